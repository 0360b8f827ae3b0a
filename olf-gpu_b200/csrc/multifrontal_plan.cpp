// Host plan of the multifrontal block LU (see multifrontal.hpp).
#include "multifrontal.hpp"

#include <algorithm>
#include <map>
#include <stdexcept>

namespace olfb200 {

namespace {

// Appends one contribution to a target's (s0, s1) pair; a third and later one goes to `extra` (target -> list).
struct Sources {
    int s0 = -1, s1 = -1;
    std::vector<int> extra;
    void add(int s) {
        if (s0 < 0) s0 = s;
        else if (s1 < 0 && extra.empty()) s1 = s;
        else extra.push_back(s);
    }
};

void finish(const Sources& s, std::vector<int>& more, int& s0, int& s1) {
    s0 = s.s0;
    s1 = s.s1;
    if (s.extra.empty()) return;
    s1 = -2 - static_cast<int>(more.size());
    more.push_back(static_cast<int>(s.extra.size()) + 1);
    more.push_back(s.s1);
    more.insert(more.end(), s.extra.begin(), s.extra.end());
}

}  // namespace

// Columns are grouped from the roots down: column k joins the node of its parent column while the node stays within
// MF_MAX_PIVOTS pivots and MF_MAX_FRONT rows and the structural zeros it takes on (the node's rows outside k's own
// pattern) are at most a third of the front.  A merge saves the column's update matrix (written and read back) and often
// a tree level, and pays for the zeros in the panel.  Columns near the leaves (fewer than MF_LEAF_LEVELS levels of the
// elimination tree below them) stay alone: there are thousands of them, and the one-pivot kernel is the cheaper one.
MfPlan buildMfPlan(const BlockPlan& p, const std::vector<int>& nodeCol) {
    MfPlan r;
    const int nb = p.nb;
    std::vector<int> parentCol(nb, -1), rep(nb, -1), piv(nb, 0), below(nb, 0), height(nb, 0);
    for (int k = 0; k < nb; k++)
        if (p.uPtr[k + 1] - p.uPtr[k] > 1) {
            parentCol[k] = p.uCol[p.uPtr[k] + 1];
            height[parentCol[k]] = std::max(height[parentCol[k]], height[k] + 1);
        }
    for (int k = nb - 1; k >= 0; k--) {
        const int d = p.uPtr[k + 1] - p.uPtr[k] - 1;
        if (d > 0 && height[k] >= MF_LEAF_LEVELS) {
            const int t = rep[parentCol[k]], m = piv[t] + below[t], zeros = m - d;
            if (piv[t] < MF_MAX_PIVOTS && m < MF_MAX_FRONT && 3 * zeros <= m) {
                rep[k] = t;
                piv[t]++;
                continue;
            }
        }
        rep[k] = k;
        piv[k] = 1;
        below[k] = d;
    }
    // nodes in ascending order of their last (top) pivot: children before parents
    std::vector<int> nodeOf(nb, -1), top;
    for (int k = 0; k < nb; k++)
        if (rep[k] == k) {
            nodeOf[k] = static_cast<int>(top.size());
            top.push_back(k);
        }
    for (int k = 0; k < nb; k++) nodeOf[k] = nodeOf[rep[k]];
    const int nn = static_cast<int>(top.size());
    r.node.assign(nn, MfNode{});
    r.parent.assign(nn, -1);
    std::vector<std::vector<int>> pivots(nn), children(nn);
    for (int k = 0; k < nb; k++) pivots[nodeOf[k]].push_back(k);
    std::vector<int> up(nn, 0), down(nn, 0);
    for (int t = 0; t < nn; t++) {
        if (parentCol[top[t]] >= 0) {
            r.parent[t] = nodeOf[parentCol[top[t]]];
            children[r.parent[t]].push_back(t);
            up[r.parent[t]] = std::max(up[r.parent[t]], up[t] + 1);
        }
    }
    for (int t = nn - 1; t >= 0; t--)
        if (r.parent[t] >= 0) down[t] = down[r.parent[t]] + 1;
    int nRows = 0, nPan = 0, nTrl = 0;
    for (int t = 0; t < nn; t++) {
        MfNode& n = r.node[t];
        n.p = static_cast<int>(pivots[t].size());
        n.q = below[top[t]];
        n.rows = nRows;
        n.pan = nPan;
        n.trl = nTrl;
        n.child = children[t].empty() ? 0 : 1;
        n.u0 = p.uPtr[pivots[t][0]];
        r.rows.insert(r.rows.end(), pivots[t].begin(), pivots[t].end());
        r.rows.insert(r.rows.end(), p.uCol.begin() + p.uPtr[top[t]] + 1, p.uCol.begin() + p.uPtr[top[t] + 1]);
        nRows += n.p + n.q;
        nPan += n.p * (n.p + 2 * n.q);
        nTrl += n.q * n.q;
    }
    auto byLevel = [&](const std::vector<int>& lev, bool smallFirst, std::vector<int>& ptr, std::vector<int>& order) {
        const int nl = nn ? 1 + *std::max_element(lev.begin(), lev.end()) : 0;
        order.resize(nn);
        for (int t = 0; t < nn; t++) order[t] = t;
        auto panel = [&](int t) { return r.node[t].p * (r.node[t].p + 2 * r.node[t].q); };
        std::sort(order.begin(), order.end(), [&](int a, int b) {
            if (lev[a] != lev[b]) return lev[a] < lev[b];
            const bool sa = mfSmall(r.node[a]), sb = mfSmall(r.node[b]);
            if (smallFirst && sa != sb) return sa;
            const int pa = panel(a), pb = panel(b);
            return pa != pb ? pa < pb : a < b;
        });
        ptr.assign(nl + 1, 0);
        for (int t = 0; t < nn; t++) ptr[lev[t] + 1]++;
        for (int l = 0; l < nl; l++) ptr[l + 1] += ptr[l];
    };
    byLevel(up, false, r.upPtr, r.upNode);
    byLevel(down, true, r.downPtr, r.downNode);
    for (size_t l = 0; l + 1 < r.downPtr.size(); l++) {
        int c = 0;
        while (r.downPtr[l] + c < r.downPtr[l + 1] && mfSmall(r.node[r.downNode[r.downPtr[l] + c]])) c++;
        r.downSmall.push_back(c);
    }
    // update matrices: first fit; a slot is free again one level after the parent's (whose launch reads it)
    {
        std::map<int, int> freeAt;      // start -> length
        int end = 0;
        auto release = [&](int start, int len) {
            auto nx = freeAt.lower_bound(start);
            if (nx != freeAt.begin()) {
                auto pv = std::prev(nx);
                if (pv->first + pv->second == start) {
                    start = pv->first;
                    len += pv->second;
                    freeAt.erase(pv);
                }
            }
            if (nx != freeAt.end() && start + len == nx->first) {
                len += nx->second;
                freeAt.erase(nx);
            }
            freeAt[start] = len;
        };
        auto size = [&](int t) { return r.node[t].q * r.node[t].q + (r.node[t].q + 1) / 2; };
        for (size_t l = 0; l + 1 < r.upPtr.size(); l++) {
            for (int x = r.upPtr[l]; x < r.upPtr[l + 1]; x++) {
                const int t = r.upNode[x], len = size(t);
                if (len == 0) continue;
                auto it = freeAt.begin();
                while (it != freeAt.end() && it->second < len) ++it;
                if (it == freeAt.end()) {
                    r.node[t].upd = end;
                    end += len;
                } else {
                    const int start = it->first, have = it->second;
                    freeAt.erase(it);
                    r.node[t].upd = start;
                    if (have > len) freeAt[start + len] = have - len;
                }
            }
            for (int x = r.upPtr[l]; x < r.upPtr[l + 1]; x++)
                for (int c : children[r.upNode[x]])
                    if (size(c) > 0) release(r.node[c].upd, size(c));
        }
        r.updBlocks = end;
    }
    // assembly: what each panel block, trailing block and right-hand-side row adds up
    r.pan.resize(nPan);
    r.trl.resize(nTrl);
    r.rhs.resize(nRows);
    std::vector<int> at(nb, -1);        // position -> front row of the node at hand
    std::vector<Sources> front, rhs;
    for (int t = 0; t < nn; t++) {
        const MfNode& n = r.node[t];
        const int m = n.p + n.q;
        const int* rows = &r.rows[n.rows];
        for (int i = 0; i < m; i++) at[rows[i]] = i;
        front.assign(static_cast<size_t>(m) * m, Sources{});
        rhs.assign(m, Sources{});
        for (int c : children[t]) {
            const MfNode& k = r.node[c];
            const int* crow = &r.rows[k.rows + k.p];
            for (int a = 0; a < k.q; a++) {
                for (int b = 0; b < k.q; b++) front[at[crow[a]] * m + at[crow[b]]].add(k.upd + a * k.q + b);
                rhs[at[crow[a]]].add((k.upd + k.q * k.q) * 2 + a);
            }
        }
        std::vector<int> out(static_cast<size_t>(m) * m, -1);
        for (int k = 0; k < n.p; k++) {
            const int pos = rows[k], u0 = p.uPtr[pos];
            out[k * m + k] = u0;
            for (int x = u0 + 1; x < p.uPtr[pos + 1]; x++) {
                const int j = at[p.uCol[x]];
                out[k * m + j] = x;
                out[j * m + k] = p.nU + p.lPtr[pos] + (x - u0 - 1);
            }
        }
        auto panel = [&](int idx, int i, int j) {
            MfPanel& e = r.pan[n.pan + idx];
            e.out = out[i * m + j];
            e.aBlock = e.out >= 0 ? p.luToA[e.out] : -1;
            finish(front[i * m + j], r.more, e.s0, e.s1);
        };
        for (int k = 0; k < n.p; k++)
            for (int j = 0; j < m; j++) panel(k * m + j, k, j);
        for (int i = n.p; i < m; i++)
            for (int k = 0; k < n.p; k++) panel(n.p * m + (i - n.p) * n.p + k, i, k);
        for (int a = 0; a < n.q; a++)
            for (int b = 0; b < n.q; b++) {
                MfTrail& e = r.trl[n.trl + a * n.q + b];
                finish(front[(n.p + a) * m + n.p + b], r.more, e.s0, e.s1);
            }
        for (int i = 0; i < m; i++) {
            MfRhs& e = r.rhs[n.rows + i];
            e.rowP = i < n.p ? nodeCol[2 * p.perm[rows[i]]] : -1;
            e.rowV = i < n.p ? nodeCol[2 * p.perm[rows[i]] + 1] : -1;
            finish(rhs[i], r.more, e.s0, e.s1);
        }
        for (int i = 0; i < m; i++) at[rows[i]] = -1;
    }
    return r;
}

std::string checkMfPlan(const BlockPlan& p, const std::vector<int>& nodeCol, const MfPlan& m) {
    const int nb = p.nb, nn = static_cast<int>(m.node.size()), nLu = p.nU + p.nL;
    auto fail = [](const std::string& what, int i) { return "multifrontal: " + what + " " + std::to_string(i); };
    std::vector<int> pivotOf(nb, -1), stored(nLu, 0), upLevel(nn, -1), downLevel(nn, -1);
    std::vector<char> aSeen(p.aCol.size(), 0);
    for (int t = 0; t < nn; t++)
        for (int k = 0; k < m.node[t].p; k++) {
            const int pos = m.rows[m.node[t].rows + k];
            if (pivotOf[pos] >= 0) return fail("position eliminated twice", pos);
            pivotOf[pos] = t;
        }
    for (int k = 0; k < nb; k++)
        if (pivotOf[k] < 0) return fail("position never eliminated", k);
    for (size_t l = 0; l + 1 < m.upPtr.size(); l++)
        for (int x = m.upPtr[l]; x < m.upPtr[l + 1]; x++) upLevel[m.upNode[x]] = static_cast<int>(l);
    for (size_t l = 0; l + 1 < m.downPtr.size(); l++)
        for (int x = m.downPtr[l]; x < m.downPtr[l + 1]; x++) downLevel[m.downNode[x]] = static_cast<int>(l);
    // owner of every update block and pair while it is live: (node, level written) per slot, replayed level by level
    std::vector<int> owner(m.updBlocks, -1), readBy(m.updBlocks, -1);
    std::vector<std::vector<int>> kids(nn);
    for (int t = 0; t < nn; t++) {
        if (upLevel[t] < 0 || downLevel[t] < 0) return fail("node on no level", t);
        const int pr = m.parent[t];
        if (pr < 0) {
            if (m.node[t].q != 0) return fail("root with rows below", t);
            continue;
        }
        kids[pr].push_back(t);
        if (upLevel[pr] <= upLevel[t] || downLevel[pr] >= downLevel[t]) return fail("child not below its parent", t);
    }
    auto sources = [&](int s0, int s1) {
        std::vector<int> v;
        if (s0 >= 0) v.push_back(s0);
        if (s1 >= 0) v.push_back(s1);
        if (s1 <= -2)
            for (int x = 0; x < m.more[-2 - s1]; x++) v.push_back(m.more[-1 - s1 + x]);
        return v;
    };
    for (size_t l = 0; l + 1 < m.upPtr.size(); l++) {
        // reads of this level first: every slot must still belong to a child of the reading node
        for (int x = m.upPtr[l]; x < m.upPtr[l + 1]; x++) {
            const int t = m.upNode[x];
            const MfNode& n = m.node[t];
            const int mm = n.p + n.q;
            const int* rows = &m.rows[n.rows];
            int blocks = 0, pairs = 0;
            auto block = [&](int s, int i, int j) -> bool {     // slot s holds a child's block of rows (i, j)
                if (s < 0 || s >= m.updBlocks || owner[s] < 0 || m.parent[owner[s]] != t || readBy[s] == t) return false;
                const MfNode& c = m.node[owner[s]];
                const int e = s - c.upd, a = e / c.q, b = e % c.q;
                readBy[s] = t;
                blocks++;
                return a < c.q && m.rows[c.rows + c.p + a] == rows[i] && m.rows[c.rows + c.p + b] == rows[j];
            };
            for (int idx = 0; idx < n.p * (mm + n.q); idx++) {
                const int i = idx < n.p * mm ? idx / mm : n.p + (idx - n.p * mm) / n.p;
                const int j = idx < n.p * mm ? idx % mm : (idx - n.p * mm) % n.p;
                const MfPanel& e = m.pan[n.pan + idx];
                if (e.out >= 0) stored[e.out]++;
                if (e.aBlock >= 0) {
                    if (e.out < 0 || p.luToA[e.out] != e.aBlock || aSeen[e.aBlock]) return fail("Jacobian block of node", t);
                    aSeen[e.aBlock] = 1;
                }
                for (int s : sources(e.s0, e.s1))
                    if (!block(s, i, j)) return fail("panel source of node", t);
            }
            for (int a = 0; a < n.q; a++)
                for (int b = 0; b < n.q; b++) {
                    const MfTrail& e = m.trl[n.trl + a * n.q + b];
                    for (int s : sources(e.s0, e.s1))
                        if (!block(s, n.p + a, n.p + b)) return fail("trailing source of node", t);
                }
            for (int i = 0; i < mm; i++) {
                const MfRhs& e = m.rhs[n.rows + i];
                if (e.rowP != (i < n.p ? nodeCol[2 * p.perm[rows[i]]] : -1) ||
                    e.rowV != (i < n.p ? nodeCol[2 * p.perm[rows[i]] + 1] : -1)) {
                    return fail("right-hand side of node", t);
                }
                for (int s : sources(e.s0, e.s1)) {
                    const int o = owner[s / 2];
                    if (o < 0 || m.parent[o] != t) return fail("right-hand-side source of node", t);
                    const MfNode& c = m.node[o];
                    const int a = s - (c.upd + c.q * c.q) * 2;
                    if (a < 0 || a >= c.q || m.rows[c.rows + c.p + a] != rows[i]) return fail("right-hand-side row of node", t);
                    pairs++;
                }
            }
            int wantBlocks = 0, wantPairs = 0;
            for (int c : kids[t]) {
                wantBlocks += m.node[c].q * m.node[c].q;
                wantPairs += m.node[c].q;
            }
            if (blocks != wantBlocks || pairs != wantPairs) return fail("update blocks left out at node", t);
            if (n.child != (kids[t].empty() ? 0 : 1)) return fail("child flag of node", t);
        }
        // then its writes: no slot may still be waiting for a parent on this level or a later one
        for (int x = m.upPtr[l]; x < m.upPtr[l + 1]; x++) {
            const int t = m.upNode[x];
            const int len = m.node[t].q * m.node[t].q + (m.node[t].q + 1) / 2;
            for (int s = m.node[t].upd; s < m.node[t].upd + len; s++) {
                if (s < 0 || s >= m.updBlocks) return fail("update matrix outside the buffer, node", t);
                if (owner[s] >= 0 && upLevel[m.parent[owner[s]]] >= static_cast<int>(l)) return fail("update matrix overwritten by node", t);
                owner[s] = t;
                readBy[s] = -1;
            }
        }
    }
    for (int id = 0; id < nLu; id++)
        if (stored[id] != 1) return fail("LU block not stored once:", id);
    for (size_t a = 0; a < aSeen.size(); a++)
        if (!aSeen[a]) return fail("Jacobian block left out:", static_cast<int>(a));
    return "";
}

}  // namespace olfb200
