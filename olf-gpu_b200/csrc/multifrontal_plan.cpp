// Host plan of the multifrontal block LU (see multifrontal.hpp).
#include "multifrontal.hpp"

#include <algorithm>
#include <cstdint>
#include <utility>

namespace olfb200 {

namespace {

// What the targets of one node add up: the first two contributions of each, the others chained in their order of arrival.
class Sources {
public:
    void reset(int targets) {
        slot.assign(targets, Slot{});
        extra.clear();
    }
    void add(int target, int s) {
        Slot& t = slot[target];
        if (t.s0 < 0) {
            t.s0 = s;
        } else if (t.s1 < 0) {
            t.s1 = s;
        } else {
            const int e = static_cast<int>(extra.size());
            extra.push_back({s, -1});
            if (t.first < 0) t.first = e;
            else extra[t.last].next = e;
            t.last = e;
            t.more++;
        }
    }
    // A target's (s0, s1); a third and later contribution goes to `more`.
    void finish(int target, std::vector<int>& more, int& s0, int& s1) const {
        const Slot& t = slot[target];
        s0 = t.s0;
        s1 = t.s1;
        if (t.more == 0) return;
        s1 = -2 - static_cast<int>(more.size());
        more.push_back(t.more + 1);
        more.push_back(t.s1);
        for (int e = t.first; e >= 0; e = extra[e].next) more.push_back(extra[e].s);
    }

private:
    struct Slot {
        int s0 = -1, s1 = -1, first = -1, last = -1, more = 0;
    };
    struct Extra {
        int s, next;
    };
    std::vector<Slot> slot;
    std::vector<Extra> extra;
};

// First fit over a buffer that grows at its end: the free stretches by start in a tree of their largest lengths, so that the
// lowest one that is long enough is found in a few steps.
class FirstFit {
public:
    explicit FirstFit(int most) {
        while (leaves < most) leaves *= 2;
        longest.assign(2 * static_cast<size_t>(leaves), 0);
        endOf.assign(most + 1, -1);
    }
    int take(int len) {
        if (longest[1] < len) {
            const int start = end;
            end += len;
            return start;
        }
        int x = 1;
        while (x < leaves) x = longest[2 * x] >= len ? 2 * x : 2 * x + 1;
        const int start = x - leaves, have = longest[x];
        set(start, 0);
        if (have > len) set(start + len, have - len);
        return start;
    }
    void give(int start, int len) {
        if (endOf[start] >= 0) {          // the stretch that ends here
            const int before = endOf[start];
            len += start - before;
            set(before, 0);
            start = before;
        }
        const int after = longest[leaves + start + len];
        if (after > 0) {
            set(start + len, 0);
            len += after;
        }
        set(start, len);
    }
    int size() const { return end; }

private:
    int leaves = 1, end = 0;
    std::vector<int> longest;      // [1]: of all; [leaves + start]: of the stretch starting there
    std::vector<int> endOf;        // position -> start of the free stretch that ends there
    void set(int start, int len) {
        const int old = longest[leaves + start];
        if (old > 0) endOf[start + old] = -1;
        if (len > 0) endOf[start + len] = start;
        int x = leaves + start;
        longest[x] = len;
        for (x /= 2; x >= 1; x /= 2) {
            const int most = std::max(longest[2 * x], longest[2 * x + 1]);
            if (longest[x] == most) break;
            longest[x] = most;
        }
    }
};

}  // namespace

// Columns are grouped from the roots down: column k joins the node of its parent column while the node stays within
// MF_MAX_PIVOTS pivots and MF_MAX_FRONT rows and the structural zeros it takes on (the node's rows outside k's own
// pattern) are at most a third of the front.  A merge saves the column's update matrix (written and read back) and often
// a tree level, and pays for the zeros in the panel.  Columns near the leaves (fewer than MF_LEAF_LEVELS levels of the
// elimination tree below them) stay alone: there are thousands of them, and the one-pivot kernel is the cheaper one.
// A column with more than MF_MAX_BELOW rows below its pivot: no plan (such a column would be a node of its own).
MfPlan buildMfPlan(const BlockPlan& p, const std::vector<int>& nodeCol) {
    MfPlan r;
    const int nb = p.nb;
    for (int k = 0; k < nb; k++)
        if (p.uPtr[k + 1] - p.uPtr[k] - 1 > MF_MAX_BELOW) return r;
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
        // by level, (small nodes first,) panel size, number
        std::vector<std::pair<uint64_t, int>> key(nn);
        for (int t = 0; t < nn; t++) {
            const MfNode& n = r.node[t];
            const uint64_t large = smallFirst && !mfSmall(n) ? 1 : 0;
            key[t] = {(static_cast<uint64_t>(lev[t]) << 32) | (large << 31) | static_cast<uint64_t>(n.p * (n.p + 2 * n.q)), t};
        }
        std::sort(key.begin(), key.end());
        order.resize(nn);
        for (int t = 0; t < nn; t++) order[t] = key[t].second;
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
        auto size = [&](int t) { return r.node[t].q * r.node[t].q + (r.node[t].q + 1) / 2; };
        int all = 0;
        for (int t = 0; t < nn; t++) all += size(t);
        FirstFit slots(all + 1);
        for (size_t l = 0; l + 1 < r.upPtr.size(); l++) {
            for (int x = r.upPtr[l]; x < r.upPtr[l + 1]; x++) {
                const int t = r.upNode[x];
                if (size(t) > 0) r.node[t].upd = slots.take(size(t));
            }
            for (int x = r.upPtr[l]; x < r.upPtr[l + 1]; x++)
                for (int c : children[r.upNode[x]])
                    if (size(c) > 0) slots.give(r.node[c].upd, size(c));
        }
        r.updBlocks = slots.size();
    }
    // assembly: what each panel block, trailing block and right-hand-side row adds up
    r.pan.resize(nPan);
    r.trl.resize(nTrl);
    r.rhs.resize(nRows);
    std::vector<int> at(nb, -1);        // position -> front row of the node at hand
    Sources front, rhs;
    std::vector<int> out;
    for (int t = 0; t < nn; t++) {
        const MfNode& n = r.node[t];
        const int m = n.p + n.q;
        const int* rows = &r.rows[n.rows];
        for (int i = 0; i < m; i++) at[rows[i]] = i;
        front.reset(m * m);
        rhs.reset(m);
        for (int c : children[t]) {
            const MfNode& k = r.node[c];
            const int* crow = &r.rows[k.rows + k.p];
            for (int a = 0; a < k.q; a++) {
                for (int b = 0; b < k.q; b++) front.add(at[crow[a]] * m + at[crow[b]], k.upd + a * k.q + b);
                rhs.add(at[crow[a]], (k.upd + k.q * k.q) * 2 + a);
            }
        }
        out.assign(static_cast<size_t>(m) * m, -1);
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
            front.finish(i * m + j, r.more, e.s0, e.s1);
        };
        for (int k = 0; k < n.p; k++)
            for (int j = 0; j < m; j++) panel(k * m + j, k, j);
        for (int i = n.p; i < m; i++)
            for (int k = 0; k < n.p; k++) panel(n.p * m + (i - n.p) * n.p + k, i, k);
        for (int a = 0; a < n.q; a++)
            for (int b = 0; b < n.q; b++) {
                MfTrail& e = r.trl[n.trl + a * n.q + b];
                front.finish((n.p + a) * m + n.p + b, r.more, e.s0, e.s1);
            }
        for (int i = 0; i < m; i++) {
            MfRhs& e = r.rhs[n.rows + i];
            e.rowP = i < n.p ? nodeCol[2 * p.perm[rows[i]]] : -1;
            e.rowV = i < n.p ? nodeCol[2 * p.perm[rows[i]] + 1] : -1;
            rhs.finish(i, r.more, e.s0, e.s1);
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
    // the shapes that the kernels' index arithmetic and shared memory are laid out for
    for (int t = 0; t < nn; t++) {
        const MfNode& n = m.node[t];
        if (n.p < 1 || n.p > MF_MAX_PIVOTS || n.q > MF_MAX_BELOW || (n.p > 1 && n.p + n.q > MF_MAX_FRONT)) return fail("shape of node", t);
    }
    for (size_t l = 0; l < MF_LEAF_LEVELS && l + 1 < m.upPtr.size(); l++)
        for (int x = m.upPtr[l]; x < m.upPtr[l + 1]; x++)
            if (m.node[m.upNode[x]].p != 1) return fail("several pivots near the leaves, node", m.upNode[x]);
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
