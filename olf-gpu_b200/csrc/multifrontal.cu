// Multifrontal form of the block LU and of its triangular solves (schedule 4's linear solve).
//
// The level kernels (kernels.cu) factorize left-looking, one 2x2 block per thread: every update reads both its operands
// from L2, 64 bytes for 16 operations, through ~120 dependent levels on the 9,241-bus plan.  Here the columns are
// grouped into the nodes of an assembly tree (multifrontal.hpp) and one launch runs a whole tree level: a node adds up
// its Jacobian blocks and its children's update matrices, eliminates its pivots and streams the Schur complement of the
// rows below to its own update matrix, each block summed in registers.  The right-hand side rides along as one more
// column, so the forward solve costs no pass of its own, and the L blocks are only stored where a later solve reads them
// (mixed precision's refinement).
//
// A thread works on two neighbouring lanes (16-byte FP64 accesses): the index arithmetic, records and addresses, which
// outnumber the FP64 instructions by far, are shared by both, and twice the bytes are in flight.  Two kinds of nodes.  Near
// the leaves there are thousands with one pivot and a few rows below it: a warp factorizes one for 64 lanes, everything in
// registers with the row count a template parameter (no shared memory, no barrier, every load of a node independent of
// the others).  Further up a CTA works on one node for G lane pairs with the pivots' panel in shared memory: thread =
// (pair g, worker).  A level with few nodes takes few pairs and many workers per pair (latency), one with many nodes small
// CTAs (their fixed latencies overlap).  Every sum has an order that does not depend on G or on the CTA's size.
//
// What bounds it: near the leaves memory (9,241 buses, 500 lanes: the first level reads and writes 0.93 GB in 0.19 ms, 5.0
// TB/s, the four after it 3.8 to 4.2 TB/s), further up the dependent loads and FP64 latencies of a node (64 lanes: 23 to 48 us a
// level; the FP64 pipe is 4 to 6 % busy, near the leaves under 10 %).
// Factorization + solves of one pass on 9,241 buses, 500 / 17 lanes: 2.68 / 1.12 ms with the level launches, 2.14 / 0.68 ms
// here; two lanes a thread took the 500-lane pass from 2.90 to 2.40 ms.
//
// The update matrices are grouped by 32 lanes, [lane group][block][4][32], so a block is one kilobyte at constant offsets.
// Lanes that are not solving are computed along with their neighbour's; nothing reads their factors or work vectors, and
// their dx, trouble and precision flags are left alone.
#include "kernels.cuh"

#include <algorithm>
#include <map>
#include <utility>

#include "multifrontal.hpp"

namespace olfb200 {

namespace {

constexpr int CTA = 256, WIDE_CTA = 512, LEAF_CTA = 128;

// Two neighbouring lanes' values.
template <typename T>
struct alignas(2 * sizeof(T)) Pair {
    T a, b;
};
template <typename T>
__device__ __forceinline__ Pair<T> fma2(const Pair<T>& x, const Pair<T>& y, const Pair<T>& z) {
    return Pair<T>{rnFma(x.a, y.a, z.a), rnFma(x.b, y.b, z.b)};
}
// z - x y
template <typename T>
__device__ __forceinline__ Pair<T> fnma2(const Pair<T>& x, const Pair<T>& y, const Pair<T>& z) {
    return Pair<T>{rnFma(-x.a, y.a, z.a), rnFma(-x.b, y.b, z.b)};
}
template <typename T>
__device__ __forceinline__ Pair<T> mul2(const Pair<T>& x, const Pair<T>& y) {
    return Pair<T>{rnMul(x.a, y.a), rnMul(x.b, y.b)};
}
template <typename T>
__device__ __forceinline__ void add2(Pair<T>& x, const Pair<T>& y) {
    x.a += y.a;
    x.b += y.b;
}

// A thread's two lanes s, s + 1 (s even) and which of them are solving.
struct Lanes {
    int s;
    bool a, b;
    __device__ __forceinline__ bool any() const { return a || b; }
};

__device__ __forceinline__ bool mfSolving(const DevBatch& b, int s) {
    return s < b.S && b.active[s] && !b.pending[s] && (!b.laneMask || b.laneMask[s]);
}
__device__ __forceinline__ Lanes lanesAt(const DevBatch& b, int s) {
    Lanes l{s, mfSolving(b, s), mfSolving(b, s + 1)};
    if (l.s >= b.S) l.s = 0;      // past the batch: any valid address (nothing is stored)
    return l;
}

template <typename T>
__device__ __forceinline__ Pair<T> ld(const T* p) {
    return *reinterpret_cast<const Pair<T>*>(p);
}
template <typename T>
__device__ __forceinline__ void st(T* p, const Pair<T>& v) {
    *reinterpret_cast<Pair<T>*>(p) = v;
}

// A lane pair's part of the update buffer.
template <typename T>
__device__ __forceinline__ T* laneUpdates(T* upd, const MfDev& mf, int s) {
    return upd + (size_t)(s >> 5) * mf.updBlocks * 128 + (s & 31);
}

// v += block blk where take is true; the loads run either way (from block 0, whose values are then left out), so that
// several of them are in flight together.
template <typename T>
__device__ __forceinline__ void addBlockIf(const T* upd, int blk, bool take, Pair<T> (&v)[4]) {
    const T* p = upd + (size_t)(take ? blk : 0) * 128;
    Pair<T> x[4];
#pragma unroll
    for (int e = 0; e < 4; e++) x[e] = ld(p + 32 * e);
    if (take) {
#pragma unroll
        for (int e = 0; e < 4; e++) add2(v[e], x[e]);
    }
}

template <typename T>
__device__ __forceinline__ void addBlock(const T* upd, int blk, Pair<T> (&v)[4]) {
    const T* p = upd + (size_t)blk * 128;
#pragma unroll
    for (int e = 0; e < 4; e++) add2(v[e], ld(p + 32 * e));
}

// The second and later children's contributions to one block.
template <typename T>
__device__ __forceinline__ void addOthers(const T* upd, const int* more, int s1, Pair<T> (&v)[4]) {
    if (s1 >= 0) addBlock(upd, s1, v);
    if (s1 <= -2) {
        const int* l = more - 2 - s1;
        const int n = l[0];
        for (int x = 1; x <= n; x++) addBlock(upd, l[x], v);
    }
}

// The children's contributions to one block (upd: the lanes' part).
template <typename T>
__device__ __forceinline__ void addSources(const T* upd, const int* more, int s0, int s1, Pair<T> (&v)[4]) {
    if (s0 >= 0) addBlock(upd, s0, v);
    addOthers(upd, more, s1, v);
}

// ... to one right-hand-side row.
template <typename T>
__device__ __forceinline__ void addRhs(const T* upd, const int* more, int s0, int s1, Pair<T> (&v)[2]) {
    auto add = [&](int s) {
        const T* p = upd + (size_t)s * 64;
        add2(v[0], ld(p));
        add2(v[1], ld(p + 32));
    };
    if (s0 >= 0) add(s0);
    if (s1 >= 0) add(s1);
    if (s1 <= -2) {
        const int* l = more - 2 - s1;
        const int n = l[0];
        for (int x = 1; x <= n; x++) add(l[x]);
    }
}

template <typename T>
__device__ __forceinline__ void storeUpdate(T* upd, int blk, const Pair<T> (&v)[4]) {
    T* p = upd + (size_t)blk * 128;
#pragma unroll
    for (int e = 0; e < 4; e++) st(p + 32 * e, v[e]);
}

template <typename T>
__device__ __forceinline__ Pair<T> ldDouble(const double* p) {
    const Pair<double> d = ld(p);
    return Pair<T>{(T)d.a, (T)d.b};
}

template <typename T>
__device__ __forceinline__ void loadJacobian(const DevBatch& b, int blk, int s, Pair<T> (&v)[4]) {
    const size_t S = b.S;
    const double* p = b.J + (size_t)blk * 4 * S + s;
    v[0] = ldDouble<T>(p);
    v[1] = ldDouble<T>(p + S);
    v[2] = ldDouble<T>(p + 2 * S);
    v[3] = ldDouble<T>(p + 3 * S);
}

template <typename T>
__device__ __forceinline__ Pair<T> loadRhs(const DevBatch& b, int row, int s) {
    const Pair<double> f = ld(b.F + (size_t)row * b.S + s);
    return Pair<T>{(T)(-f.a), (T)(-f.b)};
}

template <typename T>
__device__ __forceinline__ void storeBlock(T* p, size_t S, const Pair<T> (&v)[4]) {
    st(p, v[0]);
    st(p + S, v[1]);
    st(p + 2 * S, v[2]);
    st(p + 3 * S, v[3]);
}

// c -= l u (2x2 blocks).
template <typename T>
__device__ __forceinline__ void mulSub(Pair<T> (&c)[4], const Pair<T> (&l)[4], const Pair<T> (&u)[4]) {
    c[0] = fnma2(l[0], u[0], fnma2(l[1], u[2], c[0]));
    c[1] = fnma2(l[0], u[1], fnma2(l[1], u[3], c[1]));
    c[2] = fnma2(l[2], u[0], fnma2(l[3], u[2], c[2]));
    c[3] = fnma2(l[2], u[1], fnma2(l[3], u[3], c[3]));
}

// y -= l x (a block and a pair of rows).
template <typename T>
__device__ __forceinline__ void mulSubPair(Pair<T> (&y)[2], const Pair<T> (&l)[4], const Pair<T>& x0, const Pair<T>& x1) {
    y[0] = fnma2(l[0], x0, fnma2(l[1], x1, y[0]));
    y[1] = fnma2(l[2], x0, fnma2(l[3], x1, y[1]));
}

template <typename T>
__device__ __forceinline__ void mul(Pair<T> (&o)[4], const Pair<T> (&a)[4], const Pair<T> (&b)[4]) {
    o[0] = fma2(a[0], b[0], mul2(a[1], b[2]));
    o[1] = fma2(a[0], b[1], mul2(a[1], b[3]));
    o[2] = fma2(a[2], b[0], mul2(a[3], b[2]));
    o[3] = fma2(a[2], b[1], mul2(a[3], b[3]));
}

template <typename T>
__device__ __forceinline__ T det1(T d0, T d1, T d2, T d3) { return rnFma(d0, d3, -rnMul(d1, d2)); }

template <typename T>
__device__ __forceinline__ void invert(const Pair<T> (&d)[4], Pair<T> (&iv)[4]) {
    const T ia = (T)1 / det1(d[0].a, d[1].a, d[2].a, d[3].a), ib = (T)1 / det1(d[0].b, d[1].b, d[2].b, d[3].b);
    iv[0] = Pair<T>{d[3].a * ia, d[3].b * ib};
    iv[1] = Pair<T>{-d[1].a * ia, -d[1].b * ib};
    iv[2] = Pair<T>{-d[2].a * ia, -d[2].b * ib};
    iv[3] = Pair<T>{d[0].a * ia, d[0].b * ib};
}

template <typename T>
__device__ __forceinline__ T maxAbs(T x0, T x1, T x2, T x3) {
    return fmax(fmax(fabs(x0), fabs(x1)), fmax(fabs(x2), fabs(x3)));
}

// Flags a near-singular pivot (lu_pivot.cuh:12-18) and, in FP32, a badly conditioned or grown one (amax: max |A_kk|).
template <typename T>
__device__ __forceinline__ void checkPivot1(const DevBatch& b, int s, T d0, T d1, T d2, T d3, T amax) {
    const T det = det1(d0, d1, d2, d3);
    const T scale = fabs(d0 * d3) + fabs(d1 * d2);
    if (!(fabs(det) > (T)1e-13 * scale) || !isfinite(det)) b.trouble[s] = TROUBLE_PIVOT;
    if (sizeof(T) == 4 && b.precision64) {
        const float dmax = (float)maxAbs(d0, d1, d2, d3);
        const float kappa = dmax * dmax * fabsf((float)((T)1 / det));      // max |D| max |inv D|
        const float grow = amax > 0 ? dmax / (float)amax : 1.0f;
        if (!(kappa <= (float)b.growthLimit) || !(grow <= (float)b.growthLimit)) b.precision64[s] = 1;
    }
}
template <typename T>
__device__ __forceinline__ void checkPivot(const DevBatch& b, const Lanes& ln, const Pair<T> (&d)[4], const Pair<T>& amax) {
    if (ln.a) checkPivot1(b, ln.s, d[0].a, d[1].a, d[2].a, d[3].a, amax.a);
    if (ln.b) checkPivot1(b, ln.s + 1, d[0].b, d[1].b, d[2].b, d[3].b, amax.b);
}

__device__ __forceinline__ int4 record(const void* table, int i) { return __ldg(reinterpret_cast<const int4*>(table) + i); }

// A one-pivot node with Q rows below, two lanes (every record is the same for the warp).
template <typename T, int Q, bool STORE_L>
__device__ __forceinline__ void factorLeaf(const DevBatch& b, T* lu, T* w, size_t WS, T* us, const MfDev& mf, const MfTask& n,
                                           const Lanes& ln) {
    const size_t S = b.S;
    const int s = ln.s;
    const MfPanel* pan = mf.pan + n.pan;
    int4 ru[Q + 1];                        // the pivot's row: aBlock, out, s0, s1
#pragma unroll
    for (int c = 0; c <= Q; c++) ru[c] = record(pan, c);
    const int4 ry = record(mf.rhs + n.rows, 0);
    Pair<T> u[Q + 1][4], y[2], amax{};
#pragma unroll
    for (int c = 0; c <= Q; c++) {
#pragma unroll
        for (int e = 0; e < 4; e++) u[c][e] = Pair<T>{0, 0};
        if (ru[c].x >= 0) loadJacobian(b, ru[c].x, s, u[c]);
    }
    y[0] = loadRhs<T>(b, ry.x, s);
    y[1] = loadRhs<T>(b, ry.y, s);
    if (sizeof(T) == 4) {
        amax = Pair<T>{maxAbs(u[0][0].a, u[0][1].a, u[0][2].a, u[0][3].a), maxAbs(u[0][0].b, u[0][1].b, u[0][2].b, u[0][3].b)};
    }
    pdlWait();   // the children's update matrices (earlier levels) are read from here on
#pragma unroll
    for (int c = 0; c <= Q; c++) addSources(us, mf.more, ru[c].z, ru[c].w, u[c]);
    addRhs(us, mf.more, ry.z, ry.w, y);
    Pair<T> iv[4];
    invert(u[0], iv);
    checkPivot(b, ln, u[0], amax);
    T* uo = lu + (size_t)n.u0 * 4 * S + s;
    storeBlock(uo, S, iv);
#pragma unroll
    for (int c = 1; c <= Q; c++) storeBlock(uo + (size_t)c * 4 * S, S, u[c]);
    st(w + (size_t)(2 * n.pos) * WS, y[0]);
    st(w + (size_t)(2 * n.pos + 1) * WS, y[1]);
#pragma unroll 1
    for (int a = 0; a < Q; a++) {          // (not unrolled: the kernel's size, its instruction fetches, costs more)
        const int4 rl = record(pan, Q + 1 + a), rr = record(mf.rhs + n.rows, 1 + a);
        Pair<T> l[4], ls[4];
#pragma unroll
        for (int e = 0; e < 4; e++) l[e] = Pair<T>{0, 0};
        if (rl.x >= 0) loadJacobian(b, rl.x, s, l);
        addSources(us, mf.more, rl.z, rl.w, l);
        mul(ls, l, iv);
        if (STORE_L) storeBlock(lu + (size_t)rl.y * 4 * S + s, S, ls);
#pragma unroll
        for (int c = 0; c < Q; c++) {
            const MfTrail et = mf.trl[n.trl + a * Q + c];
            Pair<T> v[4];
#pragma unroll
            for (int e = 0; e < 4; e++) v[e] = Pair<T>{0, 0};
            addSources(us, mf.more, et.s0, et.s1, v);
            mulSub(v, ls, u[1 + c]);
            storeUpdate(us, n.upd + a * Q + c, v);
        }
        Pair<T> r[2] = {{0, 0}, {0, 0}};
        addRhs(us, mf.more, rr.z, rr.w, r);
        mulSubPair(r, ls, y[0], y[1]);
        T* ro = us + (size_t)(n.upd + Q * Q) * 128 + a * 64;
        st(ro, r[0]);
        st(ro + 32, r[1]);
    }
}

// One row below the pivot of a node with many, two lanes: the pivot and its U row are added up for every row (L1 hits).
template <typename T, bool STORE_L>
__device__ __forceinline__ void factorRow(const DevBatch& b, T* lu, T* w, size_t WS, T* us, const MfDev& mf, const MfTask& n,
                                          const Lanes& ln) {
    const size_t S = b.S;
    const int q = n.q, a = n.row, s = ln.s;
    const MfPanel* pan = mf.pan + n.pan;
    const int4 ed = record(pan, 0), el = record(pan, q + 1 + a), er = record(mf.rhs + n.rows, 0);
    Pair<T> d[4], l[4], y[2], amax{};
#pragma unroll
    for (int e = 0; e < 4; e++) d[e] = l[e] = Pair<T>{0, 0};
    if (ed.x >= 0) loadJacobian(b, ed.x, s, d);
    if (el.x >= 0) loadJacobian(b, el.x, s, l);
    y[0] = loadRhs<T>(b, er.x, s);
    y[1] = loadRhs<T>(b, er.y, s);
    if (sizeof(T) == 4) amax = Pair<T>{maxAbs(d[0].a, d[1].a, d[2].a, d[3].a), maxAbs(d[0].b, d[1].b, d[2].b, d[3].b)};
    pdlWait();   // the children's update matrices (earlier levels) are read from here on
    addSources(us, mf.more, ed.z, ed.w, d);
    addSources(us, mf.more, el.z, el.w, l);
    addRhs(us, mf.more, er.z, er.w, y);
    Pair<T> iv[4], ls[4];
    invert(d, iv);
    if (a == 0) {
        checkPivot(b, ln, d, amax);
        storeBlock(lu + (size_t)n.u0 * 4 * S + s, S, iv);
        st(w + (size_t)(2 * n.pos) * WS, y[0]);
        st(w + (size_t)(2 * n.pos + 1) * WS, y[1]);
    }
    mul(ls, l, iv);
    if (STORE_L) storeBlock(lu + (size_t)el.y * 4 * S + s, S, ls);
#pragma unroll 2
    for (int c = 0; c < q; c++) {
        const int4 eu = record(pan, 1 + c);
        const MfTrail et = mf.trl[n.trl + a * q + c];
        Pair<T> u[4], v[4];
#pragma unroll
        for (int e = 0; e < 4; e++) u[e] = v[e] = Pair<T>{0, 0};
        if (eu.x >= 0) loadJacobian(b, eu.x, s, u);
        addSources(us, mf.more, eu.z, eu.w, u);
        addSources(us, mf.more, et.s0, et.s1, v);
        if (a == 0) storeBlock(lu + (size_t)(n.u0 + 1 + c) * 4 * S + s, S, u);
        mulSub(v, ls, u);
        storeUpdate(us, n.upd + a * q + c, v);
    }
    const int4 ea = record(mf.rhs + n.rows, 1 + a);
    Pair<T> r[2] = {{0, 0}, {0, 0}};
    addRhs(us, mf.more, ea.z, ea.w, r);
    mulSubPair(r, ls, y[0], y[1]);
    T* ro = us + (size_t)(n.upd + q * q) * 128 + a * 64;
    st(ro, r[0]);
    st(ro + 32, r[1]);
}

// A solution entry of both lanes: the work vector, and dx where the lane is solving.
template <typename T>
__device__ __forceinline__ void storeDx(const DevBatch& b, const Lanes& ln, int row, const Pair<T>& x) {
    double* p = b.dx + (size_t)row * b.S + ln.s;
    if (ln.a && ln.b) {
        st(p, Pair<double>{(double)x.a, (double)x.b});
    } else {
        if (ln.a) p[0] = (double)x.a;
        if (ln.b) p[1] = (double)x.b;
    }
}

// x of a small node, two lanes: inv(D) (y - sum_j U(0, j) x_j).
template <typename T>
__device__ __forceinline__ void backwardRow(const DevBatch& b, const T* lu, T* w, size_t WS, const MfDev& mf, int node,
                                            const Lanes& ln) {
    const size_t S = b.S;
    const int s = ln.s;
    const MfNode n = mf.down[node];
    const int q = n.q;
    const int* rows = mf.rows + n.rows;
    const size_t pos = rows[0];
    const T* u = lu + (size_t)n.u0 * 4 * S + s;
    Pair<T> iv[4] = {ld(u), ld(u + S), ld(u + 2 * S), ld(u + 3 * S)};
    Pair<T> y[2] = {ld(w + (2 * pos) * WS), ld(w + (2 * pos + 1) * WS)};
    const MfRhs er = mf.rhs[n.rows];
    pdlWait();   // the ancestors' solution entries are read from here on
#pragma unroll 4
    for (int j = 1; j <= q; j++) {
        const T* uj = u + (size_t)j * 4 * S;
        const Pair<T> ub[4] = {ld(uj), ld(uj + S), ld(uj + 2 * S), ld(uj + 3 * S)};
        const T* x = w + (size_t)(2 * rows[j]) * WS;
        mulSubPair(y, ub, ld(x), ld(x + WS));
    }
    const Pair<T> x0 = fma2(iv[0], y[0], mul2(iv[1], y[1])), x1 = fma2(iv[2], y[0], mul2(iv[3], y[1]));
    st(w + (2 * pos) * WS, x0);
    st(w + (2 * pos + 1) * WS, x1);
    storeDx(b, ln, er.rowP, x0);
    storeDx(b, ln, er.rowV, x1);
}

// t / d for t d < 65536, r = (65535 + d) / d.
__device__ __forceinline__ int smallDiv(int t, unsigned r) { return (int)(((unsigned)t * r) >> 16); }

// Shared-memory blocks of G lane pairs: four rows of G pairs, padded by a fifth row where a row is shorter than a line of
// banks, so that consecutive blocks fall into different banks.
template <typename T, int G>
constexpr int blockStride() { return G * 2 * (int)sizeof(T) >= 128 ? 4 * G : 5 * G; }

template <int G, typename T>
__device__ __forceinline__ void ldBlock(const Pair<T>* M, int blk, Pair<T> (&v)[4]) {
    const Pair<T>* p = M + blk * blockStride<T, G>();
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] = p[e * G];
}

template <int G, typename T>
__device__ __forceinline__ void stBlock(Pair<T>* M, int blk, const Pair<T> (&v)[4]) {
    Pair<T>* p = M + blk * blockStride<T, G>();
#pragma unroll
    for (int e = 0; e < 4; e++) p[e * G] = v[e];
}

__device__ __forceinline__ void prefetch(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// One node, G lane pairs, one CTA: assembly, elimination, Schur complement.  sm: the panel's blocks, the pivots' inverses
// [p], the right-hand side [p][2], (FP32) the pivots' max |A_kk| [p].
template <typename T, int G, bool STORE_L>
__device__ __forceinline__ void factorNode(const DevBatch& b, T* lu, T* w, size_t WS, T* us, const MfDev& mf, int node,
                                           const Lanes& ln, Pair<T>* sm) {
    const int W = (int)blockDim.x / G;
    const int worker = (int)threadIdx.x / G, g = (int)threadIdx.x % G, s = ln.s;
    const size_t S = b.S;
    const MfNode n = mf.up[node];
    const int p = n.p, q = n.q, m = p + q, nPan = p * (m + q);
    const MfPanel* pan = mf.pan + n.pan;
    constexpr int BS = blockStride<T, G>();
    Pair<T>* M = sm + g;
    Pair<T>* IV = M + nPan * BS;
    Pair<T>* Y = IV + p * BS;
    Pair<T>* amaxS = Y + p * 2 * G;
    const Pair<T> zero{0, 0};
    constexpr int D = 2;
    // before the previous level is waited for: the Jacobian's part, two blocks in flight, and the records used later
    // brought near
    for (int t0 = worker; t0 < nPan; t0 += D * W) {
        int a[D];
        Pair<T> v[D][4];
#pragma unroll
        for (int x = 0; x < D; x++) a[x] = t0 + x * W < nPan ? pan[t0 + x * W].aBlock : -1;
#pragma unroll
        for (int x = 0; x < D; x++) loadJacobian(b, a[x] >= 0 ? a[x] : 0, s, v[x]);
#pragma unroll
        for (int x = 0; x < D; x++) {
            const int t = t0 + x * W;
            if (t >= nPan) break;
            if (a[x] < 0) v[x][0] = v[x][1] = v[x][2] = v[x][3] = zero;
            stBlock<G>(M, t, v[x]);
            if (sizeof(T) == 4 && t < p * m && t % m == t / m) {
                amaxS[(t / m) * G] = Pair<T>{maxAbs(v[x][0].a, v[x][1].a, v[x][2].a, v[x][3].a),
                                             maxAbs(v[x][0].b, v[x][1].b, v[x][2].b, v[x][3].b)};
            }
        }
    }
    for (int i = worker; i < p; i += W) {
        const MfRhs e = mf.rhs[n.rows + i];
        Y[(2 * i) * G] = loadRhs<T>(b, e.rowP, s);
        Y[(2 * i + 1) * G] = loadRhs<T>(b, e.rowV, s);
    }
    const MfTrail* trl = mf.trl + n.trl;
    for (int t = (int)threadIdx.x * 16; t < q * q; t += (int)blockDim.x * 16) prefetch(trl + t);
    for (int t = (int)threadIdx.x * 8; t < m; t += (int)blockDim.x * 8) prefetch(mf.rhs + n.rows + t);
    pdlWait();   // the children's update matrices (earlier levels) are read from here on
    if (n.child) {
        for (int t0 = worker; t0 < nPan; t0 += D * W) {
            int2 e[D];
            Pair<T> v[D][4];
#pragma unroll
            for (int x = 0; x < D; x++) {
                e[x] = make_int2(-1, -1);
                if (t0 + x * W < nPan) e[x] = make_int2(pan[t0 + x * W].s0, pan[t0 + x * W].s1);
            }
#pragma unroll
            for (int x = 0; x < D; x++) {
                v[x][0] = v[x][1] = v[x][2] = v[x][3] = zero;
                addBlockIf(us, e[x].x, e[x].x >= 0, v[x]);
            }
#pragma unroll
            for (int x = 0; x < D; x++) {
                if (e[x].x < 0) continue;
                if (e[x].y != -1) addOthers(us, mf.more, e[x].y, v[x]);
                Pair<T> o[4];
                ldBlock<G>(M, t0 + x * W, o);
#pragma unroll
                for (int c = 0; c < 4; c++) add2(o[c], v[x][c]);
                stBlock<G>(M, t0 + x * W, o);
            }
        }
        for (int i = worker; i < p; i += W) {
            const MfRhs e = mf.rhs[n.rows + i];
            Pair<T> y[2] = {zero, zero};
            addRhs(us, mf.more, e.s0, e.s1, y);
            add2(Y[(2 * i) * G], y[0]);
            add2(Y[(2 * i + 1) * G], y[1]);
        }
    }
    __syncthreads();
    if (worker == 0) {
        Pair<T> d[4], iv[4];
        ldBlock<G>(M, 0, d);
        invert(d, iv);
        stBlock<G>(IV, 0, iv);
    }
    // the pivots, right-looking within the panel, one barrier each: a task scales its row's L block for itself (the panel
    // keeps the unscaled column) and updates two blocks behind the pivot; worker 0 starts with the next pivot's row and
    // inverts that pivot
    for (int k = 0; k + 1 < p; k++) {
        __syncthreads();
        const int left = p - 1 - k, wide = m - 1 - k, hw = (wide + 1) >> 1, hl = (left + 1) >> 1;
        const unsigned rw = (65535u + hw) / hw, rl = (65535u + hl) / hl;
        const int nWide = left * hw, nAll = nWide + q * hl;
        Pair<T> iv[4];
        ldBlock<G>(IV, k, iv);
        for (int t = worker; t < nAll; t += W) {
            const bool wideRow = t < nWide;
            const int tt = wideRow ? t : t - nWide;
            const int i = smallDiv(tt, wideRow ? rw : rl);
            const int j = k + 1 + 2 * (tt - i * (wideRow ? hw : hl));
            const int row = wideRow ? (k + 1 + i) * m : p * m + i * p;
            const bool two = j + 1 < (wideRow ? m : p);
            Pair<T> l[4], ls[4], u[4], x[4];
            ldBlock<G>(M, row + k, l);
            ldBlock<G>(M, k * m + j, u);
            ldBlock<G>(M, row + j, x);
            mul(ls, l, iv);
            mulSub(x, ls, u);
            stBlock<G>(M, row + j, x);
            if (t == 0) {          // block (k + 1, k + 1) is final
                Pair<T> nx[4];
                invert(x, nx);
                stBlock<G>(IV, k + 1, nx);
            }
            if (two) {
                ldBlock<G>(M, k * m + j + 1, u);
                ldBlock<G>(M, row + j + 1, x);
                mulSub(x, ls, u);
                stBlock<G>(M, row + j + 1, x);
            }
        }
        // the right-hand side, from the last worker down
        for (int i = k + W - worker; i < p; i += W) {
            Pair<T> c[4], l[4];
            ldBlock<G>(M, i * m + k, c);
            mul(l, c, iv);
            Pair<T> y[2] = {Y[(2 * i) * G], Y[(2 * i + 1) * G]};
            mulSubPair(y, l, Y[(2 * k) * G], Y[(2 * k + 1) * G]);
            Y[(2 * i) * G] = y[0];
            Y[(2 * i + 1) * G] = y[1];
        }
    }
    __syncthreads();
    // the L blocks scaled, every one at once
    for (int t = worker; t < q * p; t += W) {
        const int k = t % p;
        Pair<T> c[4], iv[4], l[4];
        ldBlock<G>(M, p * m + t, c);
        ldBlock<G>(IV, k, iv);
        mul(l, c, iv);
        stBlock<G>(M, p * m + t, l);
    }
    __syncthreads();
    if (!ln.any()) return;
    // the U rows (and the L blocks) to the factor storage, y to the solve's work vector
    const int nOut = STORE_L ? nPan : p * m;
    const unsigned rm = (65535u + m) / m;
#pragma unroll 2
    for (int t = worker; t < nOut; t += W) {
        const int k = smallDiv(t, rm), j = t - k * m;
        const bool upper = t < p * m;
        if (upper && !STORE_L && j < k) continue;
        const int id = pan[t].out;
        if (id < 0) continue;
        Pair<T> v[4];
        ldBlock<G>(M, t, v);
        if (upper && j == k) {
            checkPivot(b, ln, v, sizeof(T) == 4 ? amaxS[k * G] : zero);
            ldBlock<G>(IV, k, v);
        } else if (upper && j < k) {      // the pivot block's L part, row k, column j
            Pair<T> iv[4], c[4];
            ldBlock<G>(IV, j, iv);
            ldBlock<G>(M, t, c);
            mul(v, c, iv);
        }
        storeBlock(lu + (size_t)id * 4 * S + s, S, v);
    }
    for (int i = worker; i < p; i += W) {
        const size_t pos = mf.rows[n.rows + i];
        st(w + (2 * pos) * WS, Y[(2 * i) * G]);
        st(w + (2 * pos + 1) * WS, Y[(2 * i + 1) * G]);
    }
    // the Schur complement: two blocks of a worker at a time, summed in registers
    const unsigned rq = q > 0 ? (65535u + q) / q : 0;
    constexpr int N = 2;
    for (int t0 = worker; t0 < q * q; t0 += N * W) {
        MfTrail e[N];
        int lc[N], ub[N];
        Pair<T> v[N][4];
#pragma unroll
        for (int x = 0; x < N; x++) {
            const int t = t0 + x * W < q * q ? t0 + x * W : t0;
            const int a = smallDiv(t, rq);
            e[x] = trl[t];
            lc[x] = p * m + a * p;
            ub[x] = p + t - a * q;
        }
#pragma unroll
        for (int x = 0; x < N; x++) {
            v[x][0] = v[x][1] = v[x][2] = v[x][3] = zero;
            addBlockIf(us, e[x].s0, e[x].s0 >= 0, v[x]);
        }
#pragma unroll
        for (int x = 0; x < N; x++)
            if (e[x].s1 != -1) addOthers(us, mf.more, e[x].s1, v[x]);
        for (int k = 0; k < p; k++) {
#pragma unroll
            for (int x = 0; x < N; x++) {
                Pair<T> l[4], u[4];
                ldBlock<G>(M, lc[x] + k, l);
                ldBlock<G>(M, k * m + ub[x], u);
                mulSub(v[x], l, u);
            }
        }
#pragma unroll
        for (int x = 0; x < N; x++)
            if (t0 + x * W < q * q) storeUpdate(us, n.upd + t0 + x * W, v[x]);
    }
    T* ro = us + (size_t)(n.upd + q * q) * 128;
    for (int a = worker; a < q; a += W) {
        const MfRhs e = mf.rhs[n.rows + p + a];
        Pair<T> y[2] = {zero, zero};
        addRhs(us, mf.more, e.s0, e.s1, y);
        for (int k = 0; k < p; k++) {
            Pair<T> l[4];
            ldBlock<G>(M, p * m + a * p + k, l);
            mulSubPair(y, l, Y[(2 * k) * G], Y[(2 * k + 1) * G]);
        }
        st(ro + a * 64, y[0]);
        st(ro + a * 64 + 32, y[1]);
    }
}

// Strands a pivot row's columns below the pivots are split into (partial sums added in strand order).
__host__ __device__ constexpr int backwardStrands(int q) { return q <= 4 ? 1 : q <= 8 ? 2 : q <= 16 ? 4 : 8; }

// The backward substitution of one node, G lane pairs, one CTA: the rows below its pivots are solved.  Their columns first
// (every pivot row and strand at once), then the pivot block is swept from its last row up.  sm: the pivot block [p][p], x
// of the front [m][2], partial sums [strands][p][2].
template <typename T, int G>
__device__ __forceinline__ void backwardNode(const DevBatch& b, const T* lu, T* wv, size_t WS, const MfDev& mf, int node,
                                             const Lanes& ln, Pair<T>* sm) {
    const int W = (int)blockDim.x / G;
    const int worker = (int)threadIdx.x / G, g = (int)threadIdx.x % G, s = ln.s;
    const size_t S = b.S;
    const MfNode n = mf.down[node];
    const int p = n.p, q = n.q, m = p + q;
    const MfPanel* pan = mf.pan + n.pan;
    const int* rows = mf.rows + n.rows;
    Pair<T>* D = sm + g;
    Pair<T>* X = D + p * p * blockStride<T, G>();
    Pair<T>* part = X + m * 2 * G;
    const Pair<T> zero{0, 0};
    const unsigned rp = (65535u + p) / p;
#pragma unroll 2
    for (int t = worker; t < p * p; t += W) {
        const int k = smallDiv(t, rp), j = t - k * p;
        const int id = j >= k ? pan[k * m + j].out : -1;
        Pair<T> v[4] = {zero, zero, zero, zero};
        if (id >= 0) {
            const T* u = lu + (size_t)id * 4 * S + s;
            v[0] = ld(u);
            v[1] = ld(u + S);
            v[2] = ld(u + 2 * S);
            v[3] = ld(u + 3 * S);
        }
        stBlock<G>(D, t, v);
    }
    for (int i = worker; i < p; i += W) {
        const T* w = wv + (size_t)(2 * rows[i]) * WS;
        X[(2 * i) * G] = ld(w);
        X[(2 * i + 1) * G] = ld(w + WS);
    }
    pdlWait();   // the ancestors' solution entries are read from here on
    for (int i = p + worker; i < m; i += W) {
        const T* w = wv + (size_t)(2 * rows[i]) * WS;
        X[(2 * i) * G] = ld(w);
        X[(2 * i + 1) * G] = ld(w + WS);
    }
    __syncthreads();
    const int C = backwardStrands(q);
    for (int t = worker; t < p * C; t += W) {
        const int c = smallDiv(t, rp), k = t - c * p;
        Pair<T> a[2] = {zero, zero};
#pragma unroll 2
        for (int j = p + c; j < m; j += C) {
            const int id = pan[k * m + j].out;
            if (id >= 0) {
                const T* u = lu + (size_t)id * 4 * S + s;
                const Pair<T> ub[4] = {ld(u), ld(u + S), ld(u + 2 * S), ld(u + 3 * S)};
                mulSubPair(a, ub, X[(2 * j) * G], X[(2 * j + 1) * G]);
            }
        }
        part[(2 * t) * G] = a[0];
        part[(2 * t + 1) * G] = a[1];
    }
    __syncthreads();
    for (int k = worker; k < p; k += W) {
        Pair<T> y0 = X[(2 * k) * G], y1 = X[(2 * k + 1) * G];
        for (int c = 0; c < C; c++) {
            add2(y0, part[(2 * (c * p + k)) * G]);
            add2(y1, part[(2 * (c * p + k) + 1) * G]);
        }
        X[(2 * k) * G] = y0;
        X[(2 * k + 1) * G] = y1;
    }
    for (int k = p - 1; k >= 0; k--) {
        __syncthreads();
        Pair<T> d[4];
        ldBlock<G>(D, k * p + k, d);
        const Pair<T> y0 = X[(2 * k) * G], y1 = X[(2 * k + 1) * G];
        const Pair<T> x0 = fma2(d[0], y0, mul2(d[1], y1)), x1 = fma2(d[2], y0, mul2(d[3], y1));
        for (int i = worker; i < k; i += W) {
            Pair<T> u[4];
            ldBlock<G>(D, i * p + k, u);
            Pair<T> y[2] = {X[(2 * i) * G], X[(2 * i + 1) * G]};
            mulSubPair(y, u, x0, x1);
            X[(2 * i) * G] = y[0];
            X[(2 * i + 1) * G] = y[1];
        }
        if (worker == W - 1 && ln.any()) {
            const MfRhs e = mf.rhs[n.rows + k];
            T* w = wv + (size_t)(2 * rows[k]) * WS;
            st(w, x0);
            st(w + WS, x1);
            storeDx(b, ln, e.rowP, x0);
            storeDx(b, ln, e.rowV, x1);
        }
    }
}

template <typename T, int G, bool FACTOR, bool STORE_L>
__device__ __forceinline__ void runTeam(const DevBatch& b, T* lu, T* wv, T* upd, const MfDev& mf, const MfSegment& sg,
                                        int cta, unsigned char* smem) {
    const int unit = cta / sg.groups, group = cta - unit * sg.groups;     // lane groups fastest
    const Lanes ln = lanesAt(b, 2 * (group * G + (int)threadIdx.x % G));
    if (!__syncthreads_or(ln.any())) {
        pdlWait();
        return;
    }
    Pair<T>* sm = reinterpret_cast<Pair<T>*>(smem);
    T* w = wv + ln.s;
    if (FACTOR) factorNode<T, G, STORE_L>(b, lu, w, b.S, laneUpdates(upd, mf, ln.s), mf, sg.first + unit, ln, sm);
    else backwardNode<T, G>(b, lu, w, b.S, mf, sg.first + unit, ln, sm);
}

template <typename T, bool STORE_L>
__device__ __forceinline__ void factorTask(const DevBatch& b, T* lu, T* w, size_t WS, T* us, const MfDev& mf, const MfTask& n,
                                           const Lanes& ln) {
    if (n.row >= 0) factorRow<T, STORE_L>(b, lu, w, WS, us, mf, n, ln);
    else if (n.q == 0) factorLeaf<T, 0, STORE_L>(b, lu, w, WS, us, mf, n, ln);
    else if (n.q == 1) factorLeaf<T, 1, STORE_L>(b, lu, w, WS, us, mf, n, ln);
    else if (n.q == 2) factorLeaf<T, 2, STORE_L>(b, lu, w, WS, us, mf, n, ln);
    else factorLeaf<T, MF_WARP_ROWS, STORE_L>(b, lu, w, WS, us, mf, n, ln);
}

// A leaf level's tasks, or a backward level's small nodes: a warp's 64 lanes on one, consecutive warps consecutive tasks,
// lane groups slowest.
template <typename T, bool FACTOR, bool STORE_L>
__device__ __forceinline__ void runTask(const DevBatch& b, T* lu, T* wv, T* upd, const MfDev& mf, const MfLevel& lv, int cta) {
    const int warps = blockDim.x >> 5, per = (lv.taskCount + warps - 1) / warps;
    int group = cta / per;
    const int k = (cta - group * per) * warps + (threadIdx.x >> 5);
    if (lv.reverse) group = (b.S + 63) / 64 - 1 - group;      // what the previous level wrote last is still in L2
    const Lanes ln = lanesAt(b, group * 64 + 2 * (threadIdx.x & 31));
    if (k >= lv.taskCount || !ln.any()) {
        pdlWait();
        return;
    }
    if (FACTOR) factorTask<T, STORE_L>(b, lu, wv + ln.s, b.S, laneUpdates(upd, mf, ln.s), mf, mf.task[lv.taskFirst + k], ln);
    else backwardRow<T>(b, lu, wv + ln.s, b.S, mf, lv.taskFirst + k, ln);
}

template <typename T, bool STORE_L>
__global__ void __launch_bounds__(LEAF_CTA, 4) mfLeafKernel(DevBatch b, T* lu, T* wv, T* upd, MfDev mf, MfLevel lv) {
    pdlTrigger();
    runTask<T, true, STORE_L>(b, lu, wv, upd, mf, lv, blockIdx.x);
}

// A level's CTA nodes, then (backward) its small nodes.
template <typename T, bool FACTOR, bool STORE_L, int MAX_THREADS>
__global__ void __launch_bounds__(MAX_THREADS, 512 / MAX_THREADS) mfLevelKernel(DevBatch b, T* lu, T* wv, T* upd, MfDev mf,
                                                                                 MfLevel lv) {
    extern __shared__ __align__(16) unsigned char mfSmem[];
    pdlTrigger();
    int cta = blockIdx.x;
    if (!FACTOR && cta >= lv.teamCtas) {
        runTask<T, false, false>(b, lu, wv, upd, mf, lv, cta - lv.teamCtas);
        return;
    }
    int x = 0;
    while (x + 1 < lv.segments && cta >= lv.seg[x].count * lv.seg[x].groups) {
        cta -= lv.seg[x].count * lv.seg[x].groups;
        x++;
    }
    const MfSegment sg = lv.seg[x];
    switch (sg.pairs) {
        case 16:   // FP32 only
            if (sizeof(T) == 4) runTeam<T, sizeof(T) == 4 ? 16 : 8, FACTOR, STORE_L>(b, lu, wv, upd, mf, sg, cta, mfSmem);
            break;
        case 8: runTeam<T, 8, FACTOR, STORE_L>(b, lu, wv, upd, mf, sg, cta, mfSmem); break;
        case 4: runTeam<T, 4, FACTOR, STORE_L>(b, lu, wv, upd, mf, sg, cta, mfSmem); break;
        case 2: runTeam<T, 2, FACTOR, STORE_L>(b, lu, wv, upd, mf, sg, cta, mfSmem); break;
        default: runTeam<T, 1, FACTOR, STORE_L>(b, lu, wv, upd, mf, sg, cta, mfSmem); break;
    }
}

template <typename T, bool FACTOR, bool STORE_L>
void launchLevels(const DevBatch& b, T* lu, T* wv, T* upd, const MfDev& mf, const std::vector<MfLevel>& levels,
                  cudaStream_t st) {
    for (size_t l = 0; l < levels.size(); l++) {
        const MfLevel& lv = levels[l];
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(lv.teamCtas + lv.taskCtas);
        cfg.blockDim = dim3(lv.threads);
        cfg.dynamicSmemBytes = lv.smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        // the first level is a normal launch: its reads before pdlWait (the Jacobian; the factors) are final then, and
        // stay so for the levels after it
        cfg.attrs = attr;
        cfg.numAttrs = l == 0 ? 0 : 1;
        if (FACTOR && lv.teamCtas == 0) cudaLaunchKernelEx(&cfg, mfLeafKernel<T, STORE_L>, b, lu, wv, upd, mf, lv);
        else if (lv.threads > CTA) cudaLaunchKernelEx(&cfg, mfLevelKernel<T, FACTOR, STORE_L, WIDE_CTA>, b, lu, wv, upd, mf, lv);
        else cudaLaunchKernelEx(&cfg, mfLevelKernel<T, FACTOR, STORE_L, CTA>, b, lu, wv, upd, mf, lv);
    }
}

constexpr int teamBytes(int p, int q, int G, int elem, bool factor) {
    const int m = p + q, bs = G * 2 * elem >= 128 ? 4 : 5;
    if (factor) return ((p * (m + q) + p) * bs + p * 3) * G * 2 * elem;
    return (p * p * bs + m * 2 + backwardStrands(q) * p * 2) * G * 2 * elem;
}
int teamBytes(const MfNode& n, int G, int elem, bool factor) { return teamBytes(n.p, n.q, G, elem, factor); }

// A plan's largest fronts (MF_MAX_PIVOTS pivots of MF_MAX_FRONT rows; one pivot over MF_MAX_BELOW) fit a CTA at one lane pair,
// and their block numbers stay in smallDiv's range.
constexpr bool frontFits(int p, int q) {
    return teamBytes(p, q, 1, 8, true) <= MF_MAX_BYTES && teamBytes(p, q, 1, 8, false) <= MF_MAX_BYTES &&
           p * (p + 2 * q) * (p + q) < 65536 && q * q * q < 65536;
}
static_assert(frontFits(MF_MAX_PIVOTS, MF_MAX_FRONT - MF_MAX_PIVOTS) && frontFits(1, MF_MAX_BELOW), "front limits");

}  // namespace

MfSchedule scheduleMf(const MfPlan& plan, const std::vector<int>& taskPtr, int nS, int S, int share, bool fp32,
                      bool factor) {
    constexpr int SMS = 148;      // B200's; only the launches' shapes follow it, no result does
    MfSchedule r;
    const std::vector<int>& ptr = factor ? plan.upPtr : plan.downPtr;
    const std::vector<int>& order = factor ? plan.upNode : plan.downNode;
    const int elem = fp32 ? 4 : 8, top = fp32 ? 16 : 8, whole = fp32 ? 4 : 2;   // whole: pairs of a sector
    const int nP = (nS + 1) / 2;
    for (size_t l = 0; l + 1 < ptr.size(); l++) {
        MfLevel lv{};
        if (factor && l + 1 < taskPtr.size()) {       // a leaf level: warps only
            lv.taskFirst = taskPtr[l];
            lv.taskCount = taskPtr[l + 1] - taskPtr[l];
            lv.threads = LEAF_CTA;
            lv.taskCtas = (lv.taskCount + LEAF_CTA / 32 - 1) / (LEAF_CTA / 32) * ((S + 63) / 64);
            lv.reverse = l & 1;
            r.levels.push_back(lv);
            continue;
        }
        const int firstTeam = ptr[l] + (factor ? 0 : plan.downSmall[l]);
        lv.taskFirst = ptr[l];
        lv.taskCount = firstTeam - ptr[l];
        // Pairs and threads per CTA: from wide CTAs down to single warps, until the level's threads fit the GPU at once (512
        // to an SM) or the CTAs are single warps; a CTA's share of shared memory goes with its threads.  Per width as many
        // pairs as the batch, the share (at least whole sectors) and a CTA for every SM allow.  Factorization + solves per
        // pass on 9,241 buses, 500 / 62 / 17 lanes: 2.14 / 0.81 / 0.68 ms; with 2,048 threads to an SM 2.42 / 0.93 / 0.75,
        // with 256 2.17 / 0.88 / 0.73; with two CTAs for every SM 2.17 / 0.83 / 0.68, with one for every other 2.15 / 0.82 /
        // 0.71.
        int cap = 1;
        auto pairs = [&](const MfNode& n, int most) {
            int G = most;
            while (G > whole && teamBytes(n, G, elem, factor) > MF_SHARE_BYTES * std::min(lv.threads, CTA) / CTA) G /= 2;
            while (G > 1 && teamBytes(n, G, elem, factor) > MF_SHARE_BYTES) G /= 2;
            return G;
        };
        std::map<std::pair<int, int>, std::pair<int, int>> shapes;      // (p, q): a node of that shape, how many
        for (int x = firstTeam; x < ptr[l + 1]; x++) {
            const MfNode& n = plan.node[order[x]];
            auto& e = shapes[{n.p, n.q}];
            e.first = order[x];
            e.second++;
        }
        auto ctas = [&] {
            long c = 0;
            for (const auto& e : shapes) {
                const int G = pairs(plan.node[e.second.first], cap);
                c += (long)e.second.second * ((nP + G - 1) / G);
            }
            return c;
        };
        const MfNode* largest = firstTeam < ptr[l + 1] ? &plan.node[order[ptr[l + 1] - 1]] : nullptr;
        for (lv.threads = WIDE_CTA;; lv.threads /= 2) {
            for (cap = 1; cap < top && cap < nP;) cap *= 2;
            while (cap > 1 && ctas() < SMS / share) cap /= 2;
            if (lv.threads == 32 || ctas() * lv.threads <= SMS * 512L / share) break;
            // (the largest panel, at whole sectors, would take more than the narrower CTAs' share)
            if (lv.threads <= CTA && largest && teamBytes(*largest, std::min(cap, whole), elem, factor) > MF_SHARE_BYTES * (lv.threads / 2) / CTA) break;
        }
        for (int x = firstTeam; x < ptr[l + 1]; x++) {
            const MfNode& n = plan.node[order[x]];
            // (never more pairs than the smaller panels before it: one segment per count)
            const int G = pairs(n, lv.segments ? std::min(cap, lv.seg[lv.segments - 1].pairs) : cap);
            const int bytes = teamBytes(n, G, elem, factor);
            MfSegment* sg = lv.segments ? &lv.seg[lv.segments - 1] : nullptr;
            if (!sg || sg->pairs != G) {
                sg = &lv.seg[lv.segments++];
                *sg = MfSegment{x, 0, G, (nP + G - 1) / G};
            }
            sg->count++;
            lv.teamCtas += sg->groups;
            lv.smem = std::max(lv.smem, bytes);
        }
        if (lv.teamCtas == 0 || (lv.taskCount > 0 && lv.threads > CTA)) lv.threads = CTA;
        lv.taskCtas = (lv.taskCount + lv.threads / 32 - 1) / (lv.threads / 32) * ((S + 63) / 64);
        r.levels.push_back(lv);
    }
    return r;
}

cudaError_t prepareMf() {
    const void* k[] = {reinterpret_cast<const void*>(mfLevelKernel<double, true, false, CTA>),
                       reinterpret_cast<const void*>(mfLevelKernel<double, true, false, WIDE_CTA>),
                       reinterpret_cast<const void*>(mfLevelKernel<float, true, true, CTA>),
                       reinterpret_cast<const void*>(mfLevelKernel<float, true, true, WIDE_CTA>),
                       reinterpret_cast<const void*>(mfLevelKernel<double, false, false, CTA>),
                       reinterpret_cast<const void*>(mfLevelKernel<double, false, false, WIDE_CTA>),
                       reinterpret_cast<const void*>(mfLevelKernel<float, false, false, CTA>),
                       reinterpret_cast<const void*>(mfLevelKernel<float, false, false, WIDE_CTA>)};
    for (const void* f : k) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, MF_MAX_BYTES);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void launchMfFactor(const DevNet&, const DevBatch& b, const MfRun& mf, bool fp32, cudaStream_t st) {
    if (fp32) launchLevels<float, true, true>(b, b.lu32, b.w32, static_cast<float*>(mf.upd), mf.dev, mf.up32->levels, st);
    else launchLevels<double, true, false>(b, b.lu64, b.w64, static_cast<double*>(mf.upd), mf.dev, mf.up64->levels, st);
}

void launchMfBackward(const DevNet&, const DevBatch& b, const MfRun& mf, bool fp32, cudaStream_t st) {
    if (fp32) launchLevels<float, false, false>(b, b.lu32, b.w32, nullptr, mf.dev, mf.down32->levels, st);
    else launchLevels<double, false, false>(b, b.lu64, b.w64, nullptr, mf.dev, mf.down64->levels, st);
}

}  // namespace olfb200
