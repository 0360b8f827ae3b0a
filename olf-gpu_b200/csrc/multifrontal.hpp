// Host plan (multifrontal_plan.cpp) of the multifrontal block LU: the elimination order's columns grouped into nodes (supernodes)
// that are factorized as small dense fronts, one tree level of nodes per launch (multifrontal.cu).
#pragma once

#include <string>
#include <vector>

#include "structure.hpp"

namespace olfb200 {

// A node eliminates the p pivots of its first p rows; its front has m = p + q rows (positions, ascending; the q others
// belong to ancestors).  Its panel is the blocks U(k, j), k < p, j < m (index k m + j; for j < k the L part of the pivot
// block) followed by L(i, k), p <= i < m (index p m + (i - p) p + k): p (m + q) blocks.  Its update matrix (the q x q
// Schur complement it passes on, then q right-hand-side pairs, two to a block) starts at block upd of a buffer whose
// slots are reused once the parent has read them.
struct MfNode {
    int p, q;
    int rows;   // first of its m entries in rows / rhs
    int pan;    // first of its panel records
    int trl;    // first of its q q trailing records
    int upd;    // first block of its update matrix
    int child;  // 1: it has children (update matrices to add)
    int u0;     // the LU block of its first pivot's diagonal (the rest of that U row follows)
};

// A warp's task near the leaves: a one-pivot node (row -1: all of it) or one row below its pivot.
struct MfTask {
    int q, row;
    int pos;                       // the pivot's position
    int rows, pan, trl, upd, u0;   // as its node's
};

// What a target adds up: s0 / s1 blocks of children's update matrices (-1 none); s1 <= -2: more[-2 - s1] = count,
// then that many further blocks.
struct MfPanel {
    int aBlock;   // the Jacobian block, -1 none
    int out;      // the LU block it ends in, -1 a structural zero of the pattern (not stored)
    int s0, s1;
};
struct MfTrail {
    int s0, s1;
};
// Right-hand side of one front row: the bus's two equation rows (their -F is added, pivot rows only; -1 else) and the
// children's pairs (scalar index / 2 into the update buffer), encoded like the blocks.
struct MfRhs {
    int rowP, rowV;
    int s0, s1;
};

struct MfPlan {
    std::vector<MfNode> node;
    std::vector<int> rows;              // positions of the front rows of every node
    std::vector<MfPanel> pan;
    std::vector<MfTrail> trl;
    std::vector<MfRhs> rhs;
    std::vector<int> more;
    std::vector<int> parent;            // node -> parent node, -1 a root
    // nodes by height above the leaves (factorization) and by depth below the roots (backward), within a level by panel
    // size (backward: the small nodes first)
    std::vector<int> upPtr, upNode, downPtr, downNode;
    std::vector<int> downSmall;         // small nodes at the head of each backward level
    int updBlocks = 0;                  // blocks of the update buffer (per lane)
};

// A node whose backward substitution one thread does per lane; the others get a CTA.
inline bool mfSmall(const MfNode& n) { return n.p == 1 && n.q <= 8; }
// Near the leaves (tree levels below MF_LEAF_LEVELS) every node has one pivot, and a warp factorizes it for 64 lanes (up
// to MF_WARP_ROWS rows below the pivot; one row of it otherwise: four rows' blocks spill); further up a CTA does.
// Factorization + solves per pass, 9,241 buses, 500 / 17 lanes, by leaf levels: 3 2.26 / 0.74 ms, 5 2.14 / 0.68 ms,
// 7 2.13 / 0.68 ms, 9 2.09 / 0.69 ms; 2,000 buses, 257 lanes: 0.31, 0.33, 0.35, 0.36 ms.
// Grids from here on take the multifrontal solve; below, the few levels of the level launches are the shorter chain.  Whole
// solves, level launches / multifrontal, ms, 1 and 130 lanes: 512 buses 0.74 / 0.77 and 3.32 / 3.55, 540 0.74 / 0.83 and 3.35 /
// 3.77, 640 0.55 / 0.57 and 3.35 / 3.47, 660 (three grids, all batch sizes) 0.5 to 11 % slower; 700 (three grids) 0.95 / 0.81
// and 4.47 / 3.45, 0.94 / 0.85 and 4.53 / 3.81, 0.79 / 0.80 and 1.38 / 1.33; 820 0.96 / 0.90 and 4.41 / 4.01; 1,000 1.32 / 1.11
// and 5.09 / 4.39; 2,000 1.28 / 0.97 and 2.28 / 1.80; 9,241 3.29 / 2.07 and 7.09 / 5.30.  Small mixed batches gain as well (8
// lanes: 2,000 buses 3.43 / 2.79, 9,241 5.45 / 3.96).  The line is one of the grid, not of the batch: a scenario's bits do not
// depend on its batch's size, on any batch that has room for the update matrices.
constexpr int MF_MIN_BUSES = 700;
constexpr int MF_MAX_PIVOTS = 16, MF_MAX_FRONT = 40, MF_LEAF_LEVELS = 5, MF_WARP_ROWS = 3;
// The most rows below a pivot: the kernels divide a node's block numbers by multiplying with a 16-bit reciprocal.  An order
// with a wider column gets no plan (no nodes), and its factorization keeps the level launches.
constexpr int MF_MAX_BELOW = 40;

// Plans that may run it (buildMfPlan may still find a column too wide).
inline bool runsMultifrontal(const BlockPlan& p) { return !p.deferredL && p.nb >= MF_MIN_BUSES; }

MfPlan buildMfPlan(const BlockPlan& p, const std::vector<int>& nodeCol);
// "" when the plan holds: every position a pivot once, every LU block stored once, every Jacobian block and every
// child's update block added exactly once and at its own row and column, children below their parents, and no update
// matrix overwritten between its node's level and its parent's; else the first violation.
std::string checkMfPlan(const BlockPlan& p, const std::vector<int>& nodeCol, const MfPlan& m);

}  // namespace olfb200
