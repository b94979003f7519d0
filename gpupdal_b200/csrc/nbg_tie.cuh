// nbg_tie.cuh — tie rows: what the tie-order resolver's kernels share.
#pragma once

#include "nbg_common.cuh"
#include "nbg_query.cuh"

namespace nbg {

// ---------------------------------------------------------------------------
// Tie-order resolver.
//
// In a tie row the points strictly inside the K-th distance D_K are the
// reference's, and the remaining m = K - less slots go to points at integer
// distance D_K.  Among those the reference keeps the smallest FP64 distances
// and, at equal FP64 distance, the ones its depth-first search meets first
// (nanoflann.hpp:178-205, :1191-1197): while fewer than m of them have been
// admitted the result set holds fewer than K points within D_K, so its worst
// distance exceeds D_K and no subtree holding one of them is pruned.  The
// search meets points of one leaf in the tree's point order and, for points in
// different leaves, first the side of their lowest common node that the query
// visits first (nanoflann.hpp:1226-1236: child1 iff (q-divlow)+(q-divhigh) < 0).
// Ordering that group therefore needs the replica's tree but not its search.
static constexpr int TIE_CAP = 32;

// True when the reference's search meets replica position pa before pb.
__device__ __forceinline__ bool kd_meets_first(const KdOrder& kd, const double q[3], uint32_t pa,
                                               uint32_t pb) {
    int node = kd.root;
    for (int depth = 0; depth < 64; ++depth) {
        const int a = __ldg(&kd.c1[node]);
        if (a < 0) break;
        const uint32_t split = __ldg(&kd.ne[a]);
        const bool la = pa < split, lb = pb < split;
        if (la == lb) {
            node = la ? a : __ldg(&kd.c2[node]);
            continue;
        }
        const double val = q[__ldg(&kd.feat[node])];
        const bool left_first =
            __dadd_rn(__dsub_rn(val, __ldg(&kd.dlo[node])), __dsub_rn(val, __ldg(&kd.dhi[node]))) < 0;
        return la == left_first;
    }
    return pa < pb;
}

struct TieArgs {
    GridView gv;
    const GridParams* gp;
    uint64_t n;
    const double* row_k;
    const int32_t* x;  // raw coordinates in caller order
    const int32_t* y;
    const int32_t* z;
    int K;
    StageGroup grp;
    Transform tf;
    ExceptionSink ex;
    const uint2* ties;
    uint32_t nties;
    uint64_t of_rows;  // rows of the query that listed them
    KdOrder kd;
    uint32_t* exact_rows;
    uint32_t* counters;
    uint32_t* ids_out;
};

}  // namespace nbg
