// nbg_kdtree.cu — exact replica of the reference's KD3 tree, and its search,
// for the rows whose neighbour set depends on nanoflann's tie order.
//
// The reference keeps, among points at equal FP64 distance, the ones its
// depth-first search meets first (vendor/nanoflann/nanoflann.hpp:178-205
// shifts only on strict >, :1191-1197 admits only dist < worst).  That order
// is a function of the tree, so rows whose k-th distance ties (and rows the
// ring search could not finish) are answered by replaying the reference's
// search over an identical tree built on the device.
//
// Tree build (nanoflann.hpp:640-690 divideTree, :779-828 middleSplit_,
// :837-873 planeSplit), level-synchronous over all segments of a level:
//   minmax    per-segment min/max of the raw coordinates (monotone in the
//             double coordinate raw*scale+offset)
//   split     cut feature among dims whose top-down span > (1-1e-5)*max span,
//             largest actual spread first; cut value = top-down midpoint
//             clamped to the segment's extent
//   pass 1/2  the two Hoare passes.  Their effect is exactly: with L the
//             count of elements satisfying the predicate, the t-th element
//             from the left failing it inside [0, L) swaps with the t-th
//             element from the right satisfying it inside [L, n).  Ranks
//             come from per-tile counts and block scans.
//   children  split index lim1 / lim2 / count/2 rule; segments of at most
//             100 points become leaves
// divlow/divhigh (child extents) are filled bottom-up afterwards.
//
// Search (nanoflann.hpp:875-893, 1059-1079, 1184-1250) is replayed per row
// in FP64 with every operation rounded as the reference rounds it.
#include <cub/cub.cuh>

#include <algorithm>
#include <string>
#include <vector>

#include "nbg_common.cuh"
#include "nbg_internal.h"

namespace nbg {

static constexpr int KD_LEAF = 100;
// Level passes: tiles of KD_THREADS * ROWS elements, each warp taking ROWS rows
// of 32 consecutive elements.  Long tiles keep the tile list of a 32M-point tree
// at 8k entries, which one block can scan; up to KD_SHORT_MAX points a tile of
// that length would leave most SMs without one (245 tiles at 1M points: 13.7 us
// a classify pass), so the tiles are a quarter as long.
static constexpr int KD_THREADS = 256;
static constexpr int KD_ROWS_LONG = 16, KD_ROWS_SHORT = 4;
static constexpr uint64_t KD_SHORT_MAX = 2500000;
// Segments of at most this many points are finished, subtree and all, in the
// shared memory of one block (kd_block_build_kernel).
static constexpr uint32_t KD_BLOCK_MAX = 4096;
static constexpr int KD_BTHREADS = 512;
static constexpr int KD_BWARPS = KD_BTHREADS / 32;
// a warp's pending subtrees: the smaller child is taken first, so at most
// log2(KD_BLOCK_MAX) larger ones wait
static constexpr int KD_BSTACK = 13;
// A build beside a running query (the plain call's speculative replica) keeps
// its level passes to 4 blocks of 256 threads per SM, walking tiles in strides,
// and starts its subtrees, whose blocks want most of an SM's shared memory, when
// the query's select pass is through (beside its FP64 finish pass).  From 16M
// points up; a smaller build would end after the query, which then waits for it.
static constexpr int kKdBesideBlocksPerSm = 4;
static constexpr uint64_t kKdBesideMinPoints = 16000000;
static constexpr uint32_t KD_WARP_RUN = 2048;  // points of a run at the cut that one warp reads
static constexpr int KD_RETRY = -100;  // kd_build: redo with room for every node
static constexpr int KD_STACK = 96;
static constexpr int KD_CAP = 66;

struct KdSeg {
    uint32_t begin, end;
    int32_t node;
    int32_t pad;   // tree
    double lo[3], hi[3];
};

// A level segment's cut and what its passes found.
struct KdSplit {
    int32_t f;
    int32_t dims;  // dimensions (bits) whose extents the children need
    // points with (uint32_t)(raw - org) below t1 are below the cut, those below
    // t2 at or below it (org: the segment's least raw value in dimension f)
    int32_t org;
    uint32_t t1, t2;
    uint32_t first;  // first tile
    double cutval;
    uint32_t L, eq;  // points below and at the cut
    uint32_t m, m2;  // misplaced pairs of pass 1 and pass 2
    // extents of the points below, at and above the cut (dimensions `dims`)
    int32_t mn[3][3], mx[3][3];
};

// Device-side state of a build: the host queues levels without reading it.
struct KdState {
    uint32_t segs;    // segments of the current level
    uint32_t tiles;   // their tiles
    uint32_t nodes;
    uint32_t errors;  // capacity overflows
    uint32_t small;   // segments for the subtree builder
    uint32_t any_eq;  // some segment of the level has points at its cut
    uint32_t ticket;  // blocks of the running pass that have finished
    uint32_t pad;
};

struct KdDev {
    const int32_t* rx;
    const int32_t* ry;
    const int32_t* rz;
    const uint32_t* rid;
    const int32_t* c1;
    const int32_t* c2;
    const int32_t* feat;
    const uint32_t* nb;
    const uint32_t* ne;
    const double* dlo;
    const double* dhi;
    int32_t root;  // the tree's root node
    double root_lo[3], root_hi[3];
};

// Storage of one or more replicas built together (a forest): the trees'
// points are concatenated (tree k owns positions [base[k], base[k] + npts[k])),
// their nodes share the node arrays, and tree k's root is node k.  Segments
// carry their tree in KdSeg::pad, nodes in ntree[].
struct KdForest {
    uint64_t n = 0;
    uint32_t grid_cap = 0;   // most blocks of a level-pass launch (0: no limit)
    bool beside = false;     // shares the SMs with a query
    int ntrees = 0;
    std::vector<uint64_t> base, npts;
    std::vector<Transform> tfh;
    std::vector<double> rootbox;  // 6 per tree: lo[3], hi[3]
    Transform* tfs = nullptr;     // device, per tree
    int32_t* ntree = nullptr;     // device, per node
    int refs = 0;
    int32_t* rx = nullptr;
    int32_t* ry = nullptr;
    int32_t* rz = nullptr;
    uint32_t* rid = nullptr;
    uint32_t* kpos = nullptr;  // base + point id -> position (inverse of rid per tree)
    uint32_t* mlpos = nullptr;
    uint32_t* mrpos = nullptr;
    // nodes
    uint32_t node_cap = 0, node_count = 0;
    int32_t* c1 = nullptr;
    int32_t* c2 = nullptr;
    int32_t* feat = nullptr;
    uint32_t* nb = nullptr;
    uint32_t* ne = nullptr;
    double* dlo = nullptr;
    double* dhi = nullptr;
    int32_t* bmin = nullptr;  // 3 per node
    int32_t* bmax = nullptr;
    // segments of the current and next level
    KdSeg* seg[2] = {nullptr, nullptr};
    KdSplit* split[2] = {nullptr, nullptr};
    uint32_t seg_cap = 0;
    KdSeg* small = nullptr;      // segments left for the subtree builder
    uint32_t small_cap = 0;
    // tiles
    uint32_t* tile_seg = nullptr;
    unsigned long long* tile_cnt = nullptr;  // per tile counts (below | at << 32), then prefix
    uint32_t tile_cap = 0;
    uint32_t tile = 0;  // elements a tile
    KdState* state = nullptr;
    uint32_t* counters = nullptr;  // [2] errors of the search replay
    uint64_t* bases = nullptr;     // device, first position per tree
    uint64_t bytes = 0;
    std::vector<std::pair<void*, size_t>> blocks;  // device blocks owned
};

// A tile's view of its replica: the forest and the tile's tree in it.
struct KdReplica {
    KdForest* f = nullptr;
    int tree = 0;
    bool built = false;
};

// ---------------------------------------------------------------------------
// build kernels
// ---------------------------------------------------------------------------
__global__ void kd_init_kernel(const int32_t* x, const int32_t* y, const int32_t* z, uint64_t n,
                               int32_t* rx, int32_t* ry, int32_t* rz, uint32_t* rid) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        rx[i] = x[i];
        ry[i] = y[i];
        rz[i] = z[i];
        rid[i] = (uint32_t)i;
    }
}

// Cut feature and value of a segment from its top-down box (lo, hi) and its
// points' extents (mn, mx): nanoflann.hpp:779-828 middleSplit_.
__device__ __forceinline__ void kd_choose_cut(const double lo[3], const double hi[3],
                                              const int32_t mn_[3], const int32_t mx_[3],
                                              const Transform& tf, int& cutfeat, double& cutval) {
    const double EPS = 0.00001;
    double max_span = __dsub_rn(hi[0], lo[0]);
    for (int i = 1; i < 3; ++i) {
        double span = __dsub_rn(hi[i], lo[i]);
        if (span > max_span) max_span = span;
    }
    double max_spread = -1;
    cutfeat = 0;
    for (int i = 0; i < 3; ++i) {
        double span = __dsub_rn(hi[i], lo[i]);
        if (span > __dmul_rn(__dsub_rn(1.0, EPS), max_span)) {
            double mn = ref_coord(mn_[i], tf.scale[i], tf.offset[i]);
            double mx = ref_coord(mx_[i], tf.scale[i], tf.offset[i]);
            double spread = __dsub_rn(mx, mn);
            if (spread > max_spread) {
                cutfeat = i;
                max_spread = spread;
            }
        }
    }
    double split_val = __dmul_rn(__dadd_rn(lo[cutfeat], hi[cutfeat]), 0.5);  // (halving is exact either way)
    double mn = ref_coord(mn_[cutfeat], tf.scale[cutfeat], tf.offset[cutfeat]);
    double mx = ref_coord(mx_[cutfeat], tf.scale[cutfeat], tf.offset[cutfeat]);
    if (split_val < mn) cutval = mn;
    else if (split_val > mx) cutval = mx;
    else cutval = split_val;
}

// The reference's coordinate is monotone in the raw integer, so a comparison
// with the cut value is one with an integer: t1 counts from mn to the smallest
// raw value of [mn, mx + 1] whose coordinate is at or above the cut, t2 to the
// smallest above it.  (The passes then read 4 bytes and compare, with no FP64
// arithmetic; as offsets from mn the bounds fit at either end of int32.)
__device__ __forceinline__ void kd_thresholds(double cut, double sc, double of, int32_t mn, int32_t mx,
                                              uint32_t& t1, uint32_t& t2) {
    const uint32_t range = (uint32_t)((long long)mx - mn) + 1u;
    auto at = [&](uint32_t k) { return ref_coord((int32_t)((long long)mn + k), sc, of); };
    const double est = (cut - of) / sc - (double)mn;
    const uint32_t near = est <= 0.0 ? 0u : est >= (double)range ? range : (uint32_t)est;
    uint32_t bound[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        uint32_t lo = q ? bound[0] : 0u, hi = range;  // the answer lies in [lo, hi]
        uint32_t probe = max(lo, min(near, hi));
        for (int step = 0; lo < hi; ++step) {
            // a few steps around the estimate settle it unless many raw values
            // share a coordinate (an offset far above the scale)
            if (step > 3) probe = lo + (hi - lo) / 2;
            probe = min(probe, hi - 1);
            const double v = at(probe);
            if (q ? v <= cut : v < cut) {
                lo = probe + 1;
                probe = lo;
            } else {
                hi = probe;
                probe = hi > lo ? hi - 1 : lo;
            }
        }
        bound[q] = lo;
    }
    t1 = bound[0];
    t2 = bound[1];
}

// The same by a whole warp: its lanes try 32 raw values around the estimate
// (inv = 1 / sc) at once.
__device__ __forceinline__ void kd_warp_thresholds(double cut, double sc, double inv, double of, int32_t mn,
                                                   int32_t mx, uint32_t& t1, uint32_t& t2) {
    const uint32_t range = (uint32_t)((long long)mx - mn) + 1u;
    const double est = (cut - of) * inv - (double)mn - 15.0;
    const uint32_t base = est <= 0.0 ? 0u : est >= (double)range ? range - 1u : (uint32_t)est;
    const uint32_t u = base + (threadIdx.x & 31u);
    const double v = ref_coord((int32_t)((long long)mn + min(u, range - 1u)), sc, of);
    const unsigned in = __ballot_sync(0xffffffffu, u < range);
    const unsigned below = __ballot_sync(0xffffffffu, u < range && v < cut);
    const unsigned upto = __ballot_sync(0xffffffffu, u < range && v <= cut);
    if ((base && !(below & 1u)) || (upto == in && base + __popc(in) < range)) {
        kd_thresholds(cut, sc, of, mn, mx, t1, t2);  // beyond the lanes' reach
        return;
    }
    t1 = base + __popc(below);
    t2 = base + __popc(upto);
}

// Hoare's pass swaps the t-th element from the left that fails the predicate
// inside [0, L) with the t-th from the right that satisfies it inside [L, n);
// with `prank` elements satisfying it before element li, a failing element's t
// is li - prank, a satisfying one's L - 1 - prank.
__device__ __forceinline__ uint32_t kd_split_index(uint32_t count, uint32_t L, uint32_t L2) {
    const uint32_t lim1 = L, lim2 = L + L2;
    return lim1 > count / 2 ? lim1 : lim2 < count / 2 ? lim2 : count / 2;
}

struct KdNodes {
    int32_t *c1, *c2, *feat;
    uint32_t *nb, *ne;
    int32_t *bmin, *bmax;
    int32_t* ntree;
    uint32_t cap;
};

// Node arrays of one split: parent `node`, children cid and cid + 1.
__device__ __forceinline__ void kd_write_children(const KdNodes& N, int32_t node, uint32_t cid, int f,
                                                  uint32_t b, uint32_t mid, uint32_t e, int32_t tree) {
    N.c1[node] = (int32_t)cid;
    N.c2[node] = (int32_t)(cid + 1);
    N.feat[node] = f;
#pragma unroll
    for (uint32_t side = 0; side < 2; ++side) {
        N.nb[cid + side] = side ? mid : b;
        N.ne[cid + side] = side ? e : mid;
        N.c1[cid + side] = -1;
        N.c2[cid + side] = -1;
        N.feat[cid + side] = 0;
        N.ntree[cid + side] = tree;
    }
}

struct KdLevel {
    const KdSeg* segs;
    KdSplit* sp;
    KdSeg* next;
    KdSplit* next_sp;
    KdSeg* small;
    uint32_t* tile_seg;
    unsigned long long* tile_cnt;
    KdState* st;
    int32_t *rx, *ry, *rz;
    uint32_t* rid;
    uint32_t *mlpos, *mrpos;
    const Transform* tfs;
    KdNodes N;
    uint32_t seg_cap, small_cap, tile_cap;
    uint32_t tile;  // elements a tile
};

// True in every thread of the block that finishes a pass last; what the other
// blocks wrote is visible to it.
__device__ __forceinline__ bool kd_last_block(KdState* st) {
    __shared__ uint32_t s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}

// Exclusive prefix of v[0 .. n] (n + 1 entries, v[n] written) by one block of
// KD_THREADS threads.
__device__ __forceinline__ void kd_block_prefix(unsigned long long* v, uint32_t n) {
    typedef cub::BlockScan<unsigned long long, KD_THREADS> Scan;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ unsigned long long s_carry;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < n; base += KD_THREADS * 8) {
        unsigned long long x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t i = base + threadIdx.x * 8 + k;
            x[k] = i < n ? __ldcg(&v[i]) : 0ull;
        }
        unsigned long long total;
        Scan(tmp).ExclusiveSum(x, x, total);
        const unsigned long long c = s_carry;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t i = base + threadIdx.x * 8 + k;
            if (i < n) v[i] = c + x[k];
        }
        if (threadIdx.x == 0) s_carry = c + total;
        __syncthreads();
    }
    if (threadIdx.x == 0) v[n] = s_carry;
}

// Rows of a tile: warp w's element of row k.
template <int ROWS>
__device__ __forceinline__ uint32_t kd_row(uint32_t begin, uint32_t tile, int k) {
    return begin + tile * (KD_THREADS * ROWS) + ((threadIdx.x >> 5) * ROWS + k) * 32 + (threadIdx.x & 31u);
}

// Per tile, pass 1: points below the cut in the low 32 bits, at it in the high
// ones; pass 2: points at the cut at or after position L (segments that have
// any).  The last block turns the counts into their prefix.
template <int PASS, int ROWS>
__global__ void __launch_bounds__(KD_THREADS) kd_count_kernel(const KdLevel lv) {
    __shared__ unsigned long long red[KD_THREADS / 32];
    const uint32_t ntiles = lv.st->tiles;
    if (!ntiles || (PASS == 2 && !lv.st->any_eq)) return;
    for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const uint32_t s = lv.tile_seg[t];
        const uint32_t b = lv.segs[s].begin, e = lv.segs[s].end;
        const KdSplit* sp = &lv.sp[s];
        const int f = sp->f, org = sp->org;
        const uint32_t t1 = sp->t1, t2 = sp->t2;
        const uint32_t from = PASS == 1 ? b : b + sp->L;
        const int32_t* rc = f == 0 ? lv.rx : (f == 1 ? lv.ry : lv.rz);
        uint32_t nlt = 0, neq = 0;
        if (PASS == 1 || sp->eq) {
            int32_t v[ROWS];
#pragma unroll
            for (int k = 0; k < ROWS; ++k) {
                const uint32_t i = kd_row<ROWS>(b, t - sp->first, k);
                v[k] = i >= from && i < e ? rc[i] - org : -1;
            }
#pragma unroll
            for (int k = 0; k < ROWS; ++k) {
                const uint32_t x = (uint32_t)v[k];  // (outside the range: above every bound)
                if (PASS == 1) nlt += x < t1;
                neq += x >= t1 && x < t2;
            }
        }
        unsigned long long c = (unsigned long long)__reduce_add_sync(0xffffffffu, nlt) |
                               (unsigned long long)__reduce_add_sync(0xffffffffu, neq) << 32;
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long r = 0;
            for (int k = 0; k < KD_THREADS / 32; ++k) r += red[k];
            lv.tile_cnt[t] = r;
        }
        __syncthreads();
    }
    if (!kd_last_block(lv.st)) return;
    kd_block_prefix(lv.tile_cnt, ntiles);
    __syncthreads();
    if (threadIdx.x == 0) lv.st->ticket = 0;
    if (PASS == 1) {
        // the segments' counts
        const uint32_t S = lv.st->segs;
        bool eq = false;
        for (uint32_t s = threadIdx.x; s < S; s += KD_THREADS) {
            KdSplit* sp = &lv.sp[s];
            const uint32_t t0 = sp->first, t1 = s + 1 < S ? lv.sp[s + 1].first : ntiles;
            const unsigned long long d = lv.tile_cnt[t1] - lv.tile_cnt[t0];
            sp->L = (uint32_t)d;
            sp->eq = (uint32_t)(d >> 32);
            sp->m = 0;
            sp->m2 = 0;
            eq = eq || sp->eq;
        }
        eq = __syncthreads_or(eq);
        if (threadIdx.x == 0) lv.st->any_eq = eq;
    }
}

// The positions of the misplaced elements (mlpos, mrpos: see kd_split_index's
// note); pass 1 also takes the extents of the points below, at and above the
// cut, the children's boxes.
template <int PASS, int ROWS>
__global__ void __launch_bounds__(KD_THREADS) kd_classify_kernel(const KdLevel lv) {
    __shared__ uint32_t s_cnt[KD_THREADS / 32];
    __shared__ int32_t s_ext[18];
    const uint32_t ntiles = lv.st->tiles;
    if (!ntiles || (PASS == 2 && !lv.st->any_eq)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const uint32_t s = lv.tile_seg[t];
        KdSplit* sp = &lv.sp[s];
        if (PASS == 2 && !sp->eq) continue;
        const uint32_t sb = lv.segs[s].begin, e = lv.segs[s].end;
        const uint32_t L1 = sp->L;
        const uint32_t b = PASS == 1 ? sb : sb + L1;      // the pass's range
        const uint32_t L = PASS == 1 ? L1 : sp->eq;       // satisfying elements in it
        const int f = sp->f, org = sp->org;
        const uint32_t t1 = sp->t1, t2 = sp->t2;
        const int dims = sp->dims;
        const int32_t* rc = f == 0 ? lv.rx : (f == 1 ? lv.ry : lv.rz);
        unsigned bal[ROWS];
        uint32_t n = 0;
        if (PASS == 1) {
            if (threadIdx.x < 18) s_ext[threadIdx.x] = threadIdx.x < 9 ? INT32_MAX : INT32_MIN;
            int32_t mn[2][3], mx[2][3];  // below, at or above
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    mn[q][d] = INT32_MAX;
                    mx[q][d] = INT32_MIN;
                }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < ROWS; ++k) {
                const uint32_t i = kd_row<ROWS>(sb, t - sp->first, k);
                const bool in = i < e;
                const int32_t c[3] = {in && dims & 1 ? lv.rx[i] : 0, in && dims & 2 ? lv.ry[i] : 0,
                                      in && dims & 4 ? lv.rz[i] : 0};
                const uint32_t v = (uint32_t)((f == 0 ? c[0] : (f == 1 ? c[1] : c[2])) - org);
                const bool p = in && v < t1;
                bal[k] = __ballot_sync(0xffffffffu, p);
                n += __popc(bal[k]);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    mn[0][d] = min(mn[0][d], p ? c[d] : INT32_MAX);
                    mx[0][d] = max(mx[0][d], p ? c[d] : INT32_MIN);
                    mn[1][d] = min(mn[1][d], in && v >= t2 ? c[d] : INT32_MAX);
                    mx[1][d] = max(mx[1][d], in && v >= t2 ? c[d] : INT32_MIN);
                }
                // at the cut: few (a ninth of all points costs as much lane by lane
                // as reduced over the warp first)
                if (in && v >= t1 && v < t2)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        atomicMin(&s_ext[3 + d], c[d]);
                        atomicMax(&s_ext[12 + d], c[d]);
                    }
            }
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int32_t a = __reduce_min_sync(0xffffffffu, mn[q][d]);
                    const int32_t z = __reduce_max_sync(0xffffffffu, mx[q][d]);
                    if (lane == 0) {
                        atomicMin(&s_ext[6 * q + d], a);
                        atomicMax(&s_ext[9 + 6 * q + d], z);
                    }
                }
        } else {
#pragma unroll
            for (int k = 0; k < ROWS; ++k) {
                const uint32_t i = kd_row<ROWS>(sb, t - sp->first, k);
                const bool in = i >= b && i < e;
                bal[k] = __ballot_sync(0xffffffffu, in && (uint32_t)(rc[in ? i : b] - org) < t2);
                n += __popc(bal[k]);
            }
        }
        if (lane == 0) s_cnt[warp] = n;
        __syncthreads();
        const unsigned long long pre = lv.tile_cnt[t] - lv.tile_cnt[sp->first];
        uint32_t before = PASS == 1 ? (uint32_t)pre : (uint32_t)(pre >> 32);
        for (int w = 0; w < warp; ++w) before += s_cnt[w];
#pragma unroll
        for (int k = 0; k < ROWS; ++k) {
            const uint32_t i = kd_row<ROWS>(sb, t - sp->first, k);
            if (i >= b && i < e) {
                const uint32_t prank = before + __popc(bal[k] & lt), li = i - b;
                const bool p = bal[k] >> lane & 1u;
                if (li < L) {
                    if (!p) lv.mlpos[b + (li - prank)] = i;
                } else {
                    if (p) lv.mrpos[b + (L - 1 - prank)] = i;
                    if (li == L) {
                        if (PASS == 1) sp->m = L - prank;
                        else sp->m2 = L - prank;
                    }
                }
            }
            before += __popc(bal[k]);
        }
        if (PASS == 1 && threadIdx.x < 18) {
            const int q = (threadIdx.x % 9) / 3, d = threadIdx.x % 3;
            if (threadIdx.x < 9) atomicMin(&sp->mn[q][d], s_ext[threadIdx.x]);
            else atomicMax(&sp->mx[q][d], s_ext[threadIdx.x]);
        }
        __syncthreads();
    }
}

// Cut, thresholds and fresh extents of a segment whose points' extents are
// (mn, mx).
__device__ __forceinline__ void kd_plan_segment(const KdSeg& sg, const int32_t mn[3], const int32_t mx[3],
                                                const Transform& tf, KdSplit* sp) {
    int f;
    double cut;
    kd_choose_cut(sg.lo, sg.hi, mn, mx, tf, f, cut);
    KdSplit p;
    p.f = f;
    p.cutval = cut;
    p.org = mn[f];
    // a child's cut is chosen among the dimensions whose side of its box comes
    // within 1e-5 of the longest; their extents decide, and the cut dimension's
    // become divlow / divhigh: the classify pass reads no others
    p.dims = 1 << f;
    for (int side = 0; side < 2; ++side) {
        double span[3], longest = 0.0;
        for (int d = 0; d < 3; ++d) {
            const double l = side && d == f ? cut : sg.lo[d], h = !side && d == f ? cut : sg.hi[d];
            span[d] = __dsub_rn(h, l);
            longest = fmax(longest, span[d]);
        }
        for (int d = 0; d < 3; ++d)
            if (span[d] >= longest * (1.0 - 2e-5)) p.dims |= 1 << d;
    }
    kd_thresholds(cut, tf.scale[f], tf.offset[f], mn[f], mx[f], p.t1, p.t2);
    p.first = 0;
    p.L = p.eq = p.m = p.m2 = 0;
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            p.mn[q][d] = INT32_MAX;
            p.mx[q][d] = INT32_MIN;
        }
    *sp = p;
}

// One block: the tile list of the S segments in segs / sp.
__device__ __forceinline__ void kd_tile_map(const KdSeg* segs, KdSplit* sp, uint32_t S, uint32_t* tile_seg,
                                            uint32_t tile_cap, uint32_t tile, KdState* st) {
    typedef cub::BlockScan<uint32_t, KD_THREADS> Scan;
    __shared__ typename Scan::TempStorage tmp;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < S; base += KD_THREADS) {
        const uint32_t s = base + threadIdx.x;
        const uint32_t nt = s < S ? (segs[s].end - segs[s].begin + tile - 1) / tile : 0u;
        uint32_t first, total;
        Scan(tmp).ExclusiveSum(nt, first, total);
        if (s < S) sp[s].first = carry + first;
        carry += total;
        __syncthreads();
    }
    if (carry > tile_cap) {
        if (threadIdx.x == 0) {
            st->errors += 1;
            st->segs = st->tiles = 0;
        }
        return;
    }
    for (uint32_t t = threadIdx.x; t < carry; t += KD_THREADS) {
        uint32_t lo = 0, hi = S;  // last segment whose first tile <= t
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sp[mid].first <= t) lo = mid;
            else hi = mid;
        }
        tile_seg[t] = lo;
    }
    if (threadIdx.x == 0) {
        st->segs = S;
        st->tiles = carry;
    }
}

// Extents of the points [from, mid) (v: least x, y, z, then greatest) and [mid, to)
// (the next six), in every lane of a warp that takes every `step`-th from
// `first` (its lanes' consecutive).
__device__ __forceinline__ void kd_run_extents(const KdLevel& lv, uint32_t from, uint32_t mid, uint32_t to,
                                               uint32_t first, uint32_t step, int32_t (&v)[12]) {
#pragma unroll
    for (int k = 0; k < 12; ++k) v[k] = k % 6 < 3 ? INT32_MAX : INT32_MIN;
#pragma unroll 4
    for (uint32_t i = from + first; i < to; i += step) {
        const int32_t c[3] = {__ldcg(&lv.rx[i]), __ldcg(&lv.ry[i]), __ldcg(&lv.rz[i])};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            v[d] = min(v[d], i < mid ? c[d] : INT32_MAX);
            v[3 + d] = max(v[3 + d], i < mid ? c[d] : INT32_MIN);
            v[6 + d] = min(v[6 + d], i < mid ? INT32_MAX : c[d]);
            v[9 + d] = max(v[9 + d], i < mid ? INT32_MIN : c[d]);
        }
    }
#pragma unroll
    for (int k = 0; k < 12; ++k)
        v[k] = k % 6 < 3 ? __reduce_min_sync(0xffffffffu, v[k]) : __reduce_max_sync(0xffffffffu, v[k]);
}

// The misplaced pairs of a tile: every load of the thread's pairs is issued
// before any store (each position belongs to exactly one pair of the level, so
// the loads never read what a store of this launch writes), which keeps the
// dependent position -> coordinate loads of all the thread's items in flight
// together instead of one item at a time.  After pass 2 the last block splits
// the segments and plans the next level (the bound keeps its registers from
// costing the swaps a resident block).
template <int PASS>
__global__ void __launch_bounds__(KD_THREADS, PASS == 1 ? 4 : 3) kd_swap_kernel(const KdLevel lv) {
    const uint32_t ntiles = lv.st->tiles;
    if (!ntiles) return;
    constexpr int ITEMS = 4;
    if (PASS == 1 || lv.st->any_eq) {
        for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
            const uint32_t s = lv.tile_seg[t];
            const KdSplit* sp = &lv.sp[s];
            const uint32_t m = PASS == 1 ? sp->m : sp->m2;
            const uint32_t b = lv.segs[s].begin + (PASS == 1 ? 0u : sp->L);
            const uint32_t end = min(m, (t - sp->first + 1) * lv.tile);
            for (uint32_t l0 = (t - sp->first) * lv.tile + threadIdx.x; l0 < end; l0 += KD_THREADS * ITEMS) {
                uint32_t a[ITEMS], z[ITEMS], ai[ITEMS], zi[ITEMS];
                int32_t ax[ITEMS], ay[ITEMS], az[ITEMS], zx[ITEMS], zy[ITEMS], zz[ITEMS];
#pragma unroll
                for (int k = 0; k < ITEMS; ++k)
                    if (l0 + k * KD_THREADS < end) {
                        a[k] = lv.mlpos[b + l0 + k * KD_THREADS];
                        z[k] = lv.mrpos[b + l0 + k * KD_THREADS];
                    }
#pragma unroll
                for (int k = 0; k < ITEMS; ++k)
                    if (l0 + k * KD_THREADS < end) {
                        ax[k] = lv.rx[a[k]];
                        ay[k] = lv.ry[a[k]];
                        az[k] = lv.rz[a[k]];
                        ai[k] = lv.rid[a[k]];
                        zx[k] = lv.rx[z[k]];
                        zy[k] = lv.ry[z[k]];
                        zz[k] = lv.rz[z[k]];
                        zi[k] = lv.rid[z[k]];
                    }
#pragma unroll
                for (int k = 0; k < ITEMS; ++k)
                    if (l0 + k * KD_THREADS < end) {
                        lv.rx[a[k]] = zx[k];
                        lv.ry[a[k]] = zy[k];
                        lv.rz[a[k]] = zz[k];
                        lv.rid[a[k]] = zi[k];
                        lv.rx[z[k]] = ax[k];
                        lv.ry[z[k]] = ay[k];
                        lv.rz[z[k]] = az[k];
                        lv.rid[z[k]] = ai[k];
                    }
            }
        }
    }
    if (PASS == 1 || !kd_last_block(lv.st)) return;
    // ---- split the segments, plan the next level
    __shared__ uint32_t s_next, s_runs, s_who, s_run[3];
    __shared__ int32_t s_rext[12];
    if (threadIdx.x == 0) s_next = s_runs = 0;
    __syncthreads();
    const uint32_t S = lv.st->segs;
    // children of a segment cut at `index`, with the extents of their points
    auto split = [&](const KdSeg& sg, const KdSplit& p, uint32_t index, const int32_t (&mn)[2][3],
                     const int32_t (&mx)[2][3]) {
        const uint32_t cid = atomicAdd(&lv.st->nodes, 2u);
        if (cid + 2 > lv.N.cap) {
            atomicAdd(&lv.st->errors, 1u);
            return;
        }
        kd_write_children(lv.N, sg.node, cid, p.f, sg.begin, sg.begin + index, sg.end, sg.pad);
        for (int side = 0; side < 2; ++side) {
            const uint32_t node = cid + side;
            for (int d = 0; d < 3; ++d) {
                lv.N.bmin[3 * node + d] = mn[side][d];
                lv.N.bmax[3 * node + d] = mx[side][d];
            }
            KdSeg ch = sg;
            if (side == 0) {
                ch.end = sg.begin + index;
                ch.hi[p.f] = p.cutval;
            } else {
                ch.begin = sg.begin + index;
                ch.lo[p.f] = p.cutval;
            }
            ch.node = (int32_t)node;
            if (ch.end - ch.begin <= KD_BLOCK_MAX) {
                const uint32_t slot = atomicAdd(&lv.st->small, 1u);
                if (slot < lv.small_cap) lv.small[slot] = ch;
                else atomicAdd(&lv.st->errors, 1u);
            } else {
                const uint32_t slot = atomicAdd(&s_next, 1u);
                if (slot < lv.seg_cap) {
                    lv.next[slot] = ch;
                    kd_plan_segment(ch, mn[side], mx[side], lv.tfs[sg.pad], &lv.next_sp[slot]);
                } else {
                    atomicAdd(&lv.st->errors, 1u);
                }
            }
        }
    };
    for (uint32_t s = threadIdx.x; s < S; s += KD_THREADS) {
        const KdSeg sg = lv.segs[s];
        const KdSplit p = lv.sp[s];
        const uint32_t index = kd_split_index(sg.end - sg.begin, p.L, p.eq);
        if (index > p.L && index < p.L + p.eq) {  // among the points at the cut: below
            s_runs = 1;
            continue;
        }
        // the points at the cut go to one side
        int32_t mn[2][3], mx[2][3];
        for (int d = 0; d < 3; ++d) {
            mn[0][d] = p.mn[0][d];
            mx[0][d] = p.mx[0][d];
            mn[1][d] = p.mn[2][d];
            mx[1][d] = p.mx[2][d];
        }
        const int at = index == p.L ? 1 : 0;
        for (int d = 0; d < 3; ++d) {
            mn[at][d] = min(mn[at][d], p.mn[1][d]);
            mx[at][d] = max(mx[at][d], p.mx[1][d]);
        }
        split(sg, p, index, mn, mx);
    }
    __syncthreads();
    // segments whose split falls among the points at their cut: the extents of the
    // two parts of that run, read by a warp, or (a long run) by the block
    const int lane = threadIdx.x & 31;
    for (uint32_t s0 = 0; s_runs && s0 < S; s0 += KD_THREADS) {
        const uint32_t s = s0 + threadIdx.x;
        const KdSeg sg = lv.segs[min(s, S - 1)];
        const KdSplit p = lv.sp[min(s, S - 1)];
        const uint32_t index = kd_split_index(sg.end - sg.begin, p.L, p.eq);
        const bool in_run = s < S && index > p.L && index < p.L + p.eq;
        const uint32_t from = sg.begin + p.L, mid = sg.begin + index, to = from + p.eq;
        int32_t run[12];
        for (unsigned m = __ballot_sync(0xffffffffu, in_run && p.eq <= KD_WARP_RUN); m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            int32_t v[12];
            kd_run_extents(lv, __shfl_sync(0xffffffffu, from, src), __shfl_sync(0xffffffffu, mid, src),
                           __shfl_sync(0xffffffffu, to, src), lane, 32u, v);
            if (lane == src)
#pragma unroll
                for (int k = 0; k < 12; ++k) run[k] = v[k];
        }
        bool wait = in_run && p.eq > KD_WARP_RUN;
        while (__syncthreads_or(wait)) {
            if (threadIdx.x == 0) s_who = KD_THREADS;
            if (threadIdx.x < 12) s_rext[threadIdx.x] = threadIdx.x % 6 < 3 ? INT32_MAX : INT32_MIN;
            __syncthreads();
            if (wait) atomicMin(&s_who, threadIdx.x);
            __syncthreads();
            const bool mine = wait && s_who == threadIdx.x;
            if (mine) {
                s_run[0] = from;
                s_run[1] = mid;
                s_run[2] = to;
            }
            __syncthreads();
            int32_t v[12];
            kd_run_extents(lv, s_run[0], s_run[1], s_run[2], threadIdx.x, KD_THREADS, v);
            if (lane == 0)
#pragma unroll
                for (int k = 0; k < 12; ++k) {
                    if (k % 6 < 3) atomicMin(&s_rext[k], v[k]);
                    else atomicMax(&s_rext[k], v[k]);
                }
            __syncthreads();
            if (mine) {
                wait = false;
#pragma unroll
                for (int k = 0; k < 12; ++k) run[k] = s_rext[k];
            }
        }
        if (!in_run) continue;
        int32_t mn[2][3], mx[2][3];
#pragma unroll
        for (int side = 0; side < 2; ++side)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                mn[side][d] = min(p.mn[2 * side][d], run[6 * side + d]);
                mx[side][d] = max(p.mx[2 * side][d], run[6 * side + 3 + d]);
            }
        split(sg, p, index, mn, mx);
    }
    __syncthreads();
    if (threadIdx.x == 0) lv.st->ticket = 0;
    kd_tile_map(lv.next, lv.next_sp, min(s_next, lv.seg_cap), lv.tile_seg, lv.tile_cap, lv.tile, lv.st);
}

// The roots: extents, cuts and tile list of the first level (one block).
__global__ void __launch_bounds__(KD_THREADS) kd_roots_kernel(const KdLevel lv, uint32_t S) {
    for (uint32_t s = threadIdx.x; s < S; s += KD_THREADS) {
        const KdSeg sg = lv.segs[s];
        kd_plan_segment(sg, &lv.N.bmin[3 * sg.node], &lv.N.bmax[3 * sg.node], lv.tfs[sg.pad], &lv.sp[s]);
    }
    __syncthreads();
    kd_tile_map(lv.segs, lv.sp, S, lv.tile_seg, lv.tile_cap, lv.tile, lv.st);
}

// ---------------------------------------------------------------------------
// Whole subtrees in shared memory, one block per segment.  The block's warps
// split with the tree: a group of W warps cuts its segment (extents, cut,
// ranks by ballot, Hoare's swaps, all in shared memory), then each half of the
// group takes one child; a single warp goes on depth first, the smaller child
// at once and the larger one stacked.  A point is read and written once; the
// inverse permutation goes out with it.
struct KdFrame16 {
    double lo[3], hi[3];
    int32_t node;
    uint16_t b, e;
};

struct KdBlockShared {
    int32_t c[3][KD_BLOCK_MAX];
    uint32_t id[KD_BLOCK_MAX];
    uint16_t ml[KD_BLOCK_MAX], mr[KD_BLOCK_MAX];
    KdFrame16 stk[KD_BWARPS][KD_BSTACK];
    int32_t ext[KD_BWARPS][6];
    uint32_t cnt[KD_BWARPS][2];
    uint32_t m[KD_BWARPS];
    uint32_t cid[KD_BWARPS];
};

// Barrier of a group of W warps starting at warp w0 (barrier 0 is the block's).
__device__ __forceinline__ void kd_group_sync(int W, int w0) {
    if (W == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + (w0 >> 1)), "r"(W * 32) : "memory");
}

// One Hoare pass of a group over [b, e) (values less than `tp` above `org`
// satisfy the predicate; L of them).
__device__ __forceinline__ void kd_group_pass(KdBlockShared& sh, const int32_t* v, uint32_t b, uint32_t e,
                                              int32_t org, uint32_t tp, uint32_t L, uint32_t before, uint32_t r0, uint32_t r1,
                                              int W, int w0) {
    const int lane = threadIdx.x & 31, t = threadIdx.x - w0 * 32;
    const unsigned lt = (1u << lane) - 1u;
    for (uint32_t r = r0; r < r1; r += 32) {
        const uint32_t i = r + lane;
        const bool in = i < e, p = in && (uint32_t)(v[in ? i : b] - org) < tp;
        const unsigned bal = __ballot_sync(0xffffffffu, p);
        if (in) {
            const uint32_t prank = before + __popc(bal & lt), li = i - b;
            if (li < L) {
                if (!p) sh.ml[b + (li - prank)] = (uint16_t)i;
            } else {
                if (p) sh.mr[b + (L - 1 - prank)] = (uint16_t)i;
                if (li == L) sh.m[w0] = L - prank;
            }
        }
        before += __popc(bal);
    }
    kd_group_sync(W, w0);
    const uint32_t m = L < e - b ? sh.m[w0] : 0u;
    for (uint32_t k = t; k < m; k += W * 32) {
        const uint32_t a = sh.ml[b + k], z = sh.mr[b + k];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int32_t x = sh.c[d][a];
            sh.c[d][a] = sh.c[d][z];
            sh.c[d][z] = x;
        }
        const uint32_t x = sh.id[a];
        sh.id[a] = sh.id[z];
        sh.id[z] = x;
    }
    kd_group_sync(W, w0);
}

__global__ void __launch_bounds__(KD_BTHREADS, 2) kd_block_build_kernel(
    const KdSeg* __restrict__ small, int32_t* rx, int32_t* ry, int32_t* rz, uint32_t* rid,
    uint32_t* kpos, const uint64_t* __restrict__ tree_base, KdNodes N, KdState* st, const Transform* tfs) {
    extern __shared__ __align__(16) unsigned char kd_smem[];
    KdBlockShared& sh = *reinterpret_cast<KdBlockShared*>(kd_smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    {
        const KdSeg root = small[blockIdx.x];
        const uint32_t base = root.begin, total = root.end - root.begin;
        const Transform tf = tfs[root.pad];
        const double inv[3] = {1.0 / tf.scale[0], 1.0 / tf.scale[1], 1.0 / tf.scale[2]};
        for (uint32_t i = threadIdx.x; i < total; i += KD_BTHREADS) {
            sh.c[0][i] = rx[base + i];
            sh.c[1][i] = ry[base + i];
            sh.c[2][i] = rz[base + i];
            sh.id[i] = rid[base + i];
        }
        __syncthreads();
        double lo[3], hi[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = root.lo[d];
            hi[d] = root.hi[d];
        }
        uint32_t b = 0, e = total;
        int32_t node = root.node;
        int W = KD_BWARPS, w0 = 0, top = 0;
        while (true) {
            const uint32_t count = e - b;
            const int t = threadIdx.x - w0 * 32;
            int32_t mn[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, mx[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
            for (uint32_t i = b + t; i < e; i += W * 32) {
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int32_t x = sh.c[d][i];
                    mn[d] = min(mn[d], x);
                    mx[d] = max(mx[d], x);
                }
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                mn[d] = __reduce_min_sync(0xffffffffu, mn[d]);
                mx[d] = __reduce_max_sync(0xffffffffu, mx[d]);
            }
            if (W > 1) {
                if (lane == 0) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        sh.ext[warp][d] = mn[d];
                        sh.ext[warp][3 + d] = mx[d];
                    }
                }
                kd_group_sync(W, w0);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    mn[d] = __reduce_min_sync(0xffffffffu, sh.ext[w0 + (lane & (W - 1))][d]);
                    mx[d] = __reduce_max_sync(0xffffffffu, sh.ext[w0 + (lane & (W - 1))][3 + d]);
                }
            }
            if (t < 3) {
                N.bmin[3 * node + t] = t == 0 ? mn[0] : (t == 1 ? mn[1] : mn[2]);
                N.bmax[3 * node + t] = t == 0 ? mx[0] : (t == 1 ? mx[1] : mx[2]);
            }
            bool split = count > (uint32_t)KD_LEAF;
            if (split) {
                // the children's numbers, asked for now and used after the passes
                uint32_t cid = 0;
                if (t == 0) cid = atomicAdd(&st->nodes, 2u);
                int f;
                double cut;
                kd_choose_cut(lo, hi, mn, mx, tf, f, cut);
                uint32_t t1, t2;
                const int32_t org = f == 0 ? mn[0] : (f == 1 ? mn[1] : mn[2]);
                kd_warp_thresholds(cut, tf.scale[f], f == 0 ? inv[0] : (f == 1 ? inv[1] : inv[2]), tf.offset[f],
                                   org, f == 0 ? mx[0] : (f == 1 ? mx[1] : mx[2]), t1, t2);
                const int32_t* v = sh.c[f];
                // each warp of the group takes a run of rows
                const uint32_t rows = (count + 31) / 32, per = (rows + W - 1) / W;
                const uint32_t r0 = min(b + (warp - w0) * per * 32, e), r1 = min(r0 + per * 32, e);
                uint32_t nlt = 0, neq = 0;
                for (uint32_t r = r0; r < r1; r += 32) {
                    const uint32_t i = r + lane;
                    const uint32_t x = i < e ? (uint32_t)(v[i] - org) : 0xFFFFFFFFu;
                    nlt += x < t1;
                    neq += x >= t1 && x < t2;
                }
                nlt = __reduce_add_sync(0xffffffffu, nlt);
                neq = __reduce_add_sync(0xffffffffu, neq);
                uint32_t L = nlt, eq = neq, before = 0;
                if (W > 1) {
                    if (lane == 0) {
                        sh.cnt[warp][0] = nlt;
                        sh.cnt[warp][1] = neq;
                    }
                    kd_group_sync(W, w0);
                    const uint32_t x = lane < W ? sh.cnt[w0 + lane][0] : 0u;
                    L = __reduce_add_sync(0xffffffffu, x);
                    eq = __reduce_add_sync(0xffffffffu, lane < W ? sh.cnt[w0 + lane][1] : 0u);
                    before = __reduce_add_sync(0xffffffffu, lane < warp - w0 ? x : 0u);
                }
                kd_group_pass(sh, v, b, e, org, t1, L, before, r0, r1, W, w0);
                if (eq) {
                    // pass 2 moves only points at the cut
                    const uint32_t b2 = b + L, rows2 = (count - L + 31) / 32, per2 = (rows2 + W - 1) / W;
                    const uint32_t q0 = min(b2 + (warp - w0) * per2 * 32, e), q1 = min(q0 + per2 * 32, e);
                    uint32_t before2 = 0;
                    if (W > 1) {
                        uint32_t k = 0;
                        for (uint32_t r = q0; r < q1; r += 32) {
                            const uint32_t i = r + lane;
                            k += i < e && (uint32_t)(v[min(i, e - 1)] - org) < t2;
                        }
                        k = __reduce_add_sync(0xffffffffu, k);
                        if (lane == 0) sh.cnt[warp][0] = k;
                        kd_group_sync(W, w0);
                        before2 = __reduce_add_sync(0xffffffffu, lane < warp - w0 ? sh.cnt[w0 + lane][0] : 0u);
                    }
                    kd_group_pass(sh, v, b2, e, org, t2, eq, before2, q0, q1, W, w0);
                }
                const uint32_t mid = b + kd_split_index(count, L, eq);
                if (t == 0) {
                    if (cid + 2 <= N.cap)
                        kd_write_children(N, node, cid, f, base + b, base + mid, base + e, root.pad);
                    else atomicAdd(&st->errors, 1u);
                    sh.cid[w0] = cid;
                }
                if (W > 1) {
                    kd_group_sync(W, w0);
                    cid = sh.cid[w0];
                    kd_group_sync(W, w0);  // (read by all before a half's leader writes it again)
                } else {
                    cid = __shfl_sync(0xffffffffu, cid, 0);
                }
                if (cid + 2 > N.cap) {
                    split = false;  // (the host builds again with more room)
                } else if (W > 1) {
                    // each half of the group takes a child
                    W >>= 1;
                    const int side = warp >= w0 + W ? 1 : 0;
                    w0 += side * W;
                    node = (int32_t)cid + side;
                    if (side) b = mid;
                    else e = mid;
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        if (d == f) {
                            if (side) lo[d] = cut;
                            else hi[d] = cut;
                        }
                } else {
                    // the larger child waits, the smaller one is next
                    const int big = e - mid > mid - b ? 1 : 0;
                    if (lane == 0) {
                        KdFrame16& fr = sh.stk[warp][top];
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            fr.lo[d] = d == f && big ? cut : lo[d];
                            fr.hi[d] = d == f && !big ? cut : hi[d];
                        }
                        fr.node = (int32_t)cid + big;
                        fr.b = (uint16_t)(big ? mid : b);
                        fr.e = (uint16_t)(big ? e : mid);
                    }
                    ++top;
                    __syncwarp();
                    node = (int32_t)cid + 1 - big;
                    if (big) e = mid;
                    else b = mid;
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        if (d == f) {
                            if (big) hi[d] = cut;
                            else lo[d] = cut;
                        }
                }
            }
            if (!split) {
                if (W > 1 || top == 0) break;  // a leaf of the whole group, or the warp's last one
                --top;
                __syncwarp();
                const KdFrame16 fr = sh.stk[warp][top];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    lo[d] = fr.lo[d];
                    hi[d] = fr.hi[d];
                }
                node = fr.node;
                b = fr.b;
                e = fr.e;
                __syncwarp();
            }
        }
        __syncthreads();
        const uint64_t tb = tree_base[root.pad];
        for (uint32_t i = threadIdx.x; i < total; i += KD_BTHREADS) {
            rx[base + i] = sh.c[0][i];
            ry[base + i] = sh.c[1][i];
            rz[base + i] = sh.c[2][i];
            const uint32_t id = sh.id[i];
            rid[base + i] = id;
            kpos[tb + id] = base + i;
        }
    }
}

__global__ void kd_div_kernel(const KdState* st, const int32_t* c1, const int32_t* c2, const int32_t* feat,
                              const int32_t* bmin, const int32_t* bmax, const Transform* tfs,
                              const int32_t* ntree, double* dlo, double* dhi, uint32_t cap) {
    // (a build out of room is made again: a number drawn past the capacity's last
    // pair has a place but no node in it)
    if (st->errors) return;
    const uint32_t nodes = min(st->nodes, cap);
    for (uint32_t node = blockIdx.x * blockDim.x + threadIdx.x; node < nodes; node += gridDim.x * blockDim.x) {
        if (c1[node] < 0) continue;
        const int f = feat[node];
        const Transform& tf = tfs[ntree[node]];
        dlo[node] = ref_coord(bmax[3 * c1[node] + f], tf.scale[f], tf.offset[f]);
        dhi[node] = ref_coord(bmin[3 * c2[node] + f], tf.scale[f], tf.offset[f]);
    }
}

// ---------------------------------------------------------------------------
// search replay
// ---------------------------------------------------------------------------
struct KdResult {
    double dist[KD_CAP];
    uint32_t idx[KD_CAP];
    int count, cap;
    __device__ __forceinline__ void init(int c) {
        cap = c;
        count = 0;
        dist[cap - 1] = DBL_MAX;
    }
    __device__ __forceinline__ double worst() const { return dist[cap - 1]; }
    __device__ __forceinline__ void add(double d, uint32_t id) {
        int i;
        for (i = count; i > 0; --i) {
            if (dist[i - 1] > d) {
                if (i < cap) {
                    dist[i] = dist[i - 1];
                    idx[i] = idx[i - 1];
                }
            } else break;
        }
        if (i < cap) {
            dist[i] = d;
            idx[i] = id;
        }
        if (count < cap) count++;
    }
};

// One DFS frame: the node, the bound it was entered with and, once its
// best child is done, the saved per-dimension distance.  The child order
// and cut distance are recomputed from the node when needed.
struct KdFrame {
    double mind, dst;
    int32_t node, phase;
};

__device__ __forceinline__ double kd_sq(double a, double b) {
    double d = __dsub_rn(a, b);
    return __dmul_rn(d, d);
}

// Squared FP64 distance from q to replica position i, as the reference forms it.
__device__ __forceinline__ double kd_point_dist(const KdDev& kd, const Transform& tf,
                                                const double q[3], uint32_t i) {
    const double p0 = ref_coord(kd.rx[i], tf.scale[0], tf.offset[0]);
    const double p1 = ref_coord(kd.ry[i], tf.scale[1], tf.offset[1]);
    const double p2 = ref_coord(kd.rz[i], tf.scale[2], tf.offset[2]);
    const double d0 = __dsub_rn(q[0], p0);
    const double d1 = __dsub_rn(q[1], p1);
    const double d2 = __dsub_rn(q[2], p2);
    return __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
}

// Returns false when the explicit stack overflowed (never for sane trees).
// WARP: the 32 lanes of a warp replay one row together.  Every lane walks the
// same nodes and keeps the same result list; a leaf's points are measured 32
// at a time and its candidates (below the worst distance taken at the leaf's
// start, as the reference's leaf loop takes it) are inserted by every lane in
// leaf order, so the list is the single-thread replay's exactly.
template <bool WARP>
__device__ bool kd_search(const KdDev& kd, const Transform& tf, const double q[3], KdResult& rs) {
    double dists[3] = {0.0, 0.0, 0.0};
    double distsq = 0.0;
    for (int i = 0; i < 3; ++i) {
        if (q[i] < kd.root_lo[i]) {
            dists[i] = kd_sq(q[i], kd.root_lo[i]);
            distsq = __dadd_rn(distsq, dists[i]);
        }
        if (q[i] > kd.root_hi[i]) {
            dists[i] = kd_sq(q[i], kd.root_hi[i]);
            distsq = __dadd_rn(distsq, dists[i]);
        }
    }
    KdFrame st[KD_STACK];
    int top = 0;
    st[0].node = kd.root;
    st[0].mind = distsq;
    st[0].phase = 0;
    while (top >= 0) {
        const int node = st[top].node;
        const int phase = st[top].phase;
        if (phase == 0 && kd.c1[node] < 0) {
            const double worst = rs.worst();
            const uint32_t b = kd.nb[node], e = kd.ne[node];
            if (WARP) {
                const int lane = threadIdx.x & 31;
                for (uint32_t base = b; base < e; base += 32) {
                    const uint32_t i = base + lane;
                    double dist = 0.0;
                    uint32_t id = 0;
                    bool c = false;
                    if (i < e) {
                        dist = kd_point_dist(kd, tf, q, i);
                        id = kd.rid[i];
                        c = dist < worst;
                    }
                    unsigned m = __ballot_sync(0xffffffffu, c);
                    while (m) {
                        const int l = __ffs(m) - 1;
                        m &= m - 1;
                        rs.add(__shfl_sync(0xffffffffu, dist, l), __shfl_sync(0xffffffffu, id, l));
                    }
                }
            } else {
                for (uint32_t i = b; i < e; ++i) {
                    const double dist = kd_point_dist(kd, tf, q, i);
                    if (dist < worst) rs.add(dist, kd.rid[i]);
                }
            }
            --top;
            continue;
        }
        const int idx = kd.feat[node];
        const double val = q[idx];
        const double diff1 = __dsub_rn(val, kd.dlo[node]);
        const double diff2 = __dsub_rn(val, kd.dhi[node]);
        const bool left_first = __dadd_rn(diff1, diff2) < 0;
        if (phase == 0) {
            st[top].phase = 1;
            if (top + 1 >= KD_STACK) return false;
            ++top;
            st[top].node = left_first ? kd.c1[node] : kd.c2[node];
            st[top].mind = st[top - 1].mind;
            st[top].phase = 0;
        } else if (phase == 1) {
            const double cut = left_first ? kd_sq(val, kd.dhi[node]) : kd_sq(val, kd.dlo[node]);
            const double dst = dists[idx];
            const double mind2 = __dsub_rn(__dadd_rn(st[top].mind, cut), dst);
            dists[idx] = cut;
            st[top].dst = dst;
            st[top].phase = 2;
            if (mind2 <= rs.worst()) {
                if (top + 1 >= KD_STACK) return false;
                ++top;
                st[top].node = left_first ? kd.c2[node] : kd.c1[node];
                st[top].mind = mind2;
                st[top].phase = 0;
            }
        } else {
            dists[idx] = st[top].dst;
            --top;
        }
    }
    return true;
}

// Replays the reference's search for each listed row, one warp per row, and
// writes its K neighbour ids (the reference's order) to nbr[r*K ...].
__global__ void __launch_bounds__(128) kd_search_kernel(KdDev kd, Transform tf, const int32_t* __restrict__ x,
                                 const int32_t* __restrict__ y, const int32_t* __restrict__ z,
                                 const uint32_t* __restrict__ rows, uint32_t nrows, int K,
                                 uint32_t* __restrict__ nbr, uint32_t* __restrict__ counts,
                                 uint32_t* errors, const double* row_k, uint64_t npts) {
    const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= nrows) return;  // whole warps leave together
    const uint32_t id = rows[r];
    const int Kr = row_neighbours(row_k, K, npts, id);  // <= K
    const double q[3] = {ref_coord(x[id], tf.scale[0], tf.offset[0]),
                         ref_coord(y[id], tf.scale[1], tf.offset[1]),
                         ref_coord(z[id], tf.scale[2], tf.offset[2])};
    if (Kr <= 0) {
        if (lane == 0) counts[r] = 0;
        return;
    }
    KdResult rs;
    rs.init(Kr);
    const bool ok = kd_search<true>(kd, tf, q, rs);
    for (int s = lane; s < K; s += 32) nbr[(uint64_t)r * K + s] = s < rs.count ? rs.idx[s] : 0u;
    if (lane == 0) {
        counts[r] = ok ? (uint32_t)rs.count : 0u;
        if (!ok) atomicAdd(errors, 1u);
    }
}

// Covariance of the replayed neighbour lists and the stage projections.
__global__ void kd_finish_kernel(Transform tf, const int32_t* __restrict__ x,
                                 const int32_t* __restrict__ y, const int32_t* __restrict__ z,
                                 const uint32_t* __restrict__ rows, uint32_t nrows, int K,
                                 const uint32_t* __restrict__ nbr,
                                 const uint32_t* __restrict__ counts, StageGroup g,
                                 ExceptionSink ex, int stride, int kpick) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrows) return;
    const uint32_t id = rows[r];
    const int32_t qraw[3] = {x[id], y[id], z[id]};
    // with a stride the reference keeps entries 0, stride, ... of its k*stride
    // list, unfilled entries reading point 0 (KDImpl.hpp:359-380)
    const int cnt = stride > 1 ? kpick : (int)counts[r];
    long long s1[3] = {0, 0, 0}, s2[6] = {0, 0, 0, 0, 0, 0};
    for (int s = 0; s < cnt; ++s) {
        const uint32_t j = nbr[(uint64_t)r * K + (uint64_t)s * (stride > 1 ? stride : 1)];
        const long long d0 = (long long)x[j] - qraw[0];
        const long long d1 = (long long)y[j] - qraw[1];
        const long long d2 = (long long)z[j] - qraw[2];
        s1[0] += d0;
        s1[1] += d1;
        s1[2] += d2;
        s2[0] += d0 * d0;
        s2[1] += d1 * d0;
        s2[2] += d1 * d1;
        s2[3] += d2 * d0;
        s2[4] += d2 * d1;
        s2[5] += d2 * d2;
    }
    const long long n = cnt;
    long long M[6];
    M[0] = n * s2[0] - s1[0] * s1[0];
    M[1] = n * s2[1] - s1[1] * s1[0];
    M[2] = n * s2[2] - s1[1] * s1[1];
    M[3] = n * s2[3] - s1[2] * s1[0];
    M[4] = n * s2[4] - s1[2] * s1[1];
    M[5] = n * s2[5] - s1[2] * s1[2];
    nbg_finish_row(g, tf, ex, id, cnt, M, qraw);
}

// A kNN consumer's epilogue over replayed lists (already in the reference's
// order: the replay is its search).
__global__ void kd_list_finish_kernel(Transform tf, const int32_t* __restrict__ x,
                                      const int32_t* __restrict__ y, const int32_t* __restrict__ z,
                                      const uint32_t* __restrict__ rows, uint32_t nrows, int K,
                                      const uint32_t* __restrict__ nbr,
                                      const uint32_t* __restrict__ counts, ListArgs L,
                                      ExceptionSink ex) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrows) return;
    const uint32_t id = rows[r];
    const int32_t qraw[3] = {x[id], y[id], z[id]};
    const double q64[3] = {ref_coord(qraw[0], tf.scale[0], tf.offset[0]),
                           ref_coord(qraw[1], tf.scale[1], tf.offset[1]),
                           ref_coord(qraw[2], tf.scale[2], tf.offset[2])};
    const int cnt = min((int)counts[r], K);
    uint32_t ids[KD_CAP];
    int off[KD_CAP][3];
    double d[KD_CAP];
    for (int j = 0; j < cnt; ++j) {
        const uint32_t p = nbr[(uint64_t)r * K + j];
        ids[j] = p;
        off[j][0] = x[p] - qraw[0];
        off[j][1] = y[p] - qraw[1];
        off[j][2] = z[p] - qraw[2];
        d[j] = ref_dist2(q64, qraw, off[j], tf);
    }
    list_consume(L, tf, ex, id, qraw, cnt, ids, off, d);
}

// Neighbour-set export: ascending ids into ids_out[id*K ...].
__global__ void kd_scatter_ids_kernel(const uint32_t* __restrict__ rows, uint32_t nrows, int K,
                                      const uint32_t* __restrict__ nbr,
                                      const uint32_t* __restrict__ counts, uint32_t* ids_out) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrows) return;
    uint32_t* row = ids_out + (uint64_t)rows[r] * K;
    const int cnt = (int)counts[r];
    for (int s = 0; s < cnt; ++s) {
        const uint32_t v = nbr[(uint64_t)r * K + s];
        int t = s - 1;
        while (t >= 0 && row[t] > v) {
            row[t + 1] = row[t];
            --t;
        }
        row[t + 1] = v;
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static int kd_alloc(Context* ctx, void** p, size_t bytes, KdForest* kd) {
    int rc = ctx_alloc(ctx, p, bytes);
    if (rc) return rc;
    kd->bytes += bytes;
    kd->blocks.emplace_back(*p, bytes);
    return NBG_OK;
}

static void kd_release(Context* ctx, KdForest* kd, void* p) {
    for (size_t i = 0; i < kd->blocks.size(); ++i)
        if (kd->blocks[i].first == p) {
            ctx_free(ctx, p, kd->blocks[i].second);
            kd->bytes -= kd->blocks[i].second;
            kd->blocks.erase(kd->blocks.begin() + i);
            return;
        }
}

static void kd_forest_free(Context* ctx, KdForest* f) {
    for (auto& b : f->blocks) ctx_free(ctx, b.first, b.second);
    delete f;
}

void kd_free(Context* ctx, Tile* t) {
    KdReplica* kd = t->kd;
    if (!kd) return;
    KdForest* f = kd->f;
    delete kd;
    t->kd = nullptr;
    if (f && --f->refs <= 0) kd_forest_free(ctx, f);
}

static unsigned grid_for(const Context* ctx, uint64_t n) {
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, ctx->sm_count * 8));
}

// Node arrays for `nc` nodes (nothing in them is kept).
static int kd_alloc_nodes(Context* ctx, KdForest* kd, uint32_t nc) {
    void** arrays[] = {(void**)&kd->c1, (void**)&kd->c2, (void**)&kd->feat, (void**)&kd->nb, (void**)&kd->ne,
                       (void**)&kd->ntree, (void**)&kd->bmin, (void**)&kd->bmax, (void**)&kd->dlo, (void**)&kd->dhi};
    static const size_t width[] = {4, 4, 4, 4, 4, 4, 12, 12, 8, 8};
    for (int i = 0; i < 10; ++i) {
        if (*arrays[i]) kd_release(ctx, kd, *arrays[i]);
        *arrays[i] = nullptr;
        const int rc = kd_alloc(ctx, arrays[i], (size_t)nc * width[i], kd);
        if (rc) return rc;
    }
    kd->node_cap = nc;
    return NBG_OK;
}

// A single tree's points, root and build state in one launch (ten small copies
// from the host cost as much as a level).
struct KdRoot {
    KdSeg seg;
    int32_t mn[3], mx[3];
    Transform tf;
};

__global__ void kd_init_one_kernel(const int32_t* __restrict__ x, const int32_t* __restrict__ y,
                                   const int32_t* __restrict__ z, uint32_t n, int32_t* rx, int32_t* ry,
                                   int32_t* rz, uint32_t* rid, const KdRoot root, KdNodes N, KdSeg* dst,
                                   Transform* tfs, uint64_t* bases, KdState* st, const KdState state) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        rx[i] = x[i];
        ry[i] = y[i];
        rz[i] = z[i];
        rid[i] = (uint32_t)i;
    }
    if (blockIdx.x || threadIdx.x) return;
    N.c1[0] = N.c2[0] = -1;
    N.feat[0] = 0;
    N.nb[0] = 0;
    N.ne[0] = n;
    N.ntree[0] = 0;
    for (int d = 0; d < 3; ++d) {
        N.bmin[d] = root.mn[d];
        N.bmax[d] = root.mx[d];
    }
    *dst = root.seg;
    *tfs = root.tf;
    *bases = 0;
    *st = state;
}

// The passes of one level.
template <int ROWS>
static void kd_level(const KdLevel& lv, unsigned blocks, cudaStream_t st) {
    kd_count_kernel<1, ROWS><<<blocks, KD_THREADS, 0, st>>>(lv);
    kd_classify_kernel<1, ROWS><<<blocks, KD_THREADS, 0, st>>>(lv);
    kd_swap_kernel<1><<<blocks, KD_THREADS, 0, st>>>(lv);
    kd_count_kernel<2, ROWS><<<blocks, KD_THREADS, 0, st>>>(lv);
    kd_classify_kernel<2, ROWS><<<blocks, KD_THREADS, 0, st>>>(lv);
    kd_swap_kernel<2><<<blocks, KD_THREADS, 0, st>>>(lv);
}

// One build of the forest over `tiles`.  Levels are queued without reading
// anything back: the kernels take the segment and tile counts from the device,
// and a level with nothing left exits at once.
static int kd_build(Context* ctx, KdForest* kd, Tile* const* tiles, cudaStream_t st) {
    const int T = kd->ntrees;
    std::vector<KdSeg> level0, small0;
    std::vector<int32_t> box(6 * (size_t)T);
    std::vector<int32_t> init(6 * (size_t)T);  // c1, c2, feat, nb, ne, ntree of the roots
    uint64_t largest = 0;
    for (int k = 0; k < T; ++k) {
        const Tile* t = tiles[k];
        const uint64_t b = kd->base[k], n = kd->npts[k];
        if (T > 1)
            kd_init_kernel<<<grid_for(ctx, n), 256, 0, st>>>(t->x, t->y, t->z, n, kd->rx + b, kd->ry + b,
                                                             kd->rz + b, kd->rid + b);
        // root: the tile's actual bounding box, as calculateBounds
        const GridParams& g = t->host_gp;
        const int32_t mn[3] = {g.minx, g.miny, g.minz}, mx[3] = {g.maxx, g.maxy, g.maxz};
        KdSeg root;
        root.begin = (uint32_t)b;
        root.end = (uint32_t)(b + n);
        root.node = k;
        root.pad = k;
        for (int d = 0; d < 3; ++d) {
            root.lo[d] = (double)mn[d] * t->tf.scale[d] + t->tf.offset[d];
            root.hi[d] = (double)mx[d] * t->tf.scale[d] + t->tf.offset[d];
            kd->rootbox[6 * k + d] = root.lo[d];
            kd->rootbox[6 * k + 3 + d] = root.hi[d];
            box[3 * k + d] = mn[d];
            box[3 * (T + k) + d] = mx[d];
        }
        init[k] = init[T + k] = -1;
        init[2 * T + k] = 0;
        init[3 * T + k] = (int32_t)root.begin;
        init[4 * T + k] = (int32_t)root.end;
        init[5 * T + k] = k;
        if (n > KD_BLOCK_MAX) level0.push_back(root);
        else small0.push_back(root);
        largest = std::max(largest, n);
    }
    NBG_LAUNCHED(T);
    if (level0.size() > kd->seg_cap || small0.size() > kd->small_cap) {
        set_err(ctx, "KD replica: too many trees for the segment lists");
        return NBG_ERR_UNSUPPORTED;
    }
    const KdNodes N{kd->c1, kd->c2, kd->feat, kd->nb, kd->ne, kd->bmin, kd->bmax, kd->ntree, kd->node_cap};
    KdState state{};
    state.nodes = (uint32_t)T;
    state.small = (uint32_t)small0.size();
    cudaError_t e = cudaSuccess;
    if (T == 1) {
        KdRoot root;
        root.seg = level0.empty() ? small0[0] : level0[0];
        for (int d = 0; d < 3; ++d) {
            root.mn[d] = box[d];
            root.mx[d] = box[3 + d];
        }
        root.tf = kd->tfh[0];
        kd_init_one_kernel<<<grid_for(ctx, kd->n), 256, 0, st>>>(
            tiles[0]->x, tiles[0]->y, tiles[0]->z, (uint32_t)kd->n, kd->rx, kd->ry, kd->rz, kd->rid, root, N,
            level0.empty() ? kd->small : kd->seg[0], kd->tfs, kd->bases, kd->state, state);
        e = cudaGetLastError();
    } else {
        // root nodes 0..T-1 (the host arrays outlive the copies: pageable sources are
        // taken before the calls return)
        void* const roots[] = {kd->c1, kd->c2, kd->feat, kd->nb, kd->ne, kd->ntree};
        for (int i = 0; i < 6 && !e; ++i)
            e = cudaMemcpyAsync(roots[i], &init[(size_t)i * T], T * 4, cudaMemcpyHostToDevice, st);
        if (!e) e = cudaMemcpyAsync(kd->bmin, &box[0], T * 12, cudaMemcpyHostToDevice, st);
        if (!e) e = cudaMemcpyAsync(kd->bmax, &box[3 * (size_t)T], T * 12, cudaMemcpyHostToDevice, st);
        if (!e) e = cudaMemcpyAsync(kd->tfs, kd->tfh.data(), T * sizeof(Transform), cudaMemcpyHostToDevice, st);
        if (!e) e = cudaMemcpyAsync(kd->bases, kd->base.data(), T * 8, cudaMemcpyHostToDevice, st);
        if (!e && !level0.empty())
            e = cudaMemcpyAsync(kd->seg[0], level0.data(), level0.size() * sizeof(KdSeg), cudaMemcpyHostToDevice, st);
        if (!e && !small0.empty())
            e = cudaMemcpyAsync(kd->small, small0.data(), small0.size() * sizeof(KdSeg), cudaMemcpyHostToDevice, st);
        if (!e) e = cudaMemcpyAsync(kd->state, &state, sizeof(state), cudaMemcpyHostToDevice, st);
    }
    if (e) {
        set_err(ctx, std::string("KD replica init failed: ") + cudaGetErrorString(e));
        return NBG_ERR_CUDA;
    }
    auto subtrees = [&](uint32_t ns) -> int {
        if (!ns) return NBG_OK;
        if (cudaFuncSetAttribute(kd_block_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(KdBlockShared)))
            return NBG_ERR_CUDA;
        if (kd->beside && cudaStreamWaitEvent(st, ctx->fev[0], 0)) return NBG_ERR_CUDA;
        kd_block_build_kernel<<<ns, KD_BTHREADS, sizeof(KdBlockShared), st>>>(
            kd->small, kd->rx, kd->ry, kd->rz, kd->rid, kd->kpos, kd->bases, N, kd->state, kd->tfs);
        NBG_LAUNCHED(1);
        return NBG_OK;
    };
    int cur = 0;
    auto level = [&](int c) {
        KdLevel lv;
        lv.segs = kd->seg[c];
        lv.sp = kd->split[c];
        lv.next = kd->seg[c ^ 1];
        lv.next_sp = kd->split[c ^ 1];
        lv.small = kd->small;
        lv.tile_seg = kd->tile_seg;
        lv.tile_cnt = kd->tile_cnt;
        lv.st = kd->state;
        lv.rx = kd->rx;
        lv.ry = kd->ry;
        lv.rz = kd->rz;
        lv.rid = kd->rid;
        lv.mlpos = kd->mlpos;
        lv.mrpos = kd->mrpos;
        lv.tfs = kd->tfs;
        lv.N = N;
        lv.seg_cap = kd->seg_cap;
        lv.small_cap = kd->small_cap;
        lv.tile_cap = kd->tile_cap;
        lv.tile = kd->tile;
        return lv;
    };
    if (!level0.empty()) {
        kd_roots_kernel<<<1, KD_THREADS, 0, st>>>(level(0), (uint32_t)level0.size());
        NBG_LAUNCHED(1);
        const uint32_t most = std::min<uint32_t>(kd->tile_cap, (uint32_t)ctx->sm_count * 8);
        const unsigned blocks = kd->grid_cap ? std::min(most, kd->grid_cap) : most;
        // halving gets the largest tree to KD_BLOCK_MAX in `depth` levels;
        // midpoint cuts are uneven, so a few more are queued before looking
        int depth = 1;
        while ((largest >> depth) > KD_BLOCK_MAX) ++depth;
        int queued = depth + 2;
        while (true) {
            for (int l = 0; l < queued; ++l) {
                const KdLevel lv = level(cur);
                if (lv.tile == KD_THREADS * KD_ROWS_SHORT) kd_level<KD_ROWS_SHORT>(lv, blocks, st);
                else kd_level<KD_ROWS_LONG>(lv, blocks, st);
                cur ^= 1;
            }
            NBG_LAUNCHED(6 * queued);
            e = cudaGetLastError();
            if (!e) e = cudaMemcpyAsync(&state, kd->state, sizeof(state), cudaMemcpyDeviceToHost, st);
            if (!e) e = cudaStreamSynchronize(st);
            if (e) {
                set_err(ctx, std::string("KD replica build failed: ") + cudaGetErrorString(e));
                return NBG_ERR_CUDA;
            }
            if (state.errors) return KD_RETRY;
            if (!state.segs) break;
            queued = 3;
        }
        const int rc = subtrees(state.small);  // (one launch: a block's latency is most of a small build)
        if (rc) return rc;
    } else {
        const int rc = subtrees(state.small);
        if (rc) return rc;
    }
    // divlow / divhigh from the children's extents
    kd_div_kernel<<<grid_for(ctx, kd->node_cap / 16), 256, 0, st>>>(kd->state, kd->c1, kd->c2, kd->feat, kd->bmin,
                                                                   kd->bmax, kd->tfs, kd->ntree, kd->dlo, kd->dhi,
                                                                   kd->node_cap);
    NBG_LAUNCHED(1);
    e = cudaGetLastError();
    if (!e) e = cudaMemcpyAsync(&state, kd->state, sizeof(state), cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaStreamSynchronize(st);
    if (e) {
        set_err(ctx, std::string("KD replica subtree build failed: ") + cudaGetErrorString(e));
        return NBG_ERR_CUDA;
    }
    if (state.errors) return KD_RETRY;
    kd->node_count = state.nodes;
    return NBG_OK;
}

// Builds one forest holding the replicas of every listed tile that has none.
int kd_ensure_many(Context* ctx, Tile* const* tiles, int count, cudaStream_t st, bool beside_query) {
    NBG_RANGE("nbg kd replica build");
    std::vector<Tile*> todo;
    for (int i = 0; i < count; ++i)
        if (!(tiles[i]->kd && tiles[i]->kd->built) && tiles[i]->n > 0) todo.push_back(tiles[i]);
    if (todo.empty()) return NBG_OK;
    for (Tile* t : todo) kd_free(ctx, t);
    KdForest* kd = new KdForest();
    kd->ntrees = (int)todo.size();
    uint64_t n = 0;
    for (Tile* t : todo) {
        kd->base.push_back(n);
        kd->npts.push_back(t->n);
        kd->tfh.push_back(t->tf);
        n += t->n;
    }
    if (n >= (1ull << 32) - 1) {
        delete kd;
        set_err(ctx, "KD replica: more than 2^32 points in one forest");
        return NBG_ERR_UNSUPPORTED;
    }
    kd->n = n;
    if (beside_query && n >= kKdBesideMinPoints) {
        kd->grid_cap = (uint32_t)(kKdBesideBlocksPerSm * ctx->sm_count);
        kd->beside = true;
    }
    kd->rootbox.assign(6 * (size_t)kd->ntrees, 0.0);
    const int T = kd->ntrees;
    int rc = kd_alloc(ctx, (void**)&kd->rx, n * 4, kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->ry, n * 4, kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->rz, n * 4, kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->rid, n * 4, kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->mlpos, n * 4, kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->mrpos, n * 4, kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->kpos, n * 4, kd);
    // a level's segments hold more than KD_BLOCK_MAX points each
    kd->seg_cap = (uint32_t)(n / KD_BLOCK_MAX + 1);
    for (int i = 0; i < 2; ++i) {
        if (!rc) rc = kd_alloc(ctx, (void**)&kd->seg[i], kd->seg_cap * sizeof(KdSeg), kd);
        if (!rc) rc = kd_alloc(ctx, (void**)&kd->split[i], kd->seg_cap * sizeof(KdSplit), kd);
    }
    kd->small_cap = (uint32_t)(n / 64 + 1024 + T);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->small, (size_t)kd->small_cap * sizeof(KdSeg), kd);
    kd->tile = KD_THREADS * (n <= KD_SHORT_MAX ? KD_ROWS_SHORT : KD_ROWS_LONG);
    kd->tile_cap = (uint32_t)(n / kd->tile + kd->seg_cap + 1);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->tile_seg, (size_t)kd->tile_cap * 4, kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->tile_cnt, ((size_t)kd->tile_cap + 1) * 8, kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->state, sizeof(KdState), kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->counters, 64, kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->tfs, (size_t)T * sizeof(Transform), kd);
    if (!rc) rc = kd_alloc(ctx, (void**)&kd->bases, (size_t)T * 8, kd);
    // room for leaves of 16 points on average (ordinary clouds, and clusters nested
    // at every scale, have 50 to 70 to a leaf)
    if (!rc) rc = kd_alloc_nodes(ctx, kd, (uint32_t)(n / 8 + 1024 + 2 * (uint64_t)T));
    if (!rc) rc = kd_build(ctx, kd, todo.data(), st);
    while (rc == KD_RETRY) {
        // a more uneven tree outgrew the node or subtree lists: build it again with
        // twice the room, up to one for every point
        const uint64_t nodes = std::min<uint64_t>(2 * n + 64 + 2 * (uint64_t)T, UINT32_MAX), smalls = n + T;
        if (kd->node_cap >= nodes && kd->small_cap >= smalls) {
            set_err(ctx, "KD replica build ran out of node capacity");
            rc = NBG_ERR_UNSUPPORTED;
            break;
        }
        kd_release(ctx, kd, kd->small);
        kd->small_cap = (uint32_t)std::min<uint64_t>(2 * (uint64_t)kd->small_cap, smalls);
        rc = kd_alloc(ctx, (void**)&kd->small, (size_t)kd->small_cap * sizeof(KdSeg), kd);
        if (!rc) rc = kd_alloc_nodes(ctx, kd, (uint32_t)std::min<uint64_t>(2 * (uint64_t)kd->node_cap, nodes));
        if (!rc) rc = kd_build(ctx, kd, todo.data(), st);
    }
    if (rc) {
        kd_forest_free(ctx, kd);
        return rc;
    }
    for (int k = 0; k < T; ++k) {
        KdReplica* v = new KdReplica();
        v->f = kd;
        v->tree = k;
        v->built = true;
        todo[k]->kd = v;
    }
    kd->refs = T;
    return NBG_OK;
}

int kd_ensure(Context* ctx, Tile* t, cudaStream_t st, bool beside_query) {
    Tile* one[1] = {t};
    return kd_ensure_many(ctx, one, 1, st, beside_query);
}

bool kd_built(const Tile* t) { return t->kd && t->kd->built; }

KdOrder kd_order(const Tile* t) {
    const KdForest* kd = t->kd->f;
    KdOrder o;
    o.c1 = kd->c1;
    o.c2 = kd->c2;
    o.feat = kd->feat;
    o.ne = kd->ne;
    o.dlo = kd->dlo;
    o.dhi = kd->dhi;
    o.kpos = kd->kpos;
    o.root = t->kd->tree;
    o.base = kd->base[t->kd->tree];
    return o;
}

static KdDev kd_view(const Tile* t) {
    const KdForest* kd = t->kd->f;
    const int k = t->kd->tree;
    KdDev v;
    v.rx = kd->rx;
    v.ry = kd->ry;
    v.rz = kd->rz;
    v.rid = kd->rid;
    v.c1 = kd->c1;
    v.c2 = kd->c2;
    v.feat = kd->feat;
    v.nb = kd->nb;
    v.ne = kd->ne;
    v.dlo = kd->dlo;
    v.dhi = kd->dhi;
    v.root = k;
    for (int d = 0; d < 3; ++d) {
        v.root_lo[d] = kd->rootbox[6 * k + d];
        v.root_hi[d] = kd->rootbox[6 * k + 3 + d];
    }
    return v;
}

// Searches the listed rows into per-call scratch (nbr, counts).
static int kd_search_rows(Context* ctx, Tile* t, int K, const uint32_t* rows, uint32_t nrows,
                          uint32_t** nbr, uint32_t** counts, cudaStream_t st,
                          const double* row_k = nullptr) {
    if (K > KD_CAP) return NBG_ERR_INVALID;
    KdForest* kd = t->kd->f;
    *nbr = nullptr;
    *counts = nullptr;
    int arc = ctx_alloc(ctx, (void**)nbr, (size_t)nrows * K * 4);
    if (!arc) arc = ctx_alloc(ctx, (void**)counts, (size_t)nrows * 4);
    if (arc) {
        if (*nbr) ctx_free(ctx, *nbr, (size_t)nrows * K * 4);
        *nbr = nullptr;
        *counts = nullptr;
        return arc;
    }
    cudaMemsetAsync(kd->counters + 2, 0, 4, st);
    kd_search_kernel<<<(nrows + 3) / 4, 128, 0, st>>>(kd_view(t), t->tf, t->x, t->y, t->z,
                                                          rows, nrows, K, *nbr, *counts,
                                                          kd->counters + 2, row_k, t->n);
    NBG_LAUNCHED(1);
    cudaError_t le = cudaGetLastError();
    uint32_t err = 0;
    if (le == cudaSuccess) le = cudaMemcpyAsync(&err, kd->counters + 2, 4, cudaMemcpyDeviceToHost, st);
    if (le == cudaSuccess) le = cudaStreamSynchronize(st);
    if (le != cudaSuccess) {
        set_err(ctx, std::string("exact KD rows: ") + cudaGetErrorString(le));
        return NBG_ERR_CUDA;
    }
    if (err) {
        set_err(ctx, "KD search stack overflow");
        return NBG_ERR_UNSUPPORTED;
    }
    return NBG_OK;
}

int kd_run_rows(Context* ctx, Tile* t, int K, const StageGroup& grp, const ExceptionSink& ex,
                const uint32_t* rows, uint32_t nrows, cudaStream_t st, const double* row_k,
                int stride, int kpick) {
    NBG_RANGE("nbg search replay");
    if (!nrows) return NBG_OK;
    uint32_t *nbr = nullptr, *counts = nullptr;
    int rc = kd_search_rows(ctx, t, K, rows, nrows, &nbr, &counts, st, row_k);
    if (!rc) {
        kd_finish_kernel<<<(nrows + 127) / 128, 128, 0, st>>>(t->tf, t->x, t->y, t->z, rows, nrows,
                                                              K, nbr, counts, grp, ex, stride,
                                                              kpick);
        NBG_LAUNCHED(1);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            set_err(ctx, std::string("exact KD finish: ") + cudaGetErrorString(e));
            rc = NBG_ERR_CUDA;
        }
    }
    if (nbr) ctx_free(ctx, nbr, (size_t)nrows * K * 4);
    if (counts) ctx_free(ctx, counts, (size_t)nrows * 4);
    return rc;
}

int kd_list_rows(Context* ctx, Tile* t, int K, const ListArgs& L, const ExceptionSink& ex,
                 const uint32_t* rows, uint32_t nrows, cudaStream_t st) {
    if (!nrows) return NBG_OK;
    uint32_t *nbr = nullptr, *counts = nullptr;
    int rc = kd_search_rows(ctx, t, K, rows, nrows, &nbr, &counts, st);
    if (!rc) {
        kd_list_finish_kernel<<<(nrows + 127) / 128, 128, 0, st>>>(t->tf, t->x, t->y, t->z, rows,
                                                                   nrows, K, nbr, counts, L, ex);
        NBG_LAUNCHED(1);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            set_err(ctx, std::string("exact KD list: ") + cudaGetErrorString(e));
            rc = NBG_ERR_CUDA;
        }
    }
    if (nbr) ctx_free(ctx, nbr, (size_t)nrows * K * 4);
    if (counts) ctx_free(ctx, counts, (size_t)nrows * 4);
    return rc;
}

int kd_neighbor_rows(Context* ctx, Tile* t, int K, const uint32_t* rows, uint32_t nrows,
                     uint32_t* ids_out, cudaStream_t st) {
    if (!nrows) return NBG_OK;
    uint32_t *nbr = nullptr, *counts = nullptr;
    int rc = kd_search_rows(ctx, t, K, rows, nrows, &nbr, &counts, st);
    if (!rc) {
        kd_scatter_ids_kernel<<<(nrows + 127) / 128, 128, 0, st>>>(rows, nrows, K, nbr, counts,
                                                                   ids_out);
        NBG_LAUNCHED(1);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            set_err(ctx, std::string("exact KD ids: ") + cudaGetErrorString(e));
            rc = NBG_ERR_CUDA;
        }
    }
    if (nbr) ctx_free(ctx, nbr, (size_t)nrows * K * 4);
    if (counts) ctx_free(ctx, counts, (size_t)nrows * 4);
    return rc;
}

// Test hook: copies the tile's replica out (point order as ids, and its
// tree's nodes renumbered in breadth-first order from its root, ranges
// relative to the tile).
int kd_export(Context* ctx, Tile* t, uint32_t* vind, uint32_t* nnodes, int32_t* c1, int32_t* c2,
              int32_t* feat, double* dlo, double* dhi, uint32_t* nb, uint32_t* ne, uint32_t cap,
              cudaStream_t st) {
    int rc = kd_ensure(ctx, t, st);
    if (rc) return rc;
    const KdForest* kd = t->kd->f;
    const int k = t->kd->tree;
    const uint64_t base = kd->base[k];
    const uint32_t nn = kd->node_count;
    std::vector<int32_t> hc1(nn), hc2(nn), hf(nn);
    std::vector<uint32_t> hnb(nn), hne(nn);
    std::vector<double> hlo(nn), hhi(nn);
    cudaMemcpyAsync(vind, kd->rid + base, t->n * 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(hc1.data(), kd->c1, nn * 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(hc2.data(), kd->c2, nn * 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(hf.data(), kd->feat, nn * 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(hlo.data(), kd->dlo, nn * 8, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(hhi.data(), kd->dhi, nn * 8, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(hnb.data(), kd->nb, nn * 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(hne.data(), kd->ne, nn * 4, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return NBG_ERR_CUDA;
    std::vector<int32_t> order{(int32_t)k};
    for (size_t q = 0; q < order.size(); ++q) {
        const int32_t v = order[q];
        if (hc1[v] >= 0) {
            order.push_back(hc1[v]);
            order.push_back(hc2[v]);
        }
    }
    std::vector<int32_t> newid(nn, -1);
    for (size_t q = 0; q < order.size(); ++q) newid[order[q]] = (int32_t)q;
    *nnodes = (uint32_t)order.size();
    const uint32_t m = std::min<uint32_t>(cap, (uint32_t)order.size());
    for (uint32_t q = 0; q < m; ++q) {
        const int32_t v = order[q];
        c1[q] = hc1[v] >= 0 ? newid[hc1[v]] : -1;
        c2[q] = hc2[v] >= 0 ? newid[hc2[v]] : -1;
        feat[q] = hf[v];
        dlo[q] = hlo[v];
        dhi[q] = hhi[v];
        nb[q] = (uint32_t)(hnb[v] - base);
        ne[q] = (uint32_t)(hne[v] - base);
    }
    return NBG_OK;
}

}  // namespace nbg
