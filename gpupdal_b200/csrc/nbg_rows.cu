// nbg_rows.cu — single rows answered by whole warps: the rows a faster select
// kernel hands back, and the tie rows.
//
// Both are few, and each can be long: a row beside a sparse region searches
// many rings, a tie row scans its rings again.  One thread per row left a
// launch waiting for its longest row (1.2 ms for 2,800 handed-back rows of the
// 4M-point stress tile, 0.8 ms for the 41k tie rows of the 1M-point one) with
// 5 % of the warps active.  Here a warp takes a row: the lanes look the ring's
// columns up together, then read its points 32 at a time.
//   handed-back rows  candidates below the current (K+1)-th distance are
//                     gathered in shared memory and, 32 at a time, sorted across
//                     the lanes and merged into the sorted list the lanes hold; a
//                     thread each where they are many (many_retries)
//   tie rows          strictly closer points are summed; a member of the group at
//                     the K-th distance goes to the lane of its number, and every
//                     lane ranks its member by (FP64 distance, visiting order);
//                     a tile whose ties are many gives a thread each (many_ties)
// The FP64 epilogue of a row is not warp work: a warp answers up to 32 rows,
// keeps row j's sums in lane j, and then every lane finishes its own row.
#include <algorithm>
#include <vector>

#include "nbg_common.cuh"
#include "nbg_internal.h"
#include "nbg_query.cuh"
#include "nbg_tie.cuh"

namespace nbg {

static constexpr int kRowThreads = 128;
static constexpr unsigned kAll = 0xffffffffu;

// Calls f(p, in) warp-uniformly for batches of up to 32 points (one per lane,
// `in` where there is one) of ring R: the cells scan_shell visits, with its
// pruning against `lim`.
template <class F>
__device__ __forceinline__ void warp_ring(const GridView& gv, const GridParams& g, const QueryCell& qc, int R,
                                          unsigned long long lim, const F& f) {
    const int lane = threadIdx.x & 31;
    const int w = 2 * R + 1, c = g.cell;
    const int zlo = qc.cz - R, zhi = qc.cz + R;
    for (int c0 = 0; c0 < w * w; c0 += 32) {
        // this lane's column: one run of points, and for an inner column (only
        // its cells at zlo and zhi belong to the ring) a second
        uint32_t st[2] = {0, 0}, len[2] = {0, 0};
        const int k = c0 + lane;
        if (k < w * w) {
            const int dy = k / w - R, dx = k % w - R;
            const int x = qc.cx + dx, y = qc.cy + dy;
            if (x >= 0 && x < g.gx && y >= 0 && y < g.gy) {
                const int gx_ = slab_gap(qc.qx, x, c), gy_ = slab_gap(qc.qy, y, c);
                const unsigned long long h2 =
                    (unsigned long long)((long long)gx_ * gx_ + (long long)gy_ * gy_);
                if (h2 <= lim) {
                    const int4 ci = __ldg(&gv.colinfo[(uint32_t)y * (uint32_t)g.gx + (uint32_t)x]);
                    int zr0 = zlo, zr1 = zhi;
                    if (lim < (1ull << 46)) {
                        const float s = sqrtf((float)(lim - h2)) + 1.0f;
                        zr0 = max(zr0, (int)floorf(((float)qc.qz - s) / (float)c));
                        zr1 = min(zr1, (int)floorf(((float)qc.qz + s) / (float)c));
                    }
                    auto run = [&](int i, int zl, int zh) {
                        zl = max(max(zl, zr0), ci.y);
                        zh = min(min(zh, zr1), ci.z);
                        if (zl > zh) return;
                        st[i] = __ldg(&gv.cstart[(uint32_t)ci.x + (uint32_t)(zl - ci.y)]);
                        len[i] = __ldg(&gv.cstart[(uint32_t)ci.x + (uint32_t)(zh - ci.y) + 1u]) - st[i];
                    };
                    if (max(abs(dx), abs(dy)) == R) {
                        run(0, zlo, zhi);
                    } else {
                        run(0, zlo, zlo);
                        run(1, zhi, zhi);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (i && !__any_sync(kAll, len[1] != 0)) break;
            uint32_t inc = len[i];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(kAll, inc, o);
                if (lane >= o) inc += v;
            }
            const uint32_t base = st[i] - (inc - len[i]);
            const uint32_t T = __shfl_sync(kAll, inc, 31);
            for (uint32_t t0 = 0; t0 < T; t0 += 32) {
                const uint32_t t = t0 + lane;
                int col = 0;  // the first column whose end passes t
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    if (__shfl_sync(kAll, inc, col + o - 1) <= t) col += o;
                const uint32_t pp = __shfl_sync(kAll, base, col) + t;
                const bool in = t < T;
                float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
                if (in) p = __ldg(&gv.sorted[pp]);
                f(p, in);
            }
        }
    }
}

// The 32 NR smallest keys seen, ascending over (register, lane).
template <int NR>
struct WarpTop {
    uint32_t v[NR];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int r = 0; r < NR; ++r) v[r] = 0xFFFFFFFFu;
    }
    // ascending bitonic merge of a rising-then-falling sequence over the lanes
    static __device__ __forceinline__ uint32_t clean(uint32_t k) {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int j = 16; j > 0; j >>= 1) {
            const uint32_t o = __shfl_xor_sync(kAll, k, j);
            k = (lane & j) ? max(k, o) : min(k, o);
        }
        return k;
    }
    static __device__ __forceinline__ uint32_t sort(uint32_t k) {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int s = 2; s <= 32; s <<= 1) {
            const bool up = (lane & s) == 0 || s == 32;
#pragma unroll
            for (int j = s >> 1; j > 0; j >>= 1) {
                const uint32_t o = __shfl_xor_sync(kAll, k, j);
                k = (up == ((lane & j) == 0)) ? min(k, o) : max(k, o);
            }
        }
        return k;
    }
    // one key of each lane
    __device__ __forceinline__ void insert(uint32_t key) {
        key = sort(key);
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const uint32_t rev = __shfl_xor_sync(kAll, key, 31);
            const uint32_t lo = min(v[r], rev), hi = max(v[r], rev);
            v[r] = clean(lo);
            // (the larger half falls, then rises: ascending from the other end too)
            if (r + 1 < NR) key = clean(hi);
        }
    }
    __device__ __forceinline__ uint32_t at(int i) const {
        uint32_t x = 0xFFFFFFFFu;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const uint32_t y = __shfl_sync(kAll, v[r], i & 31);
            if (r == i >> 5) x = y;
        }
        return x;
    }
};

// A row's sums from its lanes' parts.
__device__ __forceinline__ void warp_sums(int (&s)[9], int& cnt) {
#pragma unroll
    for (int k = 0; k < 9; ++k) s[k] = __reduce_add_sync(kAll, s[k]);
    cnt = __reduce_add_sync(kAll, cnt);
}

__device__ __forceinline__ void add_offsets(int (&s)[9], int ix, int iy, int iz) {
    s[0] += ix;
    s[1] += iy;
    s[2] += iz;
    s[3] += ix * ix;
    s[4] += iy * ix;
    s[5] += iy * iy;
    s[6] += iz * ix;
    s[7] += iz * iy;
    s[8] += iz * iz;
}

__device__ __forceinline__ QueryCell cell_of(const GridParams& g, int qx, int qy, int qz) {
    return QueryCell{qx, qy, qz, qx / g.cell, qy / g.cell, qz / g.cell};
}

// One row of the two-pass ring search by a warp: select_kth and its second
// pass.  True when answered (s: the sums over K points, in every lane);
// otherwise the row has been handed on.
template <int NR>
__device__ __forceinline__ bool warp_select(const QueryArgs& a, const GridParams& g, const float4 q, uint32_t id,
                                            int K, uint32_t* gather, int (&s)[9]) {
    const int lane = threadIdx.x & 31;
    const QueryCell qc = cell_of(g, __float2int_rz(q.x), __float2int_rz(q.y), __float2int_rz(q.z));
    WarpTop<NR> top;
    top.init();
    uint32_t thr = 0xFFFFFFFFu;  // the (K+1)-th key
    uint32_t held = 0;           // gathered keys (below 32 between batches)
    auto merge = [&]() {
        __syncwarp();
        top.insert((uint32_t)lane < held ? gather[lane] : 0xFFFFFFFFu);
        thr = top.at(K);
        // keys past the first 32 move down
        const uint32_t rest = held > 32u ? held - 32u : 0u;
        const uint32_t x = (uint32_t)lane < rest ? gather[32 + lane] : 0u;
        __syncwarp();
        if ((uint32_t)lane < rest) gather[lane] = x;
        held = rest;
    };
    auto take = [&](const float4 p, bool in) {
        const uint32_t key = in ? dist_key(p.x - q.x, p.y - q.y, p.z - q.z) : 0xFFFFFFFFu;
        const unsigned b = __ballot_sync(kAll, key < thr);
        if (key < thr) gather[held + __popc(b & ((1u << lane) - 1u))] = key;
        held += __popc(b);
        if (held >= 32u) merge();
    };
    bool complete = false;
    int R;
    for (R = 0; R <= a.rmax; ++R) {
        warp_ring(a.gv, g, qc, R, thr < KEY_EXACT_END ? (unsigned long long)(thr - KEY_BASE) : ~0ull, take);
        if (held) merge();
        const uint32_t kth = top.at(K - 1);
        const unsigned long long gap2 = outside_gap2(g, qc, R);
        if (gap2 == ~0ull) {
            complete = kth != 0xFFFFFFFFu;
            break;
        }
        if (kth < KEY_EXACT_END && (unsigned long long)(kth - KEY_BASE) < gap2) {
            complete = true;
            break;
        }
    }
    if (R > a.rmax) R = a.rmax;
    const uint32_t kk = top.at(K - 1), kk1 = top.at(K);
    bool tie = false;
    if (!complete || kk >= KEY_EXACT_END) {
        if (lane == 0) atomicAdd(&a.counters[2], 1u);
    } else if (kk1 == kk) {
        if (lane == 0) atomicAdd(&a.counters[1], 1u);
        tie = true;
    } else {
        int cnt = 0;
#pragma unroll
        for (int k = 0; k < 9; ++k) s[k] = 0;
        for (int r = 0; r <= R; ++r)
            warp_ring(a.gv, g, qc, r, (unsigned long long)(kk - KEY_BASE), [&](const float4 p, bool in) {
                const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                if (in && dist_key(dx, dy, dz) <= kk) {
                    add_offsets(s, small_int(dx), small_int(dy), small_int(dz));
                    ++cnt;
                }
            });
        warp_sums(s, cnt);
        if (cnt == K) return true;  // (always: a complete row without a tie)
    }
    if (lane == 0) defer_row(a, id, tie, kk, R);
    return false;
}

// Covariance numerators of a row's sums.
__device__ __forceinline__ void finish_sums(const StageGroup& grp, const Transform& tf, const ExceptionSink& ex,
                                            uint32_t id, int n, const int (&s)[9], const int32_t qraw[3]) {
    const long long N = n;
    const long long M[6] = {N * s[3] - (long long)s[0] * s[0], N * s[4] - (long long)s[1] * s[0],
                            N * s[5] - (long long)s[1] * s[1], N * s[6] - (long long)s[2] * s[0],
                            N * s[7] - (long long)s[2] * s[1], N * s[8] - (long long)s[2] * s[2]};
    nbg_finish_row(grp, tf, ex, id, n, M, qraw);
}

// Rows a warp takes: as many as spread the rows over all warps of the launch,
// 32 at most (one for each lane to finish).
__device__ __forceinline__ uint32_t rows_per_warp(uint32_t rows) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    return min(32u, (rows + warps - 1) / warps);
}

// Rows handed back by a select kernel (a.rows, a.nq_dev entries), searched and
// finished (their sums slots hold cnt = 0, so the finish pass over the other
// rows, which may run at the same time, skips them).
template <int NR>
__device__ __forceinline__ void retry_finish_rows(const QueryArgs& a, const uint32_t* rows, const uint32_t nr,
                                                  uint32_t (*s_gather)[64]) {
    const uint32_t rpw = rows_per_warp(nr);
    const int lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = gridDim.x * (blockDim.x >> 5);
    const GridParams g = *a.gp;
    for (uint32_t r0 = warp * rpw; r0 < nr; r0 += warps * rpw) {
        const uint32_t m = min(rpw, nr - r0);
        float4 mq = make_float4(0.f, 0.f, 0.f, 0.f);  // this lane's row
        int mk = -1;                                   // its neighbours (-1: nothing to finish)
        int ms[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        if ((uint32_t)lane < m) mq = __ldg(&a.qpts[__ldg(&rows[r0 + lane])]);
        for (uint32_t j = 0; j < m; ++j) {
            const float4 q = make_float4(__shfl_sync(kAll, mq.x, j), __shfl_sync(kAll, mq.y, j),
                                         __shfl_sync(kAll, mq.z, j), __shfl_sync(kAll, mq.w, j));
            const uint32_t id = __float_as_uint(q.w);
            const int K = row_neighbours(a.row_k, a.K, a.n, id);
            int s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            // (no neighbours: the reference's covariance of an empty set is zero)
            const bool ok = K <= 0 || warp_select<NR>(a, g, q, id, K, s_gather[threadIdx.x >> 5], s);
            if (ok && (uint32_t)lane == j) {
                mk = max(K, 0);
#pragma unroll
                for (int k = 0; k < 9; ++k) ms[k] = s[k];
            }
            __syncwarp();
        }
        if (mk >= 0) {
            const int32_t qraw[3] = {__float2int_rz(mq.x) + g.minx, __float2int_rz(mq.y) + g.miny,
                                     __float2int_rz(mq.z) + g.minz};
            finish_sums(a.grp, a.tf, a.ex, __float_as_uint(mq.w), mk, ms, qraw);
        }
        __syncwarp();
    }
}

template <int NR>
__global__ void __launch_bounds__(kRowThreads) knn_retry_finish_kernel(const QueryArgs a, uint32_t most) {
    __shared__ uint32_t s_gather[kRowThreads / 32][64];
    const uint32_t nr = *a.nq_dev;
    if (nr < most) retry_finish_rows<NR>(a, a.rows, nr, s_gather);  // (else a thread each)
}

// The same for the tiles of a batch: blockIdx.y's jobs, gridDim.y apart.
template <int NR>
__global__ void __launch_bounds__(kRowThreads) knn_retry_batch_kernel(const BatchJob* __restrict__ jobs, int njobs,
                                                                      uint32_t most) {
    __shared__ uint32_t s_gather[kRowThreads / 32][64];
    if (most != 0xFFFFFFFFu && retry_total(jobs, njobs) >= most) return;
    for (int j = blockIdx.y; j < njobs; j += gridDim.y) {
        const QueryArgs& a = jobs[j].q;
        retry_finish_rows<NR>(a, a.retry_rows, a.counters[6], s_gather);
    }
}

// One tie row by a warp (see tie_row): the sums over its K points, in every
// lane.  False when the row went to the search replay.
__device__ __forceinline__ bool warp_tie(const TieArgs& a, const GridParams& g, uint2 e, int K, int (&s)[9]) {
    const int lane = threadIdx.x & 31;
    const uint32_t id = e.x, kk = KEY_BASE + (e.y & 0xFFFFFFu);
    const int R = (int)(e.y >> 24);
    const int32_t qraw[3] = {__ldg(&a.x[id]), __ldg(&a.y[id]), __ldg(&a.z[id])};
    const QueryCell qc = cell_of(g, qraw[0] - g.minx, qraw[1] - g.miny, qraw[2] - g.minz);
    const float qx = (float)qc.qx, qy = (float)qc.qy, qz = (float)qc.qz;
#pragma unroll
    for (int k = 0; k < 9; ++k) s[k] = 0;
    int less = 0;
    uint32_t gcnt = 0, gid = 0;  // the group's size; this lane's member
    int g0 = 0, g1 = 0, g2 = 0;
    for (int r = 0; r <= R; ++r)
        warp_ring(a.gv, g, qc, r, (unsigned long long)(kk - KEY_BASE), [&](const float4 p, bool in) {
            const float dx = p.x - qx, dy = p.y - qy, dz = p.z - qz;
            const uint32_t key = in ? dist_key(dx, dy, dz) : 0xFFFFFFFFu;
            if (key < kk) {
                add_offsets(s, small_int(dx), small_int(dy), small_int(dz));
                ++less;
            }
            unsigned b = __ballot_sync(kAll, key == kk);
            // (past 32 the row goes to the search replay)
            while (b && gcnt <= 32u) {  // the lane of the member's number takes it
                const int src = __ffs(b) - 1;
                b &= b - 1;
                const float mx = __shfl_sync(kAll, dx, src), my = __shfl_sync(kAll, dy, src),
                            mz = __shfl_sync(kAll, dz, src);
                const uint32_t mi = __shfl_sync(kAll, __float_as_uint(p.w), src);
                if ((uint32_t)lane == gcnt) {
                    gid = mi;
                    g0 = small_int(mx);
                    g1 = small_int(my);
                    g2 = small_int(mz);
                }
                ++gcnt;
            }
        });
    const int m = K - __reduce_add_sync(kAll, less);
    if (gcnt > 32u || m <= 0 || m > (int)gcnt) {
        if (lane == 0) {
            const uint32_t slot = atomicAdd(&a.counters[0], 1u);
            a.exact_rows[slot] = id;
        }
        return false;
    }
    const bool member = (uint32_t)lane < gcnt;
    const double q64[3] = {ref_coord(qraw[0], a.tf.scale[0], a.tf.offset[0]),
                           ref_coord(qraw[1], a.tf.scale[1], a.tf.offset[1]),
                           ref_coord(qraw[2], a.tf.scale[2], a.tf.offset[2])};
    const int off[3] = {g0, g1, g2};
    const double d = ref_dist2(q64, qraw, off, a.tf);
    int lt = 0, le = 0;
    for (uint32_t u = 0; u < gcnt; ++u) {
        const double du = __shfl_sync(kAll, d, u);
        lt += du < d;
        le += du <= d;
    }
    // members at the m-th smallest FP64 distance; when they all have one offset
    // any of them gives the same sums, and no tree is walked (see tie_row)
    const bool last = member && lt < m && m <= le;
    const unsigned lm = __ballot_sync(kAll, last);
    const int ref = __ffs(lm) - 1;
    const int r0 = __shfl_sync(kAll, g0, ref), r1 = __shfl_sync(kAll, g1, ref), r2 = __shfl_sync(kAll, g2, ref);
    const bool any_order = __all_sync(kAll, !last || (g0 == r0 && g1 == r1 && g2 == r2));
    int rank = lt;
    // (members at other distances are in or out by distance alone)
    if (last && any_order) rank += __popc(lm & ((1u << lane) - 1u));
    if (!any_order) {
        const uint32_t mine = last ? __ldg(&a.kd.kpos[a.kd.base + gid]) : 0u;
        for (unsigned x = lm; x; x &= x - 1) {
            const int u = __ffs(x) - 1;
            const uint32_t other = __shfl_sync(kAll, mine, u);
            if (last && u != lane) rank += kd_meets_first(a.kd, q64, other, mine);
        }
    }
    __syncwarp();
    if (member && rank < m) add_offsets(s, g0, g1, g2);
    int dummy = 0;
    warp_sums(s, dummy);
    return true;
}

// Up to 32 tie rows by a warp, rows r0 .. r0 + m - 1 of a.ties.
__device__ __forceinline__ void warp_tie_rows(const TieArgs& a, uint32_t r0, uint32_t m) {
    const int lane = threadIdx.x & 31;
    const GridParams g = *a.gp;
    uint2 me = make_uint2(0, 0);
    if ((uint32_t)lane < m) me = a.ties[r0 + lane];
    int mk = -1;
    int ms[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t j = 0; j < m; ++j) {
        const uint2 e = make_uint2(__shfl_sync(kAll, me.x, j), __shfl_sync(kAll, me.y, j));
        const int K = row_neighbours(a.row_k, a.K, a.n, e.x);
        int s[9];
        const bool ok = warp_tie(a, g, e, K, s);
        if (ok && (uint32_t)lane == j) {
            mk = K;
#pragma unroll
            for (int k = 0; k < 9; ++k) ms[k] = s[k];
        }
        __syncwarp();
    }
    if (mk >= 0) {
        const int32_t qraw[3] = {__ldg(&a.x[me.x]), __ldg(&a.y[me.x]), __ldg(&a.z[me.x])};
        finish_sums(a.grp, a.tf, a.ex, me.x, mk, ms, qraw);
    }
    __syncwarp();
}

// Tie rows counted on the device (a.nties: the list's capacity), or a.nties
// rows when `count` is null; a count of `most` or more is left to the thread form.
__global__ void __launch_bounds__(kRowThreads) knn_tie_kernel(const TieArgs a, const uint32_t* count, uint32_t most) {
    const uint32_t nt = count ? min(*count, a.nties) : a.nties;
    if (nt >= most) return;
    const uint32_t rpw = rows_per_warp(nt);
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t r0 = warp * rpw; r0 < nt; r0 += warps * rpw) warp_tie_rows(a, r0, min(rpw, nt - r0));
}

// The tie rows of many tiles in one launch: jobs[j] is tile j's arguments, its
// rows are entries first[j] .. first[j+1]-1 of the launch, taken in runs of
// `run` that do not cross tiles.
__global__ void __launch_bounds__(kRowThreads) knn_tie_batch_kernel(const TieArgs* __restrict__ jobs,
                                                                    const uint64_t* __restrict__ first, int njobs,
                                                                    uint64_t runs, uint32_t run) {
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    if (warp >= runs) return;
    int lo = 0, hi = njobs;  // the job whose runs hold this one
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first[mid] <= warp) lo = mid;
        else hi = mid;
    }
    const TieArgs& a = jobs[lo];
    const uint32_t r0 = (uint32_t)(warp - first[lo]) * run;
    warp_tie_rows(a, r0, min(run, a.nties - r0));
}

// ---- launches -----------------------------------------------------------------
static constexpr uint64_t kRowBlocksPerSm = 16;

// nbg_query.cu: a thread per row
int launch_tie_threads(const TieArgs& a, cudaStream_t stream);
int launch_tie_threads_batch(const TieArgs* jobs, const uint64_t* first, int njobs, uint64_t rows,
                             cudaStream_t stream);
int launch_retry_threads(const QueryArgs& q, int slots, uint32_t least, int sms, cudaStream_t stream);
int launch_retry_threads_batch(int slots, const BatchJob* jobs, int njobs, uint32_t least, int sms,
                               cudaStream_t stream);

// From this many of a launch's `rows` up, its tie rows get a thread each, below a
// warp each.  A warp's lanes read one row's points side by side and leave no
// tail, but sort, rank and sum across lanes; neighbouring threads of a dense
// list walk the same cells.  Thread / warp, K = 17, ms: scattered ties (2 % of a
// cloud with duplicates) 0.48 / 0.23 for 44k rows of 2M, 1.15 / 1.09 for 350k of
// 16M; 7 % of a batch whose density falls with distance 10.1 / 6.8; a raster's
// (8 %) 0.30 / 0.47 for 82k of 1M; a lattice's (all) 0.23 / 0.19 for 20k, 0.24 / 0.41
// for 50k, 2.4 / 8.2 for 1M.
uint32_t many_ties(int sms, uint64_t rows) {
    return (uint32_t)std::max<uint64_t>((uint64_t)sms * 256, rows / 13);
}

// The same for the rows a select hands back: few of them are the hard rows, far
// from one another, with a long tail; when a fifth of a large tile is handed back
// the select as a whole did not fit it, and neighbouring threads walk the same
// cells again.  Whole calls, thread / warp, ms: 1 - 2 % of 4M mixture points 13.5 /
// 12.6 (K = 65) and 8.7 / 8.6 (K = 33); 17 % of 500k points far apart in raw units
// 18.9 / 12.7; 29 % of 1M points whose density falls with distance 160 / 197; 39 %
// of 500k far points 22.8 / 42.6; all of a 1M wall 24.4 / 31.5, of a 100k one 1.1 /
// 1.8; 77 % of 100k far points 20.0 / 22.2, 35 % of them 19.4 / 11.1.  A thread's
// list costs in proportion to its slots, a warp's by the third register at most:
// from 65 slots up half the rows (K = 65, 500k far points: 32 % 43.8 / 35.4, 39 %
// 93 / 85, all 182 / 219).
uint32_t many_retries(int sms, int slots, uint64_t rows) {
    return (uint32_t)std::max<uint64_t>((uint64_t)sms * 512, slots > 64 ? rows / 2 : rows / 5);
}

// may_be_many: the thread form is launched too (an idle launch costs 3 us)
int launch_retry_finish(const QueryArgs& q, int slots, bool may_be_many, int sms, cudaStream_t stream) {
    const uint64_t rows = q.nq;  // the most there can be
    const uint32_t many = may_be_many ? many_retries(sms, slots, rows) : 0xFFFFFFFFu;
    if (rows >= many) {
        const int rc = launch_retry_threads(q, slots, many, sms, stream);
        if (rc) return rc;
    }
    const unsigned blocks =
        (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((rows + 3) / 4, (uint64_t)sms * kRowBlocksPerSm));
    if (slots <= 32) knn_retry_finish_kernel<1><<<blocks, kRowThreads, 0, stream>>>(q, many);
    else if (slots <= 64) knn_retry_finish_kernel<2><<<blocks, kRowThreads, 0, stream>>>(q, many);
    else knn_retry_finish_kernel<3><<<blocks, kRowThreads, 0, stream>>>(q, many);
    NBG_LAUNCHED(1);
    return cudaGetLastError() == cudaSuccess ? NBG_OK : NBG_ERR_CUDA;
}

// Blocks for a batch's jobs, at least four a job; more jobs than fill the GPU so
// take turns (gridDim.y ends at 65535).
dim3 retry_batch_grid(int njobs, int sms) {
    const unsigned y = (unsigned)std::min<uint64_t>((uint64_t)njobs, (uint64_t)sms * kRowBlocksPerSm / 4);
    return dim3((unsigned)((uint64_t)sms * kRowBlocksPerSm / y), y);
}

// `rows`: the rows of the jobs' tiles.
int launch_retry_batch(int slots, const BatchJob* jobs, int njobs, uint64_t rows, bool may_be_many, int sms,
                       cudaStream_t stream) {
    if (!njobs) return NBG_OK;
    uint32_t many = many_retries(sms, slots, rows);
    if (may_be_many && rows >= many) {
        const int rc = launch_retry_threads_batch(slots, jobs, njobs, many, sms, stream);
        if (rc) return rc;
    } else {
        many = 0xFFFFFFFFu;  // (there cannot be as many)
    }
    const dim3 grid = retry_batch_grid(njobs, sms);
    if (slots <= 32) knn_retry_batch_kernel<1><<<grid, kRowThreads, 0, stream>>>(jobs, njobs, many);
    else if (slots <= 64) knn_retry_batch_kernel<2><<<grid, kRowThreads, 0, stream>>>(jobs, njobs, many);
    else knn_retry_batch_kernel<3><<<grid, kRowThreads, 0, stream>>>(jobs, njobs, many);
    NBG_LAUNCHED(1);
    return cudaGetLastError() == cudaSuccess ? NBG_OK : NBG_ERR_CUDA;
}

int launch_tie_rows(const TieArgs& a, const uint32_t* count, int sms, cudaStream_t stream) {
    const uint32_t many = many_ties(sms, a.of_rows);
    if (a.ids_out || (!count && a.nties >= many)) return launch_tie_threads(a, stream);
    const unsigned blocks =
        (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(((uint64_t)a.nties + 3) / 4, (uint64_t)sms * kRowBlocksPerSm));
    knn_tie_kernel<<<blocks, kRowThreads, 0, stream>>>(a, count, many);
    NBG_LAUNCHED(1);
    return cudaGetLastError() == cudaSuccess ? NBG_OK : NBG_ERR_CUDA;
}

int launch_tie_batch(Context* ctx, const std::vector<TieArgs>& jobs, cudaStream_t stream) {
    uint64_t total = 0;
    uint64_t rows = 0;
    for (const TieArgs& j : jobs) {
        total += j.nties;
        rows += j.of_rows;
    }
    if (!total) return NBG_OK;
    const uint64_t warps = (uint64_t)ctx->sm_count * kRowBlocksPerSm * (kRowThreads / 32);
    const bool threads = total >= many_ties(ctx->sm_count, rows);
    const uint32_t run = threads ? 1u : (uint32_t)std::min<uint64_t>(32, std::max<uint64_t>(1, total / warps));
    std::vector<uint64_t> first(1, 0);
    for (const TieArgs& j : jobs) first.push_back(first.back() + (j.nties + run - 1) / run);
    TieArgs* djobs = nullptr;
    uint64_t* dfirst = nullptr;
    const size_t jb = jobs.size() * sizeof(TieArgs), fb = first.size() * sizeof(uint64_t);
    int rc = ctx_alloc(ctx, (void**)&djobs, jb);
    if (!rc) rc = ctx_alloc(ctx, (void**)&dfirst, fb);
    // pageable sources: both copies complete before they return
    if (!rc) rc = host_to_device(ctx, djobs, jobs.data(), jb, stream);
    if (!rc) rc = host_to_device(ctx, dfirst, first.data(), fb, stream);
    if (!rc && threads) {
        rc = launch_tie_threads_batch(djobs, dfirst, (int)jobs.size(), total, stream);
    } else if (!rc) {
        const uint64_t runs = first.back();
        knn_tie_batch_kernel<<<(unsigned)((runs * 32 + kRowThreads - 1) / kRowThreads), kRowThreads, 0, stream>>>(
            djobs, dfirst, (int)jobs.size(), runs, run);
        NBG_LAUNCHED(1);
        if (cudaGetLastError() != cudaSuccess) rc = NBG_ERR_CUDA;
    }
    // the job table is read by the kernel: return it to the cache only after
    if (cudaStreamSynchronize(stream) != cudaSuccess && !rc) rc = NBG_ERR_CUDA;
    if (djobs) ctx_free(ctx, djobs, jb);
    if (dfirst) ctx_free(ctx, dfirst, fb);
    return rc;
}

}  // namespace nbg
