// nbg_group.cu — group select: a warp's 32 neighbouring queries share one
// candidate list.
//
// Same answer as the per-thread select (knn_select_kernel, nbg_query.cu): for
// each row, the exact integer neighbourhood sums of its K nearest points (or
// their ids, for the neighbour-set export), or the row handed to the
// tie-order resolver / the exact KD path.  The per-thread ring search gives
// every lane its own rings of cells, so a warp walks the union of its lanes'
// cells with most lanes masked, and pays the whole top-list insertion network
// (2 (K+1) min/max) whenever any lane inserts.  Here
//
//   order     a warp's 32 queries are one clump of the clump order
//             (clump_kernel, nbg_grid.cu: median splits of a block of 1024
//             points), spatially compact at any density
//   members   the clump and its siblings are the first list: after it every
//             lane holds K + 1 real points, so its (K+1)-th distance bounds
//             the search
//   rounds    a round takes the open lanes near the one of smallest bound and
//             a margin that covers theirs.  Its list is the points within the
//             margin of the box around the round's queries, found by a walk
//             down the tree of clump boxes (32 boxes a step, one per lane; the
//             warp's own block first, so the bounds fall before the rest of
//             the tree is tested).  A lane whose K-th lies inside the margin is
//             answered: the points left out are farther.  The others see the
//             shell between this margin and a wider one
//   scan      each lane forms the exact integer squared distance of every
//             staged candidate (uniform loop, two at once in packed f32
//             arithmetic) and appends the ones below its bound to a short list
//             of its own in shared memory; when a lane's list is full all lanes
//             sort theirs (a register network) and merge it into their sorted
//             top list (one bitonic merge).  A candidate costs a compare and a
//             store, and the network runs once per up to M of them with every
//             lane active
//   sums      keys pack the squared distance above the candidate's index in
//             the warp's list, so the K nearest are read back directly
//
// A list of more candidates than the index field holds is started over with
// the bounds it gave (`again`); rows that overflow it twice, or whose distances
// pass the key's field, go to the retry launch (warps of their own) through a
// list read on the device.  Ties and far rows are decided exactly as the
// per-thread select decides them.
//
// Bound by instruction issue (the data lie in L2): 2.7 candidates are scanned
// for each of the K + 1 kept, and the merges cost about as much as the scan.  Measured
// select times at the densities of the synthetic clouds, per-thread two-pass
// search -> this kernel: K = 65, 1.5M points, 8.9 -> 3.6 ms; K = 33, 4.7M
// points of 24 tiles, 12.6 -> 5.8 ms.
#include <climits>

#include "nbg_common.cuh"
#include "nbg_internal.h"
#include "nbg_query.cuh"

namespace nbg {

// ---- register networks -----------------------------------------------------
__device__ __forceinline__ void cmp_swap(uint32_t& a, uint32_t& b) {
    const uint32_t lo = min(a, b);
    b = max(a, b);
    a = lo;
}

// Batcher's odd-even merge sort of N (a power of two) registers, ascending.
template <int N, int P, int K>
__device__ __forceinline__ void oe_stage(uint32_t (&v)[N]) {
#pragma unroll
    for (int j = K % P; j + K < N; j += 2 * K)
#pragma unroll
        for (int i = 0; i < K; ++i)
            if (i + j + K < N && (i + j) / (2 * P) == (i + j + K) / (2 * P))
                cmp_swap(v[i + j], v[i + j + K]);
    if constexpr (K > 1) oe_stage<N, P, K / 2>(v);
}
template <int N, int P = 1>
__device__ __forceinline__ void oe_sort(uint32_t (&v)[N]) {
    oe_stage<N, P, P>(v);
    if constexpr (2 * P < N) oe_sort<N, 2 * P>(v);
}

// Shared-memory list of a lane: `at` is the shared-space address of its next
// slot (128 bytes apart).  Written as predicated instructions: a branch per
// candidate, with its reconvergence, costs more than the candidate.
__device__ __forceinline__ void append_below(uint32_t& at, uint32_t kb, uint32_t kthr, uint32_t key) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.lt.u32 p, %1, %2;\n\t"
        "@p st.shared.u32 [%0], %3;\n\t"
        "@p add.u32 %0, %0, 128;\n\t}"
        : "+r"(at)
        : "r"(kb), "r"(kthr), "r"(key));
}
// Takes a list slot's key and leaves the slot empty.
__device__ __forceinline__ uint32_t list_take(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];\n\tst.shared.u32 [%1], %2;" : "=&r"(v) : "r"(addr), "r"(0xFFFFFFFFu));
    return v;
}

// Two floats in one register pair, and arithmetic on both at once.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}

constexpr int next_pow2(int n) {
    int p = 1;
    while (p < n) p <<= 1;
    return p;
}

// Half-cleaners of a bitonic (rising then falling) sequence of N registers,
// taken as the last N of the next power of two with -inf in front (those
// comparators change nothing and are left out).
template <int N, int D>
__device__ __forceinline__ void bitonic_clean(uint32_t (&v)[N]) {
    constexpr int S = next_pow2(N) - N;
#pragma unroll
    for (int i = 0; i + D < N; ++i)
        if (((i + S) & D) == 0) cmp_swap(v[i], v[i + D]);
    if constexpr (D > 1) bitonic_clean<N, D / 2>(v);
}

// The N smallest of a (ascending) and b (ascending), into a (ascending).
template <int N, int M>
__device__ __forceinline__ void merge_low(uint32_t (&a)[N], const uint32_t (&b)[M]) {
#pragma unroll
    for (int i = (N > M ? N - M : 0); i < N; ++i) a[i] = min(a[i], b[N - 1 - i]);
    bitonic_clean<N, next_pow2(N) / 2>(a);
}

// ---- shape of the kernel for a top list of KS slots --------------------------
template <int KS>
struct WarpShape {
    // warps work alone; two to a block so that a long one holds little else
    static constexpr int kThreads = 64;
    static constexpr int kMinBlocks = KS > 40 ? 6 : (KS > 20 ? 10 : 12);
    static constexpr int kBatch = KS > 40 ? 32 : 16;  // appended candidates per merge
    static constexpr int kIdxBits = KS > 40 ? 11 : 10;
    static constexpr uint32_t kCap = 1u << kIdxBits;
    static constexpr uint32_t kD2Max = (1u << (32 - kIdxBits)) - 1u;  // first distance past the field
    static constexpr int kMaxMargin = KS > 40 ? 1447 : 2047;  // (group_max_margin) its square < kD2Max
    static constexpr uint32_t kMemClumps = (KS + 31) / 32;  // clumps whose points bound the search
    static constexpr size_t kBufBytes = (size_t)kBatch * 32 * 4;
    static constexpr size_t kStageBytes = 3 * 64 * 4;
    static constexpr size_t kPosBytes = (size_t)kCap * 4;
    static constexpr size_t kWarpBytes = kBufBytes + kStageBytes + kPosBytes;
    static constexpr size_t kSmem = kThreads / 32 * kWarpBytes;
};

// Smallest ring R of the grid's cube rings around qc whose outside lies
// beyond squared distance d2 (what the tie-order resolver rescans).
__device__ __forceinline__ int ring_for(const GridParams& g, const QueryCell& qc, uint32_t d2) {
    int R = 0;
    while (R < 256 && outside_gap2(g, qc, R) <= (unsigned long long)d2) ++R;
    return R;
}

__device__ __forceinline__ int ceil_sqrt(uint32_t d2) {
    int s = (int)sqrtf((float)d2);
    while ((uint32_t)s * (uint32_t)s < d2) ++s;
    return s;
}

// One warp: the rows of slots s0 .. s0 + 31 (or those entries of the launch's
// row list).
template <int KS>
__device__ __forceinline__ void group_warp(const QueryArgs& a, const uint64_t s0, const float margin0,
                                           unsigned char* wb) {
    using S = WarpShape<KS>;
    constexpr int M = S::kBatch, IB = S::kIdxBits;
    const int lane = threadIdx.x & 31;
    // this lane's appended keys, 32 words apart
    const uint32_t buf = (uint32_t)__cvta_generic_to_shared(wb) + (uint32_t)lane * 4u;
    float* stage = (float*)(wb + S::kBufBytes);  // x, y, z of up to 64 candidates, 64 apart
    uint32_t* cpos = (uint32_t*)(wb + S::kBufBytes + S::kStageBytes);
    const float finf = __int_as_float(0x7F800000);
    const uint32_t n = (uint32_t)a.n;
    // lane l keeps level l of the box tree (nodes, first box) and of the walk
    // down it (children left, node)
    uint32_t lv_count = 0, lv_left = 0, lv_node = 0;
    uint64_t lv_off = 0;
    int ltop;  // first level of at most 32 nodes
    uint32_t nclumps;
    {
        const ClumpTree tr(n);
        ltop = tr.top;
        nclumps = tr.count[0];
#pragma unroll
        for (int l = 0; l < ClumpTree::kLevels; ++l)
            if (lane == l) {
                lv_count = tr.count[l];
                lv_off = tr.off[l];
            }
    }
    const GridParams g = *a.gp;
    const bool valid = s0 + lane < (a.rows ? a.nq : a.n);
    const uint32_t pos = !valid ? 0u : a.rows ? __ldg(&a.rows[s0 + lane]) : (uint32_t)(s0 + lane);
    const float4 q = valid ? __ldg(&a.qpts[pos]) : make_float4(finf, finf, finf, 0.f);

    // ---- the lane's query
    const uint32_t id = __float_as_uint(q.w);
    const int K = valid ? row_neighbours(a.row_k, a.K, a.n, id) : 0;
    const int qx = __float2int_rz(q.x), qy = __float2int_rz(q.y), qz = __float2int_rz(q.z);
    bool retry = valid && K <= 0;  // rows without neighbours: the retry launch
    bool done = K <= 0;
    TopK<KS> top;  // the last two slots are the K-th and (K+1)-th
    top.init(done ? 0 : KS - (K + 1));
    uint32_t bnd = KEY_BASE + S::kD2Max;  // distances from here up do not matter
    uint32_t kthr = done ? 0u : bnd;      // the same while the lane takes part in a scan
    uint32_t at = buf;                    // next slot of the lane's list
    for (int k = 0; k < M; ++k) list_take(buf + k * 128);
    const uint64_t nqx = pack2(-q.x, -q.x), nqy = pack2(-q.y, -q.y), nqz = pack2(-q.z, -q.z);
    const uint64_t bias = pack2(8388608.0f, 8388608.0f);  // the integer distance in the mantissa (dist_key)

    // ---- lists.  First the members: the clumps around the warp's first row
    // bound every lane's search.  Then one list per margin of a round; a round
    // finishes the open lanes near the one of smallest bound.
    const uint32_t c0 = __shfl_sync(0xffffffffu, pos, 0) >> 5;
    // (a last clump of few points takes one more)
    const uint32_t want = min(S::kMemClumps + (c0 + 1 == nclumps && (n & 31u) ? 1u : 0u), nclumps);
    // siblings: the halves of one box of 64 points, then of one of 128
    uint32_t mem0 = S::kMemClumps == 1 ? c0 : (c0 & ~1u);
    if (S::kMemClumps == 3) mem0 -= (c0 >> 1) & 1u;
    mem0 = min(mem0, nclumps - want);
    const uint32_t own = c0 >> 5;  // the block a walk starts with
    // (beyond 3 kMaxMargin it limits neither a margin nor a round's span)
    const int mcap = (int)fminf(margin0 * 8.0f * g.r1 * sqrtf((float)a.K), 3.0f * S::kMaxMargin) + 1;
    bool again = false;      // the lane's list started over: members are not in it
    bool in = !done;         // takes part in the current round
    bool members = true;     // (uniform) the current list is the members'
    bool mem_in = true;      // (uniform) the round's lanes hold the members already
    int m = 0;               // the round's margin
    float prev2 = -1.0f;     // points up to this squared distance of the round's box are done
    float filt2 = finf;      // points up to this one are taken
    float fl0 = 0.f, fl1 = 0.f, fl2 = 0.f, fh0 = 0.f, fh1 = 0.f, fh2 = 0.f;  // the round's box
    uint32_t nc = 0;         // candidates of the round's list scanned
    uint32_t base = 0;       // the list's first index past the members
    for (int guard = 0; guard < 4096; ++guard) {
        // ---- gather and scan one list
        bool over = false;
        uint32_t nst = 0, first = mem0;
        unsigned mask = members ? (1u << want) - 1u : 0u;
        bool walking = !members;  // clumps are still to be found
        bool own_first = ltop > 0;
        int L = own_first ? 1 : ltop + 1;  // the children of `node` are of level L - 1
        uint32_t node = own_first ? own : 0u;
        float4 p = make_float4(finf, finf, finf, 0.f);
        uint32_t pp = 0;
        auto fetch = [&]() {
            pp = (first + (uint32_t)(__ffs(mask) - 1)) * 32u + lane;
            p.x = finf;
            if (mask && pp < n) p = __ldg(&a.qpts[pp]);
        };
        fetch();
        while (true) {
            // down the box tree, 32 boxes at a time; the warp's own block first (its
            // points are the nearest: the bounds fall before the rest is looked at)
            while (walking && !mask) {
                const uint32_t cn = __shfl_sync(0xffffffffu, lv_count, L - 1), ch = node * 32u + lane;
                const float* b = a.boxes + __shfl_sync(0xffffffffu, lv_off, L - 1) + ch;
                bool hit = false;
                if (ch < cn && !(L == 2 && ch == own)) {
                    const float gx = max(max(__ldg(b) - fh0, fl0 - __ldg(b + 3ull * cn)), 0.0f);
                    const float gy = max(max(__ldg(b + cn) - fh1, fl1 - __ldg(b + 4ull * cn)), 0.0f);
                    const float gz = max(max(__ldg(b + 2ull * cn) - fh2, fl2 - __ldg(b + 5ull * cn)), 0.0f);
                    hit = fmaf(gx, gx, fmaf(gy, gy, gz * gz)) <= filt2;
                }
                const unsigned hits = __ballot_sync(0xffffffffu, hit);
                if (L == 1) {
                    first = node * 32u;
                    mask = hits;
                    // members are in the list already
                    if (mem_in && mem0 + want > first && mem0 < first + 32u)
                        for (uint32_t k = 0; k < want; ++k)
                            if (mem0 + k - first < 32u) mask &= ~(1u << (mem0 + k - first));
                    fetch();
                    if (own_first) {
                        own_first = false;
                        L = ltop + 1;
                        node = 0;
                        walking = ltop > 0;
                        continue;
                    }
                    L = 2;
                } else if (lane == L) {
                    lv_left = hits;
                    lv_node = node;
                }
                unsigned left = 0;
                while (L <= ltop + 1 && !(left = __shfl_sync(0xffffffffu, lv_left, L))) ++L;
                walking = L <= ltop + 1;
                if (!walking) break;
                node = __shfl_sync(0xffffffffu, lv_node, L) * 32u + (uint32_t)(__ffs(left) - 1);
                if (lane == L) lv_left &= lv_left - 1;
                --L;
            }
            // the next clump's points (the one after is loaded ahead)
            const bool more = mask != 0;
            if (more) {
                const float4 cp = p;
                const uint32_t cpp = pp;
                mask &= mask - 1;
                fetch();
                const float gx = max(max(fl0 - cp.x, cp.x - fh0), 0.0f);
                const float gy = max(max(fl1 - cp.y, cp.y - fh1), 0.0f);
                const float gz = max(max(fl2 - cp.z, cp.z - fh2), 0.0f);
                const float d2 = fmaf(gx, gx, fmaf(gy, gy, gz * gz));
                const bool take = members ? cpp < n : d2 <= filt2 && d2 > prev2;
                const unsigned bal = __ballot_sync(0xffffffffu, take);
                if (nc + nst + __popc(bal) > S::kCap) {
                    over = true;
                    break;
                }
                if (take) {
                    const uint32_t slot = nst + __popc(bal & ((1u << lane) - 1u));
                    stage[slot] = cp.x;
                    stage[64 + slot] = cp.y;
                    stage[128 + slot] = cp.z;
                    cpos[nc + slot] = cpp;
                }
                nst += __popc(bal);
            } else if (lane < 4) {  // the list ends: far points fill it to a multiple of four
                stage[nst + lane] = finf;
                stage[64 + nst + lane] = 0.0f;
                stage[128 + nst + lane] = 0.0f;
            }
            if (more && nst < 32) continue;
            // ---- scan the staged candidates; each lane appends those below its
            // bound, and all lanes merge when one's list is full (or at the end)
            __syncwarp();
            const uint32_t np = min(nst, 32u);
            bool merged = false;
            const uint32_t groups = (np + 3u) >> 2;
#pragma unroll 1
            for (uint32_t j = 0; j < groups + (more ? 0u : 1u); ++j) {
                uint32_t limit = buf + (uint32_t)(M - 4) * 128u;
                if (j < groups) {
                    const ulonglong2 x = ((const ulonglong2*)stage)[j], y = ((const ulonglong2*)stage)[16 + j],
                                     z = ((const ulonglong2*)stage)[32 + j];
                    uint64_t d[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const uint64_t dx = add2(u ? x.y : x.x, nqx), dy = add2(u ? y.y : y.x, nqy),
                                       dz = add2(u ? z.y : z.x, nqz);
                        d[u] = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, bias)));
                    }
                    const uint32_t ci = nc + j * 4u;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const uint32_t kb = (uint32_t)(d[u >> 1] >> (u & 1 ? 32 : 0));
                        append_below(at, kb, kthr, kb * (1u << IB) + (ci + u));
                    }
                } else {
                    limit = buf;  // the end: every list is merged
                }
                if (!__any_sync(0xffffffffu, at > limit)) continue;
                if (__any_sync(0xffffffffu, at > buf + 8 * 128)) {
                    uint32_t b[M];
#pragma unroll
                    for (int s = 0; s < M; ++s) b[s] = list_take(buf + s * 128);
                    oe_sort<M>(b);
                    merge_low<KS, M>(top.k, b);
                } else {
                    uint32_t b[8];
#pragma unroll
                    for (int s = 0; s < 8; ++s) b[s] = list_take(buf + s * 128);
                    oe_sort<8>(b);
                    merge_low<KS, 8>(top.k, b);
                }
                at = buf;
                const uint32_t w = top.k[KS - 1];
                if (w != 0xFFFFFFFFu) bnd = min(bnd, KEY_BASE + (w >> IB));
                kthr = min(kthr, bnd);
                merged = true;
            }
            nc += np;
            if (!more) break;
            nst -= np;
            float kx = 0.f, ky = 0.f, kz = 0.f;
            if ((uint32_t)lane < nst) {
                kx = stage[32 + lane];
                ky = stage[96 + lane];
                kz = stage[160 + lane];
            }
            __syncwarp();
            if ((uint32_t)lane < nst) {
                stage[lane] = kx;
                stage[64 + lane] = ky;
                stage[128 + lane] = kz;
            }
            __syncwarp();
            if (merged)
                filt2 = min(filt2, members ? finf : (float)(__reduce_max_sync(0xffffffffu, in ? kthr : KEY_BASE) - KEY_BASE));
        }
        // ---- what the list answered
        bool fin = false, next_round = members;
        if (members) {
            base = nc;
            members = false;
        } else if (over) {
            // too many candidates: the lanes start over with the bounds they have
            // now (a second time the retry launch takes them)
            if (in && again) retry = done = true;
            if (in && !again) {
                again = true;
                top.init(KS - (K + 1));
                if (bnd < KEY_BASE + S::kD2Max) ++bnd;
            }
            for (int k = 0; k < M; ++k) list_take(buf + k * 128);
            at = buf;
            next_round = true;
        } else {
            // a lane whose K-th is inside the margin is answered
            const uint32_t kth = top.k[KS - 2];
            if (in && kth != 0xFFFFFFFFu && (kth >> IB) <= (uint32_t)m * (uint32_t)m) {
                done = fin = true;
                in = false;
                kthr = 0;
            }
            next_round = !__any_sync(0xffffffffu, in);
            const bool whole = fl0 <= (float)m && fl1 <= (float)m && fl2 <= (float)m &&
                               fh0 + (float)m >= (float)(g.maxx - g.minx) && fh1 + (float)m >= (float)(g.maxy - g.miny) &&
                               fh2 + (float)m >= (float)(g.maxz - g.minz);
            if (!next_round && (whole || m >= S::kMaxMargin)) {
                // fewer than K points in reach: the retry launch decides
                if (in) retry = done = true;
                next_round = true;
            }
        }
        // the answered lanes read their K nearest back while the list stands
        __syncwarp();
        if (fin) {
            const uint32_t kk = top.k[KS - 2] >> IB, kk1 = top.k[KS - 1] >> IB;
            const int off = KS - (K + 1);
            if (kk == kk1) {
                atomicAdd(&a.counters[1], 1u);
                const QueryCell qc{qx, qy, qz, qx / g.cell, qy / g.cell, qz / g.cell};
                const int R = ring_for(g, qc, kk);
                defer_row(a, id, R < 256, KEY_BASE + kk, R);
                if (a.sums) a.sums[id].cnt = 0;
            } else if (a.ids_out) {
                uint32_t* row = a.ids_out + (uint64_t)id * a.K;
                int w = 0;
#pragma unroll
                for (int s = 0; s < KS - 1; ++s)
                    if (s >= off)
                        row[w++] = __float_as_uint(__ldg(&a.qpts[cpos[top.k[s] & (S::kCap - 1u)]]).w);
                for (int s = 1; s < K; ++s) {  // ascending ids
                    const uint32_t v = row[s];
                    int t = s - 1;
                    while (t >= 0 && row[t] > v) {
                        row[t + 1] = row[t];
                        --t;
                    }
                    row[t + 1] = v;
                }
            } else {
                RowSums out;
#pragma unroll
                for (int t = 0; t < 9; ++t) out.s[t] = 0;
#pragma unroll
                for (int s = 0; s < KS - 1; ++s) {
                    if (s >= off) {
                        const float4 c = __ldg(&a.qpts[cpos[top.k[s] & (S::kCap - 1u)]]);
                        const int ix = small_int(c.x - q.x), iy = small_int(c.y - q.y),
                                  iz = small_int(c.z - q.z);
                        out.s[0] += ix;
                        out.s[1] += iy;
                        out.s[2] += iz;
                        out.s[3] += ix * ix;
                        out.s[4] += iy * ix;
                        out.s[5] += iy * iy;
                        out.s[6] += iz * ix;
                        out.s[7] += iz * iy;
                        out.s[8] += iz * iz;
                    }
                }
                out.cnt = K;
                a.sums[id] = out;
            }
        }
        __syncwarp();
        // ---- the next list: a wider margin of this round, or a new round
        const int need = min(ceil_sqrt(bnd - KEY_BASE), S::kMaxMargin);  // holds all the lane can still want
        if (next_round) {
            if (!__any_sync(0xffffffffu, !done)) break;
            const int mn = __reduce_min_sync(0xffffffffu, done ? INT_MAX : need);
            const int lead = __ffs(__ballot_sync(0xffffffffu, !done && need == mn)) - 1;
            const int span = min(6 * mn, 2 * mcap);
            mem_in = !__shfl_sync(0xffffffffu, again, lead);
            const int lx = __shfl_sync(0xffffffffu, qx, lead), ly = __shfl_sync(0xffffffffu, qy, lead),
                      lz = __shfl_sync(0xffffffffu, qz, lead);
            in = !done && again != mem_in && abs(qx - lx) <= span && abs(qy - ly) <= span && abs(qz - lz) <= span;
            fl0 = (float)__reduce_min_sync(0xffffffffu, in ? qx : INT_MAX);
            fl1 = (float)__reduce_min_sync(0xffffffffu, in ? qy : INT_MAX);
            fl2 = (float)__reduce_min_sync(0xffffffffu, in ? qz : INT_MAX);
            fh0 = (float)__reduce_max_sync(0xffffffffu, in ? qx : INT_MIN);
            fh1 = (float)__reduce_max_sync(0xffffffffu, in ? qy : INT_MIN);
            fh2 = (float)__reduce_max_sync(0xffffffffu, in ? qz : INT_MIN);
            m = max(1, min(min(__reduce_max_sync(0xffffffffu, in ? need : 0), mn + (mn >> 2) + (mn >> 4)), mcap));
            prev2 = -1.0f;
            nc = base;
            kthr = in ? bnd : 0u;
        } else {
            prev2 = (float)m * (float)m;
            m = max(m + 1, min(__reduce_max_sync(0xffffffffu, in ? need : 0), 2 * m));
        }
        filt2 = min((float)m * (float)m, (float)(__reduce_max_sync(0xffffffffu, in ? kthr : KEY_BASE) - KEY_BASE));
    }
    if (retry || !done) {
        const uint32_t slot = atomicAdd(&a.counters[6], 1u);
        a.retry_rows[slot] = pos;
        if (a.sums) a.sums[id].cnt = 0;  // the finish pass leaves the row to the retry launch
    }
}

template <int KS>
__global__ void __launch_bounds__(WarpShape<KS>::kThreads, WarpShape<KS>::kMinBlocks)
    knn_group_kernel(const QueryArgs a, const float margin0) {
    using S = WarpShape<KS>;
    extern __shared__ __align__(16) unsigned char smem[];
    const uint64_t s0 = (uint64_t)blockIdx.x * S::kThreads + (threadIdx.x & ~31u);
    if (s0 < (a.rows ? a.nq : a.n)) group_warp<KS>(a, s0, margin0, smem + (threadIdx.x >> 5) * S::kWarpBytes);
}

// The clumps of many tiles in one launch: items of 128 rows, two blocks each.
template <int KS>
__global__ void __launch_bounds__(WarpShape<KS>::kThreads, WarpShape<KS>::kMinBlocks)
    knn_group_batch_kernel(const BatchJob* __restrict__ jobs, int njobs) {
    using S = WarpShape<KS>;
    extern __shared__ __align__(16) unsigned char smem[];
    const uint64_t item = blockIdx.x >> 1;
    const BatchJob& job = jobs[job_of(jobs, njobs, item)];
    const uint64_t s0 = (item - job.first) * 128u + (blockIdx.x & 1u) * S::kThreads + (threadIdx.x & ~31u);
    if (s0 < job.q.n) group_warp<KS>(select_args(job), s0, job.margin, smem + (threadIdx.x >> 5) * S::kWarpBytes);
}

template <int KS>
static int launch_group_batch_k(const BatchJob* jobs, int njobs, uint64_t items, cudaStream_t stream) {
    using S = WarpShape<KS>;
    if (!items) return NBG_OK;
    if (cudaFuncSetAttribute(knn_group_batch_kernel<KS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)S::kSmem))
        return NBG_ERR_CUDA;
    knn_group_batch_kernel<KS><<<(unsigned)(2 * items), S::kThreads, S::kSmem, stream>>>(jobs, njobs);
    NBG_LAUNCHED(1);
    return cudaGetLastError() == cudaSuccess ? NBG_OK : NBG_ERR_CUDA;
}

int launch_group_batch(int slots, const BatchJob* jobs, int njobs, uint64_t items, cudaStream_t stream) {
    switch (slots) {
        case 10: return launch_group_batch_k<10>(jobs, njobs, items, stream);
        case 12: return launch_group_batch_k<12>(jobs, njobs, items, stream);
        case 14: return launch_group_batch_k<14>(jobs, njobs, items, stream);
        case 18: return launch_group_batch_k<18>(jobs, njobs, items, stream);
        case 26: return launch_group_batch_k<26>(jobs, njobs, items, stream);
        case 34: return launch_group_batch_k<34>(jobs, njobs, items, stream);
        case 50: return launch_group_batch_k<50>(jobs, njobs, items, stream);
        case 66: return launch_group_batch_k<66>(jobs, njobs, items, stream);
    }
    return NBG_ERR_INVALID;
}

template <int KS>
static int launch_group_k(const QueryArgs& q, float margin0, cudaStream_t stream) {
    using S = WarpShape<KS>;
    const uint64_t rows = q.rows ? q.nq : q.n;
    const uint64_t blocks = (rows + S::kThreads - 1) / S::kThreads;
    if (!blocks) return NBG_OK;
    // the warps' lists pass the 48 KB default
    if (cudaFuncSetAttribute(knn_group_kernel<KS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)S::kSmem))
        return NBG_ERR_CUDA;
    knn_group_kernel<KS><<<(unsigned)blocks, S::kThreads, S::kSmem, stream>>>(q, margin0);
    NBG_LAUNCHED(1);
    return cudaGetLastError() == cudaSuccess ? NBG_OK : NBG_ERR_CUDA;
}

// The group select for K neighbours (slots: the top list's size, K + 1 or
// more).  Rows it hands back land in q.retry_rows, counted in q.counters[6].
int launch_group_select(const QueryArgs& q, int slots, float margin0, cudaStream_t stream) {
    switch (slots) {
        case 10: return launch_group_k<10>(q, margin0, stream);
        case 12: return launch_group_k<12>(q, margin0, stream);
        case 14: return launch_group_k<14>(q, margin0, stream);
        case 18: return launch_group_k<18>(q, margin0, stream);
        case 26: return launch_group_k<26>(q, margin0, stream);
        case 34: return launch_group_k<34>(q, margin0, stream);
        case 50: return launch_group_k<50>(q, margin0, stream);
        case 66: return launch_group_k<66>(q, margin0, stream);
    }
    return NBG_ERR_INVALID;
}

}  // namespace nbg
