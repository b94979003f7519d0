// nbg_grid.cu — column-compacted device grid over quantised int32 coordinates.
//
// Replaces the reference's KD3 build on the query side (PointView::build3dIndex,
// pdal/PointView.cpp:264-290) and the fork's Morton-key CUB sort
// (src/index/SpatialIndexKernels.cu:1772-1906).
//
// Airborne point clouds are 2.5-dimensional with walls, vegetation and wires:
// a dense 3D cell table over the tile's bounding box is mostly empty, and
// capping it forces cells far larger than the neighbourhoods.  Here every
// (cx, cy) column keeps a dense run of cells over its own occupied z-range
// only:
//   colinfo[col] = {base, zmin, zmax}      (one 16-byte load per column)
//   cell (cx, cy, cz) -> table entry base + cz - zmin, for zmin <= cz <= zmax
//   cstart[entry]     first point of the cell in the sorted point array
// so a query finds any cell with two dependent loads and scans, per column,
// one contiguous z-run of cells.  The build is a counting sort keyed by the
// table entry:
//   1. bbox      min/max of the raw coordinates
//   2. config    cell edge from the planar density, grid dims (device)
//   3. zrange    per-column min/max cell layer (atomics)
//   4. bases     exclusive scan of the column extents -> table size T
//   5. count     table entry per point, histogram
//   6. scan      exclusive scan of the histogram -> cstart
//   7. scatter   points into cell order as float4 {x, y, z, id} relative to
//                the tile minimum (exact: extents < 2^24)
// Within-cell order is not fixed; no output depends on it (neighbour sets are
// exact, covariance sums are exact integers).
#include <cub/cub.cuh>

#include "nbg_common.cuh"
#include "nbg_internal.h"

namespace nbg {

static constexpr int kSmallThreads = 1024;     // grid_small_kernel
static constexpr uint64_t kSmallPoints = 12288;
static constexpr uint32_t kSmallSlots = 65536;  // column slots, cells

__global__ void bbox_init_kernel(int32_t* bb) {
    if (threadIdx.x < 3) bb[threadIdx.x] = INT32_MAX;
    else if (threadIdx.x < 6) bb[threadIdx.x] = INT32_MIN;
}

__global__ void __launch_bounds__(256) bbox_kernel(const int32_t* __restrict__ x, const int32_t* __restrict__ y,
                            const int32_t* __restrict__ z, uint64_t n, int32_t* bb) {
    int32_t lo[3] = {INT32_MAX, INT32_MAX, INT32_MAX};
    int32_t hi[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        int32_t v[3] = {x[i], y[i], z[i]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = min(lo[d], v[d]);
            hi[d] = max(hi[d], v[d]);
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        lo[d] = __reduce_min_sync(0xffffffffu, lo[d]);
        hi[d] = __reduce_max_sync(0xffffffffu, hi[d]);
    }
    // one set of atomics a block: all blocks meet at the same six words (one set
    // a warp took 40 us for 1M points)
    __shared__ int32_t red[8][6];
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            red[threadIdx.x >> 5][d] = lo[d];
            red[threadIdx.x >> 5][3 + d] = hi[d];
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        int32_t r = red[0][threadIdx.x];
        for (unsigned w = 1; w < blockDim.x / 32; ++w)
            r = threadIdx.x < 3 ? min(r, red[w][threadIdx.x]) : max(r, red[w][threadIdx.x]);
        if (threadIdx.x < 3) atomicMin(&bb[threadIdx.x], r);
        else atomicMax(&bb[threadIdx.x], r);
    }
}

// Cell edge c = ceil(cell_factor * r_k), r_k the radius holding k1 points on
// a surface of the tile's planar density; grown only when the column count
// exceeds the directory.
__device__ GridParams grid_config(const int32_t* bb, uint64_t n, int k1, float cell_factor, uint64_t cols_cap,
                                  int32_t fixed_cell) {
    GridParams g;
    g.minx = bb[0];
    g.miny = bb[1];
    g.minz = bb[2];
    g.maxx = bb[3];
    g.maxy = bb[4];
    g.maxz = bb[5];
    const double ex = (double)g.maxx - g.minx + 1.0;
    const double ey = (double)g.maxy - g.miny + 1.0;
    const double ez = (double)g.maxz - g.minz + 1.0;
    double c;
    if (fixed_cell > 0) {
        c = fixed_cell;
    } else {
        const double rho2 = (double)n / (ex * ey);
        const double r = sqrt((double)k1 / (3.14159265358979 * rho2));
        c = ceil((double)cell_factor * r);
    }
    if (c < 1.0) c = 1.0;
    g.cap_hit = 0;
    for (;;) {
        const double gx = floor((ex - 1.0) / c) + 1.0;
        const double gy = floor((ey - 1.0) / c) + 1.0;
        if (gx * gy <= (double)cols_cap) {
            g.gx = (int32_t)gx;
            g.gy = (int32_t)gy;
            g.gz = (int32_t)(floor((ez - 1.0) / c) + 1.0);
            break;
        }
        c = ceil(c * 1.25 + 1.0);
        g.cap_hit = 1;
    }
    g.cell = (int32_t)c;
    g.r1 = (float)sqrt(ex * ey / (3.14159265358979 * (double)n));
    g.ncols = (uint32_t)g.gx * (uint32_t)g.gy;
    // tiled layout of the columns' runs where its padded slots fit the directory
    const uint64_t tx = ((uint64_t)g.gx + 63) / 64, ty = ((uint64_t)g.gy + 63) / 64;
    g.tgx = tx * ty * 4096 <= cols_cap ? (int32_t)tx : 0;
    g.nslots = g.tgx ? (uint32_t)(tx * ty * 4096) : g.ncols;
    // a full column's offsets pass the single-pass select's keys, and a thin
    // one's k1 nearest lie (at its own planar density) beyond 0.8 of the group
    // select's
    g.full = 1u << loc_offset_bits(g.cell);
    const float m = 0.8f * (float)group_max_margin(k1 + 1), cf = (float)g.cell;
    g.thin = (uint32_t)fminf(4.0e9f, (float)k1 * cf * cf / (3.14159265f * m * m));
    g.heavy = (uint32_t)fminf(4.0e9f, 256.0f * fmaxf(1.0f, (float)n / (float)g.ncols));
    g.in_full = g.in_thin = g.in_heavy = g.cells = 0;
    return g;
}

__global__ void grid_config_kernel(const int32_t* bb, uint64_t n, int k1, float cell_factor,
                                   uint64_t cols_cap, int32_t fixed_cell, GridParams* gp) {
    *gp = grid_config(bb, n, k1, cell_factor, cols_cap, fixed_cell);
}

__global__ void col_init_kernel(uint32_t ncols_cap, int4* __restrict__ colinfo, uint32_t* __restrict__ ext) {
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c <= ncols_cap;
         c += gridDim.x * blockDim.x) {
        if (c < ncols_cap) colinfo[c] = make_int4(0, INT32_MAX, -1, 0);
        ext[c] = 0;
    }
}

__global__ void col_zrange_kernel(const int32_t* __restrict__ x, const int32_t* __restrict__ y,
                                  const int32_t* __restrict__ z, uint64_t n,
                                  const GridParams* __restrict__ gpp, int4* __restrict__ colinfo) {
    const GridParams g = *gpp;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t cx = (uint32_t)(x[i] - g.minx) / (uint32_t)g.cell;
        const uint32_t cy = (uint32_t)(y[i] - g.miny) / (uint32_t)g.cell;
        const int cz = (int)((uint32_t)(z[i] - g.minz) / (uint32_t)g.cell);
        int4* ci = &colinfo[cy * (uint32_t)g.gx + cx];
        atomicMin(&ci->y, cz);
        atomicMax(&ci->z, cz);
    }
}

// Extents in layout order (column_slot), one past the last slot included;
// the padded slots of edge tiles are cleared before.
__global__ void col_extent_kernel(const GridParams* __restrict__ gpp,
                                  const int4* __restrict__ colinfo, uint32_t* __restrict__ ext) {
    const GridParams g = *gpp;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < g.ncols; c += gridDim.x * blockDim.x) {
        const int4 ci = colinfo[c];
        ext[column_slot(g, c % (uint32_t)g.gx, c / (uint32_t)g.gx)] =
            ci.z >= ci.y ? (uint32_t)(ci.z - ci.y + 1) : 0u;
    }
}

__global__ void col_base_kernel(GridParams* gpp, const uint32_t* __restrict__ ext,
                                int4* __restrict__ colinfo, uint32_t* __restrict__ table_size) {
    const GridParams g = *gpp;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c <= g.ncols;
         c += gridDim.x * blockDim.x) {
        if (c < g.ncols) colinfo[c].x = (int)ext[column_slot(g, c % (uint32_t)g.gx, c / (uint32_t)g.gx)];
        else *table_size = gpp->cells = ext[g.nslots];
    }
}

// Table entry of every point and the per-entry histogram.  An entry at or
// beyond `entries` (a table too small for this grid: only the build that does
// not read the table size first can see one) sets bit 2 of cap_hit and is
// dropped; the caller rebuilds such a grid.
__global__ void cell_count_kernel(const int32_t* __restrict__ x, const int32_t* __restrict__ y,
                                  const int32_t* __restrict__ z, uint64_t n, GridParams* gpp,
                                  const int4* __restrict__ colinfo, uint32_t* __restrict__ keys,
                                  uint32_t* __restrict__ counts, uint64_t entries) {
    const GridParams g = *gpp;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t cx = (uint32_t)(x[i] - g.minx) / (uint32_t)g.cell;
        const uint32_t cy = (uint32_t)(y[i] - g.miny) / (uint32_t)g.cell;
        const int cz = (int)((uint32_t)(z[i] - g.minz) / (uint32_t)g.cell);
        const int4 ci = colinfo[cy * (uint32_t)g.gx + cx];
        const uint32_t key = (uint32_t)ci.x + (uint32_t)(cz - ci.y);
        if ((uint64_t)key >= entries) {
            keys[i] = 0xFFFFFFFFu;
            atomicOr(&gpp->cap_hit, 2u);
            continue;
        }
        keys[i] = key;
        atomicAdd(&counts[key], 1u);
    }
}

__global__ void cell_scatter_kernel(const int32_t* __restrict__ x, const int32_t* __restrict__ y,
                                    const int32_t* __restrict__ z, uint64_t n, GridParams* gpp,
                                    const uint32_t* __restrict__ keys, uint32_t* __restrict__ cursor,
                                    float4* __restrict__ sorted, const int4* __restrict__ colinfo,
                                    const uint32_t* __restrict__ cstart, uint64_t entries) {
    const GridParams g = *gpp;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        if (keys[i] == 0xFFFFFFFFu) continue;
        const uint32_t pos = atomicAdd(&cursor[keys[i]], 1u);
        float4 r;
        r.x = (float)(x[i] - g.minx);
        r.y = (float)(y[i] - g.miny);
        r.z = (float)(z[i] - g.minz);
        r.w = __uint_as_float((uint32_t)i);
        sorted[pos] = r;
    }
    // the counts of GridParams over the columns, beside the scatter: the warps
    // that have any
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
    if ((first & ~31u) >= g.ncols) return;
    uint32_t v[3] = {0, 0, 0};
    for (uint32_t c = first; c < g.ncols; c += gridDim.x * blockDim.x) {
        const int4 ci = colinfo[c];
        // (a column beyond a table that is too small, which is built again)
        if (ci.z < ci.y || (uint64_t)(uint32_t)ci.x + (uint32_t)(ci.z - ci.y) + 1 > entries) continue;
        const uint32_t p = cstart[(uint32_t)ci.x + (uint32_t)(ci.z - ci.y) + 1u] - cstart[(uint32_t)ci.x];
        v[0] += p > g.full ? p : 0u;
        v[1] += p < g.thin ? p : 0u;
        v[2] += p > g.heavy ? p : 0u;
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const uint32_t r = __reduce_add_sync(0xffffffffu, v[q]);
        if ((threadIdx.x & 31) == 0 && r) atomicAdd(&gpp->in_full + q, r);
    }
}

// Exclusive prefix sums of v[0 .. count) in place (and into w), by one block of
// kSmallThreads; returns the total in every thread.  `part` is shared, one
// word a warp.
__device__ uint32_t block_scan(uint32_t* v, uint32_t* w, uint32_t count, uint32_t* part) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t b = 0; b < count; b += kSmallThreads) {
        const uint32_t c = b + threadIdx.x;
        const uint32_t own = c < count ? v[c] : 0u;
        uint32_t x = own;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) part[warp] = x;
        __syncthreads();
        uint32_t p = lane < kSmallThreads / 32 ? part[lane] : 0u;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, p, d);
            if (lane >= d) p += y;
        }
        const uint32_t before = __shfl_sync(0xffffffffu, p, (warp + 31) & 31);
        const uint32_t r = carry + (warp ? before : 0u) + x - own;
        if (c < count) {
            v[c] = r;
            if (w) w[c] = r;
        }
        carry += __shfl_sync(0xffffffffu, p, 31);
        __syncthreads();
    }
    return carry;
}

// The whole build of a small tile in one block: the phases are the kernels'
// above, a barrier in place of a launch.  A grid of more slots or entries than
// a block should walk, or than the table holds, sets bit 2 of cap_hit and is
// left to the other builds.
//
// Bound by the phases' latency, not by work: thirteen launches and a read of the
// table size between them are what it saves (figures at grid_small).
__global__ void __launch_bounds__(kSmallThreads) grid_small_kernel(
    const int32_t* x, const int32_t* y, const int32_t* z, const uint32_t n, int k1, float cell_factor,
    uint64_t cols_cap, GridParams* gp, int32_t* bbox, int4* colinfo, uint32_t* ext, uint32_t* table_size,
    uint32_t entries, uint32_t* keys, uint32_t* cstart, uint32_t* cursor, float4* sorted) {
    __shared__ int32_t red[kSmallThreads / 32][6], bb[6];
    __shared__ uint32_t part[kSmallThreads / 32];
    __shared__ GridParams sg;
    const uint32_t tid = threadIdx.x;
    int32_t r[6] = {INT32_MAX, INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN, INT32_MIN};
    for (uint32_t i = tid; i < n; i += kSmallThreads) {
        const int32_t v[3] = {x[i], y[i], z[i]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            r[d] = min(r[d], v[d]);
            r[3 + d] = max(r[3 + d], v[d]);
        }
    }
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        r[d] = d < 3 ? __reduce_min_sync(0xffffffffu, r[d]) : __reduce_max_sync(0xffffffffu, r[d]);
        if ((tid & 31) == 0) red[tid >> 5][d] = r[d];
    }
    __syncthreads();
    if (tid < 32) {
#pragma unroll
        for (int d = 0; d < 6; ++d) {
            const int32_t v = red[tid][d];
            const int32_t m = d < 3 ? __reduce_min_sync(0xffffffffu, v) : __reduce_max_sync(0xffffffffu, v);
            if (tid == 0) bb[d] = bbox[d] = m;
        }
        if (tid == 0) {
            sg = grid_config(bb, n, k1, cell_factor, cols_cap, 0);
            if (sg.nslots > kSmallSlots) sg.cap_hit |= 2u;
            *gp = sg;
        }
    }
    __syncthreads();
    const GridParams g = sg;
    if (g.cap_hit & 2u) return;
    for (uint32_t c = tid; c <= g.nslots; c += kSmallThreads) {
        if (c < g.ncols) colinfo[c] = make_int4(0, INT32_MAX, -1, 0);
        ext[c] = 0;
    }
    __syncthreads();
    for (uint32_t i = tid; i < n; i += kSmallThreads) {
        const uint32_t cx = (uint32_t)(x[i] - g.minx) / (uint32_t)g.cell;
        const uint32_t cy = (uint32_t)(y[i] - g.miny) / (uint32_t)g.cell;
        const int cz = (int)((uint32_t)(z[i] - g.minz) / (uint32_t)g.cell);
        int4* ci = &colinfo[cy * (uint32_t)g.gx + cx];
        atomicMin(&ci->y, cz);
        atomicMax(&ci->z, cz);
    }
    __syncthreads();
    for (uint32_t c = tid; c < g.ncols; c += kSmallThreads) {
        const int zlo = __ldcg(&colinfo[c].y), zhi = __ldcg(&colinfo[c].z);
        ext[column_slot(g, c % (uint32_t)g.gx, c / (uint32_t)g.gx)] = zhi >= zlo ? (uint32_t)(zhi - zlo + 1) : 0u;
    }
    __syncthreads();
    const uint32_t total = block_scan(ext, nullptr, g.nslots + 1, part);
    if (tid == 0) *table_size = gp->cells = total;
    if (total > entries || total > kSmallSlots) {  // (as *gp says to the host)
        if (tid == 0) gp->cap_hit = g.cap_hit | 2u;
        return;
    }
    for (uint32_t c = tid; c < g.ncols; c += kSmallThreads)
        colinfo[c].x = (int)ext[column_slot(g, c % (uint32_t)g.gx, c / (uint32_t)g.gx)];
    for (uint32_t c = tid; c <= total; c += kSmallThreads) cstart[c] = 0;
    __syncthreads();
    for (uint32_t i = tid; i < n; i += kSmallThreads) {
        const uint32_t cx = (uint32_t)(x[i] - g.minx) / (uint32_t)g.cell;
        const uint32_t cy = (uint32_t)(y[i] - g.miny) / (uint32_t)g.cell;
        const int cz = (int)((uint32_t)(z[i] - g.minz) / (uint32_t)g.cell);
        const int4 ci = __ldcg(&colinfo[cy * (uint32_t)g.gx + cx]);
        uint32_t key = (uint32_t)ci.x + (uint32_t)(cz - ci.y);
        if (key < total) {
            atomicAdd(&cstart[key], 1u);
        } else {  // (extents whose sum passes 32 bits)
            key = 0xFFFFFFFFu;
            atomicOr(&gp->cap_hit, 2u);
        }
        keys[i] = key;
    }
    __syncthreads();
    block_scan(cstart, cursor, total + 1, part);
    // (of a small tile's counts select_kernel reads the full columns', for lists of
    // up to 14 slots)
    if (k1 < 14) {
        uint32_t full = 0;
        for (uint32_t c = tid; c < g.ncols; c += kSmallThreads) {
            const int4 ci = __ldcg(&colinfo[c]);
            // (beyond the table: extents whose sum passes 32 bits)
            if (ci.z < ci.y || (uint64_t)(uint32_t)ci.x + (uint32_t)(ci.z - ci.y) + 1 > total) continue;
            const uint32_t p = cstart[(uint32_t)ci.x + (uint32_t)(ci.z - ci.y) + 1u] - cstart[(uint32_t)ci.x];
            full += p > g.full ? p : 0u;
        }
        if (full) atomicAdd(&gp->in_full, full);
    }
    for (uint32_t i = tid; i < n; i += kSmallThreads) {
        if (keys[i] == 0xFFFFFFFFu) continue;
        const uint32_t pos = atomicAdd(&cursor[keys[i]], 1u);
        float4 p;
        p.x = (float)(x[i] - g.minx);
        p.y = (float)(y[i] - g.miny);
        p.z = (float)(z[i] - g.minz);
        p.w = __uint_as_float(i);
        sorted[pos] = p;
    }
}

// Clump order of the group select: every block of kClumpRows consecutive rows
// (a patch of neighbouring columns) is halved at the median of its longest
// side until 32 points are left, so a clump's box is small and square: ground,
// wall and canopy points of a column come apart.  Against 32-point runs of a
// Hilbert curve through the same blocks, a clump's search examines 166 instead
// of 268 candidates (terrain, K = 17; 251 instead of 333 on the mixture).
// Writes the points in that order, the clumps' boxes and the blocks' boxes.
static constexpr int kClumpRows = 1024;

// Ascending bitonic sort of each segment of SEG threads' keys (one each):
// shuffles inside a warp, shared memory across.
template <int SEG>
__device__ __forceinline__ uint32_t sort_segment(uint32_t key, uint32_t* sh) {
    const int tid = threadIdx.x;
#pragma unroll
    for (int k = 2; k <= SEG; k <<= 1) {
        // (descending runs are sorted as ascending runs of the complement)
        const uint32_t flip = k < SEG && (tid & k) ? 0xFFFFFFFFu : 0u;
        key ^= flip;
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            uint32_t other;
            if (j >= 32) {
                __syncthreads();
                sh[tid] = key;
                __syncthreads();
                other = sh[tid ^ j];
            } else {
                other = __shfl_xor_sync(0xffffffffu, key, j);
            }
            key = (tid & j) ? max(key, other) : min(key, other);
        }
        key ^= flip;
    }
    return key;
}

__global__ void __launch_bounds__(kClumpRows) clump_kernel(const float4* __restrict__ sorted, uint64_t n,
                                                           float4* __restrict__ pts, float* __restrict__ boxes) {
    __shared__ uint32_t sh[kClumpRows];
    __shared__ int sc[3][kClumpRows];
    __shared__ uint32_t sid[kClumpRows];
    __shared__ int wbox[32][6];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint64_t base = (uint64_t)blockIdx.x * kClumpRows;
    const int rows = (int)min((uint64_t)kClumpRows, n - base);
    if (tid < rows) {
        const float4 q = __ldg(&sorted[base + tid]);
        sc[0][tid] = __float2int_rz(q.x);
        sc[1][tid] = __float2int_rz(q.y);
        sc[2][tid] = __float2int_rz(q.z);
        sid[tid] = __float_as_uint(q.w);
    }
    __syncthreads();
    uint32_t idx = (uint32_t)tid;  // the row in this thread's place
    // box of the warp's rows
    auto warp_box = [&](int (&v)[6]) {
        const bool in = idx < (uint32_t)rows;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            v[d] = __reduce_min_sync(0xffffffffu, in ? sc[d][idx] : INT32_MAX);
            v[3 + d] = __reduce_max_sync(0xffffffffu, in ? sc[d][idx] : INT32_MIN);
        }
    };
#pragma unroll 1
    for (int seg = kClumpRows; seg > 32; seg >>= 1) {
        int v[6];
        warp_box(v);
        if (lane == 0)
#pragma unroll
            for (int d = 0; d < 6; ++d) wbox[wid][d] = v[d];
        __syncthreads();
        const int sw = seg >> 5, w0 = wid & ~(sw - 1);  // the segment's warps
        int best = -1, axis = 0, lo = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int l = __reduce_min_sync(0xffffffffu, wbox[w0 + (lane & (sw - 1))][d]);
            const int h = __reduce_max_sync(0xffffffffu, wbox[w0 + (lane & (sw - 1))][3 + d]);
            const int e = h >= l ? h - l : 0;
            if (e > best) {
                best = e;
                axis = d;
                lo = l;
            }
        }
        const int s = max(0, 32 - __clz(max(best, 1)) - 21);  // (extent >> s) < 2^21
        uint32_t key = 0x80000000u | idx;  // threads past the rows sort last
        if (idx < (uint32_t)rows) key = (uint32_t)(sc[axis][idx] - lo) >> s << 10 | idx;
        switch (seg) {
            case 1024: key = sort_segment<1024>(key, sh); break;
            case 512: key = sort_segment<512>(key, sh); break;
            case 256: key = sort_segment<256>(key, sh); break;
            case 128: key = sort_segment<128>(key, sh); break;
            default: key = sort_segment<64>(key, sh); break;
        }
        idx = key & (kClumpRows - 1u);
        __syncthreads();
    }
    // (rows past the end keep the last places of the last block)
    if (base + tid < n)
        pts[base + tid] = make_float4((float)sc[0][idx], (float)sc[1][idx], (float)sc[2][idx],
                                      __uint_as_float(sid[idx]));
    const ClumpTree tr(n);
    int v[6];
    warp_box(v);
    const uint64_t clump = (base >> 5) + wid;
    if (lane < 6 && clump < tr.count[0]) {
        int r = v[0];
#pragma unroll
        for (int d = 1; d < 6; ++d)
            if (lane == d) r = v[d];
        boxes[tr.off[0] + (uint64_t)lane * tr.count[0] + clump] = (float)r;
    }
    if (lane == 0)
#pragma unroll
        for (int d = 0; d < 6; ++d) wbox[wid][d] = v[d];
    __syncthreads();
    if (wid < 6) {
        const int x = wbox[lane][wid];
        const int r = wid < 3 ? __reduce_min_sync(0xffffffffu, x) : __reduce_max_sync(0xffffffffu, x);
        if (lane == 0) boxes[tr.off[1] + (uint64_t)wid * tr.count[1] + blockIdx.x] = (float)r;
    }
}

// Boxes of a level's nodes from their 32 children's, one warp per node.
__global__ void clump_parents_kernel(float* __restrict__ boxes, uint64_t n, int level) {
    const ClumpTree tr(n);
    uint32_t nc = 0, np = 0;
    uint64_t oc = 0, op = 0;
#pragma unroll
    for (int l = 1; l < ClumpTree::kLevels; ++l)
        if (l == level) {
            nc = tr.count[l - 1];
            oc = tr.off[l - 1];
            np = tr.count[l];
            op = tr.off[l];
        }
    const uint32_t node = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (node >= np) return;
    const uint32_t ch = node * 32u + lane;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        const int none = d < 3 ? INT32_MAX : INT32_MIN;
        const int x = ch < nc ? (int)boxes[oc + (uint64_t)d * nc + ch] : none;
        const int r = d < 3 ? __reduce_min_sync(0xffffffffu, x) : __reduce_max_sync(0xffffffffu, x);
        if (lane == 0) boxes[op + (uint64_t)d * np + node] = (float)r;
    }
}

int ensure_clumps(Context* ctx, Tile* t, cudaStream_t stream) {
    (void)ctx;
    if (t->pts || !t->n) return NBG_OK;
    if (!t->clumps || !t->grid_valid) return NBG_ERR_INVALID;
    NBG_RANGE("nbg clump order");
    float4* pts = (float4*)t->cursor;
    float* boxes = (float*)t->keys;
    const ClumpTree tr(t->n);
    clump_kernel<<<(unsigned)((t->n + kClumpRows - 1) / kClumpRows), kClumpRows, 0, stream>>>(t->sorted, t->n, pts,
                                                                                              boxes);
    NBG_LAUNCHED(1);
    for (int l = 2; l <= tr.top; ++l) {
        clump_parents_kernel<<<(tr.count[l] + 3) / 4, 128, 0, stream>>>(boxes, t->n, l);
        NBG_LAUNCHED(1);
    }
    if (cudaGetLastError() != cudaSuccess) return NBG_ERR_CUDA;
    t->pts = pts;
    t->boxes = boxes;
    return NBG_OK;
}

static int grid_blocks(uint64_t n, int threads, int sms, int per_sm = 8) {
    uint64_t b = (n + threads - 1) / threads;
    uint64_t cap = (uint64_t)sms * per_sm;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

// Bytes of CUB scan storage for `items` entries.
size_t grid_temp_bytes(uint64_t items) {
    size_t b = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, b, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                  (int)items);
    return b + 256;
}

// Builds the grid of `t` on `stream`.  One host synchronisation reads the
// table size T (sum of the column extents); the table grows when needed.
int build_grid(Context* ctx, Tile* t, int k1, cudaStream_t stream) {
    t->pts = nullptr;  // (their arrays are the build's)
    const uint64_t n = t->n;
    const int sms = ctx->sm_count;
    const int nb = grid_blocks(n, 256, sms);
    // the scatter waits on a returned atomic per point: more resident threads
    // keep more of those round trips in flight
    const int sb = grid_blocks(n, 256, sms, 32);
    bbox_init_kernel<<<1, 32, 0, stream>>>(t->bbox);
    bbox_kernel<<<grid_blocks(n, 256, sms, 2), 256, 0, stream>>>(t->x, t->y, t->z, n, t->bbox);
    grid_config_kernel<<<1, 1, 0, stream>>>(t->bbox, n, k1, t->cell_factor, t->cols_cap,
                                            t->fixed_cell, t->gp);
    const int cb = grid_blocks(t->cols_cap + 1, 256, sms);
    col_init_kernel<<<cb, 256, 0, stream>>>((uint32_t)t->cols_cap, t->colinfo, t->ext);
    col_zrange_kernel<<<nb, 256, 0, stream>>>(t->x, t->y, t->z, n, t->gp, t->colinfo);
    col_extent_kernel<<<cb, 256, 0, stream>>>(t->gp, t->colinfo, t->ext);
    size_t tmp = t->grid_tmp_bytes;
    if (cub::DeviceScan::ExclusiveSum(t->grid_tmp, tmp, t->ext, t->ext, (int)(t->cols_cap + 1),
                                      stream))
        return NBG_ERR_CUDA;
    col_base_kernel<<<cb, 256, 0, stream>>>(t->gp, t->ext, t->colinfo, t->table_dev);
    uint32_t T = 0;
    if (cudaMemcpyAsync(&T, t->table_dev, 4, cudaMemcpyDeviceToHost, stream) ||
        cudaStreamSynchronize(stream))
        return NBG_ERR_CUDA;
    if ((uint64_t)T + 1 > t->table_cap) {
        int rc = grid_grow_table(ctx, t, (uint64_t)T + 1);
        if (rc) return rc;
    }
    t->table_size = T;
    if (cudaMemsetAsync(t->cstart, 0, ((size_t)T + 1) * sizeof(uint32_t), stream))
        return NBG_ERR_CUDA;
    cell_count_kernel<<<nb, 256, 0, stream>>>(t->x, t->y, t->z, n, t->gp, t->colinfo, t->keys,
                                              t->cstart, (uint64_t)T + 1);
    tmp = t->grid_tmp_bytes;
    if (cub::DeviceScan::ExclusiveSum(t->grid_tmp, tmp, t->cstart, t->cstart, (int)(T + 1),
                                      stream))
        return NBG_ERR_CUDA;
    if (cudaMemcpyAsync(t->cursor, t->cstart, ((size_t)T + 1) * sizeof(uint32_t),
                        cudaMemcpyDeviceToDevice, stream))
        return NBG_ERR_CUDA;
    cell_scatter_kernel<<<sb, 256, 0, stream>>>(t->x, t->y, t->z, n, t->gp, t->keys, t->cursor,
                                                t->sorted, t->colinfo, t->cstart, T);
    // bbox (2), config, col init, zrange, extent, scan (2), bases, count, scan (2), scatter
    NBG_LAUNCHED(13);
    return cudaGetLastError() == cudaSuccess ? NBG_OK : NBG_ERR_CUDA;
}

// One block's build against thirteen launches and two reads by the host: 30 us
// against 87 up to 2000 points, 42 / 86 at 4000, 56 / 84 at 8000, 65 / 86 at
// 12000, 77 / 89 at 16000 (a call's time as before there), 140 / 88 at 32000.  A
// cell edge fixed by a radius may give any number of columns: not here.
bool grid_small(const Tile* t) { return t->n <= kSmallPoints && !t->fixed_cell; }

// A small tile's build in one launch (grid_small), without synchronisation; bit 2
// of cap_hit as build_grid_async.
int build_grid_small(Context* ctx, Tile* t, int k1, cudaStream_t stream) {
    (void)ctx;
    t->pts = nullptr;  // (their arrays are the build's)
    const uint64_t entries = t->table_cap - 1;  // cstart needs entries + 1 slots
    grid_small_kernel<<<1, kSmallThreads, 0, stream>>>(
        t->x, t->y, t->z, (uint32_t)t->n, k1, t->cell_factor, t->cols_cap, t->gp, t->bbox, t->colinfo, t->ext,
        t->table_dev, (uint32_t)std::min<uint64_t>(entries, UINT32_MAX), t->keys, t->cstart, t->cursor, t->sorted);
    NBG_LAUNCHED(1);
    t->table_size = entries;
    return cudaGetLastError() == cudaSuccess ? NBG_OK : NBG_ERR_CUDA;
}

// The same build without reading the table size on the host (no
// synchronisation, so it can be captured in a CUDA graph): the histogram and
// its scan cover the whole table capacity.  A grid whose table would not fit
// sets bit 2 of cap_hit; the caller rebuilds it with build_grid.
int build_grid_async(Context* ctx, Tile* t, int k1, cudaStream_t stream) {
    t->pts = nullptr;  // (their arrays are the build's)
    const uint64_t n = t->n;
    const int sms = ctx->sm_count;
    const int nb = grid_blocks(n, 256, sms);
    // the scatter waits on a returned atomic per point: more resident threads
    // keep more of those round trips in flight
    const int sb = grid_blocks(n, 256, sms, 32);
    const uint64_t entries = t->table_cap - 1;  // cstart needs entries + 1 slots
    bbox_init_kernel<<<1, 32, 0, stream>>>(t->bbox);
    bbox_kernel<<<grid_blocks(n, 256, sms, 2), 256, 0, stream>>>(t->x, t->y, t->z, n, t->bbox);
    grid_config_kernel<<<1, 1, 0, stream>>>(t->bbox, n, k1, t->cell_factor, t->cols_cap,
                                            t->fixed_cell, t->gp);
    const int cb = grid_blocks(t->cols_cap + 1, 256, sms);
    col_init_kernel<<<cb, 256, 0, stream>>>((uint32_t)t->cols_cap, t->colinfo, t->ext);
    col_zrange_kernel<<<nb, 256, 0, stream>>>(t->x, t->y, t->z, n, t->gp, t->colinfo);
    col_extent_kernel<<<cb, 256, 0, stream>>>(t->gp, t->colinfo, t->ext);
    size_t tmp = t->grid_tmp_bytes;
    if (cub::DeviceScan::ExclusiveSum(t->grid_tmp, tmp, t->ext, t->ext, (int)(t->cols_cap + 1),
                                      stream))
        return NBG_ERR_CUDA;
    col_base_kernel<<<cb, 256, 0, stream>>>(t->gp, t->ext, t->colinfo, t->table_dev);
    if (cudaMemsetAsync(t->cstart, 0, (size_t)(entries + 1) * sizeof(uint32_t), stream))
        return NBG_ERR_CUDA;
    cell_count_kernel<<<nb, 256, 0, stream>>>(t->x, t->y, t->z, n, t->gp, t->colinfo, t->keys,
                                              t->cstart, entries);
    tmp = t->grid_tmp_bytes;
    if (cub::DeviceScan::ExclusiveSum(t->grid_tmp, tmp, t->cstart, t->cstart, (int)(entries + 1),
                                      stream))
        return NBG_ERR_CUDA;
    if (cudaMemcpyAsync(t->cursor, t->cstart, (size_t)(entries + 1) * sizeof(uint32_t),
                        cudaMemcpyDeviceToDevice, stream))
        return NBG_ERR_CUDA;
    cell_scatter_kernel<<<sb, 256, 0, stream>>>(t->x, t->y, t->z, n, t->gp, t->keys, t->cursor,
                                                t->sorted, t->colinfo, t->cstart, entries);
    NBG_LAUNCHED(13);
    t->table_size = entries;
    return cudaGetLastError() == cudaSuccess ? NBG_OK : NBG_ERR_CUDA;
}

}  // namespace nbg
