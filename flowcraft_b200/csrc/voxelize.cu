// Mesh voxelizer on the device: FlowCraft's Voxelizer::Voxelize
// (FlowCraft/Voxelizer.cpp:136-485) producing the solver's boundary input, the
// VoxelGrid solid mask and signed distance (FlowCraft/VoxelGrid.h:13-61),
// bit-identical to the reference's CPU build.
//
// Pipeline (one stream, blocking call):
//   1. grid: bounds of the vertices by a two-level reduction whose ties keep
//      the lowest vertex index, which is std::min/std::max's first-wins rule
//      (Mesh.h:56-59) even for signed zeros; then the padded domain, cell size
//      and dims exactly as Voxelizer.cpp:146-166;
//   2. triangles: one thread per triangle computes its unit normal and its
//      clamped cell box (Voxelizer.cpp:206-235) and counts the 8x8x8 raster
//      tiles the box touches; an exclusive scan places every (tile, triangle)
//      pair, written in triangle order; a stable radix sort on the tile id
//      groups them by tile keeping triangle order inside each tile, and a
//      run-length encode gives each occupied tile its triangle list;
//   3. raster: a block per occupied tile where its list is short, else one per
//      box of 4x4x2 cells, which tests the tile's triangles against the box and
//      computes the distances of those that overlap it, many at a time. Each
//      cell's running signed distance, best normal projection and solid bit
//      follow the
//      reference's update rule (Voxelizer.cpp:236-293) over the triangles
//      whose box holds the cell, in index order, so every cell sees the same
//      triangles in the same order as the CPU loop and rounds the same IEEE
//      operations (the library is built without FMA contraction, with IEEE
//      division and square root);
//   4. flood fill: fluid cells 6-connected to cell (0,0,0) are the exterior
//      (Voxelizer.cpp:295-454). A tile without triangles holds no solid cell
//      and is one node; in an occupied tile every x-run of fluid cells in an
//      8-cell row is a node. Nodes are joined across rows, layers and tile
//      faces with a lock-free union-find that links larger roots under
//      smaller ones (Playne & Hawick, "A new algorithm for parallel
//      connected-component labelling on GPUs", IEEE TPDS 2018). Occupied
//      tiles are the few along the surface, so the forest is small (the
//      aircraft at 640 cells: 0.3M nodes for 31M cells) and stays in L2;
//   5. finalize: one pass writes every cell: unreached fluid becomes solid and
//      the signed distance is reconciled with the classification
//      (Voxelizer.cpp:456-481). Tiles without triangles are written without
//      being read.
// Measured on a B200, the 57,516-triangle aircraft on 640x308x158 cells, mesh
// and grid on the device: 3.30 -> 0.57 ms (flood fill and finalize 2.0 -> 0.13,
// raster 0.95 -> 0.29).
//
// Every loop over the union-find forest is bounded: labels strictly decrease
// along a parent chain, and the loops also stop after a fixed iteration count,
// setting an error bit the host turns into FC_LBM_ERR_CUDA.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_run_length_encode.cuh>
#include <cub/device/device_scan.cuh>

#include "fc_lbm.h"
#include "host_wait.h"

namespace {

constexpr int kTile = 8;                    // raster tile edge (cells)
constexpr int kTileCells = kTile * kTile * kTile;
constexpr int kTileRows = kTile * kTile;    // 8-cell x rows of a tile
constexpr int kTriWords = 20;               // a[3] b[3] c[3] n[3] lo[3] hi[3] pad[2]
constexpr int kBoundsBlocks = 148;
constexpr int kBoundsThreads = 256;
constexpr unsigned kMaxFindHops = 1u << 26;
constexpr int kMaxMergeRetries = 1 << 20;
constexpr int kWaitTimeoutMs = 600000;
constexpr int kErrBadIndex = 1;
constexpr int kErrUnionBound = 2;

struct alignas(16) Tri {  // read as 16-byte vectors
    float a[3], b[3], c[3], n[3];
    int lo[3], hi[3];  // clamped cell box, grid axes (x spans world y, y spans world x)
    int pad[2];
};
static_assert(sizeof(Tri) == kTriWords * 4, "triangle record layout");

struct V3 {
    float x, y, z;
};

__device__ __forceinline__ V3 vsub(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 vadd(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 vmul(V3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ float vdot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 vcross(V3 a, V3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float vlen(V3 v) { return sqrtf(v.x * v.x + v.y * v.y + v.z * v.z); }
__device__ __forceinline__ float min3(float a, float b, float c) {
    float m = a;
    if (b < m) m = b;
    if (c < m) m = c;
    return m;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float m = a;
    if (m < b) m = b;
    if (m < c) m = c;
    return m;
}

// float -> int as the x86-64 host converts it (cvttss2si): truncation in
// range, INT_MIN for NaN and out-of-range values. The device's own conversion
// saturates instead, which would change the clamped box of a triangle lying
// more than 2^31 cells outside the grid.
__device__ __forceinline__ int to_int_host(float f) {
    return (f >= -2147483648.0f && f < 2147483648.0f) ? (int)f : INT_MIN;
}

// Closest point on triangle (a, b, c) to p: Ericson's Voronoi-region method,
// the operation order of Voxelizer.cpp:89-129.
__device__ __forceinline__ V3 closest_on_triangle(V3 p, V3 a, V3 b, V3 c) {
    const V3 ab = vsub(b, a), ac = vsub(c, a), ap = vsub(p, a);
    const float d1 = vdot(ab, ap), d2 = vdot(ac, ap);
    if (d1 <= 0.0f && d2 <= 0.0f) return a;
    const V3 bp = vsub(p, b);
    const float d3 = vdot(ab, bp), d4 = vdot(ac, bp);
    if (d3 >= 0.0f && d4 <= d3) return b;
    const float vc = d1 * d4 - d3 * d2;
    if (vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f) {
        const float v = d1 / (d1 - d3);
        return vadd(a, vmul(ab, v));
    }
    const V3 cp = vsub(p, c);
    const float d5 = vdot(ab, cp), d6 = vdot(ac, cp);
    if (d6 >= 0.0f && d5 <= d6) return c;
    const float vb = d5 * d2 - d1 * d6;
    if (vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f) {
        const float w = d2 / (d2 - d6);
        return vadd(a, vmul(ac, w));
    }
    const float va = d3 * d6 - d5 * d4;
    if (va <= 0.0f && (d4 - d3) >= 0.0f && (d5 - d6) >= 0.0f) {
        const float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        return vadd(b, vmul(vsub(c, b), w));
    }
    const float denom = 1.0f / (va + vb + vc);
    const float v = vb * denom, w = vc * denom;
    return vadd(vadd(a, vmul(ab, v)), vmul(ac, w));
}

// ---- 1. grid from the mesh bounds ----

// (value, vertex index) with "smaller value, then smaller index" order: the
// minimum over a set is the first vertex holding the smallest value, which is
// what a sequential `min = std::min(min, v)` keeps (it never replaces an equal
// value, so -0.0 and +0.0 keep whichever came first). For the maximum the
// value order flips and the index order stays.
struct Pick {
    float v;
    unsigned i;
};
__device__ __forceinline__ Pick pick_min(Pick a, Pick b) {
    return (b.v < a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}
__device__ __forceinline__ Pick pick_max(Pick a, Pick b) {
    return (a.v < b.v || (b.v == a.v && b.i < a.i)) ? b : a;
}

__device__ __forceinline__ Pick shfl_pick(Pick p, int off) {
    p.v = __shfl_down_sync(0xffffffffu, p.v, off);
    p.i = __shfl_down_sync(0xffffffffu, p.i, off);
    return p;
}

// The reduction's identity is the reference's starting value (FLT_MAX for the
// minimum, lowest() for the maximum) with an index behind every vertex, so a
// vertex equal to it (or NaN, which never compares less) leaves the same
// bits the sequential loop leaves.
__global__ void __launch_bounds__(kBoundsThreads) k_bounds_partial(const float* __restrict__ pos, unsigned nv,
                                                                   Pick* __restrict__ partial) {
    Pick mn[3], mx[3];
    for (int k = 0; k < 3; ++k) {
        mn[k] = {3.402823466e38f, 0xffffffffu};
        mx[k] = {-3.402823466e38f, 0xffffffffu};
    }
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
        for (int k = 0; k < 3; ++k) {
            const Pick p{pos[3 * (size_t)i + k], i};
            mn[k] = pick_min(mn[k], p);
            mx[k] = pick_max(mx[k], p);
        }
    }
    __shared__ Pick s[6][kBoundsThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < 3; ++k) {
        for (int off = 16; off > 0; off >>= 1) {
            mn[k] = pick_min(mn[k], shfl_pick(mn[k], off));
            mx[k] = pick_max(mx[k], shfl_pick(mx[k], off));
        }
        if (lane == 0) {
            s[k][warp] = mn[k];
            s[3 + k][warp] = mx[k];
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int k = threadIdx.x;
        Pick r = s[k][0];
        for (int w = 1; w < kBoundsThreads / 32; ++w) r = k < 3 ? pick_min(r, s[k][w]) : pick_max(r, s[k][w]);
        partial[blockIdx.x * 6 + k] = r;
    }
}

struct GridOut {
    int dims[3];
    float cell;
    float origin[3];
};

// Voxelizer.cpp:146-166: a warp per bound, then one thread.
constexpr int kGridThreads = 6 * 32;
__global__ void __launch_bounds__(kGridThreads) k_grid_final(const Pick* __restrict__ partial, int blocks, int target_res, float padx, float pady,
                             float padz, GridOut* out) {
    __shared__ Pick r[6];
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Pick p = partial[k];
    for (int b = lane; b < blocks; b += 32) p = k < 3 ? pick_min(p, partial[b * 6 + k]) : pick_max(p, partial[b * 6 + k]);
    for (int off = 16; off > 0; off >>= 1) p = k < 3 ? pick_min(p, shfl_pick(p, off)) : pick_max(p, shfl_pick(p, off));
    if (lane == 0) r[k] = p;
    __syncthreads();
    if (threadIdx.x != 0) return;
    const V3 mn{r[0].v, r[1].v, r[2].v}, mx{r[3].v, r[4].v, r[5].v};
    const V3 size = vsub(mx, mn);
    const V3 pad{size.x * padx, size.y * pady, size.z * padz};
    const V3 dmin = vsub(mn, pad), dmax = vadd(mx, pad);
    const V3 dsize = vsub(dmax, dmin);
    const float longest = max3(dsize.x, dsize.y, dsize.z);
    const int res = target_res > 4 ? target_res : 4;
    float cs = longest / (float)res;
    if (cs < 1e-6f) cs = 1e-6f;
    const int nx = to_int_host(ceilf(dsize.y / cs)), ny = to_int_host(ceilf(dsize.x / cs)),
              nz = to_int_host(ceilf(dsize.z / cs));
    out->dims[0] = nx > 1 ? nx : 1;
    out->dims[1] = ny > 1 ? ny : 1;
    out->dims[2] = nz > 1 ? nz : 1;
    out->cell = cs;
    out->origin[0] = dmin.x;
    out->origin[1] = dmin.y;
    out->origin[2] = dmin.z;
}

// ---- 2. triangle records and tile binning ----

struct GridDev {
    int nx, ny, nz;
    int tx, ty, tz;  // tiles per axis
    float cs, cr;
    float ox, oy, oz;
};

// Status words of a call: error bits, the tiles that hold a triangle, and the
// tiles with long lists.
struct Status {
    int err;
    unsigned occupied, longest, long_tiles;
};

// Marks tile (x, y, z) in `slot`; 1 where it was not marked before.
__device__ __forceinline__ unsigned mark_tile(uint32_t* __restrict__ slot, const GridDev& g, int x, int y, int z) {
    uint32_t* m = slot + (((size_t)z * g.ty + y) * g.tx + x);
    return __ldcg(m) == 0u && atomicExch(m, 1u) == 0u ? 1u : 0u;
}

// The record and pair count of triangle t, and where its box holds at most
// kOwnTiles tiles their marks in `slot`; true where it holds more.
constexpr unsigned kOwnTiles = 32;
__device__ __forceinline__ bool prep_triangle(const float* __restrict__ pos, unsigned nv,
                                              const uint32_t* __restrict__ idx, unsigned ntri, const GridDev& g,
                                              Tri* tris, unsigned long long* __restrict__ counts, uint32_t* slot,
                                              Status* st, unsigned t) {
    if (t > ntri) return false;
    if (t == ntri) {  // the scan's trailing slot, so offsets[ntri] is the pair total
        counts[t] = 0;
        return false;
    }
    const uint32_t i0 = idx[3 * (size_t)t], i1 = idx[3 * (size_t)t + 1], i2 = idx[3 * (size_t)t + 2];
    if (i0 >= nv || i1 >= nv || i2 >= nv) {
        atomicOr(&st->err, kErrBadIndex);
        counts[t] = 0;
        return false;
    }
    const V3 a{pos[3 * (size_t)i0], pos[3 * (size_t)i0 + 1], pos[3 * (size_t)i0 + 2]};
    const V3 b{pos[3 * (size_t)i1], pos[3 * (size_t)i1 + 1], pos[3 * (size_t)i1 + 2]};
    const V3 c{pos[3 * (size_t)i2], pos[3 * (size_t)i2 + 1], pos[3 * (size_t)i2 + 2]};
    const V3 rn = vcross(vsub(b, a), vsub(c, a));
    const float nl = vlen(rn);
    Tri r{};
    r.a[0] = a.x, r.a[1] = a.y, r.a[2] = a.z;
    r.b[0] = b.x, r.b[1] = b.y, r.b[2] = b.z;
    r.c[0] = c.x, r.c[1] = c.y, r.c[2] = c.z;
    unsigned long long cnt = 0;
    if (nl <= 1e-12f) {  // zero-area triangles touch no cell
        r.n[0] = r.n[1] = r.n[2] = 0.0f;
        r.lo[0] = r.lo[1] = r.lo[2] = 1;
        r.hi[0] = r.hi[1] = r.hi[2] = 0;
    } else {
        const V3 un = vmul(rn, 1.0f / nl);
        r.n[0] = un.x, r.n[1] = un.y, r.n[2] = un.z;
        const V3 tmin{min3(a.x, b.x, c.x), min3(a.y, b.y, c.y), min3(a.z, b.z, c.z)};
        const V3 tmax{max3(a.x, b.x, c.x), max3(a.y, b.y, c.y), max3(a.z, b.z, c.z)};
        int lo0 = to_int_host(floorf((tmin.y - g.cr - g.oy) / g.cs));
        int lo1 = to_int_host(floorf((tmin.x - g.cr - g.ox) / g.cs));
        int lo2 = to_int_host(floorf((tmin.z - g.cr - g.oz) / g.cs));
        int hi0 = to_int_host(ceilf((tmax.y + g.cr - g.oy) / g.cs));
        int hi1 = to_int_host(ceilf((tmax.x + g.cr - g.ox) / g.cs));
        int hi2 = to_int_host(ceilf((tmax.z + g.cr - g.oz) / g.cs));
        lo0 = lo0 < 0 ? 0 : lo0;
        lo1 = lo1 < 0 ? 0 : lo1;
        lo2 = lo2 < 0 ? 0 : lo2;
        hi0 = hi0 > g.nx - 1 ? g.nx - 1 : hi0;
        hi1 = hi1 > g.ny - 1 ? g.ny - 1 : hi1;
        hi2 = hi2 > g.nz - 1 ? g.nz - 1 : hi2;
        r.lo[0] = lo0, r.lo[1] = lo1, r.lo[2] = lo2;
        r.hi[0] = hi0, r.hi[1] = hi1, r.hi[2] = hi2;
        if (lo0 <= hi0 && lo1 <= hi1 && lo2 <= hi2) {
            cnt = (unsigned long long)(hi0 / kTile - lo0 / kTile + 1) * (hi1 / kTile - lo1 / kTile + 1) *
                  (hi2 / kTile - lo2 / kTile + 1);
            if (cnt <= kOwnTiles) {
                unsigned fresh = 0;
                for (int z = lo2 / kTile; z <= hi2 / kTile; ++z)
                    for (int y = lo1 / kTile; y <= hi1 / kTile; ++y)
                        for (int x = lo0 / kTile; x <= hi0 / kTile; ++x) fresh += mark_tile(slot, g, x, y, z);
                if (fresh) atomicAdd(&st->occupied, fresh);
            }
        }
    }
    tris[t] = r;
    counts[t] = cnt;
    return cnt > kOwnTiles;
}

// Also marks every tile a triangle's box touches in `slot` (zeroed) and counts
// the marked tiles. A tile is a trip to memory, so a box of many is marked by
// the whole block, four tiles per thread in flight: two facets across a
// 1024x512x512 grid took 316 ms with all tiles of a box on its thread.
constexpr int kPrepThreads = 256;
__global__ void __launch_bounds__(kPrepThreads) k_tri_prep(const float* __restrict__ pos, unsigned nv,
                                                           const uint32_t* __restrict__ idx, unsigned ntri, GridDev g,
                                                           Tri* tris, unsigned long long* __restrict__ counts,
                                                           uint32_t* slot, Status* st) {
    __shared__ unsigned s_big[kPrepThreads], s_count;
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    const unsigned t = blockIdx.x * kPrepThreads + threadIdx.x;
    if (prep_triangle(pos, nv, idx, ntri, g, tris, counts, slot, st, t)) s_big[atomicAdd(&s_count, 1u)] = t;
    __syncthreads();
    unsigned fresh = 0;
    for (unsigned b = 0; b < s_count; ++b) {
        const Tri& r = tris[s_big[b]];
        const int x0 = r.lo[0] / kTile, y0 = r.lo[1] / kTile, z0 = r.lo[2] / kTile;
        const unsigned wx = r.hi[0] / kTile - x0 + 1, wy = r.hi[1] / kTile - y0 + 1, wz = r.hi[2] / kTile - z0 + 1;
        const uint64_t count = (uint64_t)wx * wy * wz;
        for (uint64_t k0 = threadIdx.x; k0 < count; k0 += 4 * kPrepThreads) {
            uint32_t* m[4];
            uint32_t old[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint64_t k = k0 + u * kPrepThreads < count ? k0 + u * kPrepThreads : k0;
                const uint64_t row = k / wx;
                m[u] = slot + (((size_t)z0 + row / wy) * g.ty + y0 + row % wy) * g.tx + x0 + (k - row * wx);
                old[u] = __ldcg(m[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (old[u] == 0u && atomicExch(m[u], 1u) == 0u) ++fresh;
        }
    }
    if (fresh) atomicAdd(&st->occupied, fresh);
}

__global__ void k_tri_emit(const Tri* __restrict__ tris, const unsigned long long* __restrict__ offsets,
                           unsigned ntri, GridDev g, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntri) return;
    const unsigned long long off = offsets[t], end = offsets[t + 1];
    if (off == end) return;
    const Tri& r = tris[t];
    const int x0 = r.lo[0] / kTile, x1 = r.hi[0] / kTile;
    const int y0 = r.lo[1] / kTile, y1 = r.hi[1] / kTile;
    const int z0 = r.lo[2] / kTile, z1 = r.hi[2] / kTile;
    unsigned long long o = off;
    for (int z = z0; z <= z1; ++z)
        for (int y = y0; y <= y1; ++y)
            for (int x = x0; x <= x1; ++x) {
                keys[o] = (uint32_t)(((size_t)z * g.ty + y) * g.tx + x);
                vals[o] = t;
                ++o;
            }
}

// ---- 3. raster ----

// A tile with at most kShortList triangles is rasterized by one block, one with
// more by a block per box (k_vox_raster).
// Whole call on a B200, every tile by one block / by boxes, average list in
// brackets: two facets across 640x320x320 (2) 6.5 / 13.7 ms; icosphere of 1280
// triangles at 640 cells (4) 0.84 / 1.23 ms, of 20480 (20) 0.98 / 1.12, of 5120
// at 128 cells (87) 0.54 / 0.48; wing at 256 cells (54) 0.62 / 0.56; aircraft at
// 640 (274) 2.11 / 0.86, at 96 (6781) 10.7 / 2.1.
constexpr unsigned kShortList = 32, kLongestList = 512;

// slot[tile] = its place in the list of occupied tiles + 1 (0: no triangle);
// the places of the tiles with long lists in `long_tiles`: more than
// kLongestList triangles from the front, the others from the back.
__global__ void k_tile_slots(const uint32_t* __restrict__ run_tile, const uint32_t* __restrict__ run_len,
                             unsigned runs, uint32_t* __restrict__ slot, uint32_t* __restrict__ long_tiles,
                             Status* __restrict__ st) {
    const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= runs) return;
    slot[run_tile[k]] = k + 1u;
    if (run_len[k] > kLongestList)
        long_tiles[atomicAdd(&st->longest, 1u)] = k;
    else if (run_len[k] > kShortList)
        long_tiles[runs - 1u - atomicAdd(&st->long_tiles, 1u)] = k;
}

// A cell's running state, and the update by one more triangle of its list
// (distance, signed normal projection; a NaN distance changes nothing).
struct CellState {
    float sd = INFINITY, bp = -1.0f;
    bool sol = false;
    __device__ __forceinline__ void add(float dist, float nd, float tie, float cr) {
        const float and_ = fabsf(nd);
        const float bd = fabsf(sd);
        // Voxelizer.cpp:258-290: a clearly nearer triangle replaces the
        // cell's distance; within the tie tolerance the one whose normal
        // points more directly at the cell decides the sign
        if (dist + tie < bd) {
            sd = nd < 0.0f ? -dist : dist;
            bp = and_;
        } else if (dist <= bd + tie) {
            if (and_ > bp) {
                const float md = dist < bd ? dist : bd;
                sd = nd < 0.0f ? -md : md;
                bp = and_;
            } else if (dist < bd) {
                sd = sd < 0.0f ? -dist : dist;
            }
        }
        if (dist <= cr) sol = true;
    }
};

// Short lists: a block per tile, two cells per thread, the triangles staged
// through shared memory in list order. What a block costs before and after its
// triangles is paid once per tile here, once per box in the other form.
constexpr int kRasterThreads = 256;
__device__ __forceinline__ void raster_tile(unsigned tile_at, uint32_t tile, unsigned count,
                                            const uint32_t* __restrict__ list, const Tri* __restrict__ tris,
                                            const GridDev& g, uint8_t* __restrict__ solid, float* __restrict__ sdf,
                                            uint8_t* __restrict__ mask) {
    __shared__ Tri s_tri[kShortList];
    if (threadIdx.x < count) s_tri[threadIdx.x] = tris[list[threadIdx.x]];
    __syncthreads();
    const int x = (int)(tile % (uint32_t)g.tx) * kTile + (threadIdx.x & 7);
    const int y = (int)((tile / (uint32_t)g.tx) % (uint32_t)g.ty) * kTile + ((threadIdx.x >> 3) & 7);
    const int z0 = (int)(tile / ((uint32_t)g.tx * (uint32_t)g.ty)) * kTile;
    const float tie = g.cs * 1e-3f;
#pragma unroll 1
    for (int c = threadIdx.x; c < kTileCells; c += kRasterThreads) {
        const int z = z0 + (c >> 6);
        const bool inside = x < g.nx && y < g.ny && z < g.nz;
        // CellCenter: world x from grid y, world y from grid x (VoxelGrid.h:43-56)
        const V3 at{g.ox + ((float)y + 0.5f) * g.cs, g.oy + ((float)x + 0.5f) * g.cs, g.oz + ((float)z + 0.5f) * g.cs};
        CellState cell;
        for (unsigned k = 0; inside && k < count; ++k) {
            const Tri& r = s_tri[k];
            if (x < r.lo[0] || x > r.hi[0] || y < r.lo[1] || y > r.hi[1] || z < r.lo[2] || z > r.hi[2]) continue;
            const V3 a{r.a[0], r.a[1], r.a[2]}, b{r.b[0], r.b[1], r.b[2]}, d{r.c[0], r.c[1], r.c[2]};
            const V3 diff = vsub(at, closest_on_triangle(at, a, b, d));
            cell.add(vlen(diff), vdot(diff, V3{r.n[0], r.n[1], r.n[2]}), tie, g.cr);
        }
        const unsigned fluid = __ballot_sync(0xffffffffu, inside && !cell.sol);
        if (inside) {
            const size_t i = ((size_t)z * g.ny + y) * g.nx + x;
            solid[i] = cell.sol ? 1 : 0;
            sdf[i] = cell.sd;
        }
        const unsigned lane = threadIdx.x & 31u;
        if (lane < 4) {  // the warp's four rows, eight bits each
            const unsigned r = (fluid >> (8 * lane)) & 0xffu;
            reinterpret_cast<uint16_t*>(mask)[(size_t)tile_at * kTileRows + (c >> 5) * 4 + lane] =
                (uint16_t)((r & 0xfu) | (r >> 4) << 8);
        }
    }
}

// The first 16 x most blocks take the tiles with long lists, box by box: block
// 16k + w box w (4x4x2 cells, one per lane) of the k-th such tile, the longest
// lists first, since a box of thousands of triangles outlasts the rest. The
// other blocks take the short ones and fill in behind. The list order matters only to the running state, not to a triangle's distance
// from a cell, so all threads compute the distances of a chunk of the box's
// triangles at once, one (triangle, cell) pair each, for the cells inside the
// triangle's own box only; warp 0 then applies the update rule to them in
// order. A list can be long (thousands of triangles where a mesh comes to a
// point), and a triangle's box covers a fifth of the cells of the boxes it
// overlaps. The 57,516-triangle aircraft on 31M cells, B200: one triangle after
// another per cell 0.78 ms, a triangle per warp 0.35 ms, a pair per thread in
// blocks of 256 0.29 ms (of 512 0.35). What is left is latency: a block's
// chain of list, box and triangle loads, at 46 % of the warp slots and 35 % of
// the issue slots; a branch-free closest_on_triangle measured the same. Also
// writes the fluid bits of the box's rows, which the flood fill runs on.
constexpr int kRasterWarps = kRasterThreads / 32;
constexpr int kRasterChunk = 64;  // distances kept at a time
constexpr int kTileBoxes = kTileCells / 32;
__global__ void __launch_bounds__(kRasterThreads, 4) k_vox_raster(
    const Tri* __restrict__ tris, const uint32_t* __restrict__ tile_tris, const uint32_t* __restrict__ run_tile,
    const uint32_t* __restrict__ run_len, const unsigned long long* __restrict__ run_off, unsigned runs,
    const uint32_t* __restrict__ long_tiles, unsigned most, const Status* __restrict__ st, GridDev g,
    uint8_t* __restrict__ solid, float* __restrict__ sdf, uint8_t* __restrict__ mask) {
    unsigned k;
    if (blockIdx.x >= kTileBoxes * most) {
        k = blockIdx.x - kTileBoxes * most;
        if (run_len[k] <= kShortList)
            raster_tile(k, run_tile[k], run_len[k], tile_tris + run_off[k], tris, g, solid, sdf, mask);
        return;
    }
    k = blockIdx.x / kTileBoxes;
    const unsigned longest = st->longest;
    if (k >= longest + st->long_tiles) return;
    k = long_tiles[k < longest ? k : runs - 1u - (k - longest)];
    __shared__ uint32_t s_hit[kRasterThreads];
    __shared__ float2 s_res[kRasterChunk][32];  // distance and signed normal projection; NaN: outside the box
    __shared__ unsigned s_count[kRasterWarps];
    // the chunk's triangles: their cells of the box (first cell and size per
    // axis) and the pairs up to and including each
    __shared__ uint32_t s_clip[kRasterChunk], s_pairs[kRasterChunk], s_part[kRasterChunk / 32];
    const unsigned w = blockIdx.x % kTileBoxes;
    const uint32_t tile = run_tile[k];
    const unsigned count = run_len[k];
    const uint32_t* list = tile_tris + run_off[k];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the block's box, and this lane's cell in it
    const int lx = (w & 1) * 4, ly = ((w >> 1) & 1) * 4, lz = (w >> 2) * 2;
    const int bx = (int)(tile % (uint32_t)g.tx) * kTile + lx;
    const int by = (int)((tile / (uint32_t)g.tx) % (uint32_t)g.ty) * kTile + ly;
    const int bz = (int)(tile / ((uint32_t)g.tx * (uint32_t)g.ty)) * kTile + lz;
    const int x = bx + (lane & 3), y = by + ((lane >> 2) & 3), z = bz + (lane >> 4);
    const bool inside = x < g.nx && y < g.ny && z < g.nz;
    const float tie = g.cs * 1e-3f;
    CellState cell;
    const bool empty = bx >= g.nx || by >= g.ny || bz >= g.nz;  // a box behind the grid's edge
    for (unsigned base = 0; base < count && !empty; base += kRasterThreads) {
        // the list's next triangles that overlap the box, in list order
        bool hit = false;
        uint32_t mine = 0;
        if (base + threadIdx.x < count) {
            mine = list[base + threadIdx.x];
            const int4* r = reinterpret_cast<const int4*>(tris + mine) + 3;
            const int4 u = __ldg(r), v = __ldg(r + 1);  // lo[0..2] hi[0] | hi[1..2]
            hit = bx <= u.w && bx + 3 >= u.x && by <= v.x && by + 3 >= u.y && bz <= v.y && bz + 1 >= u.z;
        }
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) s_count[warp] = __popc(hits);
        __syncthreads();
        unsigned place = 0, m = 0;
        for (int j = 0; j < kRasterWarps; ++j) {
            if (j < warp) place += s_count[j];
            m += s_count[j];
        }
        if (hit) s_hit[place + __popc(hits & ((1u << lane) - 1u))] = mine;
        __syncthreads();
        for (unsigned c0 = 0; c0 < m; c0 += kRasterChunk) {
            const unsigned c1 = c0 + kRasterChunk < m ? c0 + kRasterChunk : m;
            if (threadIdx.x < kRasterChunk) {
                unsigned n = 0;
                if (c0 + threadIdx.x < c1) {
                    const int4* r = reinterpret_cast<const int4*>(tris + s_hit[c0 + threadIdx.x]) + 3;
                    const int4 u = __ldg(r), v = __ldg(r + 1);
                    const int x0 = max(u.x, bx), x1 = min(u.w, bx + 3), y0 = max(u.y, by), y1 = min(v.x, by + 3),
                              z0 = max(u.z, bz), z1 = min(v.y, bz + 1);
                    s_clip[threadIdx.x] = (uint32_t)((x0 - bx) | (y0 - by) << 2 | (z0 - bz) << 4 | (x1 - x0) << 5 |
                                                     (y1 - y0) << 7 | (z1 - z0) << 9);
                    n = (unsigned)((x1 - x0 + 1) * (y1 - y0 + 1) * (z1 - z0 + 1));
                }
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned t = __shfl_up_sync(0xffffffffu, n, o);
                    if (lane >= o) n += t;
                }
                s_pairs[threadIdx.x] = n;
                if (lane == 31) s_part[warp] = n;
            }
            for (unsigned r = threadIdx.x; r < (c1 - c0) * 32u; r += kRasterThreads)
                s_res[r >> 5][r & 31u].x = __int_as_float(0x7fffffff);
            __syncthreads();
            if (threadIdx.x < kRasterChunk) {
                unsigned n = s_pairs[threadIdx.x];
                for (int j = 0; j < warp; ++j) n += s_part[j];
                s_pairs[threadIdx.x] = n;
            }
            __syncthreads();
            const unsigned total = s_pairs[kRasterChunk - 1];
            for (unsigned pr = threadIdx.x; pr < total; pr += kRasterThreads) {
                unsigned lo = 0, hi = c1 - c0 - 1;  // the first triangle whose pairs pass pr
                while (lo < hi) {
                    const unsigned mid = (lo + hi) >> 1;
                    if (s_pairs[mid] > pr)
                        hi = mid;
                    else
                        lo = mid + 1;
                }
                const unsigned first = lo ? s_pairs[lo - 1] : 0u, clip = s_clip[lo];
                const unsigned wx = ((clip >> 5) & 3u) + 1u, wy = ((clip >> 7) & 3u) + 1u;
                const unsigned q = pr - first, qy = q / wx, qz = qy / wy;
                const unsigned cx = (clip & 3u) + q - qy * wx, cy = ((clip >> 2) & 3u) + qy - qz * wy,
                               cz = ((clip >> 4) & 1u) + qz;
                // CellCenter: world x from grid y, world y from grid x (VoxelGrid.h:43-56)
                const V3 at{g.ox + ((float)(by + (int)cy) + 0.5f) * g.cs, g.oy + ((float)(bx + (int)cx) + 0.5f) * g.cs,
                            g.oz + ((float)(bz + (int)cz) + 0.5f) * g.cs};
                const float4* r = reinterpret_cast<const float4*>(tris + s_hit[c0 + lo]);
                const float4 f0 = __ldg(r), f1 = __ldg(r + 1), f2 = __ldg(r + 2);
                const V3 a{f0.x, f0.y, f0.z}, b{f0.w, f1.x, f1.y}, c{f1.z, f1.w, f2.x};
                const V3 diff = vsub(at, closest_on_triangle(at, a, b, c));
                s_res[lo][cx | cy << 2 | cz << 4] = make_float2(vlen(diff), vdot(diff, V3{f2.y, f2.z, f2.w}));
            }
            __syncthreads();
            if (warp == 0) {
#pragma unroll 4
                for (unsigned h = c0; h < c1; ++h) {
                    cell.add(s_res[h - c0][lane].x, s_res[h - c0][lane].y, tie, g.cr);
                }
            }
            __syncthreads();
        }
    }
    if (warp != 0) return;
    const unsigned fluid = __ballot_sync(0xffffffffu, inside && !cell.sol);
    if (inside) {
        const size_t i = ((size_t)z * g.ny + y) * g.nx + x;
        solid[i] = cell.sol ? 1 : 0;
        sdf[i] = cell.sd;
    }
    if (lane < 8)  // row (y, z) of the box: four bits
        mask[((size_t)k * kTileRows + (lz + (lane >> 2)) * kTile + ly + (lane & 3)) * 2 + (w & 1)] =
            (uint8_t)((fluid >> (4 * lane)) & 0xfu);
}

// ---- 4. flood fill (connected components of fluid nodes) ----

// Node ids: a tile without triangles is its tile index; the run of fluid
// cells that starts at bit b of row (y, z) of occupied tile k is ntiles +
// nodes k + (ry z + y) rx + b / 2 (two runs of a row are at least two bits
// apart), with rx = 4 and ry = 8 and fewer in grids thinner than a tile, so that
// there are no more nodes than a tile has cells. Id is 32 bits wherever the ids
// fit.
template <class Id>
struct Flood {
    int tx, ty, tz;
    int rx, ry, nodes;
    Id ntiles;
    const uint32_t* slot;
    const uint8_t* mask;  // fluid bits of the occupied tiles' rows: a byte per four cells
    Id* L;
    int* err;
    __device__ __forceinline__ Id run(uint32_t slot1, int row, unsigned m, int bit) const {
        const unsigned starts = m & ~(m << 1);
        const int b = 31 - __clz(starts & ((2u << bit) - 1u));
        return ntiles + (Id)(slot1 - 1u) * (Id)nodes + (Id)((row / kTile * ry + row % kTile) * rx + (b >> 1));
    }
    __device__ __forceinline__ unsigned row_mask(uint32_t slot1, int row) const {
        const unsigned v = reinterpret_cast<const uint16_t*>(mask)[(size_t)(slot1 - 1u) * kTileRows + row];
        return (v & 0xfu) | (v >> 4);
    }
};

template <class Id>
__device__ __forceinline__ Id find_root(const Id* __restrict__ L, Id a, int* err) {
    for (unsigned hop = 0; hop < kMaxFindHops; ++hop) {
        const Id p = __ldcg(L + a);
        if (p == a) return a;
        a = p;
    }
    atomicOr(err, kErrUnionBound);
    return a;
}

template <class Id>
__device__ void unite(Id* L, Id a, Id b, int* err) {
    for (int it = 0; it < kMaxMergeRetries; ++it) {
        a = find_root(L, a, err);
        b = find_root(L, b, err);
        if (a == b) return;
        if (a < b) {
            const Id old = atomicMin(L + b, a);
            if (old == b) return;
            b = old;
        } else {
            const Id old = atomicMin(L + a, b);
            if (old == a) return;
            a = old;
        }
    }
    atomicOr(err, kErrUnionBound);
}

// Labels: one thread per tile row gives each empty tile the first tile of its
// x-run of empty tiles; the runs of occupied tiles label themselves.
template <class Id>
__global__ void k_ff_label(Flood<Id> f, unsigned occupied) {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t row = t; row < (size_t)f.ty * f.tz; row += step) {
        Id start = 0;
        bool open = false;
        for (int x = 0; x < f.tx; ++x) {
            const Id i = (Id)(row * f.tx + x);
            const bool empty = f.slot[i] == 0u;
            if (empty && !open) start = i;
            open = empty;
            f.L[i] = empty ? start : i;
        }
    }
    for (size_t k = t; k < (size_t)occupied * f.nodes; k += step) f.L[f.ntiles + k] = (Id)(f.ntiles + k);
}

// Joins empty tiles with the row below and the layer below, once per stretch
// of tiles that are empty on both sides.
template <class Id>
__global__ void k_ff_tiles(Flood<Id> f) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)f.ntiles || f.slot[i] != 0u) return;
    const int x = (int)(i % f.tx);
    const size_t row = i / f.tx;
    const int y = (int)(row % f.ty), z = (int)(row / f.ty);
    const bool left = x > 0 && f.slot[i - 1] == 0u;
    auto join = [&](size_t below) {
        if (f.slot[below] == 0u && !(left && f.slot[below - 1] == 0u)) unite<Id>(f.L, (Id)i, (Id)below, f.err);
    };
    if (y > 0) join(i - f.tx);
    if (z > 0) join(i - (size_t)f.tx * f.ty);
}

// Joins the runs of an occupied tile (one thread per row) with those of the
// row below, the layer below and the tile to the left, and with empty tiles
// on every side.
template <class Id>
__global__ void __launch_bounds__(kTileRows) k_ff_runs(Flood<Id> f, const uint32_t* __restrict__ run_tile) {
    const uint32_t s1 = blockIdx.x + 1u, tile = run_tile[blockIdx.x];
    const int row = threadIdx.x, ly = row & (kTile - 1), lz = row / kTile;
    const unsigned m = f.row_mask(s1, row);
    if (!m) return;
    const int x = (int)(tile % (uint32_t)f.tx);
    const uint32_t tr = tile / (uint32_t)f.tx;
    const int y = (int)(tr % (uint32_t)f.ty), z = (int)(tr / (uint32_t)f.ty);
    // this row with row `r2` of the tile `other` (s2 = its slot; 0: empty, all fluid)
    auto rows = [&](uint32_t other, uint32_t s2, int r2) {
        const unsigned o = s2 ? f.row_mask(s2, r2) : 0xffu;
        const unsigned both = m & o;
        for (unsigned b = both & ~(both << 1); b; b &= b - 1u) {
            const int bit = __ffs(b) - 1;
            unite<Id>(f.L, f.run(s1, row, m, bit), s2 ? f.run(s2, r2, o, bit) : (Id)other, f.err);
        }
    };
    const uint32_t dy = (uint32_t)f.tx, dz = (uint32_t)f.tx * (uint32_t)f.ty;
    if (ly > 0)
        rows(tile, s1, row - 1);
    else if (y > 0)
        rows(tile - dy, f.slot[tile - dy], row + kTile - 1);
    if (lz > 0)
        rows(tile, s1, row - kTile);
    else if (z > 0)
        rows(tile - dz, f.slot[tile - dz], row + kTileRows - kTile);
    if (ly == kTile - 1 && y + 1 < f.ty && f.slot[tile + dy] == 0u) rows(tile + dy, 0u, 0);
    if (lz == kTile - 1 && z + 1 < f.tz && f.slot[tile + dz] == 0u) rows(tile + dz, 0u, 0);
    if ((m & 1u) && x > 0) {
        const uint32_t s2 = f.slot[tile - 1];
        if (!s2) {
            unite<Id>(f.L, f.run(s1, row, m, 0), (Id)(tile - 1), f.err);
        } else {
            const unsigned o = f.row_mask(s2, row);
            if (o & 0x80u) unite<Id>(f.L, f.run(s1, row, m, 0), f.run(s2, row, o, 7), f.err);
        }
    }
    if ((m & 0x80u) && x + 1 < f.tx && f.slot[tile + 1] == 0u)
        unite<Id>(f.L, f.run(s1, row, m, 7), (Id)(tile + 1), f.err);
}

// The reached cells: a byte per empty tile, the bits of every row of the
// occupied tiles. Nothing is reached when cell 0 is solid.
template <class Id>
__global__ void k_ff_reached(Flood<Id> f, unsigned occupied, uint8_t* __restrict__ tile_reached,
                             uint8_t* __restrict__ row_reached) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)f.ntiles + (size_t)occupied * kTileRows) return;
    const uint32_t s0 = f.slot[0];
    const unsigned m0 = s0 ? f.row_mask(s0, 0) : 1u;
    const bool seed = (m0 & 1u) != 0u;
    const Id r0 = seed ? find_root<Id>(f.L, s0 ? f.run(s0, 0, m0, 0) : (Id)0, f.err) : (Id)0;
    if (i < (size_t)f.ntiles) {
        if (f.slot[i] == 0u) tile_reached[i] = seed && find_root<Id>(f.L, (Id)i, f.err) == r0 ? 1 : 0;
        return;
    }
    const size_t k = i - (size_t)f.ntiles;
    const uint32_t s1 = (uint32_t)(k / kTileRows) + 1u;
    const int row = (int)(k % kTileRows);
    const unsigned m = f.row_mask(s1, row);
    unsigned r = 0;
    if (seed)
        for (unsigned b = m & ~(m << 1); b; b &= b - 1u) {
            const int bit = __ffs(b) - 1;
            if (find_root<Id>(f.L, f.run(s1, row, m, bit), f.err) == r0)
                r |= m & ~(m + (1u << bit));  // the run: the carry out of its lowest bit clears it
        }
    row_reached[k] = (uint8_t)r;
}

// ---- 5. finalize ----

// One warp per 128-cell segment of an x row, four cells of one tile per lane
// (tiles start on multiples of 8). kVec: rows start on four-cell boundaries
// and the arrays are aligned, so the four cells move as one vector.
template <bool kVec>
__global__ void __launch_bounds__(256) k_vox_finalize(uint8_t* __restrict__ solid, float* __restrict__ sdf, GridDev g,
                                                      const uint32_t* __restrict__ slot,
                                                      const uint8_t* __restrict__ tile_reached,
                                                      const uint8_t* __restrict__ row_reached, int segs) {
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t row = warp / (size_t)segs;
    if (row >= (size_t)g.ny * g.nz) return;
    const int x = (int)(warp - row * (size_t)segs) * 128 + (int)(threadIdx.x & 31) * 4;
    if (x >= g.nx) return;
    const int y = (int)(row % (size_t)g.ny), z = (int)(row / (size_t)g.ny);
    const size_t tile = ((size_t)(z / kTile) * g.ty + y / kTile) * g.tx + x / kTile;
    const uint32_t s1 = slot[tile];
    const size_t i = row * g.nx + x;
    const int n = g.nx - x < 4 ? g.nx - x : 4;
    uint8_t s[4];
    float d[4];
    if (!s1) {
        const bool out = tile_reached[tile] != 0;
        for (int k = 0; k < 4; ++k) {
            s[k] = out ? 0 : 1;
            d[k] = out ? INFINITY : -INFINITY;
        }
    } else {
        const unsigned r = row_reached[(size_t)(s1 - 1u) * kTileRows + (z & (kTile - 1)) * kTile + (y & (kTile - 1))] >>
                           (x & (kTile - 1));
        if constexpr (kVec) {
            const uchar4 a = *reinterpret_cast<const uchar4*>(solid + i);
            const float4 b = *reinterpret_cast<const float4*>(sdf + i);
            s[0] = a.x, s[1] = a.y, s[2] = a.z, s[3] = a.w;
            d[0] = b.x, d[1] = b.y, d[2] = b.z, d[3] = b.w;
        } else {
            for (int k = 0; k < n; ++k) s[k] = solid[i + k], d[k] = sdf[i + k];
        }
        for (int k = 0; k < 4; ++k) {
            if (!kVec && k >= n) break;
            const bool so = s[k] != 0 || !((r >> k) & 1u);
            const float a = fabsf(d[k]);
            if (!so)
                d[k] = a;
            else if (a > g.cr)
                d[k] = -a;
            s[k] = so ? 1 : 0;
        }
    }
    if constexpr (kVec) {
        *reinterpret_cast<uchar4*>(solid + i) = make_uchar4(s[0], s[1], s[2], s[3]);
        *reinterpret_cast<float4*>(sdf + i) = make_float4(d[0], d[1], d[2], d[3]);
    } else {
        for (int k = 0; k < n; ++k) solid[i + k] = s[k], sdf[i + k] = d[k];
    }
}

// ---- host side ----

int wait_on(cudaStream_t s) {
    cudaEvent_t ev;
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return FC_LBM_ERR_CUDA;
    if (cudaEventRecord(ev, s) != cudaSuccess) {
        cudaEventDestroy(ev);
        return FC_LBM_ERR_CUDA;
    }
    const cudaError_t e = fc::poll_until([&] { return cudaEventQuery(ev); }, kWaitTimeoutMs);
    const int rc = e == cudaSuccess ? FC_LBM_OK : (e == cudaErrorNotReady ? FC_LBM_ERR_TIMEOUT : FC_LBM_ERR_CUDA);
    cudaEventDestroy(ev);
    return rc;
}

// One array of a combined allocation.
struct Part {
    void** p;
    size_t bytes;
    template <class T>
    Part(T** q, size_t count) : p(reinterpret_cast<void**>(q)), bytes(count * sizeof(T)) {}
    Part(void** q, size_t b) : p(q), bytes(b) {}
};

// Stream-ordered scratch allocations, freed together on the same stream when
// the call returns (every path that hands results back has waited first).
struct Scratch {
    cudaStream_t s;
    void* ptrs[8] = {};
    int n = 0;
    explicit Scratch(cudaStream_t st) : s(st) {}
    template <class T>
    cudaError_t get(T** p, size_t bytes) {
        *p = nullptr;
        if (n >= 8) return cudaErrorInvalidValue;
        void* q = nullptr;
        const cudaError_t e = cudaMallocAsync(&q, bytes ? bytes : 16, s);
        if (e != cudaSuccess) return e;
        ptrs[n++] = q;
        *p = static_cast<T*>(q);
        return cudaSuccess;
    }
    // Several arrays in one allocation, each on a 256-byte boundary: the calls
    // in a pipeline of short kernels are host time that the device waits for.
    cudaError_t get_all(std::initializer_list<Part> parts) {
        size_t total = 0;
        for (const Part& p : parts) total += (p.bytes + 255) / 256 * 256;
        char* base = nullptr;
        const cudaError_t e = get(&base, total);
        if (e != cudaSuccess) return e;
        for (const Part& p : parts) {
            *p.p = base;
            base += (p.bytes + 255) / 256 * 256;
        }
        return cudaSuccess;
    }
    ~Scratch() {
        for (int i = n - 1; i >= 0; --i) cudaFreeAsync(ptrs[i], s);
    }
};

// A driver function, or null.
template <class Fn>
Fn driver_function(const char* name) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return q == cudaDriverEntryPointSuccess ? reinterpret_cast<Fn>(p) : nullptr;
}

// The id of the calling thread's current context, never given twice in a
// process; 0 if there is none.
unsigned long long context_id() {
    using Current = CUresult (*)(CUcontext*);
    using Id = CUresult (*)(CUcontext, unsigned long long*);
    static const auto current = driver_function<Current>("cuCtxGetCurrent");
    static const auto id_of = driver_function<Id>("cuCtxGetId");
    CUcontext c = nullptr;
    unsigned long long id = 0;
    return current && id_of && current(&c) == CUDA_SUCCESS && c && id_of(c, &id) == CUDA_SUCCESS ? id : 0;
}

// A few pinned bytes per host thread for the sizes and status a call reads
// back. A copy to pageable memory waits for the stream inside the driver, and
// the memory pool gives its memory back at such waits: the next call then maps
// it anew, which costs more than the call's kernels. The bytes die with the
// context they were allocated in (cudaDeviceReset): where another one is
// current, the call takes pageable memory.
struct HostWords {
    void* p = nullptr;
    int device = -1;
    unsigned long long context = 0;
    HostWords() {
        context = context_id();
        if (!context || cudaGetDevice(&device) != cudaSuccess || cudaHostAlloc(&p, 64, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();  // the caller falls back to pageable memory
            p = nullptr;
        }
    }
    bool usable() const { return p && context_id() == context; }
    ~HostWords() {
        if (!p) return;
        if (!usable()) {  // the thread has moved to another device since, or the context is gone
            using Get = CUresult (*)(CUdevice*, int);
            using State = CUresult (*)(CUdevice, unsigned*, int*);
            const auto get = driver_function<Get>("cuDeviceGet");
            const auto state = driver_function<State>("cuDevicePrimaryCtxGetState");
            CUdevice d = 0;
            unsigned flags = 0;
            int active = 0;
            if (!get || !state || get(&d, device) != CUDA_SUCCESS || state(d, &flags, &active) != CUDA_SUCCESS ||
                !active || cudaSetDevice(device) != cudaSuccess || !usable())
                return;
        }
        cudaFreeHost(p);
    }
};

struct Answer {
    unsigned long long pairs;
    Status st;
    GridOut grid;
};
static_assert(sizeof(Answer) <= 64, "one HostWords block");

Answer* host_answer(Answer* fallback) {
    static thread_local HostWords w;
    return w.usable() ? static_cast<Answer*>(w.p) : fallback;
}

int code_of(cudaError_t e) {
    if (e == cudaSuccess) return FC_LBM_OK;
    if (e == cudaErrorMemoryAllocation) return FC_LBM_ERR_OUT_OF_MEMORY;
    return FC_LBM_ERR_CUDA;
}

#define VX_TRY(expr)                                   \
    do {                                               \
        const cudaError_t _e = (expr);                 \
        if (_e != cudaSuccess) return code_of(_e);     \
    } while (0)

#define VX_RC(expr)                     \
    do {                                \
        const int _rc = (expr);         \
        if (_rc != FC_LBM_OK) return _rc; \
    } while (0)

int bits_for(uint64_t v) {
    int b = 1;
    while (b < 32 && (uint64_t(1) << b) <= v) ++b;
    return b;
}

int grid_on_device(const float* d_pos, size_t nv, const fc_voxel_params* p, cudaStream_t s, Scratch& sc,
                   GridOut* host) {
    Pick* partial = nullptr;
    GridOut* d_out = nullptr;
    VX_TRY(sc.get(&partial, sizeof(Pick) * 6 * kBoundsBlocks));
    VX_TRY(sc.get(&d_out, sizeof(GridOut)));
    k_bounds_partial<<<kBoundsBlocks, kBoundsThreads, 0, s>>>(d_pos, (unsigned)nv, partial);
    VX_TRY(cudaGetLastError());
    k_grid_final<<<1, kGridThreads, 0, s>>>(partial, kBoundsBlocks, p->target_resolution, p->padding[0], p->padding[1],
                                  p->padding[2], d_out);
    VX_TRY(cudaGetLastError());
    Answer own;
    Answer* ans = host_answer(&own);
    VX_TRY(cudaMemcpyAsync(&ans->grid, d_out, sizeof(GridOut), cudaMemcpyDeviceToHost, s));
    VX_RC(wait_on(s));
    *host = ans->grid;
    return FC_LBM_OK;
}

// Runs that a row of a tile, and a tile, of the grid can hold.
int row_nodes(const GridDev& g) { return (std::min(g.nx, kTile) + 1) / 2; }
int tile_nodes(const GridDev& g) { return row_nodes(g) * std::min(g.ny, kTile) * std::min(g.nz, kTile); }

// The flood fill's kernels: labels, joins, reached flags.
template <class Id>
int flood(const GridDev& g, uint64_t ntiles, unsigned occupied, const uint32_t* slot, const uint8_t* mask,
          const uint32_t* run_tile, Id* L, uint8_t* tile_reached, uint8_t* row_reached, Status* st, cudaStream_t s) {
    const int rx = row_nodes(g), ry = std::min(g.ny, kTile), nodes = tile_nodes(g);
    const Flood<Id> f{g.tx, g.ty, g.tz, rx, ry, nodes, (Id)ntiles, slot, mask, L, &st->err};
    const uint64_t rows = std::max<uint64_t>((uint64_t)g.ty * g.tz, (uint64_t)occupied * nodes);
    k_ff_label<Id><<<(unsigned)std::min<uint64_t>((rows + 127) / 128, 148 * 32), 128, 0, s>>>(f, occupied);
    VX_TRY(cudaGetLastError());
    const uint64_t tile_blocks = (ntiles + 127) / 128;
    const uint64_t reach_blocks = (ntiles + (uint64_t)occupied * kTileRows + 127) / 128;
    if (reach_blocks > (uint64_t)INT32_MAX) return FC_LBM_ERR_TOO_LARGE;
    k_ff_tiles<Id><<<(unsigned)tile_blocks, 128, 0, s>>>(f);
    VX_TRY(cudaGetLastError());
    if (occupied > 0) {
        k_ff_runs<Id><<<occupied, kTileRows, 0, s>>>(f, run_tile);
        VX_TRY(cudaGetLastError());
    }
    k_ff_reached<Id><<<(unsigned)reach_blocks, 128, 0, s>>>(f, occupied, tile_reached, row_reached);
    VX_TRY(cudaGetLastError());
    return FC_LBM_OK;
}

int voxelize_on_device(const float* d_pos, size_t nv, const uint32_t* d_idx, size_t ni, const int32_t dims[3],
                       float cell_size, const float origin[3], uint8_t* d_solid, float* d_sdf, cudaStream_t s,
                       Scratch& sc) {
    const int nx = dims[0], ny = dims[1], nz = dims[2];
    GridDev g;
    g.nx = nx, g.ny = ny, g.nz = nz;
    g.tx = (nx + kTile - 1) / kTile, g.ty = (ny + kTile - 1) / kTile, g.tz = (nz + kTile - 1) / kTile;
    g.cs = cell_size;
    g.cr = cell_size * 0.8660254f;
    g.ox = origin[0], g.oy = origin[1], g.oz = origin[2];
    const unsigned ntri = (unsigned)(ni / 3);
    const uint64_t ntiles = (uint64_t)g.tx * g.ty * g.tz;

    // the first half: triangle records, tile marks, and the sizes of the rest
    Status* d_st = nullptr;
    uint32_t* slot = nullptr;
    Tri* tris = nullptr;
    unsigned long long *counts = nullptr, *offsets = nullptr;
    void* tmp = nullptr;
    size_t tmp_bytes = 0;
    if (ntri > 0)
        VX_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, counts, offsets, (int64_t)ntri + 1, s));
    VX_TRY(sc.get_all({{&d_st, 1}, {&slot, ntiles}, {&tris, ntri}, {&counts, (size_t)ntri + 1},
                       {&offsets, (size_t)ntri + 1}, {&tmp, tmp_bytes}}));
    VX_TRY(cudaMemsetAsync(d_st, 0, sizeof(Status), s));
    VX_TRY(cudaMemsetAsync(slot, 0, sizeof(uint32_t) * ntiles, s));
    Status st{};
    unsigned long long pairs = 0;
    Answer own;
    Answer* ans = host_answer(&own);
    if (ntri > 0) {
        k_tri_prep<<<(ntri + kPrepThreads) / kPrepThreads, kPrepThreads, 0, s>>>(d_pos, (unsigned)nv, d_idx, ntri, g,
                                                                               tris, counts, slot, d_st);
        VX_TRY(cudaGetLastError());
        VX_TRY(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, counts, offsets, (int64_t)ntri + 1, s));
        VX_TRY(cudaMemcpyAsync(&ans->pairs, offsets + ntri, sizeof(pairs), cudaMemcpyDeviceToHost, s));
        VX_TRY(cudaMemcpyAsync(&ans->st, d_st, sizeof(st), cudaMemcpyDeviceToHost, s));
        VX_RC(wait_on(s));
        pairs = ans->pairs;
        st = ans->st;
        if (st.err & kErrBadIndex) return FC_LBM_ERR_INVALID_ARG;
        if (pairs > (unsigned long long)INT32_MAX) return FC_LBM_ERR_TOO_LARGE;
    }
    // the second half: the tiles' triangle lists and the flood fill's nodes
    const unsigned runs = st.occupied;  // the runs of equal tile ids after the sort
    const uint64_t nodes = ntiles + (uint64_t)runs * tile_nodes(g);
    const bool wide = nodes >= 0xffffffffull;
    uint32_t *k0 = nullptr, *k1 = nullptr, *v0 = nullptr, *v1 = nullptr;
    uint32_t *run_tile = nullptr, *run_len = nullptr, *long_tiles = nullptr;
    unsigned long long* run_off = nullptr;
    int* d_runs = nullptr;
    uint8_t *mask = nullptr, *tile_reached = nullptr, *row_reached = nullptr;
    char* labels = nullptr;
    size_t sort_bytes = 0, rle_bytes = 0, scan_bytes = 0;
    const int end_bit = bits_for(ntiles);
    if (pairs > 0) {
        cub::DoubleBuffer<uint32_t> kb(k0, k1), vb(v0, v1);
        VX_TRY(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, kb, vb, (int)pairs, 0, end_bit, s));
        VX_TRY(cub::DeviceRunLengthEncode::Encode(nullptr, rle_bytes, k0, run_tile, run_len, d_runs, (int)pairs, s));
        VX_TRY(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, run_len, run_off, (int64_t)runs, s));
    }
    VX_TRY(sc.get_all({{&k0, pairs}, {&k1, pairs}, {&v0, pairs}, {&v1, pairs}, {&run_tile, runs}, {&run_len, runs},
                       {&long_tiles, runs},
                       {&run_off, runs}, {&d_runs, 1}, {&mask, (size_t)runs * kTileRows * 2}, {&tile_reached, ntiles},
                       {&row_reached, (size_t)runs * kTileRows}, {&labels, nodes * (wide ? 8 : 4)},
                       {&tmp, std::max(sort_bytes, std::max(rle_bytes, scan_bytes))}}));
    if (pairs > 0) {
        k_tri_emit<<<(ntri + 255) / 256, 256, 0, s>>>(tris, offsets, ntri, g, k0, v0);
        VX_TRY(cudaGetLastError());
        cub::DoubleBuffer<uint32_t> kb(k0, k1), vb(v0, v1);
        VX_TRY(cub::DeviceRadixSort::SortPairs(tmp, sort_bytes, kb, vb, (int)pairs, 0, end_bit, s));
        VX_TRY(cub::DeviceRunLengthEncode::Encode(tmp, rle_bytes, kb.Current(), run_tile, run_len, d_runs, (int)pairs,
                                                   s));
        VX_TRY(cub::DeviceScan::ExclusiveSum(tmp, scan_bytes, run_len, run_off, (int64_t)runs, s));
        k_tile_slots<<<(runs + 255) / 256, 256, 0, s>>>(run_tile, run_len, runs, slot, long_tiles, d_st);
        VX_TRY(cudaGetLastError());
        // as many tiles as can have a long list, a block per box, and a block per tile:
        // below 2^31 blocks (pairs < 2^31, and runs <= 2^29, since a grid of below 2^32
        // cells has at least eight for each of its tiles)
        const unsigned most = std::min<unsigned>(runs, (unsigned)(pairs / (kShortList + 1)));
        k_vox_raster<<<kTileBoxes * most + runs, kRasterThreads, 0, s>>>(tris, vb.Current(), run_tile, run_len, run_off,
                                                                       runs, long_tiles, most, d_st, g, d_solid, d_sdf,
                                                                       mask);
        VX_TRY(cudaGetLastError());
    }
    VX_RC(wide ? flood(g, ntiles, runs, slot, mask, run_tile, reinterpret_cast<unsigned long long*>(labels),
                       tile_reached, row_reached, d_st, s)
               : flood(g, ntiles, runs, slot, mask, run_tile, reinterpret_cast<uint32_t*>(labels), tile_reached,
                       row_reached, d_st, s));
    const int segs = (nx + 127) / 128;
    const size_t fin_blocks = ((size_t)segs * ny * nz * 32 + 255) / 256;
    if (fin_blocks > (size_t)INT32_MAX) return FC_LBM_ERR_TOO_LARGE;
    const bool vec = nx % 4 == 0 && reinterpret_cast<uintptr_t>(d_solid) % 4 == 0 &&
                     reinterpret_cast<uintptr_t>(d_sdf) % 16 == 0;
    if (vec)
        k_vox_finalize<true><<<(unsigned)fin_blocks, 256, 0, s>>>(d_solid, d_sdf, g, slot, tile_reached, row_reached,
                                                                  segs);
    else
        k_vox_finalize<false><<<(unsigned)fin_blocks, 256, 0, s>>>(d_solid, d_sdf, g, slot, tile_reached, row_reached,
                                                                   segs);
    VX_TRY(cudaGetLastError());
    VX_TRY(cudaMemcpyAsync(&ans->st, d_st, sizeof(st), cudaMemcpyDeviceToHost, s));
    VX_RC(wait_on(s));
    return ans->st.err ? FC_LBM_ERR_CUDA : FC_LBM_OK;
}

bool finite3(const float* v) { return std::isfinite(v[0]) && std::isfinite(v[1]) && std::isfinite(v[2]); }

}  // namespace

extern "C" {

FC_LBM_API int fc_lbm_voxel_grid(const float* positions, size_t vertex_count, const fc_voxel_params* params,
                                 int32_t memory, int32_t dims[3], float* cell_size, float origin[3], void* stream) {
    if (!positions || !params || !dims || !cell_size || !origin) return FC_LBM_ERR_INVALID_ARG;
    if (memory != FC_MEMORY_HOST && memory != FC_MEMORY_DEVICE) return FC_LBM_ERR_INVALID_ARG;
    if (vertex_count == 0 || vertex_count >= 0xffffffffu) return FC_LBM_ERR_INVALID_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    GridOut out{};
    int rc;
    {
        Scratch sc(s);
        const float* d_pos = positions;
        if (memory == FC_MEMORY_HOST) {
            float* p = nullptr;
            VX_TRY(sc.get(&p, 12 * vertex_count));
            VX_TRY(cudaMemcpyAsync(p, positions, 12 * vertex_count, cudaMemcpyHostToDevice, s));
            d_pos = p;
        }
        rc = grid_on_device(d_pos, vertex_count, params, s, sc, &out);
    }
    if (rc != FC_LBM_OK) return rc;
    for (int k = 0; k < 3; ++k) {
        dims[k] = out.dims[k];
        origin[k] = out.origin[k];
    }
    *cell_size = out.cell;
    return FC_LBM_OK;
}

FC_LBM_API int fc_lbm_voxelize(const float* positions, size_t vertex_count, const uint32_t* indices,
                               size_t index_count, const int32_t dims[3], float cell_size, const float origin[3],
                               int32_t memory, uint8_t* solid, float* signed_distance, void* stream) {
    if (!dims || !origin || !solid || !signed_distance) return FC_LBM_ERR_INVALID_ARG;
    if (memory != FC_MEMORY_HOST && memory != FC_MEMORY_DEVICE) return FC_LBM_ERR_INVALID_ARG;
    if (dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0) return FC_LBM_ERR_INVALID_ARG;
    if (!(cell_size > 0.0f) || !std::isfinite(cell_size) || !finite3(origin)) return FC_LBM_ERR_INVALID_ARG;
    if (index_count >= 3 && (!positions || !indices || vertex_count == 0)) return FC_LBM_ERR_INVALID_ARG;
    if (vertex_count >= 0xffffffffu || index_count / 3 >= 0xffffffffu) return FC_LBM_ERR_TOO_LARGE;
    const size_t n = (size_t)dims[0] * dims[1] * dims[2];
    if (n >= 0xffffffffull) return FC_LBM_ERR_TOO_LARGE;  // tiles and cells count below 2^32
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Scratch sc(s);
    const float* d_pos = positions;
    const uint32_t* d_idx = indices;
    uint8_t* d_solid = solid;
    float* d_sdf = signed_distance;
    const size_t ni = index_count - index_count % 3;
    if (memory == FC_MEMORY_HOST) {
        if (ni > 0) {
            float* p = nullptr;
            uint32_t* q = nullptr;
            VX_TRY(sc.get(&p, 12 * vertex_count));
            VX_TRY(sc.get(&q, 4 * ni));
            VX_TRY(cudaMemcpyAsync(p, positions, 12 * vertex_count, cudaMemcpyHostToDevice, s));
            VX_TRY(cudaMemcpyAsync(q, indices, 4 * ni, cudaMemcpyHostToDevice, s));
            d_pos = p;
            d_idx = q;
        }
        VX_TRY(sc.get(&d_solid, n));
        VX_TRY(sc.get(&d_sdf, 4 * n));
    }
    VX_RC(voxelize_on_device(d_pos, vertex_count, d_idx, ni, dims, cell_size, origin, d_solid, d_sdf, s, sc));
    if (memory == FC_MEMORY_HOST) {
        VX_TRY(cudaMemcpyAsync(solid, d_solid, n, cudaMemcpyDeviceToHost, s));
        VX_TRY(cudaMemcpyAsync(signed_distance, d_sdf, 4 * n, cudaMemcpyDeviceToHost, s));
        VX_RC(wait_on(s));
    }
    return FC_LBM_OK;
}

}  // extern "C"
