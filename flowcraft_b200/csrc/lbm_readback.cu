// Readback kernels: macroscopic field, raw populations, and the FP64
// statistics reduction.
//
// The field follows LbmReference::ReadbackField (LbmReference.cpp:475-500):
// fluid cells get (rho, ux, uy, uz) from the current post-collision state;
// solid cells get the momentum-exchange force of their fluid neighbours,
// (|F| / (6 sum w), Fx, Fy, Fz) (LbmReference::SolidCellForce,
// LbmReference.cpp:127-148), with the same Bouzidi reconstruction the step
// uses. Only the moments are computed — the step never writes a
// 16-byte-per-cell macro buffer the way the reference's GPU kernel does
// (shaders/lbm_step.comp.glsl:360-363), which saves 16 B of HBM traffic per
// cell update.
#include <algorithm>
#include <mutex>

#include "aa.cuh"
#include "collide.cuh"
#include "collide2.cuh"
#include "fc_lbm.h"
#include "lbm_internal.h"
#include "storage.cuh"

namespace fc {

__device__ __forceinline__ bool inb(const Geom& g, int x, int y, int z) {
    return x >= 0 && y >= 0 && z >= 0 && x < g.nx && y < g.ny && z < g.nz;
}
__device__ __forceinline__ size_t cidx(const Geom& g, int x, int y, int z) { return ((size_t)z * g.ny + y) * g.nx + x; }

// Post-collision population P of cell c = (x, y, z) under `layout` (aa.cuh).
template <int Q, class S, int P>
__device__ __forceinline__ float load_at(const typename S::T* __restrict__ f, size_t c, int x, int y, int z,
                                         const Geom& g, int layout) {
    return S::dec(S::ld(f + pop_slot<Q, P>(c, x, y, z, g, layout)), Lattice<Q>::w(P));
}

// InterpolatedBounceBack for fluid node a (cell ca) whose direction-i
// upstream neighbour s (cell cs) is solid (LbmReference.cpp:100-122).
template <int Q, class S, int I>
__device__ float bounce_rt(const typename S::T* __restrict__ f, const uint8_t* __restrict__ solid,
                           const float* __restrict__ sdf, const Geom& g, int ax, int ay, int az, size_t ca,
                           size_t cs, int layout) {
    using L = Lattice<Q>;
    constexpr int op = L::opp(I);
    const float plain = load_at<Q, S, op>(f, ca, ax, ay, az, g, layout);
    if (!sdf) return plain;
    const float phi_f = sdf[ca], phi_s = sdf[cs];
    if (!isfinite(phi_f) || !isfinite(phi_s)) return plain;
    const float denom = phi_f - phi_s;
    if (!(denom > 1e-4f)) return plain;
    float q = phi_f / denom;
    q = (q < 0.0f) ? 0.0f : ((1.0f < q) ? 1.0f : q);
    if (q < 0.5f) {
        const int fx = ax + L::ex(I), fy = ay + L::ey(I), fz = az + L::ez(I);
        if (!inb(g, fx, fy, fz) || solid[cidx(g, fx, fy, fz)]) return plain;
        return 2.0f * q * plain + (1.0f - 2.0f * q) * load_at<Q, S, op>(f, cidx(g, fx, fy, fz), fx, fy, fz, g, layout);
    }
    const float inv = 1.0f / (2.0f * q);
    return inv * plain + (1.0f - inv) * load_at<Q, S, I>(f, ca, ax, ay, az, g, layout);
}

// The directions to a solid cell's fluid neighbours, their flags loaded
// together. Most solid cells of a body have none and carry no force.
template <int Q>
__device__ __forceinline__ unsigned open_links(const uint8_t* __restrict__ solid, const Geom& g, int x, int y, int z) {
    using L = Lattice<Q>;
    unsigned open = 0;
    static_for<1, Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        const int ax = x + L::ex(i), ay = y + L::ey(i), az = z + L::ez(i);
        if (inb(g, ax, ay, az) && !solid[cidx(g, ax, ay, az)]) open |= 1u << i;
    });
    return open;
}

template <int Q, class S>
__device__ float4 solid_force(const typename S::T* __restrict__ f, const uint8_t* __restrict__ solid,
                              const float* __restrict__ sdf, const Geom& g, int x, int y, int z, size_t c,
                              int layout) {
    using L = Lattice<Q>;
    float fx = 0.0f, fy = 0.0f, fz = 0.0f, ws = 0.0f;
    const unsigned open = open_links<Q>(solid, g, x, y, z);
    if (!open) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    static_for<1, Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        constexpr int X = L::ex(i), Y = L::ey(i), Z = L::ez(i);
        if (!((open >> i) & 1u)) return;
        const int ax = x + X, ay = y + Y, az = z + Z;
        const size_t ca = cidx(g, ax, ay, az);
        const float plain = load_at<Q, S, L::opp(i)>(f, ca, ax, ay, az, g, layout);
        const float bounced = bounce_rt<Q, S, i>(f, solid, sdf, g, ax, ay, az, ca, c, layout);
        const float dp = (plain + bounced) - 2.0f * L::w(i);
        if constexpr (X > 0) fx = fx - dp;
        if constexpr (X < 0) fx = fx + dp;
        if constexpr (Y > 0) fy = fy - dp;
        if constexpr (Y < 0) fy = fy + dp;
        if constexpr (Z > 0) fz = fz - dp;
        if constexpr (Z < 0) fz = fz + dp;
        ws = ws + L::w(i);
    });
    const float mag = sqrtf((fx * fx + fy * fy) + fz * fz);
    const float stress = (ws > 0.0f) ? (mag / (6.0f * ws)) : 0.0f;
    return make_float4(stress, fx, fy, fz);
}

template <int Q, class S>
__device__ __forceinline__ float4 fluid_moments(const typename S::T* __restrict__ f, const Geom& g, size_t c, int x,
                                                int y, int z, int layout) {
    float p[Q];
    static_for<0, Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        p[i] = load_at<Q, S, i>(f, c, x, y, z, g, layout);
    });
    float rho, ux, uy, uz;
    moments<Q>(p, rho, ux, uy, uz);
    return make_float4(rho, ux, uy, uz);
}

// The same for a cell off every face in the layout an in-place even step
// leaves: no neighbour is tested for being inside.
template <int Q, class S>
__device__ __forceinline__ float4 inner_moments(const typename S::T* __restrict__ f, const Geom& g, size_t c) {
    float p[Q];
    static_for<0, Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        p[i] = S::dec(S::ld(f + (size_t)i * g.ps + (size_t)((long long)c + aa_link<Q>(i, g))), Lattice<Q>::w(i));
    });
    float rho, ux, uy, uz;
    moments<Q>(p, rho, ux, uy, uz);
    return make_float4(rho, ux, uy, uz);
}

template <int Q, class S, int Lay>
__global__ void __launch_bounds__(256) k_field(const typename S::T* __restrict__ f, const uint8_t* __restrict__ solid,
                                                const float* __restrict__ sdf, Geom g, size_t cell0, size_t cells,
                                                float4* __restrict__ out, int layout_in) {
    // the layout is a compile-time constant, so every slot folds to its
    // formula (plane * n + c for plane-major states)
    const int layout = Lay;
    (void)layout_in;
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= cells) return;
    const size_t c = cell0 + k;
    const int z = (int)(c / (size_t)g.nxy);
    const size_t rem = c - (size_t)z * g.nxy;
    const int y = (int)(rem / g.nx);
    const int x = (int)(rem - (size_t)y * g.nx);
    out[k] = solid[c] ? solid_force<Q, S>(f, solid, sdf, g, x, y, z, c, layout)
                      : fluid_moments<Q, S>(f, g, c, x, y, z, layout);
}

// ProbeSliceHealth's verdict on the device (LbmSolver.cpp:699-716): the
// field values k_field gives for cells [cell0, cell0 + cells), then every
// value finite, and for fluid cells rho > 0 and |u|^2 <= 4 (the same float
// operations as the host check). Any failing cell sets *flag.
template <int Q, class S, int Lay>
__global__ void __launch_bounds__(256) k_probe_health(const typename S::T* __restrict__ f,
                                                       const uint8_t* __restrict__ solid, const float* __restrict__ sdf,
                                                       Geom g, size_t cell0, size_t cells, int* __restrict__ flag,
                                                       int layout_in) {
    const int layout = Lay;
    (void)layout_in;
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool bad = false;
    if (k < cells) {
        const size_t c = cell0 + k;
        const int z = (int)(c / (size_t)g.nxy);
        const size_t rem = c - (size_t)z * g.nxy;
        const int y = (int)(rem / g.nx);
        const int x = (int)(rem - (size_t)y * g.nx);
        const bool sc = solid[c] != 0;
        const float4 v = sc ? solid_force<Q, S>(f, solid, sdf, g, x, y, z, c, layout)
                            : fluid_moments<Q, S>(f, g, c, x, y, z, layout);
        bad = !isfinite(v.x) || !isfinite(v.y) || !isfinite(v.z) || !isfinite(v.w);
        if (!bad && !sc) {
            const float sp2 = v.y * v.y + v.z * v.z + v.w * v.w;
            bad = v.x <= 0.0f || sp2 > 4.0f;
        }
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

template <int Q, class S, int Lay>
__global__ void k_pops_out(const typename S::T* __restrict__ f, const uint8_t* __restrict__ solid,
                           int solid_is_weight, Geom g, size_t cell0, size_t cells, float* __restrict__ out,
                           int layout_in) {
    // the layout is a compile-time constant, so every slot folds to its
    // formula (plane * n + c for plane-major states)
    const int layout = Lay;
    (void)layout_in;
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= cells) return;
    const size_t c = cell0 + k;
    int x = 0, y = 0, z = 0;
    if (layout != kLayoutPlanes) {  // the plane-major slot needs no coordinates
        z = (int)(c / (size_t)g.nxy);
        const size_t rem = c - (size_t)z * g.nxy;
        y = (int)(rem / g.nx);
        x = (int)(rem - (size_t)y * g.nx);
    }
    const bool sw = solid_is_weight && solid[c];
    static_for<0, Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        out[(size_t)i * cells + k] = sw ? Lattice<Q>::w(i) : load_at<Q, S, i>(f, c, x, y, z, g, layout);
    });
}

template <int Q, class S, int Lay>
__global__ void k_pops_in(typename S::T* __restrict__ f, Geom g, size_t cell0, size_t cells,
                          const float* __restrict__ in, int layout_in) {
    // the layout is a compile-time constant, so every slot folds to its
    // formula (plane * n + c for plane-major states)
    const int layout = Lay;
    (void)layout_in;
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= cells) return;
    const size_t c = cell0 + k;
    int x = 0, y = 0, z = 0;
    if (layout != kLayoutPlanes) {
        z = (int)(c / (size_t)g.nxy);
        const size_t rem = c - (size_t)z * g.nxy;
        y = (int)(rem / g.nx);
        x = (int)(rem - (size_t)y * g.nx);
    }
    static_for<0, Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        f[pop_slot<Q, i>(c, x, y, z, g, layout)] = S::enc(in[(size_t)i * cells + k], Lattice<Q>::w(i));
    });
}

// ---- statistics (LbmReference::ComputeStats, LbmReference.cpp:502-585) ----
// Slots: 0 density sum, 1 speed sum, 2 mass, 3..5 force sums, 6 fluid count,
// 7 min density, 8 max density, 9 max speed, 10 max stress, 11 NaN flag.
constexpr int kStatsThreads = 256;

struct StatAcc {
    double dsum = 0.0, ssum = 0.0, fx = 0.0, fy = 0.0, fz = 0.0, count = 0.0;
    float mn = 1e30f, mx = -1e30f, vmax = 0.0f, smax = 0.0f;
    int nan = 0;
};

__device__ __forceinline__ void stat_merge(StatAcc& a, const StatAcc& b) {
    a.dsum += b.dsum;
    a.ssum += b.ssum;
    a.fx += b.fx;
    a.fy += b.fy;
    a.fz += b.fz;
    a.count += b.count;
    a.mn = fminf(a.mn, b.mn);
    a.mx = fmaxf(a.mx, b.mx);
    a.vmax = fmaxf(a.vmax, b.vmax);
    a.smax = fmaxf(a.smax, b.smax);
    a.nan |= b.nan;
}

__device__ __forceinline__ void stat_block_reduce(StatAcc& acc, double* out) {
    __shared__ StatAcc sh[kStatsThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        StatAcc b;
        b.dsum = __shfl_down_sync(0xffffffffu, acc.dsum, o);
        b.ssum = __shfl_down_sync(0xffffffffu, acc.ssum, o);
        b.fx = __shfl_down_sync(0xffffffffu, acc.fx, o);
        b.fy = __shfl_down_sync(0xffffffffu, acc.fy, o);
        b.fz = __shfl_down_sync(0xffffffffu, acc.fz, o);
        b.count = __shfl_down_sync(0xffffffffu, acc.count, o);
        b.mn = __shfl_down_sync(0xffffffffu, acc.mn, o);
        b.mx = __shfl_down_sync(0xffffffffu, acc.mx, o);
        b.vmax = __shfl_down_sync(0xffffffffu, acc.vmax, o);
        b.smax = __shfl_down_sync(0xffffffffu, acc.smax, o);
        b.nan = __shfl_down_sync(0xffffffffu, acc.nan, o);
        stat_merge(acc, b);
    }
    if (lane == 0) sh[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        StatAcc t = sh[0];
        for (int w = 1; w < kStatsThreads / 32; ++w) stat_merge(t, sh[w]);
        out[0] = t.dsum;
        out[1] = t.ssum;
        out[2] = t.dsum;  // mass: the reference sums rho over fluid cells
        out[3] = t.fx;
        out[4] = t.fy;
        out[5] = t.fz;
        out[6] = t.count;
        out[7] = t.mn;
        out[8] = t.mx;
        out[9] = t.vmax;
        out[10] = t.smax;
        out[11] = t.nan;
    }
}

// The reductions run over groups of 128 cells, one warp per group, four cells
// per lane: one 4-byte load of solid flags per lane. The solid cells of a
// group are listed in shared memory and shared out over the lanes; those with
// a fluid neighbour, the few that carry a force, collect in a queue of the
// warp and are evaluated 32 at a time, so that the long force code runs with
// full warps instead of in the few lanes that hit one. Lane l holds cells 4l
// .. 4l + 3 of a plane-major group, which lets its populations come four at a
// time, and cells l, l + 32, ... of an in-place one.
constexpr int kGroup = 128;
constexpr int kStatsWarps = kStatsThreads / 32;
// Resident blocks per SM. The grids stop at one wave of them: each block ends
// in a barrier and a reduction. Plane-major k_stats holds four cells per lane
// and takes three blocks (four spill: 444 us against 417; with three only D3Q15
// in 16 bits does, 84 bytes, and 512x256x256 still take 347 us, 438 without
// groups). The in-place ones hold one cell and take four: 512x256x256 after
// an even step, D3Q19 FP16 780 us, D3Q15 663, with three 809 and 705.
constexpr int kAeroPerSm = 2;
constexpr int stats_per_sm(int layout) { return layout == kLayoutPlanes ? 3 : 4; }
constexpr int kMostStatsBlocks = 148 * 4;

__device__ __forceinline__ size_t group_cell(size_t base, int lane, int j, bool planes) {
    return base + (planes ? 4 * lane + j : lane + 32 * j);
}

// The flags of this lane's four cells of a group, a byte each (nonzero:
// solid); cells past the lattice read as fluid. words: `solid` is on a 4-byte
// boundary.
__device__ __forceinline__ uint32_t group_word(const uint8_t* __restrict__ solid, size_t base, size_t n, int lane,
                                               bool planes, bool words) {
    if (planes && words && base + 4 * lane + 4 <= n)
        return __ldg(reinterpret_cast<const uint32_t*>(solid + base + 4 * lane));
    uint32_t w = 0;
    for (int j = 0; j < 4; ++j) {
        const size_t c = group_cell(base, lane, j, planes);
        if (c < n) w |= (uint32_t)solid[c] << (8 * j);
    }
    return w;
}

// Bit j: this lane's j-th cell is solid.
__device__ __forceinline__ unsigned solid_bits(uint32_t w) {
    unsigned b = 0;
    for (int j = 0; j < 4; ++j) b |= ((w >> (8 * j)) & 0xffu) ? 1u << j : 0u;
    return b;
}

// Bit j: this lane's j-th cell lies inside the lattice.
__device__ __forceinline__ unsigned inside_bits(size_t base, size_t n, int lane, bool planes) {
    if (base + kGroup <= n) return 0xfu;
    unsigned b = 0;
    for (int j = 0; j < 4; ++j) b |= group_cell(base, lane, j, planes) < n ? 1u << j : 0u;
    return b;
}

__device__ __forceinline__ void cell_xyz(const Geom& g, size_t c, int& x, int& y, int& z) {
    // cells and layers count below 2^32: 32-bit divisions
    const uint32_t cc = (uint32_t)c, nxy = (uint32_t)g.nxy, zz = cc / nxy, rem = cc - zz * nxy,
                   yy = rem / (uint32_t)g.nx;
    z = (int)zz;
    y = (int)yy;
    x = (int)(rem - yy * (uint32_t)g.nx);
}

// Group of warp w (of W) in its k-th turn, rotated from turn to turn: with a
// plain stride a warp would meet the same part of every row, and a body would
// fall to a few warps.
__device__ __forceinline__ size_t group_base(unsigned w, unsigned W, unsigned k) {
    return ((size_t)k * W + (w + 37u * (k % W)) % W) * kGroup;
}

struct SolidLists {
    uint8_t group[kGroup];   // the group's solid cells, relative to its base
    uint32_t queue[64];      // solid cells with a fluid neighbour, not evaluated yet
};

// every(x, y, z) for each solid cell of the group (bits `sol` of this lane),
// force(cell) for each queued cell once 32 are queued; with `last`, for all.
template <int Q, class Every, class Force>
__device__ __forceinline__ void group_solids(SolidLists& sl, unsigned& queued, size_t base, int lane, bool planes,
                                             unsigned sol, bool last, const uint8_t* __restrict__ solid,
                                             const Geom& g, Every&& every, Force&& force) {
    if (!last && !__any_sync(0xffffffffu, sol != 0u)) return;
    unsigned at = __popc(sol);
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += t;
    }
    const unsigned total = __shfl_sync(0xffffffffu, at, 31);
    at -= __popc(sol);
    for (int j = 0; j < 4; ++j)
        if ((sol >> j) & 1u) sl.group[at++] = (uint8_t)(group_cell(0, lane, j, planes));
    __syncwarp();
#pragma unroll 1
    for (unsigned k = 0; k < total || (last && queued > 0); k += 32) {
        bool open = false;
        size_t c = 0;
        if (k + lane < total) {
            c = base + sl.group[k + lane];
            int x, y, z;
            cell_xyz(g, c, x, y, z);
            every(x, y, z);
            open = open_links<Q>(solid, g, x, y, z) != 0u;
        }
        const unsigned hits = __ballot_sync(0xffffffffu, open);
        if (open) sl.queue[queued + __popc(hits & ((1u << lane) - 1u))] = (uint32_t)c;  // below 32 + 32
        queued += __popc(hits);
        __syncwarp();
        if (queued >= 32 || (last && k + 32 >= total)) {
            if (lane < (int)queued) force((size_t)sl.queue[lane]);
            const uint32_t rest = sl.queue[32 + lane];
            __syncwarp();
            sl.queue[lane] = rest;
            queued -= queued < 32 ? queued : 32;
            __syncwarp();
        }
    }
    __syncwarp();
}

// Four populations of one plane from an address on a four-element boundary,
// as two pairs.
template <class S>
__device__ __forceinline__ void load4(const typename S::T* p, float w, float2& lo, float2& hi) {
    using T2 = typename S::T2;
    if constexpr (S::kBytes == 4) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(p));
        lo = make_float2(q.x, q.y), hi = make_float2(q.z, q.w);
    } else {
        const uint2 q = __ldg(reinterpret_cast<const uint2*>(p));
        // dec: h / 2^8 + w
        lo = fma2(S::raw2(*reinterpret_cast<const T2*>(&q.x)), bc2(kOffsetScaleInv), bc2(w));
        hi = fma2(S::raw2(*reinterpret_cast<const T2*>(&q.y)), bc2(kOffsetScaleInv), bc2(w));
    }
}

// B200, 512x256x256 D3Q19 FP16 with a wing: 501 -> 372 us (one cell per thread,
// 2-byte loads, the force in the lanes that hit a solid cell, before); what is
// left is arithmetic: the IEEE divisions and roots of four cells per lane.
template <int Q, class S, int Lay>
__global__ void __launch_bounds__(kStatsThreads, stats_per_sm(Lay)) k_stats(const typename S::T* __restrict__ f,
                                                         const uint8_t* __restrict__ solid,
                                                         const float* __restrict__ sdf, Geom g,
                                                         double* __restrict__ partials, bool words, bool vec) {
    using L = Lattice<Q>;
    // the layout is a compile-time constant, so every slot folds to its
    // formula (plane * stride + c for plane-major states)
    constexpr bool planes = Lay == kLayoutPlanes;
    __shared__ SolidLists s_lists[kStatsWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned w = blockIdx.x * kStatsWarps + warp, W = gridDim.x * kStatsWarps;
    StatAcc acc;
    unsigned queued = 0;
    bool last = false;
    for (unsigned k = 0; !last; ++k) {  // the last turn has no group: it empties the queue
        last = (size_t)k * W * kGroup >= g.n;
        const size_t base = group_base(w, W, k);
        unsigned fluid = 0, sol = 0;
        if (!last) {
            sol = solid_bits(group_word(solid, base, g.n, lane, planes, words));
            fluid = inside_bits(base, g.n, lane, planes) & ~sol;
        }
        auto add = [&](const float4& m) {
            if (!isfinite(m.x) || !isfinite(m.y) || !isfinite(m.z) || !isfinite(m.w)) {
                acc.nan = 1;
                return;
            }
            const float sp = sqrtf(speed2(m.y, m.z, m.w));
            acc.mn = fminf(acc.mn, m.x);
            acc.mx = fmaxf(acc.mx, m.x);
            acc.vmax = fmaxf(acc.vmax, sp);
            acc.dsum += (double)m.x;
            acc.ssum += (double)sp;
            acc.count += 1.0;
        };
        if constexpr (!planes) {
            // One cell at a time, since four in flight spill, and without the
            // tests for the faces where none is near: 1024x512x512 after an even
            // step, D3Q15 FP16 9.1 -> 4.6 ms, D3Q19 FP32 9.4 -> 5.2.
#pragma unroll 1
            for (int j = 0; j < 4; ++j) {
                if (!((fluid >> j) & 1u)) continue;
                const size_t c = group_cell(base, lane, j, planes);
                int x, y, z;
                cell_xyz(g, c, x, y, z);
                const bool inner = x > 0 && y > 0 && z > 0 && x < g.nx - 1 && y < g.ny - 1 && z < g.nz - 1;
                add(Lay == kLayoutAAEven && inner ? inner_moments<Q, S>(f, g, c)
                                                  : fluid_moments<Q, S>(f, g, c, x, y, z, Lay));
            }
        } else {
            float4 m[4];
            if (vec && base + kGroup <= g.n) {  // moments<Q> of four cells
                if (fluid) {
                    const float2 zero = bc2(0.0f);
                    float2 r[2] = {zero, zero}, a[2] = {zero, zero}, b[2] = {zero, zero}, c[2] = {zero, zero};
                    static_for<0, Q>([&](auto I) {
                        constexpr int i = decltype(I)::value;
                        constexpr int X = L::ex(i), Y = L::ey(i), Z = L::ez(i);
                        float2 v[2];
                        load4<S>(f + (size_t)i * g.ps + base + 4 * lane, L::w(i), v[0], v[1]);
                        for (int j = 0; j < 2; ++j) {
                            r[j] = add2(r[j], v[j]);
                            if constexpr (X > 0) a[j] = add2(a[j], v[j]);
                            if constexpr (X < 0) a[j] = sub2(a[j], v[j]);
                            if constexpr (Y > 0) b[j] = add2(b[j], v[j]);
                            if constexpr (Y < 0) b[j] = sub2(b[j], v[j]);
                            if constexpr (Z > 0) c[j] = add2(c[j], v[j]);
                            if constexpr (Z < 0) c[j] = sub2(c[j], v[j]);
                        }
                    });
                    for (int j = 0; j < 2; ++j) {
                        if (r[j].x > 1e-6f) a[j].x /= r[j].x, b[j].x /= r[j].x, c[j].x /= r[j].x;
                        if (r[j].y > 1e-6f) a[j].y /= r[j].y, b[j].y /= r[j].y, c[j].y /= r[j].y;
                        m[2 * j] = make_float4(r[j].x, a[j].x, b[j].x, c[j].x);
                        m[2 * j + 1] = make_float4(r[j].y, a[j].y, b[j].y, c[j].y);
                    }
                }
            } else {
                for (int j = 0; j < 4; ++j)
                    if ((fluid >> j) & 1u) m[j] = fluid_moments<Q, S>(f, g, group_cell(base, lane, j, planes), 0, 0, 0, Lay);
            }
            for (int j = 0; j < 4; ++j)
                if ((fluid >> j) & 1u) add(m[j]);
        }
        group_solids<Q>(s_lists[warp], queued, base, lane, planes, sol, last, solid, g, [](int, int, int) {},
                        [&](size_t c) {
            int x, y, z;
            cell_xyz(g, c, x, y, z);
            const float4 v = solid_force<Q, S>(f, solid, sdf, g, x, y, z, c, Lay);
            if (isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w)) {
                acc.fx += (double)v.y;
                acc.fy += (double)v.z;
                acc.fz += (double)v.w;
                acc.smax = fmaxf(acc.smax, v.x);
            }
        });
    }
    stat_block_reduce(acc, partials + (size_t)blockIdx.x * kStatsSlots);
}

__global__ void __launch_bounds__(kStatsThreads) k_stats_final(const double* __restrict__ partials, int blocks,
                                                               double* __restrict__ result) {
    StatAcc acc;
    for (int b = threadIdx.x; b < blocks; b += blockDim.x) {
        const double* p = partials + (size_t)b * kStatsSlots;
        StatAcc t;
        t.dsum = p[0];
        t.ssum = p[1];
        t.fx = p[3];
        t.fy = p[4];
        t.fz = p[5];
        t.count = p[6];
        t.mn = (float)p[7];
        t.mx = (float)p[8];
        t.vmax = (float)p[9];
        t.smax = (float)p[10];
        t.nan = p[11] != 0.0;
        stat_merge(acc, t);
    }
    stat_block_reduce(acc, result);
}

// ---- aerodynamic forces (FieldOverlay::ComputeAerodynamicForces, FieldOverlay.cpp:469-621) ----
// Slots: 0-2 force sums, 3 lift weight sum, 4-6 lift-weighted position sums,
// 7 force weight sum, 8-10 force-weighted sums, 11-13 geometric position sums,
// 14 solid count, 15 max solid z, 16 min loaded stress, 17 max loaded stress,
// 18 NaN flag. All sums are FP64; a solid cell whose field entry is not finite
// only raises the flag (the reference skips it after counting its position).
enum AeroSlot { kAfx = 0, kAlw = 3, kAlwx = 4, kAfw = 7, kAfwx = 8, kAgx = 11, kAcount = 14, kAmaxz = 15,
                kAlo = 16, kAhi = 17, kAnan = 18 };

__device__ __forceinline__ void aero_init(double* a) {
    for (int k = 0; k < kAeroSlots; ++k) a[k] = 0.0;
    a[kAmaxz] = -1.0;
    a[kAlo] = 1e30;
    a[kAhi] = -1e30;
}

__device__ __forceinline__ void aero_merge(double* a, const double* b) {
    for (int k = 0; k <= kAcount; ++k) a[k] += b[k];
    a[kAmaxz] = fmax(a[kAmaxz], b[kAmaxz]);
    a[kAlo] = fmin(a[kAlo], b[kAlo]);
    a[kAhi] = fmax(a[kAhi], b[kAhi]);
    a[kAnan] = fmax(a[kAnan], b[kAnan]);
}

// Block reduction in a fixed order (shuffle tree, then warps in order).
__device__ void aero_block_reduce(double* a, double* out) {
    __shared__ double sh[kStatsThreads / 32][kAeroSlots];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        double b[kAeroSlots];
        for (int k = 0; k < kAeroSlots; ++k) b[k] = __shfl_down_sync(0xffffffffu, a[k], o);
        aero_merge(a, b);
    }
    if (lane == 0)
        for (int k = 0; k < kAeroSlots; ++k) sh[warp][k] = a[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kStatsThreads / 32; ++w) aero_merge(a, sh[w]);
        for (int k = 0; k < kAeroSlots; ++k) out[k] = a[k];
    }
}

// B200, 512x256x256 D3Q19 FP16 with a wing: 392 -> 112 us, and the final kernel 75
// -> 13 us (one flag per thread and load, the force in the lanes that hit a
// solid cell, one thread per column of the final patch, before).
template <int Q, class S, int Lay>
__global__ void __launch_bounds__(kStatsThreads) k_aero(const typename S::T* __restrict__ f,
                                                        const uint8_t* __restrict__ solid,
                                                        const float* __restrict__ sdf, Geom g, float cs, float ox,
                                                        float oy, float oz, double* __restrict__ partials,
                                                        bool words) {
    // the layout is a compile-time constant, as in k_stats
    constexpr bool planes = Lay == kLayoutPlanes;
    __shared__ SolidLists s_lists[kStatsWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned w = blockIdx.x * kStatsWarps + warp, W = gridDim.x * kStatsWarps;
    double a[kAeroSlots];
    aero_init(a);
    unsigned queued = 0;
    bool last = false, any = false;
    // the flags of several groups in one trip to memory: a pass over a lattice
    // is mostly flags without a solid cell
    constexpr int kAhead = 4;
    unsigned rot = w;  // group_base's rotation, stepped
    size_t from[kAhead];
    for (unsigned k0 = 0; !last; k0 += kAhead) {  // the last turn has no groups: it empties the queue
        last = (size_t)k0 * W * kGroup >= g.n;
        uint32_t flags[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const unsigned r = rot + 37u * k;
            from[k] = ((size_t)(k0 + k) * W + (r < W ? r : r % W)) * kGroup;
            flags[k] = last ? 0u : group_word(solid, from[k], g.n, lane, planes, words);
        }
        rot = (rot + 37u * kAhead) % W;
        if (!last && !__any_sync(0xffffffffu, (flags[0] | flags[1] | flags[2] | flags[3]) != 0u)) continue;
        any = any || !last;
        // (one copy of the force code: the group is picked at run time)
#pragma unroll 1
        for (int k = 0; k < kAhead; ++k) {
            const unsigned bits = solid_bits(k == 0 ? flags[0] : (k == 1 ? flags[1] : (k == 2 ? flags[2] : flags[3])));
            const size_t base = k == 0 ? from[0] : (k == 1 ? from[1] : (k == 2 ? from[2] : from[3]));
            auto every = [&](int x, int y, int z) {
                // VoxelGrid::CellCenter (VoxelGrid.h:53-55) in float
                a[kAgx] += (double)(ox + ((float)y + 0.5f) * cs);
                a[kAgx + 1] += (double)(oy + ((float)x + 0.5f) * cs);
                a[kAgx + 2] += (double)(oz + ((float)z + 0.5f) * cs);
                a[kAcount] += 1.0;
                a[kAmaxz] = fmax(a[kAmaxz], (double)z);
            };
            group_solids<Q>(s_lists[warp], queued, base, lane, planes, bits, last, solid, g, every,
                            [&](size_t c) {
                int x, y, z;
                cell_xyz(g, c, x, y, z);
                const float px = ox + ((float)y + 0.5f) * cs;
                const float py = oy + ((float)x + 0.5f) * cs;
                const float pz = oz + ((float)z + 0.5f) * cs;
                const float4 v = solid_force<Q, S>(f, solid, sdf, g, x, y, z, c, Lay);
                if (!isfinite(v.x) || !isfinite(v.y) || !isfinite(v.z) || !isfinite(v.w)) {
                    a[kAnan] = 1.0;
                    return;
                }
                a[kAfx] += (double)v.y;
                a[kAfx + 1] += (double)v.z;
                a[kAfx + 2] += (double)v.w;
                const double wl = fabs((double)v.w);
                a[kAlw] += wl;
                a[kAlwx] += wl * px;
                a[kAlwx + 1] += wl * py;
                a[kAlwx + 2] += wl * pz;
                const double wf = sqrt((double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w);
                a[kAfw] += wf;
                a[kAfwx] += wf * px;
                a[kAfwx + 1] += wf * py;
                a[kAfwx + 2] += wf * pz;
                if (v.x > 0.0f) {
                    a[kAlo] = fmin(a[kAlo], (double)v.x);
                    a[kAhi] = fmax(a[kAhi], (double)v.x);
                }
            });
        }
    }
    // most blocks meet no solid cell: their partials are the initial values
    if (__syncthreads_or(any))
        aero_block_reduce(a, partials + (size_t)blockIdx.x * kAeroSlots);
    else if (threadIdx.x < 1)
        for (int k = 0; k < kAeroSlots; ++k) partials[(size_t)blockIdx.x * kAeroSlots + k] = a[k];
}

// Reduces the partials, then computes the centre of pressure and the lift
// arrow's base from a 5x5 patch of columns around it (FieldOverlay.cpp:
// 580-618): the highest solid cell of the patch, all its cells over the
// block's threads.
__global__ void __launch_bounds__(kStatsThreads) k_aero_final(const double* __restrict__ partials, int blocks,
                                                              const uint8_t* __restrict__ solid, Geom g, float cs,
                                                              float ox, float oy, float oz,
                                                              double* __restrict__ result) {
    __shared__ double tot[kAeroSlots];
    __shared__ float cp[3];
    __shared__ int col_top;
    double a[kAeroSlots];
    aero_init(a);
    for (int b = threadIdx.x; b < blocks; b += blockDim.x) aero_merge(a, partials + (size_t)b * kAeroSlots);
    aero_block_reduce(a, tot);
    if (threadIdx.x == 0) {
        col_top = -1;
        const double lw = tot[kAlw], fw = tot[kAfw], count = tot[kAcount];
        float c0 = 0.0f, c1 = 0.0f, c2 = 0.0f;
        if (lw > 1e-9) {
            c0 = (float)(tot[kAlwx] / lw), c1 = (float)(tot[kAlwx + 1] / lw), c2 = (float)(tot[kAlwx + 2] / lw);
        } else if (fw > 1e-9) {
            c0 = (float)(tot[kAfwx] / fw), c1 = (float)(tot[kAfwx + 1] / fw), c2 = (float)(tot[kAfwx + 2] / fw);
        } else if (count > 0.0) {
            const double inv = 1.0 / count;
            c0 = (float)(tot[kAgx] * inv), c1 = (float)(tot[kAgx + 1] * inv), c2 = (float)(tot[kAgx + 2] * inv);
        }
        cp[0] = c0, cp[1] = c1, cp[2] = c2;
    }
    __syncthreads();
    {
        const int nxm = g.nx - 1 > 0 ? g.nx - 1 : 0, nym = g.ny - 1 > 0 ? g.ny - 1 : 0;
        int gx = (int)floorf((cp[1] - oy) / cs), gy = (int)floorf((cp[0] - ox) / cs);
        gx = gx < 0 ? 0 : (gx > nxm ? nxm : gx);
        gy = gy < 0 ? 0 : (gy > nym ? nym : gy);
        int top = -1;
#pragma unroll 8
        for (int k = threadIdx.x; k < 25 * g.nz; k += kStatsThreads) {
            const int z = k / 25, col = k - 25 * z;
            int x = gx + col % 5 - 2, y = gy + col / 5 - 2;
            x = x < 0 ? 0 : (x > nxm ? nxm : x);
            y = y < 0 ? 0 : (y > nym ? nym : y);
            if (solid[((size_t)z * g.ny + y) * g.nx + x]) top = z;
        }
        if (top >= 0) atomicMax(&col_top, top);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int maxz = (int)tot[kAmaxz];
        const int eff = col_top >= 0 ? col_top : (maxz > 0 ? maxz : 0);
        float lo = (float)tot[kAlo], hi = (float)tot[kAhi];
        if (lo > hi) {
            lo = 0.0f;
            hi = 1e-6f;
        } else {
            lo = 0.0f;
            if (!(hi > lo)) hi = lo + 1e-6f;
        }
        result[0] = tot[kAfx];
        result[1] = tot[kAfx + 1];
        result[2] = tot[kAfx + 2];
        result[3] = tot[kAlw];
        result[4] = tot[kAfw];
        result[5] = tot[kAcount];
        result[6] = lo;
        result[7] = hi;
        result[8] = tot[kAnan];
        result[9] = cp[0];
        result[10] = cp[1];
        result[11] = cp[2];
        result[12] = cp[0];
        result[13] = cp[1];
        result[14] = oz + ((float)eff + 1.0f) * cs;
        result[15] = (double)maxz;
    }
}

static bool words_of(const uint8_t* solid) { return reinterpret_cast<uintptr_t>(solid) % 4 == 0; }

int stats_blocks(const Geom& g) {
    const size_t want = (g.n + kStatsThreads * 8 - 1) / (kStatsThreads * 8);
    return (int)std::min<size_t>(std::max<size_t>(want, 1), kMostStatsBlocks);
}

// Launches KERNEL<Q, S, layout> for the run-time `layout` (PopLayout).
#define FC_LAYOUT_LAUNCH(KERNEL, GRID, BLOCK, ...)                                        \
    do {                                                                                  \
        if (layout == kLayoutAAEven)                                                      \
            KERNEL<Q, S, kLayoutAAEven><<<GRID, BLOCK, 0, s>>>(__VA_ARGS__);              \
        else if (layout == kLayoutAAOdd)                                                  \
            KERNEL<Q, S, kLayoutAAOdd><<<GRID, BLOCK, 0, s>>>(__VA_ARGS__);               \
        else                                                                              \
            KERNEL<Q, S, kLayoutPlanes><<<GRID, BLOCK, 0, s>>>(__VA_ARGS__);              \
    } while (0)

template <int Q, class S>
static cudaError_t field_t(const void* f, const uint8_t* solid, const float* sdf, const Geom& g, size_t cell0,
                           size_t cells, float* out, int layout, cudaStream_t s) {
    if (cells == 0) return cudaSuccess;
    FC_LAYOUT_LAUNCH(k_field, (unsigned)((cells + 255) / 256), 256, (const typename S::T*)f, solid, sdf, g, cell0,
                     cells, (float4*)out, layout);
    return cudaGetLastError();
}

template <int Q, class S>
static cudaError_t probe_health_t(const void* f, const uint8_t* solid, const float* sdf, const Geom& g, size_t cell0,
                                  size_t cells, int* flag, int layout, cudaStream_t s) {
    if (cells == 0) return cudaSuccess;
    FC_LAYOUT_LAUNCH(k_probe_health, (unsigned)((cells + 255) / 256), 256, (const typename S::T*)f, solid, sdf, g,
                     cell0, cells, flag, layout);
    return cudaGetLastError();
}

template <int Q, class S>
static cudaError_t pops_out_t(const void* f, const uint8_t* solid, int sw, const Geom& g, size_t cell0, size_t cells,
                              float* out, int layout, cudaStream_t s) {
    if (cells == 0) return cudaSuccess;
    FC_LAYOUT_LAUNCH(k_pops_out, (unsigned)((cells + 255) / 256), 256, (const typename S::T*)f, solid, sw, g, cell0,
                     cells, out, layout);
    return cudaGetLastError();
}

template <int Q, class S>
static cudaError_t pops_in_t(void* f, const Geom& g, size_t cell0, size_t cells, const float* in, int layout,
                             cudaStream_t s) {
    if (cells == 0) return cudaSuccess;
    FC_LAYOUT_LAUNCH(k_pops_in, (unsigned)((cells + 255) / 256), 256, (typename S::T*)f, g, cell0, cells, in, layout);
    return cudaGetLastError();
}

template <int Q, class S>
static cudaError_t stats_t(const void* f, const uint8_t* solid, const float* sdf, const Geom& g, double* partials,
                           int blocks, double* result, int layout, cudaStream_t s) {
    // four populations at a time where every plane and cell group starts on
    // such a boundary
    blocks = std::min(blocks, stats_per_sm(layout) * 148);
    const bool vec = g.ps % 4 == 0 && reinterpret_cast<uintptr_t>(f) % (4 * S::kBytes) == 0;
    FC_LAYOUT_LAUNCH(k_stats, blocks, kStatsThreads, (const typename S::T*)f, solid, sdf, g, partials, words_of(solid),
                     vec);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_stats_final<<<1, kStatsThreads, 0, s>>>(partials, blocks, result);
    return cudaGetLastError();
}

#define FC_DISPATCH(q, storage, FN, ...)                               \
    do {                                                               \
        if ((q) == 19) {                                               \
            if ((storage) == 0) return FN<19, StoreF32>(__VA_ARGS__);  \
            if ((storage) == 1) return FN<19, StoreF16>(__VA_ARGS__);  \
            if ((storage) == 2) return FN<19, StoreBF16>(__VA_ARGS__); \
        } else if ((q) == 15) {                                        \
            if ((storage) == 0) return FN<15, StoreF32>(__VA_ARGS__);  \
            if ((storage) == 1) return FN<15, StoreF16>(__VA_ARGS__);  \
            if ((storage) == 2) return FN<15, StoreBF16>(__VA_ARGS__); \
        }                                                              \
        return cudaErrorInvalidValue;                                  \
    } while (0)

cudaError_t launch_field(int q, int storage, const void* f, const uint8_t* solid, const float* sdf, const Geom& g,
                         size_t cell0, size_t cells, float* out, int layout, cudaStream_t s) {
    FC_DISPATCH(q, storage, field_t, f, solid, sdf, g, cell0, cells, out, layout, s);
}

cudaError_t launch_probe_health(int q, int storage, const void* f, const uint8_t* solid, const float* sdf,
                                const Geom& g, size_t cell0, size_t cells, int* flag, int layout, cudaStream_t s) {
    FC_DISPATCH(q, storage, probe_health_t, f, solid, sdf, g, cell0, cells, flag, layout, s);
}

cudaError_t launch_pops_out(int q, int storage, const void* f, const uint8_t* solid, int solid_is_weight,
                            const Geom& g, size_t cell0, size_t cells, float* out, int layout, cudaStream_t s) {
    FC_DISPATCH(q, storage, pops_out_t, f, solid, solid_is_weight, g, cell0, cells, out, layout, s);
}

cudaError_t launch_pops_in(int q, int storage, void* f, const Geom& g, size_t cell0, size_t cells, const float* in,
                           int layout, cudaStream_t s) {
    FC_DISPATCH(q, storage, pops_in_t, f, g, cell0, cells, in, layout, s);
}

cudaError_t launch_stats(int q, int storage, const void* f, const uint8_t* solid, const float* sdf, const Geom& g,
                         double* partials, int blocks, double* result, int layout, cudaStream_t s) {
    FC_DISPATCH(q, storage, stats_t, f, solid, sdf, g, partials, blocks, result, layout, s);
}

template <int Q, class S>
static cudaError_t aero_t(const void* f, const uint8_t* solid, const float* sdf, const Geom& g, float cs, float ox,
                          float oy, float oz, double* partials, int blocks, double* result, int layout,
                          cudaStream_t s) {
    blocks = std::min(blocks, kAeroPerSm * 148);
    FC_LAYOUT_LAUNCH(k_aero, blocks, kStatsThreads, (const typename S::T*)f, solid, sdf, g, cs, ox, oy, oz, partials,
                     words_of(solid));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_aero_final<<<1, kStatsThreads, 0, s>>>(partials, blocks, solid, g, cs, ox, oy, oz, result);
    return cudaGetLastError();
}

cudaError_t launch_aero(int q, int storage, const void* f, const uint8_t* solid, const float* sdf, const Geom& g,
                        float cell_size, float ox, float oy, float oz, double* partials, int blocks, double* result,
                        int layout, cudaStream_t s) {
    FC_DISPATCH(q, storage, aero_t, f, solid, sdf, g, cell_size, ox, oy, oz, partials, blocks, result, layout, s);
}

}  // namespace fc

// ---- statistics without allocation (fc_lbm_stats_noalloc) ----
// The same k_stats / k_stats_final kernels as fc_lbm_readback_stats, with the
// per-block partials in a fixed file-scope device array instead of memory the
// solver allocated: as many blocks' as a launch of either path has at most
// (592 * 12 doubles = 56 KiB). Both paths take the same number of blocks. Lattices are limited
// to 2^29 cells. Each launch writes every slot of the partials it uses before
// the final kernel reads them, so nothing has to be cleared between calls.
//
// The device address of the array is looked up once per device and cached for
// the life of the process. A cudaDeviceReset destroys the module that holds
// the array, so that cached address does not survive a reset; the header
// documents this.
namespace {

static_assert(fc::kStatsSlots == FC_LBM_STATS_SLOTS, "slot count must match the header");

static __device__ __align__(256) double g_noalloc_partials[fc::kMostStatsBlocks * fc::kStatsSlots];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
double* g_noalloc_scratch[kNoAllocMaxDevices] = {};

}  // namespace

extern "C" FC_LBM_API int fc_lbm_stats_noalloc(const void* populations, const uint8_t* solid,
                                               const float* signed_distance, int32_t nx, int32_t ny, int32_t nz,
                                               int32_t model, int32_t storage, double* out_slots, void* stream) {
    if (!populations || !solid || !out_slots) return FC_LBM_ERR_INVALID_ARG;
    if (nx <= 0 || ny <= 0 || nz <= 0) return FC_LBM_ERR_INVALID_ARG;
    if (model != FC_LATTICE_D3Q15 && model != FC_LATTICE_D3Q19) return FC_LBM_ERR_INVALID_ARG;
    if (storage < FC_STORAGE_FP32 || storage > FC_STORAGE_BF16_OFFSET) return FC_LBM_ERR_INVALID_ARG;
    const size_t n = (size_t)nx * (size_t)ny * (size_t)nz;
    if (n > FC_LBM_NOALLOC_MAX_CELLS) return FC_LBM_ERR_TOO_LARGE;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return FC_LBM_ERR_CUDA;
    if (dev >= kNoAllocMaxDevices) return FC_LBM_ERR_UNSUPPORTED;
    double* scratch = nullptr;
    {
        // set-up, once per device, with that device current: the symbol's
        // host-side name is not a device address
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_scratch[dev]) {
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_partials) != cudaSuccess || !p) return FC_LBM_ERR_CUDA;
            g_noalloc_scratch[dev] = static_cast<double*>(p);
        }
        scratch = g_noalloc_scratch[dev];
    }
    fc::Geom g{};
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    g.wpr = (nx + 31) / 32;
    g.nxy = (long long)nx * ny;
    g.n = n;
    g.ps = n;  // the caller's planes: no padding
    const int q = model == FC_LATTICE_D3Q19 ? 19 : 15;
    const cudaError_t e = fc::launch_stats(q, storage, populations, solid, signed_distance, g, scratch,
                                           fc::stats_blocks(g), out_slots, fc::kLayoutPlanes, static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? FC_LBM_OK : FC_LBM_ERR_CUDA;
}
