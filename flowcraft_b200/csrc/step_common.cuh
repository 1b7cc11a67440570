// Pieces shared by the step kernels (lbm_step.cu: ping-pong; lbm_step_aa.cu:
// one set streamed in place).
#pragma once

#include "collide.cuh"
#include "collide2.cuh"
#include "lbm_internal.h"
#include "storage.cuh"

#include <algorithm>
#include <type_traits>

namespace fc {

constexpr int kBulkRows = 8;  // block = 32 x-lanes x 8 rows
constexpr int kBatchChunk = 8;  // consecutive tiles a block of the batch kernel takes at a time

// Chained steps overlap their ends: a step kernel lets the next one of its
// lattice start as soon as its own blocks have all started
// (programmatic dependent launch), and the next one's blocks, on SMs that the
// last wave leaves idle, run up to here: launch, index arithmetic and the
// loads of what no step writes (bulk mask, boundary list). The populations
// wait until the step before is complete. They come by ordinary loads
// (ld_plain): a read-only load asks for data that nothing writes during the
// kernel's life, and here the step before still does at its start (the two
// kinds measured the same, within 1 % from 48x24x24 to 1024x512x512). Passing
// the cell index through the wait makes every population address depend on
// it, so that no load moves ahead of it.
// B200, us per step, with the boundary list in its own kernel and full
// serialization / now: 48x24x24 FP32 14.6 / 6.7, FP16 18.5 / 9.0; 128x64x64
// FP32 27.0 / 19.5, FP16 30.0 / 15.3; 512x256x256 FP16 571 / 554.
__device__ __forceinline__ uint32_t after_previous_step(uint32_t c) {
    asm volatile("griddepcontrol.wait;" : "+r"(c)::"memory");
    return c;
}

// The same for the in-place kernels, whose population loads are ordinary ones
// that stay behind a memory clobber (with the index passed through, the FP32
// kernels spill more and lost 2 % at 512x256x256).
__device__ __forceinline__ void previous_step_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// First thing in a chained kernel. One thread waits whatever its block holds:
// a step is never complete before the one it was chained to, so the wait above
// covers every earlier step too.
__device__ __forceinline__ void step_enter() {
    asm volatile("griddepcontrol.launch_dependents;");
    if ((blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x | threadIdx.y) == 0)
        asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Host: launches a step kernel, chained to the launch before it if asked.
template <class... P, class... A>
cudaError_t launch_step_kernel(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, bool chained, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Blocks of a step launch that take boundary-list entries (BoundarySpan):
// true for those, with the entry of this thread (one past the end for none).
__device__ __forceinline__ bool boundary_block(const BoundarySpan& b, uint32_t& entry) {
    if (blockIdx.z >= b.slabs) return false;
    const size_t block = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    const size_t e = (size_t)b.begin + block * (32 * kBulkRows) + threadIdx.y * 32 + threadIdx.x;
    entry = e < b.end ? (uint32_t)e : b.end;
    return true;
}

// Host: the launches of a step's `layers` layers and the entries of `b`, in
// slabs of gx x gy blocks ahead of the layers: launch(span, layers) enqueues
// one kernel of span.slabs + layers block layers. Normally that is one; a grid
// holds 65535 block layers, so entries that do not fit beside the layers (very
// tall, narrow lattices) go out in launches of their own first.
template <class F>
cudaError_t launch_with_slabs(BoundarySpan b, unsigned gx, unsigned gy, unsigned layers, int* launched, F&& launch) {
    constexpr size_t kMost = 65535;
    const size_t per = (size_t)gx * gy * 32 * kBulkRows;
    for (;;) {
        const size_t slabs = b.end > b.begin ? (b.end - b.begin + per - 1) / per : 0;
        const bool whole = slabs + layers <= kMost;
        if (whole && slabs + layers == 0) return cudaSuccess;
        BoundarySpan part = b;
        part.slabs = (unsigned)(whole ? slabs : std::min(slabs, kMost));
        if (part.slabs * per < b.end - b.begin) part.end = (uint32_t)(b.begin + part.slabs * per);
        const cudaError_t e = launch(part, whole ? layers : 0u);
        if (e != cudaSuccess) return e;
        ++*launched;
        if (whole) return cudaSuccess;
        b.begin = part.end;
        b.chained = false;
    }
}

template <int Q>
__device__ __forceinline__ long long link_offset(int i, const Geom& g) {
    return (long long)Lattice<Q>::ex(i) + (long long)Lattice<Q>::ey(i) * g.nx + (long long)Lattice<Q>::ez(i) * g.nxy;
}

// Source of population i for a fluid cell whose upstream neighbour is off
// the Y and/or Z edge (oy / oz): the free-slip mirror when every wall crossed
// is free-slip, else plain bounce-back (LbmReference.cpp:370-380). Returns the
// plane to read at the cell itself; every candidate has the weight of i.
template <int Q, int I>
__device__ __forceinline__ int edge_plane(bool oy, bool oz, const StepParams& p) {
    const bool mirror = (!oy || p.slip_y) && (!oz || p.slip_z);
    if (!mirror) return Lattice<Q>::opp(I);
    if (oy && oz) return mirror_z<Q>(mirror_y<Q>(I));
    return oy ? mirror_y<Q>(I) : mirror_z<Q>(I);
}

template <int Q, class S>
__device__ __forceinline__ float load_plane(const typename S::T* f, int plane, size_t n, size_t cell, float w) {
    return S::dec(ld_plain<S>(f + (size_t)plane * n + cell), w);
}

// Both cells of a pair through the collision the storage format uses;
// returns a two-bit divergence mask (bit 0: cell A, bit 1: cell B).
template <int Q, class S>
__device__ __forceinline__ unsigned collide_pair(float2 (&v)[Q], float tau, float cs) {
    if constexpr (S::kExact) {  // bit-exact path: the scalar reference-order collision per cell
        float a[Q], b[Q];
        static_for<0, Q>([&](auto I) {
            constexpr int i = decltype(I)::value;
            a[i] = v[i].x;
            b[i] = v[i].y;
        });
        const unsigned bad = (collide_regularized<Q>(a, tau, cs) ? 1u : 0u) | (collide_regularized<Q>(b, tau, cs) ? 2u : 0u);
        static_for<0, Q>([&](auto I) {
            constexpr int i = decltype(I)::value;
            v[i] = make_float2(a[i], b[i]);
        });
        return bad;
    } else {
        return collide_offsets2<Q>(v, tau, cs);
    }
}

// Lattice constants for a run-time direction i (lane i of a warp that
// shares one cell's populations): the weight, and each component of e_i from
// a table packed two bits per direction (component + 1).
template <int Q>
__device__ __forceinline__ float lattice_w_rt(unsigned i) {
    return i == 0 ? Lattice<Q>::w(0) : (i < 7 ? Lattice<Q>::w(1) : Lattice<Q>::w(Q - 1));
}

// Component `axis` of e_i for a run-time direction: the table packed two bits
// per direction (component + 1) into one compile-time constant.
template <int Q>
__host__ __device__ constexpr unsigned long long lattice_e_bits(int axis) {
    unsigned long long b = 0;
    for (int i = 0; i < Q; ++i) {
        const int e = axis == 0 ? Lattice<Q>::ex(i) : (axis == 1 ? Lattice<Q>::ey(i) : Lattice<Q>::ez(i));
        b |= (unsigned long long)(e + 1) << (2 * i);
    }
    return b;
}

template <int Q, int Axis>
__device__ __forceinline__ float lattice_e_rt(unsigned i) {
    constexpr unsigned long long bits = lattice_e_bits<Q>(Axis);
    return (float)((int)((bits >> (2 * i)) & 3ull) - 1);
}

// equilibrium<Q, I> for a run-time direction: e.u as ((ex ux + ey uy) + ez uz)
// with e in {-1, 0, 1}, which equals edotu's sum of the non-zero terms (a
// zero term adds +-0, and only the sign of a zero result can differ, which
// the equilibrium does not see), then the same operations.
template <int Q>
__device__ __forceinline__ float equilibrium_rt(unsigned i, float rho, float ux, float uy, float uz, float u2) {
    const float eu = (lattice_e_rt<Q, 0>(i) * ux + lattice_e_rt<Q, 1>(i) * uy) + lattice_e_rt<Q, 2>(i) * uz;
    return (lattice_w_rt<Q>(i) * rho) * (((1.0f + 3.0f * eu) + (4.5f * eu) * eu) - 1.5f * u2);
}

// Storage code of a format (0 FP32, 1 FP16 offset, 2 BF16 offset).
template <class S>
constexpr int storage_code() {
    return S::kBytes == 4 ? 0 : (std::is_same<S, StoreF16>::value ? 1 : 2);
}

}  // namespace fc
