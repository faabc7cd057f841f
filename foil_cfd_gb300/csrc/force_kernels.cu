// Momentum-exchange force on the solid (reference forceReductionKernel,
// src/sim/lbm_core.cu:573-637): every fluid cell with a solid neighbour at
// +c_q hands the wall c_q (2 f_q - 6 w_q (c_q . u_w)) per step, f_q being the
// post-collision population and u_w the wall-model slip velocity (zero when
// the model is off).
//
// GB300 design: instead of sweeping every cell and reading 18 neighbour flags
// (the reference), the kernel walks a compact list of wall-adjacent cells with
// a per-cell solid-link bit mask, built once per flag upload. Per-link terms
// are formed in FP32 as the reference does, then summed in FP64: per thread,
// per warp (shuffles), per block, and over the blocks' sums in a fixed order
// by the block that finishes last, so the result is deterministic run to run.
//
// A short list is a chain of latencies, a long one bound by the FP64 adds
// (1/64 of the FP32 rate). So a cell's populations are all under way before
// the first is added; a link adds to the components it has (30 adds for 18
// links instead of 54); blocks are of 64 threads, so that a short list spreads
// over the SMs and their FP64 units; and the sum over the blocks is no launch
// of its own. Under a profiler (caches cold): 1216 cells 17.9 -> 9.8 us, the
// 0.45 million cells around a 640-cell tunnel's patch 98 -> 70 us.
#include "d3q19.cuh"
#include "kernels.h"
#include "pdl.cuh"

#include <cuda_runtime.h>

#include <algorithm>

namespace fcfd {
namespace {

constexpr int kForceBlock = 64;
constexpr int kMaxForceBlocks = 4096;

__host__ __device__ int force_blocks(int count) {
    const int b = (count + kForceBlock - 1) / kForceBlock;
    return b < 1 ? 1 : b > kMaxForceBlocks ? kMaxForceBlocks : b;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

/// Block-wide FP64 sum of (a, b, c); the result is valid in thread 0.
__device__ __forceinline__ void block_sum3(double& a, double& b, double& c) {
    __shared__ double sh[3][kForceBlock / 32];
    a = warp_sum(a); b = warp_sum(b); c = warp_sum(c);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sh[0][warp] = a; sh[1][warp] = b; sh[2][warp] = c; }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < kForceBlock / 32; ++w) { a += sh[0][w]; b += sh[1][w]; c += sh[2][w]; }
    }
}

/// Momentum exchange of list blockIdx.y; blocks past the list's own count return.
template <class S, bool WM, int N>
__global__ void __launch_bounds__(kForceBlock)
force_kernel(const __grid_constant__ ForceLists<N> L) {
    using T = typename S::T;
    __shared__ bool last;
    pdl_wait();
    const ForceList& l = L.list[blockIdx.y];
    const unsigned nb = force_blocks(l.count);
    if (blockIdx.x >= nb) return;
    const T* f = static_cast<const T*>(l.f);
    double fx = 0.0, fy = 0.0, fz = 0.0;
    float probe = 0.0f;
    for (int i = blockIdx.x * kForceBlock + threadIdx.x; i < l.count; i += nb * kForceBlock) {
        const std::uint32_t c = l.cells[i];
        const std::uint32_t m = l.masks[i];
        float v[kQ];
#pragma unroll
        for (int q = 1; q < kQ; ++q) v[q] = m & (1u << q) ? S::ld(f + q * l.n, c, wgt(q)) : 0.0f;
        float uwx = 0.0f, uwy = 0.0f, uwz = 0.0f;
        if constexpr (WM) {
            uwx = __half2float(__ushort_as_half(l.slip.uwx[c]));
            uwy = __half2float(__ushort_as_half(l.slip.uwy[c]));
            uwz = __half2float(__ushort_as_half(l.slip.uwz[c]));
        }
#pragma unroll
        for (int q = 1; q < kQ; ++q) {
            if (!(m & (1u << q))) continue;
            // Rounded as the allocation-free variant's expression is.
            float corr = 0.0f;
            if constexpr (WM) corr = __fmul_rn(6.0f * wgt(q), cx(q) * uwx + cy(q) * uwy + cz(q) * uwz);
            const float t = __fmaf_rn(2.0f, v[q], -corr);
            // A component that the link lacks gets 0 t: nothing, or NaN.
            probe += 0.0f * t;
            if (cx(q) != 0) fx += static_cast<double>(cx(q) * t);
            if (cy(q) != 0) fy += static_cast<double>(cy(q) * t);
            if (cz(q) != 0) fz += static_cast<double>(cz(q) * t);
        }
    }
    fx += static_cast<double>(probe);
    fy += static_cast<double>(probe);
    fz += static_cast<double>(probe);
    block_sum3(fx, fy, fz);
    double* partials = l.scratch + 1;
    unsigned* ticket = reinterpret_cast<unsigned*>(l.scratch);
    if (threadIdx.x == 0) {
        partials[3 * blockIdx.x + 0] = fx;
        partials[3 * blockIdx.x + 1] = fy;
        partials[3 * blockIdx.x + 2] = fz;
        __threadfence();
        last = atomicAdd(ticket, 1u) == nb - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    fx = fy = fz = 0.0;
    for (unsigned b = threadIdx.x; b < nb; b += kForceBlock) {
        fx += __ldcg(partials + 3 * b + 0);
        fy += __ldcg(partials + 3 * b + 1);
        fz += __ldcg(partials + 3 * b + 2);
    }
    block_sum3(fx, fy, fz);
    if (threadIdx.x == 0) {
        l.out[0] = fx; l.out[1] = fy; l.out[2] = fz;
        *ticket = 0;   // for the next reduction
    }
}

template <int N>
cudaError_t launch_lists(Storage s, const ForceLists<N>& L, int lists, cudaStream_t st) {
    int nb = 1;
    bool wm = false;
    for (int i = 0; i < lists; ++i) {
        const ForceList& l = L.list[i];
        if (!l.f || !l.scratch || !l.out || l.n <= 0 || l.count < 0) return cudaErrorInvalidValue;
        nb = std::max(nb, force_blocks(l.count));
        wm = wm || l.slip.active();
    }
    const dim3 grid(static_cast<unsigned>(nb), static_cast<unsigned>(lists));
    if constexpr (N == 1) {
        if (wm)
            return launch_pdl(s == Storage::F32 ? force_kernel<StoreF32, true, N> : force_kernel<StoreF16, true, N>, grid,
                              kForceBlock, st, L);
    }
    return launch_pdl(s == Storage::F32 ? force_kernel<StoreF32, false, N> : force_kernel<StoreF16, false, N>, grid,
                      kForceBlock, st, L);
}

} // namespace

size_t force_scratch_bytes(int count) { return (1 + 3 * static_cast<size_t>(force_blocks(count))) * sizeof(double); }

cudaError_t launch_force(Storage s, const ForceList& list, cudaStream_t st) {
    return launch_lists(s, ForceLists<1>{{list}}, 1, st);
}

cudaError_t launch_forces(Storage s, const ForceLists<kMaxForceLists>& lists, int n, cudaStream_t st) {
    if (n < 1 || n > kMaxForceLists) return cudaErrorInvalidValue;
    return launch_lists(s, lists, n, st);
}

} // namespace fcfd
