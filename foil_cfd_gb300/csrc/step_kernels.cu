// Per-level kernels around the stream-collide: equilibrium / speck / macroscopic initialisation, the NaN
// watchdog, FP32 <-> storage conversion, the AA layout's conversions, and the
// FP16-storage stream-collide (the deviation collision body of
// collide_common.cuh; the FP32 storage collide lives in collide_f32.cu,
// compiled without contraction).
//
// GB300 layout choices (not in the reference): the buffers are unpadded SoA
// and all three axes wrap periodically in the index math, so there is no
// ghost-plane refresh pass; a per-cell kind byte marks the fluid cells that
// touch a wall, so bulk cells stream without reading 18 neighbour flags.
#include "collide_common.cuh"

namespace fcfd {
namespace {

constexpr int kBlock1D = 256;

/// Cold start of both buffers (f2 null: of one): equilibrium at the inlet speed
/// (at rest inside solids) and the spanwise speck perturbation (reference
/// lbm_core.cu:130-160), 3 w_q c_z w'(x, z) on the fluid cells' populations,
/// added to the value as stored. Two launches per buffer, the second over what
/// the first had written, moved 3 x these bytes: 23.6 million cells FP32
/// 1.10 ms, 0.50 ms in one pass over both.
template <class S>
__global__ void __launch_bounds__(kBlock1D)
reset_kernel(typename S::T* __restrict__ f, typename S::T* __restrict__ f2, const std::uint8_t* __restrict__ kind,
             unsigned n, int nx, int nz, FastDiv divX, FastDiv divXY, float uIn, float amp, float ph1, float ph2,
             float phX) {
    const unsigned c = blockIdx.x * kBlock1D + threadIdx.x;
    if (c >= n) return;
    const int flag = kind[c] & kFlagMask;
    const float ux = flag == kSolid ? 0.0f : uIn;
    float v[kQ];
    if constexpr (std::is_same_v<S, StoreF32>) {
        feq_rn(1.0f, ux, 0.0f, 0.0f, v);   // the FP32 storage's expressions, uncontracted
    } else {
        const float usq = 1.5f * (ux * ux);
#pragma unroll
        for (int q = 0; q < kQ; ++q) v[q] = feq_q(q, 1.0f, ux, 0.0f, 0.0f, usq);
    }
    if (flag == kFluid) {
        const unsigned zu = fdiv(c, divXY), rem = c - zu * divXY.d;
        const int z = static_cast<int>(zu), x = static_cast<int>(rem - fdiv(rem, divX) * divX.d);
        const float tz = 6.2831853f * (static_cast<float>(z) + 0.5f) / nz;
        const float tx = 6.2831853f * (static_cast<float>(x) + 0.5f) / nx;
        const float wz = amp * (0.6f * __sinf(3.0f * tz + ph1) + 0.4f * __sinf(7.0f * tz + ph2))
                       * (1.0f + 0.3f * __sinf(2.0f * tx + phX));
#pragma unroll
        for (int q = 1; q < kQ; ++q)
            if (cz(q) != 0) v[q] = S::rt(v[q], wgt(q)) + 3.0f * wgt(q) * cz(q) * wz;
    }
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        S::st(f + static_cast<long long>(q) * n, c, v[q], wgt(q));
        if (f2) S::st(f2 + static_cast<long long>(q) * n, c, v[q], wgt(q));
    }
}

template <class S>
__global__ void init_macro_kernel(typename S::T* __restrict__ f, const std::uint8_t* __restrict__ kind,
                                  long long n, const float* __restrict__ rho,
                                  const float* __restrict__ u, const float* __restrict__ v,
                                  const float* __restrict__ w) {
    const long long c = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const bool solid = (kind[c] & kFlagMask) == kSolid;
    const float r = solid ? 1.0f : rho[c];
    const float ux = solid ? 0.0f : u[c], uy = solid ? 0.0f : v[c], uz = solid ? 0.0f : w[c];
    const float usq = 1.5f * (ux * ux + uy * uy + uz * uz);
#pragma unroll
    for (int q = 0; q < kQ; ++q) S::st(f + q * n, c, feq_q(q, r, ux, uy, uz, usq), wgt(q));
}

/// NaN / runaway watchdog on a prime-strided sample (lbm_core.cu:526-559):
/// verdict base+1 = non-finite populations, base+2 = |u| pinned at the cap.
template <class S>
__global__ void watchdog_kernel(const typename S::T* __restrict__ f, long long n,
                                long long offset, int* flag, int flagBase) {
    const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long long c = t * 4093 + offset;
    if (c >= n) return;
    float s = 0.0f, jx = 0.0f, jy = 0.0f, jz = 0.0f;
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        const float v = S::ld(f + q * n, c, wgt(q));
        s += v; jx += cx(q) * v; jy += cy(q) * v; jz += cz(q) * v;
    }
    if (!isfinite(s)) {
        *flag = flagBase + 1;
    } else {
        const float sp2 = (jx * jx + jy * jy + jz * jz) / fmaxf(s * s, 1e-12f);
        const float cap = 0.95f * kMaxSimSpeed;
        if (sp2 > cap * cap) *flag = flagBase + 2;
    }
}

template <class S>
__global__ void f32_to_store_kernel(const float* __restrict__ in, typename S::T* __restrict__ out,
                                    long long n) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n * kQ) return;
    const int q = static_cast<int>(i / n);
    S::st(out, i, in[i], wgt(q));
}

template <class S>
__global__ void store_to_f32_kernel(const typename S::T* __restrict__ in, float* __restrict__ out,
                                    long long n) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n * kQ) return;
    const int q = static_cast<int>(i / n);
    out[i] = S::ld(in, i, wgt(q));
}

/// AA pattern: out[x] = in[x + s] of one direction slice, periodic on all
/// three axes.
template <class E>
__global__ void aa_shift_kernel(const E* __restrict__ in, E* __restrict__ out, int nx, int ny, int nz, int sx,
                                int sy, int sz) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= nx) return;
    const int y = blockIdx.y, z = blockIdx.z;
    int xs = x + sx, ys = y + sy, zs = z + sz;
    xs = xs < 0 ? xs + nx : (xs >= nx ? xs - nx : xs);
    ys = ys < 0 ? ys + ny : (ys >= ny ? ys - ny : ys);
    zs = zs < 0 ? zs + nz : (zs >= nz ? zs - nz : zs);
    out[x + static_cast<long long>(nx) * (y + static_cast<long long>(ny) * z)] =
        in[xs + static_cast<long long>(nx) * (ys + static_cast<long long>(ny) * zs)];
}

__global__ void fill_kernel(float* __restrict__ d, long long n, float v) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) d[i] = v;
}

inline unsigned blocks_for(long long n) {
    return static_cast<unsigned>((n + kBlock1D - 1) / kBlock1D);
}

inline dim3 plane_grid(const LevelDims& d, int bx) {
    return dim3(static_cast<unsigned>((d.nx + bx - 1) / bx), static_cast<unsigned>(d.ny),
                static_cast<unsigned>(d.nz));
}

} // namespace

cudaError_t launch_collide(Storage s, const void* src, void* dst, const std::uint8_t* kind, LevelDims d,
                           const CollideParams& p, float* rho, float* u, float* v, float* w, SlipField slip,
                           cudaStream_t st) {
    if (!src || !dst || !kind || d.cells() <= 0) return cudaErrorInvalidValue;
    // FP32 storage runs the reference-order kernels (bit-identical to the
    // reference step without FMA contraction); FP16 storage runs the
    // pair-sum collision. The staged kernel is used only when selected.
    if (s == Storage::F32)
        return launch_collide_f32_ref(static_cast<const float*>(src), static_cast<float*>(dst), kind, d, p,
                                      rho, u, v, w, slip, st);
    return launch_collide_impl<StoreF16, false>(src, dst, kind, d, p, rho, u, v, w, slip, st);
}

cudaError_t launch_collide_aa(Storage s, void* f, LevelDims d, const CollideParams& p, int odd, float* rho,
                              float* u, float* v, float* w, cudaStream_t st) {
    if (!f || d.cells() <= 0) return cudaErrorInvalidValue;
    if (s == Storage::F32) return launch_collide_aa_f32(static_cast<float*>(f), d, p, odd, rho, u, v, w, st);
    return launch_collide_aa_impl<StoreF16, false>(f, d, p, odd, rho, u, v, w, st);
}

namespace {
/// f*_q(x) = A[opp(q)][x + c_q]: the two slices of a pair change places, each
/// shifted along its own velocity, through one slice of scratch.
template <class E>
cudaError_t aa_shift_pairs(E* f, E* slice, LevelDims d, cudaStream_t st) {
    const long long n = d.cells();
    const dim3 grid = plane_grid(d, 128);
    for (int q = 1; q < kQ; q += 2) {
        E *a = f + q * n, *b = f + (q + 1) * n;
        aa_shift_kernel<E><<<grid, 128, 0, st>>>(b, slice, d.nx, d.ny, d.nz, cx(q), cy(q), cz(q));
        aa_shift_kernel<E><<<grid, 128, 0, st>>>(a, b, d.nx, d.ny, d.nz, -cx(q), -cy(q), -cz(q));
        if (auto e = cudaGetLastError(); e != cudaSuccess) return e;
        if (auto e = cudaMemcpyAsync(a, slice, static_cast<size_t>(n) * sizeof(E), cudaMemcpyDeviceToDevice, st);
            e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}
} // namespace

cudaError_t launch_aa_shift(Storage s, void* f, void* slice, LevelDims d, cudaStream_t st) {
    if (!f || !slice || d.cells() <= 0) return cudaErrorInvalidValue;
    if (s == Storage::F32) return aa_shift_pairs(static_cast<unsigned*>(f), static_cast<unsigned*>(slice), d, st);
    return aa_shift_pairs(static_cast<unsigned short*>(f), static_cast<unsigned short*>(slice), d, st);
}

cudaError_t launch_collide_child(Storage s, const void* src, void* dst, const std::uint8_t* kind, LevelDims d,
                                 const CollideParams& p, SlipField slip, const ChildFuse& cf, cudaStream_t st) {
    if (!src || !dst || !kind || d.cells() <= 0) return cudaErrorInvalidValue;
    if (s == Storage::F32)
        return launch_collide_child_f32(static_cast<const float*>(src), static_cast<float*>(dst), kind, d, p, slip,
                                        cf, st);
    return launch_collide_child_impl<StoreF16, false>(src, dst, kind, d, p, slip, cf, st);
}

cudaError_t launch_apply_flag_edits(Storage s, void* fA, void* fB, const std::uint8_t* flags,
                                    const std::uint8_t* mask, LevelDims d, cudaStream_t st) {
    if (!fA || !fB || !flags || !mask || d.cells() <= 0) return cudaErrorInvalidValue;
    if (s == Storage::F32)
        return launch_apply_flag_edits_f32(static_cast<float*>(fA), static_cast<float*>(fB), flags, mask, d, st);
    return launch_apply_flag_edits_impl<StoreF16>(fA, fB, flags, mask, d, st);
}

cudaError_t launch_reset(Storage s, void* f, void* f2, const std::uint8_t* kind, LevelDims d, float uInlet,
                         float amplitude, unsigned seed, cudaStream_t st) {
    const long long n = d.cells();
    if (!f || !kind || n <= 0) return cudaErrorInvalidValue;
    // Seeded phases through a Knuth multiplicative hash, as the reference
    // derives them (lbm_core.cu:761-767), so cold starts are reproducible.
    auto phase = [seed](unsigned salt) {
        unsigned h = (seed + salt) * 2654435761u;
        h ^= h >> 16;
        return 6.2831853f * static_cast<float>(h & 0xFFFFFFu) / 16777216.0f;
    };
    const FastDiv dx = fast_div(static_cast<unsigned>(d.nx));
    const FastDiv dxy = fast_div(static_cast<unsigned>(d.nx) * static_cast<unsigned>(d.ny));
    if (s == Storage::F32)
        reset_kernel<StoreF32><<<blocks_for(n), kBlock1D, 0, st>>>(
            static_cast<float*>(f), static_cast<float*>(f2), kind, static_cast<unsigned>(n), d.nx, d.nz, dx, dxy, uInlet,
            amplitude, phase(1u), phase(2u), phase(3u));
    else
        reset_kernel<StoreF16><<<blocks_for(n), kBlock1D, 0, st>>>(
            static_cast<__half*>(f), static_cast<__half*>(f2), kind, static_cast<unsigned>(n), d.nx, d.nz, dx, dxy, uInlet,
            amplitude, phase(1u), phase(2u), phase(3u));
    return cudaGetLastError();
}

cudaError_t launch_init_from_macro(Storage s, void* f, const std::uint8_t* kind, LevelDims d,
                                   const float* rho, const float* u, const float* v,
                                   const float* w, cudaStream_t st) {
    const long long n = d.cells();
    if (!f || !kind || n <= 0 || !rho || !u || !v || !w) return cudaErrorInvalidValue;
    if (s == Storage::F32)
        return launch_init_macro_f32(static_cast<float*>(f), kind, n, rho, u, v, w, st);
    else
        init_macro_kernel<StoreF16><<<blocks_for(n), kBlock1D, 0, st>>>(static_cast<__half*>(f), kind, n, rho, u, v, w);
    return cudaGetLastError();
}

cudaError_t launch_watchdog(Storage s, const void* f, LevelDims d, int* flag, long long offset,
                            int flagBase, cudaStream_t st) {
    const long long n = d.cells();
    if (!f || !flag || n <= 0) return cudaErrorInvalidValue;
    const long long off = ((offset % 4093) + 4093) % 4093;
    const long long samples = (n + 4092) / 4093;
    if (s == Storage::F32)
        watchdog_kernel<StoreF32><<<blocks_for(samples), kBlock1D, 0, st>>>(
            static_cast<const float*>(f), n, off, flag, flagBase);
    else
        watchdog_kernel<StoreF16><<<blocks_for(samples), kBlock1D, 0, st>>>(
            static_cast<const __half*>(f), n, off, flag, flagBase);
    return cudaGetLastError();
}

cudaError_t launch_f32_to_store(Storage s, const float* in, void* out, long long cells,
                                cudaStream_t st) {
    if (!in || !out || cells <= 0) return cudaErrorInvalidValue;
    if (s == Storage::F32)
        return cudaMemcpyAsync(out, in, static_cast<size_t>(cells) * kQ * sizeof(float),
                               cudaMemcpyDeviceToDevice, st);
    f32_to_store_kernel<StoreF16><<<blocks_for(cells * kQ), kBlock1D, 0, st>>>(in, static_cast<__half*>(out), cells);
    return cudaGetLastError();
}

cudaError_t launch_store_to_f32(Storage s, const void* in, float* out, long long cells,
                                cudaStream_t st) {
    if (!in || !out || cells <= 0) return cudaErrorInvalidValue;
    if (s == Storage::F32)
        return cudaMemcpyAsync(out, in, static_cast<size_t>(cells) * kQ * sizeof(float),
                               cudaMemcpyDeviceToDevice, st);
    store_to_f32_kernel<StoreF16><<<blocks_for(cells * kQ), kBlock1D, 0, st>>>(static_cast<const __half*>(in), out, cells);
    return cudaGetLastError();
}

cudaError_t launch_fill(float* dst, long long n, float v, cudaStream_t st) {
    if (!dst || n <= 0) return cudaErrorInvalidValue;
    fill_kernel<<<blocks_for(n), kBlock1D, 0, st>>>(dst, n, v);
    return cudaGetLastError();
}

} // namespace fcfd
