// 2:1 (generally m:1, m = 2..4) refinement-patch coupling, the reference's
// src/sim/lbm_refine.cu:70-429 physics on a GB300 work decomposition.
//
// Coarse -> fine fill: each target fine cell samples the 19 populations at
// its centre by trilinear interpolation over the 8 surrounding coarse cells
// (solid corners dropped and the weights renormalised), blended linearly
// between the two coarse time levels, splits them into feq + fneq, projects
// fneq onto the stress (Latt & Chopard 2006) and rescales it by
// tau_f / (m tau_c) (Dupuis & Chopard 2003). The reference launches this over
// every fine cell and exits early off the interface shell; here the launch
// covers a compact list of target cells (the shell per sub-step, or every
// non-solid fine cell when seeding).
//
// Fine -> coarse restriction: per coarse fluid cell of the patch minus a
// 2-cell band, average the m^3 fine children (solid children skipped), take
// fneq against the average's own equilibrium, filter fneq over the cell and
// its 18 lattice neighbours (Lagrava et al. 2012), regularise, rescale by
// m tau_c / tau_f and blend into the coarse post-collision state over a
// 3-cell edge ramp. The reference recomputes each neighbour's child average
// inside the filter (19 averages per cell); here pass 1 stores every child
// average once in scratch (one 96-byte record per coarse cell, stored
// planar: see child_record.cuh) and pass 2 filters from scratch.
//
// Built with --fmad=false: every expression keeps the reference's rounding,
// so fill and restriction are bit-identical to the reference kernels
// compiled without contraction (the limiter's rsqrtf is the same hardware
// instruction the reference's GPU build uses).
#include "child_record.cuh"
#include "d3q19.cuh"
#include "kernels.h"
#include "pdl.cuh"

#include <cuda_runtime.h>

#include <type_traits>

namespace fcfd {
namespace {

constexpr int kRefineBlock = 128;
constexpr int kRestrictBand = 2;   // coarse band skipped by the restriction
constexpr int kRestrictBlend = 3;  // edge-blend ramp width (coarse cells)

/// v folded into [0, n) for v in [-n, 2n): the fill's corners lie at most one
/// cell outside the coarse domain, so a compare replaces the division.
__device__ __forceinline__ int wrap1(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }

/// Latt-Chopard projection of fneq onto the second-order Hermite space
/// (zero-coefficient terms left out, as in child_record.cuh; the rest part, all
/// of whose coefficients are 0, is then not read: limited_moments has made every
/// part of a cell with a bad population NaN).
__device__ __forceinline__ void regularize(float (&fneq)[kQ]) {
    float pxx = fneq[1], pyy = fneq[3], pzz = fneq[5], pxy = fneq[7], pxz = fneq[9], pyz = fneq[11];
#pragma unroll
    for (int q = 2; q < kQ; ++q) {
        const float v = fneq[q];
        if (cx(q) != 0) pxx += v;
        if (cy(q) != 0 && q != 3) pyy += v;
        if (cz(q) != 0 && q != 5) pzz += v;
        if (cx(q) * cy(q) != 0 && q != 7) pxy = cx(q) * cy(q) > 0 ? pxy + v : pxy - v;
        if (cx(q) * cz(q) != 0 && q != 9) pxz = cx(q) * cz(q) > 0 ? pxz + v : pxz - v;
        if (cy(q) * cz(q) != 0 && q != 11) pyz = cy(q) * cz(q) > 0 ? pyz + v : pyz - v;
    }
    const float trace = (1.0f / 3.0f) * (pxx + pyy + pzz);
    fneq[0] = 4.5f * wgt(0) * (0.0f - trace);
#pragma unroll
    for (int p = 1; p <= 9; ++p) {   // c and -c project alike
        const int q = 2 * p - 1;
        float d = 0.0f;
        bool any = false;
        if (cx(q) != 0) { d = pxx; any = true; }
        if (cy(q) != 0) { d = any ? d + pyy : pyy; any = true; }
        if (cz(q) != 0) d = any ? d + pzz : pzz;
        if (cx(q) * cy(q) != 0) d = cx(q) * cy(q) > 0 ? d + 2.0f * pxy : d - 2.0f * pxy;
        if (cx(q) * cz(q) != 0) d = cx(q) * cz(q) > 0 ? d + 2.0f * pxz : d - 2.0f * pxz;
        if (cy(q) * cz(q) != 0) d = cy(q) * cz(q) > 0 ? d + 2.0f * pyz : d - 2.0f * pyz;
        fneq[q] = fneq[q + 1] = 4.5f * wgt(q) * (d - trace);
    }
}

/// Slice pointers of a fill: the coarse level's two time levels and the fine level.
template <class T>
struct FillPtrs {
    const T* t0[kQ];
    const T* t1[kQ];
    T* out[kQ];
    __host__ FillPtrs(const T* c0, const T* c1, T* f, long long cn, long long fn) {
        for (int q = 0; q < kQ; ++q) {
            t0[q] = c0 + q * cn;
            t1[q] = c1 + q * cn;
            out[q] = f + q * fn;
        }
    }
};

/// Interpolated populations -> equilibrium + neqScale x the regularised rest.
__device__ __forceinline__ void rescale(float (&fi)[kQ], float neqScale) {
    float rho, ux, uy, uz;
    limited_moments(fi, rho, ux, uy, uz);
    float feq[kQ];
    feq_rn(rho, ux, uy, uz, feq);
#pragma unroll
    for (int q = 0; q < kQ; ++q) fi[q] -= feq[q];
    regularize(fi);
#pragma unroll
    for (int q = 0; q < kQ; ++q) fi[q] = feq[q] + neqScale * fi[q];
}

/// BLEND false: a time weight of 0, where s0 + 0 (s1 - s0) is s0 itself
/// (the sign of a zero sum aside, for which s1 is read), so the second time
/// level is not read. Identical to the blended form whenever the second
/// level is finite.
/// The eight corners lie in four pairs of x neighbours (a patch keeps a cell
/// away from the coarse domain's x and y faces, so only z wraps): four cell
/// indices, the second of a pair one element on.
template <class S, bool BLEND>
__global__ void __launch_bounds__(kRefineBlock)
fill_kernel(const __grid_constant__ FillPtrs<typename S::T> fp, const std::uint8_t* __restrict__ ckind,
            const std::uint32_t* __restrict__ targets, unsigned count, RefineGeom g, float invFactor, float tw,
            float neqScale, FastDiv divX, FastDiv divXY) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait(i);
    if (i >= count) return;
    const std::uint32_t t = targets[i];
    const unsigned zu = fdiv(t, divXY);
    const unsigned rem = t - zu * divXY.d;
    const unsigned yu = fdiv(rem, divX);
    const int zf = static_cast<int>(zu), yf = static_cast<int>(yu), xf = static_cast<int>(rem - yu * divX.d);

    const float gx = static_cast<float>(g.boxX0) + (static_cast<float>(xf) + 0.5f) * invFactor - 0.5f;
    const float gy = static_cast<float>(g.boxY0) + (static_cast<float>(yf) + 0.5f) * invFactor - 0.5f;
    const float gz = (static_cast<float>(zf) + 0.5f) * invFactor - 0.5f;
    const int ix = static_cast<int>(floorf(gx)), iy = static_cast<int>(floorf(gy));
    const int iz = static_cast<int>(floorf(gz));
    const float tx = gx - ix, ty = gy - iy, tz = gz - iz;

    float w8[8];
    w8[0] = (1 - tx) * (1 - ty) * (1 - tz);
    w8[1] = tx * (1 - ty) * (1 - tz);
    w8[2] = (1 - tx) * ty * (1 - tz);
    w8[3] = tx * ty * (1 - tz);
    w8[4] = (1 - tx) * (1 - ty) * tz;
    w8[5] = tx * (1 - ty) * tz;
    w8[6] = (1 - tx) * ty * tz;
    w8[7] = tx * ty * tz;
    const unsigned cnx = g.coarse.nx, cny = g.coarse.ny;
    std::uint32_t row[4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
        row[r] = static_cast<unsigned>(ix) + cnx * (static_cast<unsigned>(iy + (r & 1))
                                                    + cny * static_cast<unsigned>(wrap1(iz + (r >> 1), g.coarse.nz)));
    float wsum = 0.0f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        if ((ckind[row[c >> 1] + (c & 1)] & kFlagMask) == kSolid) w8[c] = 0.0f;
        wsum += w8[c];
    }
    if (wsum < 1e-6f) return; // fully inside a parent solid: leave it
    const float iws = 1.0f / wsum;
#pragma unroll
    for (int c = 0; c < 8; ++c) w8[c] *= iws;

    float fi[kQ];
    // FP16 storage sums the stored deviations and adds w_q once: with the
    // corner weights summing to one, sum w8 (w_q + g) = w_q + sum w8 g up to
    // rounding, without a weight add per corner load. FP32 keeps the
    // reference's expression.
    constexpr bool kDev = std::is_same_v<S, StoreF16>;
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const unsigned e = row[c >> 1];
            if constexpr (kDev) {
                s0 += w8[c] * S::template ld_dev<kIndexed>(fp.t0[q] + e, c & 1, wgt(q));
                if constexpr (BLEND) s1 += w8[c] * S::template ld_dev<kIndexed>(fp.t1[q] + e, c & 1, wgt(q));
            } else {
                s0 += w8[c] * S::template ld<kIndexed>(fp.t0[q] + e, c & 1, wgt(q));
                if constexpr (BLEND) s1 += w8[c] * S::template ld<kIndexed>(fp.t1[q] + e, c & 1, wgt(q));
            }
        }
        if constexpr (kDev) {
            fi[q] = wgt(q) + (BLEND ? s0 + tw * (s1 - s0) : s0);
        } else if constexpr (BLEND) {
            fi[q] = s0 + tw * (s1 - s0);
        } else {
            if (s0 == 0.0f) {
#pragma unroll
                for (int c = 0; c < 8; ++c) s1 += w8[c] * S::template ld<kIndexed>(fp.t1[q] + row[c >> 1], c & 1, wgt(q));
                s0 = s0 + tw * (s1 - s0);
            }
            fi[q] = s0;
        }
    }
    rescale(fi, neqScale);
#pragma unroll
    for (int q = 0; q < kQ; ++q) S::st(fp.out[q], t, fi[q], wgt(q));
}

/// Seeds a whole fine level: every cell that is not solid, in both buffers
/// (`twin` elements apart), as fill_kernel does from one time level. G = 2,
/// for factor 2: a thread has the two cells, one above the other, that lie
/// between the same coarse planes and reads their eight corners once. One cell
/// at a time waited for its 152 loads: 41.7 million cells FP32 2.01 ms, 1.68 by
/// pairs (at 80 registers; 1.77 at 128, 1.69 at 64).
template <class S, int G>
__global__ void __launch_bounds__(kRefineBlock, G == 2 ? 6 : 10)
seed_kernel(const __grid_constant__ FillPtrs<typename S::T> fp, const std::uint8_t* __restrict__ ckind,
            const std::uint8_t* __restrict__ fkind, unsigned count, RefineGeom g, float invFactor, float neqScale,
            FastDiv divX, FastDiv divXY, long long twin) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait(i);
    if (i >= count) return;
    const unsigned zu = fdiv(i, divXY);
    const unsigned rem = i - zu * divXY.d;
    const unsigned yu = fdiv(rem, divX);
    const int yf = static_cast<int>(yu), xf = static_cast<int>(rem - yu * divX.d);
    const int z0 = G == 2 ? 2 * static_cast<int>(zu) - 1 : static_cast<int>(zu);
    bool on[G];
    bool any = false;
#pragma unroll
    for (int k = 0; k < G; ++k) {
        const int z = z0 + k;
        on[k] = z >= 0 && z < g.fine.nz && (fkind[rem + divXY.d * static_cast<unsigned>(z)] & kFlagMask) != kSolid;
        any = any || on[k];
    }
    if (!any) return;

    const float gx = static_cast<float>(g.boxX0) + (static_cast<float>(xf) + 0.5f) * invFactor - 0.5f;
    const float gy = static_cast<float>(g.boxY0) + (static_cast<float>(yf) + 0.5f) * invFactor - 0.5f;
    const int ix = static_cast<int>(floorf(gx)), iy = static_cast<int>(floorf(gy));
    const int iz = static_cast<int>(floorf((static_cast<float>(z0 + G - 1) + 0.5f) * invFactor - 0.5f));
    const float tx = gx - ix, ty = gy - iy;
    const unsigned cnx = g.coarse.nx, cny = g.coarse.ny;
    std::uint32_t row[4];
    bool solid[8];
#pragma unroll
    for (int r = 0; r < 4; ++r)
        row[r] = static_cast<unsigned>(ix) + cnx * (static_cast<unsigned>(iy + (r & 1))
                                                    + cny * static_cast<unsigned>(wrap1(iz + (r >> 1), g.coarse.nz)));
#pragma unroll
    for (int c = 0; c < 8; ++c) solid[c] = (ckind[row[c >> 1] + (c & 1)] & kFlagMask) == kSolid;
    const float w4[4] = {(1 - tx) * (1 - ty), tx * (1 - ty), (1 - tx) * ty, tx * ty};
    float w8[G][8];
#pragma unroll
    for (int k = 0; k < G; ++k) {
        const float tz = ((static_cast<float>(z0 + k) + 0.5f) * invFactor - 0.5f) - iz;
        float wsum = 0.0f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            w8[k][c] = solid[c] ? 0.0f : w4[c & 3] * (c < 4 ? 1 - tz : tz);
            wsum += w8[k][c];
        }
        on[k] = on[k] && !(wsum < 1e-6f);   // fully inside a parent solid: leave it
        const float iws = 1.0f / wsum;
#pragma unroll
        for (int c = 0; c < 8; ++c) w8[k][c] *= iws;
    }
    constexpr bool kDev = std::is_same_v<S, StoreF16>;
    float fi[G][kQ];
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        float v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const auto* p = fp.t0[q] + row[c >> 1];
            v[c] = kDev ? S::template ld_dev<kIndexed>(p, c & 1, wgt(q)) : S::template ld<kIndexed>(p, c & 1, wgt(q));
        }
#pragma unroll
        for (int k = 0; k < G; ++k) {
            float s0 = 0.0f;
#pragma unroll
            for (int c = 0; c < 8; ++c) s0 += w8[k][c] * v[c];
            fi[k][q] = kDev ? wgt(q) + s0 : s0 + 0.0f;   // the sign of a zero: that of fill_kernel's s0 + 0 (s0 - s0)
        }
    }
#pragma unroll
    for (int k = 0; k < G; ++k) {
        if (!on[k]) continue;
        rescale(fi[k], neqScale);
        const unsigned t = rem + divXY.d * static_cast<unsigned>(z0 + k);
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
            S::st(fp.out[q], t, fi[k][q], wgt(q));
            S::st(fp.out[q] + twin, t, fi[k][q], wgt(q));
        }
    }
}

/// Pass 1: child average of every coarse cell of the restricted sub-box, as
/// one 96-byte record per coarse cell (six float4).
template <class S>
__global__ void __launch_bounds__(kRefineBlock)
child_avg_kernel(const typename S::T* __restrict__ ff, const std::uint8_t* __restrict__ fkind,
                 RefineGeom g, int rx0, int ry0, RecordGrid rg, float* __restrict__ scratch) {
    int lx = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait(lx);
    if (lx >= rg.w) return;
    const int ly = blockIdx.y, zc = blockIdx.z;
    const int m = g.factor;
    const int fx = m * (rx0 + lx - g.boxX0), fy = m * (ry0 + ly - g.boxY0), fz = m * zc;
    const long long fn = g.fine.cells();
    const unsigned fnx = g.fine.nx, fnxy = static_cast<unsigned>(g.fine.nx) * g.fine.ny;
    float fi[kQ];
#pragma unroll
    for (int q = 0; q < kQ; ++q) fi[q] = 0.0f;
    int nFluid = 0;
    for (int k = 0; k < m; ++k)
        for (int j = 0; j < m; ++j)
            for (int i = 0; i < m; ++i) {
                const unsigned c = static_cast<unsigned>(fx + i) + fnx * static_cast<unsigned>(fy + j)
                                 + fnxy * static_cast<unsigned>(fz + k);
                if ((fkind[c] & kFlagMask) == kSolid) continue;
                ++nFluid;
#pragma unroll
                for (int q = 0; q < kQ; ++q) fi[q] += S::template ld<kIndexed>(ff + q * fn, c, wgt(q));
            }
    write_child_record<S>(fi, nFluid, reinterpret_cast<float4*>(scratch) + rg.index(lx, ly, zc),
                          rg.count(g.coarse.nz));
}

/// Every record of a new scratch without fluid children (the border stays so).
template <class S>
__global__ void __launch_bounds__(kRefineBlock) clear_records_kernel(float* __restrict__ scratch, unsigned count) {
    const unsigned t = blockIdx.x * kRefineBlock + threadIdx.x;
    if (t < count) ChildRecord<S>::write_invalid(reinterpret_cast<float4*>(scratch) + t, count);
}

constexpr int kRestrictTX = 32, kRestrictTY = 2, kRestrictTZ = 2;

template <class S>
__global__ void __launch_bounds__(kRestrictTX * kRestrictTY * kRestrictTZ)
restrict_kernel(typename S::T* __restrict__ fc, const std::uint8_t* __restrict__ ckind,
                RefineGeom g, int rx0, int ry0, RecordGrid rg, float neqScaleInv,
                const __grid_constant__ RecordPlanes rec, float* __restrict__ mRho,
                float* __restrict__ mU, float* __restrict__ mV, float* __restrict__ mW) {
    int lx = blockIdx.x * kRestrictTX + threadIdx.x;
    pdl_wait(lx);
    const int ly = blockIdx.y * kRestrictTY + threadIdx.y;
    const int zc = blockIdx.z * kRestrictTZ + threadIdx.z;
    const int nz = g.coarse.nz;
    if (lx >= rg.w || ly >= rg.h || zc >= nz) return;
    const unsigned t = rg.index(lx, ly, zc);
    const int xc = rx0 + lx, yc = ry0 + ly;
    const long long cn = g.coarse.cells();
    const unsigned cell = static_cast<unsigned>(xc) + static_cast<unsigned>(g.coarse.nx)
                        * (static_cast<unsigned>(yc) + static_cast<unsigned>(g.coarse.ny) * zc);
    if ((ckind[cell] & kFlagMask) != kFluid) return;
    float fneq[kQ], stencil;
    using Rec = ChildRecord<S>;
    typename Rec::Raw raw[2];
    Rec::fetch(rec, t, raw[0]);
    Rec::template add<true>(raw[0], fneq, stencil);
    if (stencil == 0.0f) return;

    const int dEdge = min(min(lx, rg.w - 1 - lx), min(ly, rg.h - 1 - ly));
    const float blend = fminf(1.0f, static_cast<float>(dEdge + 1) / static_cast<float>(kRestrictBlend + 1));

    // The neighbours in the reference's order. A record in the border or
    // without fluid children adds nothing, so no load waits on a test, and the
    // next neighbour's loads are under way while one is added: left to the
    // compiler, ordinary loads came out at 64 registers and waited more
    // (321x101x33 with a patch, FP32: 23.5 us a launch, so 21.7, through the
    // read-only path 21.2; at 80 registers 20.4, but a step of the 640-cell
    // tunnel takes 0.4 % longer, with FP16 storage 1.2 %).
    const int zm = zc == 0 ? nz - 1 : zc - 1, zp = zc == nz - 1 ? 0 : zc + 1;
    auto at = [&](int nb) { return rg.index(lx + cx(nb), ly + cy(nb), cz(nb) < 0 ? zm : (cz(nb) > 0 ? zp : zc)); };
    Rec::fetch(rec, at(1), raw[1]);
#pragma unroll
    for (int nb = 1; nb < kQ; ++nb) {
        if (nb + 1 < kQ) Rec::fetch(rec, at(nb + 1), raw[(nb + 1) & 1]);
        Rec::template add<false>(raw[nb & 1], fneq, stencil);
    }
    const float invS = 1.0f / stencil;
#pragma unroll
    for (int q = 0; q < kQ; ++q) fneq[q] *= invS;
    regularize(fneq);
    const float4 m4 = ChildRecord<S>::moments(rec, t);
    float feq[kQ];
    feq_rn(m4.x, m4.y, m4.z, m4.w, feq);
    // The coarse collide, whose result this replaces, ran before the fine
    // sub-steps: earlier than the launch before this one.
    float b[kQ];
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        const float restricted = feq[q] + neqScaleInv * fneq[q];
        const float existing = S::template ld<kEarlier>(fc + q * cn, cell, wgt(q));
        b[q] = existing + blend * (restricted - existing);
        S::st(fc + q * cn, cell, b[q], wgt(q));
    }
    if (mRho) {
        float br = b[0], bjx = b[1], bjy = b[3], bjz = b[5];
#pragma unroll
        for (int q = 1; q < kQ; ++q) {
            br += b[q];
            if (cx(q) != 0 && q != 1) bjx = cx(q) > 0 ? bjx + b[q] : bjx - b[q];
            if (cy(q) != 0 && q != 3) bjy = cy(q) > 0 ? bjy + b[q] : bjy - b[q];
            if (cz(q) != 0 && q != 5) bjz = cz(q) > 0 ? bjz + b[q] : bjz - b[q];
        }
        bjx = __fmaf_rn(0.0f, br, bjx); bjy = __fmaf_rn(0.0f, br, bjy); bjz = __fmaf_rn(0.0f, br, bjz);
        br = fmaxf(br, kRhoFloor);
        const float bi = 1.0f / br;
        mRho[cell] = br; mU[cell] = bjx * bi; mV[cell] = bjy * bi; mW[cell] = bjz * bi;
    }
}

inline void sub_box(const RefineGeom& g, int& rx0, int& ry0, int& rw, int& rh) {
    rx0 = g.boxX0 + kRestrictBand;
    ry0 = g.boxY0 + kRestrictBand;
    rw = (g.boxX1 - kRestrictBand) - rx0;
    rh = (g.boxY1 - kRestrictBand) - ry0;
}

} // namespace

template <class S>
static cudaError_t launch_fill_impl(const void* cT0, const void* cT1, const std::uint8_t* coarseKind, void* fineF,
                                    const std::uint32_t* targets, int count, const RefineGeom& g, float timeWeight,
                                    float neqScale, cudaStream_t st) {
    using T = typename S::T;
    const FillPtrs<T> fp(static_cast<const T*>(cT0), static_cast<const T*>(cT1), static_cast<T*>(fineF),
                         g.coarse.cells(), g.fine.cells());
    const unsigned nb = static_cast<unsigned>((count + kRefineBlock - 1) / kRefineBlock);
    const FastDiv dx = fast_div(static_cast<unsigned>(g.fine.nx));
    const FastDiv dxy = fast_div(static_cast<unsigned>(g.fine.nx) * static_cast<unsigned>(g.fine.ny));
    return launch_pdl(timeWeight != 0.0f ? fill_kernel<S, true> : fill_kernel<S, false>, nb, kRefineBlock, st, fp,
                      coarseKind, targets, static_cast<unsigned>(count), g, 1.0f / static_cast<float>(g.factor),
                      timeWeight, neqScale, dx, dxy);
}

template <class S>
static cudaError_t launch_seed_impl(const void* coarseF, const std::uint8_t* coarseKind, void* fine0, void* fine1,
                                    const std::uint8_t* fineKind, const RefineGeom& g, float neqScale, cudaStream_t st) {
    using T = typename S::T;
    const FillPtrs<T> fp(static_cast<const T*>(coarseF), static_cast<const T*>(coarseF), static_cast<T*>(fine0),
                         g.coarse.cells(), g.fine.cells());
    const long long plane = static_cast<long long>(g.fine.nx) * g.fine.ny;
    const bool pairs = g.factor == 2 && g.fine.nz == 2 * g.coarse.nz;
    const long long count = plane * (pairs ? g.coarse.nz + 1 : g.fine.nz);
    const unsigned nb = static_cast<unsigned>((count + kRefineBlock - 1) / kRefineBlock);
    return launch_pdl(pairs ? seed_kernel<S, 2> : seed_kernel<S, 1>, nb, kRefineBlock, st, fp, coarseKind, fineKind,
                      static_cast<unsigned>(count), g, 1.0f / static_cast<float>(g.factor), neqScale,
                      fast_div(static_cast<unsigned>(g.fine.nx)), fast_div(static_cast<unsigned>(plane)),
                      static_cast<long long>(static_cast<T*>(fine1) - static_cast<T*>(fine0)));
}

cudaError_t launch_fill_c2f(Storage s, const void* cT0, const void* cT1,
                            const std::uint8_t* coarseKind, void* fineF,
                            const std::uint32_t* targets, int count, const RefineGeom& g,
                            float timeWeight, float neqScale, cudaStream_t st) {
    if (!cT0 || !cT1 || !coarseKind || !fineF || g.factor < 2 || g.factor > 4)
        return cudaErrorInvalidValue;
    if (count <= 0) return cudaSuccess;
    return (s == Storage::F32 ? launch_fill_impl<StoreF32> : launch_fill_impl<StoreF16>)(
        cT0, cT1, coarseKind, fineF, targets, count, g, timeWeight, neqScale, st);
}

cudaError_t launch_seed_c2f(Storage s, const void* coarseF, const std::uint8_t* coarseKind, void* fine0, void* fine1,
                            const std::uint8_t* fineKind, const RefineGeom& g, float neqScale, cudaStream_t st) {
    if (!coarseF || !coarseKind || !fine0 || !fine1 || !fineKind || g.factor < 2 || g.factor > 4)
        return cudaErrorInvalidValue;
    return (s == Storage::F32 ? launch_seed_impl<StoreF32> : launch_seed_impl<StoreF16>)(
        coarseF, coarseKind, fine0, fine1, fineKind, g, neqScale, st);
}

static RecordGrid record_grid(const RefineGeom& g, int& rx0, int& ry0) {
    RecordGrid rg;
    sub_box(g, rx0, ry0, rg.w, rg.h);
    return rg;
}

long long restrict_scratch_floats(const RefineGeom& g) {
    int rx0, ry0;
    const RecordGrid rg = record_grid(g, rx0, ry0);
    if (rg.w <= 0 || rg.h <= 0) return 0;
    return kScratchVals * rg.count(g.coarse.nz);
}

cudaError_t launch_clear_scratch(Storage s, const RefineGeom& g, float* scratch, cudaStream_t st) {
    int rx0, ry0;
    const long long n = record_grid(g, rx0, ry0).count(g.coarse.nz);
    if (!scratch || n <= 0) return cudaErrorInvalidValue;
    const unsigned nb = static_cast<unsigned>((n + kRefineBlock - 1) / kRefineBlock);
    if (s == Storage::F32) clear_records_kernel<StoreF32><<<nb, kRefineBlock, 0, st>>>(scratch, static_cast<unsigned>(n));
    else clear_records_kernel<StoreF16><<<nb, kRefineBlock, 0, st>>>(scratch, static_cast<unsigned>(n));
    return cudaGetLastError();
}

void restrict_sub_box(const RefineGeom& g, int& rx0, int& ry0, int& rw, int& rh) { sub_box(g, rx0, ry0, rw, rh); }

template <class S>
static cudaError_t launch_restrict_impl(const void* fineF, const std::uint8_t* fineKind, void* coarseF,
                                        const std::uint8_t* coarseKind, const RefineGeom& g, float neqScaleInv,
                                        float* scratch, float* rho, float* u, float* v, float* w, cudaStream_t st,
                                        bool childDone) {
    using T = typename S::T;
    int rx0, ry0;
    const RecordGrid rg = record_grid(g, rx0, ry0);
    if (rg.w <= 0 || rg.h <= 0) return cudaErrorInvalidValue;
    if (!childDone) {
        const dim3 grid(static_cast<unsigned>((rg.w + kRefineBlock - 1) / kRefineBlock), static_cast<unsigned>(rg.h),
                        static_cast<unsigned>(g.coarse.nz));
        if (auto e = launch_pdl(child_avg_kernel<S>, grid, kRefineBlock, st, static_cast<const T*>(fineF), fineKind, g,
                                rx0, ry0, rg, scratch);
            e != cudaSuccess)
            return e;
    }
    const dim3 block(kRestrictTX, kRestrictTY, kRestrictTZ);
    const dim3 grid(static_cast<unsigned>((rg.w + kRestrictTX - 1) / kRestrictTX),
                    static_cast<unsigned>((rg.h + kRestrictTY - 1) / kRestrictTY),
                    static_cast<unsigned>((g.coarse.nz + kRestrictTZ - 1) / kRestrictTZ));
    return launch_pdl(restrict_kernel<S>, grid, block, st, static_cast<T*>(coarseF), coarseKind, g, rx0, ry0, rg,
                      neqScaleInv, RecordPlanes::of(scratch, rg.count(g.coarse.nz)), u && v && w ? rho : nullptr, u, v,
                      w);
}

cudaError_t launch_restrict_f2c(Storage s, const void* fineF, const std::uint8_t* fineKind,
                                void* coarseF, const std::uint8_t* coarseKind,
                                const RefineGeom& g, float neqScaleInv, float* scratch,
                                float* rho, float* u, float* v, float* w, cudaStream_t st, bool childDone) {
    if (!fineF || !fineKind || !coarseF || !coarseKind || !scratch || g.factor < 2 || g.factor > 4)
        return cudaErrorInvalidValue;
    return (s == Storage::F32 ? launch_restrict_impl<StoreF32> : launch_restrict_impl<StoreF16>)(
        fineF, fineKind, coarseF, coarseKind, g, neqScaleInv, scratch, rho, u, v, w, st, childDone);
}

} // namespace fcfd
