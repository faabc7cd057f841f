// Per-cell building blocks of the stream-collide kernels and the kernel
// templates built from them: the one-cell-per-thread kernel over the
// flattened lattice, its form for 16-bit populations with tiles staged through
// shared memory, the fine collide with the restriction's child sums fused in,
// the staged kernel that streams x-rows through shared memory
// with bulk async copies, and the AA-pattern in-place kernels.
//
// Physics follows the reference step (src/sim/lbm_core.cu:213-475): per link
// the upstream neighbour's flag selects plain streaming, half-way bounce-back
// (opposite slot of this cell) or specular free slip (mirrored slot of the
// tangentially displaced cell); inlet cells are written with feq(1, u_in),
// outlets copy the upstream column; moments with a density floor of 0.05; a
// |u| <= 0.3 limiter; Smagorinsky tau_eff from the non-equilibrium stress
// (Hou et al. 1996); TRT with magic parameter Lambda.
//
// Two collision bodies, selected by the EXACT template flag:
//  * collide_exact: the reference kernel's expression tree (lbm_core.cu:
//    386-467) with zero-coefficient terms skipped (an exact identity). It is
//    bit-identical to the reference only in a translation unit compiled with
//    --fmad=false (collide_f32.cu), where no multiply-add is contracted.
//  * collide_dev: the same TRT + Smagorinsky update on the deviations
//    g_q = f_q - w_q (the FP16 storage format), with moments, stress and
//    TRT formed from opposite-pair sums/differences and the equilibrium's
//    second moment in closed form (rho/3 I + rho u u); reciprocals and square
//    roots by the hardware approximations. Fewer instructions, no weight add
//    per load or subtract per store, FP32-rounding-level different.
// Population access follows the body: Pop<S, DEV> loads and stores f (exact
// body) or g (deviation body); a bounce-back or mirrored slot has the weight
// of the link it replaces and the Ladd and interpolated bounce-back terms are
// affine with unit coefficient sum, so every gather path is the same in both
// forms.
//
// This header is included by exactly one translation unit per instantiation
// set; the kernels live in an anonymous namespace.
#pragma once

#include "child_record.cuh"
#include "d3q19.cuh"
#include "kernels.h"
#include "pdl.cuh"

#include <cuda_runtime.h>

#include <type_traits>

namespace fcfd {
namespace {

struct CollideArgs {
    int nx, ny, nz;
    long long n; // cells per direction slice
    float tau0, lambda, smagPre, uIn;
    int writeMacro;
    float *rho, *u, *v, *w;
    const std::uint16_t *uwx, *uwy, *uwz;
    int* status; // staged kernel: nonzero when a pipeline wait timed out
    const std::uint8_t* qFrac;   // q-LIBB cut bytes [cell * 19 + q], or null
    const std::uint32_t* ffMask; // q-LIBB two-node bits [cell]
    const uint2* links;          // pull-link classes per cell (build_level_tables), or null
};

/// Slice pointers of one launch, passed as a __grid_constant__ kernel
/// parameter: pull[q][cell] is the source x - c_q of an interior cell (no
/// periodic wrap on any axis) in slice q, own[q][cell] the cell itself in
/// slice q of the source buffer, out[q][cell] in the destination. A load or
/// store of such a cell is one 32 x 32 + 64-bit multiply-add of the cell index
/// and a constant-bank pointer, where a wrapped 3-D index, a slice product or
/// a 64-bit offset added to a base pointer each take more instructions.
template <class T>
struct SlicePtrs {
    const T* pull[kQ];
    const T* own[kQ];
    T* out[kQ];
};

template <class T>
__host__ SlicePtrs<T> slice_ptrs(const T* src, T* dst, int nx, int ny, long long n) {
    SlicePtrs<T> o;
    const long long sx = nx, sxy = static_cast<long long>(nx) * ny;
    for (int q = 0; q < kQ; ++q) {
        o.own[q] = src + q * n;
        o.out[q] = dst + q * n;
        o.pull[q] = src + (q * n - (cx(q) + sx * cy(q) + sxy * cz(q)));
    }
    return o;
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

/// True when no pull of (x, y, z) wraps around a periodic axis.
__device__ __forceinline__ bool interior(int x, int y, int z, const CollideArgs& a) {
    return x > 0 && x < a.nx - 1 && y > 0 && y < a.ny - 1 && z > 0 && z < a.nz - 1;
}

/// Population access in f (DEV false) or deviation g = f - w_q (DEV true).
template <class S, bool DEV>
struct Pop {
    using T = typename S::T;
    __device__ __forceinline__ static float ld(const T* __restrict__ p, long long i, float w) {
        if constexpr (DEV) return S::ld_dev(p, i, w);
        else return S::ld(p, i, w);
    }
    __device__ __forceinline__ static void st(T* __restrict__ p, long long i, float v, float w) {
        if constexpr (DEV) S::st_dev(p, i, v, w);
        else S::st(p, i, v, w);
    }
    __device__ __forceinline__ static float lds(unsigned row, int i, float w) {
        if constexpr (DEV) return S::lds_dev(row, i, w);
        else return S::lds(row, i, w);
    }
    /// Coherent load, for a slot this kernel may have written.
    __device__ __forceinline__ static float ld_coherent(const T* p, float w) {
        const float v = static_cast<float>(*p);
        if constexpr (DEV) return std::is_same_v<T, float> ? v - w : v;
        else return std::is_same_v<T, float> ? v : w + v;
    }
};

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// ---- equilibrium in the reference expression order ------------------------
__device__ __forceinline__ float dot_c(int q, float ux, float uy, float uz) {
    // (cx ux + cy uy) + cz uz with zero terms dropped and +-1 folded.
    float d = 0.0f;
    bool any = false;
    if (cx(q) != 0) { d = cx(q) > 0 ? ux : -ux; any = true; }
    if (cy(q) != 0) { const float t = cy(q) > 0 ? uy : -uy; d = any ? d + t : t; any = true; }
    if (cz(q) != 0) { const float t = cz(q) > 0 ? uz : -uz; d = any ? d + t : t; }
    return d;
}

/// Reference equilibrium19 (lbm_core.cu:65-73): (w rho)((1 + cu + cu cu/2) - usq).
__device__ __forceinline__ void eq19(float rho, float ux, float uy, float uz, float (&feq)[kQ]) {
    const float usq = 1.5f * (ux * ux + uy * uy + uz * uz);
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        const float cu = 3.0f * dot_c(q, ux, uy, uz);
        feq[q] = (wgt(q) * rho) * (1.0f + cu + 0.5f * cu * cu - usq);
    }
}

// Packed operations on two floats in a register pair: each rounds as the
// scalar one does, in half the instructions. The collisions take two pairs of
// directions of equal weight through them. FP16 storage, bound by instruction
// issue: 24-tunnel polar 61.0 -> 58.4 ms per 100 steps, 333x170x149 in place
// 5.76 -> 5.52 ms per 40. FP32 storage (PAIRS) where instructions or latency
// bound a kernel and it has the registers to keep the operands in pairs: 64^3
// lattice 8.6 -> 8.2 us per step, the 640-cell tunnel's step with the child
// sums in pairs 3.10 -> 3.07 ms. Not by tile codes, at 40 registers (spills
// 140-190 bytes; the 768x320x96 tunnel 0.547 -> 0.601 ms per step), nor in the
// batch (12 tunnels 36.5 -> 37.8 ms per 100 steps).
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void un2(F2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ F2 sub2(F2 a, F2 b) { F2 r; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
/// A product that goes on into a packed sum: as a b + z with z a negative zero
/// that the assembler does not know for one, since it fuses a packed product
/// and the sum after it, rounding modifiers or not.
__device__ __forceinline__ F2 mul2(F2 a, F2 b, F2 z) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(z)); return r; }
__device__ __forceinline__ F2 neg_zero(float positive) { const float z = __fmul_rn(positive, -0.0f); return f2(z, z); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }

// ---- collision bodies ------------------------------------------------------
// The exact body forms the reference's expressions with fewer operations
// where the result is the same to the bit: sums start from their first term
// instead of 0 (only the sign of a zero sum could differ, which nothing below
// sees), the equilibria of an opposite pair share 0.5 (3 c.u)^2 (3 c.u changes
// sign exactly), and the TRT halves are taken by scaling the rate
// (multiplying by 0.5 is exact: omega (0.5 a - 0.5 b) = (0.5 omega)(a - b)).
template <bool PAIRS>
__device__ __forceinline__ void collide_exact(float (&f)[kQ], float tau0, float lambda, float smagPre,
                                              float& rhoO, float& uxO, float& uyO, float& uzO) {
    float rho = f[0], jx = f[1], jy = f[3], jz = f[5];
#pragma unroll
    for (int q = 1; q < kQ; ++q) {
        rho += f[q];
        if (cx(q) != 0 && q != 1) jx = cx(q) > 0 ? jx + f[q] : jx - f[q];
        if (cy(q) != 0 && q != 3) jy = cy(q) > 0 ? jy + f[q] : jy - f[q];
        if (cz(q) != 0 && q != 5) jz = cz(q) > 0 ? jz + f[q] : jz - f[q];
    }
    rho = fmaxf(rho, kRhoFloor);
    const float invRho = 1.0f / rho;
    float ux = jx * invRho, uy = jy * invRho, uz = jz * invRho;
    float u2 = ux * ux + uy * uy + uz * uz;
    if (u2 > kMaxSimSpeed * kMaxSimSpeed) {
        // The hardware reciprocal square root, as the reference's GPU build
        // evaluates rsqrtf (lbm_core.cu:413); its CPU build and the oracle
        // use IEEE 1/sqrtf. Only cells beyond |u| = 0.3 take this branch.
        const float s = kMaxSimSpeed * rsqrtf(u2);
        ux *= s; uy *= s; uz *= s;
        u2 = ux * ux + uy * uy + uz * uz;
    }
    const float usq = 1.5f * u2;
    float feq[kQ];
    feq[0] = (wgt(0) * rho) * (1.0f - usq);
    const F2 z = neg_zero(tau0);
    auto feq1 = [&](int p) {
        const int qa = 2 * p - 1, qb = 2 * p;
        const float cu = 3.0f * dot_c(qa, ux, uy, uz);
        const float h = 0.5f * cu * cu;
        const float wr = wgt(qa) * rho;
        feq[qa] = wr * (1.0f + cu + h - usq);
        feq[qb] = wr * (1.0f - cu + h - usq);
    };
    auto feq2 = [&](int p, int q) {   // two pairs of equal weight
        const int a = 2 * p - 1, b = 2 * q - 1;
        const float wr = wgt(a) * rho;
        const F2 one = f2(1.0f, 1.0f), w2 = f2(wr, wr), u2 = f2(usq, usq);
        const F2 cu = mul2(f2(3.0f, 3.0f), f2(dot_c(a, ux, uy, uz), dot_c(b, ux, uy, uz)), z);
        const F2 h = mul2(mul2(f2(0.5f, 0.5f), cu, z), cu, z);
        un2(mul2(w2, sub2(add2(add2(one, cu), h), u2), z), feq[a], feq[b]);
        un2(mul2(w2, sub2(add2(sub2(one, cu), h), u2), z), feq[a + 1], feq[b + 1]);
    };
    if constexpr (PAIRS) {
        feq2(1, 2);
        feq1(3);
        feq2(4, 5);
        feq2(6, 7);
        feq2(8, 9);
    } else {
#pragma unroll
        for (int p = 1; p <= 9; ++p) feq1(p);
    }
    float tauEff = tau0;
    if (smagPre > 0.0f) {
        float pxx = f[1] - feq[1], pyy = f[3] - feq[3], pzz = f[5] - feq[5];
        float pxy = f[7] - feq[7], pxz = f[9] - feq[9], pyz = f[11] - feq[11];
#pragma unroll
        for (int q = 2; q < kQ; ++q) {
            const float fneq = f[q] - feq[q];
            if (cx(q) != 0) pxx += fneq;
            if (cy(q) != 0 && q != 3) pyy += fneq;
            if (cz(q) != 0 && q != 5) pzz += fneq;
            if (cx(q) * cy(q) != 0 && q != 7) pxy = cx(q) * cy(q) > 0 ? pxy + fneq : pxy - fneq;
            if (cx(q) * cz(q) != 0 && q != 9) pxz = cx(q) * cz(q) > 0 ? pxz + fneq : pxz - fneq;
            if (cy(q) * cz(q) != 0 && q != 11) pyz = cy(q) * cz(q) > 0 ? pyz + fneq : pyz - fneq;
        }
        const float qbar = sqrtf(pxx * pxx + pyy * pyy + pzz * pzz + 2.0f * (pxy * pxy + pxz * pxz + pyz * pyz));
        tauEff = 0.5f * (tau0 + sqrtf(tau0 * tau0 + smagPre * qbar * invRho));
    }
    const float omP = 1.0f / tauEff;
    const float tauM = 0.5f + lambda / (tauEff - 0.5f);
    const float omM = 1.0f / tauM;
    const float hP = 0.5f * omP, hM = 0.5f * omM;
    f[0] = f[0] - omP * (f[0] - feq[0]);
    auto relax1 = [&](int p) {
        const int qa = 2 * p - 1, qb = 2 * p;
        const float sym = hP * ((f[qa] + f[qb]) - (feq[qa] + feq[qb]));
        const float asym = hM * ((f[qa] - f[qb]) - (feq[qa] - feq[qb]));
        f[qa] = f[qa] - sym - asym;
        f[qb] = f[qb] - sym + asym;
    };
    auto relax2 = [&](int p, int q) {
        const int a = 2 * p - 1, b = 2 * q - 1;
        const F2 fa = f2(f[a], f[b]), fb = f2(f[a + 1], f[b + 1]), ea = f2(feq[a], feq[b]), eb = f2(feq[a + 1], feq[b + 1]);
        const F2 sym = mul2(f2(hP, hP), sub2(add2(fa, fb), add2(ea, eb)), z);
        const F2 asym = mul2(f2(hM, hM), sub2(sub2(fa, fb), sub2(ea, eb)), z);
        un2(sub2(sub2(fa, sym), asym), f[a], f[b]);
        un2(add2(sub2(fb, sym), asym), f[a + 1], f[b + 1]);
    };
    if constexpr (PAIRS) {
        relax2(1, 2);
        relax1(3);
        relax2(4, 5);
        relax2(6, 7);
        relax2(8, 9);
    } else {
#pragma unroll
        for (int p = 1; p <= 9; ++p) relax1(p);
    }
    rhoO = rho; uxO = ux; uyO = uy; uzO = uz;
}

// ---- arithmetic of the deviation body -----------------------------------------
// Every operation is an explicit round-to-nearest intrinsic (the fused
// multiply-adds written out where the body wants them), so the compiler
// contracts nothing on its own and the body rounds the same in every
// translation unit and kernel that includes it.
template <class V> struct Lane;
template <> struct Lane<float> {
    __device__ __forceinline__ static float s(float v) { return v; }
    __device__ __forceinline__ static float add(float a, float b) { return __fadd_rn(a, b); }
    __device__ __forceinline__ static float sub(float a, float b) { return __fsub_rn(a, b); }
    __device__ __forceinline__ static float mul(float a, float b) { return __fmul_rn(a, b); }
    __device__ __forceinline__ static float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
    __device__ __forceinline__ static float neg(float a) { return -a; }
    __device__ __forceinline__ static float rcp(float a) { return rcp_approx(a); }
    __device__ __forceinline__ static float sqrt(float a) { return sqrt_approx(a); }
};

/// Density floor of one lane: rho = max-floored 1 + dr, rm1 = rho - 1.
__device__ __forceinline__ void rho_floor(float dr, float& rho, float& rm1) {
    const float r = __fadd_rn(1.0f, dr);
    const bool floored = r < kRhoFloor;
    rho = floored ? kRhoFloor : r;
    rm1 = floored ? kRhoFloor - 1.0f : dr;
}

/// The |u| <= 0.3 limiter of one lane (u2 recomputed when it acts).
__device__ __forceinline__ void limit_u(float& ux, float& uy, float& uz, float& u2) {
    if (u2 > kMaxSimSpeed * kMaxSimSpeed) {
        const float sc = __fmul_rn(kMaxSimSpeed, rsqrtf(u2));
        ux = __fmul_rn(ux, sc); uy = __fmul_rn(uy, sc); uz = __fmul_rn(uz, sc);
        u2 = __fmaf_rn(uz, uz, __fmaf_rn(uy, uy, __fmul_rn(ux, ux)));
    }
}

/// c_a . u of pair direction a, components in the order x, y, z.
template <class V>
__device__ __forceinline__ V dot_lane(int a, V ux, V uy, V uz) {
    using L = Lane<V>;
    V d = L::s(0.0f);
    bool any = false;
    if (cx(a) != 0) { d = cx(a) > 0 ? ux : L::neg(ux); any = true; }
    if (cy(a) != 0) { d = any ? (cy(a) > 0 ? L::add(d, uy) : L::sub(d, uy)) : (cy(a) > 0 ? uy : L::neg(uy)); any = true; }
    if (cz(a) != 0) d = any ? (cz(a) > 0 ? L::add(d, uz) : L::sub(d, uz)) : (cz(a) > 0 ? uz : L::neg(uz));
    return d;
}

/// TRT + Smagorinsky collision on the deviations g_q = f_q - w_q of one cell.
template <class V>
__device__ __forceinline__ void collide_dev_lanes(V (&g)[kQ], float tau0, float lambda, float smagPre, V& rhoO,
                                                  V& uxO, V& uyO, V& uzO) {
    using L = Lane<V>;
    // Pair sums of f are s[p] + 2 w_p, differences d[p] as for f. The
    // update needs only these (symmetric and antisymmetric parts), so the
    // pair's own values are not kept.
    V s[10], d[10];
    auto halves = [&](int p, int q) {
        const F2 a = f2(g[2 * p - 1], g[2 * q - 1]), b = f2(g[2 * p], g[2 * q]);
        un2(add2(a, b), s[p], s[q]);
        un2(sub2(a, b), d[p], d[q]);
    };
    halves(1, 2);
    halves(4, 5);
    halves(6, 7);
    halves(8, 9);
    s[3] = L::add(g[5], g[6]);
    d[3] = L::sub(g[5], g[6]);
    // Pair p has velocity c_{2p-1}: p1 (1,0,0) p2 (0,1,0) p3 (0,0,1)
    // p4 (1,1,0) p5 (1,0,1) p6 (0,1,1) p7 (1,-1,0) p8 (1,0,-1) p9 (0,1,-1).
    const V dr = L::add(L::add(L::add(g[0], L::add(L::add(s[1], s[2]), L::add(s[3], s[4]))),
                               L::add(L::add(s[5], s[6]), L::add(s[7], s[8]))),
                        s[9]);
    const V jx = L::add(L::add(L::add(d[1], d[4]), L::add(d[5], d[7])), d[8]);
    const V jy = L::add(L::add(L::add(d[2], d[4]), L::sub(d[6], d[7])), d[9]);
    const V jz = L::sub(L::add(L::add(d[3], d[5]), L::sub(d[6], d[8])), d[9]);
    V rho, rm1;   // rm1 = rho - 1
    rho_floor(dr, rho, rm1);
    const V inv = L::rcp(rho);
    V ux = L::mul(jx, inv), uy = L::mul(jy, inv), uz = L::mul(jz, inv);
    V u2 = L::fma(uz, uz, L::fma(uy, uy, L::mul(ux, ux)));
    limit_u(ux, uy, uz, u2);
    const V rux = L::mul(rho, ux), ruy = L::mul(rho, uy);
    V tauEff = L::s(tau0);
    if (smagPre > 0.0f) {
        // Non-equilibrium stress: the weights' share of the diagonal
        // (sum of w_q over c_a != 0 = 1/3) cancels against rho/3 up to rho - 1.
        const V r3 = L::mul(rm1, L::s(1.0f / 3.0f));
        V nxx, nyy;
        un2(fma2(f2(L::neg(rux), L::neg(ruy)), f2(ux, uy),
                 sub2(add2(add2(add2(f2(s[1], s[2]), f2(s[4], s[4])), add2(f2(s[5], s[6]), f2(s[7], s[7]))), f2(s[8], s[9])),
                      f2(r3, r3))),
            nxx, nyy);
        const V nzz = L::fma(L::neg(L::mul(rho, uz)), uz,
                             L::sub(L::add(L::add(L::add(s[3], s[5]), L::add(s[6], s[8])), s[9]), r3));
        const V nxy = L::fma(L::neg(rux), uy, L::sub(s[4], s[7]));
        const V nxz = L::fma(L::neg(rux), uz, L::sub(s[5], s[8]));
        const V nyz = L::fma(L::neg(ruy), uz, L::sub(s[6], s[9]));
        const V dia = L::fma(nzz, nzz, L::fma(nyy, nyy, L::mul(nxx, nxx)));
        const V off = L::fma(nyz, nyz, L::fma(nxz, nxz, L::mul(nxy, nxy)));
        const V qbar = L::sqrt(L::fma(L::s(2.0f), off, dia));
        const V inner = L::fma(L::mul(L::s(smagPre), qbar), inv, L::s(__fmul_rn(tau0, tau0)));
        tauEff = L::mul(L::s(0.5f), L::add(L::s(tau0), L::sqrt(inner)));
    }
    const V omP = L::rcp(tauEff);
    const V omM = L::rcp(L::fma(L::s(lambda), L::rcp(L::sub(tauEff, L::s(0.5f))), L::s(0.5f)));
    // feq_q - w_q = w_q (A + 4.5 rho (c_q.u)^2) + 3 w_q rho (c_q.u), A = rho - 1 - 1.5 rho u^2.
    const V A = L::fma(L::mul(L::s(-1.5f), rho), u2, rm1);
    const V r45 = L::mul(L::s(4.5f), rho);
    g[0] = L::fma(L::neg(omP), L::fma(L::s(-1.0f / 3.0f), A, g[0]), g[0]);
    // Two pairs of equal weight at a time in packed operations, which round
    // as the scalar ones do.
    const F2 z = neg_zero(tau0);
    const F2 nP = f2(-omP, -omP), nM = f2(-omM, -omM), A2 = f2(A, A), r2 = f2(r45, r45);
    auto relax2 = [&](int p, int q) {
        const int a = 2 * p - 1, b = 2 * q - 1;
        const float w = wgt(a), e1 = L::mul(L::s(6.0f * w), rho);
        const F2 cu = f2(dot_lane<V>(a, ux, uy, uz), dot_lane<V>(b, ux, uy, uz));
        const F2 es = mul2(f2(2.0f * w, 2.0f * w), fma2(mul2(r2, cu, z), cu, A2), z);
        const F2 ea = mul2(f2(e1, e1), cu, z);
        const F2 sp = f2(s[p], s[q]), dp = f2(d[p], d[q]);
        const F2 sym = fma2(nP, sub2(sp, es), sp), asym = fma2(nM, sub2(dp, ea), dp);
        const F2 h = f2(0.5f, 0.5f);
        un2(mul2(h, add2(sym, asym), z), g[a], g[b]);
        un2(mul2(h, sub2(sym, asym), z), g[a + 1], g[b + 1]);
    };
    relax2(1, 2);
    relax2(4, 5);
    relax2(6, 7);
    relax2(8, 9);
    {
        const float w = wgt(5);
        const V es = L::mul(L::s(2.0f * w), L::fma(L::mul(r45, uz), uz, A));
        const V ea = L::mul(L::mul(L::s(6.0f * w), rho), uz);
        const V sym = L::fma(L::neg(omP), L::sub(s[3], es), s[3]);
        const V half = L::mul(L::s(0.5f), L::fma(L::neg(omM), L::sub(d[3], ea), d[3]));
        g[5] = L::fma(L::s(0.5f), sym, half);
        g[6] = L::fma(L::s(0.5f), sym, L::neg(half));
    }
    rhoO = rho; uxO = ux; uyO = uy; uzO = uz;
}

__device__ __forceinline__ void collide_dev(float (&g)[kQ], float tau0, float lambda, float smagPre,
                                            float& rhoO, float& uxO, float& uyO, float& uzO) {
    collide_dev_lanes<float>(g, tau0, lambda, smagPre, rhoO, uxO, uyO, uzO);
}

/// The collision of a cell's 19 populations: f with the exact body, the
/// deviations g with the fast one.
template <bool EXACT, bool PAIRS = false>
__device__ __forceinline__ void collide_body(float (&f)[kQ], const CollideArgs& a, float& r, float& ux, float& uy,
                                             float& uz) {
    if constexpr (EXACT) collide_exact<PAIRS>(f, a.tau0, a.lambda, a.smagPre, r, ux, uy, uz);
    else collide_dev(f, a.tau0, a.lambda, a.smagPre, r, ux, uy, uz);
}

// ---- per-cell pieces ---------------------------------------------------------
struct Nbr {
    unsigned sx[3], sy[3], sz[3];
};

/// Source coordinates of a pull along each velocity component (x - c, wrapped).
__device__ __forceinline__ Nbr neighbours(int x, int y, int z, int nx, int ny, int nz) {
    Nbr b;
    b.sx[0] = wrap_inc(x, nx); b.sx[1] = x; b.sx[2] = wrap_dec(x, nx);
    b.sy[0] = wrap_inc(y, ny); b.sy[1] = y; b.sy[2] = wrap_dec(y, ny);
    b.sz[0] = wrap_inc(z, nz); b.sz[1] = z; b.sz[2] = wrap_dec(z, nz);
    return b;
}

/// Boundary (non-fluid) cell: inlet feq(1, u_in), outlets from the upstream
/// column, everything else untouched (lbm_core.cu:241-283).
template <class S>
__device__ __forceinline__ void boundary_cell(const typename S::T* __restrict__ src, typename S::T* __restrict__ dst,
                                              const CollideArgs& a, int flag, unsigned cell, int x, int y, int z) {
    const long long n = a.n;
    if (flag == kInlet) {
        float feq[kQ];
        eq19(1.0f, a.uIn, 0.0f, 0.0f, feq);
#pragma unroll
        for (int q = 0; q < kQ; ++q) S::st(dst + q * n, cell, feq[q], wgt(q));
        if (a.writeMacro) { a.rho[cell] = 1.0f; a.u[cell] = a.uIn; a.v[cell] = 0.0f; a.w[cell] = 0.0f; }
    } else if (flag == kOutlet || flag == kOutletEq) {
        const unsigned up = static_cast<unsigned>(wrap_dec(x, a.nx))
                          + static_cast<unsigned>(a.nx) * (static_cast<unsigned>(y) + static_cast<unsigned>(a.ny) * z);
        float g[kQ];
        float r = 0.0f, jx = 0.0f, jy = 0.0f, jz = 0.0f;
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
            g[q] = S::ld(src + q * n, up, wgt(q));
            r += g[q];
            if (cx(q) != 0) jx = cx(q) > 0 ? jx + g[q] : jx - g[q];
            if (cy(q) != 0) jy = cy(q) > 0 ? jy + g[q] : jy - g[q];
            if (cz(q) != 0) jz = cz(q) > 0 ? jz + g[q] : jz - g[q];
        }
        const float inv = 1.0f / r;
        const float ux = jx * inv, uy = jy * inv, uz = jz * inv;
        if (flag == kOutletEq) {
            eq19(1.0f, ux, uy, uz, g);   // equilibrium outflow feq(1, u_upstream)
            r = 1.0f;
        }
#pragma unroll
        for (int q = 0; q < kQ; ++q) S::st(dst + q * n, cell, g[q], wgt(q));
        if (a.writeMacro) { a.rho[cell] = r; a.u[cell] = ux; a.v[cell] = uy; a.w[cell] = uz; }
    } else if (a.writeMacro) {
        a.rho[cell] = 1.0f; a.u[cell] = 0.0f; a.v[cell] = 0.0f; a.w[cell] = 0.0f;
    }
}

/// Bulk fluid cell: 19 plain pulls from global memory.
template <class S, bool DEV>
__device__ __forceinline__ void gather_bulk(const typename S::T* __restrict__ src, const CollideArgs& a,
                                            const Nbr& b, float (&f)[kQ]) {
    const unsigned unx = a.nx, uny = a.ny;
#pragma unroll
    for (int q = 0; q < kQ; ++q)
        f[q] = Pop<S, DEV>::ld(src + q * a.n, b.sx[1 + cx(q)] + unx * (b.sy[1 + cy(q)] + uny * b.sz[1 + cz(q)]),
                               wgt(q));
}

/// Bulk fluid cell away from the periodic faces: the same 19 pulls through
/// the constant offsets.
template <class S, bool DEV>
__device__ __forceinline__ void gather_interior(const SlicePtrs<typename S::T>& o, unsigned cell, float (&f)[kQ]) {
#pragma unroll
    for (int q = 0; q < kQ; ++q) f[q] = Pop<S, DEV>::ld(o.pull[q], cell, wgt(q));
}

/// Store the 19 populations of `cell` (slice pointers when given).
template <class S, bool DEV>
__device__ __forceinline__ void store_cell(typename S::T* __restrict__ dst, const CollideArgs& a, unsigned cell,
                                           const float (&f)[kQ], const SlicePtrs<typename S::T>* o) {
#pragma unroll
    for (int q = 0; q < kQ; ++q) Pop<S, DEV>::st(o ? o->out[q] : dst + q * a.n, cell, f[q], wgt(q));
}

/// Near-wall fluid cell: the upstream flag picks the (slot, cell) pair per
/// link; the wall-model Ladd term 6 w_q (c_q . u_w) on solid links. LW: the
/// links' classes come from the cell's link word (a.links) instead of the
/// 18 neighbours' flags.
template <class S, bool WM, bool QL, bool DEV, bool LW = false>
__device__ __forceinline__ void gather_wall(const typename S::T* __restrict__ src,
                                            const std::uint8_t* __restrict__ kind, const CollideArgs& a,
                                            const Nbr& b, unsigned cell, int y, int z, float (&f)[kQ]) {
    const unsigned unx = a.nx, uny = a.ny;
    const long long n = a.n;
    float uwx = 0.0f, uwy = 0.0f, uwz = 0.0f;
    bool uwLoaded = false;
    using P = Pop<S, DEV>;
    unsigned long long lm = 0;
    if constexpr (LW) {
        const uint2 w = __ldg(a.links + cell);
        lm = static_cast<unsigned long long>(w.x) | (static_cast<unsigned long long>(w.y) << 32);
    }
    f[0] = P::ld(src, cell, wgt(0));
#pragma unroll
    for (int q = 1; q < kQ; ++q) {
        const unsigned X = b.sx[1 + cx(q)], Y = b.sy[1 + cy(q)], Z = b.sz[1 + cz(q)];
        const unsigned pn = X + unx * (Y + uny * Z);
        bool solid, slipY, slipZ;
        if constexpr (LW) {
            solid = (lm >> (q - 1)) & 1ull;
            slipY = (lm >> (17 + q)) & 1ull;
            slipZ = (lm >> (35 + q)) & 1ull;
        } else {
            const int nf = kind[pn] & kFlagMask;
            solid = nf == kSolid;
            slipY = is_slip_y(nf);
            slipZ = is_slip_z(nf);
        }
        const unsigned pY = X + unx * (static_cast<unsigned>(y) + uny * Z);
        const unsigned pZ = X + unx * (Y + uny * static_cast<unsigned>(z));
        const int qs = solid ? opp(q) : (slipY ? mir_y(q) : (slipZ ? mir_z(q) : q));
        const unsigned cs = solid ? cell : (slipY ? pY : (slipZ ? pZ : pn));
        float fq = P::ld(src + static_cast<long long>(qs) * n, cs, wgt(q));
        // Interpolated bounce-back (Bouzidi 2001) on a solid link with an
        // analytic cut fraction, in the reference's expression order
        // (lbm_core.cu:332-364): the wall sits at q = byte/255 of the link.
        if (QL && solid) {
            const std::uint8_t qb = a.qFrac[static_cast<long long>(cell) * kQ + q];
            if (qb != 0) {
                const float qf = static_cast<float>(qb) * (1.0f / 255.0f);
                const float fOut = P::ld(src + static_cast<long long>(q) * n, cell, wgt(q));
                if (qf >= 0.5f) {
                    const float inv2q = 0.5f / qf;
                    fq = inv2q * fOut + (1.0f - inv2q) * fq;
                } else if (a.ffMask[cell] & (1u << q)) {
                    // Second fluid node x + c_q (opposite the wall).
                    const unsigned pff = b.sx[1 - cx(q)] + unx * (b.sy[1 - cy(q)] + uny * b.sz[1 - cz(q)]);
                    const float fOutFF = P::ld(src + static_cast<long long>(q) * n, pff, wgt(q));
                    fq = 2.0f * qf * fOut + (1.0f - 2.0f * qf) * fOutFF;
                }
                // else: x + c_q solid (thin vane): keep the half-way value.
            }
        }
        if constexpr (WM) {
            if (solid) {
                if (!uwLoaded) {
                    uwx = __half2float(__ushort_as_half(a.uwx[cell]));
                    uwy = __half2float(__ushort_as_half(a.uwy[cell]));
                    uwz = __half2float(__ushort_as_half(a.uwz[cell]));
                    uwLoaded = true;
                }
                fq += (6.0f * wgt(q)) * dot_c(q, uwx, uwy, uwz);
            }
        }
        f[q] = fq;
    }
}

/// Near-wall interior cell whose wall links are all solid (bit q - 1 of
/// `solidMask`): the pulls of gather_wall through the constant offsets --
/// the own cell's opposite slot on a solid link, the upstream cell
/// otherwise -- with the same interpolated bounce-back and Ladd terms.
template <class S, bool WM, bool QL, bool DEV>
__device__ __forceinline__ void gather_solid_links(const typename S::T* __restrict__ src, const CollideArgs& a,
                                                   const SlicePtrs<typename S::T>& o, unsigned cell, int x, int y, int z,
                                                   unsigned solidMask, float (&f)[kQ]) {
    using P = Pop<S, DEV>;
    float uwx = 0.0f, uwy = 0.0f, uwz = 0.0f;
    if constexpr (WM) {
        uwx = __half2float(__ushort_as_half(a.uwx[cell]));
        uwy = __half2float(__ushort_as_half(a.uwy[cell]));
        uwz = __half2float(__ushort_as_half(a.uwz[cell]));
    }
    f[0] = P::ld(o.own[0], cell, wgt(0));
#pragma unroll
    for (int q = 1; q < kQ; ++q) {
        const bool solid = (solidMask >> (q - 1)) & 1u;
        float fq = P::ld(solid ? o.own[opp(q)] : o.pull[q], cell, wgt(q));
        if (QL && solid) {
            const std::uint8_t qb = a.qFrac[static_cast<long long>(cell) * kQ + q];
            if (qb != 0) {
                const float qf = static_cast<float>(qb) * (1.0f / 255.0f);
                const float fOut = P::ld(o.own[q], cell, wgt(q));
                if (qf >= 0.5f) {
                    const float inv2q = 0.5f / qf;
                    fq = inv2q * fOut + (1.0f - inv2q) * fq;
                } else if (a.ffMask[cell] & (1u << q)) {
                    const unsigned unx = a.nx, uny = a.ny;
                    const Nbr b = neighbours(x, y, z, a.nx, a.ny, a.nz);
                    const unsigned pff = b.sx[1 - cx(q)] + unx * (b.sy[1 - cy(q)] + uny * b.sz[1 - cz(q)]);
                    const float fOutFF = P::ld(src + static_cast<long long>(q) * a.n, pff, wgt(q));
                    fq = 2.0f * qf * fOut + (1.0f - 2.0f * qf) * fOutFF;
                }
            }
        }
        if constexpr (WM) {
            if (solid) fq += (6.0f * wgt(q)) * dot_c(q, uwx, uwy, uwz);
        }
        f[q] = fq;
    }
}

template <class S, bool EXACT, bool PAIRS = false>
__device__ __forceinline__ void finish_cell(typename S::T* __restrict__ dst, const CollideArgs& a, unsigned cell,
                                            float (&f)[kQ], const SlicePtrs<typename S::T>* o = nullptr) {
    float r, ux, uy, uz;
    collide_body<EXACT, PAIRS>(f, a, r, ux, uy, uz);
    store_cell<S, !EXACT>(dst, a, cell, f, o);
    if (a.writeMacro) { a.rho[cell] = r; a.u[cell] = ux; a.v[cell] = uy; a.w[cell] = uz; }
}

/// The 19 post-streaming populations of fluid cell (x, y, z): bulk cells by
/// plain pulls (constant offsets away from the periodic faces when `o` is
/// given), near-wall cells through their neighbours' flags.
template <class S, bool WM, bool QL, bool DEV, bool LW = false>
__device__ __forceinline__ void gather_fluid(const typename S::T* __restrict__ src,
                                             const std::uint8_t* __restrict__ kind, const CollideArgs& a,
                                             std::uint8_t k, unsigned cell, int x, int y, int z, float (&f)[kQ],
                                             const SlicePtrs<typename S::T>* o) {
    if (!(k & kNearWall)) {
        if (o && interior(x, y, z, a)) gather_interior<S, DEV>(*o, cell, f);
        else gather_bulk<S, DEV>(src, a, neighbours(x, y, z, a.nx, a.ny, a.nz), f);
        return;
    }
    // Near-wall cell. With the link classes at hand, an interior cell whose
    // wall links are all solid (the cells along a foil) pulls through the
    // constant offsets, a select per link choosing its own opposite slot over
    // the upstream cell; slip-wall cells and the periodic faces take the
    // general path (measured the same as a slip-aware select path, which
    // needs more registers).
    if (a.links && o && interior(x, y, z, a)) {
        const uint2 w = __ldg(a.links + cell);
        if (w.y == 0 && (w.x >> 18) == 0) {   // solid links only (no slip-wall bit)
            gather_solid_links<S, WM, QL, DEV>(src, a, *o, cell, x, y, z, w.x, f);
            return;
        }
    }
    gather_wall<S, WM, QL, DEV, LW>(src, kind, a, neighbours(x, y, z, a.nx, a.ny, a.nz), cell, y, z, f);
}

/// One full cell update at (x, y, z): boundary cells by flag, fluid cells
/// by their 19 pulls (bulk or near-wall path) and the collision.
template <class S, bool WM, bool EXACT, bool QL = false, bool LW = false>
__device__ __forceinline__ void collide_one(const typename S::T* __restrict__ src, typename S::T* __restrict__ dst,
                                            const std::uint8_t* __restrict__ kind, const CollideArgs& a, int x, int y,
                                            int z, const SlicePtrs<typename S::T>* o = nullptr) {
    const unsigned cell = static_cast<unsigned>(x)
                        + static_cast<unsigned>(a.nx) * (static_cast<unsigned>(y) + static_cast<unsigned>(a.ny) * z);
    const std::uint8_t k = kind[cell];
    const int flag = k & kFlagMask;
    if (flag != kFluid) {
        boundary_cell<S>(src, dst, a, flag, cell, x, y, z);
        return;
    }
    float f[kQ];
    gather_fluid<S, WM, QL, !EXACT, LW>(src, kind, a, k, cell, x, y, z, f, o);
    finish_cell<S, EXACT>(dst, a, cell, f, o);
}

// ---- one cell per thread over the flattened lattice -----------------------------
// Consecutive threads take consecutive cells across row boundaries, so no
// warp is cut by a row end. (x, y, z) come from two divisions by invariant
// integers (FastDiv, d3q19.cuh). HBM-bound with FP32 storage. With codes, a
// warp of bulk interior cells reads one code byte, brought into L2 ahead of
// time, in place of 32 kind bytes that stream from HBM before its pulls can
// start, and needs no coordinates: the 768x320x96 tunnel (23.6 M cells, FP32)
// runs at 0.552 ms per step, 6.51 TB/s, against 0.591 ms by kind bytes and
// rows; with every cell taken for bulk without looking it was 0.535 ms.
constexpr int kCellBlockX = 128;   // the cells of one code word

/// Codes of blocks that start a while later into L2: the codes of eight
/// neighbouring blocks share a sector, and without it all eight wait for HBM.
constexpr unsigned kCodesAhead = 3072;   // blocks; about one and a half residencies of the GPU
__device__ __forceinline__ void prefetch_codes(const std::uint32_t* codes) {
    if ((blockIdx.x & 7) == 0 && threadIdx.x == 0 && blockIdx.x + kCodesAhead < gridDim.x)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(codes + blockIdx.x + kCodesAhead));
}

/// One cell, its warp's tile code known.
template <class S, bool WM, bool EXACT, bool QL, bool PAIRS>
__device__ __forceinline__ void collide_coded(const typename S::T* __restrict__ src, typename S::T* __restrict__ dst,
                                              const std::uint8_t* __restrict__ kind, int code, const CollideArgs& a,
                                              const SlicePtrs<typename S::T>& off, unsigned cell, const FastDiv& divX,
                                              const FastDiv& divY) {
    if (cell >= static_cast<unsigned>(a.n) || (code == kTileIdle && !a.writeMacro)) return;
    float f[kQ];
    if (code == kTileBulk) {
        gather_interior<S, !EXACT>(off, cell, f);
    } else {
        const std::uint8_t k = kind[cell];
        const unsigned row = fdiv(cell, divX), zu = fdiv(row, divY);
        const int x = static_cast<int>(cell - row * divX.d), y = static_cast<int>(row - zu * divY.d);
        const int z = static_cast<int>(zu), flag = k & kFlagMask;
        if (flag != kFluid) {
            boundary_cell<S>(src, dst, a, flag, cell, x, y, z);
            return;
        }
        gather_fluid<S, WM, QL, !EXACT>(src, kind, a, k, cell, x, y, z, f, &off);
    }
    finish_cell<S, EXACT, PAIRS>(dst, a, cell, f, &off);
}

template <class S, bool WM, bool EXACT, bool QL, bool CODED>
__global__ void __launch_bounds__(kCellBlockX, CODED ? S::kCodedMinBlocks : S::kCellMinBlocks)
collide_flat_kernel(const typename S::T* __restrict__ src, typename S::T* __restrict__ dst,
                    const std::uint8_t* __restrict__ kind, const std::uint32_t* __restrict__ codes, CollideArgs a,
                    const __grid_constant__ SlicePtrs<typename S::T> off, FastDiv divX, FastDiv divY) {
    pdl_wait();
    const unsigned cell = blockIdx.x * kCellBlockX + threadIdx.x;
    int code = kTileGeneral;
    if constexpr (CODED) {
        prefetch_codes(codes);
        code = reinterpret_cast<const std::uint8_t*>(codes)[cell >> 5];
    }
    collide_coded<S, WM, EXACT, QL, !CODED>(src, dst, kind, code, a, off, cell, divX, divY);
}

// ---- tiles staged through shared memory (16-bit populations) --------------------
// A warp's access to one slice moves 64 bytes at 2 bytes a lane, and it is
// those small requests that bound the one-cell kernel with FP16 storage: with
// its collision taken out it ran no faster. Here a block brings the pulls of
// 128 consecutive cells in by 16-byte asynchronous copies (the 17 aligned
// chunks around each slice's run) and writes its results back in 16-byte
// pieces. A block whose cells are not all bulk and off the lattice's faces
// (walls, faces, inlets, outlets) runs cell by cell.
constexpr int kTile = 128;
constexpr int kTileRow = (kTile / 8 + 1) * 16;   // bytes of a slice's run with its misalignment
constexpr std::uint32_t kTileWordBulk = kTileBulk * 0x01010101u;

/// Per slice: the 16-byte boundary at or below cell 0's element of the reads,
/// the byte offset of that element in the tile, and cell 0's element of the
/// writes.
template <class T>
struct TileMap {
    const T* in[kQ];
    T* out[kQ];
    unsigned inOff[kQ];

    __host__ void set(int q, const T* i, T* o) {
        const auto u = reinterpret_cast<std::uintptr_t>(i);
        in[q] = reinterpret_cast<const T*>(u & ~std::uintptr_t{15});
        inOff[q] = static_cast<unsigned>(q * kTileRow + (u & 15u));
        out[q] = o;
    }
};

/// Copy the runs of the 128 cells from c0 on (a multiple of 128, all of them
/// off the faces, so that a run's last chunk ends inside the buffer) into
/// `tile` and wait for them.
template <class T>
__device__ __forceinline__ void tile_in(const TileMap<T>& m, unsigned c0, unsigned tile) {
    const unsigned t = threadIdx.x;
#pragma unroll
    for (int j = 0; j < 3; ++j) {   // 16 chunks a slice
        const unsigned i = t + kTile * j, q = i >> 4, c = i & 15;
        if (q < kQ)
            asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;" ::"r"(tile + q * kTileRow + 16 * c),
                         "l"(m.in[q] + (c0 + 8 * c))
                         : "memory");
    }
    if (t >= 64 && t < 64 + kQ) {   // and the 17th (the third round left warps 2 and 3 idle)
        const unsigned q = t - 64;
        asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;" ::"r"(tile + q * kTileRow + 256),
                     "l"(m.in[q] + (c0 + kTile))
                     : "memory");
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

/// Results of the block's 128 cells to their slots by 16-byte stores through
/// `tile`, whose contents every thread has read. n a multiple of 8.
template <class S, bool DEV>
__device__ __forceinline__ void tile_out(const TileMap<typename S::T>& m, unsigned c0, const float (&f)[kQ],
                                         unsigned char* tile) {
    using T = typename S::T;
    const unsigned t = threadIdx.x;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kQ; ++q) Pop<S, DEV>::st(reinterpret_cast<T*>(tile + q * kTileRow), t, f[q], wgt(q));
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const unsigned i = t + kTile * j, q = i >> 4, c = i & 15;
        if (q < kQ)
            *reinterpret_cast<uint4*>(m.out[q] + (c0 + 8 * c)) =
                *reinterpret_cast<const uint4*>(tile + q * kTileRow + 16 * c);
    }
}

template <class S, bool WM, bool EXACT, bool QL>
__global__ void __launch_bounds__(kTile, S::kTileMinBlocks)
collide_tile_kernel(const typename S::T* __restrict__ src, typename S::T* __restrict__ dst,
                    const std::uint8_t* __restrict__ kind, const std::uint32_t* __restrict__ codes, CollideArgs a,
                    const __grid_constant__ SlicePtrs<typename S::T> off,
                    const __grid_constant__ TileMap<typename S::T> map, FastDiv divX, FastDiv divY) {
    using P = Pop<S, !EXACT>;
    __shared__ __align__(16) unsigned char tile[kQ * kTileRow];
    const unsigned c0 = blockIdx.x * kTile, t = threadIdx.x, cell = c0 + t;
    pdl_wait();
    prefetch_codes(codes);
    const std::uint32_t word = codes[blockIdx.x];
    if (word != kTileWordBulk) {
        collide_coded<S, WM, EXACT, QL, true>(src, dst, kind, static_cast<int>(word >> (8 * (t >> 5))) & 0xff, a, off, cell,
                                        divX, divY);
        return;
    }
    const unsigned tb = smem_addr(tile);
    tile_in(map, c0, tb);
    float f[kQ], r, ux, uy, uz;
#pragma unroll
    for (int q = 0; q < kQ; ++q) f[q] = P::lds(tb + map.inOff[q], t, wgt(q));
    collide_body<EXACT>(f, a, r, ux, uy, uz);
    if (a.writeMacro) { a.rho[cell] = r; a.u[cell] = ux; a.v[cell] = uy; a.w[cell] = uz; }
    if (a.n % 8 == 0) tile_out<S, !EXACT>(map, c0, f, tile);
    else store_cell<S, !EXACT>(dst, a, cell, f, &off);
}

// ---- AA-pattern in-place streaming (all-fluid periodic lattices) --------------
// One population array A instead of the A/B pair (Bailey, Myre, Walsh, Lilja,
// Wilson 2009, "Accelerating lattice Boltzmann fluid flow simulations using
// graphics processors"). Between steps the array holds one of two layouts:
//  * the A/B state: A[q][x] = f*_q(x), each cell's post-collision populations;
//  * streamed:      A[opp(q)][x] = f*_q(x - c_q), the post-streaming
//    populations, with the slots of every opposite pair exchanged.
// An odd step reads the A/B state from the upstream cells, f_q(x) =
// A[q][x - c_q], collides and writes f*_q(x) to A[opp(q)][x + c_q] -- the
// slot it read for direction opp(q) -- leaving the streamed layout. An even
// step reads A[opp(q)][x] of its own cell and writes f*_q(x) to A[q][x],
// leaving the A/B state again, which readers want and a write leaves: no pass
// turns one into the other around an even number of steps (with the pairs
// exchanged in the other layout, as usual, each such read and the step after
// it cost a pass: 0.31 ms each at 8.4 M cells in FP16, two in 40 steps of
// 0.15 ms). Every cell writes exactly the slots it read and
// no other cell touches them, so the update is in place without races, and
// the non-coherent loads never see a slot another thread has written. The
// populations entering each collision are the A/B kernel's, so the results
// are identical bit for bit. Opposite directions share a weight, so the FP16
// deviation bytes move between slots unchanged.

template <class T>
__device__ __forceinline__ const T* byte_add(const T* p, long long b) {
    return reinterpret_cast<const T*>(reinterpret_cast<const char*>(p) + b);
}
template <class T>
__device__ __forceinline__ T* byte_add(T* p, long long b) {
    return reinterpret_cast<T*>(reinterpret_cast<char*>(p) + b);
}

/// Byte offsets from &A[0][x] of the odd-step read A[q][x - c_q] of an
/// interior cell; its write A[opp(q)][x + c_q] is the read offset of opp(q).
struct AAOffsets {
    long long rd[kQ];
};

template <class T>
__host__ AAOffsets aa_offsets(int nx, int ny, long long n) {
    AAOffsets o;
    const long long sx = nx, sxy = static_cast<long long>(nx) * ny;
    for (int q = 0; q < kQ; ++q)
        o.rd[q] = (q * n - (cx(q) + sx * cy(q) + sxy * cz(q))) * static_cast<long long>(sizeof(T));
    return o;
}

/// ROWS: the grid is (row blocks, y, z) over rows of whole blocks; otherwise
/// the blocks run over the flattened lattice, so that no row end leaves lanes
/// idle, at two divisions per cell in odd steps. 40 steps, FP16: 101x100x100
/// 0.91 -> 0.74 ms, 333x170x149 6.11 -> 5.79, 40x300x300 4.59 -> 3.08, but
/// 640x192x128 9.97 -> 10.39 (FP32: 1.21 -> 0.99, 8.40 -> 8.10, 6.04 -> 4.02,
/// 14.44 -> 14.83). Tiles staged as in collide_tile_kernel measured slower
/// than either (5.79 -> 6.30, 9.97 -> 11.45 ms): the cut chunks of each run go
/// back element by element.
template <class S, bool EXACT, bool ODD, bool ROWS, bool PAIRS>
__global__ void __launch_bounds__(kCellBlockX, S::kCellMinBlocks)
collide_aa_kernel(typename S::T* __restrict__ A, CollideArgs a, const __grid_constant__ AAOffsets off, FastDiv divX,
                  FastDiv divY) {
    pdl_wait();
    const long long n = a.n;
    const unsigned unx = a.nx, uny = a.ny;
    unsigned cell = blockIdx.x * kCellBlockX + threadIdx.x;
    if constexpr (ROWS) cell += unx * (blockIdx.y + uny * blockIdx.z);
    else if (cell >= static_cast<unsigned>(n)) return;
    using P = Pop<S, !EXACT>;
    float f[kQ], r, ux, uy, uz;
    typename S::T* base = A + cell;
    if constexpr (!ODD) {
#pragma unroll
        for (int q = 0; q < kQ; ++q) f[q] = P::ld(A + opp(q) * n, cell, wgt(q));
        collide_body<EXACT, PAIRS>(f, a, r, ux, uy, uz);
#pragma unroll
        for (int q = 0; q < kQ; ++q) P::st(A + q * n, cell, f[q], wgt(q));
    } else {
        int x, y, z;
        if constexpr (ROWS) {
            x = blockIdx.x * kCellBlockX + threadIdx.x; y = blockIdx.y; z = blockIdx.z;
        } else {
            const unsigned row = fdiv(cell, divX), zu = fdiv(row, divY);
            x = static_cast<int>(cell - row * unx); y = static_cast<int>(row - zu * uny); z = static_cast<int>(zu);
        }
        // One collision body for both paths; the wrapped neighbour indices of
        // a face cell are formed again for the stores rather than held across it.
        const bool inner = interior(x, y, z, a);
        if (inner) {
#pragma unroll
            for (int q = 0; q < kQ; ++q) f[q] = P::ld(byte_add(base, off.rd[q]), 0, wgt(q));
        } else {
            const Nbr b = neighbours(x, y, z, a.nx, a.ny, a.nz);
#pragma unroll
            for (int q = 0; q < kQ; ++q)
                f[q] = P::ld(A + q * n, b.sx[1 + cx(q)] + unx * (b.sy[1 + cy(q)] + uny * b.sz[1 + cz(q)]), wgt(q));
        }
        collide_body<EXACT, PAIRS>(f, a, r, ux, uy, uz);
        if (inner) {
#pragma unroll
            for (int q = 0; q < kQ; ++q) P::st(byte_add(base, off.rd[opp(q)]), 0, f[q], wgt(q));
        } else {
            const Nbr b = neighbours(x, y, z, a.nx, a.ny, a.nz);
#pragma unroll
            for (int q = 0; q < kQ; ++q)
                P::st(A + opp(q) * n, b.sx[1 - cx(q)] + unx * (b.sy[1 - cy(q)] + uny * b.sz[1 - cz(q)]), f[q], wgt(q));
        }
    }
    if (a.writeMacro) { a.rho[cell] = r; a.u[cell] = ux; a.v[cell] = uy; a.w[cell] = uz; }
}

template <class S, bool EXACT>
cudaError_t launch_collide_aa_impl(void* fv, LevelDims d, const CollideParams& p, int odd, float* rho, float* u,
                                   float* v, float* w, cudaStream_t st) {
    using T = typename S::T;
    CollideArgs a{};
    a.nx = d.nx; a.ny = d.ny; a.nz = d.nz; a.n = d.cells();
    a.tau0 = p.tau; a.lambda = p.magicLambda; a.smagPre = p.smagPrefactor; a.uIn = p.uInlet;
    a.writeMacro = (p.writeMacro && rho && u && v && w) ? 1 : 0;
    a.rho = rho; a.u = u; a.v = v; a.w = w;
    T* f = static_cast<T*>(fv);
    const AAOffsets off = aa_offsets<T>(d.nx, d.ny, a.n);
    const bool rows = d.nx % kCellBlockX == 0;
    const dim3 grid = rows ? dim3(static_cast<unsigned>(d.nx / kCellBlockX), static_cast<unsigned>(d.ny),
                                  static_cast<unsigned>(d.nz))
                           : dim3(static_cast<unsigned>((a.n + kCellBlockX - 1) / kCellBlockX));
    auto pick = [&](auto pairs) {
        constexpr bool P = decltype(pairs)::value;
        return rows ? (odd ? collide_aa_kernel<S, EXACT, true, true, P> : collide_aa_kernel<S, EXACT, false, true, P>)
                    : (odd ? collide_aa_kernel<S, EXACT, true, false, P> : collide_aa_kernel<S, EXACT, false, false, P>);
    };
    // FP32 in pairs while the lattice is mostly in L2. 40 steps, ms without and
    // with: 1.01 M cells 0.99 and 0.88, 1.33 M 1.34 and 1.28, 1.60 M 1.65 and
    // 1.62, 2.16 M (rows) 2.25 and 2.25, 2.20 M 2.28 and 2.30, 2.74 M 2.78 and
    // 2.82, 4.49 M 4.46 and 4.57, 8.4 M 8.07 and 8.30.
    auto kern = pick(std::false_type{});
    if constexpr (EXACT)
        if (a.n < S::kPairCells) kern = pick(std::true_type{});
    return launch_pdl(kern, grid, dim3(kCellBlockX), st, f, a, off, fast_div(d.nx), fast_div(d.ny));
}

// ---- warm-restart flag edits (applyFlagEditsKernel, lbm_core.cu:644-717) -----
// mask 1: newly solid -> every population of both buffers zeroed; mask 2:
// newly fluid -> equilibrium of the mean rho, u of the neighbours (x + c_q,
// no wrap in x/y, periodic z) that are fluid and unedited, read from fA
// (rest state when there are none), written to both buffers. Edited cells
// never read each other, so the kernel has no races.
template <class S>
__global__ void apply_flag_edits_kernel(typename S::T* __restrict__ fA, typename S::T* __restrict__ fB,
                                        const std::uint8_t* __restrict__ flags,
                                        const std::uint8_t* __restrict__ mask, int nx, int ny, int nz) {
    const long long n = static_cast<long long>(nx) * ny * nz;
    const long long cell = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (cell >= n) return;
    const std::uint8_t edit = mask[cell];
    if (edit == 0) return;
    if (edit == 1) {
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
            S::st(fA + q * n, cell, 0.0f, wgt(q));
            S::st(fB + q * n, cell, 0.0f, wgt(q));
        }
        return;
    }
    const long long nxny = static_cast<long long>(nx) * ny;
    const int z = static_cast<int>(cell / nxny);
    const long long rem = cell - static_cast<long long>(z) * nxny;
    const int y = static_cast<int>(rem / nx), x = static_cast<int>(rem - static_cast<long long>(y) * nx);
    float rho = 0.0f, ux = 0.0f, uy = 0.0f, uz = 0.0f;
    int found = 0;
    for (int q = 1; q < kQ; ++q) {
        const int xn = x + cx(q), yn = y + cy(q), zn = z + cz(q);
        if (xn < 0 || xn >= nx || yn < 0 || yn >= ny) continue;
        const int znw = zn < 0 ? nz - 1 : (zn >= nz ? 0 : zn);
        const long long nc = xn + static_cast<long long>(nx) * yn + nxny * znw;
        if (flags[nc] != kFluid || mask[nc] != 0) continue;
        float r = 0.0f, jx = 0.0f, jy = 0.0f, jz = 0.0f;
#pragma unroll
        for (int p = 0; p < kQ; ++p) {
            const float fq = S::ld(fA + p * n, nc, wgt(p));
            r += fq;
            jx += cx(p) * fq; jy += cy(p) * fq; jz += cz(p) * fq;
        }
        rho += r;
        ux += jx / r; uy += jy / r; uz += jz / r;
        ++found;
    }
    if (found > 0) {
        const float inv = 1.0f / static_cast<float>(found);
        rho *= inv; ux *= inv; uy *= inv; uz *= inv;
    } else {
        rho = 1.0f; ux = uy = uz = 0.0f;
    }
    float feq[kQ];
    eq19(rho, ux, uy, uz, feq);
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        S::st(fA + q * n, cell, feq[q], wgt(q));
        S::st(fB + q * n, cell, feq[q], wgt(q));
    }
}

template <class S>
cudaError_t launch_apply_flag_edits_impl(void* fA, void* fB, const std::uint8_t* flags, const std::uint8_t* mask,
                                         LevelDims d, cudaStream_t st) {
    using T = typename S::T;
    const long long n = d.cells();
    apply_flag_edits_kernel<S><<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(
        static_cast<T*>(fA), static_cast<T*>(fB), flags, mask, d.nx, d.ny, d.nz);
    return cudaGetLastError();
}

// ---- last fine sub-step with the restriction's child averages fused in --------
// Factor-2 patches only. A thread owns one fine x column of a 2 x 2 (y, z)
// cell group and updates its four cells in the children's summation order
// (z, then y); the x partner of each child pair is the neighbouring lane.
// The child sums stay in registers split across the lane pair (even lane:
// directions 0..9, odd lane: 10..18): per cell one shuffle per direction
// pair hands each lane the partner's value it needs, and each lane adds the
// two children in the stand-alone pass's order (z, y, x; solid children
// skipped). With FP32 storage the values summed are the stored ones, exactly
// as a later load returns them (bit-identical to the separate pass); with
// FP16 storage they are the collided FP32 values before the half rounding.
// The even lane then collects the odd lane's sums and
// writes the scratch record. This saves the stand-alone pass's full re-read
// of the fine populations (measured 3 % faster than accumulating in shared
// memory).
constexpr int kFuseX = 128;

constexpr int kSplit = 10;   // directions summed by the even lane

template <class S, bool WM, bool EXACT, bool QL>
__global__ void __launch_bounds__(kFuseX, S::kChildMinBlocks)
collide_child_kernel(const typename S::T* __restrict__ src, typename S::T* __restrict__ dst,
                     const std::uint8_t* __restrict__ kind, CollideArgs a, ChildFuse cf,
                     const __grid_constant__ SlicePtrs<typename S::T> off) {
    pdl_wait();
    const int x = blockIdx.x * kFuseX + threadIdx.x;
    const bool inX = x < a.nx;
    const bool even = (threadIdx.x & 1) == 0;
    const int lx = cf.boxX0 + (x >> 1) - cf.rx0, ly = cf.boxY0 + static_cast<int>(blockIdx.y) - cf.ry0;
    // Both lanes of a pair take the record decision of the even lane.
    const int xe = x & ~1;
    const bool record = xe + 1 < a.nx && lx >= 0 && lx < cf.rw && ly >= 0 && ly < cf.rh;
    float acc[kSplit];
#pragma unroll
    for (int k = 0; k < kSplit; ++k) acc[k] = 0.0f;
    int nFluid = 0;
    // The four cells' kind bytes, read up front (one byte each in a packed
    // word), so no cell's update waits on a kind load after the previous one.
    unsigned kinds = 0;
    if (inX) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int y = 2 * blockIdx.y + (c & 1), z = 2 * blockIdx.z + (c >> 1);
            kinds |= static_cast<unsigned>(kind[static_cast<unsigned>(x) + static_cast<unsigned>(a.nx)
                                                * (static_cast<unsigned>(y) + static_cast<unsigned>(a.ny) * z)])
                   << (8 * c);
        }
    }
    for (int kz = 0; kz < 2; ++kz)
        for (int jy = 0; jy < 2; ++jy) {
            const int y = 2 * blockIdx.y + jy, z = 2 * blockIdx.z + kz;
            // A solid child, or none, adds -0 to every sum: no sum changes.
            float v[kQ];
            bool solid = true;
            const std::uint8_t k = static_cast<std::uint8_t>(kinds >> (8 * (2 * kz + jy)));
            const int flag = k & kFlagMask;
            const unsigned cell = static_cast<unsigned>(x)
                                + static_cast<unsigned>(a.nx) * (static_cast<unsigned>(y) + static_cast<unsigned>(a.ny) * z);
            if (inX && flag == kFluid) {
                gather_fluid<S, WM, QL, !EXACT>(src, kind, a, k, cell, x, y, z, v, &off);
                float rr, ux, uy, uz;
                collide_body<EXACT, true>(v, a, rr, ux, uy, uz);
                // FP32: the sums see the stored values exactly. FP16:
                // the collided FP32 values (not their half round trip),
                // the more accurate child average.
                store_cell<S, !EXACT>(dst, a, cell, v, &off);
                solid = false;
            } else {
                if (inX) boundary_cell<S>(src, dst, a, flag, cell, x, y, z);
                solid = !inX || flag == kSolid;
                // Written or untouched, the child average sees what dst holds.
#pragma unroll
                for (int q = 0; q < kQ; ++q)
                    v[q] = solid ? -0.0f : Pop<S, !EXACT>::ld_coherent(off.out[q] + cell, wgt(q));
            }
            if (!solid) ++nFluid;
            // Children in order: the even lane's first, then the odd lane's.
#pragma unroll
            for (int k2 = 0; k2 < kSplit; ++k2) {
                const int qo = k2 + kSplit < kQ ? k2 + kSplit : kQ - 1;   // odd lane's direction
                const float recv = __shfl_xor_sync(0xffffffffu, even ? v[qo] : v[k2], 1);
                const float own = even ? v[k2] : v[qo];
                acc[k2] = (acc[k2] + (even ? own : recv)) + (even ? recv : own);
            }
        }
    // The even lane gathers the odd lane's sums (directions 10..18) and the
    // child count, then writes the record.
    const int nOdd = __shfl_xor_sync(0xffffffffu, nFluid, 1);
    float fi[kQ];
#pragma unroll
    for (int k = 0; k < kSplit; ++k) fi[k] = acc[k];
#pragma unroll
    for (int k = 0; k + kSplit < kQ; ++k) fi[k + kSplit] = __shfl_xor_sync(0xffffffffu, acc[k], 1);
    if (!record || !even) return;
    const RecordGrid rg{cf.rw, cf.rh};
    write_child_record<S, !EXACT>(fi, nFluid + nOdd,
                                  reinterpret_cast<float4*>(cf.scratch) + rg.index(lx, ly, static_cast<int>(blockIdx.z)),
                                  rg.count(a.nz / 2));
}

template <class S, bool EXACT>
cudaError_t launch_collide_child_impl(const void* srcv, void* dstv, const std::uint8_t* kind, LevelDims d,
                                      const CollideParams& p, SlipField slip, const ChildFuse& cf,
                                      cudaStream_t st) {
    using T = typename S::T;
    if (d.ny % 2 || d.nz % 2 || !cf.scratch) return cudaErrorInvalidValue;
    CollideArgs a;
    a.nx = d.nx; a.ny = d.ny; a.nz = d.nz; a.n = d.cells();
    a.tau0 = p.tau; a.lambda = p.magicLambda; a.smagPre = p.smagPrefactor; a.uIn = p.uInlet;
    a.writeMacro = 0;
    a.rho = a.u = a.v = a.w = nullptr;
    a.uwx = slip.uwx; a.uwy = slip.uwy; a.uwz = slip.uwz;
    a.status = nullptr;
    a.qFrac = p.qFrac; a.ffMask = p.ffMask;
    a.links = p.links;
    const dim3 block(kFuseX);
    const dim3 grid(static_cast<unsigned>((d.nx + kFuseX - 1) / kFuseX), static_cast<unsigned>(d.ny / 2),
                    static_cast<unsigned>(d.nz / 2));
    const T* src = static_cast<const T*>(srcv);
    T* dst = static_cast<T*>(dstv);
    const bool ql = a.qFrac != nullptr;
    const SlicePtrs<T> off = slice_ptrs<T>(src, dst, d.nx, d.ny, a.n);
    auto kern = slip.active()
                    ? (ql ? collide_child_kernel<S, true, EXACT, true> : collide_child_kernel<S, true, EXACT, false>)
                    : (ql ? collide_child_kernel<S, false, EXACT, true> : collide_child_kernel<S, false, EXACT, false>);
    return launch_pdl(kern, grid, block, st, src, dst, kind, a, cf, off);
}

// ---- staged: x-rows through shared memory with bulk async copies -------------
// A persistent CTA walks rows r = blockIdx.x + k * gridDim.x (r = y + ny z).
// For every row it needs, per direction q, the full source row (y - c_y,
// z - c_z) of slice q, plus the row's kind bytes. A producer warp brings them
// into a ring of shared-memory stages with one cp.async.bulk per row piece,
// each completing on the stage's "full" mbarrier (complete_tx); consumer
// warps wait on "full", compute their cells of the row, and release the stage
// on its "empty" mbarrier (one arrive per warp). There is no block-wide
// barrier per row: warps drift by up to the ring depth, and the bytes in
// flight are set by the ring, not by resident warps. Bulk fluid cells read
// their 19 pulls from the stage (x - c_x wraps inside the row); wall-adjacent
// and boundary cells use the global-memory paths. Requires rows of a
// multiple of 16 bytes. Every wait is bounded: on a timeout the kernel sets
// *status, lets its copies in flight land (bounded) and returns.
constexpr int kConsumerWarps = 15;
constexpr int kStagedThreads = (kConsumerWarps + 1) * 32;
constexpr int kMaxStages = 8;
constexpr long long kWaitLimit = 1LL << 18; // try_wait polls (each may sleep ~20 us) before a timeout

__device__ __forceinline__ void mbar_init(std::uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(std::uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(std::uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(std::uint64_t* bar, unsigned parity) {
    // The suspend-time hint (ns) lets a waiting warp sleep until the phase
    // completes instead of re-polling and taking issue slots.
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity), "r"(20000u)
        : "memory");
    return ok != 0;
}
/// Bounded wait on a barrier phase; false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(std::uint64_t* bar, unsigned parity) {
    for (long long i = 0; i < kWaitLimit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void bulk_g2s(void* dstSmem, const void* srcGlobal, unsigned bytes, std::uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dstSmem)),
        "l"(srcGlobal), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

/// Shared-memory layout of the ring.
struct StageLayout {
    unsigned kindBytes;  // per stage, 16-byte multiple (row bytes + alignment prefix)
    unsigned popBytes;   // per stage: 19 rows
    __host__ __device__ static unsigned header() { return 256; }
};

template <class S>
__host__ __device__ inline StageLayout stage_layout(int nx) {
    StageLayout l;
    l.kindBytes = static_cast<unsigned>(((nx + 15 + 15) / 16) * 16);
    l.popBytes = static_cast<unsigned>(kQ) * static_cast<unsigned>(nx) * sizeof(typename S::T);
    return l;
}

template <class S>
__device__ __forceinline__ void issue_row(const typename S::T* __restrict__ src,
                                          const std::uint8_t* __restrict__ kind, unsigned char* kstage,
                                          typename S::T* pstage, std::uint64_t* bar, long long row,
                                          const CollideArgs& a, unsigned kindBytes) {
    using T = typename S::T;
    const int y = static_cast<int>(row % a.ny), z = static_cast<int>(row / a.ny);
    const unsigned rowBytes = static_cast<unsigned>(a.nx) * sizeof(T);
    // Kind row: copy from the 16-byte boundary at or below its start.
    const long long kstart = row * static_cast<long long>(a.nx);
    const long long kal = kstart & ~15LL;
    const unsigned kb = static_cast<unsigned>(((kstart - kal + a.nx + 15) / 16) * 16);
    mbar_expect_tx(bar, rowBytes * kQ + kb);
    bulk_g2s(kstage, kind + kal, kb, bar);
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        int ys = y - cy(q), zs = z - cz(q);
        ys = ys < 0 ? ys + a.ny : (ys >= a.ny ? ys - a.ny : ys);
        zs = zs < 0 ? zs + a.nz : (zs >= a.nz ? zs - a.nz : zs);
        const T* g = src + q * a.n + static_cast<long long>(a.nx) * (ys + static_cast<long long>(a.ny) * zs);
        bulk_g2s(pstage + q * a.nx, g, rowBytes, bar);
    }
    (void)kindBytes;
}

template <class S, bool WM, bool EXACT, bool QL>
__global__ void __launch_bounds__(kStagedThreads, 2)
collide_staged_kernel(const typename S::T* __restrict__ src, typename S::T* __restrict__ dst,
                      const std::uint8_t* __restrict__ kind, CollideArgs a, int stages) {
    using T = typename S::T;
    extern __shared__ __align__(128) unsigned char smem[];
    std::uint64_t* full = reinterpret_cast<std::uint64_t*>(smem);
    std::uint64_t* empty = full + kMaxStages;
    const StageLayout L = stage_layout<S>(a.nx);
    unsigned char* kring = smem + StageLayout::header();
    T* pring = reinterpret_cast<T*>(kring + static_cast<size_t>(L.kindBytes) * stages);
    const long long rows = static_cast<long long>(a.ny) * a.nz;
    const long long G = gridDim.x;
    const int nx = a.nx;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t stageElems = static_cast<size_t>(kQ) * nx;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kConsumerWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == kConsumerWarps) {
        // ---- producer warp: one lane issues every copy ----
        if (lane == 0) {
            long long k = 0;
            for (;; ++k) {
                const long long r = blockIdx.x + k * G;
                if (r >= rows) break;
                const int s = static_cast<int>(k % stages);
                if (k >= stages && !mbar_wait(&empty[s], static_cast<unsigned>(((k / stages) - 1) & 1))) {
                    atomicExch(a.status, 1);
                    break;
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                issue_row<S>(src, kind, kring + static_cast<size_t>(L.kindBytes) * s, pring + stageElems * s,
                             &full[s], r, a, L.kindBytes);
            }
            // Let every copy this CTA issued land before the CTA can exit.
            for (long long j = k - stages; j < k; ++j)
                if (j >= 0) (void)mbar_wait(&full[j % stages], static_cast<unsigned>((j / stages) & 1));
        }
        return;
    }

    // ---- consumer warps ----
    // Row k is cut into 32-cell chunks; chunk j goes to warp
    // (j + k * nchunks) mod W, so the assignment rotates from row to row and
    // every warp does the same work over a few rows.
    const int nchunks = (nx + 31) / 32;
    for (long long k = 0;; ++k) {
        const long long r = blockIdx.x + k * G;
        if (r >= rows) break;
        const int s = static_cast<int>(k % stages);
        if (!mbar_wait(&full[s], static_cast<unsigned>((k / stages) & 1))) {
            atomicExch(a.status, 1);
            break;
        }
        const unsigned sbase = smem_addr(pring + stageElems * s);
        const long long kstart = r * static_cast<long long>(nx);
        const unsigned kbase = smem_addr(kring + static_cast<size_t>(L.kindBytes) * s) + static_cast<unsigned>(kstart & 15);
        const int y = static_cast<int>(r % a.ny), z = static_cast<int>(r / a.ny);
        const int j0 = static_cast<int>(((warp - (k * nchunks) % kConsumerWarps) % kConsumerWarps + kConsumerWarps)
                                        % kConsumerWarps);
        for (int j = j0; j < nchunks; j += kConsumerWarps) {
            const int x = j * 32 + lane;
            if (x >= nx) continue;
            const unsigned cell = static_cast<unsigned>(x) + static_cast<unsigned>(nx) * static_cast<unsigned>(r);
            unsigned short kb16;
            asm volatile("ld.shared.u8 %0, [%1];" : "=h"(kb16) : "r"(kbase + static_cast<unsigned>(x)));
            const std::uint8_t kb = static_cast<std::uint8_t>(kb16);
            const int flag = kb & kFlagMask;
            if (flag != kFluid) {
                boundary_cell<S>(src, dst, a, flag, cell, x, y, z);
                continue;
            }
            float f[kQ];
            if (!(kb & kNearWall)) {
                const int xs[3] = {wrap_inc(x, nx), x, wrap_dec(x, nx)};
                const unsigned rowBytes = static_cast<unsigned>(nx) * sizeof(T);
#pragma unroll
                for (int q = 0; q < kQ; ++q) f[q] = Pop<S, !EXACT>::lds(sbase + q * rowBytes, xs[1 + cx(q)], wgt(q));
            } else {
                const Nbr b = neighbours(x, y, z, nx, a.ny, a.nz);
                gather_wall<S, WM, QL, !EXACT>(src, kind, a, b, cell, y, z, f);
            }
            finish_cell<S, EXACT>(dst, a, cell, f);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
    }
}

// ---- launch ------------------------------------------------------------------
struct StagedPlan {
    int stages = 0;
    size_t smem = 0;
};

template <class S>
StagedPlan staged_plan(LevelDims d) {
    StagedPlan p;
    const size_t rowBytes = static_cast<size_t>(d.nx) * sizeof(typename S::T);
    if (rowBytes % 16 != 0 || d.nx < 8) return p;
    const StageLayout L = stage_layout<S>(d.nx);
    const size_t stageBytes = static_cast<size_t>(L.kindBytes) + L.popBytes;
    // Two CTAs per SM (113 KB each), each with as deep a ring as fits
    // (2..8 stages).
    const size_t budget = 113 * 1024 - StageLayout::header();
    const long long st = static_cast<long long>(budget / stageBytes);
    if (st < 2) return p;
    p.stages = static_cast<int>(st > kMaxStages ? kMaxStages : st);
    p.smem = StageLayout::header() + stageBytes * static_cast<size_t>(p.stages);
    return p;
}

template <class S, bool EXACT>
cudaError_t launch_collide_impl(const void* srcv, void* dstv, const std::uint8_t* kind, LevelDims d,
                                const CollideParams& p, float* rho, float* u, float* v, float* w, SlipField slip,
                                cudaStream_t st) {
    using T = typename S::T;
    CollideArgs a;
    a.nx = d.nx; a.ny = d.ny; a.nz = d.nz; a.n = d.cells();
    a.tau0 = p.tau; a.lambda = p.magicLambda; a.smagPre = p.smagPrefactor; a.uIn = p.uInlet;
    a.writeMacro = (p.writeMacro && rho && u && v && w) ? 1 : 0;
    a.rho = rho; a.u = u; a.v = v; a.w = w;
    a.uwx = slip.uwx; a.uwy = slip.uwy; a.uwz = slip.uwz;
    a.status = p.status;
    a.qFrac = p.qFrac; a.ffMask = p.ffMask;
    a.links = p.links;
    const T* src = static_cast<const T*>(srcv);
    T* dst = static_cast<T*>(dstv);
    const bool wm = slip.active();
    const StagedPlan plan = staged_plan<S>(d);
    // Automatic selection takes the one-cell kernel: on a GB300 the staged
    // ring measured slower (1.43-1.57 ms vs 0.89 ms per FP32 collide launch
    // on the 640x192x192 airfoil tunnel), its consumer warps being issue-bound
    // on shared-memory reads and ring bookkeeping.
    const bool staged = p.status && plan.stages >= 2 && p.kernel == 2;
    if (staged) {
        const bool ql = a.qFrac != nullptr;
        auto kern = wm ? (ql ? collide_staged_kernel<S, true, EXACT, true> : collide_staged_kernel<S, true, EXACT, false>)
                       : (ql ? collide_staged_kernel<S, false, EXACT, true> : collide_staged_kernel<S, false, EXACT, false>);
        // The dynamic shared-memory limit is a per-kernel attribute: raise it
        // once to the device's opt-in maximum (levels of one solver use
        // different stage sizes); occupancy is cached per (kernel, size).
        static const void* raised[8] = {};
        bool isRaised = false;
        for (const void* k : raised) isRaised |= (k == reinterpret_cast<const void*>(kern));
        if (!isRaised) {
            int dev = 0, optin = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
            if (static_cast<size_t>(optin) < plan.smem) return cudaErrorInvalidValue;
            if (auto e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
                e != cudaSuccess)
                return e;
            for (const void*& k : raised)
                if (!k) { k = reinterpret_cast<const void*>(kern); break; }
        }
        struct Entry { const void* k; size_t smem; int perSm; };
        static Entry cache[16] = {};
        int perSm = 0;
        for (const Entry& c : cache)
            if (c.k == reinterpret_cast<const void*>(kern) && c.smem == plan.smem) perSm = c.perSm;
        if (perSm == 0) {
            if (auto e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kern, kStagedThreads, plan.smem);
                e != cudaSuccess)
                return e;
            if (perSm < 1) perSm = 1;
            for (Entry& c : cache)
                if (c.k == nullptr) { c = Entry{reinterpret_cast<const void*>(kern), plan.smem, perSm}; break; }
        }
        const long long rows = static_cast<long long>(d.ny) * d.nz;
        long long grid = static_cast<long long>(sm_count()) * perSm;
        if (grid > rows) grid = rows;
        kern<<<static_cast<unsigned>(grid), kStagedThreads, plan.smem, st>>>(src, dst, kind, a, plan.stages);
        return cudaGetLastError();
    }
    const SlicePtrs<T> off = slice_ptrs<T>(src, dst, d.nx, d.ny, a.n);
    const FastDiv fx = fast_div(static_cast<unsigned>(d.nx)), fy = fast_div(static_cast<unsigned>(d.ny));
    const unsigned blocks = static_cast<unsigned>((a.n + kCellBlockX - 1) / kCellBlockX);
    const bool ql = a.qFrac != nullptr;
    // Codes (and the tiles they announce) where the populations stream from
    // HBM; a lattice that stays in L2 has its kind bytes there too, and the
    // code is then one more load ahead of the pulls.
    const bool coded = p.tiles && a.n >= S::kCodedCells;
    if (coded && (sizeof(T) == 4 || p.kernel == 0)) {
        if constexpr (sizeof(T) == 2) {
            TileMap<T> map;
            for (int q = 0; q < kQ; ++q) map.set(q, off.pull[q], off.out[q]);
            auto kern = wm ? (ql ? collide_tile_kernel<S, true, EXACT, true> : collide_tile_kernel<S, true, EXACT, false>)
                           : (ql ? collide_tile_kernel<S, false, EXACT, true> : collide_tile_kernel<S, false, EXACT, false>);
            return launch_pdl(kern, blocks, kTile, st, src, dst, kind, p.tiles, a, off, map, fx, fy);
        } else {
            auto kern = wm ? (ql ? collide_flat_kernel<S, true, EXACT, true, true> : collide_flat_kernel<S, true, EXACT, false, true>)
                           : (ql ? collide_flat_kernel<S, false, EXACT, true, true> : collide_flat_kernel<S, false, EXACT, false, true>);
            return launch_pdl(kern, blocks, kCellBlockX, st, src, dst, kind, p.tiles, a, off, fx, fy);
        }
    } else {
        auto kern = wm ? (ql ? collide_flat_kernel<S, true, EXACT, true, false> : collide_flat_kernel<S, true, EXACT, false, false>)
                       : (ql ? collide_flat_kernel<S, false, EXACT, true, false> : collide_flat_kernel<S, false, EXACT, false, false>);
        return launch_pdl(kern, blocks, kCellBlockX, st, src, dst, kind, nullptr, a, off, fx, fy);
    }
}

} // namespace
} // namespace fcfd
