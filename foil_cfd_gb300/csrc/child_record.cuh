// Restriction pass 1 per coarse cell: the averaged children's moments with
// the density floor and the |u| <= 0.3 limiter, their non-equilibrium part,
// and the scratch record the restriction filter reads (fneq[19], valid
// flag, rho, ux, uy, uz; 96 B with FP32 storage, 64 B with FP16). Shared by the stand-alone
// child-average kernel and the fine collide that fuses it.
//
// The scratch is planar: float4 k of record t sits at base[k * stride + t]
// (stride = records in the scratch), so the 32 lanes of a warp reading the
// same part of the records of 32 consecutive coarse cells read 512
// contiguous bytes, not 32 pieces 96 bytes apart. Every multiply
// and add is an explicit round-to-nearest intrinsic in the reference's
// operation order, so the record rounds the same in a translation unit built
// with or without FMA contraction, and is bit-identical to the reference's
// childAvgFneq (src/sim/lbm_refine.cu:70-97) evaluated without contraction.
#pragma once

#include "d3q19.cuh"

#include <cuda_fp16.h>

namespace fcfd {

constexpr int kScratchVals = 24;   // per coarse cell: fneq[19], valid, rho, ux, uy, uz
constexpr int kScratchValid = 19;  // record layout: 6 float4, valid flag closes the fneq part
constexpr int kScratchRho = 20;

__device__ __forceinline__ float rn_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float rn_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rn_sub(float a, float b) { return __fsub_rn(a, b); }

// Terms whose lattice coefficient is 0 are left out of the sums below, and
// sums start from their first term: the same value for finite populations
// (the sign of a zero aside). What such terms do for an infinity or a NaN,
// which 0 times it passes on to every sum, is kept by one term 0 times the sum
// of all: a bad population, the rest one too, spoils the whole cell, and so
// travels on to where the watchdog looks.

/// Moments of fi with the density floor and the |u| <= 0.3 limiter.
__device__ __forceinline__ void limited_moments(const float (&fi)[kQ], float& rho, float& ux, float& uy,
                                                float& uz) {
    float r = fi[0], jx = fi[1], jy = fi[3], jz = fi[5];
#pragma unroll
    for (int q = 1; q < kQ; ++q) {
        r = rn_add(r, fi[q]);
        if (cx(q) != 0 && q != 1) jx = cx(q) > 0 ? rn_add(jx, fi[q]) : rn_sub(jx, fi[q]);
        if (cy(q) != 0 && q != 3) jy = cy(q) > 0 ? rn_add(jy, fi[q]) : rn_sub(jy, fi[q]);
        if (cz(q) != 0 && q != 5) jz = cz(q) > 0 ? rn_add(jz, fi[q]) : rn_sub(jz, fi[q]);
    }
    jx = __fmaf_rn(0.0f, r, jx); jy = __fmaf_rn(0.0f, r, jy); jz = __fmaf_rn(0.0f, r, jz);
    r = fmaxf(r, kRhoFloor);
    const float inv = 1.0f / r;
    ux = rn_mul(jx, inv); uy = rn_mul(jy, inv); uz = rn_mul(jz, inv);
    const float u2 = rn_add(rn_add(rn_mul(ux, ux), rn_mul(uy, uy)), rn_mul(uz, uz));
    if (u2 > kMaxSimSpeed * kMaxSimSpeed) {
        // The hardware rsqrtf of the reference's GPU build (lbm_refine.cu:238,
        // 309); only cells beyond |u| = 0.3 take this branch.
        const float sc = rn_mul(kMaxSimSpeed, rsqrtf(u2));
        ux = rn_mul(ux, sc); uy = rn_mul(uy, sc); uz = rn_mul(uz, sc);
    }
    rho = r;
}

/// c_q . u, the components in the order x, y, z.
__device__ __forceinline__ float dot_rn(int q, float ux, float uy, float uz) {
    float d = 0.0f;
    bool any = false;
    if (cx(q) != 0) { d = cx(q) > 0 ? ux : -ux; any = true; }
    if (cy(q) != 0) { const float t = cy(q) > 0 ? uy : -uy; d = any ? rn_add(d, t) : t; any = true; }
    if (cz(q) != 0) { const float t = cz(q) > 0 ? uz : -uz; d = any ? rn_add(d, t) : t; }
    return d;
}

/// Second-order equilibria (lbm_core.cu:65-73), operations in source order;
/// the two of an opposite pair share 0.5 (3 c.u)^2.
__device__ __forceinline__ void feq_rn(float rho, float ux, float uy, float uz, float (&feq)[kQ]) {
    const float usq = rn_mul(1.5f, rn_add(rn_add(rn_mul(ux, ux), rn_mul(uy, uy)), rn_mul(uz, uz)));
    feq[0] = rn_mul(rn_mul(wgt(0), rho), rn_sub(1.0f, usq));
#pragma unroll
    for (int p = 1; p <= 9; ++p) {
        const int a = 2 * p - 1;
        const float cu = rn_mul(3.0f, dot_rn(a, ux, uy, uz));
        const float h = rn_mul(rn_mul(0.5f, cu), cu), wr = rn_mul(wgt(a), rho);
        feq[a] = rn_mul(wr, rn_sub(rn_add(rn_add(1.0f, cu), h), usq));
        feq[a + 1] = rn_mul(wr, rn_sub(rn_add(rn_sub(1.0f, cu), h), usq));
    }
}

/// The scratch covers the restricted sub-box with a border of one cell in x
/// and y, so that every neighbour of a cell of the box has a record.
struct RecordGrid {
    int w = 0, h = 0;   // of the sub-box
    __host__ __device__ unsigned index(int lx, int ly, int z) const {
        return static_cast<unsigned>(lx + 1) + static_cast<unsigned>(w + 2)
             * (static_cast<unsigned>(ly + 1) + static_cast<unsigned>(h + 2) * static_cast<unsigned>(z));
    }
    __host__ __device__ long long count(int nz) const { return static_cast<long long>(w + 2) * (h + 2) * nz; }
};

/// Parts of a record, which the launch before wrote: ordinary loads behind the
/// wait, in the order of the source.
__device__ __forceinline__ float4 ld_rec(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ld_rec(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

/// The planes of the scratch (four or six of them), float4 k of record t at p[k][t].
struct RecordPlanes {
    const float4* p[kScratchVals / 4];
    __host__ static RecordPlanes of(const float* scratch, long long stride) {
        RecordPlanes r;
        for (int k = 0; k < kScratchVals / 4; ++k) r.p[k] = reinterpret_cast<const float4*>(scratch) + k * stride;
        return r;
    }
};

/// Layout of a coarse cell's record by storage. FP32 storage: fneq[19] in
/// FP32, the valid flag, rho, ux, uy, uz -- six float4 (96 B), so the
/// restriction is bit-identical to the reference's. FP16 storage: fneq[19]
/// as halves (the precision of the stored deviations), the valid flag and
/// rho, ux, uy, uz in FP32 -- four float4 (64 B); the restriction's 19
/// neighbour reads per coarse cell then move 48 B each instead of 80 B.
/// A record without fluid children, and the border's, holds -0 in fneq and 0
/// in the flag: adding it changes no sum (x + -0 is x for every x), so the
/// restriction adds all its neighbours without looking.
template <class S> struct ChildRecord;

template <> struct ChildRecord<StoreF32> {
    static constexpr int kVec = kScratchVals / 4;
    __device__ __forceinline__ static void write(float4* rec, long long st, const float (&fneq)[kQ], float rho,
                                                 float ux, float uy, float uz) {
        float r[kScratchVals];
#pragma unroll
        for (int q = 0; q < kQ; ++q) r[q] = fneq[q];
        r[kScratchValid] = 1.0f;
        r[kScratchRho] = rho; r[kScratchRho + 1] = ux; r[kScratchRho + 2] = uy; r[kScratchRho + 3] = uz;
#pragma unroll
        for (int k = 0; k < kVec; ++k) rec[k * st] = make_float4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
    }
    __device__ __forceinline__ static void write_invalid(float4* rec, long long st) {
#pragma unroll
        for (int k = 0; k < 4; ++k) rec[k * st] = make_float4(-0.0f, -0.0f, -0.0f, -0.0f);
        rec[4 * st] = make_float4(-0.0f, -0.0f, -0.0f, 0.0f);
    }
    /// A record's fneq and valid flag as stored.
    struct Raw { float4 a[5]; };
    __device__ __forceinline__ static void fetch(const RecordPlanes& r, unsigned t, Raw& w) {
#pragma unroll
        for (int k = 0; k < 5; ++k) w.a[k] = ld_rec(r.p[k] + t);
    }
    /// acc[q] += fneq[q], count += valid flag; SET: the record's own values.
    template <bool SET>
    __device__ __forceinline__ static void add(const Raw& w, float (&acc)[kQ], float& count) {
        const float4 (&a)[5] = w.a;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const float v[4] = {a[k].x, a[k].y, a[k].z, a[k].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int q = 4 * k + e;
                if (q < kQ) acc[q] = SET ? v[e] : acc[q] + v[e];
                else count = SET ? v[e] : count + v[e];
            }
        }
    }
    __device__ __forceinline__ static float4 moments(const RecordPlanes& r, unsigned t) {
        return ld_rec(r.p[kScratchRho / 4] + t);
    }
};

template <> struct ChildRecord<StoreF16> {
    static constexpr int kVec = 4;   // halves 0-7 | halves 8-15 | halves 16-18, valid | rho, u, v, w
    __device__ __forceinline__ static unsigned pack(float a, float b) {
        const __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<const unsigned*>(&h);
    }
    __device__ __forceinline__ static float2 unpack(unsigned u) {
        const __half2 h = *reinterpret_cast<const __half2*>(&u);
        return __half22float2(h);
    }
    __device__ __forceinline__ static void write(float4* rec, long long st, const float (&fneq)[kQ], float rho,
                                                 float ux, float uy, float uz) {
        uint4* r = reinterpret_cast<uint4*>(rec);
        r[0] = make_uint4(pack(fneq[0], fneq[1]), pack(fneq[2], fneq[3]), pack(fneq[4], fneq[5]),
                          pack(fneq[6], fneq[7]));
        r[st] = make_uint4(pack(fneq[8], fneq[9]), pack(fneq[10], fneq[11]), pack(fneq[12], fneq[13]),
                           pack(fneq[14], fneq[15]));
        r[2 * st] = make_uint4(pack(fneq[16], fneq[17]), pack(fneq[18], 0.0f), __float_as_uint(1.0f), 0u);
        rec[3 * st] = make_float4(rho, ux, uy, uz);
    }
    __device__ __forceinline__ static void write_invalid(float4* rec, long long st) {
        uint4* r = reinterpret_cast<uint4*>(rec);
        constexpr unsigned z = 0x80008000u;   // two halves of -0
        r[0] = make_uint4(z, z, z, z);
        r[st] = make_uint4(z, z, z, z);
        r[2 * st] = make_uint4(z, z, 0u, 0u);
    }
    struct Raw { uint4 c[3]; };
    __device__ __forceinline__ static void fetch(const RecordPlanes& r, unsigned t, Raw& w) {
#pragma unroll
        for (int k = 0; k < 3; ++k) w.c[k] = ld_rec(reinterpret_cast<const uint4*>(r.p[k]) + t);
    }
    template <bool SET>
    __device__ __forceinline__ static void add(const Raw& raw, float (&acc)[kQ], float& count) {
        const uint4 (&c)[3] = raw.c;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const unsigned w[4] = {c[k].x, c[k].y, c[k].z, c[k].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int q = 8 * k + 2 * j;
                if (q >= kQ) continue;
                const float2 v = unpack(w[j]);
                acc[q] = SET ? v.x : acc[q] + v.x;
                if (q + 1 < kQ) acc[q + 1] = SET ? v.y : acc[q + 1] + v.y;
            }
        }
        count = SET ? __uint_as_float(c[2].z) : count + __uint_as_float(c[2].z);
    }
    __device__ __forceinline__ static float4 moments(const RecordPlanes& r, unsigned t) { return ld_rec(r.p[3] + t); }
};

/// Record of a coarse cell from the sum fi of its nFluid fluid children
/// (sums of the deviations f - w_q when DEV), at rec = base + t of a planar
/// scratch of stride st.
template <class S, bool DEV = false>
__device__ __forceinline__ void write_child_record(float (&fi)[kQ], int nFluid, float4* rec, long long st) {
    if (nFluid == 0) {
        ChildRecord<S>::write_invalid(rec, st);
        return;
    }
    const float invN = 1.0f / static_cast<float>(nFluid);
#pragma unroll
    for (int q = 0; q < kQ; ++q) fi[q] = DEV ? rn_mul(fi[q], invN) + wgt(q) : rn_mul(fi[q], invN);
    float rho, ux, uy, uz;
    limited_moments(fi, rho, ux, uy, uz);
    float fneq[kQ];
    feq_rn(rho, ux, uy, uz, fneq);
#pragma unroll
    for (int q = 0; q < kQ; ++q) fneq[q] = rn_sub(fi[q], fneq[q]);
    ChildRecord<S>::write(rec, st, fneq, rho, ux, uy, uz);
}

} // namespace fcfd
