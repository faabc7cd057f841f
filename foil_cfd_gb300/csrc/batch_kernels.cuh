// Batched stream-collide: one launch steps every tunnel of a batch (or of a
// group of its tunnels: a contiguous range of work items).
//
// The grid walks a flat list of work items -- for each tunnel, tiles of 128
// cells of the flattened lattice, or its rows (y, z) in groups of `ROWS`,
// whose cells the block's BX threads stride through along x (the item decode
// is paid once per row) -- with a
// block-stride loop, so a grid of a few blocks per SM is persistent across
// all tunnels of unequal size, and a grid of one block per item is an
// ordinary launch. The tunnel table is a __grid_constant__ kernel parameter
// (constant bank): a block finds an item's tunnel by binary search over the
// tunnels' first items and reads that tunnel's parameters from the bank with
// a uniform index. Item decoding is 32-bit. Every cell runs the same per-cell
// update as the single-tunnel kernels (collide_one), so a batch produces the
// same populations, bit for bit, as stepping each tunnel on its own with the
// same collision body. Items of a tunnel whose watchdog latch is set are
// skipped: a diverged tunnel stops where it tripped.
#pragma once

#include "batch_types.h"
#include "collide_common.cuh"

#include <algorithm>

namespace fcfd {
namespace {

// Register cap per storage: S::kBatchThreads resident threads per SM.
template <class S, bool EXACT, int BX, int ROWS>
__global__ void __launch_bounds__(BX, S::kBatchThreads / BX)
batch_collide_kernel(const __grid_constant__ BatchTable P, unsigned itemBase, unsigned nItems, int parity) {
    pdl_wait();
    using T = typename S::T;
    // FP32: the near-wall gather reads the cells' link words (batch step
    // 1.054 -> 0.950 ms on the polar); FP16: the same path at the 64-register
    // cap spilled more and measured 3 % slower, so it reads the neighbours'
    // flags.
    constexpr bool kLinkWall = std::is_same_v<S, StoreF32>;
    const unsigned itemEnd = itemBase + nItems;
    for (unsigned item = itemBase + blockIdx.x; item < itemEnd; item += gridDim.x) {
        int lo = 0, hi = P.ntun - 1;
        while (lo < hi) {  // last tunnel whose first item <= item
            const int mid = (lo + hi + 1) >> 1;
            if (P.begins[mid] <= item) lo = mid;
            else hi = mid - 1;
        }
        if (P.latch && P.latch[lo] != 0) continue;   // a latched tunnel no longer steps
        const BatchTunnelParam& tp = P.t[lo];
        CollideArgs a;
        a.nx = tp.nx; a.ny = tp.ny; a.nz = tp.nz; a.n = tp.n;
        a.tau0 = tp.tau; a.lambda = P.lambda; a.smagPre = P.smagPre; a.uIn = tp.uIn;
        a.writeMacro = 0;
        a.rho = a.u = a.v = a.w = nullptr;
        a.uwx = a.uwy = a.uwz = nullptr;
        a.status = nullptr;
        a.qFrac = nullptr;
        a.links = tp.links;
        a.ffMask = nullptr;
        const T* src = static_cast<const T*>(tp.f[parity]);
        T* dst = static_cast<T*>(tp.f[parity ^ 1]);
        const unsigned ny = static_cast<unsigned>(tp.ny);
        const unsigned rows = ny * static_cast<unsigned>(tp.nz);
        const unsigned row0 = (item - P.begins[lo]) * ROWS;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const unsigned row = row0 + r;
            if (row >= rows) break;
            const unsigned z = row / ny;
            const int y = static_cast<int>(row - z * ny);
            for (int x = threadIdx.x; x < tp.nx; x += BX)
                collide_one<S, false, EXACT, false, kLinkWall>(src, dst, tp.kind, a, x, y, static_cast<int>(z));
        }
    }
}

// ---- tiles of the flattened lattice ------------------------------------------------
// The cells of the row kernel each decode their coordinates, read their kind
// byte and form 19 wrapped indices: 667 instructions a cell with FP16 storage,
// 43 % of the HBM rate. Here a warp of 32 bulk cells (one code byte) pulls by
// its tunnel's constant offsets, also in the two z planes, whose wrap is one
// more constant (an eighth of a 16-cell span); with 16-bit populations a block
// of such warps stages its runs as collide_tile_kernel does; and in the other
// warps (10 %, nearly all at a row's end) the bulk cells take the offsets too.
// 100 steps of the 24-tunnel polar (31.9 M cells), FP16, 69.4 -> 61.3 ms, of
// which near-wall cells take 2.6 ms and inlets and outlets 3.3; 12 tunnels
// FP32 41.3 -> 36.6 ms. The tunnel of an item comes from a table of starting
// points: a binary search took 4 ms of the 100 steps.

/// Cells to add to a pull of q that wraps around z (lowZ, highZ: the lattice's
/// cells in plane 0 and in the last one, else 0).
__device__ __forceinline__ int z_wrap(int q, int lowZ, int highZ) {
    return cz(q) > 0 ? lowZ : cz(q) < 0 ? -highZ : 0;
}

constexpr unsigned slices_of_cz(int v) {
    unsigned m = 0;
    for (int q = 0; q < kQ; ++q) m |= (cz(q) == v ? 1u : 0u) << q;
    return m;
}

template <class S, bool EXACT>
__global__ void __launch_bounds__(kTile, S::kBatchTileMinBlocks)
batch_tile_kernel(const __grid_constant__ BatchTable P, unsigned itemBase, unsigned nItems, int parity) {
    using T = typename S::T;
    using Pp = Pop<S, !EXACT>;
    constexpr bool kStages = sizeof(T) == 2;
    constexpr bool kLinkWall = std::is_same_v<S, StoreF32>;   // as in the row kernel
    __shared__ __align__(16) unsigned char tile[kStages ? kQ * kTileRow : 16];
    const unsigned t = threadIdx.x, tb = smem_addr(tile);
    pdl_wait();
    const unsigned itemEnd = itemBase + nItems;
    for (unsigned item = itemBase + blockIdx.x; item < itemEnd; item += gridDim.x) {
        if ((item & 7) == 0 && t == 0 && item + kCodesAhead < itemEnd)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(P.tiles + item + kCodesAhead));
        const std::uint32_t word = P.tiles[item];
        int lo = P.tunnelAt[item >> P.itemShift];
        while (P.begins[lo + 1] <= item) ++lo;
        const int latched = P.latch ? P.latch[lo] : 0;
        const BatchTunnelParam& tp = P.t[lo];
        const unsigned c0 = (item - P.begins[lo]) * kTile, cell = c0 + t;
        if (word == 0 || latched != 0) continue;   // idle cells; a latched tunnel no longer steps
        CollideArgs a;
        a.nx = tp.nx; a.ny = tp.ny; a.nz = tp.nz; a.n = tp.n;
        a.tau0 = tp.tau; a.lambda = P.lambda; a.smagPre = P.smagPre; a.uIn = tp.uIn;
        a.writeMacro = 0;
        a.rho = a.u = a.v = a.w = nullptr;
        a.uwx = a.uwy = a.uwz = nullptr;
        a.status = nullptr;
        a.qFrac = nullptr;
        a.links = tp.links;
        a.ffMask = nullptr;
        const T* src = static_cast<const T*>(tp.f[parity]);
        T* dst = static_cast<T*>(tp.f[parity ^ 1]);
        const int n = static_cast<int>(tp.n), code = static_cast<int>(word >> (8 * (t >> 5))) & 0xff;
        int lowZ = code == kTileLowZ ? n : 0, highZ = code == kTileHighZ ? n : 0;
        float f[kQ];
        // n a multiple of 8: a z wrap leaves the runs' alignment as it is,
        // and the results go back in whole pieces.
        const bool staged = kStages && n % 8 == 0 && code >= kTileBulk && word == static_cast<unsigned>(code) * 0x01010101u;
        if (staged) {
            if (item != itemBase + blockIdx.x) __syncthreads();   // the last item's results are read
            constexpr unsigned kUp = slices_of_cz(1), kDown = slices_of_cz(-1);
            auto chunk = [&](unsigned q, unsigned c) {
                int p = tp.pull[q];
                if ((kUp >> q) & 1u) p += lowZ;
                if ((kDown >> q) & 1u) p -= highZ;
                asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;" ::"r"(tb + q * kTileRow + 16 * c),
                             "l"(src + ((p & ~7) + static_cast<int>(c0 + 8 * c)))
                             : "memory");
            };
#pragma unroll
            for (int j = 0; j < 3; ++j) {   // as tile_in
                const unsigned i = t + kTile * j, q = i >> 4;
                if (q < kQ) chunk(q, i & 15);
            }
            if (t >= 64 && t < 64 + kQ) chunk(t - 64, 16);
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
            __syncthreads();
#pragma unroll
            for (int q = 0; q < kQ; ++q) f[q] = Pp::lds(tb + tp.inOff[q], t, wgt(q));
        } else {
            bool pulls = code >= kTileBulk;
            if (!pulls) {
                if (code == kTileIdle || cell >= static_cast<unsigned>(n)) continue;
                const std::uint8_t k = tp.kind[cell];
                const unsigned row = fdiv(cell, tp.divX), zu = fdiv(row, tp.divY);
                const int x = static_cast<int>(cell - row * tp.divX.d), y = static_cast<int>(row - zu * tp.divY.d);
                const int z = static_cast<int>(zu), flag = k & kFlagMask;
                if (flag != kFluid) {
                    boundary_cell<S>(src, dst, a, flag, cell, x, y, z);
                    continue;
                }
                pulls = !(k & kNearWall) && x > 0 && x < a.nx - 1 && y > 0 && y < a.ny - 1 && a.nz > 1;
                lowZ = z == 0 ? n : 0;
                highZ = z == a.nz - 1 ? n : 0;
                if (!pulls) gather_fluid<S, false, false, !EXACT, kLinkWall>(src, tp.kind, a, k, cell, x, y, z, f, nullptr);
            }
            if (pulls) {
#pragma unroll
                for (int q = 0; q < kQ; ++q)
                    f[q] = Pp::ld(src, static_cast<int>(cell) + (tp.pull[q] + z_wrap(q, lowZ, highZ)), wgt(q));
            }
        }
        float r, ux, uy, uz;
        collide_body<EXACT>(f, a, r, ux, uy, uz);
        if (staged) {
            __syncthreads();
#pragma unroll
            for (int q = 0; q < kQ; ++q) Pp::st(reinterpret_cast<T*>(tile + q * kTileRow), t, f[q], wgt(q));
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const unsigned i = t + kTile * j, q = i >> 4, c = i & 15;
                if (q < kQ)
                    *reinterpret_cast<uint4*>(dst + static_cast<int>(q * n + c0 + 8 * c)) =
                        *reinterpret_cast<const uint4*>(tile + q * kTileRow + 16 * c);
            }
        } else {
            store_cell<S, !EXACT>(dst, a, cell, f, nullptr);
        }
    }
}

template <class S, bool EXACT, int BX, int ROWS>
cudaError_t launch_batch_shape(const BatchTable& tab, unsigned itemBase, unsigned nItems, int parity, int grid,
                               cudaStream_t st) {
    const unsigned g = grid > 0 ? std::min<unsigned>(static_cast<unsigned>(grid), nItems) : nItems;
    if (g == 0) return cudaSuccess;
    if constexpr (BX == kTile && ROWS == 1)
        return launch_pdl(batch_tile_kernel<S, EXACT>, g, BX, st, tab, itemBase, nItems, parity);
    else
        return launch_pdl(batch_collide_kernel<S, EXACT, BX, ROWS>, g, BX, st, tab, itemBase, nItems, parity);
}

template <class S, bool EXACT, int BX, int ROWS>
int batch_occupancy_shape() {
    int b = 0;
    if constexpr (BX == kTile && ROWS == 1)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, batch_tile_kernel<S, EXACT>, BX, 0);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, batch_collide_kernel<S, EXACT, BX, ROWS>, BX, 0);
    return b;
}

#define FCFD_BATCH_SHAPES(X) \
    X(64, 1) X(64, 2) X(64, 4) X(128, 1) X(128, 2) X(128, 4) X(256, 1) X(256, 2) X(256, 4)

template <class S, bool EXACT>
cudaError_t launch_batch_impl(const BatchTable& tab, unsigned itemBase, unsigned nItems, int parity, BatchShape sh,
                              cudaStream_t st) {
    if (tab.ntun <= 0 || tab.ntun > kMaxBatchTunnels) return cudaErrorInvalidValue;
#define FCFD_BATCH_CASE(B, R) \
    if (sh.block == B && sh.rows == R) return launch_batch_shape<S, EXACT, B, R>(tab, itemBase, nItems, parity, sh.grid, st);
    FCFD_BATCH_SHAPES(FCFD_BATCH_CASE)
#undef FCFD_BATCH_CASE
    return cudaErrorInvalidValue;
}

template <class S, bool EXACT>
int batch_occupancy_impl(BatchShape sh) {
#define FCFD_BATCH_OCC(B, R) \
    if (sh.block == B && sh.rows == R) return batch_occupancy_shape<S, EXACT, B, R>();
    FCFD_BATCH_SHAPES(FCFD_BATCH_OCC)
#undef FCFD_BATCH_OCC
    return 0;
}

} // namespace
} // namespace fcfd
