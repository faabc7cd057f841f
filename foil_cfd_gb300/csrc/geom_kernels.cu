// On-device geometry builders: the flag fields, patch box and cell lists the
// solver keys off, built where they are used instead of on the host.
//
// * Airfoil rasterisation (src/geom/voxelizer.cpp:62-153, voxelizeAirfoil):
//   the outline rotated about the quarter chord and scaled to the anchor,
//   one warp per lattice row intersecting the row's cell-centre line with
//   every edge under the half-open rule, the crossings sorted, and the
//   cells between crossing pairs marked in a 2-D mask.
// * Flag field (buildBoundaryFlags, closeTrailingEdgeGaps, stampInterfaceShell,
//   voxelizer.cpp:28-60, 155-183, 223-245): one thread per cell evaluates the
//   base flag (domain faces, all fluid or an input field), the extruded mask
//   over fluid, the single-cell trailing-edge closure judged on the
//   pre-closure field (the +-y neighbours' pre-closure flags are recomputed,
//   so the pass is out of place without a copy) and the interface shell.
// * Patch box (derivePatchBox, voxelizer.cpp:265-301): a min/max reduction
//   of the solid cells' x and y.
// * Bit planes: one bit per cell and property (solid, fluid, ...), 32 cells of
//   a row per word, built once per flag field. What depends on a cell's
//   neighbours is then word arithmetic on 32 cells at a time.
// * Level tables: kind bytes, pull-link classes, tile codes, cell classes and
//   the solid bounding box of a level.
// * Cell lists in ascending cell order: selection words, one scan over the
//   tiles of 256 words, the selected cells, then one thread per entry for what
//   an entry holds: the force-link list, the wall-model cell list of
//   buildWallCellList (src/sim/wall_model.cpp:55-236: pull-solid link mask,
//   vane exclusion, 5^3 occupancy-gradient normal, sample cell along the
//   normal) and the interface-shell list of a refined level.
//
// Built without FMA contraction: the rasteriser's crossings and the wall
// normals are the host builders' values bit for bit.
#include <cuda_runtime.h>

#include <cstdint>

#include "d3q19.cuh"
#include "kernels.h"

namespace fcfd {
namespace {

constexpr std::uint8_t kFluidB = 0, kSolidB = 1, kInletB = 2, kOutletB = 3, kSlipTopB = 4, kSlipBottomB = 5;
constexpr std::uint8_t kInterfaceB = 8, kOutletEqB = 9;
constexpr int kMaxCrossings = 64;      // per lattice row; more sets the error flag
constexpr int kRowWarps = 4;           // rows per block of the rasteriser

/// Periodic index for any offset (a sample search can step several
/// periods on a thin span); equals the single wrap wherever that is in range.
__device__ __forceinline__ int wrapi(int v, int n) {
    if (static_cast<unsigned>(v) < static_cast<unsigned>(n)) return v;
    const int r = v % n;
    return r < 0 ? r + n : r;
}

// ---- rasteriser -------------------------------------------------------------

__global__ void foil_poly_kernel(const float* __restrict__ xy, int npts, float c, float s, float chord, float ax,
                                 float ay, float* __restrict__ px, float* __restrict__ py) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npts) return;
    // p - (0.25, 0), rotated by the angle whose cosine/sine are c/s, scaled, anchored.
    const float rx = xy[2 * i] - 0.25f, ry = xy[2 * i + 1] - 0.0f;
    const float qx = rx * c - ry * s, qy = rx * s + ry * c;
    px[i] = ax + qx * chord;
    py[i] = ay + qy * chord;
}

__global__ void __launch_bounds__(kRowWarps * 32)
foil_rows_kernel(const float* __restrict__ px, const float* __restrict__ py, int npts, int nx, int ny,
                 std::uint8_t* __restrict__ mask, int* __restrict__ err) {
    __shared__ float cr[kRowWarps][kMaxCrossings];
    __shared__ float srt[kRowWarps][kMaxCrossings];
    __shared__ int span[kRowWarps][kMaxCrossings];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int y = blockIdx.x * kRowWarps + warp;
    if (y >= ny) return;
    std::uint8_t* row = mask + static_cast<long long>(y) * nx;
    int m = 0;
    if (y >= 1 && y <= ny - 2) {
        const float yc = static_cast<float>(y) + 0.5f;
        for (int base = 0; base < npts; base += 32) {
            const int i = base + lane;
            bool hit = false;
            float xc = 0.0f;
            if (i < npts) {
                const int j = i + 1 == npts ? 0 : i + 1;
                const float ya = py[i], yb = py[j];
                if ((ya > yc) != (yb > yc)) {
                    const float t = (yc - ya) / (yb - ya);
                    xc = px[i] + t * (px[j] - px[i]);
                    hit = true;
                }
            }
            const unsigned b = __ballot_sync(0xffffffffu, hit);
            const int slot = m + __popc(b & ((1u << lane) - 1u));
            if (hit && slot < kMaxCrossings) cr[warp][slot] = xc;
            m += __popc(b);
        }
        if (m > kMaxCrossings) {
            if (lane == 0) atomicExch(err, 1);
            m = 0;
        }
    }
    __syncwarp();
    // Rank sort (ties broken by edge order) of the crossings.
    for (int k = lane; k < m; k += 32) {
        const float v = cr[warp][k];
        int r = 0;
        for (int j = 0; j < m; ++j) {
            const float u = cr[warp][j];
            r += (u < v) || (u == v && j < k);
        }
        srt[warp][r] = v;
    }
    __syncwarp();
    const int pairs = m / 2;
    for (int k = lane; k < pairs; k += 32) {
        const int xa = max(1, static_cast<int>(ceilf(srt[warp][2 * k] - 0.5f)));
        const int xb = min(nx - 2, static_cast<int>(floorf(srt[warp][2 * k + 1] - 0.5f)));
        span[warp][2 * k] = xa;
        span[warp][2 * k + 1] = xb;
    }
    __syncwarp();
    for (int x = lane; x < nx; x += 32) {
        bool in = false;
        for (int k = 0; k < pairs; ++k) in |= (x >= span[warp][2 * k]) && (x <= span[warp][2 * k + 1]);
        row[x] = in ? 1 : 0;
    }
}

// ---- flag field -------------------------------------------------------------

struct FlagBuild {
    int nx, ny, nz;
    int base;                          // 0 domain faces, 1 all fluid, 2 input field
    const std::uint8_t* in;            // base 2
    const std::uint8_t* mask;          // nx*ny rasterised foil, or null
    int closeGaps;
    int shell;                         // interface-shell width, 0 for none
};

__device__ __forceinline__ std::uint8_t base_flag(const FlagBuild& b, long long cell, int x, int y) {
    if (b.base == 2) return b.in[cell];
    if (b.base == 1) return kFluidB;
    // buildBoundaryFlags: slip faces, the inlet wins the x = 0 corners, the
    // outlet yields to the slip faces.
    std::uint8_t f = kFluidB;
    if (y == 0) f = kSlipBottomB;
    if (y == b.ny - 1) f = kSlipTopB;
    if (x == 0) f = kInletB;
    else if (x == b.nx - 1 && y != 0 && y != b.ny - 1) f = kOutletB;
    return f;
}

__device__ __forceinline__ std::uint8_t voxel_flag(const FlagBuild& b, long long cell, int x, int y) {
    const std::uint8_t f = base_flag(b, cell, x, y);
    if (b.mask && f == kFluidB && b.mask[static_cast<long long>(y) * b.nx + x]) return kSolidB;
    return f;
}

/// A thread has one (x, y) over a run of planes: only an input field (base 2)
/// varies along z, all else is worked out once. Cell by cell the two 64-bit
/// divisions and the tests of three cells took 182 instructions each: 41.7
/// million cells 184 us, 32 by columns.
constexpr int kFlagRun = 16;
__global__ void __launch_bounds__(256)
build_flags_kernel(FlagBuild b, std::uint8_t* __restrict__ out, int* __restrict__ closed) {
    const unsigned plane = static_cast<unsigned>(b.nx) * static_cast<unsigned>(b.ny);
    const unsigned c = blockIdx.x * 256u + threadIdx.x;
    int count = 0;
    if (c < plane) {
        const int y = static_cast<int>(c / static_cast<unsigned>(b.nx)), x = static_cast<int>(c - y * static_cast<unsigned>(b.nx));
        const int z0 = blockIdx.y * kFlagRun, z1 = min(z0 + kFlagRun, b.nz);
        std::uint8_t f = 0;
        bool close = false;
        for (int z = z0; z < z1; ++z) {
            const long long cell = c + static_cast<long long>(z) * plane;
            if (z == z0 || b.base == 2) {
                f = voxel_flag(b, cell, x, y);
                close = b.closeGaps && y >= 1 && y <= b.ny - 2 && f == kFluidB
                        && voxel_flag(b, cell - b.nx, x, y - 1) == kSolidB && voxel_flag(b, cell + b.nx, x, y + 1) == kSolidB;
                if (close) f = kSolidB;
                if (b.shell > 0 && (y < b.shell || y >= b.ny - b.shell || x < b.shell || x >= b.nx - b.shell))
                    f = kInterfaceB;
            }
            count += close;
            out[cell] = f;
        }
    }
    count = __reduce_add_sync(0xffffffffu, count);
    if (count && (threadIdx.x & 31) == 0) atomicAdd(closed, count);
}

/// Flags of a new field, in place, to the edit mask against the kind bytes of
/// the old one (1 newly solid, 2 newly fluid), four cells a thread, and the
/// number of edits.
__global__ void __launch_bounds__(256)
flag_diff_kernel(const std::uint8_t* __restrict__ kind, std::uint8_t* __restrict__ mask, unsigned n,
                 unsigned long long* __restrict__ count) {
    const unsigned i = 4u * (blockIdx.x * 256u + threadIdx.x);
    int edits = 0;
    if (i < n) {   // both arrays go on to a multiple of four
        const std::uint32_t was = __vcmpeq4(*reinterpret_cast<const std::uint32_t*>(kind + i) & 0x0f0f0f0fu, 0x01010101u * kSolidB);
        std::uint32_t now = __vcmpeq4(*reinterpret_cast<const std::uint32_t*>(mask + i), 0x01010101u * kSolidB);
        if (n - i < 4) now = (now & (0xffffffffu >> (32 - 8 * (n - i)))) | (was & ~(0xffffffffu >> (32 - 8 * (n - i))));
        edits = __popc(was ^ now) / 8;
        *reinterpret_cast<std::uint32_t*>(mask + i) = (now & ~was & 0x01010101u) | (was & ~now & 0x02020202u);
    }
    edits = __reduce_add_sync(0xffffffffu, edits);
    if (edits && (threadIdx.x & 31) == 0) atomicAdd(count, static_cast<unsigned long long>(edits));
}

// ---- bit planes -----------------------------------------------------------------
// The old builders tested 18 neighbour bytes per cell, a thread running through
// 16 cells one after the other: 0.56 ms per pass over a 42 M-cell patch. A word
// of a plane holds 32 cells of a row, so the same test is about 20 loads and
// 60 operations for 32 cells, and the planes of that patch (5.3 MB each) stay
// in L2.

struct BitGrid {
    int nx, ny, nz, words;   // words per row
    __host__ __device__ unsigned total() const {
        return static_cast<unsigned>(words) * static_cast<unsigned>(ny) * static_cast<unsigned>(nz);
    }
};
BitGrid bit_grid(LevelDims d) { return BitGrid{d.nx, d.ny, d.nz, (d.nx + 31) / 32}; }

enum Plane { kPSolid, kPFluid, kPSlip, kPInlet, kPOutlet, kPInter, kPlanes };
struct Planes {
    std::uint32_t* p[kPlanes];   // null: not wanted
};

/// Four cells' matches of one byte value as four bits.
__device__ __forceinline__ std::uint32_t match4(std::uint32_t cells, std::uint32_t value) {
    return ((__vcmpeq4(cells, value * 0x01010101u) & 0x01010101u) * 0x10204080u) >> 28;
}

/// One thread per word. ALIGN: bytes a row's words start on (16, 4 or 1).
/// keep: the bits of a flag byte that count (the step looks at the low four).
template <int ALIGN>
__global__ void __launch_bounds__(256)
planes_kernel(const std::uint8_t* __restrict__ flags, BitGrid g, Planes P, std::uint32_t keep) {
    const unsigned wi = blockIdx.x * 256u + threadIdx.x;
    if (wi >= g.total()) return;
    const unsigned row = wi / g.words, x0 = 32u * (wi - row * g.words);
    const std::uint8_t* f = flags + static_cast<size_t>(row) * g.nx + x0;
    const int valid = min(32, g.nx - static_cast<int>(x0));
    std::uint32_t c[8];
    if (ALIGN == 16 && valid == 32) {
        const uint4 a = reinterpret_cast<const uint4*>(f)[0], b = reinterpret_cast<const uint4*>(f)[1];
        c[0] = a.x; c[1] = a.y; c[2] = a.z; c[3] = a.w;
        c[4] = b.x; c[5] = b.y; c[6] = b.z; c[7] = b.w;
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            c[k] = 0xffffffffu;
            if (ALIGN >= 4 && 4 * k + 4 <= valid) {
                c[k] = reinterpret_cast<const std::uint32_t*>(f)[k];
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (4 * k + e < valid)
                        c[k] = (c[k] & ~(0xffu << (8 * e))) | (static_cast<std::uint32_t>(f[4 * k + e]) << (8 * e));
            }
        }
    }
    std::uint32_t w[kPlanes] = {};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        c[k] &= keep;
        w[kPSolid] |= match4(c[k], kSolidB) << (4 * k);
        w[kPFluid] |= match4(c[k], kFluidB) << (4 * k);
        w[kPInlet] |= match4(c[k], kInletB) << (4 * k);
        w[kPOutlet] |= (match4(c[k], kOutletB) | match4(c[k], kOutletEqB)) << (4 * k);
        w[kPInter] |= match4(c[k], kInterfaceB) << (4 * k);
        w[kPSlip] |= match4(c[k] & 0xfcfcfcfcu, kSlipTopB) << (4 * k);   // 4..7
    }
#pragma unroll
    for (int p = 0; p < kPlanes; ++p)
        if (P.p[p]) P.p[p][wi] = w[p];
}

/// Word w of row (y, z) of a plane with its neighbours x - 1 and x + 1.
/// WRAPX: periodic in x; otherwise nothing beyond the faces.
struct Word3 {
    std::uint32_t mid, xm, xp;   // bit i: cell 32 w + i, the cell before it, the cell after it
};
template <bool WRAPX, class F>
__device__ __forceinline__ Word3 word3(const F& at, const BitGrid& g, unsigned rowWord, int w) {
    Word3 r;
    r.mid = at(rowWord + w);
    const int last = g.words - 1, valid = min(32, g.nx - 32 * w);
    std::uint32_t before = 0, after = 0;
    if (w > 0) before = at(rowWord + w - 1) >> 31;
    else if (WRAPX) before = (at(rowWord + last) >> ((g.nx - 1) & 31)) & 1u;
    if (w < last) after = at(rowWord + w + 1) & 1u;
    else if (WRAPX) after = at(rowWord) & 1u;
    r.xm = (r.mid << 1) | before;
    r.xp = (r.mid >> 1) | (after << (valid - 1));
    return r;
}

/// Cells of word w of row (y, z) with a set cell among their 18 neighbours.
/// WRAPXY: periodic in x and y; otherwise nothing beyond those faces. z is
/// periodic.
template <bool WRAPXY, class F>
__device__ __forceinline__ std::uint32_t near18(const F& at, const BitGrid& g, int w, int y, int z) {
    std::uint32_t any = 0;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz) {
        const int Z = wrapi(z + dz, g.nz);
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy) {
            int Y = y + dy;
            if (WRAPXY) Y = wrapi(Y, g.ny);
            else if (Y < 0 || Y >= g.ny) continue;
            const unsigned rw = (static_cast<unsigned>(Z) * g.ny + Y) * g.words;
            if (dy != 0 && dz != 0) {
                any |= at(rw + w);
            } else {
                const Word3 r = word3<WRAPXY>(at, g, rw, w);
                any |= r.xm | r.xp | (dy != 0 || dz != 0 ? r.mid : 0u);
            }
        }
    }
    return any;
}

struct OnePlane {
    const std::uint32_t* p;
    __device__ __forceinline__ std::uint32_t operator()(unsigned i) const { return __ldg(p + i); }
};
struct OrPlanes {
    const std::uint32_t *p, *q;
    __device__ __forceinline__ std::uint32_t operator()(unsigned i) const { return __ldg(p + i) | __ldg(q + i); }
};
struct AndNotPlanes {
    const std::uint32_t *p, *q;
    __device__ __forceinline__ std::uint32_t operator()(unsigned i) const { return __ldg(p + i) & ~__ldg(q + i); }
};

__device__ __forceinline__ void word_of(const BitGrid& g, unsigned wi, int& w, int& y, int& z) {
    const unsigned row = wi / g.words;
    w = static_cast<int>(wi - row * g.words);
    z = static_cast<int>(row / g.ny);
    y = static_cast<int>(row - static_cast<unsigned>(z) * g.ny);
}

// ---- classes and bounding box ------------------------------------------------------

/// counts: cells read and written by a step, inlets, the others' complement is
/// formed by the host; box: min/max of the solid cells' x and y.
__global__ void __launch_bounds__(256)
classes_kernel(Planes P, BitGrid g, unsigned long long* __restrict__ counts, int* __restrict__ box) {
    unsigned long long rw = 0, in = 0;
    int x0 = g.nx, x1 = -1, y0 = g.ny, y1 = -1;
    for (unsigned i = blockIdx.x * 256u + threadIdx.x; i < g.total(); i += gridDim.x * 256u) {
        if (counts) {
            rw += __popc(P.p[kPFluid][i]) + __popc(P.p[kPOutlet][i]);
            in += __popc(P.p[kPInlet][i]);
        }
        const std::uint32_t s = P.p[kPSolid][i];
        if (s) {
            int w, y, z;
            word_of(g, i, w, y, z);
            x0 = min(x0, 32 * w + __ffs(static_cast<int>(s)) - 1);
            x1 = max(x1, 32 * w + 31 - __clz(static_cast<int>(s)));
            y0 = min(y0, y);
            y1 = max(y1, y);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        rw += __shfl_xor_sync(0xffffffffu, rw, o);
        in += __shfl_xor_sync(0xffffffffu, in, o);
        x0 = min(x0, __shfl_xor_sync(0xffffffffu, x0, o));
        x1 = max(x1, __shfl_xor_sync(0xffffffffu, x1, o));
        y0 = min(y0, __shfl_xor_sync(0xffffffffu, y0, o));
        y1 = max(y1, __shfl_xor_sync(0xffffffffu, y1, o));
    }
    if ((threadIdx.x & 31) == 0) {
        if (counts && rw) atomicAdd(counts + 0, rw);
        if (counts && in) atomicAdd(counts + 1, in);
        if (x1 >= 0) {
            atomicMin(box + 0, x0); atomicMax(box + 2, x1);
            atomicMin(box + 1, y0); atomicMax(box + 3, y1);
        }
    }
}

// ---- kind bytes, pull-link classes, tile codes -------------------------------------

/// kind = flag | kNearWall for fluid cells with a solid or slip pull
/// neighbour; links (when given): the classes of those cells' 18 pull links
/// (kernels.h; the other cells' words are read by nothing and not written).
/// One thread per word; the links of a word by its warp, one cell per lane.
/// ALIGN 4: rows of whole 4-byte words. (41.7 million cells in rows that are
/// not: 245 us byte by byte, 119 word by word.)
template <int ALIGN>
__global__ void __launch_bounds__(256)
classify_kernel(const std::uint8_t* __restrict__ flags, Planes P, BitGrid g, std::uint8_t* __restrict__ kind,
                uint2* __restrict__ links) {
    const unsigned wi = blockIdx.x * 256u + threadIdx.x, lane = threadIdx.x & 31;
    std::uint32_t near = 0;
    unsigned c0 = 0;
    int valid = 0;
    if (wi < g.total()) {
        int w, y, z;
        word_of(g, wi, w, y, z);
        const std::uint32_t fluid = P.p[kPFluid][wi];
        if (fluid) near = fluid & near18<true>(OrPlanes{P.p[kPSolid], P.p[kPSlip]}, g, w, y, z);
        c0 = (static_cast<unsigned>(z) * g.ny + y) * g.nx + 32u * w;
        valid = min(32, g.nx - 32 * w);
    }
    if constexpr (ALIGN >= 4) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const std::uint32_t add = ((((near >> (4 * k)) & 15u) * 0x00204081u) & 0x01010101u) << 7;
            if (4 * k + 4 <= valid)
                reinterpret_cast<std::uint32_t*>(kind + c0)[k] =
                    (reinterpret_cast<const std::uint32_t*>(flags + c0)[k] & 0x0f0f0f0fu) | add;
        }
    } else {   // word by word, a cell per lane: byte by byte each lane's accesses were a line of their own
        for (int src = 0; src < 32; ++src) {
            const unsigned c = __shfl_sync(0xffffffffu, c0, src) + lane;
            const std::uint32_t nw = __shfl_sync(0xffffffffu, near, src);
            if (static_cast<int>(lane) < __shfl_sync(0xffffffffu, valid, src))
                kind[c] = static_cast<std::uint8_t>((flags[c] & kFlagMask) | (nw >> lane & 1u) << 7);
        }
    }
    if (!links) return;
    for (unsigned todo = __ballot_sync(0xffffffffu, near != 0); todo; todo &= todo - 1) {
        const int src = __ffs(static_cast<int>(todo)) - 1;
        const std::uint32_t nw = __shfl_sync(0xffffffffu, near, src);
        if (!(nw >> lane & 1u)) continue;
        int w, y, z;
        word_of(g, wi - lane + src, w, y, z);
        const int x = 32 * w + static_cast<int>(lane);
        unsigned long long m = 0;
#pragma unroll
        for (int q = 1; q < kQ; ++q) {
            const int X = wrapi(x - cx(q), g.nx), Y = wrapi(y - cy(q), g.ny), Z = wrapi(z - cz(q), g.nz);
            const int nf = flags[(static_cast<size_t>(Z) * g.ny + Y) * g.nx + X] & kFlagMask;
            if (nf == kSolid) m |= 1ull << (q - 1);
            if (is_slip_y(nf)) m |= 1ull << (17 + q);
            if (is_slip_z(nf)) m |= 1ull << (35 + q);
        }
        links[(static_cast<size_t>(z) * g.ny + y) * g.nx + x] =
            make_uint2(static_cast<unsigned>(m), static_cast<unsigned>(m >> 32));
    }
}

/// Tile codes (kernels.h), one thread per 32 cells of the flattened lattice;
/// `kind` has 64 bytes after its last cell.
__global__ void __launch_bounds__(256)
tile_codes_kernel(const std::uint8_t* __restrict__ kind, std::uint8_t* __restrict__ codes, int nx, int ny, int nz,
                  unsigned n, unsigned ncodes) {
    const unsigned i = blockIdx.x * 256u + threadIdx.x, c0 = 32 * i;
    if (i >= ncodes) return;
    std::uint8_t code = kTileIdle;
    if (c0 < n) {
        const uint4 a = reinterpret_cast<const uint4*>(kind + c0)[0], b = reinterpret_cast<const uint4*>(kind + c0)[1];
        const bool full = c0 + 32 <= n;
        const unsigned row = c0 / nx, z = row / ny;
        const int x = static_cast<int>(c0 - row * nx), y = static_cast<int>(row - z * ny);
        if (full && (a.x | a.y | a.z | a.w | b.x | b.y | b.z | b.w) == 0) {
            // A run across a row's end holds cells of the x faces.
            const bool inner = x > 0 && x + 31 < nx - 1 && y > 0 && y < ny - 1 && nz > 1;
            const int zi = static_cast<int>(z);
            code = !inner ? kTileGeneral : zi == 0 ? kTileLowZ : zi == nz - 1 ? kTileHighZ : kTileBulk;
        } else {
            const std::uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            for (int k = 0; k < 32 && c0 + k < n; ++k) {
                const int flag = static_cast<int>(v[k >> 2] >> (8 * (k & 3))) & kFlagMask;
                if (flag == kFluid || flag == kInlet || flag == kOutlet || flag == kOutletEq) { code = kTileGeneral; break; }
            }
        }
    }
    codes[i] = code;
}

// ---- ordered lists ------------------------------------------------------------------

constexpr int kSelTile = 256;   // words per tile

enum SelectOp { kSelForce, kSelShell, kSelInter, kSelWall };

/// Selection words of a list and the number of cells in each tile.
/// kSelWall: `C` are the planes of the clean field, stats[1] counts the cells
/// left out for a link that is solid in the active field only.
template <int OP>
__global__ void __launch_bounds__(kSelTile)
select_kernel(Planes P, Planes C, BitGrid g, std::uint32_t* __restrict__ sel, int* __restrict__ tileCount,
              int* __restrict__ stats) {
    const unsigned wi = blockIdx.x * kSelTile + threadIdx.x;
    std::uint32_t s = 0;
    int vanes = 0;
    if (wi < g.total()) {
        int w, y, z;
        word_of(g, wi, w, y, z);
        if (OP == kSelInter) {
            s = P.p[kPInter][wi];
        } else {
            s = P.p[OP == kSelShell ? kPInter : kPFluid][wi];
            if (s) {
                if (OP == kSelForce) s &= near18<true>(OnePlane{P.p[kPSolid]}, g, w, y, z);
                if (OP == kSelShell) s &= near18<true>(OrPlanes{P.p[kPFluid], P.p[kPOutlet]}, g, w, y, z);
                if (OP == kSelWall) {
                    s &= near18<false>(OnePlane{P.p[kPSolid]}, g, w, y, z);
                    if (s && C.p[kPSolid] != P.p[kPSolid]) {
                        const std::uint32_t v = s & near18<false>(AndNotPlanes{P.p[kPSolid], C.p[kPSolid]}, g, w, y, z);
                        vanes = __popc(v);
                        s &= ~v;
                    }
                }
            }
        }
        sel[wi] = s;
    }
    __shared__ int warpSum[kSelTile / 32];
    int v = __popc(s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) warpSum[threadIdx.x >> 5] = v;
    if (OP == kSelWall && vanes) atomicAdd(stats + 1, vanes);
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int k = 0; k < kSelTile / 32; ++k) t += warpSum[k];
        tileCount[blockIdx.x] = t;
    }
}

/// Exclusive scan of the tile counts in place (one block); total -> *total.
__global__ void __launch_bounds__(1024) tile_scan_kernel(int* counts, int tiles, long long* total) {
    __shared__ long long carry;
    __shared__ long long warpSum[32];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int base = 0; base < tiles; base += 1024) {
        const int i = base + threadIdx.x;
        const long long v = i < tiles ? counts[i] : 0;
        long long inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) warpSum[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const long long w = warpSum[lane];
            long long wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const long long t = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += t;
            }
            warpSum[lane] = wi - w;
        }
        __syncthreads();
        const long long excl = carry + warpSum[warp] + inc - v;
        if (i < tiles) counts[i] = static_cast<int>(excl);
        __syncthreads();
        if (threadIdx.x == 1023) carry = excl + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

/// First list slot of this thread's selected cells: the tile's plus an
/// exclusive scan over the block of `cnt`.
__device__ __forceinline__ long long first_slot(int cnt, const int* __restrict__ tileOffset) {
    __shared__ int warpSum[kSelTile / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warpSum[warp] = inc;
    __syncthreads();
    int before = 0;
    for (int k = 0; k < warp; ++k) before += warpSum[k];
    return static_cast<long long>(tileOffset[blockIdx.x]) + before + inc - cnt;
}

/// Selected cells into the list, ascending.
__global__ void __launch_bounds__(kSelTile)
scatter_kernel(const std::uint32_t* __restrict__ sel, BitGrid g, const int* __restrict__ tileOffset,
               std::uint32_t* __restrict__ cells) {
    const unsigned wi = blockIdx.x * kSelTile + threadIdx.x;
    std::uint32_t s = wi < g.total() ? sel[wi] : 0;
    long long slot = first_slot(__popc(s), tileOffset);
    if (!s) return;
    const unsigned row = wi / g.words, c0 = row * static_cast<unsigned>(g.nx) + 32u * (wi - row * g.words);
    for (; s; s &= s - 1) cells[slot++] = c0 + static_cast<unsigned>(__ffs(static_cast<int>(s)) - 1);
}

/// Cell coordinates from its index.
__device__ __forceinline__ void coords(const BitGrid& g, std::uint32_t c, int& x, int& y, int& z) {
    const unsigned row = c / static_cast<unsigned>(g.nx);
    x = static_cast<int>(c - row * static_cast<unsigned>(g.nx));
    z = static_cast<int>(row / static_cast<unsigned>(g.ny));
    y = static_cast<int>(row - static_cast<unsigned>(z) * static_cast<unsigned>(g.ny));
}

/// Solid links of the listed cells, bit q: FORCE the neighbours at + c_q,
/// everything periodic; otherwise the pull neighbours at - c_q, nothing
/// beyond the x and y faces.
template <bool FORCE>
__global__ void __launch_bounds__(128)
link_mask_kernel(const std::uint8_t* __restrict__ flags, BitGrid g, const std::uint32_t* __restrict__ cells, unsigned n,
                 std::uint32_t* __restrict__ masks) {
    const unsigned i = blockIdx.x * 128u + threadIdx.x;
    if (i >= n) return;
    int x, y, z;
    coords(g, cells[i], x, y, z);
    std::uint32_t m = 0;
#pragma unroll
    for (int q = 1; q < kQ; ++q) {
        int X = x + (FORCE ? cx(q) : -cx(q)), Y = y + (FORCE ? cy(q) : -cy(q));
        const int Z = wrapi(z + (FORCE ? cz(q) : -cz(q)), g.nz);
        if (FORCE) {
            X = wrapi(X, g.nx);
            Y = wrapi(Y, g.ny);
        } else if (X < 0 || X >= g.nx || Y < 0 || Y >= g.ny) {
            continue;
        }
        if (flags[(static_cast<size_t>(Z) * g.ny + Y) * g.nx + X] == kSolidB) m |= 1u << q;
    }
    masks[i] = m;
}

// ---- wall-model list --------------------------------------------------------------
// Two lists: the candidates over the lattice (fluid cells with a pull link that
// is solid and none that is solid in the active field only), then the ones
// among them whose occupancy gradient gives a normal. Both keep the order, so
// the entries ascend by cell, as the host builder's.

/// Sum of (dx, dy, dz) over the solid cells of the 5^3 block around (x, y, z):
/// nothing solid beyond the x and y faces, z periodic. Whole numbers, so the
/// order of the sum does not matter.
__device__ __forceinline__ void occupancy_gradient(const std::uint32_t* __restrict__ solid, const BitGrid& g, int x, int y,
                                                   int z, int& gx, int& gy, int& gz) {
    gx = gy = gz = 0;
    const int w = x >> 5, b = x & 31, last = g.words - 1;
    for (int dz = -2; dz <= 2; ++dz) {
        const int Z = wrapi(z + dz, g.nz);
        for (int dy = -2; dy <= 2; ++dy) {
            const int Y = y + dy;
            if (Y < 0 || Y >= g.ny) continue;
            const std::uint32_t* r = solid + (static_cast<size_t>(Z) * g.ny + Y) * g.words;
            // Bits x - 2 .. x + 2 (the row's words hold nothing beyond nx).
            std::uint32_t v = b >= 2 ? __ldg(r + w) >> (b - 2) : __ldg(r + w) << (2 - b);
            if (b < 2 && w > 0) v |= __ldg(r + w - 1) >> (30 + b);
            if (b > 29 && w < last) v |= __ldg(r + w + 1) << (34 - b);
            v &= 31u;
            const int n = __popc(v);
            gx += static_cast<int>((v >> 3) & 1u) + 2 * static_cast<int>((v >> 4) & 1u) - static_cast<int>((v >> 1) & 1u)
                - 2 * static_cast<int>(v & 1u);
            gy += dy * n;
            gz += dz * n;
        }
    }
}

/// Candidates with a normal: their number per tile of 256, and in stats
/// [0] listed, [2] without a normal.
__global__ void __launch_bounds__(kSelTile)
normal_count_kernel(const std::uint32_t* __restrict__ solid, BitGrid g, const std::uint32_t* __restrict__ cand, unsigned n,
                    int* __restrict__ tileCount, int* __restrict__ stats) {
    const unsigned i = blockIdx.x * kSelTile + threadIdx.x;
    bool ok = false;
    if (i < n) {
        int x, y, z, gx, gy, gz;
        coords(g, cand[i], x, y, z);
        occupancy_gradient(solid, g, x, y, z, gx, gy, gz);
        ok = gx != 0 || gy != 0 || gz != 0;   // the host's |gradient| >= 1e-3
    }
    const int c = __syncthreads_count(ok);
    if (threadIdx.x == 0) {
        const int here = static_cast<int>(min(static_cast<unsigned>(kSelTile), n - blockIdx.x * kSelTile));
        tileCount[blockIdx.x] = c;
        if (c) atomicAdd(stats + 0, c);
        if (here - c) atomicAdd(stats + 2, here - c);
    }
}

__global__ void __launch_bounds__(kSelTile)
wall_entry_kernel(const std::uint32_t* __restrict__ solid, const std::uint8_t* __restrict__ active, BitGrid g,
                  int sampleCells, const std::uint32_t* __restrict__ cand, const std::uint32_t* __restrict__ masks,
                  unsigned n, const int* __restrict__ tileOffset, WallListOut o) {
    const unsigned i = blockIdx.x * kSelTile + threadIdx.x;
    int x = 0, y = 0, z = 0, ix = 0, iy = 0, iz = 0;
    std::uint32_t c = 0;
    if (i < n) {
        c = cand[i];
        coords(g, c, x, y, z);
        occupancy_gradient(solid, g, x, y, z, ix, iy, iz);
    }
    const bool ok = ix != 0 || iy != 0 || iz != 0;
    const long long slot = first_slot(ok ? 1 : 0, tileOffset);
    if (!ok) return;
    const float gx = static_cast<float>(ix), gy = static_cast<float>(iy), gz = static_cast<float>(iz);
    const float gm = sqrtf(gx * gx + gy * gy + gz * gz);
    const float nx_ = -gx / gm, ny_ = -gy / gm, nz_ = -gz / gm;
    std::uint32_t s = c;
    int sx = x, sy = y, sz = z;
    for (int k = sampleCells; k >= 1; --k) {
        const int tx = x + static_cast<int>(lroundf(nx_ * static_cast<float>(k)));
        const int ty = y + static_cast<int>(lroundf(ny_ * static_cast<float>(k)));
        const int tz = wrapi(z + static_cast<int>(lroundf(nz_ * static_cast<float>(k))), g.nz);
        if (tx < 0 || tx >= g.nx || ty < 0 || ty >= g.ny) continue;
        const std::uint32_t t = static_cast<std::uint32_t>(tx)
                              + static_cast<std::uint32_t>(g.nx) * (static_cast<std::uint32_t>(ty)
                                                                    + static_cast<std::uint32_t>(g.ny) * tz);
        if (active[t] != kFluidB) continue;
        s = t; sx = tx; sy = ty; sz = tz;
        break;
    }
    int dzw = sz - z;
    if (dzw > g.nz / 2) dzw -= g.nz;
    if (dzw < -g.nz / 2) dzw += g.nz;
    const float proj = static_cast<float>(sx - x) * nx_ + static_cast<float>(sy - y) * ny_
                     + static_cast<float>(dzw) * nz_;
    o.cell[slot] = c;
    o.sample[slot] = s;
    o.nX[slot] = nx_; o.nY[slot] = ny_; o.nZ[slot] = nz_;
    o.ys[slot] = 0.5f + fmaxf(proj, 0.0f);
    o.mask[slot] = masks[i];
}

// ---- host side of the tables ---------------------------------------------------------

inline unsigned blocks_of(unsigned long long n, unsigned b) { return static_cast<unsigned>((n + b - 1) / b); }

/// What the host reads back of a build: one copy.
struct Readback {
    unsigned long long counts[2];
    long long total[2];    // of the list, and of the wall list among its candidates
    int stats[4];
    int box[4];
};

/// A build's device memory, cut from one scratch block.
struct Carver {
    char* p;
    size_t used = 0;
    template <class T> T* take(size_t n) {
        T* r = reinterpret_cast<T*>(p + used);
        used += (n * sizeof(T) + 255) & ~size_t{255};
        return r;
    }
};

struct TableScratch {
    Readback* rb;
    Planes planes{}, clean{};
    std::uint32_t* sel = nullptr;   // null: no list wanted
    int* tiles = nullptr;
    /// Lays the parts out at `base` (null: only counts the bytes).
    size_t lay(char* base, const BitGrid& g, unsigned wanted, bool cleanSolid, bool list) {
        Carver c{base};
        rb = c.take<Readback>(1);
        const size_t words = g.total();
        for (int k = 0; k < kPlanes; ++k) planes.p[k] = (wanted >> k & 1u) ? c.take<std::uint32_t>(words) : nullptr;
        clean = Planes{};
        clean.p[kPSolid] = cleanSolid ? c.take<std::uint32_t>(words) : planes.p[kPSolid];
        if (list) {
            sel = c.take<std::uint32_t>(words);
            tiles = c.take<int>(words / kSelTile + 1);
        }
        return c.used;
    }
};

cudaError_t build_planes(const std::uint8_t* flags, const BitGrid& g, const Planes& P, cudaStream_t st,
                         std::uint32_t keep = 0xffffffffu) {
    const unsigned nb = blocks_of(g.total(), 256);
    const auto a = reinterpret_cast<std::uintptr_t>(flags);
    if (g.nx % 16 == 0 && a % 16 == 0) planes_kernel<16><<<nb, 256, 0, st>>>(flags, g, P, keep);
    else if (g.nx % 4 == 0 && a % 4 == 0) planes_kernel<4><<<nb, 256, 0, st>>>(flags, g, P, keep);
    else planes_kernel<1><<<nb, 256, 0, st>>>(flags, g, P, keep);
    return cudaGetLastError();
}

cudaError_t reset_readback(Readback* rb, const BitGrid& g, cudaStream_t st) {
    Readback init{};
    init.box[0] = g.nx; init.box[1] = g.ny; init.box[2] = init.box[3] = -1;
    return cudaMemcpyAsync(rb, &init, sizeof init, cudaMemcpyHostToDevice, st);
}

void launch_classes(const TableScratch& ts, const BitGrid& g, unsigned long long* counts, cudaStream_t st) {
    const unsigned nb = min(blocks_of(g.total(), 256), 8u * static_cast<unsigned>(sm_count()));
    classes_kernel<<<nb, 256, 0, st>>>(ts.planes, g, counts, ts.rb->box);
}

template <int OP>
void select_list(const TableScratch& ts, const BitGrid& g, cudaStream_t st) {
    const unsigned tiles = blocks_of(g.total(), kSelTile);
    select_kernel<OP><<<tiles, kSelTile, 0, st>>>(ts.planes, ts.clean, g, ts.sel, ts.tiles, ts.rb->stats);
    tile_scan_kernel<<<1, 1024, 0, st>>>(ts.tiles, static_cast<int>(tiles), &ts.rb->total[0]);
}

void scatter_list(const TableScratch& ts, const BitGrid& g, std::uint32_t* cells, cudaStream_t st) {
    scatter_kernel<<<blocks_of(g.total(), kSelTile), kSelTile, 0, st>>>(ts.sel, g, ts.tiles, cells);
}

cudaError_t read_back(const TableScratch& ts, Readback& h, cudaStream_t st) {
    if (auto e = cudaGetLastError(); e != cudaSuccess) return e;
    if (auto e = cudaMemcpyAsync(&h, ts.rb, sizeof h, cudaMemcpyDeviceToHost, st); e != cudaSuccess) return e;
    return cudaStreamSynchronize(st);
}

/// Stream-ordered scratch of a call without a GeomScratch of its own.
struct CallScratch {
    void* p = nullptr;
    cudaStream_t st;
    explicit CallScratch(cudaStream_t s) : st(s) {}
    ~CallScratch() { if (p) cudaFreeAsync(p, st); }
    cudaError_t alloc(size_t bytes) { return cudaMallocAsync(&p, bytes, st); }
};

constexpr unsigned bit(Plane p) { return 1u << p; }

/// Entries to allocate for a list of n that a changed field makes anew: every
/// allocation and release idles the device.
constexpr long long spare(long long n) { return n + n / 8 + 1; }

} // namespace

// ---- host entry points ---------------------------------------------------------

cudaError_t launch_flag_diff(const std::uint8_t* kind, std::uint8_t* mask, long long n, long long* count, cudaStream_t st) {
    if (!kind || !mask || !count || n <= 0 || n >= (1LL << 31)) return cudaErrorInvalidValue;
    flag_diff_kernel<<<static_cast<unsigned>((n + 1023) / 1024), 256, 0, st>>>(kind, mask, static_cast<unsigned>(n),
                                                                              reinterpret_cast<unsigned long long*>(count));
    return cudaGetLastError();
}

bool is_device_pointer(const void* p) {
    cudaPointerAttributes a{};
    if (!p || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice;
}

cudaError_t device_build_flags(LevelDims d, int base, const std::uint8_t* in, const FoilRaster* foil, int closeGaps,
                               int shell, std::uint8_t* out, cudaStream_t st, int* closedOut) {
    const long long n = d.cells();
    if (n <= 0 || !out || (base == 2 && (!in || in == out)) || base < 0 || base > 2) return cudaErrorInvalidValue;
    // Work block: 64 bytes of counters, the nx*ny mask (rounded to 16 bytes),
    // then the outline (2 floats per point) and its lattice x, y (1 + 1).
    const size_t maskBytes = foil ? (static_cast<size_t>(d.nx) * d.ny + 15) / 16 * 16 : 0;
    const size_t polyBytes = foil ? static_cast<size_t>(foil->npts) * 4 * sizeof(float) : 0;
    char* work = nullptr;
    if (auto e = cudaMallocAsync(reinterpret_cast<void**>(&work), 64 + maskBytes + polyBytes, st); e != cudaSuccess)
        return e;
    int* counters = reinterpret_cast<int*>(work);     // [0] closed, [1] rasteriser error
    cudaError_t e = cudaMemsetAsync(work, 0, 64, st);
    std::uint8_t* mask = nullptr;
    if (e == cudaSuccess && foil) {
        if (foil->npts < 3 || d.nx < 3 || d.ny < 3 || !foil->xy) {
            e = cudaErrorInvalidValue;
        } else {
            mask = reinterpret_cast<std::uint8_t*>(work + 64);
            float* dxy = reinterpret_cast<float*>(work + 64 + maskBytes);
            float* px = dxy + 2 * foil->npts;
            e = cudaMemcpyAsync(dxy, foil->xy, static_cast<size_t>(foil->npts) * 2 * sizeof(float),
                                cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) {
                foil_poly_kernel<<<(foil->npts + 127) / 128, 128, 0, st>>>(dxy, foil->npts, foil->cosA, foil->sinA,
                                                                          foil->chord, foil->anchorX, foil->anchorY,
                                                                          px, px + foil->npts);
                foil_rows_kernel<<<(d.ny + kRowWarps - 1) / kRowWarps, kRowWarps * 32, 0, st>>>(
                    px, px + foil->npts, foil->npts, d.nx, d.ny, mask, counters + 1);
                e = cudaGetLastError();
            }
        }
    }
    if (e == cudaSuccess) {
        FlagBuild b{d.nx, d.ny, d.nz, base, in, mask, closeGaps, shell};
        const long long plane = static_cast<long long>(d.nx) * d.ny;
        const dim3 grid(static_cast<unsigned>((plane + 255) / 256), static_cast<unsigned>((d.nz + kFlagRun - 1) / kFlagRun));
        build_flags_kernel<<<grid, 256, 0, st>>>(b, out, counters);
        e = cudaGetLastError();
    }
    int h[2] = {0, 0};
    // A rasterised outline is checked for the row-crossing limit.
    if (e == cudaSuccess && (closedOut || mask)) {
        e = cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess && h[1]) e = cudaErrorInvalidValue;   // a row with > 64 crossings
        if (e == cudaSuccess && closedOut) *closedOut = h[0];
    }
    cudaFreeAsync(work, st);
    return e;
}

cudaError_t GeomScratch::ensure(size_t bytes) {
    if (bytes <= size) return cudaSuccess;
    release();
    if (auto e = cudaMalloc(&p, bytes); e != cudaSuccess) { p = nullptr; return e; }
    size = bytes;
    return cudaSuccess;
}
void GeomScratch::release() {
    if (p) cudaFree(p);
    p = nullptr;
    size = 0;
}

cudaError_t device_solid_bbox(LevelDims d, const std::uint8_t* flags, cudaStream_t st, int box[4]) {
    if (d.cells() <= 0 || d.cells() >= (1LL << 31) || !flags) return cudaErrorInvalidValue;
    const BitGrid g = bit_grid(d);
    TableScratch ts;
    CallScratch cs(st);
    if (auto e = cs.alloc(ts.lay(nullptr, g, bit(kPSolid), false, false)); e != cudaSuccess) return e;
    ts.lay(static_cast<char*>(cs.p), g, bit(kPSolid), false, false);
    if (auto e = reset_readback(ts.rb, g, st); e != cudaSuccess) return e;
    if (auto e = build_planes(flags, g, ts.planes, st); e != cudaSuccess) return e;
    launch_classes(ts, g, nullptr, st);
    Readback h;
    if (auto e = read_back(ts, h, st); e != cudaSuccess) return e;
    for (int k = 0; k < 4; ++k) box[k] = h.box[k];
    return cudaSuccess;
}

cudaError_t build_level_tables(LevelDims d, const std::uint8_t* flags, LevelTables& t, GeomScratch& scratch,
                               cudaStream_t st) {
    const long long n = d.cells();
    if (n <= 0 || n >= (1LL << 31) || !flags || !t.kind) return cudaErrorInvalidValue;
    const BitGrid g = bit_grid(d);
    const unsigned wanted = bit(kPSolid) | bit(kPFluid) | bit(kPSlip) | bit(kPInlet) | bit(kPOutlet);
    TableScratch ts;
    if (auto e = scratch.ensure(ts.lay(nullptr, g, wanted, false, true)); e != cudaSuccess) return e;
    ts.lay(static_cast<char*>(scratch.p), g, wanted, false, true);
    if (auto e = reset_readback(ts.rb, g, st); e != cudaSuccess) return e;
    if (auto e = build_planes(flags, g, ts.planes, st, 0x0f0f0f0fu); e != cudaSuccess) return e;
    launch_classes(ts, g, ts.rb->counts, st);
    const unsigned nb = blocks_of(g.total(), 256);
    const auto a = reinterpret_cast<std::uintptr_t>(flags) | reinterpret_cast<std::uintptr_t>(t.kind);
    if (d.nx % 4 == 0 && a % 4 == 0) classify_kernel<4><<<nb, 256, 0, st>>>(flags, ts.planes, g, t.kind, t.links);
    else classify_kernel<1><<<nb, 256, 0, st>>>(flags, ts.planes, g, t.kind, t.links);
    if (t.tiles) {
        const unsigned nc = static_cast<unsigned>(tile_code_bytes(n));
        tile_codes_kernel<<<blocks_of(nc, 256), 256, 0, st>>>(t.kind, reinterpret_cast<std::uint8_t*>(t.tiles), d.nx,
                                                             d.ny, d.nz, static_cast<unsigned>(n), nc);
    }
    select_list<kSelForce>(ts, g, st);
    Readback h;
    if (auto e = read_back(ts, h, st); e != cudaSuccess) return e;
    t.classes[0] = static_cast<long long>(h.counts[0]);
    t.classes[1] = static_cast<long long>(h.counts[1]);
    t.classes[2] = n - t.classes[0] - t.classes[1];
    for (int k = 0; k < 4; ++k) t.box[k] = h.box[k];
    t.linkCount = h.total[0];
    if (!t.linkCells || t.linkCount > t.linkRoom) {
        cudaFree(t.linkCells);
        cudaFree(t.linkMasks);
        t.linkCells = t.linkMasks = nullptr;
        t.linkRoom = 0;
        const long long room = spare(t.linkCount);
        if (auto e = cudaMalloc(&t.linkCells, static_cast<size_t>(room) * 4); e != cudaSuccess) return e;
        if (auto e = cudaMalloc(&t.linkMasks, static_cast<size_t>(room) * 4); e != cudaSuccess) {
            cudaFree(t.linkCells);
            t.linkCells = nullptr;
            return e;
        }
        t.linkRoom = room;
    }
    if (t.linkCount > 0) {
        const unsigned m = static_cast<unsigned>(t.linkCount);
        scatter_list(ts, g, t.linkCells, st);
        link_mask_kernel<true><<<blocks_of(m, 128), 128, 0, st>>>(flags, g, t.linkCells, m, t.linkMasks);
    }
    return cudaGetLastError();
}

cudaError_t build_shell_list(LevelDims d, const std::uint8_t* flags, bool full, std::uint32_t** cells, long long* room,
                             long long* count, GeomScratch& scratch, cudaStream_t st) {
    if (d.cells() <= 0 || d.cells() >= (1LL << 31) || !flags || !cells || !room || !count) return cudaErrorInvalidValue;
    *count = 0;
    const BitGrid g = bit_grid(d);
    const unsigned wanted = full ? bit(kPInter) : bit(kPInter) | bit(kPFluid) | bit(kPOutlet);
    TableScratch ts;
    if (auto e = scratch.ensure(ts.lay(nullptr, g, wanted, false, true)); e != cudaSuccess) return e;
    ts.lay(static_cast<char*>(scratch.p), g, wanted, false, true);
    if (auto e = reset_readback(ts.rb, g, st); e != cudaSuccess) return e;
    if (auto e = build_planes(flags, g, ts.planes, st); e != cudaSuccess) return e;
    if (full) select_list<kSelInter>(ts, g, st);
    else select_list<kSelShell>(ts, g, st);
    Readback h;
    if (auto e = read_back(ts, h, st); e != cudaSuccess) return e;
    if (!*cells || h.total[0] > *room) {
        cudaFree(*cells);
        *cells = nullptr;
        *room = 0;
        if (auto e = cudaMalloc(cells, static_cast<size_t>(spare(h.total[0])) * 4); e != cudaSuccess) return e;
        *room = spare(h.total[0]);
    }
    *count = h.total[0];
    if (h.total[0] > 0) scatter_list(ts, g, *cells, st);
    return cudaGetLastError();
}

cudaError_t device_force_links(LevelDims d, const std::uint8_t* flags, std::uint32_t* cells, std::uint32_t* masks,
                               long long cap, long long* count, cudaStream_t st) {
    if (d.cells() <= 0 || d.cells() >= (1LL << 31) || !flags || !count) return cudaErrorInvalidValue;
    const BitGrid g = bit_grid(d);
    const unsigned wanted = bit(kPSolid) | bit(kPFluid);
    TableScratch ts;
    CallScratch cs(st);
    if (auto e = cs.alloc(ts.lay(nullptr, g, wanted, false, true)); e != cudaSuccess) return e;
    ts.lay(static_cast<char*>(cs.p), g, wanted, false, true);
    if (auto e = reset_readback(ts.rb, g, st); e != cudaSuccess) return e;
    if (auto e = build_planes(flags, g, ts.planes, st); e != cudaSuccess) return e;
    select_list<kSelForce>(ts, g, st);
    Readback h;
    if (auto e = read_back(ts, h, st); e != cudaSuccess) return e;
    *count = h.total[0];
    if (*count <= 0 || *count > cap) return cudaSuccess;
    const unsigned m = static_cast<unsigned>(*count);
    scatter_list(ts, g, cells, st);
    link_mask_kernel<true><<<blocks_of(m, 128), 128, 0, st>>>(flags, g, cells, m, masks);
    if (auto e = cudaGetLastError(); e != cudaSuccess) return e;
    return cudaStreamSynchronize(st);
}

// The wall list in two parts, so that its owner can allocate the entries once
// their number is known.
cudaError_t WallListBuild::find(LevelDims dims, const std::uint8_t* activeF, const std::uint8_t* clean, long long* count,
                                int stats[3], cudaStream_t st) {
    if (dims.cells() <= 0 || dims.cells() >= (1LL << 31) || !activeF || !count) return cudaErrorInvalidValue;
    d = dims;
    active = activeF;
    *count = n = candidates = 0;
    if (stats) stats[0] = stats[1] = stats[2] = 0;
    const BitGrid g = bit_grid(d);
    const bool own = clean && clean != activeF;
    const unsigned wanted = bit(kPSolid) | bit(kPFluid);
    TableScratch ts;
    if (auto e = cudaMallocAsync(&block, ts.lay(nullptr, g, wanted, own, true), st); e != cudaSuccess) return e;
    ts.lay(static_cast<char*>(block), g, wanted, own, true);
    if (auto e = reset_readback(ts.rb, g, st); e != cudaSuccess) return e;
    if (auto e = build_planes(activeF, g, ts.planes, st); e != cudaSuccess) return e;
    if (own)
        if (auto e = build_planes(clean, g, ts.clean, st); e != cudaSuccess) return e;
    select_list<kSelWall>(ts, g, st);
    Readback h;
    if (auto e = read_back(ts, h, st); e != cudaSuccess) return e;
    if (stats) stats[1] = h.stats[1];
    candidates = h.total[0];
    if (candidates == 0) return cudaSuccess;
    // Candidates, their link masks and the tiles of the second list.
    const unsigned nc = static_cast<unsigned>(candidates), tiles = blocks_of(nc, kSelTile);
    Carver c{nullptr};
    for (int pass = 0; pass < 2; ++pass) {
        c.used = 0;
        cand = c.take<std::uint32_t>(nc);
        masks = c.take<std::uint32_t>(nc);
        offsets = c.take<int>(tiles);
        if (pass == 0) {
            if (auto e = cudaMallocAsync(&block2, c.used, st); e != cudaSuccess) return e;
            c.p = static_cast<char*>(block2);
        }
    }
    solid = ts.clean.p[kPSolid];
    scatter_list(ts, g, cand, st);
    link_mask_kernel<false><<<blocks_of(nc, 128), 128, 0, st>>>(activeF, g, cand, nc, masks);
    normal_count_kernel<<<tiles, kSelTile, 0, st>>>(solid, g, cand, nc, offsets, ts.rb->stats);
    tile_scan_kernel<<<1, 1024, 0, st>>>(offsets, static_cast<int>(tiles), &ts.rb->total[1]);
    if (auto e = read_back(ts, h, st); e != cudaSuccess) return e;
    *count = n = h.total[1];
    if (stats) { stats[0] = h.stats[0]; stats[2] = h.stats[2]; }
    return cudaSuccess;
}

cudaError_t WallListBuild::emit(int sampleCells, const WallListOut& out, cudaStream_t st) const {
    if (n <= 0) return cudaSuccess;
    const unsigned nc = static_cast<unsigned>(candidates);
    wall_entry_kernel<<<blocks_of(nc, kSelTile), kSelTile, 0, st>>>(solid, active, bit_grid(d), sampleCells, cand, masks,
                                                                   nc, offsets, out);
    return cudaGetLastError();
}

void WallListBuild::release(cudaStream_t st) {
    if (block) cudaFreeAsync(block, st);
    if (block2) cudaFreeAsync(block2, st);
    block = block2 = nullptr;
}

cudaError_t device_wall_list(LevelDims d, const std::uint8_t* active, const std::uint8_t* clean, int sampleCells,
                             const WallListOut& out, long long cap, long long* count, int stats[3],
                             cudaStream_t st) {
    WallListBuild b;
    cudaError_t e = b.find(d, active, clean, count, stats, st);
    if (e == cudaSuccess && *count > 0 && *count <= cap) {
        e = b.emit(sampleCells, out, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    b.release(st);
    return e;
}

} // namespace fcfd
