// Plain (host + device) types of the batched multi-tunnel step.
#pragma once

#include "fast_div.h"

#include <cstdint>
#include <vector_types.h>

namespace fcfd {

constexpr int kMaxBatchTunnels = 64;
constexpr int kItemBuckets = 512;

/// One tunnel of a batch as the batched collide kernel sees it.
struct BatchTunnelParam {
    void* f[2];                  ///< A/B population buffers
    const std::uint8_t* kind;    ///< kind bytes (flag | near-wall bit)
    const uint2* links;          ///< pull-link classes per cell (build_level_tables)
    long long n;                 ///< cells
    int nx, ny, nz;
    float tau, uIn;
    FastDiv divX, divY;
    int pull[19];                ///< q n - (c_q in cells): slot of cell 0's pull of q, where none wraps
    unsigned inOff[19];          ///< of that slot in a staged tile (16-bit populations)
};

/// The whole batch, passed BY VALUE as a kernel parameter (about 16 KB): it
/// lives in the constant bank, so a block's uniform tunnel index reads the
/// tunnel's sizes and relaxation parameters like ordinary kernel parameters.
/// Work items of a launch are the tiles or row groups of each tunnel, numbered
/// tunnel after tunnel; begins[t] is tunnel t's first item.
struct BatchTable {
    int ntun;
    float lambda, smagPre;
    /// Per-tunnel watchdog latch in device memory (0 running; nonzero: the
    /// tunnel diverged and its work items are skipped).
    const int* latch;
    /// Tile codes (build_level_tables) of all tunnels, a word per 128 cells, each
    /// tunnel's after the last one's: word i is that of tile item i.
    const std::uint32_t* tiles;
    unsigned begins[kMaxBatchTunnels + 1];   ///< the last tunnel's is followed by the number of items
    /// The tunnel of items 0, 2^itemShift, 2 2^itemShift, ...: where the search
    /// for a tile item's tunnel begins.
    int itemShift;
    std::uint8_t tunnelAt[kItemBuckets];
    BatchTunnelParam t[kMaxBatchTunnels];
};

static_assert(sizeof(BatchTable) <= 32000, "a kernel's parameters are at most 32764 bytes");

/// Launch shape of the batched collide: threads per block (striding along
/// x through each row), rows per work item, grid (0: one item per block).
/// Blocks of 128 at one row take tiles of 128 cells of the flattened lattice
/// instead of rows.
struct BatchShape {
    int block = 128;
    int rows = 1;
    int grid = 0;
    bool tiles() const { return block == 128 && rows == 1; }
};

} // namespace fcfd
