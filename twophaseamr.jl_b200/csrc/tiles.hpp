// Haloed block tiles of a CSR level: the per-block data of the two fused
// V-cycle kernels of a level (csrc/tiles.cuh).
//
// A tile is one mesh block (its cells are contiguous in the reference's cell
// order) plus the cells within graph distance 3 of it in the level operator's
// sparsity pattern, listed ring by ring.  The down kernel computes both
// pre-smoothing sweeps, the residual and the restriction of the block's
// coarse cells from the right-hand side on the tile alone (each dependent
// phase shrinks the valid region by one ring); the up kernel computes the
// prolongation and both post-smoothing sweeps of the block from the coarse
// correction on the tile alone.  Halo values are recomputed redundantly in
// each tile instead of being exchanged between launches, which removes four
// of the six grid-wide dependencies a level costs per V-cycle.
#pragma once

#include <cstdint>
#include <vector>

#include "host.hpp"

namespace tpa {

// A tile's rows (rings <= 2) are cut into slices of 32 rows, one per warp, each
// as wide as its longest row: entry u of the slice's row k lies at
// 32 u + k of the slice, so that a warp's loads are consecutive.  Rows of the
// balanced tree hold at most 11 entries; a level with a longer row than
// kTileMaxRow is not tiled.
constexpr int kTileSlice = 32;
constexpr int kTileMaxRow = 12;

// a tile's parts of the level's lists
struct alignas(16) TileInfo {
    int32_t cell, slice, co, nco;  // first cell, first slice, first coarse cell and their number
    int32_t n0, n1, n2, n3;        // cells of rings <= 0, 1, 2, 3
};

struct TileLevelHost {
    bool ok = false;
    int ntiles = 0;
    int n3max = 0, n2max = 0;  // largest ring counts (cumulative) over the tiles
    std::vector<TileInfo> info;
    // the tiles' cells: the block's in order, then ring 1, ring 2, ring 3, each
    // with its tentative owner (coarse cell)
    std::vector<int32_t> cell, own;
    // slices {first entry, width}, and per entry its position in the level CSR
    // (-1: padding) and its column as a local cell index (padding: the row's own)
    std::vector<int32_t> slice, pos;
    std::vector<int16_t> col;
    // the coarse cells whose children lie in a tile and, for each, the local
    // indices of its first four children (-1: none), in the order of the level's
    // child lists
    std::vector<int32_t> co;
    std::vector<int16_t> ch;
};

// Tiles of a level with `nblocks` blocks of `cpb` cells, operator A (square,
// sorted columns) and tentative owners `owner` onto `nc` coarse cells.  ok is
// false (and the level keeps the unfused kernels) when a coarse cell's
// children do not all lie in one block, a coarse cell has more than four
// children, a row has more than kTileMaxRow entries, or a tile would exceed
// `max_cells` cells.
TileLevelHost build_tiles(const Csr& A, int64_t nblocks, int64_t cpb, const std::vector<int32_t>& owner, int64_t nc,
                          int max_cells);

}  // namespace tpa
