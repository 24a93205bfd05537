// Device memory of the tiled FP64 M2L's part sums (m2l_tile.cu): what a plan
// takes and what the serving loop sets aside for it (pure C++, shared with a
// CPU test).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace sfmm {

constexpr int kTileMinOrder = 2, kTileMaxOrder = 12;
constexpr int kTileParts = 6;
// Rows (targets x charge components) below which a tile's parts run in blocks
// of their own.  Measured, M2L apart / in turn (leaf 64): p = 10 Plummer 1.3k
// rows 0.73 / 1.48 ms, 6k 1.38 / 1.52, 12.6k 2.48 / 2.89, 18.5k 3.43 / 4.06,
// 22.6k 4.11 / 4.28; p = 6 2.6k 0.58 / 1.24, 18.5k 1.52 / 2.07, 22.6k 1.81 /
// 2.23; p = 12 18.5k 6.64 / 6.94.  Beyond, the blocks' last wave costs little
// (p = 10 32k 5.40 / 5.46, 37k 6.10 / 5.91) and the sums' memory, which grows
// with the rows, is not worth it.
constexpr int64_t kTileSplitRows = 24 * 1024;

// At most an eighth more: trees of a particle code's steps, or of a batch's
// fresh sets, differ in their node counts, and a released block is handed out
// again to requests of its own size only (memory.cu).  Plan set-up on a new
// 300,000-point tree, p = 10: exact sizes 3.2 to 3.5 ms, these 1.0; 60,000 points
// 0.73 and 0.20; a batch of 4 x 40,000 new points 9.2 and 8.1.
inline size_t coarse_bytes(size_t bytes)
{
    size_t step = 16;
    while (step * 16 <= bytes) step *= 2;
    return (bytes + step - 1) / step * step;
}

// Part sums of `rows` rows at order p: two potential rows and one field row per part.
inline size_t tile_part_bytes(int64_t rows, int p)
{
    const size_t T = (p + 1) * (p + 2) / 2, T1 = (p + 2) * (p + 3) / 2;
    return size_t(kTileParts) * 16 * (2 * T + T1) * size_t(rows);
}

// What to set aside for the part sums of n points with leaves of at most
// `leaf`.  A node that splits has more than `leaf` points and eight children at
// most, so a tree of even depth has up to 64/7 n / leaf nodes (measured: 40,000
// uniform points, leaf 64, 7.1 n / leaf; 300,007 Plummer points 4.0); a plan
// whose rows need more than it was given runs its parts in turn.  Leaves are at
// least n / leaf, so large trees take none.
inline size_t tile_part_estimate(int64_t n, int leaf, int qdim, int p)
{
    if (p < kTileMinOrder || p > kTileMaxOrder) return 0;
    const int64_t leaves = n / std::max(leaf, 1);
    if (leaves * qdim >= kTileSplitRows) return 0;
    return coarse_bytes(tile_part_bytes(std::min<int64_t>((64 * leaves / 7 + 128) * qdim, kTileSplitRows), p));
}

// Most bytes of part sums that plans made by the calling thread may take
// (m2l_tile.cu; the serving loop sets it for its requests).  No limit at first.
void set_thread_tile_part_limit(size_t bytes) noexcept;

}  // namespace sfmm
