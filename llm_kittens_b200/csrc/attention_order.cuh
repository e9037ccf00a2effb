// The order in which the tiles of causal attention start.
//
// The tiles of a sequence differ in length by up to its tile count, and a block takes an SM (or half of one) for as long as
// its tile is. With the tiles of one head next to each other the long tiles of the last heads start late and the chip
// drains behind them: Llama-3.1 8B at T = 4096 has 256 dK / dV tiles for 148 SMs, of 4 to 128 steps, which in that order end
// 1.47 times later than with all long tiles first. But the tiles of a head share its keys and values (or queries), which
// should still be in the L2 when the next one reads them. So heads are taken in equal groups whose operands fit into the
// L2, longest tiles first within a group: list scheduling with a bounded working set.
#pragma once
#include "common.cuh"

namespace llmk {

struct TileOrder {
    int tiles, heads, group;   // tiles per head; (batch, head) pairs; pairs per group
};

// head_bytes: what the tiles of one head read in common.
static inline TileOrder make_tile_order(int tiles, int heads, long head_bytes) {
    constexpr long L2_SHARE = 96l << 20;
    const long fit = L2_SHARE / (head_bytes > 0 ? head_bytes : 1);
    const long per = fit < 1 ? 1 : (fit < heads ? fit : heads);
    const int groups = (int)((heads + per - 1) / per);
    return TileOrder{tiles, heads, (heads + groups - 1) / groups};
}

// Block `idx` of tiles * heads: its (batch, head) pair and the rank of its tile, 0 = longest.
__host__ __device__ inline void tile_of(const TileOrder& o, int idx, int& rank, int& pair) {
    const int g = idx / (o.group * o.tiles), first = g * o.group;
    const int in_group = o.heads - first < o.group ? o.heads - first : o.group;
    const int r = idx - first * o.tiles;
    rank = r / in_group;
    pair = first + r - rank * in_group;
}

// The k-th tile of block `block` of a grid of fewer blocks than tiles, or `n` behind the last one: back and forth over the
// blocks. Tiles get shorter along the order, so with every block taking the same place in each turn the first one would
// have the longest of every turn (32 heads of 32 tiles on 148 blocks: 168 us one tile per block, 184 that way, 163 so).
__host__ __device__ inline int tile_of_turn(int n, int block, int blocks, int k) {
    const int idx = k * blocks + ((k & 1) ? blocks - 1 - block : block);
    return idx < n ? idx : n;
}

}  // namespace llmk
