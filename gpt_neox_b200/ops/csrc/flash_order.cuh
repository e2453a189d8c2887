// Order in which the attention kernels' CTAs (one per query or key tile and head) are started.
//
// Under a causal mask a tile's work grows with its position, so what is still running at the end decides how well the last
// round fills the machine: all heaviest tiles first, over all heads, leaves the light ones for the gaps.  Head by head, as
// the tiles were numbered before, the last heads' heavy tiles start when most SMs are about to go idle (48 heads, 2048
// rows: 384 forward CTAs take 36 units of work on the longest SM against 29 in this order and 26 on average; 768 backward
// 59 against 50 and 49).  The tiles of a head read the same keys and values, so the order is kept within groups of heads
// whose operands stay in L2 together (48 of 126 MB, leaving room for what the CTAs write).  48 heads of 64,
// 2048 rows, forward / dK, dV / dQ: 91 / 125 / 99 -> 75 / 114 / 87 us; 48 of 128, 777 rows, forward 43 -> 35 us; 256 heads of
// 96, in four groups, as before.
#pragma once

struct TileOrder {
    int tiles, heads, group;
    int plane;              // one group of all heads: the grid is heads x tiles, and a CTA's place needs no division
};

inline TileOrder tile_order(int tiles, int heads, long long bytes_per_head) {
    const long long fit = (48ll << 20) / (bytes_per_head > 0 ? bytes_per_head : 1);
    const int group = (int)(fit < 1 ? 1 : fit < heads ? fit : heads);
    return TileOrder{tiles, heads, group, group == heads && tiles <= 65535};
}

// The grid of an order; false: more CTAs than a grid takes.
inline bool tile_grid(const TileOrder& o, unsigned& x, unsigned& y) {
    const long long all = (long long)o.tiles * o.heads;
    x = (unsigned)(o.plane ? o.heads : all);
    y = (unsigned)(o.plane ? o.tiles : 1);
    return all <= 0x7fffffff;
}

// rank: 0 for the tile to start first.
__device__ __forceinline__ void pick_tile(const TileOrder& o, int& rank, int& head) {
    if (o.plane) {
        rank = blockIdx.y;
        head = blockIdx.x;
        return;
    }
    const int per = o.group * o.tiles, g = blockIdx.x / per, r = blockIdx.x - g * per;
    const int size = min(o.group, o.heads - g * o.group);
    rank = r / size;
    head = g * o.group + r % size;
}
