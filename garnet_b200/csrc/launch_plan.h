// How launches are cut into CTAs: plain host arithmetic, without CUDA headers.
#pragma once
#include <algorithm>

namespace gb200 {

constexpr int kSmCount = 148;

// Tiling of the int4 tile kernel (w4a16_tc.cu) for a batch of m rows.
constexpr int kTcMaxRows = 192;    // batch rows per tile (UMMA N): two accumulators and four A tiles fill 512 columns
constexpr int kTcMaxSlices = 8;    // CTAs of a cluster
constexpr int kTcSharedRows = 96;  // the largest tile with which two CTAs share an SM's memory
// CTAs in clusters of 2, 4 or 8 that run at once when each has an SM for itself: a cluster lies within a GPC, which has 16 or 18
// SMs or fewer, so that less than the whole GPU is left the larger the clusters are (74, 33 and 15 of them fit a B200, by
// cudaOccupancyMaxActiveClusters; a little less is asked for here).
constexpr int tc_cluster_room(int slices) { return slices <= 2 ? kSmCount : slices <= 4 ? 128 : 112; }
struct TcPlan {
    int panels, row_tiles, tile_rows, kslices;
};

// The chunks of K that slice `slice` of `slices` takes are [tc_first_chunk(slice), tc_first_chunk(slice + 1)): even shares, none
// of them empty as long as there are as many chunks as slices.  (Shares of equal length but for the last left the K of every
// second matrix in one slice: 64 rows x 5376 -> 512 took 28.5 us, 8.2 us in eight slices of 5 or 6 chunks; any number of slices up
// to eight instead of a power of two took 0.88 to 1.06 times as long on 35 shapes, and 23.6 instead of 15.3 us for
// 100 x 5888 -> 3000.)
#if defined(__CUDACC__)
__host__ __device__
#endif
constexpr int tc_first_chunk(int chunks, int slices, int slice) { return slice * chunks / slices; }

// As few even shares of the batch as tiles allow or, when that is more than a wave, up to three more, whichever makes the least
// work of whole waves (an MMA costs its N columns and some fixed time, about 24 columns' worth); K slices while the machine has
// room for twice the CTAs: a cluster that has to wait for another to finish doubles the call (256 rows x 2048 -> 1024, 16
// clusters of 8: 17.2 us; as 16 of 4: 9.3 us).
inline TcPlan tc_plan(int strips_padded, int chunks, int m)
{
    TcPlan t;
    t.panels = strips_padded / 8;
    const int fewest = (m + kTcMaxRows - 1) / kTcMaxRows;
    long long best = 0;
    for (int tiles = fewest; tiles == fewest || (tiles < fewest + 4 && t.panels * fewest > kSmCount); ++tiles) {
        const int rows = ((m + tiles - 1) / tiles + 15) / 16 * 16;
        const long long used = (m + rows - 1) / rows, waves = (t.panels * used + kSmCount - 1) / kSmCount, cost = waves * (rows + 24);
        if (tiles == fewest || cost < best) best = cost, t.row_tiles = int(used), t.tile_rows = rows;
    }
    const long long tiles = (long long)t.panels * t.row_tiles;
    t.kslices = 1;
    const auto room = [&](int slices) { return t.tile_rows > kTcSharedRows ? tc_cluster_room(slices) : kSmCount; };
    while (t.kslices < kTcMaxSlices && 2 * t.kslices <= chunks && tiles * t.kslices * 2 <= room(2 * t.kslices)) t.kslices *= 2;
    return t;
}

// Query tiles of 128 rows that a CTA of the gpt-oss prefill kernel takes (gpt_oss_prefill.cu); a tile is `tile_tokens` tokens of a
// kv head's group.  Two keep the exponential unit busy while the other tile's MMAs run, where there is a second tile at all; with
// fewer CTAs than SMs one tile each uses twice the SMs.
inline int oss_prefill_tiles(int batch, int kv_heads, int tokens, int tile_tokens)
{
    const long long pairs = (tokens + 2 * tile_tokens - 1) / (2 * tile_tokens);
    return tokens > tile_tokens && batch * (long long)kv_heads * pairs >= kSmCount ? 2 : 1;
}

}  // namespace gb200
