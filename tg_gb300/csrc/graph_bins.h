// graph_bins.h -- room for the bin references of one job of a frame graph.
#pragma once

#include <algorithm>
#include <cstdint>

// References to hold for a job of n_tiles tiles whose frame at capture had `entries`
// of them; false when a frame like that one cannot be held.
//
// Room for cameras that meet more than these ones: a replay that overflows scans all
// records for every tile (batches of 20 views at random poses, 16 of one scene: with a
// twelfth of this room, the same bytes when an entry had 96, 19 of 60 replays with new
// cameras overflowed and took 4 to 15 ms; with this room none of 100 does and they take 2).
// A place is 32 bits wide, so a job of very many entries gets less than that.
inline bool graph_bin_capacity(uint64_t n_tiles, uint64_t entries, uint64_t* out)
{
    const uint64_t most = 0xffffffffull;
    if (std::max(n_tiles * 4, entries * 3 / 2) > most) return false;
    *out = std::min(most, std::max<uint64_t>(3u << 16, std::max(n_tiles * 48, entries * 18)));
    return true;
}
