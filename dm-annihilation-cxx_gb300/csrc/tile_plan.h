// tile_plan.h -- sizes of the tiled render's buffers (disc_tile.cu) and the
// choice between the renders of a large chunk, in a header a host compiler
// also takes, so both are unit-tested on the CPU.
#pragma once
#include <algorithm>
#include <cstddef>

#include "seg_plan.h"

namespace dmann {

// A tile is kTileR rings by kTileW in-ring pixel indices, a unit up to
// kUnitMax discs of its list (fewer while the chunk has less than kUnitTarget
// units of more than kUnitMin).  A unit's FP32 sums are rounded by 1.7e-8 of their
// total at each addition, so a pixel of M deposits is off by 1.7e-8 kUnitMax /
// sqrt(3 M): with units of 512 that was most of the error of a map's bright
// regions (7e-8 of 1M particles at Nside 512, 4.8e-8 with 128), and their flush
// is as little of the time either way.
constexpr int kTileR = 32, kTileW = 64;
constexpr int kUnitMin = 32, kUnitMax = 128, kUnitTarget = 16384;
constexpr int kTileClasses = 64;
constexpr int kTileLists = 4;

inline int tile_strips(int nside) { return (4 * nside - 1 + kTileR - 1) / kTileR; }
inline int tile_cols(int nside) { return (4 * nside + kTileW - 1) / kTileW; }

// The class of a disc in its tile's list, whose classes are summed in ascending
// order: the biased FP32 exponent oct of its deposit scale below the chunk's
// largest, omax, in as few octaves per class as hold the smallest, omin (one
// up to a range of 2^64, four for every float).  So in one FP32 sum of at most
// kUnitMax discs an addend (weights are above exp(-6) = 2^-8.7) is never below
// 2^-(9 + 4 + 8.7) of the pixel's total before it, and no small deposit is lost
// on a large total.
DMANN_HD inline int tile_class(int oct, int omax, int omin) {
    return kTileClasses - 1 - (omax - oct) / ((omax - omin) / kTileClasses + 1);
}

// Every disc of a chunk in every tile.
inline size_t tile_pairs_bound(size_t n, int nside) {
    return (n > 0 ? n : 1) * (size_t)tile_strips(nside) * (size_t)tile_cols(nside);
}
// Pair list slots that the tiled render asks for: every disc in every tile
// where that is little (then no chunk can exceed it), else 96 per particle and
// 2^24 (a disc of the 16M set at Nside 2048 touches 33 tiles, one of the 134M set
// at Nside 4096 about 55; chunks with more pairs are segmented).
inline size_t tile_capacity(size_t n, int nside) {
    return std::min(tile_pairs_bound(n, nside), 96 * n + ((size_t)1 << 24));
}
// Fewer are of no use, and more than the list holds are not used.
inline size_t tile_least(size_t n, int nside) {
    return std::min(tile_pairs_bound(n, nside), 8 * n + ((size_t)1 << 16));
}
inline size_t tile_slots(size_t n, int nside, size_t list) {
    return list >= tile_least(n, nside) ? std::min(list, tile_capacity(n, nside)) : 0;
}
// Discs per unit of a list of `pairs`, and the units it makes at most on nt tiles.
DMANN_HD inline int tile_unit_len(long long pairs) {
    const long long k = pairs / kUnitTarget;
    return (int)(k < kUnitMin ? kUnitMin : k > kUnitMax ? kUnitMax : k);
}
DMANN_HD inline long long tile_units_of(long long pairs, long long nt) { return pairs / tile_unit_len(pairs) + nt; }
// The units of all lists, one behind the other.
inline size_t tile_unit_capacity(size_t slots, int nside) {
    return slots / kUnitMax + kTileLists * (2 * (size_t)kUnitTarget + (size_t)tile_strips(nside) * (size_t)tile_cols(nside));
}
inline bool tile_always_fits(size_t n, int nside, size_t slots) { return slots >= tile_pairs_bound(n, nside); }

// dmann_tuning.large_render
enum { kLargeAny = 1, kLargeTiles = 2, kLargeSegments = 3 };

// The renders launched for a chunk that may be large, from the buffers there
// are: the segments are of use where the pair list can overflow, and there the
// chunk's pairs are counted whether or not there are segments to take it -- the
// pair list's kernels write as many slots as there are pairs.
struct LargePlan {
    bool tile, seg;
    bool count;   // k_tile_pairs<0> before the mode is decided
};
inline LargePlan plan_large(bool have_tile, bool always_fits, bool have_seg) {
    const bool sure = have_tile && always_fits;
    return LargePlan{have_tile, have_seg && !sure, have_tile && !sure};
}

// A chunk's mode (k_seg_decide): 2 tiles, 1 segments, 0 per-disc kernels.
// From min_est estimated deposits on it is rendered by tiles where the pair
// list (pair_cap slots; 0: none) holds its pairs (0 when they need no count),
// else in segments where the item buffers (item_cap; 0: none) hold its items,
// else (and below min_est) by the per-disc kernels with FP64 deposits.
DMANN_HD inline int large_mode(long long est, long long min_est, long long blocks, long long pairs,
                               long long pair_cap, long long items, long long item_cap) {
    if (est < min_est || blocks <= 0) return 0;
    if (pair_cap > 0 && pairs <= pair_cap) return 2;
    return items > 0 && items <= item_cap ? 1 : 0;
}

}  // namespace dmann
