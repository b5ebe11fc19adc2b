// How the cell scan splits the boxes' cells between blocks, in plain C++ so
// that the host can check it too. Cells are counted in chunks, one pass of a
// block each; the grid's x runs over a box's chunks, its y strides through the
// rebuilding boxes.
#pragma once

#include <stdint.h>

#include "vlj_place.h"

namespace vlj {

struct ScanShape {
    uint32_t x, y;   // the grid
    uint32_t least;  // chunks that a block takes in a run at least
};

// Every block reads the counts of its box up to its run, so one chunk a block
// makes those reads grow with the square of a box's chunks. That is right
// while the chunks of all boxes are some waves of blocks (each costs about 3
// us, reading what comes before it less than that); beyond, runs get longer,
// and the boxes themselves fill the chip.
inline ScanShape scan_shape(uint32_t chunks_of_all, uint32_t chunks_of_largest, uint32_t boxes, uint32_t sms) {
    ScanShape s;
    s.least = (chunks_of_all + 8u * sms - 1u) / (8u * sms);
    if (s.least < 1u) s.least = 1u;
    s.x = (chunks_of_largest + s.least - 1u) / s.least;
    if (s.x > 64u) s.x = 64u;
    s.y = (2u * sms + s.x - 1u) / s.x;
    if (s.y < 64u) s.y = 64u;
    if (s.y > boxes) s.y = boxes;
    return s;
}

// Chunks of each block's run in a box of `chunks`, with x blocks for it.
VLJ_HOST_DEVICE uint32_t scan_run(uint32_t chunks, uint32_t x, uint32_t least) {
    const uint32_t even = (chunks + x - 1u) / x;
    return even > least ? even : least;
}

// The stand-alone grid's scan (vlj_binning.cuh): blocks that take a run of
// `per` cells each, whole tiles of kScanTile, and no more blocks than there are
// particles (their sums lie in the order's buffer). Up to four tiles one block
// takes them all, which needs no sums and so a launch less: 22.6 us against
// 25.8 for a call over 4,913 cells, the same at 15,625, 27.8 against 25.8 at
// 19,683. Beyond, a tile a block.
constexpr uint32_t kScanTile = 4096;  // cells of one pass: four a thread
constexpr uint32_t kOneBlockTiles = 4;

struct BinRuns {
    uint32_t per, blocks;
};

inline BinRuns bin_runs(uint32_t cells, uint32_t particles) {
    const uint64_t tiles = ((uint64_t)cells + kScanTile - 1u) / kScanTile;
    const uint64_t runs = tiles <= kOneBlockTiles ? 1u : (tiles < particles ? tiles : particles);
    const uint64_t per = (tiles + runs - 1u) / runs * kScanTile;
    return {(uint32_t)per, (uint32_t)((cells + per - 1u) / per)};
}

// Whether the blocks' sums are needed, a launch of their own: a single block
// has nothing before its run.
inline bool bin_needs_sums(const BinRuns& r) { return r.blocks > 1u; }

}  // namespace vlj
