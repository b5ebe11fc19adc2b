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

}  // namespace vlj
