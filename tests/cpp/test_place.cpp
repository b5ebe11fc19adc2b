// The stand-alone grid's scatter place (csrc/vlj_place.h) on the host.
//
// Each particle of a cell takes one off the cell's counter. Alone, the places
// are each cell's own, all of them. When another call clears the counters
// after `done` of the particles (two calls that overlap on one scratch), the
// order is undefined, but no place may lie outside the n words of the buffer.
#include <stdint.h>
#include <stdio.h>

#include <vector>

#include "vlj_place.h"

int main() {
    const std::vector<std::vector<uint32_t>> sets = {{1}, {2}, {3, 1}, {0, 5}, {4, 0, 0, 9}, {40, 1, 300}};
    int failed = 0;
    for (const auto& cells : sets) {
        std::vector<uint32_t> start(cells.size()), of;
        for (size_t c = 0; c < cells.size(); c++) {
            start[c] = (uint32_t)of.size();
            of.insert(of.end(), cells[c], (uint32_t)c);
        }
        const uint32_t n = (uint32_t)of.size();
        for (uint32_t done = 0; done <= n; done++) {  // done == n: nothing overlaps
            std::vector<uint32_t> left(cells), written(n, 0u);
            for (uint32_t i = 0; i < n; i++) {
                if (i == done) left.assign(cells.size(), 0u);
                uint32_t at = 0;
                if (!vlj::scatter_place(start[of[i]], left[of[i]]--, n, &at)) continue;
                if (at >= n) {
                    printf("place %u of %u, cleared after %u\n", at, n, done);
                    failed++;
                } else {
                    written[at]++;
                }
            }
            if (done == n)
                for (uint32_t k = 0; k < n; k++)
                    if (written[k] != 1u) failed++;
        }
    }
    printf("%d failed\n", failed);
    return failed != 0;
}
