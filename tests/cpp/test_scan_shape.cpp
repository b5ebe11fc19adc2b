// The cell scan's split into blocks (csrc/vlj_scan_shape.h) on the host: every
// chunk of every box belongs to one block's run, and what the blocks read of
// the cells before their runs stays within a bound that does not grow with the
// boxes' size -- half a box for each of at most 64 blocks, and for sets of
// boxes that fill the chip by themselves a few boxes' worth. And the stand-alone
// grid's split, which launches a pass of sums only for more than one block.
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <vector>

#include "vlj_scan_shape.h"

static int failed = 0;

static void check(const std::vector<uint32_t>& chunks, double bound) {
    uint64_t all = 0;
    uint32_t most = 0;
    for (uint32_t c : chunks) {
        all += c;
        most = std::max(most, c);
    }
    const vlj::ScanShape s = vlj::scan_shape((uint32_t)all, most, (uint32_t)chunks.size(), 148u);
    if (s.x < 1 || s.x > 64 || s.y < 1 || s.y > chunks.size() || s.least < 1) failed++;
    uint64_t before = 0;
    for (uint32_t n : chunks) {
        const uint32_t run = vlj::scan_run(n, s.x, s.least);
        std::vector<uint32_t> taken(n, 0u);
        for (uint32_t block = 0; block < s.x; block++) {
            if (block * run >= n) continue;
            before += block * run;
            for (uint32_t c = block * run; c < std::min(n, (block + 1) * run); c++) taken[c]++;
        }
        for (uint32_t t : taken) failed += t != 1u;
    }
    if ((double)before > bound * (double)all) {
        printf("%zu boxes, the largest of %u chunks: %.1f times the cells read before the runs\n",
               chunks.size(), most, (double)before / (double)all);
        failed++;
    }
}

// The stand-alone grid's runs: all cells, whole tiles, sums for more than one
// block only, and no more sums than particles.
static void check_runs(uint32_t cells, uint32_t particles) {
    const vlj::BinRuns r = vlj::bin_runs(cells, particles);
    const uint64_t covered = (uint64_t)r.per * r.blocks;
    bool ok = r.per > 0 && r.per % vlj::kScanTile == 0 && covered >= cells && covered - r.per < cells;
    ok = ok && r.blocks <= particles && vlj::bin_needs_sums(r) == (r.blocks > 1u);
    ok = ok && (cells > vlj::kOneBlockTiles * vlj::kScanTile || !vlj::bin_needs_sums(r));
    if (!ok) {
        printf("%u cells, %u particles: %u blocks of %u\n", cells, particles, r.blocks, r.per);
        failed++;
    }
}

int main() {
    for (uint32_t cells : {1u, 27u, 512u, 4095u, 4096u, 4097u, 8192u, 8193u, 16384u, 16385u, 216000u, 262143u, 262144u})
        for (uint32_t n : {1u, 2u, 3u, 10u, 63u, 64u, 65u, 100000u, 2147483647u}) check_runs(cells, n);
    for (uint32_t n : {1u, 2u, 63u, 64u, 65u, 68u, 127u, 252u, 256u}) {
        check({n}, 32.0);
        check(std::vector<uint32_t>(5, n), 32.0);
        check(std::vector<uint32_t>(128, n), 6.0);
        check(std::vector<uint32_t>(400, n), 6.0);
        std::vector<uint32_t> mixed(512, 1u);
        mixed[100] = n;
        check(mixed, 32.0);
        for (size_t b = 0; b < mixed.size(); b++) mixed[b] = 1u + (uint32_t)b * n / 512u;
        check(mixed, 32.0);
    }
    printf("%d failed\n", failed);
    return failed != 0;
}
