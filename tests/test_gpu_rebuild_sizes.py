"""The rebuild chain at the sizes where its launches change shape: the number
of particles at which the list build stops splitting cells, the parts it
splits them into, and the number of cells at which the scan takes another
block, or its blocks another chunk. Cell grid and lists against the oracle, bit
for bit, on a first build and on later ones that reorder or don't."""

import pytest

from test_gpu_parity import compare_rebuild

pytestmark = pytest.mark.gpu

CASES = {
    # particles: parts of two homes, of more, and none
    "split_2": (2399, [14.2] * 3), "split_3": (4801, [17.9] * 3), "split_8": (19200, [28.4] * 3),
    "whole_cells": (19201, [28.4] * 3), "split_narrow": (2000, [13.3] * 3),
    # cells: one chunk of 4,096 exactly, one cell row more, several chunks,
    # and more chunks than the grid has blocks
    "one_chunk": (3000, [44.9] * 3), "one_chunk_and_a_row": (3000, [44.9, 44.9, 47.7]),
    "chunks_dilute": (30000, [70.1, 84.1, 98.1]), "chunks_again": (25000, [182.1] * 3),
    "chunks_most": (25000, [283.5] * 3),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_rebuild_at_the_edges_of_its_launches(gpu, O, case):
    n, box = CASES[case]
    p = gpu.lattice_box(n, box, 1.3, 6)
    sim = gpu.LennardJones(p, gpu.Settings(box, dt=0.005, thermostat=gpu.Langevin(1.3, 1.0, 6)))
    # 48 steps are whole graphs; of 45 the last ones run one by one and leave
    # their decision for the next step, to which a forced rebuild adds
    for steps in (48, 45):
        sim.run(steps)
        pre = sim.read_grid()
        before = sim.grid_info().rebuilds
        sim.force_rebuild()
        compare_rebuild(sim, O, dict(x=pre["x"], v=pre["v"], ids=pre["ids"]), before % 4 == 0)
    sim.close()


def test_scan_of_more_cells_than_some_waves_of_blocks(gpu):
    # six boxes of 1,030,301 cells each: blocks take runs of chunks that a box
    # by itself would not; the same trajectories as the boxes by themselves
    box = [283.5] * 3
    parts = [gpu.lattice_box(1500 + 7 * r, box, 1.2, r) for r in range(6)]
    batch = gpu.Batch([gpu.Replica(p, box, None) for p in parts], dt=0.005)
    batch.run(37)
    got = [batch.read_particles(r) for r in range(6)]
    rebuilds = [m.list_rebuilds for m in batch.measure()]
    batch.close()
    for p, q, n in zip(parts, got, rebuilds):
        sim = gpu.LennardJones(p, gpu.Settings(box, dt=0.005))
        sim.run(37)
        assert sim.read_particles().tobytes() == q.tobytes()
        assert sim.measure_now().list_rebuilds == n > 2
        sim.close()
