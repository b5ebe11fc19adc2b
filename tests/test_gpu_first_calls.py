"""What the first call of a fresh simulation costs. Steps run from captured
graphs, and capturing one costs about as much per step of the graph as several
steps of a small box take. A first call captures the graph of 16 steps (when it
has 16) and that of one step, whatever is left over; the graphs of 8, 4 and 2
steps come later, and the trajectory is the same with them."""

import time

import pytest

pytestmark = pytest.mark.gpu


def make(gpu):
    side = (1000 / 0.8442) ** (1.0 / 3.0)
    return gpu.LennardJones(gpu.lattice(1000, side, 0.72, 3), gpu.Settings([side] * 3, dt=0.004))


def first(gpu, steps):
    """Shortest time of a fresh simulation's first run of `steps`, in us."""
    best = 1e9
    for _ in range(5):
        sim = make(gpu)
        t = time.perf_counter()
        sim.run(steps)
        best = min(best, time.perf_counter() - t)
        sim.close()
    return best * 1e6


def test_a_first_call_captures_no_graph_for_its_rest(gpu):
    first(gpu, 31)  # the kernels are loaded
    one, whole = first(gpu, 1), first(gpu, 16)
    capture = whole - one  # 16 steps and their graph, about 1,300 us
    # 15 steps one by one: some 250 us (1,200 with graphs of 8, 4 and 2 captured)
    assert first(gpu, 15) - one < 0.5 * capture
    # 15 more than a whole graph: some 450 us (1,300)
    assert first(gpu, 31) - whole < 0.7 * capture


def test_later_graphs_keep_the_trajectory(gpu):
    out = []
    for graphs in (True, False):
        sim = make(gpu)
        sim.set_graphs(graphs)
        for k in range(100):  # the 32nd call with a use for it captures each graph
            sim.step((15, 6, 4, 3)[k % 4] if k < 90 else 15)
        out.append(sim.read_particles().tobytes())
        sim.close()
    assert out[0] == out[1]
