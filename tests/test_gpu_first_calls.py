"""What the first call of a fresh simulation costs. Steps run from captured
graphs, and capturing one costs about as much per step of the graph as several
steps of a small box take. A first call captures the graph of 16 steps (when it
has 16) and that of one step, whatever is left over; the graph of four steps
comes later, and the trajectory is the same with it."""

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
    # 15 steps without a graph: some 250 us (1,200 with graphs of 8, 4 and 2)
    assert first(gpu, 15) - one < 0.5 * capture
    # 15 more than a whole graph: some 450 us (1,300)
    assert first(gpu, 31) - whole < 0.7 * capture


def test_the_short_graph_keeps_the_trajectory(gpu):
    out = []
    for graphs in (True, False):
        sim = make(gpu)
        sim.set_graphs(graphs)
        for k in range(40):  # the 32nd call with four steps left over captures their graph
            sim.step(4 + k % 3)
        out.append(sim.read_particles().tobytes())
        sim.close()
    assert out[0] == out[1]
