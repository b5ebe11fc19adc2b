"""Work that the caller captures into a CUDA graph of its own (with the
library's own graphs off, which cannot lie inside another). A captured pass over
the lists takes the rebuild decision on every launch of the graph, also when
the lists were up to date while it was captured, and a pass after a launch of a
captured step sees that step. The same bits as without capture."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BINS = 8
ENSEMBLES = ["none", "langevin", "nose_hoover", "exchange"]


def make(gpu, stream, ensemble):
    p = gpu.lattice(1000, 11.0, 1.0, 3)
    t = {"langevin": gpu.Langevin(1.0, 1.0, 5), "nose_hoover": gpu.NoseHoover(1.0, 0.5)}.get(ensemble)
    sim = gpu.LennardJones(p, gpu.Settings([11.0] * 3, dt=0.004, profile_bins=BINS, thermostat=t),
                           stream=stream.cuda_stream)
    if ensemble == "exchange":
        sim.set_heat_exchange(gpu.HeatExchange((0.0, 1.0), (5.5, 6.5), 0.01))
    sim.set_graphs(False)
    sim.step(30)
    sim.sample_profile()
    sim.measure_now()  # the lists are up to date
    sim.clear_profile()
    return sim


def profile(sim):
    p = sim.read_profile()
    return p.samples, np.array([[s.particles, *s.kinetic, *s.virial, s.potential] for s in p.slabs]).tobytes()


@pytest.mark.parametrize("ensemble", ENSEMBLES)
def test_captured_sample_takes_the_decision_on_each_launch(gpu, ensemble):
    import torch
    stream = torch.cuda.Stream()
    sim = make(gpu, stream, ensemble)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sim.sample_profile()
    sim.step(37)
    with torch.cuda.stream(stream):
        graph.replay()
    got = profile(sim)
    sim.close()
    twin = make(gpu, stream, ensemble)
    twin.step(37)
    twin.sample_profile()
    want = profile(twin)
    twin.close()
    assert got == want


@pytest.mark.parametrize("ensemble", ENSEMBLES)
def test_measurement_after_a_captured_step(gpu, ensemble):
    import torch
    stream = torch.cuda.Stream()
    sim = make(gpu, stream, ensemble)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sim.step(1)
    sim.measure_now()
    for _ in range(33):
        with torch.cuda.stream(stream):
            graph.replay()
        got = sim.measure_now()
    q = sim.read_particles()
    sim.close()
    twin = make(gpu, stream, ensemble)
    for _ in range(33):
        twin.step(1)
        want = twin.measure_now()
    r = twin.read_particles()
    twin.close()
    assert (got.potential, got.kinetic, got.virial, got.list_rebuilds) == \
        (want.potential, want.kinetic, want.virial, want.list_rebuilds)
    assert q.tobytes() == r.tobytes()
