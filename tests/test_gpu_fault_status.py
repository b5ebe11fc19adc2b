"""What the calls report once a kernel has recorded a fault. The fault word is
written from the host: no kernel fails here. A measurement reports the fault it
came with and no earlier one, and written particles are a fresh state."""

import pytest

pytestmark = pytest.mark.gpu


def make(gpu):
    p = gpu.lattice(1000, 11.0, 1.0, 3)
    return p, gpu.LennardJones(p, gpu.Settings([11.0] * 3, dt=0.004))


def test_waiting_calls_report_the_fault(gpu):
    _, sim = make(gpu)
    sim.run(3)
    for code, status in ((1, "TIMEOUT"), (9, "CUDA_ERROR")):
        sim.set_fault(code)
        for call in (sim.measure_now, sim.read_particles, lambda: sim.run(1)):
            with pytest.raises(gpu.VljError) as e:
                call()
            assert e.value.status == status
    sim.set_fault(0)
    sim.run(1)
    sim.close()


def test_a_polled_fault_does_not_outlive_its_state(gpu):
    p, sim = make(gpu)
    sim.run(3)
    sim.set_fault(1)
    assert sim.measure()
    sim.set_fault(1)  # waits for the measurement
    assert len(sim.poll()) == 1
    sim.write_particles(p)  # a fresh state, no fault
    got = sim.measure_now()
    sim.close()
    _, fresh = make(gpu)
    want = fresh.measure_now()
    fresh.close()
    assert abs(got.potential - want.potential) <= 1e-6 * abs(want.potential)
    assert abs(got.kinetic - want.kinetic) <= 1e-12 * want.kinetic + 1e-6
