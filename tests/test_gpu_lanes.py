"""Several lanes per particle in the force passes of small boxes.

The force is summed in parts of two list rows whatever the lanes, so the lanes
that a box's size selects (eight up to about 9,400 particles, four up to
18,900, two up to 37,800) and one lane give the same step to the bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, rho, thermostat", [
    (997, 0.8442, True), (1000, 0.03, False), (9470, 0.5, True), (9473, 0.5, False),
    (12001, 0.8442, True), (18950, 0.3, True), (30011, 0.6, False), (30011, 0.6, True)])
def test_lanes_of_each_size_match_one_lane(gpu, n, rho, thermostat):
    box = (n / rho) ** (1.0 / 3.0)
    p = gpu.lattice(n, box, 1.1, 4)
    t = gpu.Langevin(1.1, 1.0, 9) if thermostat else None
    out = []
    for lanes in (0, 1):
        sim = gpu.LennardJones(p, gpu.Settings([box] * 3, dt=0.004, thermostat=t, shifted_force=thermostat))
        sim.set_step_lanes(lanes)
        sim.run(40)
        m = sim.measure_now()
        q = sim.read_particles()
        out.append((q.tobytes(), m.potential, m.virial, m.kinetic, m.list_rebuilds))
        sim.close()
    assert out[0] == out[1]
