"""Several lanes per particle in the force passes of small boxes.

The forces and energies are summed in parts of two list rows whatever the lanes,
so the lanes that a box's size selects (eight up to about 9,400 particles, four
up to 18,900, two up to 37,800), one lane and any other number give the same bits
in every pass: the steps of each ensemble, measurements, particles out, batches.
"""

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


def everything(sim):
    """What the lanes' passes leave: the measurement with its partial sums, the
    drawn values of both kinds and the particles."""
    m = sim.measure_now()
    out = [m.potential, m.virial, m.kinetic, tuple(m.momentum), m.condensed, m.thermostat_energy,
           m.list_rebuilds] + [a.tobytes() for a in sim.read_partials()] + [sim.read_vel4().tobytes()]
    return out + [sim.read_particles().tobytes(), sim.read_vel4().tobytes()]


# sizes that leave a last block and a last warp partly empty with any lanes
@pytest.mark.parametrize("ensemble", ["none", "langevin", "nose_hoover", "exchange"])
@pytest.mark.parametrize("n", [1003, 2462, 40001])
def test_every_pass_gives_the_same_bits_with_any_lanes(gpu, ensemble, n):
    side = (n / 0.6) ** (1.0 / 3.0)
    p = gpu.lattice(n, side, 1.1, 4)
    t = {"langevin": gpu.Langevin(1.1, 1.0, 9), "nose_hoover": gpu.NoseHoover(1.1, 0.5)}.get(ensemble)
    out = []
    for lanes in (1, 0, 2, 4, 8):
        sim = gpu.LennardJones(p, gpu.Settings([side] * 3, dt=0.002, thermostat=t,
                                               shifted_force=ensemble != "langevin"))
        sim.set_step_lanes(lanes)
        sim.write_particles(p)  # the first forces by these lanes too
        if ensemble == "exchange":
            sim.set_heat_exchange(gpu.HeatExchange((0.0, side / 6), (side / 2, side * 2 / 3), 0.01))
        sim.run(31)
        got = everything(sim)
        sim.set_drawn(gpu.Drawn.TEMPERATURE)
        out.append(got + everything(sim))
        sim.close()
    for k in range(1, 5):
        assert out[k] == out[0]


def test_batch_gives_the_same_bits_with_any_lanes(gpu):
    reps = []
    for r, n in enumerate([531, 1000, 2047, 777, 3333]):
        side = (n / (0.2 + 0.15 * r)) ** (1.0 / 3.0)
        reps.append(gpu.Replica(gpu.lattice(n, side, 1.0, r), [side] * 3,
                                gpu.Langevin(1.0, 1.0, r) if r % 2 else None))
    out = []
    for lanes in (1, 0, 2, 4, 8):
        b = gpu.Batch(reps, dt=0.004)
        b.set_step_lanes(lanes)
        b.run(31)
        ms = [(m.potential, m.virial, m.kinetic, tuple(m.momentum), m.list_rebuilds) for m in b.measure()]
        out.append((ms, [b.read_particles(r).tobytes() for r in range(len(reps))]))
        b.close()
    for k in range(1, 5):
        assert out[k] == out[0]


def test_refused_lanes(gpu):
    sim = gpu.LennardJones(gpu.lattice(1000, 11.0, 1.0, 3), gpu.Settings([11.0] * 3))
    for lanes in (3, 5, 6, 7, 9, 16):
        with pytest.raises(gpu.VljError) as e:
            sim.set_step_lanes(lanes)
        assert e.value.status == "INVALID_ARG"
    sim.close()
