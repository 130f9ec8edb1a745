"""The diagnostics' potential does not depend on the walk's group size: a massless body more takes the size over a
limit of the rule (groups of 4 to 8, 8 to 16, 16 to 32), and with theta 0 every other body keeps the same float terms.
Their sum is kept with its rounding errors in a second float (each about 6e-8 of errors that are themselves below
half an ulp), so the rounded sums may differ for about one body in 10^4 and the energies by less than 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def potential(bh, pm, leaf):
    n = len(pm)
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, np.zeros_like(pm))
        sim.build(np.zeros(3), 16.0, leaf, bh.BH_MULTIPOLE_QUADRUPOLE)
        e, pot = sim.energy(0.0, 0.01, potential=True)
    return e["potential"], np.asarray(pot)


@pytest.mark.parametrize("leaf", [1, 8])
@pytest.mark.parametrize("limit", [12288, 24576, 196608])
def test_potential_across_group_sizes(bh, limit, leaf):
    rng = np.random.default_rng(limit)
    pm = np.zeros((limit, 4), np.float32)
    pm[:, :3] = np.clip(rng.normal(size=(limit, 3)), -7, 7)
    pm[:, 3] = 1.0 / limit
    pm[-1, 3] = 0.0
    e1, pot1 = potential(bh, pm, leaf)
    e0, pot0 = potential(bh, np.ascontiguousarray(pm[:-1]), leaf)
    assert np.mean(pot0 != pot1[:-1]) < 1e-3
    assert abs(e0 - e1) < 1e-10 * abs(e0)
