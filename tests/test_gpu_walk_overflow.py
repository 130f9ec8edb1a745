"""Accelerations that overflow: infinite, with the sign of the pull, in every group size; the others finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("multipole", [0, 1])
@pytest.mark.parametrize("n", [2, 5, 20, 32])
def test_overflowing_pair(bh, n, multipole):
    # one leaf, one buffer of the walk: a body's terms meet nothing but each other
    rng = np.random.default_rng(n)
    pm = np.zeros((n, 4), np.float32)
    pm[:, :3] = rng.uniform(-1, 1, (n, 3))
    pm[:, 3] = 1.0
    pm[0], pm[1] = (1e-10, 2e-10, -1e-10, 1e20), (-1e-10, -2e-10, 1e-10, 1e20)
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, np.zeros_like(pm))
        sim.build(np.zeros(3), 2.5, 32, multipole)
        acc = sim.force(0.5, 0.0)[:, :3]
    inf = np.inf
    assert np.array_equal(acc[0], [-inf, -inf, inf]) and np.array_equal(acc[1], [inf, inf, -inf])
    assert np.isfinite(acc[2:]).all()
