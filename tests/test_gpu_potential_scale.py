"""Potentials at scales where factors of their terms are denormal floats, which the diagnostics keep: squared
distances of tiny systems, without a softening too, against FP64 direct sums; and 1 / D^5 of the cells' quadrupoles in
large ones, against the same system at another scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("multipole", [0, 1])
@pytest.mark.parametrize("scale", [1.0, 1e-19, 1e-20])
def test_potential_at_small_scales(bh, scale, multipole):
    # a jittered lattice: distances from 0.5 to 11 of the scale, squares down to 2.5e-41, 2e4 denormal steps;
    # theta 0 takes every pair directly
    k = 7
    rng = np.random.default_rng(k)
    x = np.stack(np.meshgrid(*[np.arange(k) - (k - 1) / 2] * 3, indexing="ij"), -1).reshape(-1, 3)
    n = len(x)
    pm = np.zeros((n, 4), np.float32)
    pm[:, :3] = (x + rng.uniform(-0.2, 0.2, x.shape)) * scale
    pm[:, 3] = rng.uniform(0.5, 1.5, n) / n
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, np.zeros_like(pm))
        sim.build(np.zeros(3), 16.0 * scale, 4, multipole)
        e, pot = sim.energy(0.0, 0.0, potential=True)
    p = pm.astype(np.float64)
    r = np.linalg.norm(p[:, None, :3] - p[None, :, :3], axis=-1)
    np.fill_diagonal(r, np.inf)
    want = -(p[None, :, 3] / r).sum(1)
    assert np.abs(pot / want - 1).max() < 1e-4  # half a step of the closest squares: 2.5e-5, half that in 1 / D
    assert abs(e["potential"] / (0.5 * (p[:, 3] * want).sum()) - 1) < 1e-4


def test_quadrupoles_at_large_scales(bh):
    # 2^25: a change of exponents only, so the potentials are the same times 2^-25 but for 1 / D^5, which is
    # denormal for D above 1.2 of the scale. Below 8 of it its half step is 2^-10 of it, and the quadrupole terms are
    # a few hundredths of a potential at theta 1.
    n, scale = 1000, 2.0**25
    pm, vel = bh.plummer(6, n)
    pot = []
    for k in (1.0, scale):
        p = pm.copy()
        p[:, :3] *= np.float32(k)
        with bh.Simulation(n) as sim:
            sim.set_bodies(p, vel)
            c, size = sim.bounds()
            sim.build(c, 2 * size, 4, 1)
            pot.append(sim.energy(1.0, 0.0, potential=True)[1] * k)
    assert np.linalg.norm(pot[1] - pot[0]) < 1e-4 * np.linalg.norm(pot[0])


@pytest.mark.parametrize("others", [0, 5, 13000])
def test_overflowing_pair(bh, others):
    """Two bodies whose m / D is no float have infinite potentials, not ones that are no numbers; a far body's
    stay finite."""
    n = 2 + others
    rng = np.random.default_rng(others)
    pm = np.zeros((n, 4), np.float32)
    pm[:, :3] = rng.uniform(-1, 1, (n, 3))
    pm[:, 3] = 1.0
    pm[0], pm[1] = (1e-10, 0, 0, 1e30), (-1e-10, 0, 0, 1e30)
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, np.zeros_like(pm))
        sim.build(np.zeros(3), 2.5, 4, 1)
        e, pot = sim.energy(0.0, 0.0, potential=True)
    assert np.array_equal(pot[:2], [-np.inf, -np.inf]) and np.isfinite(pot[2:]).all()
    assert e["potential"] == -np.inf
