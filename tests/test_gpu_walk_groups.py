"""The walk's group size follows the number of bodies (4, 8, 16 or 32 bodies per warp; the smaller ones
split the warp into slots that share the entries): each size, partly empty last groups and both sides of
the limits, against the oracle's walk within the parity bars."""
import numpy as np
import pytest

from oracle.oracle import relerr

pytestmark = pytest.mark.gpu

MED, P99 = 1e-5, 1e-4


@pytest.mark.parametrize("n,leaf,mode,eps", [
    (2, 1, 1, 0.01), (5, 1, 0, 0.0), (31, 4, 1, 0.0), (1001, 1, 0, 0.01), (1003, 8, 1, 0.0),
    (12287, 1, 1, 0.01), (12289, 8, 0, 0.01), (24575, 2, 1, 0.01), (24577, 16, 1, 0.01), (24578, 8, 0, 0.0),
    (196607, 8, 1, 0.01), (196609, 16, 0, 0.01),
])
def test_every_group_size_matches_oracle(bh, orc, n, leaf, mode, eps):
    pm, vel = bh.plummer(40 + n, n)
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, vel)
        c, size = sim.bounds()
        sim.morton_keys(size)
        sim.sort_bodies()
        sim.build(c, 2 * size, leaf, mode)
        acc, st = sim.force(0.6, eps, stats=True)
        p, _, _ = sim.get_bodies()
    pos, mass = p[:, :3].astype(np.float64), p[:, 3].astype(np.float64)
    ref, ncell, npt = orc.force(pos, mass, c, 2 * size, leaf, mode, 0.6, eps, nthreads=8)
    err = relerr(acc, ref)
    assert float(np.median(err)) <= MED and float(np.percentile(err, 99)) <= P99
    assert st.error_flags == 0
    if mode:
        assert abs(st.interactions_cell - int(ncell.sum())) <= 1e-4 * ncell.sum() + 2
        assert abs(st.interactions_p2p - int(npt.sum())) <= 1e-4 * npt.sum() + 2


def test_small_ensemble_groups_match_single_systems(bh):
    """Ensembles take their group size from all their bodies: one of few and one of more bodies."""
    for sizes in ([3, 40, 700, 1], [5000, 9000, 64], [30000, 1000]):
        parts = [bh.plummer(7 + s, k) for s, k in enumerate(sizes)]
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
        prm = bh.default_params(theta=0.6, eps=0.01, dt=1e-3, leaf_capacity=4)
        pm, vv = (np.concatenate(x) for x in zip(*parts))
        with bh.Simulation(len(pm)) as sim:
            sim.batch_set(pm, vv, off)
            sim.batch_step(prm, 1)
            bp, bv, ba = sim.get_bodies()
        for s, k in enumerate(sizes):
            if k < 2:
                continue
            with bh.Simulation(k) as one:
                one.set_bodies(*parts[s])
                one.step(prm, 1)
                p, v, a = one.get_bodies()
            sl = slice(off[s], off[s + 1])
            assert np.allclose(bp[sl], p, rtol=0, atol=1e-6) and np.allclose(bv[sl], v, rtol=0, atol=1e-6)
            assert float(np.percentile(relerr(ba[sl], a), 99)) <= 1e-5


@pytest.mark.parametrize("n,leaf,mode", [(2, 1, 1), (33, 4, 0), (1001, 1, 1), (12289, 8, 1), (24577, 8, 0), (196609, 16, 1)])
def test_potential_of_every_group_size(bh, n, leaf, mode):
    """phi at theta = 0 is the direct sum (coincident bodies left out); at theta = 0.5 it follows it within the
    quadrupole tree's accuracy. FP64 reference on a seeded subset of the bodies."""
    pm, vel = bh.plummer(60 + n, n)
    if n > 100:
        pm[7, :3] = pm[70, :3]
    eps = 0.01
    rng = np.random.default_rng(n)
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, vel)
        c, size = sim.bounds()
        sim.build(c, 2 * size, leaf, mode)
        e0, phi0 = sim.energy(0.0, eps, potential=True) if n < 50000 else (None, None)
        e1, phi1 = sim.energy(0.5, eps, potential=True)
    x, m = pm[:, :3].astype(np.float64), pm[:, 3].astype(np.float64)
    pick = np.unique(np.concatenate([rng.integers(0, n, 60), [0, min(7, n - 1), min(70, n - 1)]]))
    ref = np.empty(len(pick))
    for k, i in enumerate(pick):
        r2 = ((x - x[i]) ** 2).sum(1)
        ref[k] = -(m[r2 > 0] / np.sqrt(r2[r2 > 0] + eps * eps)).sum()
    if phi0 is not None:
        # n terms in FP32 with a compensated sum: rsqrt (2 ulp) and the rounding of each term
        assert np.all(np.abs(phi0[pick] - ref) <= 1e-6 * np.abs(ref) + 1e-12)
        assert abs(e0["potential"] - 0.5 * float((m * phi0).sum())) <= 1e-9 * abs(e0["potential"])
    if mode:
        assert np.median(np.abs(phi1[pick] - ref) / np.abs(ref).clip(1e-12)) <= 1e-3
