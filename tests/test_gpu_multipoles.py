"""Node multipoles summed straight from the bodies: sizes on both sides of each limit of the split (thread,
team, warp and block nodes; chunk and super records; systems whose small nodes go one per thread), against
the oracle's upsweep. Bars as in the parity tests: mass and centre float-float (about 44 bits) against FP64,
quadrupole FP32 against its natural scale mass * edge^2, literal barycentres bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sorted_build(sim, pm, vel, leaf, mode):
    sim.set_bodies(pm, vel)
    c, size = sim.bounds()
    sim.morton_keys(size)
    sim.sort_bodies()
    p, _, _ = sim.get_bodies()
    sim.build(c, 2 * size, leaf, mode)
    return p[:, :3].astype(np.float64), p[:, 3].astype(np.float64), c, 2 * size, sim.tree_nodes()


@pytest.mark.parametrize("n,leaf,two", [
    (2, 1, False), (9, 4, False), (16, 16, False), (17, 1, False), (129, 64, False), (1025, 1, False),
    (1100, 200, True), (8192, 1, False), (8193, 1, False), (20000, 1, True), (65536, 8, False), (65537, 8, False),
    (70001, 1, True), (262144, 16, False), (262145, 8, True),
])
def test_multipoles_match_oracle(bh, orc, n, leaf, two):
    pm, vel = bh.two_spheres(n, n) if two else bh.plummer(n, n)
    pm[:, 3] *= np.random.default_rng(n).lognormal(0.0, 1.0, n).astype(np.float32)
    with bh.Simulation(n) as sim:
        for mode in (1, 0):
            pos, mass, c, edge, t = sorted_build(sim, pm, vel, leaf, mode)
            ref = orc.build(pos, mass, c, edge, leaf, mode)
            assert np.array_equal(t["keys"], ref["keys"]) and np.array_equal(t["counts"], ref["counts"])
            assert np.allclose(t["mass"], ref["mass"], rtol=1e-11)
            if mode == 0:
                assert np.array_equal(t["com"], ref["com"])
                continue
            assert np.allclose(t["com"], ref["com"], rtol=1e-9, atol=1e-11)
            depth = np.array([(int(k).bit_length() - 1) // 3 for k in t["keys"]])
            scale = ref["mass"] * (edge / 2.0 ** depth) ** 2
            assert np.all(np.abs(t["quad"] - ref["quad"]) <= 1e-5 * scale[:, None])


def test_massless_and_coincident_bodies(bh):
    """Zero masses give zero multipoles, coincident bodies their common point: every record stays finite."""
    n = 9000
    pm, vel = bh.plummer(3, n)
    pm[:4000, 3] = 0.0
    pm[5000:7000, :3] = pm[5000, :3]
    with bh.Simulation(n) as sim:
        _, _, _, _, t = sorted_build(sim, pm, vel, 1, 1)
        for k in ("mass", "com", "quad"):
            assert np.all(np.isfinite(t[k]))
        # the FP32 masses add up in the root within float-float rounding
        assert abs(t["mass"][0] - pm[:, 3].astype(np.float64).sum()) <= 1e-11
