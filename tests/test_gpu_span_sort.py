"""Sorts by tiles with a middle merge of 32 tiles (spans of 4096 or 8192 keys): sizes around a span, around the
limits between two and three launches and the radix sort, keys with heavy ties; and steps of such systems, whose
order and positions are those of the same bodies as an ensemble of one system, which sorts otherwise."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("n", [32768, 32769, 36863, 36865, 65535, 65537, 73728, 73729, 81920 + 31, 163840, 163841])
def test_sort_bodies(bh, orc, n, ties):
    rng = np.random.default_rng(n)
    pm = np.zeros((n, 4), np.float32)
    pm[:, 3] = 1.0 / n
    pm[:, :3] = rng.integers(-3, 4, (n, 3)) if ties else rng.normal(size=(n, 3))
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, np.zeros_like(pm))
        keys = sim.morton_keys(16.0)
        assert np.array_equal(sim.sort_bodies(), orc.sort_perm(keys))


@pytest.mark.parametrize("n", [65536, 65537, 73729, 98305, 163840, 163841])
def test_step_orders_like_an_ensemble(bh, n):
    rng = np.random.default_rng(n)
    pm = np.zeros((n, 4), np.float32)
    pm[:, :3] = rng.normal(size=(n, 3))
    pm[: n // 3, :3] = pm[n // 3 : 2 * (n // 3), :3]  # equal keys
    pm[:, 3] = 1.0 / n
    vel = rng.normal(size=(n, 4)).astype(np.float32) * 0.1
    vel[:, 3] = np.arange(n)  # body ids travel in w
    prm = bh.default_params(theta=1.2, eps=0.05, dt=1e-2, leaf_capacity=8)
    out = []
    for batch in (False, True):
        with bh.Simulation(n) as sim:
            if batch:
                sim.batch_set(pm, vel, np.array([0, n], np.uint32))
                sim.batch_step(prm, 2)
            else:
                sim.set_bodies(pm, vel)
                sim.step(prm, 2)
            out.append(sim.get_bodies())
    (p, v, _), (bp, bv, _) = out
    assert np.array_equal(v[:, 3], bv[:, 3])
    assert np.allclose(p, bp, rtol=0, atol=1e-5)  # one step's force differs by rounding: dt^2 of it


@pytest.mark.parametrize("n", [65537, 73729, 163841])
def test_differentiable_path_follows_the_step(bh, n):
    rng = np.random.default_rng(n)
    pm = np.zeros((n, 4), np.float32)
    pm[:, :3] = rng.normal(size=(n, 3))
    pm[:, 3] = 1.0 / n
    vel = rng.normal(size=(n, 4)).astype(np.float32) * 0.1
    vel[:, 3] = np.arange(n)
    prm = bh.default_params(theta=1.2, eps=0.05, dt=1e-2, leaf_capacity=8)
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, vel)
        sim.adjoint_forward(prm, 2, 2)
        pa, va, _ = sim.get_bodies()
    with bh.Simulation(n) as sim:  # a(x0) first, as the differentiable path has it
        sim.set_bodies(pm, vel)
        sim.adjoint_forward(prm, 1, 1)
        p1, v1, _ = sim.get_bodies()
    assert np.array_equal(va[:, 3], np.arange(n))
    # the second of the two steps again, from the state after the first
    with bh.Simulation(n) as sim:
        sim.set_bodies(p1, v1)
        sim.adjoint_forward(prm, 1, 1)
        p2, v2, _ = sim.get_bodies()
    assert np.allclose(pa, p2, rtol=0, atol=1e-5)
    # and a tree of the final positions gives each body the direct sum's force to the opening error
    tgt = np.arange(0, n, max(1, n // 257))
    d = p1[None, :, :3].astype(np.float64) - p1[tgt, None, :3].astype(np.float64)
    acc = (d * (p1[None, :, 3:4] / ((d * d).sum(-1) + 0.05**2)[..., None] ** 1.5)).sum(1)
    # p2 = p1 + dt v1 + dt^2/2 a(x1); the tree's a is within 3e-2 of |a| ~ 1
    want = p1[tgt, :3] + 1e-2 * v1[tgt, :3] + 0.5e-4 * acc
    assert np.abs(p2[tgt, :3] - want).max() < 0.5e-4 * 3e-2 * np.abs(acc).max() + 1e-6
