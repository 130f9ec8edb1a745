"""The two-launch sort (512-key tiles, then their merge): sizes around a tile, a block of the merge and the
limit of the rule, keys with heavy ties, already sorted and reversed, against the oracle's stable sort; and
ensembles, whose pairs sort by (system, key), with systems that share and straddle tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def positions(kind, n, rng):
    """Positions whose Morton order is random, tied or nearly the input order."""
    pm = np.zeros((n, 4), np.float32)
    pm[:, 3] = 1.0 / n
    if kind == "ties":
        pm[:, :3] = rng.integers(-2, 3, (n, 3))
    elif kind == "same":
        pm[:, :3] = 0.25
    else:
        pm[:, :3] = rng.normal(size=(n, 3))
    pm[0, :3], pm[-1, :3] = (4.0, -4.0, 4.0), (-4.0, 4.0, -4.0)
    return pm


@pytest.mark.parametrize("kind", ["random", "ties", "same"])
@pytest.mark.parametrize("n", [2, 31, 33, 511, 512, 513, 1024, 1055, 16384, 16897, 98303, 98304, 98305])
def test_sort_bodies_matches_stable_sort(bh, orc, n, kind):
    rng = np.random.default_rng(n)
    pm = positions(kind, n, rng)
    with bh.Simulation(n) as sim:
        for order in (np.arange(n), np.arange(n)[::-1]):
            p = np.ascontiguousarray(pm[order])
            sim.set_bodies(p, np.zeros_like(p))
            keys = sim.morton_keys(5.0)
            perm = sim.sort_bodies()
            assert np.array_equal(perm, orc.sort_perm(keys))
            # a second sort of the sorted bodies is the identity
            sim.morton_keys(5.0)
            assert np.array_equal(sim.sort_bodies(), np.arange(n, dtype=np.uint32))


@pytest.mark.parametrize("sizes", [[1] * 700 + [512, 513, 511, 3], [1024, 1, 2000, 17, 512, 512, 40],
                                   [30000, 5, 60000], [16384] * 3 + [7] * 100, [16385, 90000]])
def test_ensembles_sort_like_single_systems(bh, sizes):
    rng = np.random.default_rng(len(sizes))
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    n = int(off[-1])
    pm = np.zeros((n, 4), np.float32)
    pm[:, :3] = rng.normal(size=(n, 3))
    pm[:, 3] = 1e-3
    vel = rng.normal(size=(n, 4)).astype(np.float32) * 0.1
    vel[:, 3] = np.arange(n)  # body ids travel in w
    prm = bh.default_params(theta=0.9, eps=0.05, dt=1e-2, leaf_capacity=4)
    with bh.Simulation(n) as sim:
        sim.batch_set(pm, vel, off)
        sim.batch_step(prm, 2)
        bp, bv, _ = sim.get_bodies()
    picked = sorted({0, len(sizes) - 1, int(np.argmax(sizes)), len(sizes) // 2})
    for s in picked:
        sl = slice(int(off[s]), int(off[s + 1]))
        if sizes[s] == 1:
            assert bv[sl, 3][0] == off[s]
            continue
        with bh.Simulation(sizes[s]) as one:
            one.set_bodies(pm[sl], vel[sl])
            one.step(prm, 2)
            p, v, _ = one.get_bodies()
        assert np.array_equal(bv[sl, 3], v[:, 3])  # the same order
        assert np.allclose(bp[sl], p, rtol=0, atol=1e-5)
