"""Node edges whose squares leave the float range only near the root: the opening test of the nodes below
stays the one of the same system at another scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("multipole", [0, 1])
@pytest.mark.parametrize("n", [3000, 70001])
def test_opening_at_large_edges(bh, n, multipole):
    # a sphere in a small part of the box, so that its nodes lie deep, and two far bodies; edge 2^66 (its
    # square is beyond float's 2^128) and the same bodies scaled by 2^-40, a change of exponents only
    pm, vel = bh.plummer(11, n)
    x = pm[:, :3] * np.float32(2.0**50) + np.float32(2.0**60)
    x[-1], x[-2] = 2.0**64, -(2.0**64)
    counts = []
    for scale in (2.0**-40, 1.0):
        p = pm.copy()
        p[:, :3] = x * np.float32(scale)
        with bh.Simulation(n) as sim:
            sim.set_bodies(p, np.zeros_like(p))
            sim.build(np.zeros(3), 2.0**66 * scale, 8, multipole)
            _, st = sim.force(0.6, 0.0, stats=True)
            counts.append((st.interactions_cell, st.interactions_p2p))
    # the two far bodies, whose squared distances overflow, may open otherwise: up to n entries each
    for small, large in zip(*counts):
        assert abs(int(large) - int(small)) <= 4 * n
    assert sum(counts[1]) < 0.5 * n * n  # and not every pair
