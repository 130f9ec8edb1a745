"""An empty state has a tree without nodes: build, its queries, forces and diagnostics take it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("multipole", [0, 1])
@pytest.mark.parametrize("leaf", [1, 8, 100])
def test_tree_of_no_bodies(bh, leaf, multipole):
    none = np.zeros((0, 4), np.float32)
    pm, vel = bh.plummer(3, 16)
    with bh.Simulation(16) as sim:
        sim.set_bodies(none, none)
        sim.build(np.zeros(3), 2.0, leaf, multipole)
        assert sim.tree_size() == 0
        assert all(len(v) == 0 for v in sim.tree_nodes().values())
        assert all(len(v) == 0 for v in sim.tree_boxes())
        acc, st = sim.force(0.5, 0.01, stats=True)
        assert acc.shape == (0, 4) and st.interactions_p2p == 0 and st.error_flags == 0
        e = sim.energy(0.5, 0.01)
        assert e["mass"] == 0 and e["total"] == 0
        # the context goes on as before
        sim.set_bodies(pm, vel)
        c, size = sim.bounds()
        sim.build(c, 2 * size, leaf, multipole)
        assert sim.tree_size() >= 1 and np.isfinite(sim.force(0.5, 0.01)).all()
