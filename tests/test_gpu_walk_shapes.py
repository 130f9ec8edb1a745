"""Launch shapes of the walk: a pinned shape is the one that runs, for ensembles and small systems too."""
import numpy as np
import pytest

from oracle.oracle import relerr

pytestmark = pytest.mark.gpu


def ensemble(bh, sizes):
    parts = [bh.plummer(31 + s, k) for s, k in enumerate(sizes)]
    pm, vel = (np.concatenate(x) for x in zip(*parts))
    return pm, vel, np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)


# groups of 4, 8 and 16 by the number of bodies in all
SIZES = [[900, 33, 1, 1500], [9000, 4000, 700], [20000, 30000, 41]]


@pytest.mark.parametrize("sizes", SIZES)
def test_pinned_shape_runs_on_small_ensembles(bh, sizes):
    pm, vel, off = ensemble(bh, sizes)
    prm = bh.default_params(theta=0.6, eps=0.01, dt=1e-3, leaf_capacity=4)
    evals, acc = [], []
    for variant in (0, 1, 6, 9):
        with bh.Simulation(len(pm)) as sim:
            sim.batch_set(pm, vel, off)
            sim.set_walk_variant(variant)
            st = sim.batch_step(prm, 1)
            evals.append((st.walk_cell_evals, st.walk_point_evals))
            acc.append((sim.get_bodies()[2], st.interactions_cell, st.interactions_p2p))
    assert evals[1] != evals[0]  # groups of 32, whose warps evaluate other entries
    assert evals[2] == evals[1]  # so does shape 6
    assert evals[3] == evals[0]  # shapes 8 and up differ for single systems only
    for a, cells, points in acc[1:]:  # the reference's interaction sets all the same
        assert cells == acc[0][1] and points == acc[0][2]
        assert float(np.median(relerr(a, acc[0][0]))) < 1e-5
