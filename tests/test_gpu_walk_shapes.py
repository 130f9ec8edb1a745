"""Launch shapes of the walk for ensembles and small systems: a pinned shape is the one that runs, the
autotuner reports the shapes that it timed, and what it picks for an ensemble stays with ensembles."""
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


@pytest.mark.parametrize("sizes,group", list(zip(SIZES, (4, 8, 16))))
def test_ensemble_rows_are_what_ran(bh, sizes, group):
    pm, vel, off = ensemble(bh, sizes)
    prm = bh.default_params(theta=0.6, eps=0.01, dt=1e-3, leaf_capacity=4)
    with bh.Simulation(len(pm)) as sim:
        sim.batch_set(pm, vel, off)
        sim.batch_step(prm, 1)
        r = sim.autotune(0.6, 0.01, trials=2)
    v = r["variants"]
    assert [x["group_size"] for x in v] == [group] + [32] * 7 + [group] * 4
    assert all(x == v[0] for x in v[8:])  # the same kernel, timed once
    assert r["best"] < 8 and v[r["best"]]["ms"] == min(x["ms"] for x in v) > 0


@pytest.mark.parametrize("pin", [None, 3])
def test_ensemble_choice_stays_with_ensembles(bh, pin):
    pm, vel, off = ensemble(bh, SIZES[0])
    prm = bh.default_params(theta=0.6, eps=0.01, dt=1e-3, leaf_capacity=4)
    one, onev = bh.plummer(5, 2000)
    evals = []
    for tune in (False, True):
        with bh.Simulation(len(pm)) as sim:
            if pin is not None:
                sim.set_walk_variant(pin)
            if tune:
                sim.batch_set(pm, vel, off)
                sim.batch_step(prm, 1)
                sim.autotune(0.6, 0.01, trials=1)
            sim.set_bodies(one, onev)
            st = sim.step(prm, 1)
            evals.append((st.walk_cell_evals, st.walk_point_evals))
    assert evals[0] == evals[1]


@pytest.mark.parametrize("n,shape", [
    (2000, (2, 4)), (12287, (2, 4)), (12288, (2, 8)), (24575, (2, 8)), (49152, (2, 16)), (49153, (3, 16)),
    (196607, (3, 16)), (196608, (4, 32)),
])
def test_default_row_names_its_kernel(bh, n, shape):
    """Row 0 against the rows of the pinned shapes with the same registers: 10 and 11 (two blocks per SM),
    1 (three), 2 (two)."""
    pm, vel = bh.plummer(2, n)
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, vel)
        c, size = sim.bounds()
        sim.build(c, 2 * size, 16, 1)
        v = sim.autotune(1.0, 0.01, trials=1)["variants"]
    assert (v[0]["min_blocks_per_sm"], v[0]["group_size"]) == shape
    # registers a thread within the budget of that many blocks of 256 on the SM's 65 536
    assert 65536 // 256 // (shape[0] + 1) // 8 * 8 < v[0]["registers"] <= 65536 // 256 // shape[0]


def test_shapes_of_one_group_size_take_alike(bh):
    """Groups of 32 on a system with fewer of them than the GPU has warps: every shape spreads them over the
    SMs. The shapes differ in registers, block size and stack; their walks differ by 3%."""
    n = 65536
    pm, vel = bh.plummer(0, n)
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, vel)
        sim.step(bh.default_params(theta=0.5, eps=0.01, dt=1e-3, leaf_capacity=8), 2)
        ms = [v["ms"] for v in sim.autotune(0.5, 0.01, trials=15)["variants"][1:8]]
    assert max(ms) < 1.2 * min(ms)
