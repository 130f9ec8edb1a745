"""The backward pass walks the forward pass's own trajectory: a step recomputed from a checkpoint repeats the
forward step bit for bit, so the gradient does not depend on how many steps a checkpoint is followed by."""
import numpy as np
import pytest

from oracle.oracle import relerr

pytestmark = pytest.mark.gpu


def bodies(bh, n, dt, pairs):
    """A sphere; or n / 2 pairs some 1e-5 apart, one body of each overtaking the other in the first step, whose
    tree has both in one cell of the deepest level."""
    if not pairs:
        return bh.plummer(3, n)
    pm, vel = bh.plummer(3, n // 2)
    d = np.random.default_rng(3).uniform(1e-5, 3e-5, (n // 2, 3)).astype(np.float32)
    pm2, vel2 = pm.copy(), vel.copy()
    pm2[:, :3] -= d
    vel2[:, :3] += d / np.float32(dt)
    pm[:, 3] *= 0.7
    pm2[:, 3] *= 0.3
    return np.concatenate([pm, pm2]), np.concatenate([vel, vel2])


@pytest.mark.parametrize("pairs", [False, True])
def test_gradient_does_not_depend_on_the_checkpoints(bh, pairs):
    # Up to 16 bodies under a root that is a leaf are one group and one buffer of the walk, so nothing is
    # summed in an order of chance and gradients of the same path are the same bits. With a checkpoint at
    # every step the path is the forward pass's; with fewer it is so only if each recomputed step is.
    n, nsteps, dt = 16, 50, 0.01
    pm, vel = bodies(bh, n, dt, pairs)
    pm[:, 3] *= 100.0  # half-kicks of the size of the velocities, whose last bits then show the forces'
    prm = bh.default_params(theta=0.5, eps=0.3, dt=dt, leaf_capacity=16, multipole=1, edge_factor=1.0)
    dl = np.random.default_rng(9).normal(size=(n, 3)).astype(np.float32)
    out = []
    for every in (1, 1, 7, nsteps):
        with bh.Simulation(n) as sim:
            sim.set_bodies(pm, vel)
            sim.adjoint_forward(prm, nsteps, every)
            out.append((*sim.get_bodies(), *sim.step_backward(dl, None)))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.parametrize("n", [200, 24577, 65537, 163841])
def test_forward_step_has_the_force_of_a_fresh_tree(bh, n):
    """a(x_1) of a forward step (whose tree keys sort in the previous tree's order) against a tree built
    from the same positions, within the bars of the walk's other tests."""
    pm, vel = bh.plummer(n, n)
    prm = bh.default_params(theta=0.6, eps=0.02, dt=1e-2, leaf_capacity=8, multipole=1, edge_factor=2.0)
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, vel)
        sim.adjoint_forward(prm, 1, 1)
        p, v, a = sim.get_bodies()
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, vel)
        c, size = sim.bounds()  # a step's tree stands in the box of the positions before its drift
        sim.set_bodies(p, v)
        sim.build(c, 2 * size, 8, 1)
        want = sim.force(0.6, 0.02)
    err = relerr(a, want)
    assert float(np.median(err)) <= 1e-5 and float(np.percentile(err, 99)) <= 1e-4
