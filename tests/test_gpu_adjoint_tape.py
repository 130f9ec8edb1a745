"""The tape of the differentiable path grows while a step is recorded, and the redone step starts from the
same accelerations: a first backward pass whose tape fills gives the gradients of a second one, whose
tape is large enough from the start."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every", [1, 3])
def test_tape_overflow_on_a_step(bh, every):
    # 64 tight clusters of 64 bodies, few interactions; one step of large velocities later the bodies fill
    # the box, and at theta 0.02 nearly all pairs are direct: 128 chunks a group, where the tape holds 64
    k, per, dt, nsteps = 4, 64, 0.25, 3
    n = k**3 * per
    rng = np.random.default_rng(5)
    centres = np.stack(np.meshgrid(*[np.arange(k) + 0.5] * 3, indexing="ij"), -1).reshape(-1, 3)
    pm = np.zeros((n, 4), np.float32)
    pm[:, :3] = np.repeat(centres, per, 0) + rng.uniform(-1e-3, 1e-3, (n, 3))
    pm[:, 3] = 4.0 / n
    vel = np.zeros_like(pm)
    vel[:, :3] = (rng.uniform(0, k, (n, 3)) - pm[:, :3]) / dt
    dl = rng.normal(size=(n, 3)).astype(np.float32)
    prm = bh.default_params(theta=0.02, eps=0.05, dt=dt, leaf_capacity=8, multipole=1, edge_factor=1.0)
    with bh.Simulation(n) as sim:
        sim.set_bodies(pm, vel)
        sim.adjoint_forward(prm, nsteps, every)
        p1, v1, a1 = sim.get_bodies()
        *first, st1 = sim.step_backward(dl, None, stats=True)
        p2, v2, a2 = sim.get_bodies()
        assert np.array_equal(p1, p2) and np.array_equal(v1, v2) and np.array_equal(a1, a2)
        *second, st2 = sim.step_backward(dl, None, stats=True)
    assert st1.kernel_launches > st2.kernel_launches  # the tape did fill, and only the first time
    for a, b in zip(first, second):  # the bar of repeated backward passes: the reductions' order
        assert np.linalg.norm(a - b) < 1e-5 * np.linalg.norm(b)
