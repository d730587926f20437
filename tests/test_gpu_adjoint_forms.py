"""The adjoint gradient over the tilings that lay the kept Krylov basis out differently: the cluster form
with chunks that do not divide the trajectories, and a tiling that changes between the forward and the
backward pass (kept segments of one layout, recomputed ones of the other)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTER = {0: (16, 1, 3, 2, 13, 1), 1: (16, 2, 3, 3, 13, 1)}   # 24 trajectories: a chunk of 16, one of 8
GRID = {0: (8, 1, 2, 2, 0, 1), 1: (8, 2, 2, 3, 0, 1)}
TOL = {0: 1e-9, 1: 3e-4}   # FP64: rounding through 14 steps; mixed: the adjoint tests' bound


def _gradient(precision, forward, backward, every):
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    s = systems.lattice2d(9)
    T, LEN = 14, 64
    p = dq.Propagator(s.n, m=10, n_traj=24, dt=1.0, noise=dq.NOISE_OU, seed=3, precision=precision, max_steps=T)
    p.set_system(s)
    p.set_noise_params(np.full(s.n, 120.0), np.full(s.n, 60.0))
    p.set_coupling_classes(s.cls_off, [1.0, 0.9])
    p.set_static_energies(np.random.default_rng(4).normal(0.0, 80.0, s.n))
    p.set_initial_state(s.bright_state((1.0, 0.0, 0.0)))
    if forward:
        p.set_tiling(*forward)
    p.adjoint_setup(T, LEN, 1.0 / T, np.random.default_rng(6).normal(0.0, 0.05, LEN), checkpoint_every=every)
    loss = p.forward()
    if backward:
        p.set_tiling(*backward)
    gs, gc = p.backward()
    p.close()
    return loss, gs, gc


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("every", [0, 4])
@pytest.mark.parametrize("forward,backward", [("C", None), ("C", "G"), ("G", "C"), ("C", "C2")])
def test_gradient_over_basis_layouts(precision, every, forward, backward):
    pick = {"C": CLUSTER[precision], "G": GRID[precision], "C2": (8,) + CLUSTER[precision][1:], None: None}
    loss, gs, gc = _gradient(precision, pick[forward], pick[backward], every)
    loss0, gs0, gc0 = _gradient(0, GRID[0], None, 0)
    tol = TOL[precision]
    assert loss == pytest.approx(loss0, rel=tol)
    assert np.abs(gs - gs0).max() < tol * np.abs(gs0).max()
    assert np.abs(gc - gc0).max() < tol * np.abs(gc0).max()
