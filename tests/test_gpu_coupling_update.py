"""Couplings changed on a context that already has its ensemble workspace: the blocks built on the
device hold the new values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _context(s, tiling):
    import dynaquant_b200 as dq
    p = dq.Propagator(s.n, m=10, n_traj=16, dt=1.0, noise=dq.NOISE_OU, sigma_static=50.0, seed=4,
                      precision=dq.PREC_MIXED, max_steps=6)
    p.set_system(s)
    p.set_noise_params(np.full(s.n, 100.0), np.full(s.n, 80.0))
    p.set_initial_state(s.bright_state((1.0, 0.0, 0.0)))
    if tiling:
        p.set_tiling(*tiling)
    return p


@pytest.mark.parametrize("tiling", [None, (8, 2, 1, 3, 12, 1), (16, 2, 2, 2, 0, 1)])
def test_changed_couplings_reach_the_ensemble(tiling):
    from dynaquant_b200 import systems
    small, large = systems.lattice2d(12), systems.lattice2d(12, J_nn=-180.0, J_nnn=70.0)
    p = _context(small, tiling)
    p.run(2)
    # other scales, then another matrix of the same pattern, against contexts made with them
    for change in ("scales", "matrix"):
        q = _context(small if change == "scales" else large, tiling)
        for x in (p, q):
            if change == "scales":
                x.set_coupling_classes(small.cls_off, [1.4, 0.3])
            elif x is p:
                x.set_system(large)
            x.reset()
            x.run(6)
        assert np.array_equal(p.populations(), q.populations()), change
        assert np.array_equal(p.correlation(), q.correlation()), change
        q.close()
    p.close()
