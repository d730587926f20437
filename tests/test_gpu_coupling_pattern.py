"""Another matrix of more, or fewer, couplings on a context that already has its ensemble workspace: the
blocks built on the device follow it, in every kind of form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _context(s, precision, tiling):
    import dynaquant_b200 as dq
    p = dq.Propagator(s.n, m=10, n_traj=16, dt=1.0, noise=dq.NOISE_OU, sigma_static=50.0, seed=4, precision=precision,
                      max_steps=6)
    p.set_system(s)
    p.set_noise_params(np.full(s.n, 100.0), np.full(s.n, 80.0))
    psi0 = np.exp(0.3j * np.arange(s.n)) / np.sqrt(s.n)
    p.set_initial_state(psi0)
    p.set_tiling(*tiling)
    return p


@pytest.mark.parametrize("precision,tiling", [
    (1, (8, 2, 2, 3, 13, 1)), (0, (4, 1, 3, 2, 13, 1)), (1, (8, 2, 1, 3, 12, 1)), (1, (16, 2, 2, 2, 0, 1)),
    (0, (16, 1, 1, 2, 5, 1))])
@pytest.mark.parametrize("first,then", [("few", "many"), ("many", "few")])
def test_matrix_of_another_pattern(precision, tiling, first, then):
    from dynaquant_b200 import systems
    # 144 sites: 8 couplings a row within 13 sites, and 29 a row within 36
    s = {"few": systems.lattice2d(12), "many": systems.tube(12, 12)}
    p = _context(s[first], precision, tiling)
    p.run(2)
    p.set_system(s[then])
    p.reset()
    p.run(6)
    q = _context(s[then], precision, tiling)
    q.run(6)
    assert p.get_tiling() == q.get_tiling()
    assert np.array_equal(p.populations(), q.populations())
    assert np.array_equal(p.correlation(), q.correlation())
    p.close()
    q.close()
