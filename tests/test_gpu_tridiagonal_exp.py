"""The exponential of the Lanczos tridiagonal (a Taylor series on one warp, the dense Padé form where
the series does not apply) through one step against the FP64 oracle's Padé, over the halvings it takes,
both scaling norms and the smallest and largest Krylov dimensions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one step, every operation FP64: s <= 6 squarings of an (m+2)-row product each lose a few ulp,
# 2^6 * 34 * 2.2e-16 = 5e-13; the recurrence's own rounding is below that
PSI_TOL = 1e-11
N, B = 64, 5


def _system(oracle, m, dt, norm, dot):
    from dynaquant_b200 import systems
    s = systems.chain(N, -300.0)
    rp, col, val, diag = s.off_diagonal()
    S = oracle.System(rp, col, val, diag, m=m, dt=dt, dot_mode=dot, norm_mode=norm, noise=oracle.NOISE_GAUSS,
                      sigma=200.0, tau=100.0, sigma_static=100.0, seed=5)
    return s, S


# halvings by dt with the complex norm: 0, 1, 2, 4 (the series) and 6 (dense)
@pytest.mark.parametrize("m,dt", [(2, 0.5), (3, 2.0), (17, 4.0), (20, 8.0), (31, 30.0), (32, 130.0), (12, 130.0)])
@pytest.mark.parametrize("norm,dot", [(0, 0), (1, 0), (1, 1)])
def test_step_matches_oracle_over_scalings(oracle, m, dt, norm, dot):
    import dynaquant_b200 as dq
    s, S = _system(oracle, m, dt, norm, dot)
    p = dq.Propagator(N, m=m, n_traj=B, dt=dt, noise=dq.NOISE_GAUSS, sigma_static=100.0, seed=5, dot=dot, norm=norm,
                      precision=dq.PREC_FP64, max_steps=1)
    p.set_system(s)
    p.set_noise_params(np.full(N, 200.0))
    g = np.random.default_rng(m)
    # the unconjugated dot of a complex state is no norm: it takes a real one, as runs start from
    psi0 = g.normal(size=N) + (1j * g.normal(size=N) if dot == 1 else 0j)
    psi0 /= np.linalg.norm(psi0)
    p.set_initial_state(psi0)
    p.run(1)
    got, err = p.states(), p.error_accum()
    for b in range(B):
        eps, deps = S.traj_init(b)
        d = S.noise_update(b, 0, eps, deps)
        psi, err_o, _, _ = S.krylov_step(d, psi0)
        assert np.abs(got[b] - psi).max() < PSI_TOL
        # the estimate's rows are below the rounding of a dense quotient where they are tiny
        assert err[b] == pytest.approx(err_o, rel=1e-3, abs=1e-13)
    p.close()
