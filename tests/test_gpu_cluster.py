"""The one-launch cluster form of the ensemble step (tiling form 13) against the FP64 oracle: cluster
sizes with and without neighbours, ragged chunks and row blocks, both precisions and dots, every noise,
the adaptive dimension, and exponentials that need the dense form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

POP_TOL = {"fp64": 1e-10, "mixed": 1e-6}   # the ensemble tests' bounds
T = 6


def _density():
    om = 20.0 * np.arange(1, 9)
    return om, 40.0 * (om / 60.0) * np.exp(-om / 60.0), 20.0, 150.0


def _pair(oracle, s, precision, B, dot, noise, m=8, dt=1.0, m_min=0, m_tol=0.0):
    import dynaquant_b200 as dq
    p = dq.Propagator(s.n, m=m, n_traj=B, dt=dt, noise=noise, sigma_static=80.0, seed=9, dot=dot,
                      precision=dq.PREC_FP64 if precision == "fp64" else dq.PREC_MIXED, max_steps=T, m_min=m_min,
                      m_tol=m_tol)
    p.set_system(s)
    kw = dict(sigma=150.0, tau=70.0)
    if noise == dq.NOISE_ZZ:
        om, J, dw, temp = _density()
        p.set_zz_spectral_density(om, J, dw, temp)
        w, c = oracle.zz_coefficients(om, J, dw, temp)
        kw = dict(zz_omega=w, zz_coeff=c)
    elif noise != dq.NOISE_NONE:
        p.set_noise_params(np.full(s.n, 150.0), np.full(s.n, 70.0))
    psi0 = s.bright_state()
    p.set_initial_state(psi0)
    rp, col, val, diag = s.off_diagonal()
    S = oracle.System(rp, col, val, diag, m=m, dt=dt, dot_mode=dot, norm_mode=1, noise=noise, sigma_static=80.0,
                      seed=9, m_min=m_min, m_tol=m_tol or 1e-7, **kw)
    return p, S.run(B, T, psi0, threads=4)


def _check(p, ref, precision):
    tol = POP_TOL[precision]
    assert np.abs(p.populations() - ref["pops"]).max() < tol
    assert np.abs(p.correlation() - ref["corr"]).max() < 10 * tol   # |corr| is 1, a population 1/n


# tube 12 x 11: 132 sites, 29 couplings a row in the middle; (trajectories per chunk, CTAs, rows per block)
@pytest.mark.parametrize("precision,B,tc,cs,rows", [
    ("fp64", 5, 1, 1, 1), ("fp64", 5, 2, 3, 2), ("fp64", 5, 4, 5, 4), ("fp64", 5, 8, 16, 1), ("fp64", 40, 32, 2, 2),
    ("mixed", 10, 2, 1, 3), ("mixed", 10, 4, 3, 1), ("mixed", 10, 8, 7, 2), ("mixed", 10, 16, 16, 3),
    ("mixed", 70, 64, 2, 3)])
@pytest.mark.parametrize("dot,noise", [(1, 2), (0, 1), (1, 3), (1, 0)])
def test_cluster_step_matches_oracle(oracle, precision, B, tc, cs, rows, dot, noise):
    from dynaquant_b200 import systems
    s = systems.tube(12, 11)
    p, ref = _pair(oracle, s, precision, B, dot, noise)
    p.set_tiling(tc, 2 if precision == "mixed" else 1, cs, rows, 13, 1)
    p.run(T)
    _check(p, ref, precision)
    p.close()


# a chain too long for its records (mixed) or rows of many couplings read through L1, and n not a multiple of anything
@pytest.mark.parametrize("kind,precision,tc,cs,rows", [("chain", "mixed", 8, 3, 3), ("chain", "fp64", 2, 3, 1),
                                                       ("tube", "mixed", 8, 4, 3), ("tube", "fp64", 4, 6, 2)])
def test_cluster_step_large_rows(oracle, kind, precision, tc, cs, rows):
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    s = systems.chain(3001) if kind == "chain" else systems.tube(37, 61)
    p, ref = _pair(oracle, s, precision, 6, 1, dq.NOISE_OU)
    p.set_tiling(tc, 2 if precision == "mixed" else 1, cs, rows, 13, 1)
    p.run(T)
    _check(p, ref, precision)
    p.close()


@pytest.mark.parametrize("precision,tc,cs", [("fp64", 2, 3), ("mixed", 4, 1), ("mixed", 8, 5)])
def test_cluster_adaptive_dimension(oracle, precision, tc, cs):
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    s = systems.tube(12, 11)
    p, ref = _pair(oracle, s, precision, 6, 1, dq.NOISE_OU, m=20, dt=2.0, m_min=4, m_tol=1e-6)
    p.set_tiling(tc, 2 if precision == "mixed" else 1, cs, 2, 13, 1)
    p.run(T)
    _check(p, ref, precision)
    if precision == "fp64":
        assert np.allclose(p.error_accum(), ref["err"], rtol=1e-3, atol=1e-13)
    p.close()


# steps of norm above 2^4 / 2: the dense exponential in every check and at the end.  The Krylov space is
# far too small for such a step, so the first step alone is asked for (FP64: a projection of norm 150
# loses about three digits of the rounding; complex64 vectors would lose everything)
@pytest.mark.parametrize("tc,cs", [(2, 3), (4, 1)])
def test_cluster_adaptive_dense_exponential(oracle, tc, cs):
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    p, ref = _pair(oracle, systems.tube(12, 11), "fp64", 6, 1, dq.NOISE_OU, m=24, dt=400.0, m_min=4, m_tol=1e-6)
    p.set_tiling(tc, 1, cs, 2, 13, 1)
    p.run(1)
    assert np.abs(p.populations()[1] - ref["pops"][1]).max() < 1e-8
    p.close()


def test_cluster_form_refuses_what_it_cannot_hold():
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    s = systems.chain(30000)
    p = dq.Propagator(s.n, m=8, n_traj=8, precision=dq.PREC_MIXED, max_steps=1)
    p.set_system(s)
    p.set_initial_state(s.bright_state())
    for bad in [(8, 2, 1, 1, 13, 1), (6, 2, 4, 1, 13, 1), (8, 2, 17, 1, 13, 1), (8, 2, 8, 4, 13, 1), (8, 1, 8, 1, 13, 1),
                (8, 2, 8, 1, 13, 2), (8, 2, 8, 1, 14, 1)]:
        with pytest.raises(dq.DQError):
            p.set_tiling(*bad)
    p.set_tiling(4, 2, 16, 1, 13, 1)
    p.run(1)
    p.close()
