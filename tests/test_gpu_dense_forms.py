"""Steps whose exponential needs the dense form (the |Re|-only norm on matrices of complex norm above 1/2,
more than four halvings), in every one-launch form of the step: one CTA, a cluster, the whole grid, the
static call, ensembles with many trajectories to a CTA, the adaptive dimension's checks with what they
bring back, and matrices too large for what shared memory is left."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# FP64, one step: as the tridiagonal exponential's test, up to 2^6 squarings of an (m+2)-row product and
# the recurrence's rounding
PSI_TOL = 1e-11
POP_TOL = {"fp64": 1e-10, "mixed": 1e-6}   # the ensemble tests' bounds
ERR_TOL = dict(rel=1e-3, abs=1e-13)

# (norm, dt) for systems of ||H|| / hbar about 0.2 per fs: an unscaled quotient of norm 1.6, five or six halvings
BIG = [(0, 8.0), (1, 90.0)]


def _system(shape):
    from dynaquant_b200 import systems
    return systems.chain(*shape) if len(shape) == 1 else systems.tube(*shape)


def _needs_dense(S1, d, psi, norm):
    """The series does not cover this step, by the halvings that the oracle takes with the complex norm."""
    return S1.krylov_step(d, psi)[3] > (4 if norm == 1 else 0)


@pytest.mark.parametrize("shape,ctas", [((33,), (1, 1)), ((1025,), (2, 16)), ((23, 30), (2, 16)), ((60, 150), (17, 148))])
@pytest.mark.parametrize("norm,dt", BIG)
def test_drop_in_step(oracle, shape, ctas, norm, dt):
    import torch
    import dynaquant_b200 as dq
    s = _system(shape)
    m = 12
    rp, col, val, diag = s.off_diagonal()
    S = oracle.System(rp, col, val, diag, m=m, dt=dt, dot_mode=1, norm_mode=norm, noise=2, sigma=150.0, tau=70.0,
                      sigma_static=80.0, seed=21)
    S1 = oracle.System(rp, col, val, diag, m=m, dt=dt, dot_mode=1, norm_mode=1)
    p = dq.Propagator(s.n, m=m, n_traj=2, dt=dt, noise=dq.NOISE_OU, sigma_static=80.0, seed=21, dot=1, norm=norm,
                      precision=dq.PREC_FP64, max_steps=4)
    p.set_system(s)
    p.set_noise_params(np.full(s.n, 150.0), np.full(s.n, 70.0))
    g = np.random.default_rng(s.n)
    psi = g.normal(size=s.n) + 1j * g.normal(size=s.n)
    psi /= np.linalg.norm(psi)
    p.set_initial_state(psi)
    p.reset()
    assert ctas[0] <= p.debug_step_shape()[0] <= ctas[1]
    a = torch.from_numpy(psi).cuda()
    b = torch.empty_like(a)
    torch.cuda.synchronize()
    eps, deps = S.traj_init(1)
    for k in range(3):
        err = p.prop_step(1, k, a.data_ptr(), b.data_ptr(), want_error=True)
        d = S.noise_update(1, k, eps, deps)
        assert _needs_dense(S1, d, psi, norm)
        psi, err_o, _, _ = S.krylov_step(d, psi)
        assert np.abs(b.cpu().numpy() - psi).max() < PSI_TOL, k
        assert err == pytest.approx(err_o, **ERR_TOL)
        a, b = b, a
        psi = a.cpu().numpy()
    p.close()


@pytest.mark.parametrize("shape", [(40,), (23, 30), (58, 91)])
@pytest.mark.parametrize("norm,dt", BIG)
def test_static_step(oracle, shape, norm, dt):
    import torch
    from dynaquant_b200 import _lib
    s = _system(shape)
    m = 14
    rp, col, val, _ = s.off_diagonal()
    g = np.random.default_rng(s.n)
    diag = g.normal(0.0, 150.0, s.n)
    psi = g.normal(size=s.n) + 1j * g.normal(size=s.n)
    psi /= np.linalg.norm(psi)
    S = oracle.System(rp, col, val, np.zeros(s.n), m=m, dt=dt, dot_mode=1, norm_mode=norm)
    S1 = oracle.System(rp, col, val, np.zeros(s.n), m=m, dt=dt, dot_mode=1, norm_mode=1)
    assert _needs_dense(S1, diag, psi, norm)
    ref, err_o, _, _ = S.krylov_step(diag, psi)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (rp, col, val, diag, psi)]
    out = torch.zeros_like(d[4])
    torch.cuda.synchronize()
    err, msg = C.c_double(), C.create_string_buffer(200)
    rc = _lib.load().dq_krylov_step_static(s.n, *[x.data_ptr() for x in d], out.data_ptr(), m, dt, 0.0, 1, norm, None,
                                           C.byref(err), msg, len(msg))
    assert rc == 0, msg.value
    assert np.abs(out.cpu().numpy() - ref).max() < PSI_TOL
    assert err.value == pytest.approx(err_o, **ERR_TOL)


def _ensemble(oracle, s, precision, B, T, m, dt, norm, m_min=0, tiling=None):
    import dynaquant_b200 as dq
    kw = dict(m_min=m_min, m_tol=1e-6) if m_min else {}
    p = dq.Propagator(s.n, m=m, n_traj=B, dt=dt, noise=dq.NOISE_OU, sigma_static=80.0, seed=9, dot=1, norm=norm,
                      precision=dq.PREC_FP64 if precision == "fp64" else dq.PREC_MIXED, max_steps=T, **kw)
    p.set_system(s)
    p.set_noise_params(np.full(s.n, 150.0), np.full(s.n, 70.0))
    psi0 = s.bright_state()
    p.set_initial_state(psi0)
    if tiling:
        p.set_tiling(*tiling)
    p.run(T)
    rp, col, val, diag = s.off_diagonal()
    S = oracle.System(rp, col, val, diag, m=m, dt=dt, dot_mode=1, norm_mode=norm, noise=2, sigma=150.0, tau=70.0,
                      sigma_static=80.0, seed=9, **kw)
    ref = S.run(B, T, psi0, threads=4)
    tol = POP_TOL[precision]
    assert np.abs(p.populations() - ref["pops"]).max() < tol
    assert np.abs(p.correlation() - ref["corr"]).max() < 10 * tol   # |corr| is 1, a population 1/n
    if precision == "fp64":
        assert np.allclose(p.error_accum(), ref["err"], rtol=1e-3, atol=1e-13)
    p.close()


# one to eight trajectories side by side in a CTA, several rounds of them, ragged chunks
@pytest.mark.parametrize("precision,B,tiling", [
    ("fp64", 5, (1, 1, 1, 1, 13, 1)), ("fp64", 7, (4, 1, 5, 2, 13, 1)), ("fp64", 40, (32, 1, 1, 2, 13, 1)),
    ("fp64", 12, (8, 1, 2, 4, 13, 1)), ("mixed", 10, (8, 2, 3, 3, 13, 1)), ("mixed", 70, (64, 2, 2, 3, 13, 1)),
    ("mixed", 36, (16, 2, 1, 2, 13, 1)), ("fp64", 6, (2, 1, 2, 2, 0, 1)), ("mixed", 8, (8, 2, 2, 3, 0, 1))])
@pytest.mark.parametrize("m", [8, 20])
def test_ensemble_step(oracle, precision, B, tiling, m):
    _ensemble(oracle, _system((12, 11)), precision, B, 4, m, 6.0, 0, tiling=tiling)


def test_ensemble_matrices_beyond_shared_memory(oracle):
    """64 trajectories' scalars at m = 32 leave less than one set of matrices."""
    _ensemble(oracle, _system((40,)), "mixed", 70, 3, 32, 6.0, 0, tiling=(64, 2, 1, 1, 13, 1))


# the checks' choices, and the iterations after a check: records in shared memory or read through L1
@pytest.mark.parametrize("shape,precision,B,tiling", [
    ((12, 11), "fp64", 6, (2, 1, 3, 2, 13, 1)), ((12, 11), "fp64", 5, (4, 1, 1, 1, 13, 1)),
    ((12, 11), "fp64", 40, (32, 1, 2, 2, 13, 1)), ((12, 11), "mixed", 10, (8, 2, 5, 3, 13, 1)),
    ((12, 11), "mixed", 36, (32, 2, 1, 2, 13, 1)), ((37, 61), "mixed", 6, (8, 2, 4, 3, 13, 1)),
    ((37, 61), "fp64", 6, (4, 1, 6, 2, 13, 1)), ((12, 11), "mixed", 8, (8, 2, 2, 3, 0, 1))])
def test_adaptive_checks(oracle, shape, precision, B, tiling):
    _ensemble(oracle, _system(shape), precision, B, 3, 28, 6.0, 0, m_min=4, tiling=tiling)
