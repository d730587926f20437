"""The drop-in step as one cluster launch: system sizes around its shapes (one CTA, several, the largest,
past it), rows of very different lengths, both conventions, and the pointers it leaves to the other form."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PSI_TOL = 1e-11   # as for the step of several launches


def _oracle_step(oracle, s, m, dt, dot, norm, noise, traj, steps, psi):
    rp, col, val, diag = s.off_diagonal()
    S = oracle.System(rp, col, val, diag, m=m, dt=dt, dot_mode=dot, norm_mode=norm, noise=noise, sigma=150.0, tau=70.0,
                      sigma_static=80.0, seed=21)
    eps, deps = S.traj_init(traj)
    for k in range(steps):
        psi, err, _, _ = S.krylov_step(S.noise_update(traj, k, eps, deps), psi)
    return psi, err


@pytest.mark.parametrize("shape", [(2,), (33,), (511,), (512,), (513,), (1024,), (1025,), (4000,), (8191,), (20000,),
                                   (10, 7), (23, 30), (58, 91), (60, 150), (60, 500)])
@pytest.mark.parametrize("dot,norm", [(0, 0), (1, 1)])
def test_step_sizes_match_oracle(oracle, shape, dot, norm):
    import torch
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    s = systems.chain(*shape) if len(shape) == 1 else systems.tube(*shape)
    m = min(12, s.n)
    p = dq.Propagator(s.n, m=m, n_traj=3, dt=0.7, noise=dq.NOISE_OU, sigma_static=80.0, seed=21, dot=dot, norm=norm,
                      precision=dq.PREC_FP64, max_steps=2)
    p.set_system(s)
    p.set_noise_params(np.full(s.n, 150.0), np.full(s.n, 70.0))
    g = np.random.default_rng(s.n)
    psi = (g.normal(size=s.n) + (1j * g.normal(size=s.n) if dot == 1 else 0j)).astype(np.complex128)
    psi /= np.linalg.norm(psi)
    p.set_initial_state(psi)
    p.reset()
    # one complex value of slack: the second pass starts 8 bytes into it
    buf = torch.zeros(2 * s.n + 4, dtype=torch.float64, device="cuda")
    out = torch.empty(s.n, dtype=torch.complex128, device="cuda")
    for shift in (0, 1):
        buf[shift:shift + 2 * s.n] = torch.from_numpy(psi.view(np.float64)).cuda()
        torch.cuda.synchronize()
        err = p.prop_step(1 + shift, 0, buf.data_ptr() + 8 * shift, out.data_ptr(), want_error=True)
        ref, err_o = _oracle_step(oracle, s, m, 0.7, dot, norm, 2, 1 + shift, 1, psi)
        assert np.abs(out.cpu().numpy() - ref).max() < PSI_TOL, shift
        assert err == pytest.approx(err_o, rel=1e-3, abs=1e-14)
    p.close()


@pytest.mark.parametrize("shape", [(58, 91), (60, 150)])
def test_consecutive_steps_match_oracle(oracle, shape):
    """Steps issued one after another without a synchronisation (cluster and whole-grid form)."""
    import torch
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    s = systems.tube(*shape)
    p = dq.Propagator(s.n, m=9, n_traj=2, dt=0.7, noise=dq.NOISE_OU, sigma_static=80.0, seed=21, dot=1, norm=1,
                      precision=dq.PREC_FP64, max_steps=2)
    p.set_system(s)
    p.set_noise_params(np.full(s.n, 150.0), np.full(s.n, 70.0))
    psi = s.bright_state()
    p.set_initial_state(psi)
    p.reset()
    a = torch.from_numpy(psi).cuda()
    b = torch.empty_like(a)
    torch.cuda.synchronize()
    for k in range(5):
        p.prop_step(1, k, a.data_ptr(), b.data_ptr())
        a, b = b, a
    err = p.prop_step(1, 5, a.data_ptr(), b.data_ptr(), want_error=True)
    ref, err_o = _oracle_step(oracle, s, 9, 0.7, 1, 1, 2, 1, 6, psi)
    assert np.abs(b.cpu().numpy() - ref).max() < PSI_TOL
    assert err == pytest.approx(err_o, rel=1e-3, abs=1e-14)
    p.close()


# rows from empty to long: the static call knows neither the columns nor the rows' lengths beforehand
@pytest.mark.parametrize("n,long_row", [(40, 5), (700, 90), (3000, 20), (5278, 60), (9000, 40), (9000, 400), (20000, 6)])
def test_static_step_uneven_rows_match_oracle(oracle, n, long_row):
    import torch
    from dynaquant_b200 import _lib
    g = np.random.default_rng(n + long_row)
    # symmetric couplings between random pairs, a few rows taking many of them
    deg = np.where(g.random(n) < 0.03, long_row, g.integers(0, 4, n))
    i = np.repeat(np.arange(n), deg)
    j = g.integers(0, n, len(i))
    ok = i != j
    i, j = i[ok], j[ok]
    v = g.normal(0.0, 60.0, len(i))
    rows, cols, vals = np.concatenate([i, j]), np.concatenate([j, i]), np.concatenate([v, v])
    o = np.argsort(rows, kind="stable")
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=n), out=rp[1:])
    col, val = cols[o].astype(np.int32), vals[o]
    diag = g.normal(0.0, 200.0, n)
    psi = g.normal(size=n) + 1j * g.normal(size=n)
    psi /= np.linalg.norm(psi)
    m = 10
    ref, err_o, _, _ = oracle.System(rp, col, val, np.zeros(n), m=m, dt=0.5, dot_mode=1, norm_mode=1).krylov_step(diag, psi)
    d = {k: torch.from_numpy(np.ascontiguousarray(x)).cuda() for k, x in
         dict(rp=rp, col=col, val=val, diag=diag, psi=psi).items()}
    out = torch.zeros_like(d["psi"])
    torch.cuda.synchronize()
    err, msg = C.c_double(), C.create_string_buffer(200)
    rc = _lib.load().dq_krylov_step_static(
        n, d["rp"].data_ptr(), d["col"].data_ptr(), d["val"].data_ptr(), d["diag"].data_ptr(), d["psi"].data_ptr(),
        out.data_ptr(), m, 0.5, 0.0, 1, 1, None, C.byref(err), msg, len(msg))
    assert rc == 0, msg.value
    assert np.abs(out.cpu().numpy() - ref).max() < PSI_TOL
    assert err.value == pytest.approx(err_o, rel=1e-3, abs=1e-14)
