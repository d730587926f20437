"""The drop-in step of large systems (one cooperative launch): its grid barrier's bounded wait."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DQ_ERR_TIMEOUT = 5
PSI_TOL = 1e-11   # as for the drop-in step elsewhere


def test_grid_barrier_timeout_is_reported_and_context_recovers(oracle):
    """A count that never comes within 20,000 cycles: every CTA gives up and leaves, the step returns
    DQ_ERR_TIMEOUT, and with the default budget the same context's next steps match the oracle (the
    barrier's counts are clear again)."""
    import torch
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    s = systems.tube(60, 150)
    rp, col, val, diag = s.off_diagonal()
    S = oracle.System(rp, col, val, diag, m=9, dt=0.7, dot_mode=1, norm_mode=1)
    p = dq.Propagator(s.n, m=9, dt=0.7, dot=1, norm=1, precision=dq.PREC_FP64, max_steps=2)
    p.set_system(s)
    psi = s.bright_state()
    p.set_initial_state(psi)
    p.reset()
    assert p.debug_step_shape()[0] > 16   # CTAs: the whole-grid form
    a = torch.from_numpy(psi).cuda()
    b = torch.empty_like(a)
    torch.cuda.synchronize()
    try:
        p.debug_set_wait_cycles(-20000)
        for _ in range(2):
            with pytest.raises(dq.DQError) as e:
                p.prop_step(0, 0, a.data_ptr(), b.data_ptr(), want_error=True)
            assert e.value.code == DQ_ERR_TIMEOUT
        with pytest.raises(dq.DQError) as e:
            p.run_plain(1)
        assert e.value.code == DQ_ERR_TIMEOUT
    finally:
        p.debug_set_wait_cycles(0)
    p.reset()
    ref = psi
    for k in range(3):
        err = p.prop_step(0, k, a.data_ptr(), b.data_ptr(), want_error=True)
        ref, err_o, _, _ = S.krylov_step(S.h0diag, ref)
        assert np.abs(b.cpu().numpy() - ref).max() < PSI_TOL
        assert err == pytest.approx(err_o, rel=1e-3, abs=1e-14)
        a, b = b, a
    p.close()
