"""Taylor-Krylov ensembles at the sizes where the step's form changes: records in shared memory, records
read through L1 (with and without their row starts in shared memory), and systems of several launches,
each against the per-trajectory path on the same draws."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10   # both FP64; the Taylor-Krylov tests' bound


def _run(s, how, B, steps, p_tk, m_b, dt=1.0, dot=1, norm=1, noise=2):
    import dynaquant_b200 as dq
    val = s.val.copy()
    rows = np.repeat(np.arange(s.n), np.diff(s.rowptr))
    val[rows == s.col] = np.random.default_rng(3).normal(0.0, 60.0, s.n)
    p = dq.Propagator(s.n, m=8, n_traj=B, dt=dt, noise=noise, seed=13, dot=dot, norm=norm, pop_every=1,
                      max_steps=steps, sigma_static=70.0, precision=dq.PREC_FP64)
    p.set_system(s)
    p.set_noise_params(np.full(s.n, 120.0), np.full(s.n, 60.0))
    p.set_initial_state(s.bright_state((1.0, 1.0, 1.0)))
    p.set_taylor_krylov(p_tk, m_b, s.rowptr, s.col, val)
    p.set_ipr(True)
    getattr(p, how)(steps)
    out = p.populations(), p.correlation(), p.ipr(), p.error_accum()
    shape = p.debug_step_shape()
    p.close()
    return out, shape


# form: CTAs (None: any number, 0: several launches), whether records are asked for
@pytest.mark.parametrize("shape,B,m_b,ctas,records", [
    ((2000,), 3, 6, None, True),       # a chain whose records fit
    ((50000,), 2, 6, 16, True),        # row starts fit, records do not
    ((62000,), 2, 6, 16, False),       # not even the row starts
    ((70000,), 2, 6, 0, False),        # too large for a cluster
    ((172, 172), 16, 12, None, None),  # a lattice between the two
])
def test_forms_match_per_trajectory_path(shape, B, m_b, ctas, records):
    from dynaquant_b200 import systems
    s = systems.chain(*shape) if len(shape) == 1 else systems.lattice2d(*shape)
    got, form = _run(s, "run", B, 3, 3, m_b)
    ref, _ = _run(s, "run_plain", B, 3, 3, m_b)
    if ctas is not None:
        assert form[1] == ctas, form
    if records is not None:
        assert (form[3] > 0) == records, form
    for a, b in zip(got[:3], ref[:3]):
        assert np.abs(a - b).max() < TOL * max(1.0, np.abs(b).max())
    assert np.allclose(got[3], ref[3], rtol=1e-6, atol=1e-14)


# steps that need the dense exponential: the |Re|-only norm and, in Taylor-Krylov, any halving; one launch
# (few and many trajectories to a CTA) and several
@pytest.mark.parametrize("shape,B,m_b,one_launch", [((12, 12), 7, 10, True), ((8, 8), 70, 20, True),
                                                    ((30, 30), 33, 12, True), ((70000,), 2, 6, False)])
@pytest.mark.parametrize("norm", [0, 1])
def test_dense_exponential_matches_per_trajectory_path(shape, B, m_b, one_launch, norm):
    from dynaquant_b200 import systems
    s = systems.chain(*shape) if len(shape) == 1 else systems.lattice2d(*shape)
    got, form = _run(s, "run", B, 3, 3, m_b, dt=9.0, norm=norm)
    ref, _ = _run(s, "run_plain", B, 3, 3, m_b, dt=9.0, norm=norm)
    assert (form[1] > 0) == one_launch
    for a, b in zip(got[:3], ref[:3]):
        assert np.abs(a - b).max() < TOL * max(1.0, np.abs(b).max())
    assert np.allclose(got[3], ref[3], rtol=1e-6, atol=1e-14)
