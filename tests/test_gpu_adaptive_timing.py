"""dq_time_iteration on contexts with the adaptive Krylov dimension: an iteration costs what it costs with
the dimension fixed, whatever the ensemble would choose or chose before (autotuning compares these)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the cluster form, whose launch runs all iterations, and a grid-wide one
@pytest.mark.parametrize("tiling", [(8, 2, 4, 3, 13, 1), (16, 2, 2, 3, 0, 1)])
def test_adaptive_contexts_time_whole_iterations(tiling):
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    s = systems.tube(30, 50)
    ms = {}
    for m_min in (0, 4):
        p = dq.Propagator(s.n, m=28, n_traj=64, dt=0.5, noise=dq.NOISE_OU, seed=5, precision=dq.PREC_MIXED,
                          max_steps=4, m_min=m_min, m_tol=1e-2)   # chooses 4 of 28
        p.set_system(s)
        p.set_noise_params(np.full(s.n, 250.0), np.full(s.n, 50.0))
        p.set_initial_state(s.bright_state())
        p.set_tiling(*tiling)
        p.run(2)   # leaves its chunks' choices behind
        ms[m_min] = min(p.time_iteration(20) for _ in range(5))
        p.close()
    # the same work: far from the 4 / 28 of a run that stops early, or from none at all
    assert 0.6 < ms[4] / ms[0] < 1.6, ms


@pytest.mark.parametrize("m_min", [0, 4])
def test_autotuned_context_reproduces_an_untuned_one(m_min):
    """Autotuning, which with an adaptive dimension compares whole steps, leaves a context that starts over."""
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    s = systems.tube(20, 30)
    out = []
    for tune in (False, True):
        p = dq.Propagator(s.n, m=16, n_traj=16, dt=0.5, noise=dq.NOISE_OU, seed=5, precision=dq.PREC_FP64, max_steps=3,
                          m_min=m_min, m_tol=1e-9)
        p.set_system(s)
        p.set_noise_params(np.full(s.n, 250.0), np.full(s.n, 50.0))
        p.set_initial_state(s.bright_state())
        if tune:
            assert p.autotune_raw(1) > 0.0
            assert p.steps_done == 0
        p.run(3)
        out.append((p.populations(), p.correlation(), p.error_accum()))
        p.close()
    assert np.abs(out[0][0] - out[1][0]).max() < 1e-10 and np.abs(out[0][1] - out[1][1]).max() < 1e-9
    assert np.allclose(out[0][2], out[1][2], rtol=1e-3, atol=1e-13)
