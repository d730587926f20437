"""The tiling of an ensemble that no one tuned: the cluster form where it is the faster one (times beside
the rule), a grid-wide form where many FP64 rows per CTA make it the slower one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTER = 13


@pytest.mark.parametrize("shape,B,precision,m_min,cluster", [
    ((2000,), 64, 0, 0, True), ((8000,), 48, 0, 0, True), ((15000,), 16, 0, 0, True), ((15000,), 64, 1, 0, True),
    ((15000,), 100, 0, 0, False), ((25000,), 100, 0, 0, False), ((25000,), 200, 0, 8, False),
    ((57, 83), 100, 0, 0, True), ((60, 250), 100, 0, 0, False)])
def test_untuned_choice(shape, B, precision, m_min, cluster):
    import dynaquant_b200 as dq
    from dynaquant_b200 import systems
    s = systems.chain(*shape) if len(shape) == 1 else systems.tube(*shape)
    p = dq.Propagator(s.n, m=16, n_traj=B, dt=0.5, precision=precision, max_steps=1, m_min=m_min)
    p.set_system(s)
    p.set_initial_state(np.ones(s.n) / np.sqrt(s.n))
    assert (p.get_tiling()[4] == CLUSTER) == cluster
    p.close()
