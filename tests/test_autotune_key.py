"""What the autotuner's cache tells apart: a tiling found for one Krylov dimension or bandwidth is not
taken for another, and files written before the keys held them are still read, but for the cluster form."""
import os
import sys
import types

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from dynaquant_b200 import autotune  # noqa: E402

ENTRY = {"traj_chunk": 16, "vec": 2, "ctas_per_sm": 2, "rows_per_block": 3, "staged": 0, "groups": 1,
         "ms_per_iter": 0.5}


class FakeProp:
    """What tune() uses of a Propagator, on a chain with couplings to `reach` sites on."""

    def __init__(self, m=16, m_min=0, reach=1, n=40):
        self.cfg = types.SimpleNamespace(device=0, n_sites=n, n_traj=32, precision=1, dot_mode=1, m=m, m_min=m_min)
        pairs = sorted({(i, i) for i in range(n)} | {(i, i + reach) for i in range(n - reach)}
                       | {(i + reach, i) for i in range(n - reach)})
        self._rp = np.zeros(n + 1, np.int32)
        np.cumsum(np.bincount([i for i, _ in pairs], minlength=n), out=self._rp[1:])
        self._col = np.array([j for _, j in pairs], np.int32)
        self.tiling, self.timed = None, 0

    def set_tiling(self, *t):
        self.tiling = t

    def get_tiling(self):
        return (8, 2, 4, 3, 13, 1)

    def reset(self):
        pass

    def autotune_raw(self, reps):
        self.timed += 1
        return 0.25


@pytest.fixture(autouse=True)
def _own_cache(tmp_path, monkeypatch):
    monkeypatch.setenv("DQ_TUNE_CACHE", str(tmp_path / "tiling.json"))


@pytest.mark.parametrize("other", [dict(m=24), dict(m_min=8), dict(reach=7)])
def test_entries_of_other_problems_are_not_taken(other):
    assert not autotune.tune(FakeProp(), 118)["cached"]
    p = FakeProp()
    assert autotune.tune(p, 118)["cached"] and p.timed == 0 and p.tiling == (8, 2, 4, 3, 13, 1)
    q = FakeProp(**other)
    assert not autotune.tune(q, 118)["cached"] and q.timed == 1


@pytest.mark.parametrize("staged,taken", [(0, True), (12, True), (13, False)])
def test_entries_of_earlier_files(staged, taken):
    p = FakeProp()
    old = autotune.key(p, 118)
    autotune.store(old[:old.index("|m=")], dict(ENTRY, staged=staged))
    assert autotune.tune(p, 118)["cached"] is taken
    assert p.timed == (0 if taken else 1)
