"""The shared memory that a Taylor-Krylov cluster step asks for holds what the kernel writes into it:
whatever the sites, bandwidth and trajectories, the row starts in front of the coupling records fit the
records' part, or that part is empty (host arithmetic only)."""
import ctypes as C

import pytest

from dynaquant_b200 import _lib

SMEM_MAX = 224 * 1024


def _shape(n, ctas, traj, m_b, bw):
    smem, rec, head = C.c_int(), C.c_int(), C.c_int()
    rc = _lib.load().dq_debug_taylor_shape(n, ctas, traj, m_b, bw, C.byref(smem), C.byref(rec), C.byref(head))
    return None if rc else (smem.value, rec.value, head.value)


def _sizes():
    n = 2.0
    while n < 90000:
        yield int(n)
        n *= 1.031
    # a chain whose only shape has no room for its row starts, and lattices and tubes beside such sizes
    yield from (144 * 144, 172 * 172, 62000, 60600, 63900, 45000, 29600, 14500, 13500, 8800)


@pytest.mark.parametrize("m_b", [1, 12, 32])
@pytest.mark.parametrize("traj", [1, 2, 4, 8, 16, 32])
def test_row_starts_fit_the_records_part(m_b, traj):
    seen = [0, 0]
    for n in _sizes():
        for ctas in range(1, 17):
            for bw in {1, 12, int(n ** 0.5), 150, n // 4, n - 1}:
                got = _shape(n, ctas, traj, m_b, bw)
                if got is None:
                    continue
                smem, rec, head = got
                rows = -(-n // ctas)
                assert head >= 4 * (rows + 2)
                assert rec == 0 or head <= rec, (n, ctas, bw, got)
                assert smem <= SMEM_MAX and rec <= smem
                seen[rec == 0] += 1
    assert seen[0] and (seen[1] or traj > 2)   # small chunks do reach the sizes without records


def test_shapes_out_of_range_are_refused():
    assert _shape(1, 1, 1, 4, 1) is None and _shape(100, 17, 1, 4, 1) is None and _shape(100, 1, 3, 4, 1) is None
    assert _shape(100, 1, 64, 4, 1) is None and _shape(10 ** 6, 16, 1, 4, 1) is None
