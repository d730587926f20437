"""The drop-in step's shape stays within what the device can hold at once (clusters of fewer CTAs, fewer
CTAs of a cooperative grid), and falls back to several launches where nothing fits (host arithmetic)."""
import ctypes as C

import pytest

from dynaquant_b200 import _lib

SMEM_MAX = 224 * 1024


def _shape(n, m, bw, z, cluster, grid):
    v = [C.c_int() for _ in range(3)]
    rc = _lib.load().dq_debug_plain_shape(n, m, bw, z, cluster, grid, *[C.byref(x) for x in v])
    assert rc == 0
    return tuple(x.value for x in v)


@pytest.mark.parametrize("cluster,grid", [(16, 148), (8, 148), (16, 40), (8, 64), (1, 148), (1, 0), (0, 0)])
@pytest.mark.parametrize("m", [2, 20, 32])
def test_shape_stays_within_the_device(cluster, grid, m):
    n = 2.0
    while n < 200000:
        # chain, lattice, tube of 28 couplings, and columns unknown beforehand (the static call)
        for bw, z in ((1, 2.0), (int(n ** 0.5) + 1, 8.0), (200, 28.0), (int(n), 0.0)):
            k = int(n)
            ctas, rows, smem = _shape(k, m, min(bw, k - 1) if z else k, z, cluster, grid)
            if ctas == 0:
                continue
            assert ctas <= (cluster if ctas <= 16 else grid), (k, bw, z)
            assert ctas * rows >= k and (ctas - 1) * rows < k
            # the block starts and the dense exponential's matrices have their place in it
            assert smem <= SMEM_MAX and smem >= 6 * 16 * (m + 2) ** 2 + 4 * rows
        n *= 1.05


def test_shapes_of_a_whole_device():
    """A full device takes one CTA, a cluster and the whole grid as the sizes grow; none of them elsewhere."""
    assert _shape(64, 16, 1, 2.0, 16, 148)[0] == 1
    assert 1 < _shape(1024, 16, 1, 2.0, 16, 148)[0] <= 16
    assert 16 < _shape(30000, 20, 180, 28.0, 16, 148)[0] <= 148
    for n, bw, z in ((64, 1, 2.0), (1024, 1, 2.0), (30000, 180, 28.0)):
        assert _shape(n, 16, bw, z, 0, 0)[0] == 0
