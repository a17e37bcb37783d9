"""Graphs at the top of the range of adjacency entries (32-bit offsets hold at
most 2^32 - 2), where a place plus a step no longer fits 32 bits."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def need(gigabytes):
    import torch

    if torch.cuda.mem_get_info()[0] < gigabytes << 30:
        pytest.skip("needs %d GB of device memory" % gigabytes)


@pytest.mark.parametrize("m", [2 ** 32 - 5, 2 ** 32 - 4, 2 ** 32 - 3, 2 ** 32 - 2])
def test_row_starts(m):
    """Every row ends where the next one begins, the last one at m."""
    import everythinggraph_gb300 as eg

    need(110)
    n = 61
    ctx = eg.Context(0)
    g = ctx.er(n, m, 5).build(eg.CSR)
    ptr = np.empty(n + 1, dtype=np.uint32)
    eg.L.check(eg.lib().eg_graph_copy_adj(g._h, eg.CSR, ctypes.c_void_p(ptr.ctypes.data), None))
    deg = g.degrees()[0].astype(np.int64)
    assert ptr[0] == 0 and ptr[n] == m
    assert np.array_equal(np.diff(ptr.astype(np.int64)), deg)
    assert np.all(np.abs(deg - m / n) < 8 * (m / n) ** 0.5)  # uniform draws
    ctx.close()
