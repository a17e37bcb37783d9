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


def test_sssp_round_over_all_entries():
    """One round lists all entries but two: vertices 5 and 20 are reached at
    distances 5 and 0, their lists fill the places up to 2^32 - 4."""
    import torch

    import everythinggraph_gb300 as eg

    need(130)
    n, m = 50, 2 ** 32 - 2
    pairs = torch.empty((m, 2), dtype=torch.int32, device="cuda")
    pairs[:, 0] = 5
    pairs[:, 1] = 30
    for i in range(1, 8):  # the first entries of 5's list, which places past 2^32 would wrap to
        pairs[i::1 << 10, 1] = 30 + i
    pairs[-2, 0], pairs[-2, 1] = 10, 5
    pairs[-1, 0], pairs[-1, 1] = 10, 20
    z = 1 << 20  # more than a warp's share: the last warp's window holds vertex 20 alone
    pairs[-2 - z:-2, 0] = 20
    pairs[-2 - z:-2, 1] = 40 + torch.arange(z, dtype=torch.int32, device="cuda") % 10
    torch.cuda.synchronize()
    ctx = eg.Context(0)
    g = ctx.from_device_pairs(n, pairs.data_ptr(), m)
    ctx.sync()
    del pairs
    torch.cuda.empty_cache()
    g.build(eg.CSR)
    dist, st = g.sssp(10, eg.weights("ref"))  # u % 10 + v % 10
    ref = np.full(n, eg.UNREACHED_SSSP, dtype=np.uint32)
    ref[10], ref[5], ref[20] = 0, 5, 0
    ref[30:38] = 10 + np.arange(8)
    ref[40:50] = np.arange(10)
    assert np.array_equal(dist, ref)
    assert st.relaxations == m
    ctx.close()


@pytest.mark.parametrize("last", [33, 900, 3000])
def test_multi_bfs_pull_of_the_last_list(last):
    """The last vertex's in-list ends at entry 2^32 - 2 and has no reached
    vertex: the pull reads it to the end and no further."""
    import torch

    import everythinggraph_gb300 as eg

    need(190)
    n, m = 40, 2 ** 32 - 2
    pairs = torch.empty((m, 2), dtype=torch.int32, device="cuda")
    pairs[:, 0] = 1
    pairs[:, 1] = 3
    pairs[-last:, 0] = 2
    pairs[-last:, 1] = n - 1
    pairs[-last - 1, 0], pairs[-last - 1, 1] = 3, 7
    torch.cuda.synchronize()
    ctx = eg.Context(0)
    g = ctx.from_device_pairs(n, pairs.data_ptr(), m)
    ctx.sync()
    del pairs
    torch.cuda.empty_cache()
    g.build(eg.CSR | eg.CSC)
    lv, st = g.bfs_multi(np.array([1, 3], dtype=np.uint32))
    ref = np.zeros((2, n), dtype=np.int32)
    ref[0, [1, 3, 7]] = 1, 2, 3
    ref[1, [3, 7]] = 1, 2
    assert np.array_equal(lv, ref)
    assert st.pull_levels >= 1
    ctx.close()


def test_bfs_and_wcc_over_all_entries():
    """Lists of about 4096 entries up to entry 2^32 - 2: all vertices within
    three levels of any root, one component."""
    import torch

    import everythinggraph_gb300 as eg

    need(190)
    n, m = 1 << 20, 2 ** 32 - 2
    ctx = eg.Context(0)
    g = ctx.er(n, m, 11).build(eg.CSR | eg.CSC)
    deg = g.degrees()[0].astype(np.int64)
    start = np.concatenate([[0], np.cumsum(deg)])
    assert start[-1] == m

    class Col:
        __cuda_array_interface__ = {"shape": (m,), "typestr": "<i4", "version": 3,
                                    "data": (g.device_ptr(eg.L.EG_DEV_CSR_COL), False)}

    col = torch.as_tensor(Col(), device="cuda")
    for root in (n - 1, 12345):  # the first's list is the last one
        near = np.unique(col[int(start[root]):int(start[root + 1])].cpu().numpy())
        ref = np.full(n, 3, dtype=np.int32)
        ref[near] = 2
        ref[root] = 1
        for direction in ("auto", "push", "pull"):
            lv, par, st = g.bfs(root, direction=direction, parents=True)
            assert np.array_equal(np.minimum(lv, 3), ref) and lv.max() <= 4
            assert st.reached == n and st.edges_traversed == m
            assert np.all(lv[par] == np.maximum(lv - 1, 1))
    lab, st = g.wcc()
    assert st.components == 1 and not lab.any()
    del col
    ctx.close()
