"""Layout builds at the sizes where the sort's tiles, digit widths and pass
counts change, against numpy's stable sort, and the context's kept blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def expected(n, src, dst):
    """CSR (stable by src) and CSC (that order, stable by dst) of the entries."""
    def rows(key):
        ptr = np.zeros(n + 1, dtype=np.int64)
        np.cumsum(np.bincount(key, minlength=n), out=ptr[1:])
        return ptr

    o = np.argsort(src, kind="stable")
    rid, col = src[o], dst[o]
    p = np.argsort(col, kind="stable")
    return rows(src), col, rows(dst), rid[p]


# n: 1, 8, 9 (one 9-bit pass), 16, 17 (9 + 8), 18, 24 and 25 bits (9 + 8 + 8);
# m around the 4096-entry tile, several tiles per thread block, and m_in off
# the tile so that one tile of an undirected input holds both directions
@pytest.mark.parametrize("n", [1, 2, 256, 257, 65536, 65537, (1 << 18) - 1, (1 << 24) - 5, (1 << 24) + 3])
@pytest.mark.parametrize("m,undirected", [(0, False), (1, True), (4095, False), (4096, False), (4097, True),
                                          (2048, True), (123457, True)])
def test_build_matches_stable_sort(n, m, undirected):
    import everythinggraph_gb300 as eg

    rng = np.random.default_rng(n * 7 + m)
    pairs = rng.integers(0, n, (m, 2), dtype=np.uint32)
    if m > 100:  # runs of one key fill whole warps and tiles
        pairs[m // 4:m // 2, 0] = n - 1
        pairs[m // 3:m // 2 + 7, 1] = n // 2
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs.reshape(-1), undirected=undirected).build(eg.CSR | eg.CSC)
    src, dst = pairs[:, 0].astype(np.int64), pairs[:, 1].astype(np.int64)
    if undirected:
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    optr, ocol, iptr, icol = expected(n, src, dst)
    for layout, ptr, col in ((eg.CSR, optr, ocol), (eg.CSC, iptr, icol)):
        p, c = g.adj(layout)
        assert np.array_equal(p, ptr) and np.array_equal(c, col)
    od, idg = g.degrees(inn=True)
    assert np.array_equal(od, np.diff(optr)) and np.array_equal(idg, np.diff(iptr))
    ctx.close()


@pytest.mark.parametrize("m", [4096, 300000])
def test_bad_endpoint_is_refused(m):
    import everythinggraph_gb300 as eg

    ctx = eg.Context(0)
    for at in (0, 2 * m - 1):
        pairs = np.zeros(2 * m, dtype=np.uint32)
        pairs[at] = 77
        g = ctx.from_pairs(77, pairs)
        with pytest.raises(eg.EGError) as e:
            g.build(eg.CSR | eg.CSC)
        assert e.value.code == -7
        assert g.info().layouts == 0
        g.free()
    ctx.close()


def test_kept_blocks_are_reused_and_given_back():
    """Freed blocks serve the next graph, are not counted as in use, and give
    way when the budget has no room beside them."""
    import everythinggraph_gb300 as eg

    ctx = eg.Context(0)
    ref = None
    for _ in range(3):  # the second and third graph are built in kept blocks
        g = ctx.rmat(16, 1 << 20, 5, undirected=True).build(eg.CSR | eg.CSC)
        got = g.adj(eg.CSC)
        ref = ref or (got, ctx.bytes_in_use)
        assert np.array_equal(got[0], ref[0][0]) and np.array_equal(got[1], ref[0][1])
        assert ctx.bytes_in_use == ref[1]
        lv, _ = g.bfs(int(g.sample_roots(1, 1)[0]))
        assert lv.max() > 1
        g.free()
    ctx.close()
    # the first graph's blocks (about 33 MB) and the second's (about 67 MB)
    # do not fit the budget together
    ctx = eg.Context(0, hbm_budget=80 << 20)
    ctx.rmat(14, 1 << 20, 5).build(eg.CSR | eg.CSC).free()
    g = ctx.rmat(15, 2 << 20, 5).build(eg.CSR | eg.CSC)
    assert g.adj(eg.CSR)[0][-1] == 2 << 20
    ctx.close()
