"""WCC where ids follow the structure (a path, a mesh, a comb with ids in
order, ascending and descending): labels against the oracle's, and the time of
a path against a random graph's of the same vertices."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def shape(kind, n):
    v = np.arange(n)
    if kind == "path":
        return np.stack([v[:-1], v[1:]], 1)
    if kind == "mesh":
        a = int(n ** 0.5)
        q = np.arange(a * a).reshape(a, a)
        return np.concatenate([np.stack([q[:, :-1].ravel(), q[:, 1:].ravel()], 1),
                               np.stack([q[:-1].ravel(), q[1:].ravel()], 1)])
    if kind == "comb":  # many paths of growing length, their ends joined two by two
        cut = np.cumsum(np.arange(1, int((2 * n) ** 0.5)))
        cut = cut[cut < n - 1]
        e = np.stack([v[:-1], v[1:]], 1)
        return np.concatenate([np.delete(e, cut, 0), np.stack([cut[:-1:2], cut[1::2][: len(cut[:-1:2])]], 1)])
    return np.stack([v[:-2], v[2:]], 1)  # two interleaved paths


@pytest.mark.parametrize("undirected,csc", [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize("n", [1024, 40001, 1 << 20])
@pytest.mark.parametrize("kind", ["path", "mesh", "comb", "two"])
@pytest.mark.parametrize("down", [False, True])
def test_labels(kind, n, undirected, csc, down):
    import everythinggraph_gb300 as eg

    pairs = shape(kind, n).astype(np.uint32)
    if down:
        pairs = n - 1 - pairs
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs.reshape(-1), undirected=undirected).build(eg.CSR | (eg.CSC if csc else 0))
    ref = oracle.wcc(n, pairs.reshape(-1))
    for _ in range(2):
        lab, st = g.wcc()
        assert np.array_equal(lab, ref)
        assert st.components == len(np.unique(ref))
    ctx.close()


@pytest.mark.parametrize("n", [300000, 1 << 21])
def test_time_of_a_path(n):
    import everythinggraph_gb300 as eg

    ctx = eg.Context(0)
    t = []
    for pairs in (shape("path", n), np.random.default_rng(1).integers(0, n, (n, 2))):
        g = ctx.from_pairs(n, pairs.astype(np.uint32).reshape(-1), undirected=True).build()
        g.wcc(copy_out=False)
        t.append(min(g.wcc(copy_out=False)[1].ms for _ in range(7)))
        g.free()
    ctx.close()
    print(t)
    assert t[0] <= 1.5 * t[1], t


def test_time_of_a_path_through_shuffled_ids():
    import everythinggraph_gb300 as eg

    n = 1000000
    rng = np.random.default_rng(1)
    p = rng.permutation(n)
    ctx = eg.Context(0)
    t = []
    for pairs in (np.stack([p[:-1], p[1:]], 1), rng.integers(0, n, (n, 2))):
        g = ctx.from_pairs(n, pairs.astype(np.uint32).reshape(-1), undirected=True).build()
        g.wcc(copy_out=False)
        t.append(min(g.wcc(copy_out=False)[1].ms for _ in range(7)))
        g.free()
    ctx.close()
    print(t)
    assert t[0] <= 2.5 * t[1], t
