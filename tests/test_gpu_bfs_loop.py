"""Single-source BFS at the edges of its bitmap words, warp turns and lists
(vertex counts around 32, 128 and 4 * 32 * 8; hubs, chains, lists of one to
hundreds of entries; push, pull and both), against the oracle's levels and its
check of the parents."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def shape(kind, n, rng):
    v = np.arange(n)
    if kind == "chain":
        m = min(n, 300)
        return np.stack([v[: m - 1], v[1:m]], 1)
    if kind == "hub":  # one list of every vertex, found late from the far ones
        return np.concatenate([np.stack([v, np.full(n, n // 2)], 1), rng.integers(0, n, (n // 4 + 1, 2))])
    if kind == "dense":
        return rng.integers(0, n, (60 * n, 2))
    if kind == "two far":  # long lists without a frontier vertex until late
        h = n // 2
        a, b = rng.integers(0, h, (40 * h, 2)), rng.integers(h, n, (40 * (n - h), 2))
        return np.concatenate([a, b, [[h - 1, h]]])
    return rng.integers(0, n, (3 * n, 2))  # sparse: isolated vertices and small parts


@pytest.mark.parametrize("undirected,csc", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("n", [2, 31, 33, 127, 129, 1025, 8191, 70001])
@pytest.mark.parametrize("kind", ["chain", "hub", "dense", "two far", "sparse"])
def test_levels_and_parents(kind, n, undirected, csc):
    import everythinggraph_gb300 as eg

    pairs = shape(kind, n, np.random.default_rng(n)).astype(np.uint32).reshape(-1)
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs, undirected=undirected).build(eg.CSR | (eg.CSC if csc else 0))
    adj = oracle.build_adj(n, pairs, undirected)
    for root in (0, n - 1):
        ref = oracle.bfs_levels(n, adj.out_ptr, adj.out_col, root)
        for direction in ("auto", "push", "pull") if csc or undirected else ("push",):
            lv, par, st = g.bfs(root, direction=direction, parents=True)
            assert np.array_equal(lv, ref)
            assert oracle.bfs_tree_ok(n, adj.out_ptr, adj.out_col, root, lv, par)
            assert st.reached == np.count_nonzero(ref)
    ctx.close()
