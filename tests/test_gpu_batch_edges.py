"""Batched kernels at the list lengths where their branches change: the
bit-sliced pull's 32- and 1056-entry cuts and the personalised PageRank's
512-entry parts, against the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def hub_graph(degrees, n, seed, extra):
    """Pairs of a directed graph whose vertex i < len(degrees) has exactly
    degrees[i] in-edges; `extra` random edges among the other vertices."""
    rng = np.random.default_rng(seed)
    h = len(degrees)
    parts = [np.stack([rng.integers(h, n, d), np.full(d, i)], 1) for i, d in enumerate(degrees)]
    parts.append(rng.integers(h, n, (extra, 2)))
    pairs = np.concatenate(parts)
    return rng.permutation(pairs).astype(np.uint32).reshape(-1)


@pytest.mark.parametrize("k", [1, 31, 33, 64])
@pytest.mark.parametrize("n", [1023, 4097])
def test_multi_bfs_list_cuts(n, k):
    import everythinggraph_gb300 as eg

    degrees = [0, 1, 3, 4, 5, 31, 32, 33, 36, 1055, 1056, 1057, 2080, 2081, 6000]
    pairs = hub_graph(degrees, n, n + k, 2 * n)
    adj = oracle.build_adj(n, pairs)
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs).build(eg.CSR | eg.CSC)
    roots = np.random.default_rng(k).integers(0, n, k).astype(np.uint32)
    roots[0] = len(degrees)
    lv, st = g.bfs_multi(roots)
    for s in range(k):
        assert np.array_equal(lv[s], oracle.bfs_levels(n, adj.out_ptr, adj.out_col, int(roots[s]))), s
    assert st.reached == int((lv > 0).sum())
    ctx.close()
