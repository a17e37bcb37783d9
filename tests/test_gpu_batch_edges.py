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


@pytest.mark.parametrize("nq", [1, 5, 32])
def test_ppr_row_parts(nq):
    """Rows of 1 .. 5000 entries (parts of 512, quarters of the parts), seeds
    on rows without entries, queries that stop at different sweeps.  fp32 sums
    of up to 5000 terms: each result within relative L1 2e-6 of FP64."""
    import everythinggraph_gb300 as eg

    n = 3001
    degrees = [0, 1, 7, 8, 9, 15, 16, 510, 511, 512, 513, 1023, 1024, 1025, 2049, 5000, 0]
    pairs = hub_graph(degrees, n, 3, 4 * n)
    adj = oracle.build_adj(n, pairs)
    rng = np.random.default_rng(nq)
    seeds = [rng.integers(0, n, int(rng.integers(1, 9))) for _ in range(nq)]
    seeds[0] = np.array([0, 16, 0])  # no in-edges, one of them twice
    tol = [10.0 ** -(3 + q % 4) for q in range(nq)]
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs).build(eg.CSR | eg.CSC)
    ranks, st = g.ppr(seeds, tolerance=tol, max_iters=40)
    for q in range(nq):
        ref, its = oracle.ppr_f64(adj, adj.out_deg(), seeds[q], damping=float(np.float32(0.85)), tol=0.0,
                                  max_iters=st.iterations[q])
        assert np.abs(ranks[q] - ref).sum() <= 2e-6 * np.abs(ref).sum()
        alone, sta = g.ppr([seeds[q]], tolerance=tol[q], max_iters=40)
        assert sta.iterations[0] == st.iterations[q] and np.array_equal(alone[0], ranks[q])
    ctx.close()
