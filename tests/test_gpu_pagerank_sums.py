"""PageRank's residual and dangling mass against exact sums (math.fsum) over
the returned ranks of the last iteration and the one before it.  Both are sums
of fp32 values kept as fp32 triples, widened once: half a unit of FP64 in the
result, half in the reference, so 2^-52 of the value at most."""
import math

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -52


# one launch (contributions staged, gathered) and a launch per step
@pytest.mark.parametrize("n,m,undirected", [(5003, 40000, False), (60013, 500000, False), (300007, 900001, False),
                                            (700001, 2100000, True)])
@pytest.mark.parametrize("iterations", [2, 5])
def test_residual_is_an_exact_sum(n, m, undirected, iterations):
    import everythinggraph_gb300 as eg

    pairs = (np.random.default_rng(n).random((m, 2)) ** 2 * n).astype(np.uint32)
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs.reshape(-1), undirected=undirected).build(eg.CSR | eg.CSC)
    opts = dict(tolerance=1e-30, dangling=True)
    before, _ = g.pagerank(iterations=iterations - 1, **opts)
    rank, st = g.pagerank(iterations=iterations, **opts)
    assert st.iterations_run == iterations
    residual = math.fsum(np.abs(rank - before).tolist())
    assert abs(st.residual - residual) <= TOL * residual
    dangling = math.fsum(rank[g.degrees()[0] == 0].tolist())
    assert abs(st.dangling_mass - dangling) <= TOL * dangling
    ctx.close()


@pytest.mark.parametrize("schedule", [0, 12])
def test_dangling_mass_of_many_ranks(schedule):
    """8 M ranks of 2^-27 to 2^-13: their sum needs more than the 48 bits of
    an fp32 pair."""
    import everythinggraph_gb300 as eg

    ctx = eg.Context(0)
    g = ctx.rmat(24, 1 << 27, 3).build(eg.CSR | eg.CSC)
    g.set_row_schedule(schedule)
    none = g.degrees()[0] == 0
    for iterations in (1, 3):
        rank, st = g.pagerank(iterations=iterations, tolerance=1e-30, dangling=True)
        dangling = math.fsum(rank[none].tolist())
        assert abs(st.dangling_mass - dangling) <= TOL * dangling
    ctx.close()


def test_sums_past_fp32():
    """A total beyond fp32's range (a huge start value) stays finite."""
    import everythinggraph_gb300 as eg

    for n, m in ((5003, 40000), (300007, 900001)):
        pairs = np.random.default_rng(n).integers(0, n, 2 * m).astype(np.uint32)
        ctx = eg.Context(0)
        g = ctx.from_pairs(n, pairs).build(eg.CSR | eg.CSC)
        start = 1e35
        rank, st = g.pagerank(iterations=3, prev_init=start, tolerance=1e-30, dangling=True)
        adj = oracle.build_adj(n, pairs)
        ref = oracle.pagerank_f64(adj, adj.out_deg(), float(np.float32(start)), 3, dangling=True)
        assert np.all(np.isfinite(rank)) and math.isfinite(st.dangling_mass) and math.isfinite(st.residual)
        assert float(np.abs(rank - ref).sum() / ref.sum()) <= 1e-6
        ctx.close()
