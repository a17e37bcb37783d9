"""eg_graph_tune on a graph small enough for PageRank in one launch keeps that
form: a tuned graph launches as often as an untuned one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(10007, 120000), (90001, 600000)])
def test_tuned_small_graph_runs_in_one_launch(n, m):
    import everythinggraph_gb300 as eg

    ctx = eg.Context(0)
    g = ctx.from_pairs(n, np.random.default_rng(n).integers(0, n, 2 * m, dtype=np.uint32), undirected=True)
    g.build(eg.CSR | eg.CSC)

    def launches():
        before = ctx.kernel_launches
        rank, _ = g.pagerank(iterations=10)
        return ctx.kernel_launches - before, rank

    launches()
    untuned, ref = launches()
    cands, chosen = g.tune()
    tuned, rank = launches()
    assert cands[chosen]["ms"] == min(c["ms"] for c in cands)
    assert tuned == untuned, (chosen, [c["ms"] for c in cands])
    assert np.array_equal(rank, ref)
    g.set_row_schedule(chosen)  # the index kept from a tuning says the same
    assert launches()[0] == untuned
    ctx.close()
