"""Batched personalised PageRank: the rounding error of one row's sum, at row
lengths up to an item, one item, and rows in parts, against FP64.  Entries are
added eight by eight, the eights' sums to an item's (64 at most); parts the
same, a quarter of them per group; every entry is a quotient of a quotient, the
sum is scaled once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [7, 8, 63, 511, 512, 513, 1027, 4100, 20011])
@pytest.mark.parametrize("extra", [3, 41])
def test_row_of_equal_entries(length, extra):
    import everythinggraph_gb300 as eg

    seeds = np.arange(1, length + extra + 1)  # the first `length` have an edge to vertex 0, all eight edges
    n = len(seeds) + 9
    pairs = np.stack([np.repeat(seeds, 8), np.tile(n - 8 + np.arange(8), len(seeds))], 1)
    pairs[: 8 * length : 8, 1] = 0
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs.astype(np.uint32).reshape(-1)).build(eg.CSR | eg.CSC)
    rank, _ = g.ppr([seeds], damping=0.85, tolerance=0.0, max_iters=1)
    exact = float(np.float32(0.85)) * length / len(seeds) / 8
    parts = -(-length // 512)
    adds = 7 + min(-(-length // 8), 64) + (7 + -(-parts // 32) + 3 if parts > 1 else 0)
    assert abs(float(rank[0, 0]) - exact) <= (adds + 3) * 2.0 ** -24 * exact
    ctx.close()


def test_after_loading_layouts(tmp_path):
    """Layouts loaded into a graph that has run: the same queries, the same
    bits."""
    import everythinggraph_gb300 as eg

    ctx = eg.Context(0)
    g = ctx.rmat(14, 1 << 18, 3, undirected=True).build(eg.CSR | eg.CSC)
    seeds = [[int(s)] for s in g.sample_roots(5, 1)]
    ref, _ = g.ppr(seeds)
    path = str(tmp_path / "g.eglayout")
    g.save_layouts(path)
    for _ in range(2):
        assert g.load_layouts(path)
        rank, _ = g.ppr(seeds)
        assert np.array_equal(rank.view(np.uint32), ref.view(np.uint32))
    ctx.close()
