"""PageRank's one-launch path at the sizes where its branches change (the
staged limit of 40,960 vertices, rows of one lane, 8 lanes, a warp, a CTA,
rows without entries, more rows or fewer entries than CTAs) against FP64:
relative L1 <= 1e-6 and max relative <= 1e-5, the bounds of the other PageRank
tests."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def pairs_of(n, lengths, extra, seed):
    """Vertex i < len(lengths) has lengths[i] in-edges and the others `extra`
    random edges among them; a fifth of the vertices has no out-edge."""
    rng = np.random.default_rng(seed)
    src = np.arange(n)[: max(1, n - n // 5)]
    p = [np.stack([rng.choice(src, d), np.full(d, i % n)], 1) for i, d in enumerate(lengths)]
    p.append(np.stack([rng.choice(src, extra), rng.integers(0, max(1, n // 2), extra)], 1))
    return rng.permutation(np.concatenate(p)).astype(np.uint32).reshape(-1)


LENGTHS = [1, 7, 8, 9, 31, 33, 127, 128, 129, 1000, 4095, 4096, 4097, 9000, 20000]


@pytest.mark.parametrize("n,extra", [(1, 3), (2, 1), (1000, 0), (5003, 60000), (40960, 400000), (40961, 400000),
                                     (200003, 300000)])
@pytest.mark.parametrize("opts", [{}, {"dangling": True}, {"tolerance": 1e-5, "dangling": True},
                                  {"swap": False, "prev_init": 0.15}, {"deg_multiplier": 2, "tolerance": 1e-4}])
def test_one_launch_vs_fp64(n, extra, opts):
    import everythinggraph_gb300 as eg

    pairs = pairs_of(n, LENGTHS, extra, n)
    adj = oracle.build_adj(n, pairs)
    deg = adj.out_deg().astype(np.int64) * opts.get("deg_multiplier", 1)
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs).build(eg.CSR | eg.CSC)
    launches = ctx.kernel_launches
    got, st = g.pagerank(iterations=30 if "tolerance" in opts else 8, **opts)
    got, st = g.pagerank(iterations=30 if "tolerance" in opts else 8, **opts)
    assert ctx.kernel_launches - launches < 60  # the relabelled copy's, then two a run
    replay, _ = g.pagerank(iterations=30 if "tolerance" in opts else 8, use_graph=True, **opts)
    assert np.array_equal(got, replay)
    its = 1 if opts.get("swap") is False else st.iterations_run
    ref = oracle.pagerank_f64(adj, deg.astype(np.uint32), float(np.float32(opts.get("prev_init", 1.0 / n))), its,
                              dangling=opts.get("dangling", False), damping=float(np.float32(0.85)))
    d = np.abs(got - ref)
    assert d.sum() <= 1e-6 * ref.sum() and (d / ref).max() <= 1e-5
    if "tolerance" in opts:
        assert st.iterations_run < 30 and st.residual < opts["tolerance"]
    ctx.close()
