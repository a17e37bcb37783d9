"""PageRank with a launch per step (schedules other than the default keep small
graphs on it): rows over one, two and many tiles, neighbouring long rows, rows
without entries, vertex counts around 4, against FP64: relative L1 <= 1e-6 and
max relative <= 1e-5, the bounds of the other PageRank tests; and the residual
against the two last FP64 iterations."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", [1, 4, 6])
@pytest.mark.parametrize("n,m", [(5, 9), (4099, 30000), (50002, 700001), (300003, 900000)])
@pytest.mark.parametrize("opts", [{}, {"dangling": True}, {"tolerance": 1e-5, "dangling": True},
                                  {"tolerance": 1e-5}, {"compensated": True, "dangling": True}])
def test_launches_vs_fp64(schedule, n, m, opts):
    import everythinggraph_gb300 as eg

    rng = np.random.default_rng(m)
    src = rng.integers(0, max(1, n - n // 5), m)
    dst = rng.integers(0, max(1, n // 2), m)
    hubs = np.arange(min(n, 12)) * (n // 12 + 1) % n  # a few rows of tiles each
    long = rng.random(m) < 0.5
    dst[long] = rng.choice(hubs, int(long.sum()))
    pairs = np.stack([src, dst], 1).astype(np.uint32).reshape(-1)
    adj = oracle.build_adj(n, pairs)
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs).build(eg.CSR | eg.CSC)
    g.set_row_schedule(schedule)
    got, st = g.pagerank(iterations=40 if "tolerance" in opts else 8, **opts)
    refs = [oracle.pagerank_f64(adj, adj.out_deg(), float(np.float32(1.0 / n)), its,
                                dangling=opts.get("dangling", False), damping=float(np.float32(0.85)))
            for its in (st.iterations_run - 1, st.iterations_run)]
    d = np.abs(got - refs[1])
    assert d.sum() <= 1e-6 * refs[1].sum() and (d / refs[1]).max() <= 1e-5
    if "tolerance" in opts:
        # both iterates are within 1e-6 of their sums, so their distance is within 2e-6
        assert abs(st.residual - np.abs(refs[1] - refs[0]).sum()) <= 2e-6 * refs[1].sum()
        assert st.iterations_run < 40 and st.residual < opts["tolerance"]
    ctx.close()
