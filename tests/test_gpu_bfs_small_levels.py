"""BFS levels that one CTA takes alone: frontiers around a warp and around the
bound on their edges, in and out of wide levels and pulls; and what a level of
a path costs."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def layers(widths, rng, back):
    """Vertices in layers, every vertex with an edge from the layer before; with
    `back` extra edges inside and against the direction."""
    start = np.concatenate([[0], np.cumsum(widths)])
    e = []
    for i in range(1, len(widths)):
        v = np.arange(start[i], start[i + 1])
        u = rng.integers(start[i - 1], start[i], len(v))
        e.append(np.stack([u, v], 1))
        if back:
            e.append(np.stack([rng.permutation(v), rng.permutation(v)], 1))
            e.append(np.stack([v, rng.integers(start[i - 1], start[i], len(v))], 1))
    e = np.concatenate(e)
    ids = rng.permutation(int(start[-1]))
    return int(start[-1]), ids[e].astype(np.uint32), int(ids[0])


SHAPES = {
    "path": [1] * 700,
    "warp": [1, 31, 32, 33, 5, 33, 32, 1, 64, 65, 2],
    "bound": [1, 1023, 1024, 1025, 3, 1024, 1, 1025, 1024, 7],
    "wide": [1, 8, 400, 5000, 9000, 500, 40, 4, 1, 1, 3000, 2, 1],
    "hub": [1, 1, 1, 20000, 1, 1, 1, 600, 1],
}


@pytest.mark.parametrize("undirected", [False, True])
@pytest.mark.parametrize("back", [False, True])
@pytest.mark.parametrize("kind", sorted(SHAPES))
def test_levels_and_parents(kind, back, undirected):
    import everythinggraph_gb300 as eg

    n, e, root = layers(SHAPES[kind], np.random.default_rng(5), back)
    n += 37  # isolated
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, e.reshape(-1), undirected=undirected).build(eg.CSR | eg.CSC)
    adj = oracle.build_adj(n, e.reshape(-1), undirected=undirected)
    ref = oracle.bfs_levels(n, adj.out_ptr, adj.out_col, root)
    deg = adj.out_deg().astype(np.int64)
    edges = set(zip(np.repeat(np.arange(n), deg).tolist(), adj.out_col.tolist()))
    for direction in ("push", "auto", "pull"):
        for divisor in (None, 3.0):
            for _ in range(2):
                lv, par, st = g.bfs(root, direction=direction, switch_divisor=divisor, parents=True)
                assert np.array_equal(lv, ref)
                on = np.flatnonzero(ref)
                assert st.reached == len(on) and st.edges_traversed == deg[on].sum()
                assert st.levels == ref.max()
                on = on[on != root]
                assert par[root] == root and np.all(lv[par[on]] == lv[on] - 1)
                assert all((int(p), int(v)) in edges for p, v in zip(par[on], on))
                assert np.all(par[ref == 0] == -1)
    ctx.close()


@pytest.mark.parametrize("n", [20000, 300000])
def test_a_level_of_a_path(n):
    """6.1 and 7.2 us with a list and two grid barriers per level; 2.9 and 2.7
    in the host loop that this replaced."""
    import everythinggraph_gb300 as eg

    ctx = eg.Context(0)
    p = np.random.default_rng(1).permutation(n)
    g = ctx.from_pairs(n, np.stack([p[:-1], p[1:]], 1).astype(np.uint32).reshape(-1), undirected=True).build()
    ms = min(g.bfs(int(p[0]), copy_out=False, host_loop=True)[1].ms for _ in range(3))
    print(ms / n * 1e3)
    assert ms / n * 1e3 < 4.0
    ctx.close()
