"""WCC on graphs that reach each of its steps (one tree from the seeds, rounds
of hooks, hooks with finds; directed and undirected; no CSC), against the
oracle's labels."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def shape(kind, n, rng):
    v = np.arange(n)
    if kind == "path":  # one long chain through shuffled ids
        p = rng.permutation(n)
        return np.stack([p[:-1], p[1:]], 1)
    if kind == "high hubs":  # stars around the largest ids, joined by one edge
        h = n - 1 - rng.integers(0, 3, n)
        return np.concatenate([np.stack([v, h], 1), [[n - 1, n - 2]]])
    if kind == "halves":  # two random components of equal size
        e = rng.integers(0, n // 2, (4 * n, 2))
        return e * 2 + rng.integers(0, 2, 4 * n)[:, None]
    if kind == "pairs":
        return np.stack([v[: n // 2 * 2 : 2], v[1 : n // 2 * 2 : 2]], 1)
    if kind == "sparse":
        return rng.integers(0, n, (n, 2))
    if kind == "loops":
        return np.stack([v[::3], v[::3]], 1)
    return rng.integers(0, n, (8 * n, 2))  # uniform


@pytest.mark.parametrize("undirected,csc", [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize("n", [1023, 1024, 1027, 70001])
@pytest.mark.parametrize("kind", ["path", "high hubs", "halves", "pairs", "sparse", "loops", "uniform"])
def test_labels(kind, n, undirected, csc):
    import everythinggraph_gb300 as eg

    pairs = shape(kind, n, np.random.default_rng(n)).astype(np.uint32)
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs.reshape(-1), undirected=undirected).build(eg.CSR | (eg.CSC if csc else 0))
    ref = oracle.wcc(n, pairs.reshape(-1))
    for _ in range(2):
        lab, st = g.wcc()
        assert np.array_equal(lab, ref)
        assert st.components == len(np.unique(ref))
    ctx.close()
