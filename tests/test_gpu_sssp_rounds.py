"""Single-source SSSP on graphs that reach each branch of its round order,
against the oracle: every weight rule, weights of 0 and up to 2^32 - 1, chains
longer than the bucket range, hubs, sizes around the 32-vertex words and the
8192-vertex groups, and enough edges for a round to hold only part of the
active vertices (more than 2^22)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def graph(n, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "chain":
        p = np.stack([np.arange(n - 1), np.arange(1, n)], 1)
    elif kind == "hub":
        p = np.concatenate([np.stack([np.zeros(5 * n, np.int64), rng.integers(0, n, 5 * n)], 1),
                            np.stack([rng.integers(0, n, 5 * n), np.zeros(5 * n, np.int64)], 1)])
    else:
        p = rng.integers(0, n, (8 * n, 2))
    return p.astype(np.uint32)


def distances(n, pairs, w, root, f32):
    """Bellman-Ford to the fixed point in the rule's arithmetic."""
    dt = np.float32 if f32 else np.uint64
    top = np.float32(np.inf) if f32 else np.uint64(0xFFFFFFFE)
    d = np.full(n, top, dtype=dt)
    d[root] = 0
    s, t = pairs[:, 0], pairs[:, 1]
    for _ in range(n + 1):
        nd = (d[s] + w.astype(dt)).astype(dt)
        if not f32:
            nd = np.where(d[s] == top, top, np.minimum(nd, top))
        e = d.copy()
        np.minimum.at(e, t, nd)
        if np.array_equal(e, d):
            break
        d = e
    return d if f32 else d.astype(np.uint32)


@pytest.mark.parametrize("kind", ["chain", "hub", "random"])
@pytest.mark.parametrize("n", [1, 2, 33, 700])
@pytest.mark.parametrize("rule", ["ref", "unit", "hash", "wide", "zero", "f32"])
def test_rounds_reach_the_fixed_point(n, kind, rule):
    import everythinggraph_gb300 as eg

    pairs = graph(n, kind, n)
    lo, hi = {"wide": (1 << 28, 0xFFFFFFFF), "zero": (0, 1)}.get(rule, (1, 255))
    w = eg.weights("hash" if rule in ("wide", "zero") else rule, seed=6, lo=lo, hi=hi)
    s, t = pairs[:, 0], pairs[:, 1]
    wt = {"ref": lambda: s % 10 + t % 10, "unit": lambda: np.ones(len(s), np.uint32),
          "f32": lambda: oracle.hash_weights_f32(s, t, 6)}.get(rule, lambda: oracle.hash_weights(s, t, 6, lo, hi))()
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs.reshape(-1)).build(eg.CSR)
    for root in {0, n // 2}:
        d, st = g.sssp(root, w)
        ref = distances(n, pairs, wt, root, rule == "f32")
        assert np.array_equal(d.view(np.uint32), ref.view(np.uint32))
        assert st.reached == int((ref != (np.inf if rule == "f32" else 0xFFFFFFFE)).sum())
    ctx.close()


@pytest.mark.parametrize("n", [8191, 8193, 400001])
def test_partial_rounds(n):
    import everythinggraph_gb300 as eg

    rng = np.random.default_rng(n)
    m = 9 << 20  # a round holds 2^22 edges at most of the random lists
    pairs = (rng.random((m, 2)) ** 2 * n).astype(np.uint32)
    adj = oracle.build_adj(n, pairs.reshape(-1))
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs.reshape(-1)).build(eg.CSR)
    rows = np.repeat(np.arange(n, dtype=np.uint32), np.diff(adj.out_ptr.astype(np.int64)))
    wt = oracle.hash_weights(rows, adj.out_col, 6, 1, 255)
    for root in (0, n - 1):
        d, _ = g.sssp(root, eg.weights("hash", seed=6, lo=1, hi=255))
        assert np.array_equal(d, oracle.sssp(n, adj.out_ptr, adj.out_col, wt, root))
    ctx.close()


@pytest.mark.parametrize("k", [2, 3, 33, 64, 70])
@pytest.mark.parametrize("kind,n", [("chain", 97), ("hub", 500), ("random", 700)])
@pytest.mark.parametrize("rule", ["ref", "zero", "wide", "f32"])
def test_batched_rounds_reach_the_fixed_point(rule, kind, n, k):
    """Batch sizes off the words of 32 and the rows of 4 sources."""
    import everythinggraph_gb300 as eg

    pairs = graph(n, kind, n + 1)
    lo, hi = {"wide": (1 << 28, 0xFFFFFFFF), "zero": (0, 1)}.get(rule, (1, 255))
    w = eg.weights("hash" if rule in ("wide", "zero") else rule, seed=6, lo=lo, hi=hi)
    s, t = pairs[:, 0], pairs[:, 1]
    wt = {"ref": lambda: s % 10 + t % 10,
          "f32": lambda: oracle.hash_weights_f32(s, t, 6)}.get(rule, lambda: oracle.hash_weights(s, t, 6, lo, hi))()
    roots = np.random.default_rng(k).integers(0, n, k).astype(np.uint32)
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs.reshape(-1)).build(eg.CSR)
    d, _ = g.sssp_multi(roots, w)
    seen = {}
    for i, r in enumerate(roots):
        r = int(r)
        if r not in seen:
            seen[r] = distances(n, pairs, wt, r, rule == "f32").view(np.uint32)
        assert np.array_equal(d[i].view(np.uint32), seen[r]), i
    ctx.close()


@pytest.mark.parametrize("n", [1023, 150001])
def test_batched_partial_rounds(n):
    import everythinggraph_gb300 as eg

    rng = np.random.default_rng(n)
    m = 3 << 20  # more places than a round's 2^21 with two words of sources
    pairs = (rng.random((m, 2)) ** 2 * n).astype(np.uint32)
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs.reshape(-1)).build(eg.CSR)
    roots = rng.integers(0, n, 40).astype(np.uint32)
    w = eg.weights("hash", seed=6, lo=1, hi=255)
    d, _ = g.sssp_multi(roots, w)
    for i in range(0, 40, 3):
        one, _ = g.sssp(int(roots[i]), w)
        assert np.array_equal(d[i], one)
    ctx.close()
