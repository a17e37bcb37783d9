"""SpMV over rows that end, begin and run on at the tiles' edges (empty rows,
rows of one entry, rows over many tiles), with integer values so that every
order of the sums gives the same numbers; and the FP64 products bit for bit,
subnormals, zeros, infinities and NaN among them."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 127, 128, 129, 1024, 5000, 300001, 778241, 1556481, 3112961, 6225921])
@pytest.mark.parametrize("hub", [0.0, 0.4])
def test_integer_sums(m, hub):
    import everythinggraph_gb300 as eg

    n = max(2, m // 9)
    rng = np.random.default_rng(m)
    pairs = rng.integers(0, n, (m, 2)).astype(np.uint32)
    pairs[rng.random(m) < hub, 1] = n // 3  # one row over many tiles
    adj = oracle.build_adj(n, pairs.reshape(-1))
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, pairs.reshape(-1)).build(eg.CSR | eg.CSC)
    x = rng.integers(0, 4, n)  # sums below 2^24: exact in fp32
    ref = np.bincount(pairs[:, 1], weights=x[pairs[:, 0]], minlength=n)
    for kind in ("f32", "f32_comp", "f64"):
        y, _ = g.spmv(x.astype(np.float32), kind=kind, unit_values=True)
        assert np.array_equal(y, ref), kind
    x = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    y, _ = g.spmv(x, kind="u32_pull")
    assert np.array_equal(y, oracle.spmv_u32(n, adj.in_ptr, adj.in_col, x, 0))
    ctx.close()


@pytest.mark.parametrize("unit", [False, True])
def test_f64_products(unit):
    import everythinggraph_gb300 as eg

    n = 1 << 16
    rng = np.random.default_rng(5)
    src = rng.permutation(n).astype(np.uint32)  # one entry per row
    ctx = eg.Context(0)
    g = ctx.from_pairs(n, np.stack([src, np.arange(n, dtype=np.uint32)], 1).reshape(-1)).build(eg.CSR | eg.CSC)
    x = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32).view(np.float32)  # every exponent and sign
    x[:8] = [0.0, -0.0, np.inf, -np.inf, np.nan, np.float32(1e-45), np.finfo(np.float32).max, np.finfo(np.float32).tiny]
    vals, _ = g.spmv(np.ones(n, np.float32), kind="f32", value_seed=7, unit_values=unit)
    y, _ = g.spmv(x, kind="f64", value_seed=7, unit_values=unit)
    with np.errstate(invalid="ignore"):
        ref = vals.astype(np.float64) * x[src].astype(np.float64) + 0.0  # a row's sum starts at +0
    assert np.array_equal(np.isnan(y), np.isnan(ref))
    ok = ~np.isnan(ref)
    assert np.array_equal(y[ok].view(np.uint64), ref[ok].view(np.uint64))
    ctx.close()
