"""The histogram kernel over feature-group widths, row counts and bin
counts: root histograms and, through the leaf values, the gathered levels,
against FP64 sums on the host.

Tolerance.  A row is rounded to the item's fixed-point grid 2^-e with
2^e * S + rows / 2 < 2^46 and e the largest such, S the item's sum of |x|, so
one row is off by at most 2^-(e+1) <= S * 2^-46 (1 + a rounding of the
margin), a bin of m rows by m * S * 2^-46 and every bin by at most
n * S * 2^-45 over all items; the FP64 additions add n * 2^-52 of S at most.
Leaves are that sum over H + lambda in FP32: 2^-23 relative on top.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bins_to_hist(bins, g, h):
    f, n = bins.shape
    out = np.zeros((f, 256, 2))
    for j in range(f):
        out[j, :, 0] = np.bincount(bins[j], weights=g.astype(np.float64), minlength=256)
        out[j, :, 1] = np.bincount(bins[j], weights=h.astype(np.float64), minlength=256)
    return out


def _table(n, f, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, f)).astype(np.float32)
    X[:, ::3] = np.round(X[:, ::3] * 2) / 2  # few bins
    if f > 2:
        X[rng.random(n) < 0.1, 2] = np.nan
    if f > 4:
        X[:, 4] = 1.0  # constant
    return X


@pytest.mark.parametrize("n,f", [(1, 1), (31, 4), (32, 5), (33, 8), (1000, 9), (1025, 16), (4099, 17), (4096, 20),
                                 (5000, 24), (3001, 25), (2049, 32), (2000, 33), (1999, 50), (70_001, 37),
                                 (140_000, 3)])
def test_given_gradients(engine, capi, n, f):
    rng = np.random.default_rng(n * 131 + f)
    X = _table(n, f, n + f)
    g = (rng.standard_normal(n) * 10.0 ** rng.uniform(-3, 1, n)).astype(np.float32)
    h = rng.uniform(1e-6, 2.0, n).astype(np.float32)
    ds = engine.upload(X, np.zeros(n, np.float32))
    ds.quantize(255, compat_u8=False)
    bins = ds.bins()
    p = capi.params(loss="mse", n_estimators=1, max_depth=4, lambda_l2=1.0, min_child_weight=0.0)
    t = engine.build_tree(ds, g, h, p, want_hist=True)
    sg, sh = np.abs(g).astype(np.float64).sum(), h.astype(np.float64).sum()
    tol = n * 2.0 ** -45
    if t["depth"] > 0:  # a tree that stops at the root builds no histogram
        want = _bins_to_hist(bins, g, h)
        assert np.abs(t["root_hist"][..., 0] - want[..., 0]).max() <= tol * sg
        assert np.abs(t["root_hist"][..., 1] - want[..., 1]).max() <= tol * sh
    leaf = t["leaf_index"].astype(np.int64)
    for q in range(1 << t["depth"]):
        m = leaf == q
        G, H = g[m].astype(np.float64).sum(), h[m].astype(np.float64).sum()
        if H >= 1e-9:
            want = -G / (H + 1.0)
            # children by subtraction: the error of a bin of the root, over every level
            err = 8 * tol * (sg + abs(want) * sh) / (H + 1.0) + 2.0 ** -23 * abs(want)
            assert abs(float(t["leaves"][q]) - want) <= err + 1e-30
    ds.close()


@pytest.mark.parametrize("n,f", [(5, 1), (100, 4), (1000, 20), (3000, 36), (70_003, 18)])
def test_counted_hessian(engine, capi, n, f):
    """MSE on every row: the kernel counts rows instead of adding hessians."""
    X = _table(n, f, 7 * n + f)
    y = (np.nan_to_num(X).sum(1) + np.random.default_rng(n).standard_normal(n)).astype(np.float32)
    ds = engine.upload(X, y)
    ds.quantize(255, compat_u8=False)
    p = capi.params(loss="mse", n_estimators=1, max_depth=3, learning_rate=1.0, lambda_l2=0.5, min_child_weight=0.0)
    m, _ = engine.train(ds, p)
    e = m.export()
    base = np.float32(m.info.base_prediction)
    g = (np.float32(2.0) * (base - y)).astype(np.float64)
    leaf = np.zeros(n, np.int64)
    for d in range(e["depth"][0]):
        x = X[:, e["feature"][0, d]]
        leaf = 2 * leaf + (x >= e["threshold"][0, d])
    tol = n * 2.0 ** -45 * np.abs(g).sum()
    for q in range(1 << e["depth"][0]):
        c = int((leaf == q).sum())
        if c:
            want = -g[leaf == q].sum() / (2.0 * c + 0.5)
            assert abs(float(e["leaves"][0, q]) - want) <= 8 * tol / (2.0 * c) + 2.0 ** -23 * abs(want) + 1e-30
    m.close()
    ds.close()
