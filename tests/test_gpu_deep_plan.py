"""The level plan and the reduction at depths where a level has more than 128
sibling pairs (and, with classes, more segments than the plan keeps at hand):
leaf values and leaf membership of one tree against FP64 sums on the host, and
the batched iterations against the plain ones, class by class.

Tolerances: as for the histogram shapes, a child's sum is off by at most
n * S * 2^-45 per level (S the sum of |x|); the leaf is that over H + lambda,
rounded to FP32.  Batched and plain paths take the same exact sums: only the
FP64 addition order differs, so equal splits and leaves within FP32 rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth,n", [(1, 5000), (8, 30_000), (9, 60_000), (10, 60_000), (12, 90_000)])
def test_leaves(engine, capi, depth, n):
    rng = np.random.default_rng(depth)
    X = rng.standard_normal((n, 13)).astype(np.float32)
    g = rng.standard_normal(n).astype(np.float32)
    h = rng.uniform(0.1, 2.0, n).astype(np.float32)
    ds = engine.upload(X, np.zeros(n, np.float32))
    ds.quantize(255, compat_u8=False)
    t = engine.build_tree(ds, g, h, capi.params(loss="mse", n_estimators=1, max_depth=depth, lambda_l2=1.0,
                                                min_child_weight=0.0))
    assert t["depth"] == depth
    leaf = t["leaf_index"].astype(np.int64)
    bins, want = ds.bins(), np.zeros(n, np.int64)
    for d in range(depth):
        b = bins[t["feature"][d]]
        want = 2 * want + ((b != 255) & (b > t["bin"][d]))
    assert np.array_equal(leaf, want)
    G = np.bincount(leaf, weights=g.astype(np.float64), minlength=1 << depth)
    H = np.bincount(leaf, weights=h.astype(np.float64), minlength=1 << depth)
    tol = depth * n * 2.0 ** -45
    v = np.where(H >= 1e-10, -G / (H + 1.0), 0.0)
    bound = (tol * np.abs(g.astype(np.float64)).sum() + np.abs(v) * tol * h.astype(np.float64).sum()) / (H + 1.0)
    assert (np.abs(t["leaves"] - v) <= bound + np.abs(v) * 2.0 ** -23 + 1e-30).all()
    ds.close()


@pytest.mark.parametrize("classes,depth", [(3, 9), (12, 10)])
def test_batched_equals_plain(engine, capi, classes, depth):
    n = 40_000
    rng = np.random.default_rng(classes)
    X = rng.standard_normal((n, 6)).astype(np.float32)
    y = rng.integers(0, classes, n).astype(np.float32)
    ds = engine.upload(X, y)
    ds.quantize(255, compat_u8=False)
    out = []
    for batched in (1, 0):
        p = capi.params(loss="softmax", n_classes=classes, n_estimators=2, max_depth=depth, min_child_weight=1e-3,
                        batched=batched)
        tr = engine.trainer(ds, p)
        tr.step(2)
        out.append(tr.model().export())
        tr.close()
    a, b = out
    assert np.array_equal(a["depth"], b["depth"]) and a["depth"].max() == depth
    # (entries past a tree's depth are not set)
    for t in range(len(a["depth"])):
        d = a["depth"][t]
        assert np.array_equal(a["feature"][t][:d], b["feature"][t][:d])
        assert np.array_equal(a["bin"][t][:d], b["bin"][t][:d])
        np.testing.assert_allclose(a["leaves"][t], b["leaves"][t], rtol=2.0 ** -21, atol=1e-9)
    ds.close()
