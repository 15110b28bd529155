"""Regular trees grown on the device (depth <= 8) and with the host in every
level (deeper) are the same trees, bit for bit, where the depth limit does not
bind: both sum exactly, so nothing may differ but the header's depth."""
import numpy as np
import pytest

import oracle as O
from datagen import binary_c1

pytestmark = pytest.mark.gpu

FIELDS = ("is_leaf", "left", "right", "feature", "split_bin", "value")


@pytest.mark.parametrize("n,f,msl,bins", [(1, 1, 1, 255), (2, 3, 1, 255), (64, 2, 3, 255), (700, 1, 9, 255),
                                          (3000, 5, 40, 31), (8192, 12, 150, 255), (9001, 40, 170, 255),
                                          (20_000, 3, 400, 255), (33_000, 150, 700, 255)])
@pytest.mark.parametrize("nan", [False, True])
def test_device_and_host_growth_agree(engine, capi, n, f, msl, bins, nan):
    X, y = binary_c1(n, max(f, 2), seed=n + f)
    X = np.ascontiguousarray(X[:, :f])
    if nan:
        X[np.random.default_rng(n).random(X.shape) < 0.05] = np.nan
    if n > 1:
        y[0], y[1] = 0.0, 1.0
    ds = engine.upload(X, y)
    ds.quantize(bins, compat_u8=False)
    trees = []
    for depth in (8, 9):
        p = capi.params(loss="logloss", n_estimators=3, max_depth=depth, learning_rate=0.3, max_bins=bins,
                        min_samples_leaf=msl, min_child_weight=0.0)
        m, st = engine.train_regular(ds, p)
        assert st.n_trees == 3
        trees.append(O.parse_tcat_regular(m.tcat()).trees)
        m.close()
    for a, b in zip(*trees):
        if _depth(b) > 8:  # the limit binds from here on
            break
        for k in FIELDS:
            assert np.array_equal(a[k], b[k]), k
    ds.close()


def _depth(t):
    d = np.zeros(len(t["is_leaf"]), int)
    for i in range(len(d)):  # children follow their parents
        if not t["is_leaf"][i]:
            d[t["left"][i]] = d[t["right"][i]] = d[i] + 1
    return d.max()


@pytest.mark.parametrize("depth", [1, 2, 7, 8])
def test_depth_limit(engine, capi, depth):
    """A binding depth limit: the trees of the limit are the deeper run's, cut."""
    X, y = binary_c1(4000, 6, seed=depth)
    ds = engine.upload(X, y)
    ds.quantize(255, compat_u8=False)
    p = capi.params(loss="logloss", n_estimators=1, max_depth=depth, learning_rate=0.3, min_samples_leaf=20)
    m, _ = engine.train_regular(ds, p)
    t = O.parse_tcat_regular(m.tcat()).trees[0]
    b = O.quantize(X, 255, False)
    pr = np.full(len(y), O.init_prediction("logloss", y), np.float32)
    g, h = O.gradients("logloss", y, pr)
    want = O.build_regular_tree(b, g, h, O.Hyper(loss="logloss", n_estimators=1, max_depth=depth, learning_rate=0.3,
                                                 min_samples_leaf=20), fp32=False)
    for k in ("is_leaf", "left", "right"):
        assert np.array_equal(t[k], want[k])
    sp = ~want["is_leaf"]
    assert np.array_equal(t["feature"][sp], want["feature"][sp])
    assert np.array_equal(t["split_bin"][sp], want["split_bin"][sp])
    # leaves: the sum of at most 4000 terms, each rounded to 2^-46 of the total
    # or better, then FP32
    assert np.allclose(t["value"], want["value"], rtol=2.0 ** -23, atol=1e-9)
    m.close()
    ds.close()
