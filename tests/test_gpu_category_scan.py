"""The ordered encoding's prefix sums over tiles of 4096 sorted positions, at
the edges of warps, tiles and of the 32 tiles that a warp scans at a time:
bit-exact against the oracle (integer labels add exactly in any order)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 33, 511, 513, 4095, 4096, 4097, 8193, 32 * 4096, 32 * 4096 + 1, 33 * 4096 + 517])
def test_ordered_prefix(engine, n):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 3)).astype(np.float32)
    X[:, 0] = rng.integers(0, 5, n)
    X[:, 2] = rng.integers(0, max(2, n // 7), n)
    X[rng.random(n) < 0.1, 0] = np.nan
    X[rng.random(n) < 0.02, 2] = np.nan
    y = rng.integers(-3, 4, n).astype(np.float32)
    order = rng.permutation(n).astype(np.uint32)
    want, tab, _ = O.ordered_ts(X, y, [0, 2], order, 1.0)
    ds = engine.upload(X, y)
    ds.encode_categorical([0, 2], "ordered", prior_weight=1.0, order=order)
    assert np.array_equal(ds.features().view(np.uint32), np.ascontiguousarray(want, np.float32).view(np.uint32))
    for j in (0, 2):
        keys, vals = ds.category_table(j)
        assert np.array_equal(keys, tab[j][0])
        assert np.array_equal(vals.view(np.uint32), np.asarray(tab[j][1], np.float32).view(np.uint32))
    ds.close()
