"""Sort, edge pick and bin assignment at the edges of their tiles: bins, edges
and edge counts bit-exact against the oracle, and the sort's payload through
the categorical encoding."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _table(n, f, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, f)).astype(np.float32)
    X[:, ::3] = np.round(X[:, ::3] * 4) / 4  # duplicates
    X[rng.random((n, f)) < 0.02] = np.nan
    for v in (0.0, -0.0, np.inf, -np.inf, 1e-42, -1e-42):
        X[rng.random((n, f)) < 0.01] = v
    if f > 3:
        X[:, 3] = np.nan  # no value at all
    if f > 4:
        X[:, 4] = 2.5     # one value
    return X


@pytest.mark.parametrize("n,f", [(1, 1), (2, 5), (31, 33), (64, 4), (65, 8), (257, 32), (1023, 7), (4095, 3), (4096, 6),
                                 (4097, 40), (8193, 2), (20_001, 17), (300_007, 3), (40_000, 65)])
@pytest.mark.parametrize("max_bins,compat", [(255, True), (255, False), (16, False)])
def test_bins_against_the_oracle(engine, n, f, max_bins, compat):
    X = _table(n, f, n + f)
    ds = engine.upload(X)
    edges, ne = ds.quantize(max_bins, compat_u8=compat)
    want = O.quantize(X, max_bins, compat)
    assert np.array_equal(ne, want.n_edges)
    assert np.array_equal(edges, want.edges)  # by value: the device folds -0.0 onto +0.0, the oracle keeps either
    # NaN rows hold bin 255 on the device whatever max_bins is (the reference: max_bins)
    assert np.array_equal(ds.bins(), np.where(np.isnan(X).T, np.uint8(255), want.bins))
    ds.close()


@pytest.mark.parametrize("n,card", [(1, 3), (5, 2), (4095, 300), (4096, 70_000), (4097, 1), (50_001, 1000)])
def test_sorted_payload(engine, n, card):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 3)).astype(np.float32)
    X[:, 1] = rng.integers(0, card, n)
    X[rng.random(n) < 0.05, 1] = np.nan
    y = rng.integers(0, 2, n).astype(np.float32)
    order = rng.permutation(n).astype(np.uint32)
    want, tab, _ = O.ordered_ts(X, y, [1], order)
    ds = engine.upload(X, y)
    ds.encode_categorical([1], "ordered", order=order)
    assert np.array_equal(ds.features().view(np.uint32), want.view(np.uint32))
    keys, vals = ds.category_table(1)
    assert np.array_equal(keys, tab[1][0]) and np.array_equal(vals.view(np.uint32), tab[1][1].view(np.uint32))
    ds.quantize(255)
    assert np.array_equal(ds.bins(), O.quantize_ts(want, [1]).bins)
    ds.close()
