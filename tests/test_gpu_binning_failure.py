"""A binning that fails half-way leaves a dataset without bins, not one whose old
bins are gone: what needs bins refuses it until it is binned again."""
import numpy as np
import pytest

from datagen import binary_c1

pytestmark = pytest.mark.gpu


def test_failed_held_out_binning(capi):
    eng = capi.Engine(0)
    X, y = binary_c1(2000, 8, seed=1)
    ref, ds = eng.upload(X, y), eng.upload(X[::-1].copy(), y[::-1].copy())
    ref.quantize(255)
    ds.quantize(63)
    p = capi.params(loss="logloss", n_estimators=2, max_depth=3)
    eng.fail_next_allocs(1)
    with pytest.raises(capi.TCError):
        ds.apply_bins(ref)
    for call in (lambda: eng.train(ds, p), lambda: eng.train_regular(ds, p), ds.bins,
                 lambda: ref.apply_bins(ds)):
        with pytest.raises(capi.TCError):
            call()
    ds.apply_bins(ref)
    assert np.array_equal(ds.bins(), ref.bins()[:, ::-1])
    eng.train(ds, p)[0].close()
    # a re-binning whose first scratch buffer fails keeps the bins
    eng.fail_next_allocs(1)
    with pytest.raises(capi.TCError):
        ds.quantize(31)
    assert np.array_equal(ds.bins(), ref.bins()[:, ::-1])
    ds.close()
    ref.close()
    eng.close()
