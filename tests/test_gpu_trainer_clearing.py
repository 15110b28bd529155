"""A trainer's accumulators and completion counters are zero before its first
kernel, whatever their blocks held before, however large the accumulators are
and whatever the default stream is doing: the same model as a fresh context's,
bit for bit."""
import numpy as np
import pytest

from datagen import binary_c1

pytestmark = pytest.mark.gpu

ARRAYS = ("depth", "feature", "bin", "threshold", "gain", "leaves")


def _table(n, f, seed):
    X, y = binary_c1(n, f, seed=seed)
    rng = np.random.default_rng(seed + 1)
    return X, y, rng.standard_normal(n).astype(np.float32), rng.uniform(0.05, 1.0, n).astype(np.float32)


def _results(eng, capi, table, depth, busy=None):
    """A fit (two trees, so no tuning) and a tree of given gradients."""
    X, y, g, h = table
    ds = eng.upload(X, y)
    ds.quantize(255)
    p = capi.params(loss="logloss", n_estimators=2, max_depth=depth, min_child_weight=0.0)
    if busy:
        busy()
    tr = eng.trainer(ds, p)
    tr.step(2)
    m = tr.model()
    tr.close()
    if busy:
        busy()
    t = eng.build_tree(ds, g, h, p, want_hist=True)
    e = m.export()
    m.close()
    ds.close()
    return [e[k] for k in ARRAYS] + [t[k] for k in ("feature", "bin", "gain", "second", "leaves", "leaf_index",
                                                    "root_hist")]


def _fresh(capi, *a):
    eng = capi.Engine(0)
    out = _results(eng, capi, *a)
    eng.close()
    return out


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def _dirty(eng, capi):
    """Leaves kept blocks of several sizes behind, filled with a fit's data."""
    for n, f, d in ((4000, 30, 6), (900, 90, 7), (20_000, 12, 4), (300, 5, 3)):
        _results(eng, capi, _table(n, f, n), d)


def test_large_accumulators(capi):
    """Depth 12 and 200 features: three buffers of 1.6 GiB, whose clearing takes
    longer than the launches behind it."""
    table = _table(1500, 200, 3)
    want = _fresh(capi, table, 12)
    eng = capi.Engine(0)
    _dirty(eng, capi)
    for _ in range(2):
        assert _same(_results(eng, capi, table, 12), want)
    eng.close()


def test_busy_default_stream(capi):
    """Work queued on the default stream (torch's) delays nothing a trainer
    needs, and nothing of a trainer runs behind it."""
    import torch

    table = _table(6000, 40, 5)
    want = _fresh(capi, table, 6)
    eng = capi.Engine(0)
    _dirty(eng, capi)

    def busy():
        torch.cuda._sleep(200_000_000)  # about 0.1 s

    for _ in range(2):
        assert _same(_results(eng, capi, table, 6, busy), want)
        torch.cuda.synchronize()
        assert _same(_results(eng, capi, table, 6), want)
    eng.close()


def test_first_small_request_behind_a_busy_default_stream(capi):
    """The small-request path's counters are cleared on the stream that uses
    them: the first request of a context is answered in full."""
    import torch

    rng = np.random.default_rng(9)
    T, D, F = 600, 6, 20
    a = dict(depth=np.full(T, D, np.int32), feature=rng.integers(0, F, (T, D)).astype(np.uint16),
             threshold=rng.standard_normal((T, D)).astype(np.float32),
             leaves=rng.standard_normal((T, 1 << D)).astype(np.float32), weights=np.full(T, 0.1, np.float32))
    info = capi.ModelInfo(T, 1, D, F, 0, 0.3, 0.1, 1.0)
    X = rng.standard_normal((64, F)).astype(np.float32)
    eng = capi.Engine(0)
    m = eng.import_model(info, a)
    eng.set_latency_worker(False)
    torch.cuda._sleep(200_000_000)
    first = m.predict(X, "raw")
    torch.cuda.synchronize()
    for _ in range(2):
        assert np.array_equal(m.predict(X, "raw"), first)
    wide = m.predict(np.concatenate([X, X]), "raw")[:64]  # the tile kernel
    assert np.abs(first - wide).max() <= 2 * T * 2.0 ** -24 * (0.3 + 0.1 * np.abs(a["leaves"]).max(1).sum())
    m.close()
    eng.close()
