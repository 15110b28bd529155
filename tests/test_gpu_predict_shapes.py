"""The tile prediction kernel over tile remainders, depths, class counts and
model forms against an FP64 walk of the same arrays on the host.

Tolerance: every row sums at most T leaves in FP32 in some order, so the error
is at most T * 2^-24 of the sum of |leaf| (plus the base), and the transforms
have slopes of at most 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(engine, capi, seed, T, D, F, K, wide=False):
    """depth in [max(0, D-2), D]; thresholds from few values per feature, or
    (`wide`) so many that the columns of bins take 128-row tiles or none."""
    rng = np.random.default_rng(seed)
    depth = rng.integers(max(0, D - 2), D + 1, T).astype(np.int32)
    thr = rng.standard_normal((T, D)).astype(np.float32)
    if not wide:
        thr = np.round(thr * 8) / 8
    a = dict(depth=depth, feature=rng.integers(0, F, (T, D)).astype(np.uint16), threshold=thr.astype(np.float32),
             leaves=(0.1 * rng.standard_normal((T, 1 << D))).astype(np.float32), weights=np.full(T, 0.1, np.float32))
    info = capi.ModelInfo(T, K, D, F, 1 if K > 1 else 0, 0.0 if K > 1 else 0.3, 0.1, 1.0)
    return engine.import_model(info, a), a


def _walk64(a, X, K, base):
    T = len(a["depth"])
    out = np.full((len(X), K), float(base))
    mag = np.full((len(X), K), abs(float(base)))
    for t in range(T):
        idx = np.zeros(len(X), np.int64)
        for d in range(a["depth"][t]):
            with np.errstate(invalid="ignore"):
                idx = 2 * idx + (X[:, a["feature"][t, d]] >= a["threshold"][t, d])
        v = a["leaves"][t, idx].astype(np.float64) * float(a["weights"][t])
        out[:, t % K] += v
        mag[:, t % K] += np.abs(v)
    return out, mag


CASES = [(T, D, F, K) for T, D, F, K in [
    (1, 1, 1, 1), (17, 2, 3, 1), (33, 3, 7, 1), (100, 4, 100, 1), (65, 5, 31, 1), (130, 6, 30, 1), (40, 7, 12, 1),
    (200, 8, 101, 1), (31, 9, 20, 1), (64, 10, 64, 1), (9, 12, 5, 1), (3, 3, 4, 3), (2, 4, 4, 3), (250, 6, 50, 10),
    (35, 5, 9, 5), (48, 7, 21, 16), (30, 1, 6, 4)]]


@pytest.mark.parametrize("T,D,F,K", CASES)
def test_depths_and_classes(engine, capi, T, D, F, K):
    m, a = _model(engine, capi, T + D + F + K, T, D, F, K)
    rng = np.random.default_rng(F)
    for n in (65, 127, 128, 129, 255, 256, 257, 1000):
        X = np.round(rng.standard_normal((n, F)) * 8).astype(np.float32) / 8  # on the borders often
        X[rng.random((n, F)) < 0.05] = np.nan
        want, mag = _walk64(a, X, K, m.info.base_prediction)
        assert np.abs(m.predict(X, "raw") - want).max() <= (T + 8) * 2.0 ** -24 * mag.max() + 1e-30
    if K > 1:
        e = np.exp(want - want.max(1, keepdims=True))
        p = e / e.sum(1, keepdims=True)
        assert np.abs(m.predict(X, "softmax") - p).max() <= (T + 8) * 2.0 ** -23 * mag.max() + 2.0 ** -20
    m.close()


def test_tile_sizes_give_the_same_bits(engine, capi):
    """A row's sum does not depend on the launch: 128-row tiles (few rows) and
    256-row ones (many) agree bit for bit, one class and several."""
    import torch

    for K in (1, 4):
        m, _ = _model(engine, capi, 11, 120, 6, 40, K)
        X = torch.randn(120_000, 40, device="cuda")
        big = torch.empty(120_000, K, device="cuda")
        m.predict_device(X.data_ptr(), 120_000, 40, big.data_ptr(), "raw", 1)
        for r0, n in ((0, 3000), (777, 129), (119_000, 1000)):
            o = torch.empty(n, K, device="cuda")
            m.predict_device(X[r0:].data_ptr(), n, 40, o.data_ptr(), "raw", 1)
            assert torch.equal(o, big[r0:r0 + n])
        torch.cuda.synchronize()
        m.close()


@pytest.mark.parametrize("F,T", [(240, 1800), (340, 1400), (340, 6000), (330, 200)])
def test_many_borders(engine, capi, F, T):
    """Models whose bin columns fit only 128-row tiles, and ones without a
    binned form (more virtual features, or more borders, than fit)."""
    m, a = _model(engine, capi, F + T, T, 6, F, 1, wide=True)
    X = np.random.default_rng(1).standard_normal((300, F)).astype(np.float32)
    want, mag = _walk64(a, X, 1, m.info.base_prediction)
    assert np.abs(m.predict(X, "raw") - want).max() <= (T + 8) * 2.0 ** -24 * mag.max()
    m.close()
