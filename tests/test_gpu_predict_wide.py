"""The 256-row tiles of the prediction kernel, which launches of more 128-row
tiles than the device has multiprocessors take: every depth and several class
counts against an FP64 walk, over the remainders of the last tile.

Tolerance: a row sums at most T leaves in FP32 in some order, so the error is at
most T * 2^-24 of the sum of |leaf| (plus the base), and the transforms have
slopes of at most 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(engine, capi, seed, T, D, F, K, coarse=True):
    rng = np.random.default_rng(seed)
    thr = rng.standard_normal((T, D)).astype(np.float32)
    if coarse:
        thr = np.round(thr * 8) / np.float32(8)
    a = dict(depth=rng.integers(max(0, D - 2), D + 1, T).astype(np.int32),
             feature=rng.integers(0, F, (T, D)).astype(np.uint16), threshold=thr,
             leaves=(0.1 * rng.standard_normal((T, 1 << D))).astype(np.float32), weights=np.full(T, 0.1, np.float32))
    info = capi.ModelInfo(T, K, D, F, 1 if K > 1 else 0, 0.0 if K > 1 else 0.3, 0.1, 1.0)
    return engine.import_model(info, a), a


def _walk64(a, X, K, base):
    out = np.full((len(X), K), float(base))
    mag = np.full((len(X), K), abs(float(base)))
    for t in range(len(a["depth"])):
        idx = np.zeros(len(X), np.int64)
        for d in range(a["depth"][t]):
            with np.errstate(invalid="ignore"):
                idx = 2 * idx + (X[:, a["feature"][t, d]] >= a["threshold"][t, d])
        v = a["leaves"][t, idx].astype(np.float64) * float(a["weights"][t])
        out[:, t % K] += v
        mag[:, t % K] += np.abs(v)
    return out, mag


def _check(m, a, F, K, T):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    half = (sms + 2) // 2 * 2  # 128-row tiles: an even count, a little more than one each
    rng = np.random.default_rng(F)
    n_max = (half + 1) * 128
    X = np.round(rng.standard_normal((n_max, F)) * 8).astype(np.float32) / 8  # on the borders often
    X[rng.random((n_max, F)) < 0.05] = np.nan
    dX = torch.from_numpy(X).cuda()
    base = m.info.base_prediction
    want, mag = {}, 0.0
    rows = np.unique(np.concatenate([np.arange(300), np.arange((half - 2) * 128 - 3, n_max),
                                     rng.integers(0, n_max, 200)]))
    want, mag = _walk64(a, X[rows], K, base)
    # the last 256-row tile full, one short, of 129 rows; then a 128-row one of 1, 127 and 128 rows
    for n in (half * 128, half * 128 - 1, half * 128 - 127, half * 128 + 1, half * 128 + 127, n_max):
        out = torch.full((n, K), -7.0, device="cuda")
        m.predict_device(dX.data_ptr(), n, F, out.data_ptr(), "raw", torch.cuda.current_stream().cuda_stream or 1)
        got = out.cpu().numpy()
        at = rows < n
        assert np.abs(got[rows[at]] - want[at]).max() <= (T + 8) * 2.0 ** -24 * mag.max() + 1e-30, n
    if K > 1:
        z = want - want.max(1, keepdims=True)
        p = np.exp(z) / np.exp(z).sum(1, keepdims=True)
        out = torch.empty((n_max, K), device="cuda")
        m.predict_device(dX.data_ptr(), n_max, F, out.data_ptr(), "softmax", 1)
        torch.cuda.synchronize()
        assert np.abs(out.cpu().numpy()[rows] - p).max() <= (T + 8) * 2.0 ** -23 * mag.max() + 2.0 ** -20


@pytest.mark.parametrize("T,D,F,K", [
    (17, 1, 3, 1), (33, 2, 7, 1), (100, 3, 101, 1), (65, 4, 31, 1), (130, 5, 30, 1), (250, 6, 40, 1), (40, 7, 12, 1),
    (200, 8, 64, 1), (31, 9, 20, 1), (64, 10, 50, 1), (48, 11, 9, 1), (20, 12, 5, 1), (37, 13, 16, 1), (2, 4, 4, 3),
    (200, 6, 50, 10), (35, 5, 9, 5), (48, 7, 21, 16), (50, 13, 8, 3)])
def test_depths_and_classes(engine, capi, T, D, F, K):
    m, a = _model(engine, capi, T + D + F + K, T, D, F, K)
    _check(m, a, F, K, T)
    m.close()


def test_without_a_binned_form(engine, capi):
    """More than 512 virtual features of 127 thresholds each: the float walk."""
    T, D, F = 8000, 10, 100
    m, a = _model(engine, capi, 1, T, D, F, 1, coarse=False)
    used = np.arange(D)[None, :] < a["depth"][:, None]
    assert sum(-(-np.unique(a["threshold"][used & (a["feature"] == j)]).size // 127) for j in range(F)) > 512
    _check(m, a, F, 1, T)
    m.close()
