"""Models without a binned form (more than 512 virtual features of 127 borders,
or more borders than fit shared memory): the float walk's rows, alone and in the
mix with models of other shapes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(engine, capi, T, D, F, K=1, levels=0):
    rng = np.random.default_rng(T + D + F + K)
    feature = rng.integers(0, F, (T, D)).astype(np.uint16)
    thr = rng.standard_normal((T, D)).astype(np.float32)
    if levels:
        thr = np.round(thr * levels) / np.float32(levels)
    a = dict(depth=rng.integers(max(1, D - 2), D + 1, T).astype(np.int32), feature=feature, threshold=thr,
             leaves=rng.standard_normal((T, 1 << D)).astype(np.float32), weights=np.full(T, 0.1, np.float32))
    return engine.import_model(capi.ModelInfo(T, K, D, F, 1 if K > 1 else 0, 0.0, 0.1, 1.0), a), a


def _virtual_features(a, F):
    """How many 127-border virtual features the model's thresholds make."""
    used = np.arange(a["threshold"].shape[1])[None, :] < a["depth"][:, None]
    return sum(-(-np.unique(a["threshold"][used & (a["feature"] == j)]).size // 127) for j in range(F))


def _walk64(a, X, K):
    out = np.zeros((len(X), K))
    mag = np.zeros((len(X), K))
    for t in range(len(a["depth"])):
        idx = np.zeros(len(X), np.int64)
        for d in range(a["depth"][t]):
            with np.errstate(invalid="ignore"):
                idx = 2 * idx + (X[:, a["feature"][t, d]] >= a["threshold"][t, d])
        v = a["leaves"][t, idx].astype(np.float64) * float(a["weights"][t])
        out[:, t % K] += v
        mag[:, t % K] += np.abs(v)
    return out, mag


@pytest.mark.parametrize("T,D,F,K", [(8000, 10, 100, 1), (9000, 9, 90, 3), (6200, 13, 100, 1)])
def test_same_bits_alone_and_in_the_mix(engine, capi, T, D, F, K):
    """The same rows alone, and served beside deeper and shallower models with
    which the launch's chunks of trees are other ones."""
    m, a = _model(engine, capi, T, D, F, K)
    assert _virtual_features(a, F) > 512
    rng = np.random.default_rng(1)
    X = rng.standard_normal((420, F)).astype(np.float32)
    X[rng.random(X.shape) < 0.03] = np.nan
    want, mag = _walk64(a, X, K)
    others = [_model(engine, capi, 50, 13, F, levels=8)[0], _model(engine, capi, 40, 3, F, levels=8)[0],
              _model(engine, capi, 1200, 6, F)[0]]
    alone = {n: m.predict(X[:n], "raw") for n in (65, 70, 128, 129, 255, 420)}
    for n, got in alone.items():
        assert np.abs(got - want[:n]).max() <= (T + 8) * 2.0 ** -24 * mag.max()
    for mix in ([others[0]], [others[1]], [others[2]], others):
        srv = capi.Server(engine, staging_bytes=0, max_batch_rows=16384, coalesce=True, max_inflight=2)
        mid = srv.add_model(m)
        oid = [srv.add_model(o) for o in mix]
        outs, tickets, keep = [], [], []
        for n in alone:
            o = np.zeros((n, K), np.float32)
            outs.append((n, o))
            tickets.append(srv.submit(mid, X[:n], o, "raw"))
            for i in oid:
                p = np.zeros((200, 1), np.float32)
                keep.append(p)
                tickets.append(srv.submit(i, X[:200], p, "raw"))
        for t in tickets:
            assert srv.poll(t, 10_000_000)[0]
        for n, o in outs:
            assert np.array_equal(o, alone[n]), (len(mix), n)
        srv.close()
    for o in others + [m]:
        o.close()
