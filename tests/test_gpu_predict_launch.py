"""Launch shapes of the tile prediction kernel, by their times on the device
(the least of many; each bound lies between the two shapes' measured ratios)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _model(engine, capi, T, D, F, levels=0):
    """T trees; thresholds of `levels` values a feature (0: all different, so
    many that the model has no binned form)."""
    rng = np.random.default_rng(T + D)
    feature = rng.integers(0, F, (T, D)).astype(np.uint16)
    thr = rng.standard_normal((T, D)).astype(np.float32)
    if levels:
        q = np.sort(rng.standard_normal((F, levels)).astype(np.float32), 1)
        thr = q[feature, rng.integers(0, levels, (T, D))]
    a = dict(depth=np.full(T, D, np.int32), feature=feature, threshold=thr,
             leaves=rng.standard_normal((T, 1 << D)).astype(np.float32), weights=np.full(T, 0.1, np.float32))
    return engine.import_model(capi.ModelInfo(T, 1, D, F, 0, 0.0, 0.1, 1.0), a)


def _least_us(m, n, F, reps=12):
    import torch

    X = torch.randn(n, F, device="cuda")
    out = torch.empty(n, device="cuda")
    st = torch.cuda.Stream()
    time.sleep(0.03)  # a latency worker of a test before leaves after 20 ms without a request
    t = []
    for _ in range(reps):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record(st)
        m.predict_device(X.data_ptr(), n, F, out.data_ptr(), "raw", st.cuda_stream)
        b.record(st)
        b.synchronize()
        t.append(a.elapsed_time(b) * 1e3)
    return min(t)


def test_float_walk_takes_128_row_tiles(engine, capi):
    """One 128-row tile more than the device has multiprocessors: about a third
    longer than one each (two blocks share a multiprocessor), not twice, as
    256-row tiles, which walk their halves one after the other, would take."""
    F, rows = 100, _sms() * 128
    m = _model(engine, capi, 7600, 10, F)
    assert _least_us(m, rows + 128, F) < 1.65 * _least_us(m, rows, F)
    m.close()


def test_rows_past_a_whole_wave(engine, capi):
    """A 256-row tile for every multiprocessor and almost half as many rows
    again: the rest in 128-row tiles takes about half as long again; as 256-row
    tiles beside half of the others it took 1.8 times as long."""
    F, rows = 37, _sms() * 256
    m = _model(engine, capi, 1000, 10, F, 254)
    assert _least_us(m, rows + rows // 2 - 128, F, 30) < 1.66 * _least_us(m, rows, F, 30)
    m.close()


def test_few_tiles_take_the_larger_chunks(engine, capi):
    """With at most a block per multiprocessor the room for a second one is worth
    nothing: 73 features (two blocks fit, with the smallest chunks of trees) take
    no longer than 120 (they do not fit)."""
    t = []
    for F in (73, 120):
        m = _model(engine, capi, 2000, 10, F, 254)
        t.append(_least_us(m, 200, F, 30))
        m.close()
    assert t[0] < 1.15 * t[1], t


def test_a_long_model_in_a_mixed_burst(engine, capi):
    """A burst's tiles of a model of many trees end a burst of other rows: they
    take 128 rows while the multiprocessors hold one each, and start first.  (A
    256-row tile takes about 1.45 times as long.)"""
    F, heavy_rows, light_rows = 8, 12_800, 15_000
    heavy, light = _model(engine, capi, 30_000, 6, F, 254), _model(engine, capi, 200, 4, F, 254)
    srv = capi.Server(engine, staging_bytes=0, max_batch_rows=131_072, coalesce=True, max_inflight=4)
    h, li = srv.add_model(heavy), srv.add_model(light)
    rng = np.random.default_rng(0)

    def request(mid, n):
        import torch

        X = torch.empty((n, F), pin_memory=True).numpy()
        X[:] = rng.standard_normal((n, F))
        return 0.0, mid, X, torch.empty((n, 1), pin_memory=True).numpy(), "raw"

    alone = [request(h, heavy_rows)]
    # (a first request takes the server's first launch; the others share the next)
    mixed = [request(li, 1)] + alone + [request(li, light_rows) for _ in range(4)]
    time.sleep(0.03)
    tries = []
    for _ in range(3):  # (host threads take part: another try where they were held up)
        t = [float(np.median([srv.replay(reqs)[1] for _ in range(25)])) for reqs in (alone, mixed)]
        tries.append(t[1] / t[0])
        if tries[-1] < 1.25:
            break
    assert min(tries) < 1.25, tries
    srv.close()
    heavy.close()
    light.close()
