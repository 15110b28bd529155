"""Device memory that a binning and an encoding need: no more than their sort,
scan and result buffers, so what fitted a budget fits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tiles(n):
    return (n + 4095) // 4096


def _bins_bytes(n, f):
    groups, last = (f + 31) // 32, f - 32 * ((f + 31) // 32 - 1)
    wide = 4 if last <= 4 else 8 if last <= 8 else 16 if last <= 16 else 32
    nt = (n + 31) // 32 * 32
    return (groups - 1) * 32 * nt + wide * nt + f * ((n + 15) // 16 * 16)


@pytest.mark.parametrize("n,f", [(1000, 32), (1000, 33), (300, 64), (9000, 7), (20_000, 100)])
def test_quantize(capi, n, f):
    X = np.random.default_rng(n).standard_normal((n, f)).astype(np.float32)
    sort = 2 * n * f * 4 + f * 256 * _tiles(n) * 4 + f * _tiles(n) * 4 + f * 4
    need = n * f * 4 + sort + f * 256 * 4 + f * 2 + f * 4 + _bins_bytes(n, f)
    eng = capi.Engine(0, mem_budget=need)
    ds = eng.upload(X)
    edges, ne = ds.quantize(255, compat_u8=False)
    assert eng.memory()[1] <= need
    free = capi.Engine(0)
    want = free.upload(X)
    we, wn = want.quantize(255, compat_u8=False)
    assert np.array_equal(edges, we) and np.array_equal(ne, wn) and np.array_equal(ds.bins(), want.bins())
    for x in (ds, want, eng, free):
        x.close()


@pytest.mark.parametrize("n,nc", [(1000, 2), (256, 1), (12_000, 3)])
def test_encode(capi, n, nc):
    rng = np.random.default_rng(n)
    f = nc + 1
    X = rng.integers(0, 9, (n, f)).astype(np.float32)
    y = rng.integers(0, 2, n).astype(np.float32)
    t = _tiles(n)
    sort = 4 * nc * n * 4 + nc * 256 * t * 4 + nc * t * 4 + nc * 4 + 2 * nc * n * 4
    exact = 4 + 16 + 4 + nc * t * 12 + nc * (n + 1) * 12
    need = n * f * 4 + n * 4 + sort + exact + nc * 2 + nc * 4 + nc * 4 + f + 9 * nc * 8
    eng = capi.Engine(0, mem_budget=need)
    ds = eng.upload(X, y)
    ds.encode_categorical(range(nc), "ordered", seed=3)
    free = capi.Engine(0)
    want = free.upload(X, y)
    want.encode_categorical(range(nc), "ordered", seed=3)
    assert np.array_equal(ds.features(), want.features())
    for x in (ds, want, eng, free):
        x.close()


@pytest.mark.parametrize("n,f", [(1000, 32), (300, 64), (20_000, 96)])
def test_apply_bins(capi, n, f):
    """A held-out table's bins and its copy of the edges, in whole groups of 32
    features (the last group's table takes up to 31 KB more than its edges)."""
    rng = np.random.default_rng(n + 1)
    X, T = (rng.standard_normal((n, f)).astype(np.float32) for _ in range(2))
    free = capi.Engine(0)
    ref, want = free.upload(X), free.upload(T)
    ref.quantize(255, compat_u8=False)
    want.apply_bins(ref)
    result = f * 256 * 4 + f * 2 + f * 4 + _bins_bytes(n, f)
    budget = 64 << 20
    eng = capi.Engine(0, mem_budget=budget)
    r, t = eng.upload(X), eng.upload(T)
    r.quantize(255, compat_u8=False)
    filler = eng.upload(np.zeros(((budget - eng.memory()[0] - result) // 4, 1), np.float32))
    t.apply_bins(r)
    assert np.array_equal(t.bins(), want.bins())
    for x in (r, t, filler, ref, want, eng, free):
        x.close()
