"""Device buffers kept for reuse: objects made from reused blocks give the same
results as fresh ones, and the kept blocks stay within the budget."""
import numpy as np
import pytest

from datagen import binary_c1

pytestmark = pytest.mark.gpu


def _fit(eng, capi, n, f, seed):
    X, y = binary_c1(n, f, seed=seed)
    ds = eng.upload(X, y)
    edges, ne = ds.quantize(255)
    m, _ = eng.train(ds, capi.params(loss="logloss", n_estimators=4, max_depth=5, hist_features_per_block=32))
    out = (edges, ne, ds.bins(), m.export())
    m.close()
    ds.close()
    return out


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3])) and all(
        np.array_equal(a[3][k], b[3][k]) for k in ("depth", "feature", "bin", "threshold", "leaves"))


def test_reused_blocks_give_the_same_results(capi):
    shapes = [(3000, 12, 1), (5000, 7, 2), (2900, 12, 3), (400, 30, 4)]
    fresh = []
    for s in shapes:
        eng = capi.Engine(0)
        fresh.append(_fit(eng, capi, *s))
        eng.close()
    eng = capi.Engine(0)
    base = eng.memory()[0]
    for _ in range(2):
        for s, want in zip(shapes, fresh):
            assert _equal(_fit(eng, capi, *s), want)
            assert eng.memory()[0] == base  # kept blocks are not in use
    eng.close()


def test_kept_blocks_count_against_the_budget(capi):
    """A context with a budget: what a destroyed dataset left behind makes room
    for a larger one, and the budget still refuses what does not fit."""
    X = np.zeros((1000, 256), np.float32)  # 1 MB
    eng = capi.Engine(0, mem_budget=4 << 20)
    for rows in (1000, 2000, 3000, 1000, 3500):
        ds = eng.upload(np.repeat(X, 4, axis=0)[:rows])
        assert eng.memory()[0] <= 4 << 20
        ds.close()
    with pytest.raises(capi.TCError):
        eng.upload(np.repeat(X, 6, axis=0)[:5000])
    eng.upload(X).close()
    eng.close()


def test_the_longest_kept_blocks_make_room(capi):
    """More than 4 GiB released: at most 4 GiB stay mapped, and a block of
    another size released after that is kept all the same."""
    import torch

    eng = capi.Engine(0)
    X = np.zeros((600_000, 256), np.float32)  # 586 MiB
    eng.upload(X[:1000]).close()
    free0 = torch.cuda.mem_get_info(0)[0]
    for ds in [eng.upload(X) for _ in range(8)]:
        ds.close()
    eng.upload(X[:250_000]).close()  # too small for any of the kept blocks
    left = torch.cuda.mem_get_info(0)[0]
    assert free0 - left <= (4 << 30) + (64 << 20)
    ds = eng.upload(X[:250_000])
    assert torch.cuda.mem_get_info(0)[0] == left
    ds.close()
    eng.close()
