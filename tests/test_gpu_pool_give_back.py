"""Kept device buffers are given back: by a call, and to another context of the
process whose allocation would fail without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS, BLOCK = 600_000, 600_000 * 256 * 4  # 586 MiB
SLACK = 64 << 20


def _free():
    import torch

    return torch.cuda.mem_get_info(0)[0]


def _keep(eng, X, count):
    for ds in [eng.upload(X) for _ in range(count)]:
        ds.close()


def test_trim_gives_the_kept_blocks_back(capi):
    eng = capi.Engine(0)
    X = np.zeros((ROWS, 256), np.float32)
    eng.upload(X[:100]).close()
    alive = eng.upload(X[:1000])
    free0 = _free()
    _keep(eng, X, 3)
    assert free0 - _free() >= 3 * BLOCK - SLACK  # (they are kept)
    eng.trim()
    assert free0 - _free() <= SLACK
    assert np.array_equal(alive.features(), X[:1000])
    eng.trim()  # nothing kept
    alive.close()
    eng.close()


def test_another_context_takes_the_kept_blocks(capi):
    import torch

    a, b = capi.Engine(0), capi.Engine(0)
    X = np.zeros((ROWS, 256), np.float32)
    for eng in (a, b):
        eng.upload(X[:100]).close()
    _keep(a, X, 3)
    torch.cuda.empty_cache()
    filler = torch.empty(_free() - BLOCK // 2, dtype=torch.uint8, device="cuda")  # half a block stays free
    try:
        ds = b.upload(X)
        ds.close()
    finally:
        del filler
        torch.cuda.empty_cache()
    a.close()
    b.close()


def test_the_facade_gives_back(engine):
    """Buffers of 4 bytes x 250k x 64 and more stay after a fit and go with the call."""
    import turbocat

    rng = np.random.default_rng(0)
    X = rng.standard_normal((250_000, 64)).astype(np.float32)
    y = (X[:, 0] > 0).astype(np.float32)
    turbocat.release_device_memory()
    turbocat.TurboCatClassifier(n_estimators=3, max_depth=3, verbosity=0).fit(X, y)
    kept = _free()
    turbocat.release_device_memory()
    assert _free() - kept >= X.nbytes // 2
