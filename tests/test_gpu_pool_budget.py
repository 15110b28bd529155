"""What a context counts and what it refuses do not depend on the objects it
had before, and the memory it maps stays within its budget."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KIB = 1024


def _upload(eng, rows):
    return eng.upload(np.zeros((rows, 256), np.float32))  # 1 KiB a row


def test_a_fitting_sequence_fits_after_larger_shapes(capi):
    """Under a budget of 4 MiB: 1000 and 2900 KiB together, on a fresh context
    and on one that keeps a block of 1200 KiB."""
    for before in ((), (1200,), (1200, 1050, 1100)):
        eng = capi.Engine(0, mem_budget=4096 * KIB)
        for rows in before:
            _upload(eng, rows).close()
        a = _upload(eng, 1000)
        b = _upload(eng, 2900)
        assert eng.memory()[0] == 3900 * KIB
        with pytest.raises(capi.TCError):  # and 3900 + 200 do not fit
            _upload(eng, 200)
        a.close()
        b.close()
        eng.close()


@pytest.mark.parametrize("budget", [0, 64 << 20])
def test_counted_bytes_are_the_bytes_asked_for(capi, budget):
    eng = capi.Engine(0, mem_budget=budget)
    base = eng.memory()[0]
    _upload(eng, 1200).close()
    peak = eng.memory()[1]
    a = _upload(eng, 1000)
    assert eng.memory() == (base + 1000 * KIB, peak)
    a.close()
    assert eng.memory() == (base, peak)
    eng.close()


def test_mapped_memory_stays_within_the_budget(capi):
    """Live and kept blocks together, measured on the device, after every
    release and every larger upload (64 MiB: the driver's own granularity)."""
    import torch

    budget, slack = 600 << 20, 64 << 20
    eng = capi.Engine(0, mem_budget=budget)
    _upload(eng, 100).close()
    free0 = torch.cuda.mem_get_info(0)[0]
    X = np.zeros((560_000, 256), np.float32)
    for rows in (300_000, 500_000, 200_000, 350_000, 560_000, 150_000):
        ds = eng.upload(X[:rows])
        assert free0 - torch.cuda.mem_get_info(0)[0] <= budget + slack
        ds.close()
        assert free0 - torch.cuda.mem_get_info(0)[0] <= budget + slack
    two = [eng.upload(X[:280_000]) for _ in range(2)]
    assert free0 - torch.cuda.mem_get_info(0)[0] <= budget + slack
    for ds in two:
        ds.close()
    assert free0 - torch.cuda.mem_get_info(0)[0] <= budget + slack
    eng.close()
