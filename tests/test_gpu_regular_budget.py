"""Regular trees under a memory budget."""
import pytest

from datagen import binary_c1

pytestmark = pytest.mark.gpu


def test_regular_trees(capi):
    """A budget without room for the histograms of every possible node of depth 8
    (19.7 MB here): the same model, grown with the nodes that are open."""
    n, f, depth = 3000, 20, 8
    X, y = binary_c1(n, f, seed=4)
    p = capi.params(loss="logloss", n_estimators=4, max_depth=depth, min_samples_leaf=60)

    def fit(budget):
        eng = capi.Engine(0, mem_budget=budget)
        ds = eng.upload(X, y)
        ds.quantize(255, compat_u8=False)
        held = eng.memory()[0]
        m, _ = eng.train_regular(ds, p)
        out = m.tcat()
        m.close()
        ds.close()
        peak = eng.memory()[1]
        eng.close()
        return out, held, peak

    want, held, peak = fit(0)
    # (the host's growth holds at most 25 open nodes of more than 2 x 60 rows)
    budget = held + 25 * f * 256 * 20 + n * 64 + (2 << 20)
    assert budget < peak
    assert fit(budget)[0] == want
