"""The work a user has this framework do, as measurable cases.

Each case is one call (or the short sequence of calls that belongs together)
through the public entry points in `turbocat._capi`, at sizes of the
repository's configurations (tests/datagen.py, bench.py) or generic ones:
fits from host arrays, boosting on a resident dataset, binning, categorical
target statistics, and prediction from one row to half a million.
`listed()` gives the fixed cases, `draw(rng)` further ones of the same ranges.
`exact(case, seed)` restates binning, boosting and prediction in 64 bits with
plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "turbo-cat_b200"))

from turbocat import _capi  # noqa: E402

_engine = None
_resident = {}  # models that a scoring program loads once, by shape


def engine():
    """One engine per process, as a program keeps it."""
    global _engine
    if _engine is None:
        _engine = _capi.Engine(0)
    return _engine


# ------------------------------------------------------------------- cases --

def listed():
    return [
        # A small table fitted from host arrays with the plain settings
        # (upload, binning, 100 trees, model back): latency and launches count.
        dict(name="fit_binary_50k", kind="fit", loss="logloss", n=50_000, f=20, depth=6, trees=100, lr=0.1, lam=1.0),
        # A regression fit on a resident, binned table of the regression
        # configuration's shape: 20 of its 500 trees.
        dict(name="train_regression_1m", kind="train", loss="mse", n=1_000_000, f=100, depth=8, trees=20, lr=0.05,
             lam=0.0),
        # Boosting iterations of the multiclass configuration (10 classes).
        dict(name="boost_multiclass_1m", kind="boost", loss="softmax", classes=10, n=1_000_000, f=50, depth=6, trees=4,
             lr=0.1, lam=1.0),
        # Boosting iterations of the imbalanced focal configuration: the
        # largest table; a small min_child_weight since focal hessians are tiny.
        dict(name="boost_focal_2m5", kind="boost", loss="focal", n=2_500_000, f=200, depth=8, trees=8, lr=0.1, lam=1.0,
             mcw=1e-3),
        # The facade's default row sampling (0.8) with a validation set and
        # early stopping, odd sizes.
        dict(name="train_sampled_valid_200k", kind="train", loss="logloss", n=200_003, f=37, depth=6, trees=24, lr=0.1,
             lam=1.0, subsample=0.8, n_valid=20_001),
        # mode="small": regular (depth-wise) trees, then scores of the table.
        dict(name="regular_50k", kind="regular", n=50_000, f=20, depth=6, trees=10, lr=0.1, lam=1.0),
        # Binning a table (3% NaN, a few low-cardinality columns) and applying
        # the bins to a held-out one.
        dict(name="quantize_1m", kind="quantize", n=1_000_003, f=100, n_test=10_007, bins=255),
        # The front end of a fit with categorical columns: upload, ordered
        # target statistics, binning.
        dict(name="encode_categorical_1m", kind="encode", n=1_000_000, f=20, n_cat=4, cardinality=1000,
             method="ordered"),
        # One row through a resident model from host memory: pure latency.
        dict(name="predict_row_1000xd6", kind="predict", where="host", n=1, f=100, trees=1000, depth=6, classes=1),
        # A burst of requests of uneven sizes (log-uniform) on four resident
        # models through the serving loop.
        dict(name="serve_burst", kind="serve", requests=48, max_rows=16_384, f=100),
        # Batch scoring of resident rows with the serving configuration's model.
        dict(name="predict_resident_500k", kind="predict", where="device", n=500_000, f=100, trees=1000, depth=6,
             classes=1),
        # Batch scoring with a ten-class model (200 iterations x 10 trees).
        dict(name="predict_multiclass_200k", kind="predict", where="device", n=200_000, f=50, trees=2000, depth=6,
             classes=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "train", "boost", "regular", "quantize", "encode", "predict", "predict", "predict_host",
                       "serve"])
    if kind in ("fit", "train", "boost"):
        loss = rng.choice(["logloss", "mse", "softmax", "focal"])
        depth = rng.randint(3, 8)
        f = _log_int(rng, 5, 200)
        n = _log_int(rng, 2_000, min(2_000_000, 200_000_000 // f))
        c = dict(kind=kind, loss=loss, n=n, f=f, depth=depth, trees=rng.randint(4, 12), lr=rng.choice([0.05, 0.1, 0.3]),
                 lam=rng.choice([0.5, 1.0, 3.0]))
        if loss == "softmax":
            c["classes"] = rng.randint(3, 10)
            c["n"] = max(2_000, c["n"] // c["classes"])
        if loss == "focal":
            c["mcw"] = 1e-3
        if kind == "train" and c["n"] <= 300_000 and rng.random() < 0.5:
            c["subsample"] = round(rng.uniform(0.5, 0.95), 2)
            c["n_valid"] = max(500, c["n"] // 10)
        return c
    if kind == "regular":
        return dict(kind=kind, n=_log_int(rng, 1_000, 100_000), f=_log_int(rng, 4, 60), depth=rng.randint(3, 7),
                    trees=rng.randint(4, 12), lr=0.1, lam=1.0)
    if kind == "quantize":
        f = _log_int(rng, 3, 200)
        return dict(kind=kind, n=_log_int(rng, 1_000, min(2_000_000, 100_000_000 // f)), f=f,
                    n_test=_log_int(rng, 100, 20_000), bins=rng.choice([255, 255, 128, 64, 15]))
    if kind == "encode":
        return dict(kind=kind, n=_log_int(rng, 2_000, 1_000_000), f=rng.randint(9, 30), n_cat=rng.randint(1, 4),
                    cardinality=_log_int(rng, 5, 50_000), method=rng.choice(["ordered", "cv"]))
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(12, 60), max_rows=_log_int(rng, 64, 16_384), f=rng.randint(20, 120))
    depth = rng.randint(3, 10)
    trees = _log_int(rng, 50, max(60, min(2_000, 10_000 // depth)))
    classes = rng.choice([1, 1, 1, rng.randint(3, 10)])
    trees = max(classes, trees // classes * classes)
    f = rng.randint(10, 150)
    if kind == "predict_host":
        return dict(kind="predict", where="host", n=_log_int(rng, 1, 20_000), f=f, trees=trees, depth=depth,
                    classes=classes)
    return dict(kind="predict", where="device", n=_log_int(rng, 100, 400_000), f=f, trees=trees, depth=depth,
                classes=classes)


# ------------------------------------------------------------------ inputs --

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=_dev(), dtype=torch.float32)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=_dev(), dtype=torch.float32)


def _table(g, n, f):
    """Half normal, a quarter uniform, a quarter log-normal columns."""
    X = _randn(g, n, f)
    a, b = f // 2, f // 2 + f // 4
    X[:, a:b] = _rand(g, n, b - a) * 6.0 - 3.0
    X[:, b:] = torch.exp(X[:, b:])
    return X


def _labels(g, X, loss, classes):
    n, f = X.shape
    k = min(f, 20)
    if loss == "mse":
        return torch.sin(X[:, : min(10, f)]).sum(1) + X[:, 0] * X[:, f - 1] + 0.1 * _randn(g, n)
    if loss == "softmax":
        W = _randn(g, k, classes)
        gumbel = -torch.log(-torch.log(_rand(g, n, classes).clamp_(1e-6, 1 - 1e-6)))
        return torch.argmax(X[:, :k] @ W + gumbel, dim=1).float()
    s = X[:, :k] @ _randn(g, k)
    if loss == "focal":  # about 1% positives
        s = s + 0.5 * _randn(g, n)
        q = torch.quantile(s[: min(n, 1_000_000)], 0.99)
        return (s > q).float()
    s = s - s.median()
    return (_rand(g, n) < torch.sigmoid(s + 0.5 * X[:, 0] * X[:, 1])).float()


def _host(t):
    """A page-locked host array, where a program that trains repeatedly keeps its table."""
    if not torch.cuda.is_available():
        return t.numpy()
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    torch.cuda.synchronize()
    return h.numpy()


def _train_table(case, seed):
    g = _gen(seed)
    n, nv = case["n"], case.get("n_valid", 0)
    loss = case.get("loss", "logloss")
    X = _table(g, n + nv, case["f"])
    y = _labels(g, X, loss, case.get("classes", 1))
    return X, y


def _quantize_table(case, seed):
    g = _gen(seed)
    X = _table(g, case["n"] + case["n_test"], case["f"])
    X[:, ::7] = torch.round(X[:, ::7] * 4.0) / 4.0  # low-cardinality columns
    X[_rand(g, *X.shape) < 0.03] = float("nan")
    return X[: case["n"]].contiguous(), X[case["n"]:].contiguous()


def _cat_table(case, seed):
    g = _gen(seed)
    n = case["n"]
    X = _randn(g, n, case["f"])
    s = X[:, 0].clone()
    for c in range(case["n_cat"]):
        j = 2 * c + 1
        cat = torch.floor(_rand(g, n) * case["cardinality"])
        s += (cat % 7 - 3) * 0.5
        cat[_rand(g, n) < 0.03] = float("nan")
        X[:, j] = cat
    y = (_rand(g, n) < torch.sigmoid(s)).float()
    return X, y, [2 * c + 1 for c in range(case["n_cat"])]


def _ensemble(g, f, trees, depth, classes):
    """Arrays of a model: thresholds are edges of a 255-bin normal column, as a trained model's are."""
    q = torch.arange(1, 255, device=_dev(), dtype=torch.float64) / 255.0
    edges = (math.sqrt(2.0) * torch.erfinv(2.0 * q - 1.0)).float()
    shift = 0.01 * _randn(g, f, 1)
    table = edges[None, :] + shift  # [f][254]
    feature = torch.randint(0, f, (trees, depth), generator=g, device=_dev())
    rank = torch.randint(0, 254, (trees, depth), generator=g, device=_dev())
    thr = table[feature, rank]
    leaves = _randn(g, trees, 1 << depth)
    arrays = dict(depth=np.full(trees, depth, np.int32), feature=feature.cpu().numpy().astype(np.uint16),
                  bin=rank.cpu().numpy().astype(np.uint8), threshold=thr.cpu().numpy(), leaves=leaves.cpu().numpy(),
                  weights=np.full(trees, 0.1, np.float32))
    info = _capi.ModelInfo(trees, classes, depth, f, 1 if classes > 1 else 0, 0.0 if classes > 1 else -0.25, 0.1, 1.0)
    return info, arrays


def _resident_model(f, trees, depth, classes):
    """The model of a program that answers small requests: loaded once, new rows with every call."""
    key = (f, trees, depth, classes)
    if key not in _resident:
        _resident[key] = engine().import_model(*_ensemble(_gen(4), *key))
    return _resident[key]


def _transform(classes):
    return "softmax" if classes > 1 else "sigmoid"


def _serve_models(g, f):
    """The serving configuration's four models: (trees, depth)."""
    return [_ensemble(g, f, t, d, 1) for t, d in ((1000, 6), (200, 4), (500, 8), (2000, 10))]


def _serve_requests(case, seed):
    # the burst's shape belongs to the case; its rows to the seed
    r = np.random.default_rng([case["requests"], case["max_rows"], case["f"]])
    rows = np.exp(r.uniform(0.0, math.log(case["max_rows"] + 1), case["requests"])).astype(np.int64)
    rows = np.clip(rows, 1, case["max_rows"])
    model = r.integers(0, 4, case["requests"])
    pool = _randn(_gen(seed + 1_000_003), int(rows.sum()), case["f"])
    return rows, model, pool


def _params(case):
    return _capi.params(loss=case.get("loss", "logloss"), n_classes=case.get("classes", 1), n_estimators=case["trees"],
                        max_depth=case["depth"], learning_rate=case["lr"], lambda_l2=case["lam"],
                        min_child_weight=case.get("mcw", 1.0), subsample=case.get("subsample", 1.0),
                        colsample_bytree=case.get("subsample", 1.0))


def prepare(case, seed):
    eng = engine()
    kind = case["kind"]
    st = dict(case=case, eng=eng)
    if kind in ("fit", "train", "boost", "regular"):
        X, y = _train_table(case, seed)
        n = case["n"]
        hX, hy = _host(X[:n]), _host(y[:n])
        st["params"] = _params(case)
        if kind == "fit":
            st.update(X=hX, y=hy)
            return st
        st["ds"] = eng.upload(hX, hy)
        st["ds"].quantize(255)
        if kind == "regular":
            st["X"] = hX
        elif kind == "boost":
            st["trainer"] = eng.trainer(st["ds"], st["params"])
        elif case.get("n_valid"):
            st["valid"] = eng.upload(_host(X[n:]), _host(y[n:]))
        return st
    if kind == "quantize":
        X, T = _quantize_table(case, seed)
        st.update(ds=eng.upload(_host(X)), test=eng.upload(_host(T)))
        return st
    if kind == "encode":
        X, y, feats = _cat_table(case, seed)
        st.update(X=_host(X), y=_host(y), feats=feats)
        return st
    if kind == "serve":
        rows, model, pool = _serve_requests(case, seed)
        g = _gen(seed + 7)
        st["models"] = [eng.import_model(i, a) for i, a in _serve_models(g, case["f"])]
        st["server"] = _capi.Server(eng, staging_bytes=0, max_batch_rows=131_072, coalesce=True, max_inflight=4)
        ids = [st["server"].add_model(m) for m in st["models"]]
        pool = _host(pool)
        off = np.concatenate([[0], np.cumsum(rows)])
        out = torch.empty((int(off[-1]), 1), dtype=torch.float32, pin_memory=True).numpy()
        st["reqs"] = [(ids[model[i]], pool[off[i]:off[i + 1]], out[off[i]:off[i + 1]]) for i in range(len(rows))]
        st["out"] = out
        return st
    X = _randn(_gen(seed), case["n"], case["f"])
    shape = (case["f"], case["trees"], case["depth"], case["classes"])
    if case["where"] == "host":
        st["model"] = _resident_model(*shape)
        st["X"] = _host(X)
    else:
        st["model"] = eng.import_model(*_ensemble(_gen(seed + 7), *shape))
        st["X"] = X
        st["out"] = torch.empty((case["n"], case["classes"]), dtype=torch.float32, device=X.device)
    return st


def _model_out(m):
    e = m.export()
    return {k: e[k] for k in ("depth", "feature", "bin", "threshold", "gain", "leaves")}


def run(st):
    case, eng, kind = st["case"], st["eng"], st["case"]["kind"]
    if kind == "fit":
        ds = eng.upload(st["X"], st["y"])
        ds.quantize(255)
        m, _ = eng.train(ds, st["params"])
        out = _model_out(m)
        m.close()
        ds.close()
        return out
    if kind == "train":
        if "valid" in st:
            tr = eng.trainer(st["ds"], st["params"])
            tr.set_validation(st["valid"], 50)
            tr.step(case["trees"])
            out = dict(loss=tr.valid_loss())
            m = tr.model()
            tr.close()
        else:
            m, _ = eng.train(st["ds"], st["params"])
            out = {}
        out.update(_model_out(m))
        m.close()
        return out
    if kind == "boost":
        tr = st["trainer"]
        tr.reset()
        tr.step(case["trees"])
        m = tr.model()
        out = _model_out(m)
        m.close()
        return out
    if kind == "regular":
        m, _ = eng.train_regular(st["ds"], st["params"])
        # the model file's bytes in a buffer that takes any tree count's nodes
        model = np.zeros(64 + case["f"] * 1028 + case["trees"] * (32 + 16 * 255), np.uint8)
        tcat = np.frombuffer(m.tcat(), np.uint8)
        model[: tcat.size] = tcat
        out = dict(model=model, scores=m.predict(st["X"]))
        m.close()
        return out
    if kind == "quantize":
        edges, n_edges = st["ds"].quantize(case["bins"])
        st["test"].apply_bins(st["ds"])
        return dict(edges=edges, n_edges=n_edges, test_bins=st["test"].bins())
    if kind == "encode":
        ds = eng.upload(st["X"], st["y"])
        ds.encode_categorical(st["feats"], case["method"], seed=11)
        categories = np.zeros((len(st["feats"]), case["cardinality"]), np.uint32)
        encodings = np.zeros((len(st["feats"]), case["cardinality"]), np.float32)
        for c, j in enumerate(st["feats"]):
            keys, vals = ds.category_table(j)
            categories[c, : keys.size], encodings[c, : vals.size] = keys, vals
        edges, n_edges = ds.quantize(255)
        ds.close()
        return dict(categories=categories, encodings=encodings, edges=edges, n_edges=n_edges)
    if kind == "serve":
        srv = st["server"]
        tickets = [srv.submit(mid, X, out, "sigmoid") for mid, X, out in st["reqs"]]
        for t in tickets:
            while not srv.poll(t)[0]:
                pass
        return st["out"]
    if case["where"] == "host":
        return st["model"].predict(st["X"], _transform(case["classes"]))
    # on torch's stream, as a program that makes the rows with torch calls it
    st["model"].predict_device(st["X"].data_ptr(), case["n"], case["f"], st["out"].data_ptr(),
                               _transform(case["classes"]), torch.cuda.current_stream().cuda_stream or 1)
    return st["out"]


def work(case):
    """What a pass cannot do without: inputs read once, outputs written once
    (training: the binned table, the labels and the scores once per tree)."""
    kind, f = case["kind"], case["f"]
    if kind in ("fit", "train", "boost", "regular"):
        n, tk = case["n"], case["trees"] * case.get("classes", 1)
        b = tk * n * (f + 12.0) + (4.0 * n * f if kind == "fit" else 0.0)
        b += case["trees"] * 4.0 * case.get("n_valid", 0) * f
        return dict(bytes=b, flops=2.0 * tk * n * f)
    n = case.get("n", 0)
    if kind == "quantize":
        return dict(bytes=(n + case["n_test"]) * f * 5.0, flops=0.0)
    if kind == "encode":
        return dict(bytes=n * f * 5.0 + n * case["n_cat"] * 8.0, flops=0.0)
    if kind == "serve":
        rows = case["requests"] * case["max_rows"] / math.log(case["max_rows"] + 1)  # mean of the log-uniform sizes
        return dict(bytes=rows * (f + 1) * 4.0, flops=rows * (6000 + 800 + 4000 + 20000) / 4.0)
    trees, depth = case["trees"], case["depth"]
    return dict(bytes=n * 4.0 * (f + case["classes"]) + trees * (8.0 * depth + 4.0 * (1 << depth)),
                flops=float(n) * trees * (depth + 1))


# ------------------------------------------------------- values in 64 bits --

def _edges_of(x, max_bins):
    """One column's quantile edges (Dataset.quantize with its uint8 count rule)."""
    x = x[~torch.isnan(x)]
    if x.numel() == 0:
        return torch.zeros(1, dtype=torch.float32, device=x.device)
    u = torch.unique(torch.where(x == 0, torch.zeros_like(x), x))
    U = u.numel()
    A = min(max_bins, U & 255)
    if A < 2:
        return u[:0]
    b = torch.arange(1, A, device=x.device, dtype=torch.int64)
    return u[b * U // A]


def _pad_edges(edges):
    out = np.zeros((len(edges), 255), np.float64)
    for j, e in enumerate(edges):
        out[j, : e.numel()] = e.double().cpu().numpy()
    return out


def _predict64(info, a, X, classes):
    """Scores [n][classes] in FP64."""
    dev = X.device
    out = torch.full((X.shape[0], classes), float(info.base_prediction), dtype=torch.float64, device=dev)
    feat = torch.from_numpy(a["feature"].astype(np.int64))
    thr = torch.from_numpy(a["threshold"]).to(dev)
    leaves = torch.from_numpy(a["leaves"]).to(dev).double() * 0.1
    Xt = X.t().contiguous()
    for t in range(feat.shape[0]):
        idx = torch.zeros(X.shape[0], dtype=torch.int64, device=dev)
        for d in range(feat.shape[1]):
            idx = 2 * idx + (Xt[int(feat[t, d])] >= thr[t, d]).long()
        out[:, t % classes] += leaves[t][idx]
    return torch.softmax(out, 1) if classes > 1 else torch.sigmoid(out)


def _sigmoid64(p):
    """The trainer's logloss probability: a degree-5 polynomial of 2^fraction (its definition), here in FP64."""
    x = (-p.clamp(-15.0, 15.0)).clamp(-88.0, 88.0) * 1.4426950408889634
    i = torch.round(x)
    f = x - i
    e = f * 0.0013333558146428443 + 0.009618129107628477
    for c in (0.05550410866482046, 0.2402265069591007, 0.6931471805599453, 1.0):
        e = e * f + c
    return 1.0 / (1.0 + e * torch.exp2(i))


def _gradients64(loss, pred, y):
    if loss == "mse":
        return 2.0 * (pred - y[None]), torch.full_like(pred, 2.0)
    if loss == "softmax":
        p = torch.softmax(pred, 0)
        g = p.clone()
        g[y.long(), torch.arange(y.numel(), device=y.device)] -= 1.0
        return g, (p * (1.0 - p)).clamp_min(1e-6)
    p = _sigmoid64(pred)
    nv = y.numel() // 8 * 8
    p[:, nv:] = torch.sigmoid(pred[:, nv:].clamp(-15.0, 15.0))
    return p - y[None], (p * (1.0 - p)).clamp_min(1e-6)


def _level_gain(bins, node, nn, g, h, lam):
    """[f][254] summed gain of every (feature, bin) and whether any node of the level allows it."""
    f = bins.shape[0]
    total = torch.empty((f, 254), dtype=torch.float64, device=bins.device)
    allowed = torch.empty((f, 254), dtype=torch.bool, device=bins.device)
    base = node * 256
    gh = torch.stack((g, h), 1)
    for j in range(f):
        hist = torch.zeros((nn * 256, 2), dtype=torch.float64, device=bins.device)
        hist.index_add_(0, base + bins[j].long(), gh)
        hist = hist.view(nn, 256, 2)
        c = hist[:, :255].cumsum(1)
        all_ = c[:, -1:]
        L = c[:, :254]
        R = (hist[:, :255].flip(1).cumsum(1).flip(1))[:, 1:]
        gl, hl, gr, hr = L[..., 0], L[..., 1], R[..., 0], R[..., 1]
        G, H = all_[..., 0], all_[..., 1]
        par = torch.where(H > 1e-10, G * G / (H + lam), torch.zeros_like(G))
        ok = (hl >= 1e-10) & (hr >= 1e-10)
        v = 0.5 * (gl * gl / (hl + lam) + gr * gr / (hr + lam) - par)
        total[j] = torch.where(ok, v, torch.zeros_like(v)).sum(0)
        allowed[j] = ok.any(0)
    return total, allowed


def _boost64(case, X, y):
    """The symmetric-tree boosting loop on all rows in FP64."""
    loss, K, D, lam, lr = case["loss"], case.get("classes", 1), case["depth"], case["lam"], case["lr"]
    lam, lr, mcw = float(np.float32(lam)), float(np.float32(lr)), case.get("mcw", 1.0)
    dev, n, f = X.device, X.shape[0], X.shape[1]
    edges = [_edges_of(X[:, j].contiguous(), 255) for j in range(f)]
    bins = torch.empty((f, n), dtype=torch.uint8, device=dev)
    for j in range(f):
        bins[j] = torch.bucketize(X[:, j].contiguous(), edges[j], right=True).to(torch.uint8)
    yd = y.double()
    if loss == "softmax":
        base = 0.0
    else:
        # the reference's start: an FP32 running sum of the labels
        s = np.cumsum(y.cpu().numpy(), dtype=np.float32)[-1]
        p = float(s / np.float32(n))
        base = p if loss == "mse" else math.log(min(max(p, 1e-7), 1 - 1e-7) / (1 - min(max(p, 1e-7), 1 - 1e-7)))
    pred = torch.full((K, n), base, dtype=torch.float64, device=dev)
    T = case["trees"] * K
    out = dict(threshold=np.zeros((T, D)), gain=np.zeros((T, D)), leaves=np.zeros((T, 1 << D)))
    t = 0
    for _ in range(case["trees"]):
        G, H = _gradients64(loss, pred, yd)
        for k in range(K):
            g, h = G[k], H[k]
            node = torch.zeros(n, dtype=torch.int64, device=dev)
            depth = 0
            for d in range(D):
                cnt = torch.bincount(node, minlength=1 << d)
                hn = torch.zeros(1 << d, dtype=torch.float64, device=dev).index_add_(0, node, h)
                if not bool(((cnt >= 2) & (hn >= 2.0 * mcw)).any()):
                    break
                gain, ok = _level_gain(bins, node, 1 << d, g, h, lam)
                if d == 0:
                    gain = torch.where(ok, gain, torch.full_like(gain, -1e300))
                q = int(torch.argmax(gain.view(-1)))
                best = float(gain.view(-1)[q])
                if best < 0.0:
                    break
                j, b = q // 254, q % 254
                ne = edges[j].numel()
                out["threshold"][t, d] = float(edges[j][min(b, ne - 1)]) if ne else 0.0
                out["gain"][t, d] = best
                node = 2 * node + (bins[j] > b).long()
                depth = d + 1
            L = 1 << depth
            gs = torch.zeros(L, dtype=torch.float64, device=dev).index_add_(0, node, g)
            hs = torch.zeros(L, dtype=torch.float64, device=dev).index_add_(0, node, h)
            leaf = torch.where(hs >= 1e-10, -gs / (hs + lam), torch.zeros_like(gs))
            out["leaves"][t, :L] = leaf.cpu().numpy()
            pred[k] += lr * leaf[node]
            t += 1
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("fit", "train", "boost"):
        K = case.get("classes", 1)
        pairs = float(case["n"]) * case["f"] * case["depth"] * case["trees"] * K
        steps = float(case["f"]) * case["depth"] * case["trees"] * K
        # row samples come from the C++ library's 64-bit Mersenne twister and
        # shuffle, which plain torch or numpy does not have
        # the focal loss's FP32 gradients span six orders of magnitude and their
        # rounding decides between nearly tied thresholds: no 64-bit value
        if case.get("subsample", 1.0) < 1.0 or case["loss"] == "focal" or pairs * 0.25e-9 + steps * 0.4e-3 > 18.0:
            return None
        X, y = _train_table(case, seed)
        e = _boost64(case, X, y)
        return dict(depth=None, feature=None, bin=None, **e)
    if kind == "regular":
        return None  # its growth order and leaf cap are the trainer's own
    if kind == "quantize":
        X, _ = _quantize_table(case, seed)
        edges = [_edges_of(X[:, j].contiguous(), case["bins"]) for j in range(case["f"])]
        return dict(edges=_pad_edges(edges), n_edges=None, test_bins=None)
    if kind == "encode":
        X, y, feats = _cat_table(case, seed)
        prior = float(y.double().mean())
        enc = np.zeros((len(feats), case["cardinality"]))
        for c, j in enumerate(feats):
            ok = ~torch.isnan(X[:, j])
            cat = X[ok, j].long()
            cnt = torch.bincount(cat)
            s = torch.bincount(cat, weights=y[ok].double())
            e = ((s + prior) / (cnt + 1.0))[cnt > 0].cpu().numpy()
            enc[c, : e.size] = e
        return dict(categories=None, encodings=enc, edges=None, n_edges=None)
    if kind == "serve":
        rows, model, pool = _serve_requests(case, seed)
        models = _serve_models(_gen(seed + 7), case["f"])
        off = np.concatenate([[0], np.cumsum(rows)])
        out = np.zeros((int(off[-1]), 1))
        for k, (info, a) in enumerate(models):
            at = np.concatenate([np.arange(off[i], off[i + 1]) for i in range(len(rows)) if model[i] == k] or
                                [np.zeros(0, np.int64)])
            if len(at):
                out[at] = _predict64(info, a, pool[torch.from_numpy(at).to(pool.device)], 1).cpu().numpy()
        return out
    X = _randn(_gen(seed), case["n"], case["f"])
    info, arrays = _ensemble(_gen(4 if case["where"] == "host" else seed + 7), case["f"], case["trees"], case["depth"],
                             case["classes"])
    return _predict64(info, arrays, X, case["classes"])
