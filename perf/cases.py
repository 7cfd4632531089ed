"""The work that is timed when this framework's speed is looked at.

Each case is one call, or one short run of calls, as a program makes them
through the package's public API: training from host rows (`train`,
`train_with_eval`, `train_many`), boosting rounds over a matrix that is
already binned on the device (`GHistIndex.from_device` + `Booster`), the
histogram backend seam (`GpuBackend.build`), and prediction (`predict`,
`predict_contribs`, the serving loop). Data has the distributions of
`datagen.py`: N(0,1), lognormal and Bernoulli(0.05) columns, categorical
codes, missing entries; labels follow from the features.

A case is a dict of plain values; `kind` says which call it is. Models for the
prediction cases are generated (splits inside the range that reaches a node,
covers as the split shares them out), so that 64-bit values can be computed
beside them. Trained trees have no such value: which split wins depends on
every bit before it, and outputs of training are compared as they are.
"""
import importlib
import math
import os

import numpy as np
import torch

# the serving loop's streams want more than the default 8 hardware queues
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")
sb = importlib.import_module("sequoia-boost_b200")

DEV = "cuda"


def listed():
    return [
        # One small job, as a fold or a grid point trains alone: launches and host work count.
        _train("train_small", rows=1_500, cols=20, rounds=50, depth=4, max_bin=64, eta=0.3),
        # The reference's README workload: 100k x 30, 100 rounds from pageable host rows.
        _train("train_regression", rows=100_000, cols=30, rounds=100, depth=6, eta=0.1),
        # A whole training call whose upload, cuts and binning weigh as much as its rounds;
        # ragged rows, missing entries, row and column sampling, pinned host rows.
        _train("train_binary_host", rows=1_000_003, cols=100, rounds=20, depth=8, eta=0.05,
               objective="binary:logistic", missing=0.1, subsample=0.8, colsample=0.8, pinned=True),
        # Boosting rounds of the large binary workload over its resident index.
        _train("rounds_binary_10m", kind="rounds", rows=10_000_000, cols=100, rounds=12, depth=8, eta=0.05,
               objective="binary:logistic", missing=0.1, subsample=0.8, colsample=0.8),
        # Multiclass trees grown leaf by leaf, categorical and monotone features: 10 trees a round.
        _train("rounds_multiclass_lossguide", kind="rounds", rows=2_000_000, cols=200, rounds=3, depth=0,
               max_leaves=255, classes=10, objective="multi:softprob", categorical=5, monotone=True, eta=0.3),
        # A parameter sweep: uneven jobs trained together.
        _train("sweep_64_jobs", kind="sweep", rows=100_000, cols=50, jobs=64, rounds=50, depth=8, max_bin=64),
        # Training with an eval set, its metrics each round and early stopping; row weights.
        _train("train_eval", kind="eval", rows=200_000, cols=50, eval_rows=50_000, rounds=40, depth=6, eta=0.1,
               weighted=True, missing=0.02),
        # One decision at a time: 16 rows through a large model.
        _predict("predict_16_rows", "predict", rows=16, trees=1000, depth=8),
        # The largest request of the serving workload, as one call.
        _predict("predict_65536_rows", "predict", rows=65_536, trees=1000, depth=8),
        # Explanations for a batch of rows.
        _predict("contribs_4096_rows", "contribs", rows=4_096, trees=1000, depth=8),
        # A burst of mixed requests to the serving loop: margins of 1..4096 rows, some explanations.
        _predict("serve_burst", "serve", rows=4_096, trees=1000, depth=8, requests=48),
        # The reference's HistogramBackend seam in f32: host gradient pairs and rows in, f64 sums out.
        {"name": "hist_build_fp32", "kind": "hist", "rows": 1_000_000, "cols": 50, "max_bin": 256, "share": 0.5,
         "precision": "fp32", "missing": 0.05},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.randrange(11)
    objective = rng.choice(["reg:squarederror", "reg:pseudohubererror", "binary:logistic"])
    common = {"objective": objective, "eta": rng.choice([0.05, 0.1, 0.3]), "max_bin": rng.choice([63, 64, 255, 256]),
              "missing": rng.choice([0.0, 0.02, 0.1]), "weighted": rng.random() < 0.3}
    sampled = rng.choice([{}, {"subsample": 0.8}, {"subsample": 0.8, "colsample": 0.8}, {"colsample": 0.5}])
    if what == 0:
        c = _train("", rows=log_int(300, 6_000), cols=rng.randint(4, 40), rounds=rng.randint(20, 60),
                   depth=rng.randint(3, 6), **common, **sampled)
    elif what == 1:
        c = _train("", rows=log_int(10_000, 200_000), cols=rng.randint(8, 60), rounds=rng.randint(30, 100),
                   depth=rng.randint(4, 8), **common, **sampled)
    elif what == 2:
        c = _train("", rows=log_int(150_000, 1_000_000), cols=rng.randint(40, 100), rounds=rng.randint(8, 20),
                   depth=rng.randint(6, 8), pinned=True, **common, **sampled)
    elif what == 3:
        c = _train("", kind="rounds", rows=log_int(1_000_000, 8_000_000), cols=rng.randint(30, 100),
                   rounds=rng.randint(4, 12), depth=rng.randint(5, 8), **common, **sampled)
    elif what == 4:
        classes = rng.randint(3, 10)
        c = _train("", kind="rounds", rows=log_int(100_000, 1_500_000), cols=rng.randint(30, 200), rounds=3,
                   depth=0, max_leaves=rng.choice([31, 63, 127, 255]), classes=classes,
                   objective="multi:softprob", categorical=rng.randint(0, 5), monotone=rng.random() < 0.5, eta=0.3)
    elif what == 5:
        c = _train("", kind="sweep", rows=log_int(5_000, 100_000), cols=rng.randint(24, 50),
                   jobs=rng.randint(6, 60), rounds=rng.randint(10, 50), depth=8, max_bin=rng.choice([64, 256]))
    elif what == 6:
        c = _train("", kind="eval", rows=log_int(20_000, 200_000), cols=rng.randint(10, 50),
                   eval_rows=log_int(2_000, 50_000), rounds=rng.randint(10, 40), depth=rng.randint(4, 8), **common,
                   **sampled)
    elif what == 7:
        c = _predict("", "predict", rows=log_int(1, 60_000), trees=log_int(50, 1000), depth=rng.randint(4, 8),
                     cols=rng.randint(10, 120), classes=rng.choice([1, 1, 1, 3, 10]))
    elif what == 8:
        c = _predict("", "contribs", rows=log_int(1, 4_000), trees=log_int(50, 1000), depth=rng.randint(4, 8),
                     cols=rng.randint(10, 120))
    elif what == 9:
        c = _predict("", "serve", rows=log_int(64, 4_000), trees=log_int(100, 1000), depth=rng.randint(5, 8),
                     cols=rng.randint(20, 110), requests=rng.randint(8, 48))
    else:
        c = {"name": "", "kind": "hist", "rows": log_int(20_000, 1_000_000), "cols": rng.randint(8, 50),
             "max_bin": rng.choice([63, 255, 256]), "share": round(rng.uniform(0.02, 1.0), 3),
             "precision": rng.choice(["fp32", "fixed"]), "missing": rng.choice([0.0, 0.1])}
    del c["name"]
    return c


def _train(name, kind="train", rows=0, cols=0, rounds=1, depth=6, max_bin=256, eta=0.3, max_leaves=0, classes=1,
           objective="reg:squarederror", missing=0.0, subsample=1.0, colsample=1.0, categorical=0, monotone=False,
           weighted=False, pinned=False, eval_rows=0, jobs=0):
    return {"name": name, "kind": kind, "rows": rows, "cols": cols, "rounds": rounds, "depth": depth,
            "max_bin": max_bin, "eta": eta, "max_leaves": max_leaves, "classes": classes, "objective": objective,
            "missing": missing, "subsample": subsample, "colsample": colsample, "categorical": categorical,
            "monotone": monotone, "weighted": weighted, "pinned": pinned, "eval_rows": eval_rows, "jobs": jobs}


def _predict(name, kind, rows, trees, depth, cols=100, classes=1, requests=0):
    return {"name": name, "kind": kind, "rows": rows, "trees": trees, "depth": depth, "cols": cols,
            "classes": classes, "requests": requests, "missing": 0.1}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _table(g, n, f, missing=0.0, categorical=0):
    """[n][f] f32 on the GPU: 70 % N(0,1), 20 % lognormal, 10 % Bernoulli(0.05)
    columns, the last `categorical` ones integer codes 0..31."""
    x = torch.randn(n, f, generator=g, device=DEV)
    a, b = (7 * f) // 10, (9 * f) // 10
    x[:, a:b].exp_()
    x[:, b:] = (x[:, b:] < -1.6449).float()
    if categorical:
        x[:, f - categorical:] = torch.randint(0, 32, (n, categorical), generator=g, device=DEV).float()
    return x, missing


def _holes(g, x, missing):
    if missing:
        step = max(1, (1 << 28) // x.shape[1])
        for i in range(0, x.shape[0], step):
            part = x[i:i + step]
            part[torch.rand(part.shape, generator=g, device=DEV) < missing] = float("nan")
    return x


def _labels(g, x, case):
    """Labels from the complete values, column by column in a fixed order."""
    n, f = x.shape
    objective, k = case["objective"], case["classes"]
    if objective.startswith("multi:"):
        w = torch.randn(f, k, generator=g, device=DEV)
        s = -torch.log(-torch.log(torch.rand(n, k, generator=g, device=DEV).clamp_(1e-7, 1 - 1e-7)))
        for j in range(f):
            s.addcmul_(x[:, j:j + 1], w[j:j + 1])
        return s.argmax(dim=1).float()
    s = 0.5 * x[:, 0] * x[:, 1]
    w = torch.rand(f, generator=g, device=DEV) * 2 - 1
    for j in range(f):
        s.add_(torch.sin(x[:, j]) * w[j])
    if objective == "binary:logistic":
        return (torch.rand(n, generator=g, device=DEV) < torch.sigmoid(s)).float()
    return s + 0.1 * torch.randn(n, generator=g, device=DEV)


def _host(t, pinned=False):
    if not pinned:
        return t.cpu().numpy()
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _rows(case, seed, n=None, f=None):
    """Device rows with their holes, labels and weights of one dataset."""
    g = _gen(seed)
    n, f = n or case["rows"], f or case["cols"]
    x, miss = _table(g, n, f, case["missing"], case["categorical"])
    y = _labels(g, x, case)
    w = 0.5 + torch.rand(n, generator=g, device=DEV) if case["weighted"] else None
    return _holes(g, x, miss), y, w


def _params(case, **over):
    lossguide = case["max_leaves"] > 0
    p = dict(objective=case["objective"], num_class=case["classes"] if case["classes"] > 1 else 0, eta=case["eta"],
             max_depth=case["depth"], max_leaves=case["max_leaves"], max_bin=case["max_bin"],
             grow_policy="lossguide" if lossguide else "depthwise", subsample=case["subsample"],
             colsample_bytree=case["colsample"], monotone_constraints=[1, -1] if case["monotone"] else [], seed=7)
    return sb.TrainingParams(**{**p, **over})


def _job_sizes(case):
    """Rows and features of a sweep's jobs: log-uniform from a hundredth of `rows`, 20 columns and up."""
    r = np.random.default_rng(case["jobs"])
    n = np.exp(r.uniform(math.log(max(200, case["rows"] / 100)), math.log(case["rows"]), case["jobs"])).astype(int)
    f = r.integers(20, case["cols"] + 1, case["jobs"])
    d = r.choice([4, 6, 8], case["jobs"])
    e = r.choice([0.05, 0.1, 0.3], case["jobs"])
    return [(int(a), int(b), int(c), float(h)) for a, b, c, h in zip(n, f, d, e)]


# ----------------------------------------------------------- generated models
def _forest(case, seed):
    """`trees` trees as level-order node arrays. A split's condition lies
    inside the range that reaches its node, its children's covers are the
    N(0,1) share on either side, and a node of small cover is a leaf."""
    r = np.random.default_rng(seed)
    T, D, F = case["trees"], case["depth"], case["cols"]
    ndtr = lambda v: torch.special.ndtr(torch.from_numpy(v)).numpy()  # noqa: E731
    ndtri = lambda v: torch.special.ndtri(torch.from_numpy(v)).numpy()  # noqa: E731
    share = r.dirichlet(np.full(F, 0.5))  # some features are split on often
    feat, cond, alive, cover = [], [], [np.ones((T, 1), bool)], [np.full((T, 1), 1e5)]
    inner = []
    for d in range(D):
        m = 1 << d
        f = r.choice(F, size=(T, m), p=share)
        lo, hi = np.full((T, m), -np.inf), np.full((T, m), np.inf)
        at = np.arange(m)
        for a in range(d):
            up = at >> (d - a)
            right = (at >> (d - a - 1)) & 1
            same = feat[a][:, up] == f
            c = cond[a][:, up]
            hi = np.where(same & (right == 0), np.minimum(hi, c), hi)
            lo = np.where(same & (right == 1), np.maximum(lo, c), lo)
        pl, ph = ndtr(lo), ndtr(hi)
        q = r.beta(2.0, 2.0, (T, m)) * 0.9 + 0.05
        c = ndtri(np.clip(pl + (ph - pl) * q, 1e-12, 1 - 1e-12)).astype(np.float32)
        grow = alive[d] & (cover[d] > 150.0) & (ph - pl > 1e-6) & ((r.random((T, m)) > 0.03) | (d < 2))
        feat.append(f)
        cond.append(c.astype(np.float64))
        inner.append(grow)
        alive.append(np.repeat(grow, 2, axis=1))
        child = np.empty((T, 2 * m))
        child[:, 0::2], child[:, 1::2] = cover[d] * q, cover[d] * (1 - q)
        cover.append(child)
    inner.append(np.zeros((T, 1 << D), bool))
    level = np.stack([a.sum(axis=1) for a in alive], axis=1)
    first = np.concatenate([np.zeros((T, 1), int), np.cumsum(level, axis=1)], axis=1)
    off = np.concatenate([[0], np.cumsum(first[:, -1])]).astype(np.int64)
    nodes = np.zeros(off[-1], sb.api.NODE_DTYPE)
    nodes["left"] = nodes["right"] = -1
    for d in range(D + 1):
        t, j = np.nonzero(alive[d])
        rank = (np.cumsum(alive[d], axis=1) - 1)[t, j]
        at = off[t] + first[t, d] + rank
        nodes["sum_hess"][at] = cover[d][t, j]
        g = inner[d][t, j]
        nodes["leaf_value"][at[~g]] = 0.02 * r.standard_normal(int((~g).sum()))
        if g.any():
            t, j, at = t[g], j[g], at[g]
            kid = first[t, d + 1] + 2 * (np.cumsum(inner[d], axis=1) - 1)[t, j]
            nodes["left"][at], nodes["right"][at] = kid, kid + 1
            nodes["split_feature"][at], nodes["split_cond"][at] = feat[d][t, j], cond[d][t, j]
            nodes["split_gain"][at] = 1.0
            nodes["default_left"][at] = r.random(len(at)) < 0.5
    return off, nodes


def _model(case, seed):
    off, nodes = _forest(case, seed)
    multi = case["classes"] > 1
    return sb.BoostedModel.from_arrays(off, nodes, np.zeros(len(off), np.int64), [], 0.1,
                                       case["classes"] if multi else 0, case["cols"],
                                       objective="multi:softprob" if multi else "binary:logistic")


def _request_rows(case, seed, n):
    g = _gen(seed)
    return _holes(g, torch.randn(n, case["cols"], generator=g, device=DEV), case["missing"])


def _requests(case):
    """(first row, rows, kind) of a burst: rows log-uniform in [1, `rows`], every twelfth an explanation of fewer."""
    r = np.random.default_rng(case["requests"])
    n = np.exp(r.uniform(0.0, math.log(case["rows"]), case["requests"])).astype(int).clip(1, case["rows"])
    out = []
    for i, m in enumerate(n):
        m = max(1, int(m) // 8) if i % 12 == 5 else int(m)
        out.append((int(r.integers(0, case["rows"] - m + 1)), m, "contribs" if i % 12 == 5 else "margin"))
    return out


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, y, w = _rows(case, seed)
        d = sb.DMatrix(_host(x, case["pinned"]), labels=_host(y, case["pinned"]),
                       weights=None if w is None else _host(w))
        return {"kind": kind, "data": d, "params": _params(case), "rounds": case["rounds"],
                "room": _room([(case["rounds"], 1 << case["depth"])])}
    if kind == "rounds":
        x, y, w = _rows(case, seed)
        types = None
        if case["categorical"]:
            types = [0] * (case["cols"] - case["categorical"]) + [1] * case["categorical"]
        torch.cuda.synchronize()
        index = sb.GHistIndex.from_device(x.data_ptr(), case["rows"], case["cols"], max_bin=case["max_bin"],
                                          feature_types=types)
        return {"kind": kind, "index": index, "labels": _host(y, True), "weights": None if w is None else _host(w),
                "params": _params(case), "rounds": case["rounds"],
                "room": _room([(case["rounds"] * case["classes"], case["max_leaves"] or 1 << case["depth"])],
                              case["categorical"])}
    if kind == "sweep":
        jobs = []
        for i, (n, f, depth, eta) in enumerate(_job_sizes(case)):
            x, y, _ = _rows(case, seed * 1000 + i, n, f)
            jobs.append((_params(case, max_depth=depth, eta=eta), sb.DMatrix(_host(x), labels=_host(y)),
                         case["rounds"]))
        return {"kind": kind, "jobs": jobs,
                "room": _room([(case["rounds"], 1 << depth) for _, _, depth, _ in _job_sizes(case)])}
    if kind == "eval":
        n = case["rows"]
        x, y, w = _rows(case, seed, n=n + case["eval_rows"])
        x, y, w = _host(x), _host(y), None if w is None else _host(w)
        part = lambda a, b: sb.DMatrix(x[a:b], labels=y[a:b], weights=None if w is None else w[a:b])  # noqa: E731
        return {"kind": kind, "train": part(0, n), "valid": part(n, None), "rounds": case["rounds"],
                "room": _room([(case["rounds"], 1 << case["depth"])]),
                "params": _params(case, eval_metric=["logloss", "error"] if case["objective"] == "binary:logistic"
                                  else ["mae", "rmse"])}
    if kind in ("predict", "contribs"):
        # request rows sit in page-locked memory, as the benchmark's request pool does
        return {"kind": kind, "model": _model(case, seed),
                "data": sb.DMatrix(_host(_request_rows(case, seed, case["rows"]), True))}
    if kind == "serve":
        model = _model(case, seed)
        x = _host(_request_rows(case, seed, case["rows"]), True)
        want = _requests(case)
        outs = [torch.empty(m * (case["cols"] + 1 if k == "contribs" else 1), pin_memory=True).numpy()
                for _, m, k in want]
        return {"kind": kind, "server": sb.Server(model, mem_bytes=4 << 30, n_slots=8), "x": x, "requests": want,
                "outs": outs}
    g = _gen(seed)
    x, miss = _table(g, case["rows"], case["cols"], case["missing"])
    x = _holes(g, x, miss)
    rows, pairs = _hist_inputs(g, case)
    torch.cuda.synchronize()
    index = sb.GHistIndex.from_device(x.data_ptr(), case["rows"], case["cols"], max_bin=case["max_bin"])
    return {"kind": kind, "index": index, "backend": sb.GpuBackend(case["precision"]),
            "rows": rows.cpu().numpy().astype(np.uint32), "pairs": _host(pairs)}


def _hist_inputs(g, case):
    rows = torch.nonzero(torch.rand(case["rows"], generator=g, device=DEV) < case["share"]).reshape(-1)
    p = torch.rand(case["rows"], generator=g, device=DEV)
    y = (torch.rand(case["rows"], generator=g, device=DEV) < 0.3).float()
    return rows, torch.stack([p - y, (p * (1 - p)).clamp_min(1e-16)], dim=1)


# ---------------------------------------------------------------------- run
FIELDS = ("left", "right", "split_feature", "split_cond", "leaf_value", "sum_hess", "split_gain", "default_left",
          "is_categorical")


def _room(sizes, categorical=0):
    """Arrays that hold the trees of any run, by (rounds * classes, most
    leaves) of each model; zeros after what is used."""
    n = sum(t * (2 * leaves - 1) for t, leaves in sizes)
    return {"nodes": np.zeros(n, sb.api.NODE_DTYPE), "offsets": np.zeros(sum(t + 1 for t, _ in sizes), np.int64),
            "categories": np.zeros(n * 32 if categorical else 1, np.uint32), "used": [0, 0, 0]}


def _arrays(room, models):
    """The models' trees, one array per node field."""
    got = [m.export() for m in models]
    for i, (name, part) in enumerate((("nodes", 1), ("offsets", 0), ("categories", 3))):
        at = 0
        for e in got:
            room[name][at:at + len(e[part])] = e[part]
            at += len(e[part])
        room[name][at:room["used"][i]] = 0
        room["used"][i] = at
    nodes = room["nodes"]
    out = {name: nodes[name].view(np.int32) if name == "split_feature" else nodes[name] for name in FIELDS}
    out["offsets"], out["categories"] = room["offsets"], room["categories"].view(np.int32)
    return out


def run(state):
    kind = state["kind"]
    if kind == "train":
        return _arrays(state["room"], [sb.train(state["params"], state["data"], state["rounds"])])
    if kind == "rounds":
        b = sb.Booster(state["index"], state["params"], state["labels"], weights=state["weights"])
        b.update(state["rounds"])
        return _arrays(state["room"], [b.model()])
    if kind == "sweep":
        return _arrays(state["room"], sb.train_many(state["jobs"]))
    if kind == "eval":
        r = sb.train_with_eval(state["params"], state["train"], state["rounds"], evals=[(state["valid"], "valid")],
                               early_stopping_rounds=10)
        out = _arrays(state["room"], [r.model])
        out["history"] = np.zeros((state["rounds"], 2))
        for h in r.history:
            out["history"][h.iteration] = [s[2] for s in h.scores]
        return out
    if kind == "predict":
        return state["model"].predict(state["data"])
    if kind == "contribs":
        return state["model"].predict_contribs(state["data"])
    if kind == "serve":
        srv, x = state["server"], state["x"]
        tickets = [srv.submit(x[a:a + m], kind=k, out=o) for (a, m, k), o in zip(state["requests"], state["outs"])]
        return [srv.wait(t)[0] for t in tickets]
    return state["backend"].build(state["index"], state["rows"], state["pairs"])


# --------------------------------------------------------------------- work
def _training_work(n, f, case, depth, trees, host):
    """Per round and tree: the codes of the sampled rows once, at a byte each,
    a row id and the split feature's code per level; labels, margins and
    gradient pairs once. From host rows, X once more. Two adds per code."""
    s, c = case["subsample"], case["colsample"]
    per_tree = n * s * f * c + n * s * depth * 5
    per_round = n * (4 + 16 * trees) + trees * per_tree
    return (n * f * 4 if host else n * f) + case["rounds"] * per_round, case["rounds"] * trees * n * s * f * c * 2


def work(case):
    kind = case["kind"]
    if kind in ("train", "rounds", "eval"):
        depth = case["depth"] or math.log2(case["max_leaves"])
        b, f = _training_work(case["rows"], case["cols"], case, depth, case["classes"], kind != "rounds")
        e = case["eval_rows"]
        return {"bytes": b + e * case["cols"] * 4 + case["rounds"] * e * 12, "flops": f + case["rounds"] * e * depth}
    if kind == "sweep":
        each = [_training_work(n, f, case, d, 1, True) for n, f, d, _ in _job_sizes(case)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    if kind == "hist":
        m = case["rows"] * case["share"]
        return {"bytes": m * (case["cols"] + 12) + case["cols"] * case["max_bin"] * 16, "flops": 2 * m * case["cols"]}
    nodes = case["trees"] * (1 << case["depth"]) * 1.4
    leaves = nodes / 2
    if kind == "serve":
        want = _requests(case)
        margin = sum(m for _, m, k in want if k == "margin")
        shap = sum(m for _, m, k in want if k == "contribs")
    else:
        margin, shap = (case["rows"], 0) if kind == "predict" else (0, case["rows"])
    out = margin * case["classes"] + shap * (case["cols"] + 1)
    return {"bytes": (margin + shap) * case["cols"] * 4 + out * 4 + nodes * 16,
            "flops": margin * case["trees"] * (case["depth"] + 1) + shap * leaves * case["depth"] * 2}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    kind = case["kind"]
    if kind == "hist":
        return _exact_hist(case, seed)
    if kind not in ("predict", "contribs", "serve"):
        return None  # trained trees
    off, nodes = _forest(case, seed)
    x = _request_rows(case, seed, case["rows"])
    if kind == "predict":
        return _exact_predict(case, off, nodes, x).reshape(-1)
    if kind == "contribs":
        return _exact_contribs(case, off, nodes, x).reshape(-1)
    margins = _exact_margins(case, off, nodes, x)
    return [margins[a:a + m].reshape(-1) if k == "margin"
            else _exact_contribs(case, off, nodes, x[a:a + m]).reshape(-1) for a, m, k in _requests(case)]


def _exact_margins(case, off, nodes, x):
    """[n][K] margins: the f32 base score and leaf values added in 64 bits."""
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    left, right = dev(nodes["left"]).long(), dev(nodes["right"]).long()
    feat, cond = dev(nodes["split_feature"].astype(np.int64)), dev(nodes["split_cond"])
    dflt, leaf = dev(nodes["default_left"]).bool(), dev(nodes["leaf_value"]).double()
    n, k = x.shape[0], case["classes"]
    out = torch.full((n, k), float(np.float32(0.1)), dtype=torch.float64, device=DEV)
    root = dev(off[:-1])
    for r0 in range(0, n, 8192):
        xr = x[r0:r0 + 8192]
        base = root.expand(xr.shape[0], -1)
        at = base.clone()
        for _ in range(case["depth"]):
            v = torch.gather(xr, 1, feat[at])
            go = torch.where(torch.isnan(v), dflt[at], v < cond[at])
            kid = torch.where(go, left[at], right[at])
            at = torch.where(left[at] < 0, at, base + kid)
        v = leaf[at]
        for c in range(k):
            out[r0:r0 + 8192, c] += v[:, c::k].sum(dim=1)
    return out


def _exact_predict(case, off, nodes, x):
    m = _exact_margins(case, off, nodes, x)
    return torch.softmax(m, dim=1) if case["classes"] > 1 else torch.sigmoid(m)


def _paths(case, off, nodes):
    """Every root-to-leaf path with its splits merged by feature: feature (or
    -1), range [lo, hi), whether missing values follow, the cover fraction."""
    left, right, D = nodes["left"], nodes["right"], case["depth"]
    at = off[:-1].astype(np.int64)
    base = at.copy()
    P = len(at)
    F = np.full((P, D), -1)
    lo, hi = np.full((P, D), -np.inf, np.float32), np.full((P, D), np.inf, np.float32)
    ok, z = np.ones((P, D), bool), np.ones((P, D))
    done = []
    for d in range(D + 1):
        end = left[at] < 0
        done.append([a[end] for a in (F, lo, hi, ok, z, at, base)])
        F, lo, hi, ok, z, at, base = (a[~end] for a in (F, lo, hi, ok, z, at, base))
        if not len(at):
            break
        grown = []
        f, c = nodes["split_feature"][at].astype(np.int64), nodes["split_cond"][at]
        for side in (0, 1):
            kid = base + (left if side == 0 else right)[at]
            G, l2, h2, o2, z2 = F.copy(), lo.copy(), hi.copy(), ok.copy(), z.copy()
            same = (G == f[:, None]) & (G >= 0)
            slot = np.where(same.any(axis=1), same.argmax(axis=1), (G < 0).argmax(axis=1))
            i = np.arange(len(at))
            G[i, slot] = f
            if side == 0:
                h2[i, slot] = np.minimum(h2[i, slot], c)
            else:
                l2[i, slot] = np.maximum(l2[i, slot], c)
            o2[i, slot] &= nodes["default_left"][at].astype(bool) == (side == 0)
            z2[i, slot] *= nodes["sum_hess"][kid].astype(np.float64) / nodes["sum_hess"][at].astype(np.float64)
            grown.append((G, l2, h2, o2, z2, kid, base))
        F, lo, hi, ok, z, at, base = (np.concatenate(a) for a in zip(*grown))
    return [np.concatenate(a) for a in zip(*done)]


def _exact_contribs(case, off, nodes, x):
    """Path-dependent TreeSHAP in 64 bits, from the definition: element e of a
    path with D elements (absent ones count as certain: z = o = 1) gets
    leaf * (o_e - z_e) * sum over subsets S of the others of
    |S|! (D - |S| - 1)! / D! * prod_S o * prod_not-S z."""
    D, Fc, n = case["depth"], case["cols"], x.shape[0]
    F, lo, hi, ok, z, leaf_at, _ = _paths(case, off, nodes)
    w = [math.factorial(s) * math.factorial(D - s - 1) / math.factorial(D) for s in range(D)]
    pat = (torch.arange(1 << D, device=DEV)[:, None] >> torch.arange(D, device=DEV)) & 1
    o_all = pat.double()
    out = torch.zeros(Fc + 1, n, dtype=torch.float64, device=DEV)
    xt = torch.cat([x.t().contiguous(), torch.zeros(1, n, device=DEV)])
    miss = torch.isnan(xt)
    leaf = nodes["leaf_value"][leaf_at].astype(np.float64)
    cut = max(64, (1 << 24) // max(n, 1 << D))
    for p0 in range(0, len(leaf), cut):
        s = slice(p0, p0 + cut)
        f, zz = torch.from_numpy(F[s]).to(DEV), torch.from_numpy(z[s]).to(DEV)
        lo_t, hi_t = torch.from_numpy(lo[s]).to(DEV), torch.from_numpy(hi[s]).to(DEV)
        ok_t, lv = torch.from_numpy(ok[s]).to(DEV), torch.from_numpy(leaf[s]).to(DEV)
        P = f.shape[0]
        # contributions of every pattern of one_fractions
        tab = torch.empty(P, 1 << D, D, dtype=torch.float64, device=DEV)
        for e in range(D):
            poly = torch.zeros(D, P, 1 << D, dtype=torch.float64, device=DEV)  # by subset size
            poly[0] = 1.0
            used = 0
            for q in range(D):
                if q == e:
                    continue
                used += 1
                zq, oq = zz[:, q:q + 1], o_all[:, q][None]
                for k in range(min(used, D - 1), 0, -1):
                    poly[k] = poly[k] * zq + poly[k - 1] * oq
                poly[0] = poly[0] * zq
            total = sum(w[k] * poly[k] for k in range(D))
            tab[:, :, e] = lv[:, None] * (o_all[:, e][None] - zz[:, e:e + 1]) * total
        # each row's pattern on each path
        code = torch.zeros(P, n, dtype=torch.long, device=DEV)
        fi = torch.where(f < 0, Fc, f)
        for e in range(D):
            v = xt[fi[:, e]]
            o = torch.where(miss[fi[:, e]], ok_t[:, e:e + 1], (v >= lo_t[:, e:e + 1]) & (v < hi_t[:, e:e + 1]))
            code |= (o | (f[:, e:e + 1] < 0)).long() << e
        for e in range(D):
            out.index_add_(0, fi[:, e], torch.gather(tab[:, :, e], 1, code))
    out[Fc] = float(np.float32(0.1)) + sum(_mean(off, nodes))
    return out.t().contiguous()


def _mean(off, nodes):
    """Every tree's cover-weighted mean leaf value."""
    left, right = nodes["left"], nodes["right"]
    cover = nodes["sum_hess"].astype(np.float64)
    value = nodes["leaf_value"].astype(np.float64)
    for t in range(len(off) - 1):
        a = off[t]
        for i in range(off[t + 1] - 1, a - 1, -1):  # children come after their parent
            if left[i] >= 0:
                l, r = a + left[i], a + right[i]
                value[i] = (cover[l] * value[l] + cover[r] * value[r]) / cover[i]
    return value[off[:-1]]


def _exact_hist(case, seed):
    """Quantile cuts from sorted columns, bins, and the pairs' sums per bin in 64 bits."""
    g = _gen(seed)
    x, miss = _table(g, case["rows"], case["cols"], case["missing"])
    x = _holes(g, x, miss)
    rows, pairs = _hist_inputs(g, case)
    pairs = pairs.double()[rows]
    out = []
    for j in range(case["cols"]):
        col = x[:, j]
        v = torch.sort(col[~torch.isnan(col)]).values
        u = torch.unique_consecutive(v)
        if u.numel() > case["max_bin"]:
            b = torch.arange(1, case["max_bin"] + 1, device=DEV, dtype=torch.float64) / case["max_bin"]
            at = (torch.ceil(b * v.numel()).long().clamp_min(1) - 1).clamp_max(v.numel() - 1)
            u = torch.unique_consecutive(v[at])
        top = torch.nextafter(v[-1:], torch.full((1,), float("inf"), device=DEV))
        cuts = torch.cat([u, top])
        c = col[rows]
        here = ~torch.isnan(c)
        at = torch.searchsorted(cuts, c[here].contiguous(), right=True).clamp_max(cuts.numel() - 1)
        h = torch.zeros(cuts.numel(), 2, dtype=torch.float64, device=DEV)
        h.index_add_(0, at, pairs[here])
        out.append(h)
    return torch.cat(out)
