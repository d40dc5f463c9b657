"""The work that a user of this framework has it do, as cases that can be timed.

Each case is one use of the public Python API (dsgdpp_b200/__init__.py):

* ``fit``      a whole run on a loaded matrix: the factors go in, ``epochs`` epochs under
               BoldDriver with the training and the test loss after each (as ``mfdsgdpp``
               and the README run it), the factors come out: in page-locked buffers that the
               program keeps, as bench.py does, or in plain arrays (the quick start).
               Throughput epochs (FP32 and BF16 factors) and the exact FP64 replay of the
               sequential point order.
* ``tracked``  a user's own step rule, as dsgdpp_b200/controller.py runs its epochs: snapshot,
               epoch at a proposed step, loss and size of the update.
* ``losses``   the losses of given factors, without training.
* ``load``     host arrays to the device (blocking, counts) and the factors back.
* ``batch``    many small problems advanced together.
* ``propose``, ``gradient``  the step-size network: one forward pass per decision, and the
               gradient of a training batch.

Matrices are drawn on the GPU from the seed with the generators that the benchmark and the
controller's training use (dsgdpp_b200/synth_gpu.py).
"""
import math

import numpy as np
import torch

import dsgdpp_b200 as P
from dsgdpp_b200 import synth_gpu


def listed():
    return [
        # One decision of the step controller: the smallest call, all latency.
        dict(name="propose_1", kind="propose", batch=1),
        # One training batch of the controller network (dsgdpp_b200/controller.py: 256 states).
        dict(name="gradient_256", kind="gradient", batch=256),
        # The README's quick start, FP32: short epochs, where launches and latency count.
        _fit("quick_fp32", 100_000, 100_000, 1_000_000, 10, 4, "fp32", epochs=20, pinned=False),
        # The same in the exact FP64 mode, which repeats the reference's sequential order.
        _fit("quick_replay", 100_000, 100_000, 1_000_000, 10, 4, "fp64", mode="replay", epochs=1,
             pinned=False),
        # The headline workload: 2M x 500k, 100M entries, Zipf degrees, rank 32, L2; d as tuned.
        _fit("zipf_100m_fp32", 2_000_000, 500_000, 100_000_000, 32, 64, "fp32", zipf=1.1, l2=0.05,
             epochs=10),
        # Its 20M-entry form with BF16 factors at the rank of the 300M-entry workload.
        _fit("zipf_20m_bf16", 400_000, 100_000, 20_000_000, 64, 64, "bf16", zipf=1.1, l2=0.05,
             epochs=5),
        # Ratings of the Netflix shape (1..5, lognormal rows), a quarter of the entries, rank 128.
        _fit("ratings_25m_fp32", 480_189, 17_770, 25_000_000, 128, 64, "fp32", ratings=True,
             epochs=5),
        # DSGD, more columns than rows, ragged sizes, a rank that fills no whole vector.
        _fit("dsgd_3m_fp32", 60_011, 230_017, 3_000_000, 50, 12, "fp32", method="dsgd",
             update="Nzsl_Nzl2", loss="Nzsl_Nzl2", epochs=10),
        # A matrix of the controller's training family, stepped by the user's own rule.
        dict(name="tracked_2m_fp32", kind="tracked", m=90_000, n=30_000, nnz=2_000_000, rank=64,
             d=16, precision="fp32", zipf=1.1, l2=0.02, epochs=5, pinned=True),
        # The losses of given factors: how a model is judged on training and test entries.
        dict(name="losses_20m_fp32", kind="losses", m=400_000, n=100_000, nnz=20_000_000, rank=32,
             d=64, precision="fp32", zipf=1.1),
        # A matrix in host memory, as a reader leaves it, to blocked records on the device.
        dict(name="load_10m_fp32", kind="load", m=300_000, n=80_000, nnz=10_000_000, rank=16,
             d=32, precision="fp32", zipf=1.1),
        # Small problems of uneven sizes and ranks together (rows, columns and density log-uniform).
        dict(name="batch_24_fp32", kind="batch", count=24, precision="fp32", epochs=10),
    ]


def _fit(name, m, n, nnz, rank, d, precision, mode="hogwild", method="dsgdpp", zipf=0.0,
         ratings=False, l2=0.0, update="Nzsl_L2", loss="Nzsl_L2", epochs=5, pinned=True):
    return dict(name=name, kind="fit", m=m, n=n, nnz=nnz, rank=rank, d=d, precision=precision,
                mode=mode, method=method, zipf=zipf, ratings=ratings, l2=l2, update=update,
                loss=loss, epochs=epochs, pinned=pinned)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit"] * 6 + ["replay"] * 2 + ["tracked", "losses", "load", "batch",
                                                      "propose", "gradient"])
    if kind in ("propose", "gradient"):
        return dict(kind=kind, batch=_log(rng, 2, 2048))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(4, 28), epochs=rng.randint(4, 10),
                    precision=rng.choice(["fp32", "fp32", "bf16"]))
    m, n = _log(rng, 20_000, 600_000), _log(rng, 5_000, 200_000)
    zipf = rng.choice([0.0, 1.1, 1.1])
    if kind == "replay":
        nnz = min(_log(rng, 50_000, 1_000_000), m * n // 50)
        c = _fit("", m, n, nnz, rng.randint(4, 64), rng.randint(4, 32), "fp64", mode="replay",
                 zipf=zipf, l2=rng.choice([0.0, 0.05]), epochs=1,
                 update=rng.choice(["Nzsl", "Nzsl_L2", "Nzsl_Nzl2"]))
        del c["name"]
        return c
    # at most one entry in 50 cells: degree-weighted positions stay distinct
    nnz = min(_log(rng, 300_000, 20_000_000), m * n // 50)
    rank = _log(rng, 4, 128)
    d = max(2, min(128, int(nnz / 8000) or 1, _log(rng, 4, 128)))
    precision = rng.choice(["fp32", "fp32", "bf16"])
    if kind == "fit":
        c = _fit("", m, n, nnz, rank, d, precision, zipf=zipf, l2=rng.choice([0.0, 0.05]),
                 method=rng.choice(["dsgdpp", "dsgdpp", "dsgd"]), epochs=rng.randint(2, 8),
                 pinned=rng.random() < 0.75)
        c["update"] = c["loss"] = rng.choice(["Nzsl_L2", "Nzsl_L2", "Nzsl_Nzl2"])
        del c["name"]
        return c
    c = dict(kind=kind, m=m, n=n, nnz=nnz, rank=rank, d=d, precision=precision, zipf=zipf)
    if kind == "tracked":
        c.update(l2=rng.choice([0.0, 0.02, 0.05]), epochs=rng.randint(2, 6), pinned=True)
    return c


# ---- inputs ---------------------------------------------------------------------------------
def _test_size(nnz):
    return max(1000, nnz // 100)


def _data(c, seed):
    if c.get("ratings"):
        return synth_gpu.make_ratings(c["m"], c["n"], c["nnz"], _test_size(c["nnz"]), c["rank"],
                                      seed)
    s = c["zipf"] or None
    return synth_gpu.make(c["m"], c["n"], c["nnz"], _test_size(c["nnz"]),
                          rank_true=min(c["rank"], 32), r=c["rank"], noise=0.2 if s else 0.1,
                          seed=seed, s_row=s, s_col=s)


def _config(c):
    return P.Config(m=c["m"], n=c["n"], rank=c["rank"], d=c["d"], precision=c["precision"],
                    exec=c.get("mode", "hogwild"), method=c.get("method", "dsgdpp"),
                    launch="stream" if c.get("mode") == "replay" else "graph",
                    update=c.get("update", "Nzsl_L2"), loss=c.get("loss", "Nzsl_L2"),
                    regularize="L2" if c.get("l2") else "None",
                    regularize_lambda=c.get("l2", 0.0))


def _context(c, data):
    ctx = P.Context(_config(c))
    ctx.set_matrix(P.TRAIN, data["rows"], data["cols"], data["vals"])
    ctx.set_matrix(P.TEST, data["trows"], data["tcols"], data["tvals"])
    return ctx


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _batch_problems(c, seed):
    """Shapes as the batched benchmark draws them (dsgdpp_b200/batchbench.py), entries capped."""
    rng = np.random.default_rng(4)  # the sizes belong to the case, the entries to the seed
    out = []
    for k in range(c["count"]):
        m = int(round(math.exp(rng.uniform(math.log(1_000), math.log(200_000)))))
        n = int(round(math.exp(rng.uniform(math.log(1_000), math.log(50_000)))))
        density = math.exp(rng.uniform(math.log(1e-4), math.log(1e-2)))
        r = int(rng.choice([8, 16, 32, 64]))
        nnz = min(2_000_000, max(16, int(round(density * m * n))))
        out.append((m, n, nnz, r, seed * 1009 + 7919 * k))
    return out


def _mlp_arrays(c, seed):
    g = np.random.default_rng(seed)
    w = [g.standard_normal((64, 16)) / 4, g.standard_normal(64) / 10,
         g.standard_normal((64, 64)) / 8, g.standard_normal(64) / 10,
         g.standard_normal(64) / 8, g.standard_normal(1) / 10]
    params = np.concatenate([a.ravel() for a in w]).astype(np.float32)
    x = g.uniform(-2, 2, (c["batch"], P.Mlp.INPUTS)).astype(np.float32)
    y = g.uniform(-1, 1, c["batch"]).astype(np.float32)
    return params, x, y


def prepare(case, seed):
    c, kind = case, case["kind"]
    state = dict(case=c)
    if kind in ("propose", "gradient"):
        params, state["x"], state["y"] = _mlp_arrays(c, seed)
        state["mlp"] = P.Mlp()
        state["mlp"].params = params
        return state
    if kind == "batch":
        problems = []
        for k, (m, n, nnz, r, s) in enumerate(_batch_problems(c, seed)):
            a = synth_gpu.make(m, n, nnz, max(1, nnz // 100), rank_true=10, r=r, noise=0.1, seed=s)
            problems.append(dict(m=m, n=n, rank=r, rows=a["rows"], cols=a["cols"], vals=a["vals"],
                                 trows=a["trows"], tcols=a["tcols"], tvals=a["tvals"],
                                 W=a["W0"], H=a["H0"], seed=1000 + k, eps0=0.001))
        cfg = P.Config(m=1, n=1, rank=1, d=1, precision=c["precision"], regularize="L2",
                       regularize_lambda=0.02)
        state["batch"] = P.Batch(cfg, problems)
        return state
    data = _data(c, seed)
    if kind == "load":
        state.update(data=data, ctx=P.Context(_config(c)))
        return state
    state["ctx"] = _context(c, data)
    W, H = data["W0"], data["H0"]
    if c.get("pinned"):
        W, H = _pinned(W), _pinned(H)
        state["out"] = (torch.empty(W.shape, dtype=torch.float64, pin_memory=True).numpy(),
                        torch.empty(H.shape, dtype=torch.float64, pin_memory=True).numpy())
    if kind == "losses":
        state["ctx"].set_factors(W, H)
    else:
        state.update(W=W, H=H)
    return state


# ---- one pass -------------------------------------------------------------------------------
def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "propose":
        return state["mlp"].forward(state["x"])
    if kind == "gradient":
        return state["mlp"].gradient(state["x"], state["y"])
    if kind == "batch":
        b = state["batch"]
        train, test, _ = b.run(c["epochs"], decrease=1.0, increase=1.0)
        return train, test, [b.get_factors(k) for k in range(c["count"])]
    ctx = state["ctx"]
    if kind == "losses":
        return [ctx.loss(), ctx.nzsl(P.TEST), ctx.l2(), ctx.nzl2()]
    if kind == "load":
        d = state["data"]
        ctx.set_matrix(P.TRAIN, d["rows"], d["cols"], d["vals"])
        ctx.set_matrix(P.TEST, d["trows"], d["tcols"], d["tvals"])
        ctx.set_factors(d["W0"], d["H0"])
        nnz1, nnz2, top = ctx.nnz12()
        return [ctx.block_nnz(), nnz1.astype(np.int64), nnz2.astype(np.int64), top,
                ctx.get_factors()]
    ctx.set_factors(state["W"], state["H"])
    ctx.seed(1)
    if kind == "tracked":
        told, eps = [], 0.001
        for _ in range(c["epochs"]):
            ctx.save_factors()
            ctx.epoch(eps)
            told.append([ctx.loss(), ctx.nzsl(P.TEST), *ctx.update_norms()])
            eps *= 1.5
        return [np.array(told), _factors(state)]
    trace = ctx.run(c["epochs"], "BoldDriver", 0.001)
    told = np.array([[t["loss"], t["test_loss"]] for t in trace])
    return [told, _factors(state)]


def _factors(state):
    if "out" not in state:
        return state["ctx"].get_factors()
    state["ctx"].get_factors_into(*state["out"])
    return state["out"]


# ---- what a pass cannot do without, and its results in 64 bits ------------------------------
def work(case):
    c, kind = case, case["kind"]
    if kind in ("propose", "gradient"):
        macs = 16 * 64 + 64 * 64 + 64
        times = 1 if kind == "propose" else 3
        return {"bytes": 4 * (5313 * (1 if times == 1 else 2) + 17 * c["batch"]),
                "flops": 2 * macs * times * c["batch"]}
    size = {"fp64": 8, "fp32": 4, "bf16": 2}[c["precision"]]
    shapes = ([s[:4] for s in _batch_problems(c, 0)] if kind == "batch"
              else [(c["m"], c["n"], c["nnz"], c["rank"])])
    total = {"bytes": 0, "flops": 0}
    for m, n, nnz, r in shapes:
        entry = 8 + (8 if c["precision"] == "fp64" else 4)
        factors, host = (m + n) * r * size, (m + n) * r * 8
        test = nnz // 100
        loss = (nnz + test) * entry + factors
        if kind == "losses":
            total["bytes"] += loss
            total["flops"] += (nnz + test) * 2 * r + 4 * (m + n) * r
        elif kind == "load":
            total["bytes"] += (nnz + test) * (16 + entry) + 2 * host + 2 * factors
        else:
            epoch = nnz * entry + 2 * factors + 4 * (m + n) + loss
            total["bytes"] += c["epochs"] * epoch + 2 * host
            total["flops"] += c["epochs"] * (8 * nnz * r + 2 * (nnz + test) * r)
    return total


def _net(params, x):
    w1, b1, w2, b2, w3, b3 = torch.split(params, [64 * 16, 64, 64 * 64, 64, 64, 1])
    gelu = torch.nn.functional.gelu
    h = gelu(x @ w1.view(64, 16).T + b1)
    return gelu(h @ w2.view(64, 64).T + b2) @ w3 + b3


def _squared_error(rows, cols, vals, W, H):
    total = 0.0
    for a in range(0, len(vals), 2_000_000):
        i, j, x = (torch.from_numpy(v[a:a + 2_000_000].astype(t)).cuda()
                   for v, t in ((rows, np.int64), (cols, np.int64), (vals, np.float64)))
        total += float((x - (W[i] * H[j]).sum(1)).square().sum())
    return total


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("propose", "gradient"):
        params, x, y = (torch.from_numpy(a.astype(np.float64)) for a in _mlp_arrays(c, seed))
        if kind == "propose":
            return _net(params, x).clamp(-1, 1).numpy()
        params.requires_grad_()
        loss = (_net(params, x) - y).square().mean()
        loss.backward()
        return float(loss.detach()), params.grad.numpy()
    if kind not in ("losses", "load"):
        return None  # the order of concurrent updates is not fixed; a replay is compared as it is
    d = _data(c, seed)
    if kind == "load":
        return [None, None, None, None, (d["W0"], d["H0"])]
    # the stored form of the inputs: values in FP32, factors in the precision of the case
    store = torch.bfloat16 if c["precision"] == "bf16" else torch.float32
    W, H = (torch.from_numpy(d[k]).cuda().to(store).double() for k in ("W0", "H0"))
    val, tval = (d[k].astype(np.float32) for k in ("vals", "tvals"))
    n1, n2 = (torch.from_numpy(np.bincount(d[k], minlength=s).astype(np.float64)).cuda()
              for k, s in (("rows", c["m"]), ("cols", c["n"])))
    w2, h2 = W.square().sum(1), H.square().sum(1)
    l2 = (float(w2.sum()), float(h2.sum()))
    return [_squared_error(d["rows"], d["cols"], val, W, H) + l2[0] + l2[1],
            _squared_error(d["trows"], d["tcols"], tval, W, H), l2,
            (float((n1 * w2).sum()), float((n2 * h2).sum()))]
