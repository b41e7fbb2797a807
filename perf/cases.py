"""The fitter's work as its users call it, as cases that can be timed and compared.

Every case goes through the public entry points with new inputs made from a
seed: the per-voxel Levenberg-Marquardt fit from one region of interest to a
whole volume, in each state and solve precision; the IVIM notebook's flow
(segmented start, per-voxel bounds); mixed models in one launch; the
warm-started fit on the device and streamed from host memory; the training of
its network; the multi-start search.

``exact`` restates the same computations in 64 bits in plain torch (the LM of
pycompute/cuda/lsqnonlin.py:823-924 with the GMW81 solve of
pycompute/cuda/solver.py:23-95, all in double).
"""
import functools
import io
import math

import numpy as np
import torch

NAN = float("nan")


def _linspace(lo, hi, n):
    return [lo + (hi - lo) * i / (n - 1) for i in range(n)]


_IVIM = dict(expr="S0*(f*exp(-b*D_1)+(1-f)*exp(-b*D_2))", pars=["S0", "f", "D_1", "D_2"], consts=["b"],
             ranges=[(500.0, 1500.0), (0.05, 0.35), (5e-3, 5e-2), (0.5e-3, 2.5e-3)], snr=(50.0, 50.0),
             lb=[0.0, 1e-3, 1e-6, 1e-8], ub=[20000.0, 0.999, 0.1, 0.02], init=[NAN, 0.1, 1e-2, 1e-3], form="ivim")
# the package's own workloads: protocol, ranges of the true parameters, bounds, start (NaN: the largest sample), noise
MODELS = {
    "ivim10": dict(_IVIM, protocol=[0, 10, 20, 50, 100, 200, 400, 600, 800, 1000]),
    "ivim16": dict(_IVIM, protocol=[0.0] + [10.0 * 100.0 ** (i / 14) for i in range(15)]),
    "ivim21": dict(_IVIM, protocol=[0, 10, 20, 30, 40, 50, 60, 70, 80, 90, 100, 120, 140, 160, 180, 200, 300, 400, 500,
                                    600, 1000]),
    "vfa8": dict(expr="S0*sin(a)*(1-exp(-15/T1))/(1-cos(a)*exp(-15/T1))", pars=["S0", "T1"], consts=["a"],
                 protocol=[math.radians(x) for x in _linspace(2.0, 30.0, 8)], ranges=[(500.0, 1500.0), (300.0, 3000.0)],
                 lb=[0.0, 10.0], ub=[50000.0, 10000.0], snr=(30.0, 100.0), init=[NAN, 1000.0], form="vfa"),
    "t2s16": dict(expr="S0*exp(-TE*R2s/1000)+c", pars=["S0", "R2s", "c"], consts=["TE"],
                  protocol=_linspace(2.0, 40.0, 16), ranges=[(500.0, 1500.0), (10.0, 200.0), (0.0, 50.0)],
                  lb=[0.0, 0.0, -1000.0], ub=[50000.0, 1000.0, 1000.0], snr=(30.0, 100.0), init=[NAN, 50.0, 0.0],
                  form="t2s"),
    "biexp32": dict(expr="S0*(f*exp(-TE/T2s)+(1-f)*exp(-TE/T2l))+c", pars=["S0", "f", "T2s", "T2l", "c"],
                    consts=["TE"], protocol=_linspace(10.0, 320.0, 32),
                    ranges=[(500.0, 1500.0), (0.1, 0.5), (10.0, 40.0), (60.0, 300.0), (0.0, 50.0)],
                    lb=[0.0, 0.0, 1.0, 20.0, -1000.0], ub=[50000.0, 1.0, 60.0, 2000.0, 1000.0], snr=(30.0, 100.0),
                    init=[NAN, 0.3, 20.0, 100.0, 0.0], form="biexp"),
}
MIXED = ("vfa8", "t2s16", "ivim10", "biexp32")
LOW_ROWS, HIGH_ROWS = (0, 11), (15, 21)  # b <= 100 and b >= 200 of the 21-value protocol: the segmented start's two fits


def listed():
    return [
        # one region of interest, fitted by itself: launches and latency count
        {"name": "roi", "kind": "fit", "model": "ivim10", "n": 300, "iters": 50, "dtype": "f32", "solve": "f64"},
        # one slab of a scan (32 x 32 x 16), the reference's iteration limit: too few voxels to fill the GPU
        {"name": "slab", "kind": "fit", "model": "ivim10", "n": 16384, "iters": 100, "dtype": "f32", "solve": "f64"},
        # a whole 256 x 256 x 128 volume, the same fit
        {"name": "volume", "kind": "fit", "model": "ivim10", "n": 8388608, "iters": 100, "dtype": "f32",
         "solve": "f64"},
        # five parameters, 32 echoes, the reference's all-fp32 arithmetic, a masked (ragged) voxel count
        {"name": "biexp fp32 solve", "kind": "fit", "model": "biexp32", "n": 300007, "iters": 40, "dtype": "f32",
         "solve": "f32"},
        # the double-precision fitter, where fp32 does not resolve a model or as the error reference of other fits
        {"name": "double", "kind": "fit", "model": "ivim10", "n": 65536, "iters": 40, "dtype": "f64", "solve": "f64"},
        # the IVIM notebook: segmented start, protocol tiled per voxel, data-driven bounds, run(50, 1e-10)
        {"name": "notebook", "kind": "notebook", "n": 53217, "iters": 50},
        # four models of a quantitative protocol in one persistent launch
        {"name": "mixed models", "kind": "mixed", "n": 262147, "iters": 100},
        # the warm-started fit of a large volume (network, 2 iterations, fallback) ...
        {"name": "warm start", "kind": "warm", "n": 16777216},
        # ... of one slice ...
        {"name": "warm start slice", "kind": "warm", "n": 50021},
        # ... and of a series of volumes that live in host memory
        {"name": "warm start from host", "kind": "stream", "n": 1000003, "volumes": 4},
        # training the warm start's network on a protocol's simulated signals
        {"name": "train network", "kind": "train", "n": 262144, "batch": 8192, "epochs": 2},
        # multi-start fit: every draw refined by 20 LM iterations
        {"name": "multi-start", "kind": "search", "n": 16001, "draws": 10, "iters": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("fit", "fit", "fit", "fit", "fit", "notebook", "mixed", "warm", "stream", "train", "search"))
    if kind == "fit":
        model = rng.choice(sorted(MODELS))
        dtype, solve = rng.choice((("f32", "f64"), ("f32", "f64"), ("f32", "f32"), ("f64", "f64")))
        iters = _log_int(rng, 3, 100)
        # at most the work of the listed volume (8.4 M voxels x 100 iterations x 10 samples); double costs far more
        most = (2e8 if dtype == "f64" else 3e9) / (iters * len(MODELS[model]["protocol"]))
        n = _log_int(rng, 200, max(400, min(8388608, most)))
        return {"kind": kind, "model": model, "n": n, "iters": iters, "dtype": dtype, "solve": solve}
    if kind == "notebook":
        return {"kind": kind, "n": _log_int(rng, 2000, 400000), "iters": _log_int(rng, 10, 80)}
    if kind == "mixed":
        return {"kind": kind, "n": _log_int(rng, 3000, 400000), "iters": _log_int(rng, 10, 100)}
    if kind == "warm":
        return {"kind": kind, "n": _log_int(rng, 3000, 16777216)}
    if kind == "stream":
        return {"kind": kind, "n": _log_int(rng, 30000, 1500000), "volumes": rng.randint(2, 5)}
    if kind == "train":
        batch = rng.choice((1024, 2048, 4096, 8192))
        return {"kind": kind, "n": batch * rng.randint(4, 32) + rng.randint(1, 900), "batch": batch,
                "epochs": rng.randint(1, 3)}
    return {"kind": kind, "n": _log_int(rng, 1000, 60000), "draws": rng.randint(3, 12), "iters": rng.randint(8, 25)}


# ---- inputs -------------------------------------------------------------------


def _model_value(form, p, c):
    if form == "ivim":
        return p[0] * (p[1] * torch.exp(-c * p[2]) + (1 - p[1]) * torch.exp(-c * p[3]))
    if form == "vfa":
        e = torch.exp(-15.0 / p[1])
        return p[0] * torch.sin(c) * (1 - e) / (1 - torch.cos(c) * e)
    if form == "t2s":
        return p[0] * torch.exp(-c * p[1] / 1000) + p[2]
    return p[0] * (p[1] * torch.exp(-c / p[2]) + (1 - p[1]) * torch.exp(-c / p[3])) + p[4]


def _signals(model, n, seed, device="cuda"):
    """(true parameters (P, n), signals (M, n)) fp32: uniform parameters, Rician noise of sigma = S0 / SNR."""
    m = MODELS[model]
    g = torch.Generator(device=device).manual_seed(seed * 1000003 + n)
    u = lambda lo, hi: torch.rand(n, generator=g, device=device) * (hi - lo) + lo  # noqa: E731
    true = torch.stack([u(lo, hi) for lo, hi in m["ranges"]])
    sigma = true[0] / u(*m["snr"])
    rows = []
    for c in m["protocol"]:
        s = _model_value(m["form"], true, torch.tensor(float(c), device=device))
        n1 = torch.randn(n, generator=g, device=device)
        n2 = torch.randn(n, generator=g, device=device)
        rows.append(torch.sqrt((s + sigma * n1) ** 2 + (sigma * n2) ** 2))
    return true, torch.stack(rows)


def _start(model, data):
    smax = data.max(dim=0).values
    return torch.stack([smax if math.isnan(v) else torch.full_like(smax, v) for v in MODELS[model]["init"]])


def _fit_inputs(case, seed):
    dt = torch.float64 if case["dtype"] == "f64" else torch.float32
    _, data = _signals(case["model"], case["n"], seed)
    data = data.to(dt)
    m = MODELS[case["model"]]
    t = lambda v: torch.tensor(v, dtype=dt, device="cuda")  # noqa: E731
    return data, _start(case["model"], data), t([float(x) for x in m["protocol"]]), t(m["lb"]), t(m["ub"])


@functools.lru_cache(maxsize=1)
def _network():
    """Weights of a warm-start network for the 16-value protocol, as a user loads them from a file: 16 -> 128 -> 128 ->
    128 -> 4, trained here in plain torch on simulated signals (the same ones for every seed of the inputs)."""
    true, sig = _signals("ivim16", 262144, 9176)
    smax = sig.max(dim=0).values
    x = torch.log((sig / smax).clamp_min(1e-6)).T.contiguous()
    y = torch.stack([true[0] / smax, true[1], torch.log(true[2]), torch.log(true[3])], 1)
    mean, std = y.mean(0), y.std(0)
    y = (y - mean) / std
    g = torch.Generator().manual_seed(41)
    dims = [(16, 128), (128, 128), (128, 128), (128, 4)]
    ws = [((torch.rand(o, i, generator=g) * 2 - 1) * (6.0 / i) ** 0.5 * (0.5 if o == 4 else 1.0)).cuda()
          for i, o in dims]
    ps = ws + [torch.zeros(o, device="cuda") for _, o in dims]
    for p in ps:
        p.requires_grad_(True)
    opt = torch.optim.Adam(ps, lr=4e-3)
    steps, batch = 512, 8192
    for s in range(steps):
        opt.param_groups[0]["lr"] = 2e-3 * (1 + math.cos(math.pi * s / steps))
        b = s % (len(x) // batch) * batch
        h = x[b:b + batch]
        for k in range(4):
            h = torch.nn.functional.linear(h, ps[k], ps[4 + k])
            if k < 3:
                h = torch.nn.functional.gelu(h, approximate="tanh")
        loss = ((h - y[b:b + batch]) ** 2).mean()
        opt.zero_grad(set_to_none=True)
        loss.backward()
        opt.step()
    return [(w.detach().cpu().numpy(), b.detach().cpu().numpy()) for w, b in zip(ps[:4], ps[4:])], \
        mean.cpu().numpy(), std.cpu().numpy()


def _load_network():
    from pycompute_gb300.warmstart import WarmStartMLP

    layers, mean, std = _network()
    m = MODELS["ivim16"]
    d = {"nin": 16, "nout": 4, "log_in": 1, "kinds": np.array([0, 1, 2, 2]), "lb": np.array(m["lb"]),
         "ub": np.array(m["ub"]), "mean": mean, "std": std, "step": 512}
    for k, (w, b) in enumerate(layers):
        a = np.zeros(((w.shape[0] + 7) // 8 * 8, w.shape[1] + 8), np.float32)
        a[:w.shape[0], :w.shape[1]] = w
        a[:w.shape[0], w.shape[1]] = b
        d["w%d" % k] = a
    f = io.BytesIO()
    np.savez(f, **d)
    f.seek(0)
    return WarmStartMLP.load(f, "cuda")


def _workload(model):
    from pycompute_gb300.synth import Workload

    m = MODELS[model]
    return Workload(name=model, expr=m["expr"], pars=list(m["pars"]), consts=list(m["consts"]),
                    protocol=[float(x) for x in m["protocol"]], ranges=list(m["ranges"]), lb=list(m["lb"]),
                    ub=list(m["ub"]), snr=m["snr"], init_values=list(m["init"]))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "fit":
        from pycompute_gb300 import Expr, SecondOrderLevenbergMarquardt

        m = MODELS[case["model"]]
        dt = torch.float64 if case["dtype"] == "f64" else torch.float32
        s["data"], s["init"], s["prot"], s["lb"], s["ub"] = _fit_inputs(case, seed)
        s["solm"] = SecondOrderLevenbergMarquardt(
            Expr(m["expr"], m["pars"], m["consts"]), None, len(m["protocol"]), dt,
            solve_dtype=torch.float64 if case["solve"] == "f64" else torch.float32)
    elif kind == "notebook":
        from pycompute_gb300 import SecondOrderLevenbergMarquardt

        m = MODELS["ivim21"]
        s["data"] = _signals("ivim21", case["n"], seed)[1]
        b = torch.tensor([float(x) for x in m["protocol"]], device="cuda")
        s["consts"] = b[:, None].expand(len(b), case["n"]).contiguous()
        s["solm"] = SecondOrderLevenbergMarquardt(m["expr"], m["pars"], m["consts"], ndata=21, dtype=torch.float32)
    elif kind == "mixed":
        from pycompute_gb300 import Expr
        from pycompute_gb300.multi import MultiJob, MultiModelFitter

        ms = [MODELS[k] for k in MIXED]
        s["fitter"] = MultiModelFitter([(Expr(m["expr"], m["pars"], m["consts"]), len(m["protocol"])) for m in ms])
        s["jobs"], s["inits"] = [], []
        for j, k in enumerate(MIXED):
            data = _signals(k, case["n"] + 31 * j, seed)[1]
            s["inits"].append(_start(k, data))
            m = MODELS[k]
            s["jobs"].append(MultiJob(s["inits"][-1].clone(), data, m["protocol"], m["lb"], m["ub"]))
        s["fitter"].build()
    elif kind in ("warm", "stream"):
        from pycompute_gb300.pipeline import WarmStartFitter

        s["fitter"] = WarmStartFitter(_workload("ivim16"), _load_network())
        if kind == "warm":
            s["data"] = _signals("ivim16", case["n"], seed)[1]
            s["pars"] = torch.empty((4, case["n"]), device="cuda")
        else:
            s["volumes"] = []
            for v in range(case["volumes"]):
                data = _signals("ivim16", case["n"], seed * 16 + v)[1]
                host = torch.empty(data.shape, pin_memory=True)
                host.copy_(data)
                s["volumes"].append((host, torch.empty((4, case["n"]), pin_memory=True)))
    elif kind == "train":
        s["labels"], s["data"] = _signals("ivim16", case["n"], seed)
        s["seed"] = seed % 1000
    else:
        from pycompute_gb300 import SecondOrderRandomSearch

        m = MODELS["ivim21"]
        s["data"] = _signals("ivim21", case["n"], seed)[1]
        t = lambda v: torch.tensor([float(x) for x in v], device="cuda")  # noqa: E731
        s["prot"], s["lb"], s["ub"] = t(m["protocol"]), t(m["lb"]), t(m["ub"])
        s["search"] = SecondOrderRandomSearch(m["expr"], m["pars"], m["consts"], 21, torch.float32)
        s["seed"] = seed
    return s


# ---- one pass -----------------------------------------------------------------


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "fit":
        solm, pars = s["solm"], s["init"].clone()
        solm.setup(pars, s["prot"], s["data"], s["lb"], s["ub"])
        solm.run(case["iters"])
        return {"pars": pars, "first_f": solm.first_f, "last_f": solm.last_f, "lam": solm.lam_t,
                "step_type": solm.step_type_t}
    if kind == "notebook":
        from pycompute_gb300.pipeline import ivim_segmented_init

        m = MODELS["ivim21"]
        pars, lb, ub = ivim_segmented_init(s["data"], m["protocol"], LOW_ROWS, HIGH_ROWS, m["lb"], m["ub"])
        solm = s["solm"]
        solm.setup(pars, s["consts"], s["data"], lb, ub)
        solm.run(case["iters"], 1e-10)
        return {"pars": pars, "first_f": solm.first_f, "last_f": solm.last_f, "step_type": solm.step_type_t,
                "lower": lb, "upper": ub}
    if kind == "mixed":
        for j, p0 in zip(s["jobs"], s["inits"]):
            j.reset(p0)
        s["fitter"].fit(s["jobs"], case["iters"])
        return [{"pars": j.pars, "first_f": j.first_f, "last_f": j.last_f, "step_type": j.step_type}
                for j in s["jobs"]]
    if kind == "warm":
        r = s["fitter"].fit(s["data"], iters_warm=2, iters_fallback=8, pars_out=s["pars"], lam0=3e-3)
        return {"pars": r.pars, "step_type": r.step_type, "counts": r.counts}
    if kind == "stream":
        counts = s["fitter"].fit_stream(s["volumes"], iters_warm=2, iters_fallback=8, lam0=3e-3)
        return {"pars": [out for _, out in s["volumes"]], "counts": counts}
    if kind == "train":
        from pycompute_gb300.warmstart import WarmStartMLP

        m = MODELS["ivim16"]
        net = WarmStartMLP(16, 4, [0, 1, 2, 2], m["lb"], m["ub"], "cuda", seed=s["seed"])
        net.train(s["data"], s["labels"], epochs=case["epochs"], batch=case["batch"], lr=2e-3)
        return {"weights": [layer.master for layer in net.layers], "loss": net.loss_sum}
    rs = s["search"]
    rs.setup(s["prot"], s["data"], s["lb"], s["ub"])
    rs.run(case["draws"], lm_iters=case["iters"], seed=s["seed"])
    return {"best_pars": rs.best_pars_t, "best_f": rs.best_f_t}


# ---- what a pass cannot do without ----------------------------------------------


def _lm_work(model, n, iters, state_bytes=4):
    """Signals and start in, parameters and state out; per sample of an iteration the model twice (8 operations for an
    exponential and its argument), its derivatives, residual and the accumulation of f, J^T r and the two Hessians;
    per iteration the LDL^T solve and the predicted reduction."""
    m = MODELS[model]
    M, P = len(m["protocol"]), len(m["pars"])
    H = P * (P + 1) // 2
    nexp = {"ivim": 2, "biexp": 2, "t2s": 1, "vfa": 1}[m["form"]]
    sample = 2 * (8 * nexp + 6) + 2 * P + 2 * H + 4 + 2 * P + 4 * H + 3 * P
    solve = P ** 3 / 3 + 5 * P * P + 4 * H
    return state_bytes * n * (M + 2 * P + 3) + n, float(n) * iters * (M * sample + solve)


def work(case):
    kind, n = case["kind"], case["n"]
    net = 2 * (16 * 128 + 2 * 128 * 128 + 128 * 4)
    if kind == "fit":
        b, f = _lm_work(case["model"], n, case["iters"], 8 if case["dtype"] == "f64" else 4)
    elif kind == "notebook":
        b, f = _lm_work("ivim21", n, case["iters"])
        b += 4 * n * (21 + 2 * 4)
    elif kind == "mixed":
        b = f = 0
        for j, k in enumerate(MIXED):
            x = _lm_work(k, n + 31 * j, case["iters"])
            b, f = b + x[0], f + x[1]
    elif kind in ("warm", "stream"):
        v = n * case.get("volumes", 1)
        b, f = v * (16 * 4 + 4 * 4 + (1 if kind == "warm" else 0)), v * net + _lm_work("ivim16", v, 2)[1]
    elif kind == "train":
        steps = n // case["batch"] * case["epochs"]
        b, f = n * 20 * 4 + 2 * 4 * 36000, 3.0 * net * case["batch"] * steps
    else:
        b, f = _lm_work("ivim21", n, case["iters"] * case["draws"])
    return {"bytes": float(b), "flops": float(f)}


# ---- the same in 64 bits --------------------------------------------------------


def _derivatives(form, p, c):
    """m, [dm/dp_k], {(i, j): d2m/dp_i dp_j, j <= i} (structural zeros left out); p[k] (n,), c (M, 1) or (M, n)."""
    if form == "ivim":
        s0, f, d1, d2 = p
        e1, e2 = torch.exp(-c * d1), torch.exp(-c * d2)
        m0 = f * e1 + (1 - f) * e2
        return s0 * m0, [m0, s0 * (e1 - e2), -c * s0 * f * e1, -c * s0 * (1 - f) * e2], {
            (1, 0): e1 - e2, (2, 0): -c * f * e1, (2, 1): -c * s0 * e1, (2, 2): c * c * s0 * f * e1,
            (3, 0): -c * (1 - f) * e2, (3, 1): c * s0 * e2, (3, 3): c * c * s0 * (1 - f) * e2}
    if form == "vfa":
        s0, t1 = p
        e = torch.exp(-15.0 / t1)
        de, dde = 15.0 / t1 ** 2 * e, (225.0 / t1 ** 4 - 30.0 / t1 ** 3) * e
        q, co = 1 - torch.cos(c) * e, torch.cos(c)
        a = torch.sin(c)
        m0 = a * (1 - e) / q
        dm = a * (co - 1) / q ** 2            # d m0 / d e
        ddm = 2 * a * (co - 1) * co / q ** 3  # d2 m0 / d e2
        return s0 * m0, [m0, s0 * dm * de], {(1, 0): dm * de, (1, 1): s0 * (ddm * de * de + dm * dde)}
    if form == "t2s":
        s0, r, o = p
        k = -c / 1000
        e = torch.exp(k * r)
        return s0 * e + o, [e, s0 * k * e, torch.ones_like(e)], {(1, 0): k * e, (1, 1): s0 * k * k * e}
    s0, f, ts, tl, o = p
    e1, e2 = torch.exp(-c / ts), torch.exp(-c / tl)
    g1, g2 = c / ts ** 2 * e1, c / tl ** 2 * e2
    h1, h2 = (c * c / ts ** 4 - 2 * c / ts ** 3) * e1, (c * c / tl ** 4 - 2 * c / tl ** 3) * e2
    m0 = f * e1 + (1 - f) * e2
    return s0 * m0 + o, [m0, s0 * (e1 - e2), s0 * f * g1, s0 * (1 - f) * g2, torch.ones_like(e1)], {
        (1, 0): e1 - e2, (2, 0): f * g1, (2, 1): s0 * g1, (2, 2): s0 * f * h1, (3, 0): (1 - f) * g2,
        (3, 1): -s0 * g2, (3, 3): s0 * (1 - f) * h2}


def _gmw81(A, b):
    """Solve with the modified LDL^T: A {(i, j): (n,), j <= i}, b [(n,)]; rotated by one, Jacobi-scaled."""
    P = len(b)
    rot = [P - 1] + list(range(P - 1))
    get = lambda i, j: A[(i, j)] if i >= j else A[(j, i)]  # noqa: E731
    L = {(i, j): get(rot[i], rot[j]) for i in range(P) for j in range(i + 1)}
    s = [torch.sqrt(L[(i, i)].abs()) for i in range(P)]
    r = [b[rot[i]] / s[i] for i in range(P)]
    for i in range(P):
        for j in range(i + 1):
            L[(i, j)] = L[(i, j)] / (s[i] * s[j])
    zero = torch.zeros_like(s[0])
    gam, nu = zero, zero
    for (i, j), v in L.items():
        if i == j:
            gam = torch.maximum(gam, v.abs())
        else:
            nu = torch.maximum(nu, v.abs())
    nu = nu / math.sqrt(max(1, P * P - 1))
    beta2 = torch.clamp_min(torch.maximum(gam, nu), 4e-16)
    delta = 4e-16 * torch.clamp_min(gam + nu, 1.0)
    D = []
    for j in range(P):
        for q in range(j):
            L[(j, q)] = L[(j, q)] / D[q]
        th = zero
        for i in range(j + 1, P):
            for q in range(j):
                L[(i, j)] = L[(i, j)] - L[(j, q)] * L[(i, q)]
            th = torch.maximum(th, L[(i, j)].abs())
        D.append(torch.maximum(torch.maximum(L[(j, j)].abs(), delta), th * th / beta2))
        for i in range(j + 1, P):
            L[(i, i)] = L[(i, i)] - L[(i, j)] ** 2 / D[j]
    y = []
    for i in range(P):
        t = r[i]
        for j in range(i):
            t = t - L[(i, j)] * D[j] * y[j]
        y.append(t / D[i])
    for i in reversed(range(P)):
        for j in range(i + 1, P):
            y[i] = y[i] - L[(j, i)] * y[j]
    x = [None] * P
    for i in range(P):
        x[rot[i]] = y[i] / s[i]
    return x


def _lm64(form, prot, p, data, lb, ub, iters, tol=1e-8, lam=5.0):
    """The LM in double; returns p, first and last cost, damping, step codes, cost at p. lb, ub: lists of floats or
    (n,) rows."""
    P, n = p.shape
    c = torch.as_tensor(prot, dtype=torch.float64, device=data.device).reshape(-1, 1)
    lb = [torch.as_tensor(v, dtype=torch.float64, device=data.device) for v in lb]
    ub = [torch.as_tensor(v, dtype=torch.float64, device=data.device) for v in ub]
    lam = torch.full((n,), float(lam), dtype=torch.float64, device=data.device)
    st = torch.ones(n, dtype=torch.int64, device=data.device)
    first, last = torch.zeros_like(lam), torch.zeros_like(lam)
    for it in range(iters):
        act = st != 0
        if not bool(act.any()):
            break
        m, J, H2 = _derivatives(form, list(p), c)
        r = m - data
        f = (r * r).sum(0)
        g = [(Jk * r).sum(0) for Jk in J]
        h, hd = {}, []
        for i in range(P):
            for j in range(i + 1):
                jt = J[i] * J[j]
                hj = jt + H2[(i, j)] * r if (i, j) in H2 else jt
                h[(i, j)] = hj.sum(0)
                if i == j:
                    hd.append((hj + torch.clamp_min(lam * jt, 1e-4)).sum(0))
        first = f if it == 0 else first
        last = torch.where(act, f, last)
        step = _gmw81({(i, j): hd[i] if i == j else h[(i, j)] for i in range(P) for j in range(i + 1)}, g)
        step = [torch.where(torch.isfinite(x), x, torch.zeros_like(x)) for x in step]
        clamped = torch.zeros_like(act)
        nrm = torch.zeros_like(f)
        for k in range(P):
            t = p[k] - g[k]
            clamped = clamped | (t > ub[k]) | (t < lb[k])
            nrm = nrm + (p[k] - torch.minimum(torch.maximum(t, lb[k]), ub[k])) ** 2
        conv = act & (nrm < tol * (1 + f)) & (((st & 1) != 0) | clamped)
        st = torch.where(conv, torch.zeros_like(st), st)
        go = act & ~conv
        pt = torch.stack([p[k] - step[k] for k in range(P)])
        ftp = ((_model_value(form, list(pt), c) - data) ** 2).sum(0)
        actual = 0.5 * (f - ftp)
        pred = torch.zeros_like(f)
        for (i, j), v in h.items():
            pred = pred - v * step[i] * step[j] * (0.5 if i == j else 1.0)
        for k in range(P):
            pred = pred + step[k] * g[k]
        rho = actual / pred
        accept = go & (rho > 0.25) & (actual > 0)
        very = rho > 0.75
        lam = torch.where(go, torch.where(accept, torch.where(very, lam * 0.2, lam), lam * 2), lam)
        st = torch.where(go, torch.where(accept, torch.where(very, 1, 2), 4), st)
        neg = go & (pred < 0)
        lam = torch.where(neg, lam * 2, lam)
        st = torch.where(neg, st | 8, st)
        p = torch.where(accept, pt, p)
        q = torch.stack([torch.minimum(torch.maximum(p[k], lb[k]), ub[k]) for k in range(P)])
        p = torch.where(go, q, p)
    return p, first, last, lam, st


def _chunks(n, size=1 << 20):
    return [(a, min(n, a + size)) for a in range(0, n, size)]


def _cost64(form, prot, p, data):
    c = torch.as_tensor(prot, dtype=torch.float64, device=data.device).reshape(-1, 1)
    return ((_model_value(form, list(p), c) - data) ** 2).sum(0)


def _gelu64(z):
    return 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))


def _warm64(data):
    """Network start, 2 iterations from damping 3e-3, refit of flagged voxels from the constant start, lower cost."""
    m = MODELS["ivim16"]
    layers, mean, std = _network()
    t = lambda a: torch.as_tensor(a, device=data.device).double()  # noqa: E731
    lb, ub = t(m["lb"])[:, None], t(m["ub"])[:, None]
    out = []
    for a, b in _chunks(data.shape[1], 1 << 19):
        d = data[:, a:b].double()
        smax = d.max(dim=0).values
        h = torch.log((d / smax).clamp_min(1e-6)).T
        for k, (w, bias) in enumerate(layers):
            h = h @ t(w).T + t(bias)
            h = _gelu64(h) if k < 3 else h
        y = h * t(std) + t(mean)
        p = torch.stack([y[:, 0] * smax, y[:, 1], torch.exp(y[:, 2]), torch.exp(y[:, 3])])
        p = torch.minimum(torch.maximum(p, lb), ub)
        p = _lm64("ivim", m["protocol"], p, d, m["lb"], m["ub"], 2, lam=3e-3)[0]
        p0 = torch.stack([smax if math.isnan(v) else torch.full_like(smax, v) for v in m["init"]])
        c, c0 = _cost64("ivim", m["protocol"], p, d), _cost64("ivim", m["protocol"], p0, d)
        idx = torch.nonzero(~torch.isfinite(c) | ~(c < c0) | ((p <= lb) | (p >= ub)).any(0))[:, 0]
        if len(idx):
            q = _lm64("ivim", m["protocol"], p0[:, idx], d[:, idx], m["lb"], m["ub"], 8)[0]
            better = _cost64("ivim", m["protocol"], q, d[:, idx]) < c[idx]
            p[:, idx] = torch.where(better, q, p[:, idx])
        out.append(p)
    return torch.cat(out, 1)


def _train64(case, data, labels, seed):
    """The same batches, start and Adam steps in double with unrounded weights and activations."""
    n, B = case["n"], case["batch"]
    d, lab = data.double(), labels.double()
    smax = d.max(dim=0).values
    y = torch.stack([lab[0] / smax, lab[1], torch.log(lab[2]), torch.log(lab[3])], 1)
    y = (y - y.mean(0)) / y.std(0, unbiased=False)
    x = torch.log((d / smax).clamp_min(1e-6)).T
    perm = torch.from_numpy(np.random.default_rng(0).permutation(n)).to(d.device)
    x, y = x[perm], y[perm]
    g = torch.Generator().manual_seed(seed)
    dims = [(16, 128), (128, 128), (128, 128), (128, 4)]
    ps = []
    for i, o in dims:
        ps.append(((torch.rand(o, i, generator=g) * 2 - 1) * ((6.0 / i) ** 0.5 * (0.5 if o == 4 else 1.0))).double()
                  .to(d.device))
    ps += [torch.zeros(o, dtype=torch.float64, device=d.device) for _, o in dims]
    mom, var = [torch.zeros_like(p) for p in ps], [torch.zeros_like(p) for p in ps]
    nb, total, loss_sum, s = n // B, case["epochs"] * (n // B), 0.0, 0
    for _ in range(case["epochs"]):
        for b in range(nb):
            for p in ps:
                p.requires_grad_(True)
            h = x[b * B:(b + 1) * B]
            for k in range(4):
                h = h @ ps[k].T + ps[4 + k]
                h = _gelu64(h) if k < 3 else h
            loss = ((h - y[b * B:(b + 1) * B]) ** 2).mean()
            grads = torch.autograd.grad(loss, ps)
            loss_sum += loss.detach()
            s += 1
            lr = 2e-3 * 0.5 * (1 + math.cos(math.pi * (s - 1) / total))
            with torch.no_grad():
                for q in range(8):
                    mom[q] = 0.9 * mom[q] + 0.1 * grads[q]
                    var[q] = 0.999 * var[q] + 0.001 * grads[q] ** 2
                    ps[q] = ps[q].detach() - lr * (mom[q] / (1 - 0.9 ** s)) / ((var[q] / (1 - 0.999 ** s)).sqrt() + 1e-8)
    out = []
    for k, (i, o) in enumerate(dims):
        a = torch.zeros(((o + 7) // 8 * 8, i + 8), dtype=torch.float64, device=d.device)
        a[:o, :i], a[:o, i] = ps[k].detach(), ps[4 + k].detach()
        out.append(a)
    return {"weights": out, "loss": loss_sum.reshape(1)}


def _notebook64(case, data):
    """The notebook's start and bounds from two log-linear fits (test_ivim.ipynb cells 6 and 10), then the LM."""
    m = MODELS["ivim21"]
    d = data.double()
    b = torch.tensor([float(v) for v in m["protocol"]], dtype=torch.float64, device=d.device)

    def line(lo, hi):
        X = torch.stack([torch.ones(hi - lo, dtype=torch.float64, device=d.device), -b[lo:hi]], 1)
        return torch.linalg.solve(X.T @ X, X.T @ torch.log(d[lo:hi]))

    low, high = line(*LOW_ROWS), line(*HIGH_ROWS)
    p = [torch.exp(low[0]), 1 - torch.exp(high[0]) / torch.exp(low[0]), low[1], high[1]]
    p = [torch.nan_to_num(v, 0.0, 0.0, 0.0).clamp(lo, hi) for v, lo, hi in zip(p, m["lb"], m["ub"])]
    lb = [(p[0] / 2).clamp_min(500.0), (p[1] - 0.4).clamp_min(0.001), (p[2] / 200).clamp_min(1e-6),
          (p[3] / 200).clamp_min(1e-8)]
    ub = [(p[0] * 2).clamp_max(20000.0), (p[1] + 0.4).clamp_max(0.999), (p[2] * 200).clamp_max(0.1),
          (p[3] * 200).clamp_max(0.02)]
    q, first, _, _, _ = _lm64("ivim", m["protocol"], torch.stack(p), d, lb, ub, case["iters"], tol=1e-10)
    return {"pars": q, "first_f": first[None], "last_f": None, "step_type": None, "lower": torch.stack(lb),
            "upper": torch.stack(ub)}


def _mix64(z):
    """splitmix64's output function on int64 bit patterns."""
    shr = lambda v, k: (v >> k) & ((1 << (64 - k)) - 1)  # noqa: E731
    z = (z ^ shr(z, 30)) * (0xBF58476D1CE4E5B9 - (1 << 64))
    z = (z ^ shr(z, 27)) * (0x94D049BB133111EB - (1 << 64))
    return z ^ shr(z, 31)


def _search64(case, data, seed):
    m = MODELS["ivim21"]
    d = data.double()
    n = case["n"]
    wrap = lambda v: (v + (1 << 63)) % (1 << 64) - (1 << 63)  # noqa: E731
    key = _mix64(torch.arange(1, n + 1, device=d.device) * wrap(0x9E3779B97F4A7C15) + wrap(seed))
    best_f = torch.full((n,), math.inf, dtype=torch.float64, device=d.device)
    best = torch.tensor(m["lb"], dtype=torch.float64, device=d.device)[:, None].expand(4, n)
    for dr in range(case["draws"]):
        rows = []
        for k in range(4):
            u = ((_mix64(key ^ (dr << 8 | k)) >> 40) & 0xFFFFFF).double() / 16777216.0
            rows.append(u * (m["ub"][k] - m["lb"][k]) + m["lb"][k])
        p = _lm64("ivim", m["protocol"], torch.stack(rows), d, m["lb"], m["ub"], case["iters"])[0]
        f = _cost64("ivim", m["protocol"], p, d)
        best = torch.where(f < best_f, p, best)
        best_f = torch.minimum(f, best_f)
    return {"best_pars": best, "best_f": best_f[None]}


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "fit":
        m = MODELS[case["model"]]
        data, init, _, _, _ = _fit_inputs(case, seed)
        parts = [_lm64(m["form"], m["protocol"], init[:, a:b].double(), data[:, a:b].double(), m["lb"], m["ub"],
                       case["iters"]) for a, b in _chunks(n)]
        p, first, last, lam = (torch.cat([x[k] for x in parts], -1) for k in range(4))
        # the damping counts accepted and rejected steps, which rounding decides once a voxel is at rest; the final
        # cost of an fp32 fit is carried by the few voxels that rounding sends to another minimum
        return {"pars": p, "first_f": first[None], "last_f": last[None] if case["dtype"] == "f64" else None,
                "lam": None, "step_type": None}
    if kind == "mixed":
        out = []
        for j, k in enumerate(MIXED):
            m = MODELS[k]
            data = _signals(k, n + 31 * j, seed)[1]
            p, first, _, _, _ = _lm64(m["form"], m["protocol"], _start(k, data).double(), data.double(), m["lb"],
                                         m["ub"], case["iters"])
            out.append({"pars": p, "first_f": first, "last_f": None, "step_type": None})
        return out
    if kind == "warm":
        return {"pars": _warm64(_signals("ivim16", n, seed)[1]), "step_type": None, "counts": None}
    if kind == "stream":
        return {"pars": [_warm64(_signals("ivim16", n, seed * 16 + v)[1]) for v in range(case["volumes"])],
                "counts": None}
    if kind == "train":
        labels, data = _signals("ivim16", n, seed)
        return _train64(case, data, labels, seed % 1000)
    if kind == "search":
        return _search64(case, _signals("ivim21", n, seed)[1], seed)
    return _notebook64(case, _signals("ivim21", n, seed)[1])
