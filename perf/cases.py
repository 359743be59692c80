"""The calls whose time this package is judged by, from the smallest LP to the largest.

Every case goes through the package's public entry points on LPs of its own
generators (``sovereign_solver_gb300.workloads``):

* ``oneshot``   ``solve_lp_pdhg``: problem in, result out (upload, layout,
                scaling, solve, read-back), what a caller of one LP does;
* ``engine``    ``PDHGEngine.solve`` on a resident problem (re-solves);
* ``batch``     ``PDHGBatch.solve``: many LPs of uneven sizes in one launch;
* ``children``  ``branching.child_gains``: the child LPs of a branch-and-bound
                node, built, solved as one batch and read back;
* ``predict`` / ``gradient``  the warm-start network's forward pass and its
                training loss and gradient;
* ``check``     ``sps_kkt_noalloc``: a point's KKT error in device memory.

``attempts`` of a case is what its LPs take (for ``work`` alone): ``max_iters``
where the call runs to its limit, else a typical count to the tolerance.
"""

import ctypes
import math

import numpy as np
import torch

import sovereign_solver_gb300 as sps
from sovereign_solver_gb300 import _native, branching, workloads
from sovereign_solver_gb300.gnn import WarmStartGNN, rhs, stacked_rows
from sovereign_solver_gb300.pdhg import PDHGEngine


def listed():
    return [
        # a textbook-size LP with every option at its default (FP32, tolerance 1e-6, continued in FP64
        # where FP32 stalls): the latency of one call
        {"name": "oneshot_40x100", "kind": "oneshot", "family": "planted", "m": 40, "n": 100, "nnz": 600,
         "precision": "fp32", "tol": 1e-6, "max_iters": 20000, "attempts": 1000},
        # the same call in FP64, an odd size with '<=' and '=' rows and free upper bounds
        {"name": "oneshot_fp64_37x53", "kind": "oneshot", "family": "transport", "m": 37, "n": 53, "nnz": 0,
         "precision": "fp64", "tol": 1e-6, "max_iters": 3000, "attempts": 2500},
        # the plain-PDHG workload of the benchmark: 200 x 500, 5 % density, to 1e-4, resident
        {"name": "planted_200x500", "kind": "engine", "family": "planted", "m": 200, "n": 500, "nnz": 5000,
         "mode": "adaptive", "precision": "fp32", "form": "lagrangian", "tol": 1e-4, "max_iters": 100000,
         "attempts": 600},
        # an ordinary sparse model
        {"name": "planted_2003x5009", "kind": "engine", "family": "planted", "m": 2003, "n": 5009, "nnz": 50000,
         "mode": "adaptive", "precision": "fp32", "form": "lagrangian", "tol": 1e-4, "max_iters": 100000,
         "attempts": 900},
        # the benchmark's default workload: the transportation LP of 2M variables, to 1e-4
        {"name": "transport_1000x2000", "kind": "engine", "family": "transport", "m": 1000, "n": 2000, "nnz": 0,
         "mode": "adaptive", "precision": "fp32", "form": "lagrangian", "tol": 1e-4, "max_iters": 100000,
         "attempts": 2600},
        # the power-law LP of the SpMV roofline at half its size, in PDLP's error form, to an
        # iteration limit (its solve to 1e-4 takes seconds)
        {"name": "powerlaw_500kx1M", "kind": "engine", "family": "powerlaw", "m": 500_000, "n": 1_000_000,
         "nnz": 10_000_000, "mode": "adaptive", "precision": "fp32", "form": "pdlp", "tol": 1e-4,
         "max_iters": 256, "attempts": 256},
        # the reference's own rules and iteration counts in FP64, to an iteration limit as its
        # benchmark runner sets one
        {"name": "reference_fp64_100x200", "kind": "engine", "family": "transport", "m": 100, "n": 200, "nnz": 0,
         "mode": "reference", "precision": "fp64", "form": "lagrangian", "tol": 1e-6, "max_iters": 2000,
         "attempts": 2000},
        # the batched workload: planted LPs of log-uniform sizes, more of them than the GPU runs at once
        {"name": "batch_640", "kind": "batch", "count": 640, "m_lo": 50, "m_hi": 1000, "tol": 1e-4,
         "max_iters": 100000, "attempts": 900},
        # strong branching at a set-covering node: the 40 children of its 20 most fractional variables
        {"name": "children_200x2000", "kind": "children", "m": 200, "n": 2000, "candidates": 20, "tol": 1e-4,
         "max_iters": 100000, "attempts": 700},
        # warm starts for 16 instances of the 200 x 400 transportation family (trained weights)
        {"name": "predict_16", "kind": "predict", "src": 200, "dst": 400, "hidden": 64, "layers": 3, "batch": 16},
        # one training minibatch of the same family
        {"name": "gradient_8", "kind": "gradient", "src": 200, "dst": 400, "hidden": 64, "layers": 3, "batch": 8},
        # a candidate point checked on an LP that already lives in device memory
        {"name": "check_60kx150k", "kind": "check", "m": 60_000, "n": 150_000, "nnz": 1_500_000},
    ]


def _between(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["oneshot", "engine", "engine", "engine", "reference", "batch", "children", "predict",
                       "gradient", "check"])
    if kind == "oneshot":
        m = _between(rng, 12, 600)
        n = int(m * rng.uniform(2.2, 3.0))
        it = rng.choice([1000, 2000, 4000])
        return {"kind": "oneshot", "family": "planted", "m": m, "n": n, "nnz": int(n * rng.uniform(4, 12)),
                "precision": rng.choice(["fp32", "fp64"]), "tol": rng.choice([1e-4, 1e-6]), "max_iters": it,
                "attempts": it // 2}
    if kind == "engine":
        family = rng.choice(["planted", "planted", "transport", "powerlaw"])
        it = rng.choice([128, 192, 320, 512])
        if family == "planted":
            m = _between(rng, 100, 40_000)
            n = int(m * rng.uniform(1.5, 3.0))
            nnz = int(n * rng.uniform(3, 20))
        elif family == "transport":
            m, nnz = _between(rng, 20, 900), 0
            n = int(m * rng.uniform(1.0, 2.0))
        else:
            m = _between(rng, 5_000, 200_000)
            n = 2 * m + rng.randrange(100)
            nnz = int(n * rng.uniform(6, 10))
        return {"kind": "engine", "family": family, "m": m, "n": n, "nnz": nnz, "mode": "adaptive",
                "precision": rng.choice(["fp32", "fp32", "fp64"]), "form": rng.choice(["lagrangian", "pdlp"]),
                "tol": 1e-6, "max_iters": it, "attempts": it}
    if kind == "reference":
        m = _between(rng, 8, 120)
        it = rng.choice([500, 1000, 2000])
        return {"kind": "engine", "family": "transport", "m": m, "n": int(m * rng.uniform(1.0, 2.0)), "nnz": 0,
                "mode": "reference", "precision": rng.choice(["fp32", "fp64"]), "form": "lagrangian", "tol": 1e-6,
                "max_iters": it, "attempts": it}
    if kind == "batch":
        return {"kind": "batch", "count": _between(rng, 30, 640), "m_lo": 50, "m_hi": _between(rng, 200, 1000),
                "tol": 1e-4, "max_iters": 640, "attempts": 600}
    if kind == "children":
        m = _between(rng, 60, 250)
        return {"kind": "children", "m": m, "n": int(m * rng.uniform(5, 10)), "candidates": rng.randrange(4, 20),
                "tol": 1e-4, "max_iters": 20000, "attempts": 700}
    if kind == "check":
        m = _between(rng, 100, 100_000)
        n = int(m * rng.uniform(1.5, 2.5))
        return {"kind": "check", "m": m, "n": n, "nnz": int(n * rng.uniform(4, 12))}
    s = _between(rng, 20, 200)
    return {"kind": kind, "src": s, "dst": int(s * rng.uniform(1.0, 2.0)), "hidden": rng.choice([32, 64, 64]),
            "layers": rng.randrange(2, 5), "batch": rng.randrange(1, 17 if kind == "predict" else 9)}


# ---------------------------------------------------------------- inputs

def _problem(case, seed):
    """The case's LP and what its generator knows of the optimum."""
    if case["family"] == "planted":
        return workloads.planted_lp(case["m"], case["n"], case["nnz"] / (case["m"] * case["n"]), seed=seed) \
            if case["m"] * case["n"] <= 40_000_000 else _planted_sparse(case, seed)
    if case["family"] == "transport":
        return workloads.transportation_lp(case["m"], case["n"], seed=seed)
    return workloads.powerlaw_lp(case["m"], case["n"], case["nnz"], seed=seed)


def _planted_sparse(case, seed):
    """The planted construction at sizes where ``planted_lp``'s dense mask would take gigabytes:
    columns of equal length, as the batched workload draws them."""
    k = max(1, round(case["nnz"] / case["n"]))
    ratio = case["n"] / case["m"]
    return workloads.batch_planted_lp(seed, m_range=(case["m"], case["m"]), n_ratio=(ratio, ratio), col_nnz=(k, k))


def _batch(case, seed):
    """The batched workload's construction, its sizes spread evenly over their logarithm: m in
    [m_lo, m_hi] in a shuffled order, n / m in [1.5, 3], the same for every seed."""
    count, (lo, hi) = case["count"], (case["m_lo"], case["m_hi"])
    for k in range(count):
        m = round(lo * (hi / lo) ** ((k * 0.6180339887) % 1.0))
        r = 1.5 + 1.5 * ((k * 0.7548776662) % 1.0)
        yield workloads.batch_planted_lp(10_000 * (seed % 10_000) + k, m_range=(m, m), n_ratio=(r, r))


def _family(case):
    return workloads.TransportFamily(case["src"], case["dst"])


def _network(case, fam, template):
    trained = (case["src"], case["dst"], case["hidden"], case["layers"]) == (200, 400, 64, 3)
    if trained:
        return WarmStartGNN.load("sovereign-solver_gb300/data/warmstart_transport_200x400.npz", template,
                                 max_batch=case["batch"])
    return WarmStartGNN(template, hidden=case["hidden"], layers=case["layers"], max_batch=case["batch"], seed=1)


def _minibatch(case, seed, net, fam):
    """Features and targets of the case's instances: each sink served by its cheapest source, the
    row prices its cost (near a transportation LP's solution: as sparse, of the same size)."""
    fvs, fcs, xts, yts, lts = [], [], [], [], []
    for k in range(case["batch"]):
        cost, supply, demand = fam.params(1000 * (seed % 100_000) + k)
        fv, fc = net.features_from(cost, np.concatenate([supply, demand]))
        C = cost.reshape(fam.S, fam.D)
        src = C.argmin(0)
        x = np.zeros((fam.S, fam.D))
        x[src, np.arange(fam.D)] = demand
        y = np.concatenate([np.zeros(fam.S), C.min(0)])
        xt, yt, lt = net.targets(x.ravel(), y, math.exp(0.1 * (k % 5) - 0.2))
        fvs.append(fv)
        fcs.append(fc)
        xts.append(xt)
        yts.append(yt)
        lts.append(lt)
    return fvs, fcs, xts, yts, np.asarray(lts, np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "oneshot":
        p, _ = _problem(case, seed)
        return {"kind": kind, "p": p, "opts": dict(tol=case["tol"], max_iters=case["max_iters"],
                                                   precision=case["precision"])}
    if kind == "engine":
        p, _ = _problem(case, seed)
        return {"kind": kind, "eng": PDHGEngine(p, mode=case["mode"], precision=case["precision"],
                                                kkt_form=case["form"], tol=case["tol"],
                                                max_iters=case["max_iters"])}
    if kind == "batch":
        return {"kind": kind, "batch": sps.PDHGBatch([p for p, _ in _batch(case, seed)], tol=case["tol"],
                                                     max_iters=case["max_iters"])}
    if kind == "children":
        p, _ = workloads.set_cover_milp(case["m"], case["n"], seed=seed)
        r = sps.solve_lp_pdhg(p, tol=1e-4, precision="fp64", max_iters=20000)   # the node's own LP
        n = p.n_vars
        return {"kind": kind, "p": p, "x": r.x, "y": r.y, "obj": r.objective,
                "cands": branching.strong_candidates(r.x, p.integer_mask, case["candidates"]),
                "lo": np.full(n, -np.inf), "hi": np.full(n, np.inf), "tol": case["tol"], "it": case["max_iters"]}
    if kind in ("predict", "gradient"):
        fam = _family(case)
        net = _network(case, fam, fam.problem(0))
        return {"kind": kind, "net": net, "data": _minibatch(case, seed, net, fam)}
    lp, x, y = _device_lp(case, seed)
    st = {"kind": kind, "lp": lp, "x": x, "y": y, "out": torch.empty(6, dtype=torch.float64, device="cuda")}
    st["desc"] = _native.DeviceLP(lp["n"], 0, lp["m"], *[lp[k].data_ptr() for k in
                                                         ("ptr", "idx", "val", "c", "rhs", "lb", "ub")])
    return st


def _device_lp(case, seed):
    """An LP of `nnz` entries (uniform columns, '=' rows, bounds [0, 10]) and a point, built on the GPU."""
    m, n = case["m"], case["n"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = lambda k: torch.rand(k, generator=g, device="cuda", dtype=torch.float64)          # noqa: E731
    nrm = lambda k: torch.randn(k, generator=g, device="cuda", dtype=torch.float64)       # noqa: E731
    length = (1 + u(m) * (2.0 * case["nnz"] / m - 1)).long().clamp_(1, n)
    ptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(length, 0)
    nnz = int(ptr[-1])
    idx = (u(nnz) * n).long().clamp_(0, n - 1).int()
    val, x, y = nrm(nnz), u(n), nrm(m)
    row = torch.repeat_interleave(torch.arange(m, device="cuda"), length)
    b = torch.zeros(m, dtype=torch.float64, device="cuda").index_add_(0, row, val * x[idx.long()]) + 1e-3 * nrm(m)
    lp = {"n": n, "m": m, "ptr": ptr.int(), "idx": idx, "val": val, "c": nrm(n), "rhs": b,
          "lb": torch.zeros(n, dtype=torch.float64, device="cuda"),
          "ub": torch.full((n,), 10.0, dtype=torch.float64, device="cuda")}
    return lp, x, y


# ---------------------------------------------------------------- the calls

def _result(r):
    return {"x": r.x, "y": r.y, "objective": r.objective, "iterations": r.iterations}


def run(st):
    kind = st["kind"]
    if kind == "oneshot":
        return _result(sps.solve_lp_pdhg(st["p"], **st["opts"]))
    if kind == "engine":
        return _result(st["eng"].solve())
    if kind == "batch":
        rs = st["batch"].solve()
        return {"x": np.concatenate([r.x for r in rs]), "y": np.concatenate([r.y for r in rs]),
                "objective": np.array([r.objective for r in rs]), "iterations": np.array([r.iterations for r in rs])}
    if kind == "children":
        down, up, rs = branching.child_gains(st["p"], st["cands"], st["x"], st["lo"], st["hi"], st["obj"], y=st["y"],
                                             tol=st["tol"], max_iters=st["it"], return_results=True)
        return {"down": down, "up": up, "x": np.stack([r.x for r in rs])}
    if kind == "predict":
        x, y, lw = st["net"].predict_features(*st["data"][:2])
        return {"x": x, "y": y, "log_omega": lw}
    if kind == "gradient":
        loss, g = st["net"].loss_grad(*st["data"])
        return {"loss": loss, "gradient": g}
    _native.check(_native.load().sps_kkt_noalloc(ctypes.byref(st["desc"]), st["x"].data_ptr(), st["y"].data_ptr(),
                                                 st["out"].data_ptr(), torch.cuda.current_stream().cuda_stream))
    return st["out"]


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind in ("oneshot", "engine"):
        if case["family"] == "transport":
            m, n, nnz = case["m"] + case["n"], case["m"] * case["n"], 2 * case["m"] * case["n"]
        else:
            m, n, nnz = case["m"], case["n"], case["nnz"]
        v = 4 if case["precision"] == "fp32" else 8
        # per attempt: both orientations once (value and index), six column vectors and eight of the rows
        each = 2 * nnz * (4 + v) + v * (7 * n + 9 * m)
        return {"bytes": case["attempts"] * each + 8 * (n + m), "flops": case["attempts"] * 4 * nnz}
    if kind in ("batch", "children"):
        if kind == "batch":
            lo, hi = case["m_lo"], case["m_hi"]
            m = (hi - lo) / math.log(hi / lo) if hi > lo else lo     # mean of a log-uniform size
            count, n = case["count"], 2.25 * m
            nnz = 30 * n
        else:
            count, m, n = 2 * case["candidates"], case["m"], case["n"]
            nnz = 0.02 * m * n
        each = 16 * nnz + 4 * (7 * n + 9 * m)
        return {"bytes": count * (case["attempts"] * each + 8 * (n + m)), "flops": count * case["attempts"] * 4 * nnz}
    if kind in ("predict", "gradient"):
        n, m, B, H, L = case["src"] * case["dst"], case["src"] + case["dst"], case["batch"], case["hidden"], case["layers"]
        dense, edges = 4 * H * H * (n + m) * B * L, 2 * 2 * H * (2 * n) * B * L
        hv = 4 * H * (n + m) * B                                     # one layer's activations
        if kind == "predict":      # inputs and outputs; every layer reads and writes its activations once
            return {"bytes": 8 * (n + m) * B + 2 * L * hv, "flops": dense + edges}
        return {"bytes": 12 * (n + m) * B + 6 * L * hv, "flops": 3 * (dense + edges)}
    m, n, nnz = case["m"], case["n"], case["nnz"]
    return {"bytes": 12 * nnz + 4 * m + 8 * (4 * n + 2 * m), "flops": 4 * nnz}


# ---------------------------------------------------------------- values in 64 bits

def exact(case, seed):
    kind = case["kind"]
    if kind in ("oneshot", "engine"):
        # the optimum is known where it was planted and the call reaches it (not at an iteration
        # limit); x has no single value (300 of 500 columns lie strictly inside their bounds, more
        # than there are rows), the prices and the objective have
        if case["family"] != "planted" or case.get("mode") == "reference" or case["max_iters"] < 20000:
            return None
        _, info = _problem(case, seed)
        return {"x": None, "y": info["y_star"], "objective": info["obj_star"], "iterations": None}
    if kind == "batch":
        if case["max_iters"] < 20000:
            return None
        obj = np.array([info["obj_star"] for _, info in _batch(case, seed)])
        return {"x": None, "y": None, "objective": obj, "iterations": None}
    if kind == "children":
        return None                  # the gains have no closed value: each is another LP's optimum
    if kind in ("predict", "gradient"):
        return _exact_network(case, seed)
    lp, x, y = _device_lp(case, seed)
    m, n = lp["m"], lp["n"]
    row = torch.repeat_interleave(torch.arange(m, device="cuda"), torch.diff(lp["ptr"].long()))
    col = lp["idx"].long()
    ax = torch.zeros(m, dtype=torch.float64, device="cuda").index_add_(0, row, lp["val"] * x[col])
    aty = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, col, lp["val"] * y[row])
    rp = (ax - lp["rhs"]).norm() / (1 + lp["rhs"].norm())
    rc = lp["c"] - aty               # every column has both bounds: no reduced cost is left over
    po = lp["c"] @ x
    do = lp["rhs"] @ y + (lp["lb"] * rc.clamp(min=0) + lp["ub"] * rc.clamp(max=0)).sum()
    gap = (po - do).abs() / (1 + po.abs() + do.abs())
    rd = torch.zeros((), dtype=torch.float64, device="cuda")
    return torch.stack([torch.maximum(rp, gap), rp, rd, gap, po, do])


def _exact_network(case, seed):
    """The network of include/sps_gnn.h in FP64 (BF16-rounded matrices and head vectors)."""
    dev, f64 = "cuda", torch.float64
    fam = _family(case)
    template = fam.problem(0)
    with _network(case, fam, template) as net:
        P = torch.from_numpy(net.params()).to(dev)
        fvs, fcs, xts, yts, lts = _minibatch(case, seed, net, fam)
    H, L, B, n, m = case["hidden"], case["layers"], case["batch"], fam.S * fam.D, fam.S + fam.D
    K = stacked_rows(template)
    K.sort_indices()
    deg = torch.from_numpy(np.diff(K.indptr).astype(np.int64)).to(dev)
    row = torch.repeat_interleave(torch.arange(m, device=dev), deg)
    col = torch.from_numpy(K.indices.astype(np.int64)).to(dev)
    val = torch.from_numpy(K.data.astype(np.float32)).to(dev)
    degv = torch.bincount(col, minlength=n)
    a_c, a_v = (val / deg[row].float()).to(f64), (val / degv[col].float()).to(f64)   # FP32 edge weights
    at = [0]

    def take(*shape, rounded):
        k = math.prod(shape)
        v = P[at[0]:at[0] + k]
        at[0] += k
        v = (v.bfloat16() if rounded else v).to(f64).reshape(shape)
        return v.requires_grad_(case["kind"] == "gradient")

    W = [take(H, 4, rounded=True), take(H, rounded=False), take(H, 4, rounded=True), take(H, rounded=False)]
    layers = []
    for _ in range(L):
        layers.append([take(H, H, rounded=True), take(H, H, rounded=True), take(H, rounded=False),
                       take(H, H, rounded=True), take(H, H, rounded=True), take(H, rounded=False)])
    heads = [take(H, rounded=True), take(1, rounded=False), take(H, rounded=True), take(1, rounded=False),
             take(2 * H, rounded=True), take(1, rounded=False)]
    every = W + [w for l in layers for w in l] + heads
    kind = torch.zeros(m, dtype=f64, device=dev)
    kind[: fam.S] = 1.0
    le = kind[row]
    n_le = torch.zeros(n, dtype=f64, device=dev).index_add_(0, col, le).clamp(min=1)
    n_eq = torch.zeros(n, dtype=f64, device=dev).index_add_(0, col, 1 - le).clamp(min=1)
    xs, ys, lws, total, grads = [], [], [], 0.0, None
    weights = (1.0, 1.0, float(np.float32(0.1)))
    for s in range(B):               # instance by instance: the activations of one in FP64 at a time
        c = torch.from_numpy(fvs[s][:, 0]).to(dev, f64)
        b = torch.from_numpy(fcs[s][:, 0]).to(dev, f64)
        cmin = torch.full((m,), math.inf, dtype=f64, device=dev).scatter_reduce_(0, row, c[col], "amin")
        gap = c[col] - cmin[row]
        fv = torch.stack([c, torch.zeros(n, dtype=f64, device=dev).index_add_(0, col, gap * le) / n_le,
                          torch.zeros(n, dtype=f64, device=dev).index_add_(0, col, gap * (1 - le)) / n_eq,
                          torch.ones(n, dtype=f64, device=dev)], 1)
        fc = torch.stack([b, kind, cmin, torch.ones(m, dtype=f64, device=dev)], 1)
        hv, hc = torch.relu(fv @ W[0].T + W[1]), torch.relu(fc @ W[2].T + W[3])
        for Uc, Mc, bc, Uv, Mv, bv in layers:
            ac = torch.zeros(m, H, dtype=f64, device=dev).index_add(0, row, a_c[:, None] * hv[col])
            hc = torch.relu(hc @ Uc.T + ac @ Mc.T + bc)
            av = torch.zeros(n, H, dtype=f64, device=dev).index_add(0, col, a_v[:, None] * hc[row])
            hv = torch.relu(hv @ Uv.T + av @ Mv.T + bv)
        x0, y0 = hv @ heads[0] + heads[1], hc @ heads[2] + heads[3]
        lw = torch.cat([hc.mean(0), hv.mean(0)]) @ heads[4] + heads[5][0]
        if case["kind"] == "gradient":
            t = [torch.from_numpy(np.ascontiguousarray(v)).to(dev, f64) for v in (xts[s], yts[s])]
            loss = (weights[0] * ((x0 - t[0]) ** 2).mean() + weights[1] * ((y0 - t[1]) ** 2).mean()
                    + weights[2] * (lw - float(lts[s])) ** 2) / B
            g = torch.cat([v.reshape(-1) for v in torch.autograd.grad(loss, every)])
            grads = g if grads is None else grads + g
            total += float(loss)
        else:
            xs.append(x0)
            ys.append(y0)
            lws.append(lw)
    if case["kind"] == "gradient":
        return {"loss": torch.tensor(total, dtype=f64), "gradient": grads}
    return {"x": torch.stack(xs), "y": torch.stack(ys), "log_omega": torch.stack(lws)}
