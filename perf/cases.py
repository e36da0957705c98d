"""Performance cases: the work that users of this library have it do, through its public entry points.

Kinds of case (the "kind" of a case dict):

  kkt     cuOptComputeKKTErrorsNoAlloc on a candidate point of an LP in device memory: the call
          that a heuristic or a monitoring loop makes for every candidate (latency counts).
  device  cuOptSolveDevice: one LP whose arrays live in device memory, solved to a tolerance.
  host    Solve(DataModel, SolverSettings): the Python (C API) route from host arrays and back.
  batch   BatchSolve: independent LPs of uneven sizes, from host arrays, in one call.
  branch  BatchPDLPStrongBranching: the down and up branches of fractional variables of one LP.
  layer   the differentiable torch layer (lp_solve_batch): its backward pass, or a training step
          (forward with crossover, then backward).

Three recipes of LP, all with an optimum known by construction (the recipes of
cuopt_b200.generators, made on the device): "constructed" (equality rows, boxed columns, uniform
sparsity, k non-zeros per column; y* and the reduced costs are unique, x* is not), "vertex"
(the same with a unique non-degenerate vertex, on which derivatives exist) and "skewed" (Zipf row
lengths, mixed senses, free columns; ill-conditioned, run to an iteration limit).
"""
import ctypes as C
import math

import numpy as np
import torch

from cuopt_b200 import linear_programming as lpm
from cuopt_b200._lib import lib
from cuopt_b200.torch_layer import LPInstance, lp_solve_batch

F64 = torch.float64


def listed():
    return [
        # A candidate check inside a heuristic's loop: the smallest call, all launch latency.
        {"name": "kkt_small", "kind": "kkt", "m": 300, "n": 700, "k": 8},
        # The same check near its largest number of variables: atomics and memory.
        {"name": "kkt_large", "kind": "kkt", "m": 200000, "n": 500000, "k": 8},
        # One tiny LP from Python, odd sizes: set-up, launches and copies.
        {"name": "host_tiny", "kind": "host", "m": 313, "n": 709, "k": 7, "mixed": False,
         "tol": 1e-6},
        # The 2000 x 5000 benchmark LP, FP64 (the reference's precision).
        {"name": "device_small_fp64", "kind": "device", "recipe": "constructed", "m": 2000,
         "n": 5000, "k": 8, "mixed": False, "tol": 1e-6},
        # A medium LP in mixed precision at the default tolerance of the settings.
        {"name": "device_medium_mixed", "kind": "device", "recipe": "constructed", "m": 12007,
         "n": 30011, "k": 9, "mixed": True, "tol": 1e-4},
        # A large LP in FP64: matrix and vectors beyond L2.
        {"name": "device_large_fp64", "kind": "device", "recipe": "constructed", "m": 200000,
         "n": 500000, "k": 8, "mixed": False, "tol": 1e-6},
        # The headline LP of the benchmark (1M x 2M, 16M non-zeros, mixed precision, 1e-6).
        {"name": "device_1m_mixed", "kind": "device", "recipe": "constructed", "m": 1000000,
         "n": 2000000, "k": 8, "mixed": True, "tol": 1e-6},
        # Skewed sparsity (Zipf rows up to 5000 long), FP64, to an iteration limit.
        {"name": "device_skewed_fp64", "kind": "device", "recipe": "skewed", "m": 20000,
         "n": 60000, "k": 0, "mixed": False, "tol": 1e-6, "limit": 1000},
        # A batch of independent LPs of uneven sizes, FP64.
        {"name": "batch_fp64", "kind": "batch", "count": 64, "m_lo": 200, "m_hi": 20000,
         "mixed": False, "tol": 1e-6},
        # Many small LPs in mixed precision at the default tolerance.
        {"name": "batch_mixed", "kind": "batch", "count": 48, "m_lo": 200, "m_hi": 3000,
         "mixed": True, "tol": 1e-4},
        # Strong branching: 32 branches of one LP (both directions of 16 variables).
        {"name": "branch_small", "kind": "branch", "m": 2000, "n": 5000, "k": 8, "count": 16,
         "tol": 1e-6},
        # The backward pass of the differentiable layer after a batched forward with crossover.
        {"name": "layer_backward", "kind": "layer", "train": False, "count": 6, "m": 800,
         "n": 1700, "k": 8, "tol": 1e-6},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["kkt", "device", "device", "host", "batch", "branch", "layer"])
    k = rng.randint(6, 12)
    if kind == "kkt":
        m = _log_uniform(rng, 100, 200000)
        return {"kind": kind, "m": m, "n": int(m * rng.uniform(1.8, 2.6)), "k": k}
    if kind == "host":
        m = _log_uniform(rng, 100, 4000)
        return {"kind": kind, "m": m, "n": int(m * rng.uniform(2.0, 2.6)), "k": k,
                "mixed": rng.random() < 0.3, "tol": rng.choice([1e-4, 1e-6])}
    if kind == "device":
        mixed = rng.random() < 0.4
        if rng.random() < 0.2:
            m = _log_uniform(rng, 2000, 20000)
            return {"kind": kind, "recipe": "skewed", "m": m, "n": int(m * rng.uniform(2.0, 3.0)),
                    "k": 0, "mixed": False, "tol": 1e-6, "limit": rng.choice([400, 1000])}
        m = _log_uniform(rng, 500, 250000)
        return {"kind": kind, "recipe": "constructed", "m": m, "n": int(m * rng.uniform(2.0, 2.6)),
                "k": k, "mixed": mixed, "tol": rng.choice([1e-4, 1e-6])}
    if kind == "batch":
        lo = _log_uniform(rng, 100, 600)
        return {"kind": kind, "count": _log_uniform(rng, 8, 64), "m_lo": lo,
                "m_hi": lo * rng.randint(2, 20), "mixed": rng.random() < 0.4,
                "tol": rng.choice([1e-4, 1e-6])}
    if kind == "branch":
        m = _log_uniform(rng, 300, 3000)
        return {"kind": kind, "m": m, "n": int(m * rng.uniform(2.2, 2.6)), "k": 8,
                "count": rng.randint(2, 20), "tol": rng.choice([1e-4, 1e-6])}
    train = rng.random() < 0.5
    m = _log_uniform(rng, 100, 250 if train else 900)
    return {"kind": kind, "train": train, "count": rng.randint(1, 8), "m": m,
            "n": int(m * rng.uniform(1.8, 2.4)), "k": 8, "tol": 1e-6}


# ---------------------------------------------------------------------------------------------
# Inputs, made on the device from the seed alone (sums in a fixed order, so that the same seed
# gives the same bits).


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=F64)


def _offsets(rows, m):
    off = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    return off


def _row_sums(values, off):
    return torch.segment_reduce(values, "sum", offsets=off, axis=0, initial=0.0)


def _columns(g, m, n, k):
    """[n, k] row indices, distinct inside each column."""
    r = torch.randint(0, m, (n, k), generator=g, device="cuda")
    while True:
        s = torch.sort(r, dim=1).values
        bad = torch.nonzero((s[:, 1:] == s[:, :-1]).any(1)).ravel()
        if bad.numel() == 0:
            return r
        r[bad] = torch.randint(0, m, (bad.numel(), k), generator=g, device="cuda")


def _uniform_lp(m, n, k, seed, vertex):
    g = _gen(seed)
    rows = _columns(g, m, n, k)
    vals = torch.randn(n, k, generator=g, device="cuda", dtype=F64)
    upper = 10.0
    if vertex:  # basic column basic[i] holds row i with a value of magnitude in [1, 2]
        basic = torch.randperm(n, generator=g, device="cuda")[:m]
        want = torch.arange(m, device="cuda")
        hit = rows[basic] == want[:, None]
        has = hit.any(1)
        pos = torch.where(has, hit.to(torch.int64).argmax(1), 0)
        rows[basic[~has], 0] = want[~has]
        sign = torch.where(_uniform(g, m) < 0.5, -1.0, 1.0).to(F64)
        vals[basic, pos] = sign * _uniform(g, m, 1.0, 2.0)
        is_basic = torch.zeros(n, dtype=torch.bool, device="cuda")
        is_basic[basic] = True
        at_up = (~is_basic) & (_uniform(g, n) < 0.2)
        x = torch.where(is_basic, _uniform(g, n, 0.5, upper - 0.5), torch.where(at_up, upper, 0.0))
        mag = _uniform(g, n, 0.1, 1.0)
        s = torch.where(is_basic, 0.0, torch.where(at_up, -mag, mag))
    else:
        x = _uniform(g, n, 0.5, 5.0)
        zero = _uniform(g, n) < 0.3
        x[zero] = 0.0
        s = torch.where(zero, _uniform(g, n, 0.1, 1.0), 0.0)
    y = torch.randn(m, generator=g, device="cuda", dtype=F64)
    c = (vals * y[rows]).sum(1) + s
    key = (rows * n + torch.arange(n, device="cuda")[:, None]).ravel()
    order = torch.argsort(key)
    key = key[order]
    row, col, val = key // n, key % n, vals.ravel()[order]
    off = _offsets(row, m)
    b = _row_sums(val * x[col], off)
    return {"m": m, "n": n, "off": off.int(), "idx": col.int(), "val": val, "c": c, "lo": b,
            "up": b.clone(), "vl": torch.zeros(n, dtype=F64, device="cuda"),
            "vu": torch.full((n,), upper, dtype=F64, device="cuda"), "x": x, "y": y, "s": s}


def _skewed_lp(m, n, seed, a=1.3, cap=5000):
    g = _gen(seed)
    w = torch.cumsum(torch.arange(1, cap + 1, device="cuda", dtype=F64) ** -a, 0)
    lens = torch.searchsorted(w / w[-1], _uniform(g, m), right=True) + 1
    lens = torch.clamp(lens, max=min(cap, n))
    row = torch.repeat_interleave(torch.arange(m, device="cuda"), lens)
    key = torch.unique(row * n + torch.randint(0, n, (row.numel(),), generator=g, device="cuda"))
    row, col = key // n, key % n
    sign = torch.where(_uniform(g, key.numel()) < 0.5, -1.0, 1.0).to(F64)
    val = 10.0 ** _uniform(g, key.numel(), -3.0, 3.0) * sign
    off = _offsets(row, m)
    free = _uniform(g, n) < 0.1
    vl = torch.where(free, -math.inf, torch.zeros(n, dtype=F64, device="cuda"))
    vu = torch.where(free, math.inf, _uniform(g, n, 1.0, 100.0))
    u = _uniform(g, n)
    at_lo, at_up = (~free) & (u < 0.3), (~free) & (u >= 0.3) & (u < 0.4)
    inside = _uniform(g, n, 0.1, 0.9)
    x = torch.where(free, torch.randn(n, generator=g, device="cuda", dtype=F64),
                    inside * torch.where(free, 1.0, vu))
    x = torch.where(at_lo, 0.0, torch.where(at_up, vu, x))
    mag = _uniform(g, n, 0.1, 1.0)
    s = torch.where(at_lo, mag, torch.where(at_up, -mag, 0.0))
    ax = _row_sums(val * x[col], off)
    eq, active = _uniform(g, m) < 0.5, _uniform(g, m) < 0.5
    y = torch.where(eq, torch.randn(m, generator=g, device="cuda", dtype=F64),
                    torch.where(active, -_uniform(g, m, 0.1, 1.0), 0.0))
    slack = torch.where((~eq) & (~active), _uniform(g, m, 0.1, 1.0) * (1.0 + ax.abs()), 0.0)
    by_col = torch.argsort(col * m + row)
    c = _row_sums((val * y[row])[by_col], _offsets(col, n)) + s
    return {"m": m, "n": n, "off": off.int(), "idx": col.int(), "val": val, "c": c,
            "lo": torch.where(eq, ax, -math.inf), "up": ax + slack, "vl": vl, "vu": vu, "x": x,
            "y": y, "s": s}


def _batch_lps(case, seed):
    # The sizes belong to the case, the values to the seed.
    rng = np.random.default_rng(case["count"])
    ms = np.exp(rng.uniform(math.log(case["m_lo"]), math.log(case["m_hi"]), case["count"]))
    ks = rng.integers(6, 13, size=case["count"])
    return [_uniform_lp(int(m), int(2.5 * int(m)), int(k), 1000 * seed + i, False)
            for i, (m, k) in enumerate(zip(ms, ks))]


def _settings(case):
    s = lpm.SolverSettings()
    s.set_optimality_tolerance(case["tol"])
    s.set_parameter(lpm.CUOPT_METHOD, int(lpm.SolverMethod.PDLP))
    s.set_parameter(lpm.CUOPT_LOG_TO_CONSOLE, False)
    if case.get("mixed"):
        s.set_parameter(lpm.CUOPT_PDLP_PRECISION, int(lpm.PDLPPrecision.Mixed))
    if case.get("limit"):
        s.set_parameter(lpm.CUOPT_ITERATION_LIMIT, int(case["limit"]))
    if case["kind"] == "layer":
        s.set_parameter(lpm.CUOPT_CROSSOVER, True)
    return s


def _data_model(p):
    h = {key: v.cpu().numpy() for key, v in p.items() if isinstance(v, torch.Tensor)}
    d = lpm.DataModel()
    d.set_csr_constraint_matrix(h["val"], h["idx"], h["off"])
    d.set_objective_coefficients(h["c"])
    d.set_constraint_lower_bounds(h["lo"])
    d.set_constraint_upper_bounds(h["up"])
    d.set_variable_lower_bounds(h["vl"])
    d.set_variable_upper_bounds(h["vu"])
    return d


def _one_lp(case, seed):
    if case.get("recipe") == "skewed":
        return _skewed_lp(case["m"], case["n"], seed)
    return _uniform_lp(case["m"], case["n"], case["k"], seed, False)


def _candidate(p, seed):
    """A point near the optimum, as a heuristic would have it checked."""
    g = _gen(seed + 77)
    x = p["x"] * (1.0 + 1e-3 * torch.randn(p["n"], generator=g, device="cuda", dtype=F64))
    y = p["y"] * (1.0 + 1e-3 * torch.randn(p["m"], generator=g, device="cuda", dtype=F64))
    return torch.minimum(torch.maximum(x, p["vl"]), p["vu"]), y, p["s"].clone()


def _layer_lps(case, seed):
    return [_uniform_lp(case["m"], case["n"], case["k"], 1000 * seed + i, True)
            for i in range(case["count"])]


def _layer_weights(case, seed):
    g = _gen(seed + 99)
    return torch.randn(case["count"], case["n"], generator=g, device="cuda", dtype=F64)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "kkt":
        p = _one_lp(case, seed)
        state.update(lp=p, point=_candidate(p, seed),
                     out=torch.empty(9, dtype=F64, device="cuda"))
    elif kind == "device":
        p = _one_lp(case, seed)
        state.update(lp=p, settings=_settings(case)._create(),
                     x=torch.empty(p["n"], dtype=F64, device="cuda"),
                     y=torch.empty(p["m"], dtype=F64, device="cuda"),
                     rc=torch.empty(p["n"], dtype=F64, device="cuda"))
    elif kind == "host":
        state.update(model=_data_model(_one_lp(case, seed)), settings=_settings(case))
    elif kind == "batch":
        state.update(models=[_data_model(p) for p in _batch_lps(case, seed)],
                     settings=_settings(case))
    elif kind == "branch":
        p = _one_lp(case, seed)
        # A relaxation's solution with `count` fractional variables among those between bounds.
        inside = torch.nonzero(p["x"] > 1.0).ravel()
        g = _gen(seed + 55)
        pick = torch.randperm(inside.numel(), generator=g, device="cuda")[:case["count"]]
        frac = inside[pick]
        state.update(model=_data_model(p), settings=_settings(case),
                     frac=frac.int().cpu().numpy(), root=p["x"][frac].cpu().numpy())
    else:
        lps = _layer_lps(case, seed)
        tensors = [LPInstance(p["c"], p["lo"], p["up"], p["val"], p["off"], p["idx"], p["vl"],
                              p["vu"]) for p in lps]
        for t in tensors:
            for v in (t.c, t.con_lo, t.con_up, t.values):
                v.requires_grad_(True)
        state.update(lps=tensors, weights=_layer_weights(case, seed), settings=_settings(case))
        if not case["train"]:
            state["solved"] = lp_solve_batch(tensors, state["settings"])
    torch.cuda.synchronize()
    return state


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _check(code, where):
    if code != 0:
        raise RuntimeError("%s returned %d" % (where, code))


def _run_kkt(s):
    p, (x, y, rc) = s["lp"], s["point"]
    _check(lib().cuOptComputeKKTErrorsNoAlloc(
        p["m"], p["n"], 1, 0.0, _ptr(p["c"]), _ptr(p["off"]), _ptr(p["idx"]), _ptr(p["val"]),
        _ptr(p["lo"]), _ptr(p["up"]), _ptr(x), _ptr(y), _ptr(rc),
        C.c_void_p(torch.cuda.current_stream().cuda_stream), _ptr(s["out"])), "KKT errors")
    return s["out"]


def _run_device(s):
    p, status = s["lp"], C.c_int32()
    _check(lib().cuOptSolveDevice(
        p["m"], p["n"], 1, 0.0, _ptr(p["c"]), _ptr(p["off"]), _ptr(p["idx"]), _ptr(p["val"]),
        _ptr(p["lo"]), _ptr(p["up"]), _ptr(p["vl"]), _ptr(p["vu"]), s["settings"],
        C.c_void_p(torch.cuda.current_stream().cuda_stream), _ptr(s["x"]), _ptr(s["y"]),
        _ptr(s["rc"]), None, C.byref(status)), "cuOptSolveDevice")
    return {"x": s["x"], "y": s["y"], "rc": s["rc"], "status": status.value}


def _vectors(solutions):
    """The solutions of a list of LPs, each kind of vector in one array."""
    return {"x": np.concatenate([v.get_primal_solution() for v in solutions]),
            "y": np.concatenate([v.get_dual_solution() for v in solutions]),
            "rc": np.concatenate([v.get_reduced_cost() for v in solutions]),
            "status": np.array([int(v.get_termination_status()) for v in solutions])}


def _run_layer(s):
    solved = s.get("solved") or lp_solve_batch(s["lps"], s["settings"])
    loss = sum((w * x).sum() for w, (x, _) in zip(s["weights"], solved))
    leaves = [v for t in s["lps"] for v in (t.c, t.con_lo, t.con_up, t.values)]
    grads = torch.autograd.grad(loss, leaves, retain_graph="solved" in s)
    out = {key: torch.cat(grads[i::4]) for i, key in enumerate(("dc", "dlo", "dup", "dval"))}
    if "solved" not in s:
        out.update(x=torch.cat([x.detach() for x, _ in solved]),
                   y=torch.cat([y.detach() for _, y in solved]))
    return out


def run(state):
    kind = state["case"]["kind"]
    if kind == "kkt":
        return _run_kkt(state)
    if kind == "device":
        return _run_device(state)
    if kind == "host":
        return _vectors([lpm.Solve(state["model"], state["settings"])])
    if kind == "batch":
        return _vectors(lpm.BatchSolve(state["models"], state["settings"])[0])
    if kind == "branch":
        return _vectors(lpm.BatchPDLPStrongBranching(state["model"], state["frac"], state["root"],
                                                     state["settings"])[0])
    return _run_layer(state)


# ---------------------------------------------------------------------------------------------


def _finite(v):
    return torch.where(torch.isfinite(v), v, 0.0)


def _exact_kkt(case, seed):
    p = _one_lp(case, seed)
    x, y, rc = _candidate(p, seed)
    off, idx = p["off"].long(), p["idx"].long()
    row = torch.repeat_interleave(torch.arange(p["m"], device="cuda"), off[1:] - off[:-1])
    ax = _row_sums(p["val"] * x[idx], off)
    by_col = torch.argsort(idx * p["m"] + row)
    aty = _row_sums((p["val"] * y[row])[by_col], _offsets(idx, p["n"]))
    rp = ax - torch.minimum(torch.maximum(ax, p["lo"]), p["up"])
    rd = p["c"] - aty - rc
    b2 = (torch.where(torch.isfinite(p["lo"]) & (p["lo"] != p["up"]), p["lo"], 0.0) ** 2).sum() + \
        (_finite(p["up"]) ** 2).sum()
    l2p, l2d = rp.norm(), rd.norm()
    primal = (p["c"] * x).sum()
    dual = (y.clamp(min=0) * _finite(p["lo"]) + y.clamp(max=0) * _finite(p["up"])).sum() + \
        (rc * x).sum()
    gap = (primal - dual).abs()
    return torch.stack([l2p, l2d, primal, dual, gap, l2p / (1 + b2.sqrt()),
                        l2d / (1 + p["c"].norm()), gap / (1 + primal.abs() + dual.abs()),
                        torch.zeros_like(gap)])


def _exact_layer(case, seed):
    """The vertex, and the implicit derivatives of sum(w x) there, from dense solves."""
    got = {key: [] for key in ("x", "y", "dlo", "dup", "dc", "dval")}
    for p, w in zip(_layer_lps(case, seed), _layer_weights(case, seed)):
        off, idx = p["off"].long(), p["idx"].long()
        row = torch.repeat_interleave(torch.arange(p["m"], device="cuda"), off[1:] - off[:-1])
        dense = torch.zeros(p["m"], p["n"], dtype=F64, device="cuda")
        dense[row, idx] = p["val"]
        basic = torch.nonzero(p["s"] == 0).ravel()
        lam = torch.linalg.solve(dense[:, basic].T, w[basic])
        got["x"].append(p["x"])
        got["y"].append(p["y"])
        got["dlo"].append(lam)
        got["dup"].append(torch.zeros_like(lam))
        got["dc"].append(torch.zeros_like(p["c"]))
        got["dval"].append(-lam[row] * p["x"][idx])
    return {key: torch.cat(v) for key, v in got.items()
            if case["train"] or key not in ("x", "y")}


def exact(case, seed):
    kind = case["kind"]
    if kind == "kkt":
        return _exact_kkt(case, seed)
    if kind == "layer":
        return _exact_layer(case, seed)
    if kind == "branch" or case.get("recipe") == "skewed":
        return None  # no closed form: another LP per branch; a run that ends at its limit
    lps = _batch_lps(case, seed) if kind == "batch" else [_one_lp(case, seed)]
    # The optimal duals and reduced costs are unique; the primal optimum is one of a face.
    return {"x": None, "y": torch.cat([p["y"] for p in lps]),
            "rc": torch.cat([p["s"] for p in lps]), "status": None}


def work(case):
    """One pass's necessary bytes (every input once, every output once) and operations.  A solve
    needs at least one product with A and one with its transpose; the iterations that it takes
    depend on the LP and are not counted."""
    kind = case["kind"]
    if kind == "batch":
        mid = (case["m_hi"] - case["m_lo"]) / math.log(case["m_hi"] / case["m_lo"])
        m = case["count"] * mid
        n, nnz = 2.5 * m, 2.5 * m * 9
    elif case.get("recipe") == "skewed":
        m, n, nnz = case["m"], case["n"], case["m"] * 150
    else:
        m, n = case["m"], case["n"]
        nnz = n * case["k"]
        if kind == "layer":
            # The backward pass: the matrix and the solution in, the four gradients out.
            m, n, nnz = m * case["count"], n * case["count"], nnz * case["count"]
    read = nnz * 12 + (m + 1) * 4 + 8 * (n + 2 * m)
    if kind == "kkt":
        return {"bytes": read + 8 * (2 * n + m) + 72, "flops": 4 * nnz + 8 * n + 8 * m}
    copies = 2 * case["count"] if kind == "branch" else 1
    flops = 4 * nnz * (2 if kind == "layer" else 1)
    written = 8 * (2 * n + m) + (8 * (nnz + n + 2 * m) if kind == "layer" else 0)
    return {"bytes": read + 16 * n + copies * written, "flops": copies * flops}
