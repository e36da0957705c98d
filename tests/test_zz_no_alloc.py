"""GPU test of cuOptComputeKKTErrorsNoAlloc, the KKT evaluation that allocates no device memory.

It must report, for the point cuOptSolveDevice returns, the residuals, objectives and gap that
cuOptSolveDevice itself reports in its statistics, on two calls in a row (its static scratch is
cleared on every call); flag malformed column indices and row offsets with NaN outputs and a
count, and clear that count on the next call; and leave the device's free memory unchanged.
Tolerances: residual norms and relative errors within 1e-7 relative (summation order and the
atomic A^T y accumulation differ), objectives within 1e-10 relative, the gap within
1e-10 x (1 + |primal| + |dual|).

The file name keeps it last in collection order, after the tests that use the allocating paths.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from cuopt_b200 import generators as gen
from cuopt_b200._lib import PDLPStatistics, lib

pytestmark = pytest.mark.gpu

MAX_COLS = 1 << 19
RES_RTOL = 1e-7
OBJ_RTOL = 1e-10


def _settings(L, tol, iteration_limit=None):
    h = C.c_void_p()
    assert L.cuOptCreateSolverSettings(C.byref(h)) == 0
    for name in ("absolute_primal_tolerance", "relative_primal_tolerance", "absolute_dual_tolerance",
                 "relative_dual_tolerance", "absolute_gap_tolerance", "relative_gap_tolerance"):
        assert L.cuOptSetFloatParameter(h, name.encode(), tol) == 0
    assert L.cuOptSetParameter(h, b"log_to_console", b"false") == 0
    if iteration_limit is not None:
        assert L.cuOptSetIntegerParameter(h, b"iteration_limit", iteration_limit) == 0
    return h


def _device(lp, torch, c=None):
    dev = torch.device("cuda", 0)
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a), device=dev, dtype=dt)
    return {"c": t(lp.c if c is None else c, torch.float64), "off": t(lp.row_off, torch.int32),
            "idx": t(lp.col_idx, torch.int32), "val": t(lp.val, torch.float64),
            "lo": t(lp.con_lo, torch.float64), "up": t(lp.con_up, torch.float64),
            "vlo": t(lp.var_lo, torch.float64), "vup": t(lp.var_up, torch.float64),
            "x": torch.empty(lp.n, device=dev, dtype=torch.float64),
            "y": torch.empty(lp.m, device=dev, dtype=torch.float64),
            "rc": torch.empty(lp.n, device=dev, dtype=torch.float64)}


def _p(t):
    return C.c_void_p(t.data_ptr())


def _solve(L, torch, d, lp, sense, offset, settings):
    st, status = PDLPStatistics(), C.c_int32()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = L.cuOptSolveDevice(lp.m, lp.n, sense, offset, _p(d["c"]), _p(d["off"]), _p(d["idx"]),
                            _p(d["val"]), _p(d["lo"]), _p(d["up"]), _p(d["vlo"]), _p(d["vup"]),
                            settings, stream, _p(d["x"]), _p(d["y"]), _p(d["rc"]), C.byref(st),
                            C.byref(status))
    assert rc == 0
    torch.cuda.synchronize()
    return st, status.value


def _no_alloc(L, torch, d, lp, sense, offset, n=None, out=None, idx=None, off=None):
    if out is None:
        out = torch.full((9,), -1.0, device="cuda", dtype=torch.float64)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = L.cuOptComputeKKTErrorsNoAlloc(lp.m, lp.n if n is None else n, sense, offset, _p(d["c"]),
                                        _p(d["off"] if off is None else off),
                                        _p(d["idx"] if idx is None else idx), _p(d["val"]),
                                        _p(d["lo"]), _p(d["up"]), _p(d["x"]), _p(d["y"]),
                                        _p(d["rc"]), stream, _p(out))
    torch.cuda.synchronize()
    return rc, out.cpu().numpy()


def _check(st, out):
    assert out[8] == 0.0
    for got, want in ((out[0], st.l2_primal_residual), (out[1], st.l2_dual_residual),
                      (out[5], st.l2_relative_primal_residual),
                      (out[6], st.l2_relative_dual_residual), (out[7], st.relative_gap)):
        assert abs(got - want) <= RES_RTOL * abs(want) + 1e-14, (got, want)
    for got, want in ((out[2], st.primal_objective), (out[3], st.dual_objective)):
        assert abs(got - want) <= OBJ_RTOL * max(1.0, abs(want)), (got, want)
    scale = 1.0 + abs(st.primal_objective) + abs(st.dual_objective)
    assert abs(out[4] - st.gap) <= 1e-10 * scale


@pytest.mark.parametrize("sense,offset,iteration_limit", [(1, 0.0, None), (1, 0.0, 300),
                                                          (-1, 2.5, None)])
def test_no_alloc_matches_solver_statistics(sense, offset, iteration_limit):
    torch = pytest.importorskip("torch")
    L = lib()
    lp = gen.constructed_lp(2000, 5000, 8, seed=0)
    d = _device(lp, torch, c=lp.c if sense == 1 else -lp.c)
    s = _settings(L, 1e-6, iteration_limit)
    try:
        st, status = _solve(L, torch, d, lp, sense, offset, s)
    finally:
        L.cuOptDestroySolverSettings(C.byref(s))
    assert status == (1 if iteration_limit is None else 4)
    rc1, out1 = _no_alloc(L, torch, d, lp, sense, offset)
    rc2, out2 = _no_alloc(L, torch, d, lp, sense, offset)
    assert rc1 == 0 and rc2 == 0
    _check(st, out1)
    _check(st, out2)


def test_no_alloc_rejects_too_many_variables():
    torch = pytest.importorskip("torch")
    L = lib()
    lp = gen.constructed_lp(200, 500, 8, seed=1)
    d = _device(lp, torch)
    rc, out = _no_alloc(L, torch, d, lp, 1, 0.0, n=MAX_COLS + 1)
    assert rc == 1  # CUOPT_INVALID_ARGUMENT, before any device work
    assert np.all(out == -1.0)


def _solved_c0(L, torch):
    lp = gen.constructed_lp(2000, 5000, 8, seed=0)
    d = _device(lp, torch)
    s = _settings(L, 1e-6)
    try:
        st, status = _solve(L, torch, d, lp, 1, 0.0, s)
    finally:
        L.cuOptDestroySolverSettings(C.byref(s))
    assert status == 1
    return lp, d, st


def test_no_alloc_flags_bad_column_then_clears():
    """A column index equal to n is counted and skipped (NaN outputs); the next call with the
    original indices starts from a cleared count and gives the solver's statistics again."""
    torch = pytest.importorskip("torch")
    L = lib()
    lp, d, st = _solved_c0(L, torch)
    bad_idx = d["idx"].clone()
    bad_idx[123] = lp.n
    rc, out = _no_alloc(L, torch, d, lp, 1, 0.0, idx=bad_idx)
    assert rc == 0
    assert out[8] == 1.0
    assert np.all(np.isnan(out[:8]))
    rc, out = _no_alloc(L, torch, d, lp, 1, 0.0)
    assert rc == 0
    _check(st, out)


def test_no_alloc_flags_decreasing_row_offsets():
    """Row 5 given an end offset below its start is counted and skipped; every access stays inside
    the arrays (the neighbouring rows only grow or shrink within them)."""
    torch = pytest.importorskip("torch")
    L = lib()
    lp, d, st = _solved_c0(L, torch)
    off = d["off"].clone()
    assert int(off[5]) > 0
    off[6] = off[5] - 1
    rc, out = _no_alloc(L, torch, d, lp, 1, 0.0, off=off)
    assert rc == 0
    assert out[8] == 1.0
    assert np.all(np.isnan(out[:8]))
    rc, out = _no_alloc(L, torch, d, lp, 1, 0.0)
    assert rc == 0
    _check(st, out)


def test_no_alloc_leaves_free_memory_unchanged():
    """After a first call (which loads the library's device code and its static scratch), further
    calls take no device memory: the device's free bytes are the same before and after them."""
    torch = pytest.importorskip("torch")
    L = lib()
    lp, d, st = _solved_c0(L, torch)
    out = torch.full((9,), -1.0, device="cuda", dtype=torch.float64)
    rc, _ = _no_alloc(L, torch, d, lp, 1, 0.0, out=out)
    assert rc == 0
    torch.cuda.synchronize()
    free_before, _ = torch.cuda.mem_get_info()
    for _ in range(5):
        rc, res = _no_alloc(L, torch, d, lp, 1, 0.0, out=out)
        assert rc == 0
    torch.cuda.synchronize()
    free_after, _ = torch.cuda.mem_get_info()
    assert free_after == free_before
    _check(st, res)


@pytest.mark.parametrize("m,n,length", [
    (1, 1, 1), (1, 700, 700), (700, 1, 1), (1024, 1024, 5), (1024, 1025, 5),
    (512, 512, 5), (512, 513, 5), (40, 1280, 9), (40, 1281, 9),                # m n = 2^18, n = 32 m
    (3001, 5003, 12), (3001, 5003, 13), (1200, 5003, 48), (1200, 5003, 49),   # lanes per row
    (37, 900, 900), (9001, 400, 33)])
def test_no_alloc_sizes_against_numpy(m, n, length):
    """The evaluation of an arbitrary point at the edges of its forms (one cluster or two kernels,
    4, 8 or 32 lanes per row) against numpy; a row of every size down to empty, infinite bounds,
    an equality, and the second call after one on other sizes."""
    torch = pytest.importorskip("torch")
    L = lib()
    rng = np.random.default_rng(m + 7 * n + length)
    lens = np.full(m, min(length, n))
    lens[rng.random(m) < 0.1] = 0
    lens[0] = min(n, length + 40)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(0, n, off[-1]).astype(np.int32)
    val = rng.standard_normal(off[-1])
    x, rc, c = (rng.standard_normal(n) for _ in range(3))
    y = rng.standard_normal(m)
    lo = np.where(rng.random(m) < 0.3, -np.inf, rng.standard_normal(m))
    up = np.where(rng.random(m) < 0.3, np.inf, np.where(np.isfinite(lo), lo, 0.0) + 0.5)
    up[m // 2] = lo[m // 2] = 0.25
    rows = np.repeat(np.arange(m), lens)
    ax = np.bincount(rows, weights=val * x[idx], minlength=m)
    aty = np.bincount(idx, weights=val * y[rows], minlength=n)
    fin = lambda v: np.where(np.isfinite(v), v, 0.0)
    b2 = (np.where(lo != up, fin(lo), 0.0) ** 2).sum() + (fin(up) ** 2).sum()
    l2p, l2d = (np.linalg.norm(v) for v in (ax - np.clip(ax, lo, up), c - aty - rc))
    primal = c @ x + 2.5
    dual = np.maximum(y, 0) @ fin(lo) + np.minimum(y, 0) @ fin(up) + rc @ x + 2.5
    gap = abs(primal - dual)
    want = [l2p, l2d, primal, dual, gap, l2p / (1 + np.sqrt(b2)), l2d / (1 + np.linalg.norm(c)),
            gap / (1 + abs(primal) + abs(dual))]
    t = lambda a, dt=torch.float64: torch.as_tensor(a, device="cuda", dtype=dt)
    d = {"c": t(c), "off": t(off, torch.int32), "idx": t(idx, torch.int32), "val": t(val),
         "lo": t(lo), "up": t(up), "x": t(x), "y": t(y), "rc": t(rc)}
    lp = type("Sizes", (), {"m": m, "n": n})
    for _ in range(2):
        code, got = _no_alloc(L, torch, d, lp, 1, 2.5)
        assert code == 0 and got[8] == 0
        # Sums of at most a million terms of order 1 in FP64; the objectives are sums with
        # cancellation, so they are held relative to the size of their terms.
        size = 1 + np.abs(c * x).sum() + np.abs(rc * x).sum() + np.abs(y * fin(lo)).sum() + \
            np.abs(y * fin(up)).sum()
        for q in (0, 1, 5, 6):
            assert abs(got[q] - want[q]) <= 1e-12 * (1 + abs(want[q]))
        for q in (2, 3, 4, 7):
            assert abs(got[q] - want[q]) <= 1e-13 * size
    other = {**d, "off": t([0] * (m + 1), torch.int32)}
    code, got = _no_alloc(L, torch, other, lp, 1, 0.0)  # no entries: A x = 0, A^T y = 0
    assert code == 0 and abs(got[1] - np.linalg.norm(c - rc)) <= 1e-12 * (1 + got[1])


def _kkt_us(L, torch, m, n, lens):
    """Microseconds of one evaluation (best of seven times twenty)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    off = np.concatenate([[0], np.cumsum(lens)])
    f = lambda k: torch.randn(k, device="cuda", dtype=torch.float64, generator=g)
    d = {"c": f(n), "x": f(n), "rc": f(n), "y": f(m), "lo": f(m), "val": f(int(off[-1])),
         "off": torch.as_tensor(off, device="cuda", dtype=torch.int32),
         "idx": torch.arange(int(off[-1]), device="cuda", dtype=torch.int32) % n}
    d["up"] = d["lo"] + 1.0
    lp = type("Sizes", (), {"m": m, "n": n})
    out = torch.zeros(9, device="cuda", dtype=torch.float64)
    best = np.inf
    for _ in range(7):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record()
        for _ in range(20):
            assert L.cuOptComputeKKTErrorsNoAlloc(
                m, n, 1, 0.0, _p(d["c"]), _p(d["off"]), _p(d["idx"]), _p(d["val"]), _p(d["lo"]),
                _p(d["up"]), _p(d["x"]), _p(d["y"]), _p(d["rc"]),
                C.c_void_p(torch.cuda.current_stream().cuda_stream), _p(out)) == 0
        e1.record()
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1) * 50.0)
    assert out[8].item() == 0.0
    return best


@pytest.mark.parametrize("rest", [8, 20])  # 4 and 8 lanes for the other rows
def test_no_alloc_long_row_among_short_ones_takes_a_warp(rest):
    """One row over all variables among short ones costs what it costs alone, on a whole warp, and
    not what the few lanes of its neighbours take for it."""
    torch = pytest.importorskip("torch")
    L = lib()
    m, n = 20000, 50000
    lens = np.full(m, rest)
    short = _kkt_us(L, torch, m, n, lens)
    lens[777] = n
    assert _kkt_us(L, torch, m, n, lens) <= 1.25 * _kkt_us(L, torch, 1, n, [n]) + short


@pytest.mark.parametrize("m,n,length", [(1000, 1000, 1000), (64, 4096, 1024)])
def test_no_alloc_small_dense_rows_use_the_chip(m, n, length):
    """Entries of few rows and columns are spread over the SMs: the time of the same entries, in the same
    columns, among empty rows that make the LP a large one (1000 x 1000 on eight SMs took 68 us and
    not 44, 64 rows on two SMs 37 us and not 20)."""
    torch = pytest.importorskip("torch")
    L = lib()
    large = np.zeros((1 << 20) // n + 20, dtype=np.int64)
    large[:m] = length
    reference = _kkt_us(L, torch, len(large), n, large)
    assert _kkt_us(L, torch, m, n, np.full(m, length)) <= 1.25 * reference + 2.0


@pytest.mark.parametrize("m,n,rest,longs", [
    (300, 9000, 5, {0: 129, 1: 128, 2: 9000, 3: 257, 299: 130}),      # 4 lanes: from 129 on
    (333, 9000, 20, {0: 257, 7: 256, 8: 9000, 15: 300, 332: 9000})])  # 8 lanes: from 257 on
def test_no_alloc_long_rows_against_numpy(m, n, rest, longs):
    torch = pytest.importorskip("torch")
    L = lib()
    rng = np.random.default_rng(m)
    lens = np.full(m, rest)
    for i, l in longs.items():
        lens[i] = l
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(0, n, off[-1]).astype(np.int32)
    val = rng.standard_normal(off[-1])
    c, x, rc = (rng.standard_normal(n) for _ in range(3))
    y = rng.standard_normal(m)
    rows = np.repeat(np.arange(m), lens)
    ax = np.bincount(rows, weights=val * x[idx], minlength=m)
    aty = np.bincount(idx, weights=val * y[rows], minlength=n)
    t = lambda a, dt=torch.float64: torch.as_tensor(a, device="cuda", dtype=dt)
    d = {"c": t(c), "off": t(off, torch.int32), "idx": t(idx, torch.int32), "val": t(val),
         "lo": t(np.zeros(m)), "up": t(np.full(m, 0.5)), "x": t(x), "y": t(y), "rc": t(rc)}
    code, got = _no_alloc(L, torch, d, type("Sizes", (), {"m": m, "n": n}), 1, 0.0)
    assert code == 0 and got[8] == 0
    # Sums of at most 9000 terms of order 1 in FP64, as in test_no_alloc_sizes_against_numpy.
    for q, want in ((0, np.linalg.norm(ax - np.clip(ax, 0.0, 0.5))),
                    (1, np.linalg.norm(c - aty - rc))):
        assert abs(got[q] - want) <= 1e-12 * (1 + want)


@pytest.mark.parametrize("n", [700, 5003])  # one cluster, two kernels
def test_no_alloc_row_without_bounds_is_not_skipped(n):
    """A row whose bounds are both NaN restricts nothing (residual 0 for a finite product), but one
    whose product is not finite shows in the primal residual, and an infinite dual in the objective."""
    torch = pytest.importorskip("torch")
    L = lib()
    m = 300
    rng = np.random.default_rng(n)
    t = lambda a, dt=torch.float64: torch.as_tensor(a, device="cuda", dtype=dt)
    off, idx = np.arange(0, 2 * m + 1, 2), np.arange(2 * m) % n
    lo = np.zeros(m)
    up = np.full(m, 1.0)
    lo[7] = up[7] = np.nan
    x = np.zeros(n)
    x[idx[14]] = 1.0
    d = {"c": t(np.zeros(n)), "off": t(off, torch.int32), "idx": t(idx, torch.int32),
         "val": t(rng.uniform(1.0, 2.0, 2 * m)), "lo": t(lo), "up": t(up), "x": t(x),
         "y": t(np.zeros(m)), "rc": t(np.zeros(n))}
    lp = type("Sizes", (), {"m": m, "n": n})
    code, got = _no_alloc(L, torch, d, lp, 1, 0.0)
    assert code == 0 and got[0] == 0.0 and got[8] == 0.0
    x[idx[14]] = np.inf
    code, got = _no_alloc(L, torch, {**d, "x": t(x)}, lp, 1, 0.0)
    assert code == 0 and np.isnan(got[0]) and got[8] == 0.0
    y = np.zeros(m)
    y[7] = np.inf
    code, got = _no_alloc(L, torch, {**d, "y": t(y)}, lp, 1, 0.0)
    assert code == 0 and np.isnan(got[3]) and got[8] == 0.0
