"""The reference's power iteration taken from Golub-Kahan coefficients (krylov_power_iteration):
on the CPU against the iteration itself in numpy, on the GPU against the oracle's."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from cuopt_b200 import generators as gen
from cuopt_b200 import linear_programming as lpm
from .helpers import datamodel_from_lp, rel, settings

ROOT = Path(__file__).resolve().parents[1]
TOL, LIMIT = 1e-4, 5000
# Both sides round in every step; sigma_max^2 is a Rayleigh quotient, insensitive to that.
SIGMA_RTOL = 1e-12


@pytest.fixture(scope="module")
def in_krylov(tmp_path_factory):
    d = tmp_path_factory.mktemp("krylov")
    (d / "k.cpp").write_text(
        '#include "pdlp_schedule.hpp"\n'
        'using cuopt_b200::krylov_power_iteration;\n'
        'extern "C" void* fresh() { return new krylov_power_iteration; }\n'
        'extern "C" void release(void* p) { delete (krylov_power_iteration*)p; }\n'
        'extern "C" int advance(void* p, const double* a, const double* b, int steps, double* s2,'
        ' int* iters) {\n'
        '  auto& k = *(krylov_power_iteration*)p; const bool done = k.advance(a, b, steps);\n'
        '  *s2 = k.sigma2(); *iters = k.iterations(); return done; }\n')
    so = d / "k.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                    f"-I{ROOT / 'cuopt_b200' / 'csrc'}", str(d / "k.cpp"), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))
    lib.fresh.restype = C.c_void_p

    def call(coefficients, steps):
        """advance() of one object with each count of `steps` in turn, until it has ended."""
        p = C.c_void_p(lib.fresh())
        s2, it, ok = C.c_double(), C.c_int(), False
        for k in steps:
            a, b = (np.ascontiguousarray(v, dtype=np.float64) for v in coefficients(k))
            ok = bool(lib.advance(p, a.ctypes.data_as(C.c_void_p), b.ctypes.data_as(C.c_void_p),
                                  len(a), C.byref(s2), C.byref(it)))
            if ok:
                break
        lib.release(p)
        return ok, s2.value, it.value

    return call


def power(A, z):
    for k in range(1, LIMIT + 1):
        q = z / np.linalg.norm(z)
        z = A @ (A.T @ q)
        s2 = float(q @ z)
        if np.linalg.norm(z - s2 * q) < TOL:
            break
    return s2, k


def golub_kahan(A, z, steps):
    u, v, beta = z / np.linalg.norm(z), np.zeros(A.shape[1]), 0.0
    a, b = [], []
    with np.errstate(all="ignore"):
        for _ in range(steps):
            p = A.T @ u - beta * v
            a.append(np.linalg.norm(p))
            v = p / a[-1]
            q = A @ v - a[-1] * u
            beta = np.linalg.norm(q)
            b.append(beta)
            u = q / beta
    return a, b


@pytest.mark.parametrize("m,n,top", [(1, 1, None), (1, 7, None), (2, 2, None), (5, 3, None),
                                     (15, 40, None), (16, 40, None), (17, 40, None),
                                     (200, 450, None), (300, 500, 0.999), (120, 400, 0.9999)])
def test_krylov_power_iteration_matches_the_iteration(in_krylov, m, n, top):
    """Small and rank-deficient matrices (the recurrence ends early), random ones, and ones whose
    two largest singular values are close (thousands of power iterations)."""
    rng = np.random.default_rng(100 * m + n)
    A = rng.standard_normal((m, n)) / np.sqrt(n)
    if top is not None:
        U, s, V = np.linalg.svd(A, full_matrices=False)
        s = np.linspace(0.1, 0.8, len(s))[::-1].copy()
        s[0], s[1] = 1.0, top
        A = (U * s) @ V
    z = rng.standard_normal(m)
    want, k = power(A, z.copy())
    # Taken up again with 16 more steps each time, and from the steps it needs at once.
    for counts in (range(16, 1025, 16), [512]):
        ok, got, it = in_krylov(lambda steps: golub_kahan(A, z, steps), counts)
        assert ok and it == k
        assert abs(got - want) <= SIGMA_RTOL * want


def test_krylov_power_iteration_degenerate_input(in_krylov):
    """A zero matrix gives 0 at once, non-finite values never converge, and too few steps are not
    taken for a result."""
    nan = float("nan")
    assert in_krylov(lambda _: ([0.0, nan], [nan, nan]), [2]) == (True, 0.0, 1)
    ok, s2, it = in_krylov(lambda _: ([nan, nan], [nan, nan]), [2])
    assert ok and np.isnan(s2) and it == LIMIT
    rng = np.random.default_rng(3)
    A = rng.standard_normal((300, 600)) / 25.0
    z = rng.standard_normal(300)
    assert not in_krylov(lambda steps: golub_kahan(A, z, steps), [8])[0]


@pytest.mark.gpu
@pytest.mark.parametrize("lp", [
    gen.constructed_lp(1, 3, 1, seed=1), gen.constructed_lp(33, 70, 3, seed=2),
    gen.constructed_lp(313, 709, 7, seed=3), gen.constructed_lp(2000, 5000, 8, seed=4),
    gen.constructed_lp(9001, 20011, 6, seed=5), gen.vertex_lp(800, 1700, 8, seed=6),
    gen.skewed_lp(900, 3000, seed=7)], ids=lambda lp: f"{lp.name}{lp.m}")
def test_step_size_and_power_iterations_match_the_oracle(lp):
    """The step size and the reported number of power iterations are the oracle's, alone and in a
    batch."""
    from oracle import oracle as O

    want = O.solve(lp, tol=1e-12, iteration_limit=0)[0]
    s = settings(tol=1e-12, iteration_limit=0)
    single = lpm.Solve(datamodel_from_lp(lp), s)
    other = gen.constructed_lp(150, 330, 5, seed=9)
    batch, _ = lpm.BatchSolve([datamodel_from_lp(other), datamodel_from_lp(lp)], s)
    for sol in (single, batch[1]):
        assert rel(sol.stats["step_size"], want["step_size"]) <= SIGMA_RTOL
        assert sol.stats["power_iterations"] == want["power_iterations"]


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(5000, 65536), (65537, 30000), (5000, 65537)])
def test_step_size_where_the_norms_change_place(m, n):
    """Sweeps of 256 blocks sum the norm in the sweep that follows, sweeps of 257 in their last."""
    from oracle import oracle as O

    lp = gen.constructed_lp(m, n, 3, seed=n)
    want = O.solve(lp, tol=1e-12, iteration_limit=0)[0]
    got = lpm.Solve(datamodel_from_lp(lp), settings(tol=1e-12, iteration_limit=0)).stats
    assert rel(got["step_size"], want["step_size"]) <= SIGMA_RTOL
    assert got["power_iterations"] == want["power_iterations"]
