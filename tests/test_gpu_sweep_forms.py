"""Edges of the sweeps' forms: every form of the plain iterations and every block shape computes the
same iterates bit for bit, at the sizes where slices, wide rows and cluster shares begin and end,
and the oracle's to its parity tolerance."""
from __future__ import annotations

import numpy as np
import pytest

from cuopt_b200 import generators as gen
from cuopt_b200 import linear_programming as lpm
from .helpers import datamodel_from_lp, settings

pytestmark = pytest.mark.gpu

GRAPHS, PERSISTENT, CLUSTER = 0, 1, 2
ITERATE_RTOL = 1e-9  # the repository's parity tolerance for iterates against the oracle


def _solve(lp, form, limit, precision=0, wpb=0):
    s = settings(tol=1e-13, iteration_limit=limit, precision=precision)
    s.set_parameter(lpm.CUOPT_PDLP_PERSISTENT_ITERATIONS, form)
    if wpb:
        s.set_parameter(lpm.CUOPT_PDLP_SWEEP_WARPS_PER_BLOCK, wpb)
    return lpm.Solve(datamodel_from_lp(lp), s)


def _same(a, b):
    assert a.get_lp_stats()["nb_iterations"] == b.get_lp_stats()["nb_iterations"]
    for f in ("get_primal_solution", "get_dual_solution", "get_reduced_cost"):
        assert np.array_equal(getattr(a, f)(), getattr(b, f)())


def _lp(kind, m, n, k):
    if kind == "wide":  # rows on both sides of 512 elements, and of several thousand
        return gen.skewed_lp(m, n, seed=m + n, zipf_a=0.7, cap=k)
    return gen.constructed_lp(m, n, k, seed=m + n)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind,m,n,k", [
    ("plain", 1, 2, 1), ("plain", 31, 64, 3), ("plain", 32, 65, 3), ("plain", 33, 96, 5),
    ("plain", 511, 1025, 4), ("plain", 1500, 3601, 13),  # shares of more than one unit a warp
    ("wide", 60, 2500, 2500), ("wide", 37, 520, 520)])
def test_forms_are_bit_identical(kind, m, n, k, precision):
    """230 iterations: checks every 10, a restart at 200 (so that the anchor is not zero)."""
    lp = _lp(kind, m, n, k)
    ref = _solve(lp, GRAPHS, 230, precision)
    _same(ref, _solve(lp, PERSISTENT, 230, precision))
    c = _solve(lp, CLUSTER, 230, precision)
    assert c.stats["plain_iteration_form"] == CLUSTER
    _same(ref, c)
    for wpb in (4, 16):
        _same(ref, _solve(lp, GRAPHS, 230, precision, wpb))


@pytest.mark.parametrize("m,n,k", [(300, 1280, 4), (300, 1281, 4),     # 4 blocks of 10 slices; 8
                                   (2560, 700, 5), (2561, 700, 5),     # 8 blocks of 10 slices; 16
                                   (2000, 5120, 5), (2000, 5121, 5)])  # 16 of 10; several a warp
def test_cluster_sizes_at_their_last_slice(m, n, k):
    """One slice a warp while a side has at most 10 per block, in the smallest cluster that holds it."""
    lp = gen.constructed_lp(m, n, k, seed=m + n)
    for precision in (0, 1):
        c = _solve(lp, CLUSTER, 230, precision)
        assert c.stats["plain_iteration_form"] == CLUSTER
        _same(_solve(lp, GRAPHS, 230, precision), c)


@pytest.mark.parametrize("m,n,k", [(65, 161, 30), (33, 161, 14), (320, 1280, 15)])
def test_cluster_exchange_behind_long_gathers(m, n, k):
    """A slice's first entry releases the vector that its other lanes have just gathered: slices of
    many chunks (long gathers between the wait and the sends), last slices of one row (lane 0 sends
    alone) and of 32, over 590 iterations."""
    lp = gen.constructed_lp(m, n, k, seed=m + n)
    for precision in (0, 1):
        c = _solve(lp, CLUSTER, 590, precision)
        assert c.stats["plain_iteration_form"] == CLUSTER
        _same(_solve(lp, GRAPHS, 590, precision), c)


@pytest.mark.parametrize("limit", [1200, 1300])
def test_cluster_form_checks_every_hundred_iterations(limit):
    lp = gen.constructed_lp(150, 333, 5, seed=4)
    _same(_solve(lp, GRAPHS, limit), _solve(lp, CLUSTER, limit))


@pytest.mark.parametrize("form", [PERSISTENT, CLUSTER])
@pytest.mark.parametrize("tol,refine", [(1e-5, True), (1e-10, False)])
def test_fp64_continuation_takes_over_the_kept_iterates(form, tol, refine):
    """The FP64 continuation starts from the iterates of the check that ended the mixed solve: one that
    met its tolerance and is refined, and one that stalled (FP32 does not reach 1e-10)."""
    lp = gen.constructed_lp(300, 700, 6, seed=12)
    out = []
    for f in (GRAPHS, form):
        s = settings(tol=tol, precision=1)
        s.set_parameter(lpm.CUOPT_PDLP_PERSISTENT_ITERATIONS, f)
        if refine:
            s.set_parameter(lpm.CUOPT_PDLP_REFINEMENT_PASSES, 1)
            s.set_parameter(lpm.CUOPT_PDLP_REFINEMENT_TOLERANCE, 1e-8)
        out.append(lpm.Solve(datamodel_from_lp(lp), s))
        assert out[-1].get_termination_status() == lpm.LPTerminationStatus.Optimal
        assert out[-1].stats["refinement_passes"] == 1
        assert out[-1].stats["plain_iteration_form"] == f
    _same(out[0], out[1])


@pytest.mark.parametrize("m,n,cap", [(400, 7000, 5000), (2500, 9000, 1200)])
def test_wide_rows_follow_the_oracle(m, n, cap):
    from oracle import oracle as O

    lp = gen.skewed_lp(m, n, seed=m, cap=cap)
    assert np.diff(lp.row_off).max() > 512
    for limit in (10, 200, 210):
        res, x, y, _ = O.solve(lp, tol=1e-13, iteration_limit=limit)
        sol = _solve(lp, GRAPHS, limit)
        assert sol.get_lp_stats()["nb_iterations"] == res["iterations"]
        for got, want in ((sol.get_primal_solution(), x), (sol.get_dual_solution(), y)):
            assert np.max(np.abs(got - want)) <= ITERATE_RTOL * (1 + np.abs(want).max())


@pytest.mark.parametrize("kind", ["plain", "long", "wide"])
@pytest.mark.parametrize("limit", [10, 190])
def test_climbers_and_batches_follow_single_solves_bit_by_bit(kind, limit):
    """Before the first restart nothing but the rows' sums can differ: climbers and batch instances
    have a single solve's iterates, also with rows of more than 512 elements."""
    lp = {"plain": lambda: gen.constructed_lp(300, 700, 6, seed=3),
          "long": lambda: gen.skewed_lp(60, 400, seed=9, zipf_a=0.7, cap=400),
          "wide": lambda: gen.skewed_lp(60, 2500, seed=9, zipf_a=0.7, cap=2500)}[kind]()
    s = settings(tol=1e-13, iteration_limit=limit)
    single = lpm.Solve(datamodel_from_lp(lp), s)
    var = np.array([0, lp.n // 2, lp.n - 1], np.int32)
    for sol in (lpm.SolveClimbers(datamodel_from_lp(lp), var, lp.var_lo[var], lp.var_up[var], s)[0] +
                lpm.BatchSolve([datamodel_from_lp(lp)] * 2, s)[0]):
        _same(single, sol)
        assert sol.stats["step_size"] == single.stats["step_size"]


@pytest.mark.parametrize("seed", range(4))
def test_tiled_copy_with_a_gap_behind_the_long_rows(seed):
    """Long rows whose elements end off a chunk leave a gap before the slices; the tiled copy takes
    its elements for padding (tiles are refused or not, the FP32 iterates stay close)."""
    lp = gen.skewed_lp(300, 2000 + seed, seed=20 + seed, zipf_a=0.7, cap=300)
    out = []
    for tiled in (0, 1):
        s = settings(tol=1e-13, iteration_limit=20, precision=1)
        s.set_parameter(lpm.CUOPT_PDLP_TILED_SWEEPS, tiled)
        out.append(lpm.Solve(datamodel_from_lp(lp), s).get_primal_solution())
    assert np.linalg.norm(out[0] - out[1]) <= 1e-4 * np.linalg.norm(out[0])
