"""Active-set solves over the cluster shapes of the LSQR kernel: one system (the largest clusters),
many at once (small ones), sizes around a slice, operators that do not fit in shared memory, and
vectors that do not (one block, everything in global memory);
the gradients are those of the constructed vertex's basis (SciPy), to the adjoint tests' 1e-7."""
from __future__ import annotations

import numpy as np
import pytest

from cuopt_b200 import generators as gen
from .test_gpu_adjoint import _basis_derivatives, _close, _settings, _tensors

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _check(lps):
    from cuopt_b200.torch_layer import LPInstance, lp_solve_batch

    tensors = [_tensors(lp) for lp in lps]
    out = lp_solve_batch([LPInstance(**t) for t in tensors], _settings(tol=1e-6))
    rng = np.random.default_rng(5)
    w = [rng.standard_normal(lp.n) for lp in lps]
    v = [rng.standard_normal(lp.m) for lp in lps]
    f = lambda a: torch.tensor(a, device="cuda")
    sum((f(a) * x).sum() + (f(b) * y).sum() for a, b, (x, y) in zip(w, v, out)).backward()
    for lp, t, a, b in zip(lps, tensors, w, v):
        mu, lam, dval = _basis_derivatives(lp, a, b)
        _close(t["c"].grad.cpu().numpy(), mu, 1e-7)
        _close(t["con_lo"].grad.cpu().numpy(), lam, 1e-7)
        _close(t["values"].grad.cpu().numpy(), dval, 1e-7)


@pytest.mark.parametrize("m,n,k", [(3, 8, 2), (31, 64, 5), (32, 70, 5), (33, 70, 5), (257, 520, 6),
                                   (1500, 3100, 140)])  # the last: 4 MB of operators
def test_one_system(m, n, k):
    _check([gen.vertex_lp(m, n, k, seed=m)])


@pytest.mark.parametrize("count", [7, 40])
def test_many_systems(count):
    sizes = [(9, 20, 3), (33, 70, 5), (130, 260, 6), (300, 640, 7)]
    _check([gen.vertex_lp(*sizes[i % 4], seed=100 + i) for i in range(count)])


@pytest.mark.parametrize("m", [7200, 10000, 15000])
def test_vectors_beyond_shared_memory(m):
    """Rows and columns around what one block (7 100), then a cluster of 8 (12 500) holds; at 15 000,
    u, v, x and w are in global memory and one block runs the system."""
    _check([gen.vertex_lp(m, 2 * m + 100, 2, seed=9)])
