"""The tensor-core exhaustive pass of the screened form (ct_digits.cuh) against the general exhaustive
kernels, which calls with few overflowed queries take.  Every pass computes a returned pair's distance
from the same double-float dot and kernel value, so the rows agree bit for bit.
"""
import numpy as np
import pytest

from tests._data import gaussian_case, mixture_case

pytestmark = pytest.mark.gpu


def _check(idx, q, k, predecessor=False, few=15, checked=150):
    gi, gd = idx.knn(q, k, predecessor=predecessor, form="screened")
    assert idx.last_stats["overflow_queries"] > 0
    for s in range(0, min(len(q), checked), few):
        hi, hd = idx.knn(q[s:s + few], k, predecessor=predecessor, form="screened")
        assert np.array_equal(hi, gi[s:s + few])
        assert np.array_equal(hd.view(np.uint32), gd[s:s + few].view(np.uint32))


@pytest.mark.parametrize("n,d,m,kt,k,nq,predecessor", [
    (40001, 1, 32, 0, 1, 4225, False),    # the smallest m; one candidate in the last tile, one query in the last row tile
    (30000, 3, 96, 1, 40, 5000, True),    # more rows than a batch
    (24000, 8, 512, 0, 50, 1500, False),
    (6000, 2, 800, 1, 7, 3000, True),     # the largest m
    (6000, 2, 832, 1, 7, 3000, True),     # one chunk above it: the general kernels
    (30000, 3, 64, 1, 64, 8000, True),    # the largest k, rows with few predecessors
])
def test_digit_pass_equals_general_pass(cuda_available, monkeypatch, n, d, m, kt, k, nq, predecessor):
    from covertreex_gb300.device import CudaResidualIndex

    case = gaussian_case(n, d, m, kt, 2.0, seed=5)
    idx = CudaResidualIndex(case["V"], case["p"], case["X"], variance=1.0, lengthscale=case["ls"], kernel_type=kt,
                            build_tree=False)
    monkeypatch.setenv("CT_SCREEN_SURVIVOR_CAP", "64")  # overflows most queries
    q = np.random.default_rng(6).choice(n, nq, replace=False).astype(np.int64)
    q[:30] = np.sort(q)[:30] if predecessor else q[:30]
    _check(idx, q, k, predecessor)


def test_digit_pass_repeated_rows_and_tiny_residuals(cuda_available):
    """Inducing points (p at its floor) and rows that occur thousands of times: more ties than a row's
    survivor list holds, which go back to the general kernels."""
    from covertreex_gb300.device import CudaResidualIndex

    case = mixture_case(20000, 2, 64, 2.0)
    X, V, p = (case[x].copy() for x in ("X", "V", "p"))
    X[3000:9000], V[3000:9000], p[3000:9000] = X[17], V[17], p[17]
    idx = CudaResidualIndex(V, p, X, variance=1.0, lengthscale=case["ls"], kernel_type=0, build_tree=False)
    q = np.concatenate([np.asarray(case["inducing"][:64]), np.arange(3000, 3040), np.arange(9000, 11000)])
    _check(idx, q.astype(np.int64), 20)


def test_digit_pass_leaves_norms_without_a_scale_to_the_general_pass(cuda_available, monkeypatch):
    """One V row whose squared norm overflows: no scale of the digits holds it."""
    from covertreex_gb300.device import CudaResidualIndex

    case = gaussian_case(24000, 3, 128, 1, 2.0, seed=5)
    V = case["V"].copy()
    V[777] = 1e20
    idx = CudaResidualIndex(V, case["p"], case["X"], variance=1.0, lengthscale=case["ls"], kernel_type=1,
                            build_tree=False)
    monkeypatch.setenv("CT_SCREEN_SURVIVOR_CAP", "64")
    q = np.random.default_rng(6).choice(np.delete(np.arange(24000), 777), 1500, replace=False).astype(np.int64)
    _check(idx, q, 20)
