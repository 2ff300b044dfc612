"""The tensor-core exhaustive pass of the screened form (ct_digits.cuh) against the general exhaustive
kernels, which calls with few overflowed queries take.  Every pass computes a returned pair's distance
from the same double-float dot and kernel value, so the rows agree bit for bit.
"""
import numpy as np
import pytest

from oracle import oracle as O
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


def _check_healthy_rows(case, bad, q, gi, k, predecessor):
    """Neighbours other than the rows `bad` against the FP64 search over the rest: a row whose distances are
    not numbers takes no other row's place but its own."""
    n = len(case["p"])
    keep = np.delete(np.arange(n), bad)
    rank = np.cumsum(np.isin(np.arange(n), bad, invert=True)) - 1
    V, p, X = case["V"][keep], case["p"][keep], case["X"][keep]
    kk = k - len(bad)
    ri, _ = O.brute_knn_f64(V, p, X, 1.0, case["ls"], case["kt"], rank[q], kk, predecessor)
    got = np.full((len(q), kk), -1, np.int64)
    for r in range(len(q)):
        g = gi[r][(gi[r] >= 0) & ~np.isin(gi[r], bad)][:kk]
        got[r, :g.size] = rank[g]
    assert np.array_equal(got >= 0, ri >= 0)

    def dist_fn(r, ids):
        return O.residual_dist_f64(V, p, X, 1.0, case["ls"], case["kt"], np.array([rank[q[r]]]), ids)[0]

    _, mism = O.near_tie_mismatches(got, ri, dist_fn)
    assert not [t for t in mism if t[3] >= 1e-6]


# Rows of at most 2 x 2048 candidates: their survivor lists hold every candidate, so nothing but the
# pass's own rules can send them to the general kernels.
SHORT_ROWS = [(3000, 0, 3000, False), (24000, 1024, 4096, True)]


@pytest.mark.parametrize("n,lo,hi,predecessor", SHORT_ROWS)
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e20])
def test_digit_pass_short_rows_beside_a_row_without_a_scale(cuda_available, monkeypatch, n, lo, hi, predecessor, value):
    from covertreex_gb300.device import CudaResidualIndex

    case = gaussian_case(n, 3, 128, 1, 2.0, seed=5)
    V = case["V"].copy()
    V[777] = value
    idx = CudaResidualIndex(V, case["p"], case["X"], variance=1.0, lengthscale=case["ls"], kernel_type=1,
                            build_tree=False)
    monkeypatch.setenv("CT_SCREEN_SURVIVOR_CAP", "64")
    ids = np.delete(np.arange(n), 777)
    ids = ids[(ids >= lo) & (ids < hi)]
    q = np.sort(np.random.default_rng(6).choice(ids, 1500, replace=False)).astype(np.int64)
    gi, _ = idx.knn(q, 20, predecessor=predecessor, form="screened")
    assert idx.last_stats["overflow_queries"] > 0
    _check_healthy_rows(case, [777], q, gi, 20, predecessor)


@pytest.mark.parametrize("n,lo,hi,predecessor", SHORT_ROWS)
def test_digit_pass_short_rows_beside_residuals_without_a_root(cuda_available, monkeypatch, n, lo, hi, predecessor):
    """Negative, NaN and zero p: the pair's normalisation is the floor, so that such a row lies at distance 0
    of every query that is searched exhaustively; 1 / sqrt(p) is no number or infinite."""
    from covertreex_gb300.device import CudaResidualIndex

    case = gaussian_case(n, 3, 128, 1, 2.0, seed=5)
    bad = [100, 777, 1000]
    p = case["p"].copy()
    p[bad] = [-0.25, np.nan, 0.0]
    idx = CudaResidualIndex(case["V"], p, case["X"], variance=1.0, lengthscale=case["ls"], kernel_type=1,
                            build_tree=False)
    monkeypatch.setenv("CT_SCREEN_SURVIVOR_CAP", "64")
    ids = np.delete(np.arange(n), bad)
    ids = ids[(ids >= lo) & (ids < hi)]
    q = np.sort(np.random.default_rng(6).choice(ids, 1500, replace=False)).astype(np.int64)
    gi, _ = idx.knn(q, 20, predecessor=predecessor, form="screened")
    assert idx.last_stats["overflow_queries"] > 0
    _check_healthy_rows(case, bad, q, gi, 20, predecessor)
    if n == 3000:  # one candidate part: an overflowed query is searched over all rows, the others are screened,
        # which leaves rows without a number out
        listed = np.isin(gi, [100, 777]).sum(axis=1)
        assert np.all((listed == 0) | (listed == 2))
        assert np.count_nonzero(listed == 2) == idx.last_stats["overflow_queries"]


@pytest.mark.parametrize("n,d,m,kt,k,nq", [(6001, 2, 512, 0, 20, 3000), (20001, 1, 32, 0, 1, 6000), (6001, 2, 800, 1, 7, 3000)])
def test_digit_pass_against_the_general_kernels_of_the_same_call(cuda_available, monkeypatch, n, d, m, kt, k, nq):
    """One call on both passes: a last row with p = NaN, which no query below it sees, sends the second index's
    calls to the general kernels.  Every p is tiny here, where those evaluate each candidate exactly and the
    digit pass only its survivors, which shows which of the two ran."""
    from covertreex_gb300.device import CudaResidualIndex

    case = gaussian_case(n, d, m, kt, 2.0, seed=5)
    monkeypatch.setenv("CT_SCREEN_SURVIVOR_CAP", "64")
    q = np.random.default_rng(6).choice(np.arange(1024, n - 1), nq, replace=False).astype(np.int64)
    p = case["p"].copy()
    p[n - 1] = np.nan
    rows, share = [], []
    for pp in (case["p"], p):
        idx = CudaResidualIndex(case["V"], pp, case["X"], variance=1.0, lengthscale=case["ls"], kernel_type=kt,
                                build_tree=False)
        rows.append(idx.knn(q, k, predecessor=True, form="screened"))
        share.append(idx.last_stats["pairs_rescored"] / idx.last_stats["pairs_exhaustive"])
    assert share[0] < 0.5 and share[1] > 0.9, share
    assert np.array_equal(rows[0][0], rows[1][0])
    assert np.array_equal(rows[0][1].view(np.uint32), rows[1][1].view(np.uint32))


@pytest.mark.parametrize("m,k,nq", [(512, 64, 700), (512, 1, 700), (544, 64, 700), (96, 50, 3000)])
@pytest.mark.parametrize("predecessor", [False, True])
def test_survivor_pass_with_listed_slots(cuda_available, m, k, nq, predecessor):
    """More slots than one wave of full buffers: those with over 512 survivors are listed for a kernel of their
    own (at m = 544 none, one kernel takes all); calls of 40 queries are one kernel throughout."""
    from covertreex_gb300.device import CudaResidualIndex

    case = mixture_case(16384, 8, m, 2.0)
    idx = CudaResidualIndex(case["V"], case["p"], case["X"], variance=1.0, lengthscale=case["ls"], kernel_type=0,
                            build_tree=False)
    q = np.random.default_rng(8).choice(16384, nq, replace=False).astype(np.int64)
    gi, gd = idx.knn(q, k, predecessor=predecessor, form="screened")
    for s in range(0, 400, 40):
        hi, hd = idx.knn(q[s:s + 40], k, predecessor=predecessor, form="screened")
        assert np.array_equal(hi, gi[s:s + 40])
        assert np.array_equal(hd.view(np.uint32), gd[s:s + 40].view(np.uint32))
