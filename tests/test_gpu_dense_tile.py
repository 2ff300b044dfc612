"""The dense tile at the sizes where its dispatch changes, bit for bit against the f32 oracle:
every column layout (straight-line stages at m = 64, 128, 256, 512; the general loop; the narrow
stages and two-word operands), tile and list edges, candidate splits, and residual variances that
are zero, negative, subnormal or infinite (no pair may be skipped that the reference's arithmetic
keeps)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(n, d, m, seed, special=False):
    r = np.random.default_rng(seed)
    X = r.standard_normal((n, d)).astype(np.float32)
    if n > 8:
        X[n // 2] = X[0]  # a duplicate point: equal distances, ties by index
    V = (r.standard_normal((n, m)) * np.sqrt(0.8 / m)).astype(np.float32)
    p = r.uniform(1e-3, 1.0, n).astype(np.float32)
    if special:
        p[::7] = r.choice(np.float32([0.0, -0.25, 1e-30, 1e-9, np.inf, 3e38]), p[::7].size)
    return V, p, X


def _check(V, p, X, kt, ls, q, k, pred, points=None):
    from covertreex_gb300.device import CudaResidualIndex

    lsv = np.full(X.shape[1], ls, np.float32)
    index = CudaResidualIndex(V, p, X, variance=1.0, lengthscale=lsv, kernel_type=kt, build_tree=False)
    gi, gd = index.knn(q, k, predecessor=pred, form="dense")
    oi, od = O.brute_knn_f32(V, p, X, 1.0, lsv, kt, q, k, pred)
    assert np.array_equal(gi, oi)
    assert np.array_equal(gd.view(np.uint32), od.view(np.uint32))


@pytest.mark.parametrize("m", [16, 32, 48, 64, 96, 128, 160, 256, 288, 512, 528, 640, 1024])
@pytest.mark.parametrize("special", [False, True])
def test_every_column_layout(cuda_available, m, special):
    V, p, X = _case(700, 3, m, 10 + m, special)
    q = np.random.default_rng(m).choice(700, 70, replace=False)
    _check(V, p, X, m // 16 % 2, 0.9, q, 20, False)
    _check(V, p, X, 1 - m // 16 % 2, 0.9, q, 20, True)


@pytest.mark.parametrize("n", [1, 2, 31, 63, 64, 65, 127, 129, 1025])
@pytest.mark.parametrize("k", [1, 32, 33, 64, 65, 128])
def test_tile_and_list_edges(cuda_available, n, k):
    V, p, X = _case(n, 2, 64, 100 + n)
    q = np.arange(n)[:: max(1, n // 40)]
    _check(V, p, X, 1, 1.0, q, k, False)
    _check(V, p, X, 0, 1.0, q, k, True)


@pytest.mark.parametrize("nq", [1, 15, 16, 17, 33, 257])
@pytest.mark.parametrize("d", [1, 3, 9])
def test_few_queries_split_over_the_chip(cuda_available, nq, d):
    V, p, X = _case(9000, d, 128, 7 * nq + d)
    q = np.random.default_rng(nq).integers(0, 9000, nq)
    _check(V, p, X, 1, 1.1, q, 50, False)
    _check(V, p, X, 0, 1.1, q, 50, True)


@pytest.mark.parametrize("kt,var", [(0, 2.5), (1, 0.3)])
def test_variance_scales_the_skip_test(cuda_available, kt, var):
    from covertreex_gb300.device import CudaResidualIndex

    V, p, X = _case(1500, 3, 256, 5)
    ls = np.float32([0.7, 1.3, 2.0])
    q = np.arange(0, 1500, 11)
    index = CudaResidualIndex(V, p, X, variance=var, lengthscale=ls, kernel_type=kt, build_tree=False)
    gi, gd = index.knn(q, 30, form="dense")
    oi, od = O.brute_knn_f32(V, p, X, var, ls, kt, q, 30, False)
    assert np.array_equal(gi, oi) and np.array_equal(gd.view(np.uint32), od.view(np.uint32))


@pytest.mark.parametrize("m,d,k", [(1936, 51, 113), (1936, 64, 80), (1952, 64, 68), (1968, 64, 56), (1936, 3, 128)])
@pytest.mark.parametrize("pred", [False, True])
def test_widest_rows_with_many_coordinates(cuda_available, m, d, k, pred):
    """The largest shared-memory needs of the 16-row tile, through the id, batch and allocation-free entry points."""
    import torch

    from covertreex_gb300 import _lib
    from covertreex_gb300.device import CudaBatch, CudaResidualIndex
    from tests.test_zz_no_alloc import _noalloc

    V, p, X = _case(300, d, m, m + d + k)
    ls = np.full(d, 2.0, np.float32)
    q = np.arange(0, 300, 7)
    index = CudaResidualIndex(V, p, X, variance=1.0, lengthscale=ls, kernel_type=1, build_tree=False)
    oi, od = O.brute_knn_f32(V, p, X, 1.0, ls, 1, q, k, pred)
    batch = CudaBatch()
    bi, bd = batch.add_ids(index, q, k, predecessor=pred)
    batch.run()
    rc, ni, nd = _noalloc(_lib.load(), dict(V=V, p=p, X=X, var=1.0, ls=ls, kt=1), q, k, pred, torch,
                          torch.cuda.current_stream())
    assert rc == 0
    for gi, gd in (index.knn(q, k, predecessor=pred, form="dense"), (bi.cpu().numpy(), bd.cpu().numpy()), (ni, nd)):
        assert np.array_equal(gi, oi) and np.array_equal(gd.view(np.uint32), od.view(np.uint32))


@pytest.mark.parametrize("m,d,k", [(1936, 51, 115), (1936, 64, 83), (1952, 64, 71), (1968, 64, 59)])
def test_widest_rows_of_the_single_tree_form(cuda_available, m, d, k):
    """The last sizes the 227 KB of a block hold (the batch kernel's own scalars leave it a little less)."""
    V, p, X = _case(300, d, m, m + d + k)
    _check(V, p, X, 1, 2.0, np.arange(0, 300, 7), k, False)
