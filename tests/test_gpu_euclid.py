"""Exact Euclidean kNN at the edges of its tiles, steps and lists: sets and distances against FP64
(float32 sums of d squared differences are within (d + 2) 2^-24 of the exact square, relative),
ties to the lower index, rows with fewer neighbours padded."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _f32_brute(P, Q, k, pred):
    """The kernel's arithmetic (one FMA per axis, emulated in FP64: a product of two 24-bit
    differences and the sum are exact to 2^-53, rounded once to f32) and its (d^2, index) order."""
    s = np.zeros((Q.shape[0], P.shape[0]), np.float32)
    for c in range(P.shape[1]):
        df = (Q[:, None, c] - P[None, :, c]).astype(np.float32)
        s = (df.astype(np.float64) ** 2 + s).astype(np.float32)
    n = P.shape[0]
    idx = np.full((Q.shape[0], k), -1, np.int64)
    d2 = np.full((Q.shape[0], k), np.inf, np.float32)
    for i in range(Q.shape[0]):
        lim = min(i, n) if pred else n
        o = np.lexsort((np.arange(lim), s[i, :lim]))[:k]
        idx[i, :o.size], d2[i, :o.size] = o, s[i, o]
    return idx, d2


def _check(P, Q, k, pred):
    from covertreex_gb300.euclidean import EuclideanTree

    gi, gd = EuclideanTree(P).knn_device(Q, k, predecessor=pred)
    gi, gd = gi.cpu().numpy(), gd.cpu().numpy()
    oi, od2 = _f32_brute(P, Q, k, pred)
    assert np.array_equal(gi >= 0, oi >= 0)
    ok = oi >= 0
    # double rounding of the emulated FMA can differ from the device's in the last bit, so the
    # order is compared through distances, and the indices wherever neighbours are not that close
    od = np.sqrt(od2.astype(np.float64))
    tol = (P.shape[1] + 2) * 2.0 ** -24 * np.where(ok, od, 0) + 1e-30
    assert np.all(np.abs(gd.astype(np.float64) - np.where(ok, od, 0))[ok] <= tol[ok])
    assert np.all(gd[~ok] == np.float32(3.402823466e38))
    gap = np.minimum(np.diff(od, axis=1, prepend=-np.inf), np.diff(od, axis=1, append=np.inf))
    clear = ok & (gap > 4 * tol)
    assert np.array_equal(gi[clear], oi[clear])
    assert np.mean(clear[ok]) > 0.5 or P.shape[0] < 64


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 8, 16])
@pytest.mark.parametrize("n,nq", [(1, 1), (31, 40), (256, 33), (257, 32), (3000, 100)])
def test_tile_edges(cuda_available, d, n, nq):
    r = np.random.default_rng(d * 1000 + n)
    P = r.standard_normal((n, d)).astype(np.float32)
    Q = r.standard_normal((nq, d)).astype(np.float32)
    for k in (1, 10, 33, 64):
        _check(P, Q, k, False)
    _check(P, P[:nq], 10, True)


def test_ties_keep_the_lower_index_and_splits_agree(cuda_available):
    """Every point four times over: each query's list is its groups of four in index order."""
    from covertreex_gb300.euclidean import EuclideanTree

    r = np.random.default_rng(3)
    base = r.integers(-50, 50, (2500, 3)).astype(np.float32)  # exact squares, many ties
    P = np.concatenate([base] * 4)
    Q = base[:17]
    gi, gd = EuclideanTree(P).knn_device(Q, 30)
    s = ((Q[:, None].astype(np.int64) - P[None].astype(np.int64)) ** 2).sum(2)
    for i in range(17):
        o = np.lexsort((np.arange(P.shape[0]), s[i]))[:30]
        assert np.array_equal(gi[i].cpu().numpy(), o)
        assert np.array_equal(gd[i].cpu().numpy(), np.sqrt(s[i, o].astype(np.float32)))


def test_infinite_and_nan_points_are_no_neighbours(cuda_available):
    from covertreex_gb300.euclidean import EuclideanTree

    P = np.random.default_rng(1).standard_normal((300, 3)).astype(np.float32)
    P[5], P[6, 1], P[7, 2] = np.nan, np.inf, 3e38
    gi, _ = EuclideanTree(P).knn_device(P[:4], 64)
    assert not np.isin(gi.cpu().numpy(), [5, 6, 7]).any()


@pytest.mark.parametrize("n,nq,k", [(592, 40, 1), (593, 40, 1), (472, 9, 16), (473, 9, 16), (568, 8, 4), (560, 8, 5),
                                    (408, 33, 24), (409, 33, 24), (400, 12, 17), (512, 390, 10), (512, 400, 10),
                                    (16, 20000, 4), (300, 20000, 10)])
@pytest.mark.parametrize("d", [1, 3, 16])
def test_few_points_on_both_sides_of_the_line(cuda_available, n, nq, k, d):
    """The warp-per-query form and the tile around the line between them, with repeated points (ties by index)
    and points that are no neighbours."""
    r = np.random.default_rng(n + nq + k + d)
    P = r.standard_normal((n, d)).astype(np.float32)
    P[n // 2:n // 2 + 8] = P[:8]
    Q = P[r.integers(0, n, nq)] if nq <= n else r.standard_normal((nq, d)).astype(np.float32)
    _check(P, Q, k, False)
    _check(P, P[:min(n, nq)], k, True)
    P[5], P[n - 3] = np.nan, np.inf
    _check(P, Q, k, False)
