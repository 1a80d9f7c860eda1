"""Cholesky factorization of tiles with +Inf on the diagonal (an overflowed covariance):
LAPACK's pivot test passes it, so the pivot becomes Inf, its column zero and info
stays 0, and the other rows and columns are the factor of the tile without that row
and column; and of tiles scaled so that pivots lie next to the ends of FP64's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _factor(hc, mats, up):
    import torch

    d = [torch.from_numpy(np.ascontiguousarray(m.T)).cuda() for m in mats]
    infos = hc.potrf_batched([hc.PotrfTask(uplo=ord(up), n=m.shape[0], A=x.data_ptr(), lda=m.shape[0])
                              for m, x in zip(mats, d)])
    tri = np.tril if up == "L" else np.triu
    out = [tri(x.cpu().numpy().T) for x in d]
    return infos, [x if up == "L" else x.T for x in out]


@pytest.mark.parametrize("up", ["L", "U"])
def test_infinite_pivots(hc, up):
    rng = np.random.default_rng(3)
    cases = [(1, 0), (16, 15), (20, 5), (40, 16), (64, 33), (70, 66), (130, 3), (130, 63), (200, 128)]
    mats, want = [], []
    for n, j in cases:
        X = rng.standard_normal((n, n))
        S = X @ X.T / n + np.eye(n)
        keep = np.arange(n) != j
        L = np.zeros((n, n))
        L[np.ix_(keep, keep)] = np.linalg.cholesky(S[np.ix_(keep, keep)]) if n > 1 else 0
        # row j: L(j, :j) from the columns before it
        L[j, :j] = np.linalg.solve(L[:j, :j], S[:j, j]) if j else 0
        L[j, j] = np.inf
        S[j, j] = np.inf
        mats.append(S)
        want.append(L)
    infos, got = _factor(hc, mats, up)
    assert list(infos) == [0] * len(cases)
    for (n, j), x, y in zip(cases, got, want):
        assert x[j, j] == np.inf and np.isinf(x).sum() == 1, (n, j)
        x[j, j] = y[j, j] = 0
        assert np.abs(x - y).max() <= 1e-12 * max(np.abs(y).max(), 1), (n, j)


def test_pivots_at_the_ends_of_the_range(hc):
    """a tile whose largest entry is FP64's largest number, against the same tile scaled down;
    a diagonal tile of subnormal, smallest and largest normal pivots"""
    rng = np.random.default_rng(4)
    X = rng.standard_normal((50, 50))
    S = X @ X.T / 50 + np.eye(50)
    S = S / np.abs(S).max()
    infos, (a, b) = _factor(hc, [S, np.ldexp(S * (1 - 2.0 ** -53), 1024)], "L")
    assert list(infos) == [0, 0] and np.isfinite(b).all()
    assert np.abs(np.ldexp(b, -512) - a).max() <= 1e-12
    d = np.array([5e-324, 1e-310, 2.2250738585072014e-308, 4.45e-308, np.finfo(float).max])
    infos, (x,) = _factor(hc, [np.diag(d)], "L")
    assert list(infos) == [0]
    assert np.abs(np.diag(x) / np.sqrt(d) - 1).max() <= 2.0 ** -52
