"""Entry-wise accuracy of syrk and gemmcd updates with graded inner factors whose inner
product S is exact (columns of disjoint support): the factor AU S has columns of very
different sizes, and each keeps its own relative accuracy.

Bound: the product's (tests/test_gpu_dense_entrywise.py), (1.25 K + 1) 2^-45, and FP64 sums of K
terms in the factor, K 2^-52, of the sum of the terms' magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EXT = np.longdouble


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("M,r,n", [(300, 20, 1), (1024, 24, 80), (1024, 205, 1)])
def test_graded_inner_factors(hc, kind, M, r, n):
    import torch

    rng = np.random.default_rng(M + r + kind)
    U, V, W = rng.standard_normal((M, r)), np.zeros((M, r)), rng.standard_normal((M, r))
    V[np.arange(M), np.arange(M) % r] = rng.choice([-1.0, 1.0], M)
    V *= 2.0 ** -np.linspace(0, 60, r).round()
    u, v, w = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (U, V, W))
    cd = torch.zeros((n, M, M), dtype=torch.float64, device="cuda")
    if kind == 1:   # CD = -U (V^T V) Bu^T, Bu of the identity's columns on top: the factor's columns, one by one
        W[:] = 0
        W[np.arange(r), np.arange(r)] = 1
        w = torch.from_numpy(np.ascontiguousarray(W.T)).cuda()
    hc.dense_batched([hc.DenseTask(kind=kind, M=M, a=r, b=r, alpha=-1.0, Au=u.data_ptr(), Av=v.data_ptr(), lda=M,
                                   Bu=w.data_ptr(), Bv=v.data_ptr(), ldb=M, CD=cd[t].data_ptr(), ldcd=M)
                      for t in range(n)])
    out = cd.cpu().numpy()
    assert (out == out[:1]).all()
    X = U if kind == 0 else W
    S = np.diag(V.T @ V)   # (exact: powers of two, and nothing off the diagonal)
    rows = rng.choice(M, 60, replace=False)
    exact, total = -(U[rows].astype(EXT) * S) @ X.T.astype(EXT), (np.abs(U[rows]).astype(EXT) * S) @ np.abs(X).T.astype(EXT)
    err = np.abs(out[0].T[rows].astype(EXT) - exact)
    if kind == 0:
        upper = np.arange(M)[None, :] > rows[:, None]
        assert (out[0].T[rows][upper] == 0).all()
        err[upper] = 0
    assert (err <= ((1.25 * min(r, 128) + 1) * 2.0 ** -45 + r * 2.0 ** -52) * total).all()
