"""The dense tiles' products on the tensor cores (hc_dense_tc.cu) at the edges
of their blocks: rows around 32 and 128, inner dimensions around 16, 32 and 128
and several chunks, list order with scaling and zeroing between chunks, columns
whose scales compensate each other, subnormal and non-finite entries; against
the same products in numpy.

Tolerance: every term of an entry carries at most 2^-53 of the largest product
of a row with a row, and each chunk's addition rounds once; K + 8 times 2^-52 of
that product bounds both with a factor of two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def _dev(x):
    """column-major device copy of a numpy matrix"""
    import torch

    return torch.from_numpy(np.ascontiguousarray(x.T)).cuda()


def _uncompress(hc, U, V, cd0=None):
    import torch

    M, K = U.shape
    N = V.shape[0]
    out = torch.full((N, M), float("nan"), dtype=torch.float64, device="cuda") if cd0 is None else _dev(cd0)
    u, v = _dev(U), _dev(V)
    hc.dense_batched([hc.DenseTask(kind=2, M=M, N=N, a=K, Au=u.data_ptr(), lda=M, Bv=v.data_ptr(), ldb=N,
                                   CD=out.data_ptr(), ldcd=M)])
    return out.cpu().numpy().T


@pytest.mark.parametrize("M,N", [(1, 1), (31, 33), (32, 128), (127, 31), (128, 32), (129, 129), (260, 70)])
@pytest.mark.parametrize("K", [1, 15, 16, 17, 32, 33, 127, 128, 129, 300])
def test_uncompress_edges(hc, M, N, K):
    rng = np.random.default_rng(M * 1000 + N * 10 + K)
    U, V = rng.standard_normal((M, K)), rng.standard_normal((N, K)) * 10.0 ** rng.uniform(-3, 0, K)
    got = _uncompress(hc, U, V)
    bound = (K + 8) * EPS * np.abs(U).max() * np.abs(V).max()
    assert np.abs(got - U @ V.T).max() <= bound


def test_columns_with_compensating_scales(hc):
    """P's column 1e140 times and Q's 1e-140 times as large: an FP64 sum does not notice"""
    rng = np.random.default_rng(5)
    U, V = rng.standard_normal((200, 20)), rng.standard_normal((90, 20))
    f = 10.0 ** rng.uniform(-140, 140, 20)
    got = _uncompress(hc, U * f, V / f)
    assert np.abs(got - (U * f) @ (V / f).T).max() <= 28 * EPS * np.abs(U).max() * np.abs(V).max() * 4


def test_subnormal_products_and_zero_rows(hc):
    rng = np.random.default_rng(6)
    U, V = rng.standard_normal((140, 9)) * 1e-160, rng.standard_normal((40, 9)) * 1e-155
    U[7] = 0.0
    got = _uncompress(hc, U, V)
    assert np.abs(got - U @ V.T).max() <= 10 * 5e-324 * 2 + 17 * EPS * np.abs(U).max() * np.abs(V).max()
    assert (got[7] == 0).all()


def test_non_finite_entries_stay_where_they_are(hc):
    rng = np.random.default_rng(7)
    U, V = rng.standard_normal((150, 12)), rng.standard_normal((70, 12))
    U[3, 2], U[130, 0], V[40, 11] = np.nan, np.inf, -np.inf
    with np.errstate(invalid="ignore"):
        ref = U @ V.T
    got = _uncompress(hc, U, V)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    inf = np.isinf(ref)
    assert np.array_equal(got[inf], ref[inf])
    ok = np.isfinite(ref)
    assert np.abs(got[ok] - ref[ok]).max() <= 20 * EPS * 25


@pytest.mark.parametrize("M", [33, 128, 200])
def test_one_tile_in_list_order(hc, M):
    """syrk runs, products after them (also above the diagonal), a scaled and a beta = 0 task"""
    rng = np.random.default_rng(M)
    r = 11
    cd0 = rng.standard_normal((M, M))
    F = [rng.standard_normal((M, r)) for _ in range(8)]
    d = [_dev(x) for x in F]
    out = _dev(cd0)
    p = lambda i: d[i].data_ptr()  # noqa: E731
    syrk = lambda i, j: hc.DenseTask(kind=0, M=M, a=r, alpha=-0.5, Au=p(i), Av=p(j), lda=M, CD=out.data_ptr(), ldcd=M)  # noqa: E731
    gemm = lambda i, j, k, l: hc.DenseTask(kind=1, M=M, a=r, b=r, Au=p(i), Av=p(j), lda=M, Bu=p(k), Bv=p(l), ldb=M,  # noqa: E731
                                           CD=out.data_ptr(), ldcd=M)
    bd = rng.standard_normal((M, M))
    dbd = _dev(bd)
    scaled = hc.DenseTask(kind=3, M=M, N=M, a=r, alpha=2.0, beta=-0.25, kdim=M, Au=p(0), Av=p(1), lda=M,
                          Bd=dbd.data_ptr(), ldb=M, CD=out.data_ptr(), ldcd=M)
    hc.dense_batched([gemm(0, 1, 2, 3), syrk(0, 1), syrk(2, 3), gemm(4, 5, 6, 7), scaled, gemm(1, 2, 3, 4)])
    ref = cd0 - F[0] @ (F[1].T @ F[3]) @ F[2].T
    for i, j in ((0, 1), (2, 3)):
        ref = np.tril(ref - 0.5 * F[i] @ (F[j].T @ F[j]) @ F[i].T)
    ref = ref - F[4] @ (F[5].T @ F[7]) @ F[6].T
    ref = -0.25 * ref + 2.0 * F[0] @ (F[1].T @ bd)
    ref = ref - F[1] @ (F[2].T @ F[4]) @ F[3].T
    got = out.cpu().numpy().T
    # the factors' inner products over M rows carry M eps of their own
    assert np.abs(got - ref).max() <= 16 * M * EPS * np.abs(ref).max()


@pytest.mark.parametrize("M,N,K,r", [(1, 3, 5, 2), (40, 33, 129, 20), (130, 127, 300, 70), (64, 200, 16, 130)])
def test_low_rank_times_dense(hc, M, N, K, r):
    rng = np.random.default_rng(M + N)
    ld = max(M, K)
    U, V = rng.standard_normal((ld, r)), rng.standard_normal((ld, r))
    bd, cd = rng.standard_normal((K, N)), rng.standard_normal((M, N))
    du, dv, db, out = _dev(U), _dev(V), _dev(bd), _dev(cd)
    hc.dense_batched([hc.DenseTask(kind=3, M=M, N=N, a=r, alpha=-1.5, beta=0.5, kdim=K, Au=du.data_ptr(),
                                   Av=dv.data_ptr(), lda=ld, Bd=db.data_ptr(), ldb=K, CD=out.data_ptr(), ldcd=M)])
    ref = 0.5 * cd - 1.5 * U[:M] @ (V[:K].T @ bd)
    assert np.abs(out.cpu().numpy().T - ref).max() <= 16 * (K + r) * EPS * np.abs(ref).max()
