"""Entry-wise accuracy of the products on the tensor cores (hc_dense_tc.cu): an entry is
off by at most a small multiple of the sum of its terms' magnitudes, as in an FP64 sum,
also where the rows' largest entries meet small ones only, so that the entry is far
below the product of the rows' scales.

Bound.  In units of the rows' scales times 2^-55 a column's two rounded factors are off by
half a unit each times a value below 1, the dropped digit products of a column by less than
an eighth, the last rounding by half: 1.125 K + 0.5 units for K columns of a chunk.  Entries
whose result is below 2^45 units, as is the entry that it is added to, and whose rows share no
column within 2^-4 of both tops are summed in FP64; any other's terms, the old entry among them,
add up to 2^45 units at least.  So the error is at most (1.25 K + 1) 2^-45 of that sum, chunk by
chunk; FP64's own share, K 2^-53, is inside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NOTRANS, TRANS, UPPER, LOWER, NONUNIT, UNIT, LEFT, RIGHT = 111, 112, 121, 122, 131, 132, 141, 142
EXT = np.longdouble


def _dev(x, ld=None):
    import torch

    ld = ld or x.shape[0]
    d = torch.full((x.shape[1], ld), float("nan"), dtype=torch.float64, device="cuda")
    d[:, :x.shape[0]] = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    return d


def _check(hc, P, Q):
    import torch

    (M, K), N = P.shape, Q.shape[0]
    p, q, out = _dev(P), _dev(Q), torch.zeros((N, M), dtype=torch.float64, device="cuda")
    hc.dense_batched([hc.DenseTask(kind=2, M=M, N=N, a=K, Au=p.data_ptr(), lda=M, Bv=q.data_ptr(), ldb=N,
                                   CD=out.data_ptr(), ldcd=M)])
    exact, total = P.astype(EXT) @ Q.astype(EXT).T, np.abs(P).astype(EXT) @ np.abs(Q).astype(EXT).T
    bound = (1.25 * min(K, 128) + 1) * 2.0 ** -45 * total + 1e-322
    assert (np.abs(out.cpu().numpy().T.astype(EXT) - exact) <= bound).all()


@pytest.mark.parametrize("e", [1e-2, 1e-3, 1e-5, 1e-10, 1e-14, 1e-18, 1e-100])
def test_large_entries_that_meet_small_ones(hc, e):
    """the two by two pattern, alone and spread over rows and columns of a larger product"""
    a, b = 4 / 3, 8 / 7
    P, Q = np.array([[1, a * e], [b * e, 1]]), np.array([[e, a], [b, e]])
    _check(hc, P, Q)
    rng = np.random.default_rng(2)
    for K, at in ((20, (3, 17)), (50, (30, 40)), (128, (100, 5)), (200, (0, 199))):
        X, Y = np.zeros((40, K)), np.zeros((70, K))
        X[:, at[0]], X[:, at[1]] = rng.uniform(1, 2, 40), e * rng.uniform(1, 2, 40)
        Y[:, at[0]], Y[:, at[1]] = e * rng.uniform(1, 2, 70), rng.uniform(1, 2, 70)
        X[::2, list(at)] = X[::2, list(at[::-1])]
        Y[::3, list(at)] = Y[::3, list(at[::-1])]
        _check(hc, X, Y)


@pytest.mark.parametrize("K", [1, 2, 5, 17, 32, 33, 64, 127, 128, 129, 300])
@pytest.mark.parametrize("decades", [2, 8, 30])
def test_entries_of_any_size(hc, K, decades):
    rng = np.random.default_rng(100 * K + decades)
    draw = lambda n: rng.standard_normal((n, K)) * 10.0 ** rng.uniform(-decades, 0, (n, K))  # noqa: E731
    P, Q = draw(150), draw(70)
    P[rng.random(P.shape) < 0.1] = 0
    P[7] = 0
    _check(hc, P, Q)


@pytest.mark.parametrize("n", [448, 513])
def test_every_solve_by_blocks_of_a_graded_triangle(hc, n):
    """80 vectors a task, 1280 together: enough for the solve by blocks (a solve by blocks, and only it, has
    waits that can give up).  Off-diagonal entries of any size up to 1 / n, rows and columns scaled besides;
    the residual's bound is that of the products, 64 columns each, and of n FP64 operations."""
    rng = np.random.default_rng(n)
    tasks, keep = [], []
    for side in (LEFT, RIGHT):
        for uplo in (UPPER, LOWER):
            for tr in (NOTRANS, TRANS):
                for dg in (NONUNIT, UNIT):
                    M, N = (n, 80) if side == LEFT else (80, n)
                    A = rng.choice([-1.0, 1.0], (n, n)) * 10.0 ** rng.uniform(-14, 0, (n, n)) / n
                    A[np.arange(n), np.arange(n)] = 1.0 if dg == UNIT else 1.0 + rng.random(n)
                    if dg == NONUNIT:
                        A = (10.0 ** rng.uniform(-6, 6, n))[:, None] * A * 10.0 ** rng.uniform(-6, 6, n)
                    A = np.tril(A) if uplo == LOWER else np.triu(A)
                    stored = A.copy()
                    if dg == UNIT:
                        stored[np.arange(n), np.arange(n)] = np.nan
                    B = rng.standard_normal((M, N)) * 10.0 ** rng.uniform(-8, 0, (M, N))
                    dA, dB = _dev(stored, n + 2), _dev(B, M + 5)
                    keep.append((A if tr == NOTRANS else A.T, B, dA, dB, side))
                    tasks.append(hc.TrsmTask(side=side, uplo=uplo, trans=tr, diag=dg, M=M, N=N, alpha=-0.75,
                                             A=dA.data_ptr(), lda=n + 2, B=dB.data_ptr(), ldb=M + 5))
    before = [k[3].clone() for k in keep]
    hc.lib().hcore_gpu_test_wait_cycles(1)
    try:
        with pytest.raises(hc.HcoreError, match="gave up"):
            hc.trsm_batched(tasks)
    finally:
        hc.lib().hcore_gpu_test_wait_cycles(0)
    for k, b in zip(keep, before):
        k[3].copy_(b)
    hc.trsm_batched(tasks)
    for A, B, _, dB, side in keep:
        X = dB.cpu().numpy()[:, :B.shape[0]].T
        if side == RIGHT:   # X op(A) = alpha B, transposed
            A, B, X = A.T, B.T, X.T
        cols = rng.choice(B.shape[1], 3, replace=False)
        A, X, B = A.astype(EXT), X[:, cols].astype(EXT), B[:, cols].astype(EXT)
        total = np.abs(A) @ np.abs(X) + 0.75 * np.abs(B)
        assert (np.abs(A @ X + 0.75 * B) <= ((1.25 * 64 + 1) * 2.0 ** -45 + 4 * n * 2.0 ** -53) * total).all()
