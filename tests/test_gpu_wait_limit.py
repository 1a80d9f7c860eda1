"""A bounded wait that gives up inside the products on the tensor cores is an error of
the call that launched them, not a result: with a bound of one clock cycle every
caller reports it (POTRF does not take the NaN for a failed pivot, the compressor not
for a tile to hand to the pivoted QR), the tiles hold NaN, and the next call, with the
built-in bound, is right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def short_waits(hc):
    class Switch:
        def __enter__(self):
            hc.lib().hcore_gpu_test_wait_cycles(1)

        def __exit__(self, *a):
            hc.lib().hcore_gpu_test_wait_cycles(0)

    yield Switch()
    hc.lib().hcore_gpu_test_wait_cycles(0)


def _dev(x):
    import torch

    return torch.from_numpy(np.ascontiguousarray(x.T)).cuda()


@pytest.mark.parametrize("tiles,M", [(1, 40), (6, 700)])
def test_dense_tasks_and_plans(hc, short_waits, tiles, M):
    import torch

    rng = np.random.default_rng(M)
    U, V = rng.standard_normal((M, 20)), rng.standard_normal((M, 20))
    u, v, out = _dev(U), _dev(V), torch.zeros((tiles, M, M), dtype=torch.float64, device="cuda")
    tasks = [hc.DenseTask(kind=2, M=M, a=20, Au=u.data_ptr(), lda=M, Bv=v.data_ptr(), ldb=M,
                          CD=out[t].data_ptr(), ldcd=M) for t in range(tiles)]

    def right():
        ok = (out.cpu().numpy() == out[:1].cpu().numpy()).all() and np.abs(out[0].cpu().numpy().T - U @ V.T).max() < 1e-12
        out.zero_()
        return ok

    with short_waits, pytest.raises(hc.HcoreError, match="gave up"):
        hc.dense_batched(tasks)
    assert torch.isnan(out).any()
    hc.dense_batched(tasks)
    assert right()
    plan = hc.DensePlan(tasks)
    with short_waits:
        plan.execute()
        with pytest.raises(hc.HcoreError, match="gave up"):
            plan.status()
    plan.status()   # (reported once)
    plan.execute()
    plan.status()
    assert right()
    plan.close()


def test_factorization(hc, short_waits):
    rng = np.random.default_rng(1)
    n = 700
    X = rng.standard_normal((n, n))
    S = X @ X.T / n + np.eye(n)
    tiles = [_dev(S) for _ in range(4)]
    tasks = [hc.PotrfTask(uplo=ord("L"), n=n, A=d.data_ptr(), lda=n) for d in tiles]
    with short_waits, pytest.raises(hc.HcoreError, match="gave up"):
        hc.potrf_batched(tasks)
    for d in tiles:
        d.copy_(_dev(S))
    assert not np.any(hc.potrf_batched(tasks))
    assert np.abs(np.tril(tiles[3].cpu().numpy().T) - np.linalg.cholesky(S)).max() < 1e-12


def test_solves(hc, short_waits):
    rng = np.random.default_rng(2)
    n, vec = 700, 1300   # (more vectors than 8 * 152: by blocks)
    A = np.tril(rng.standard_normal((n, n)) / n) + np.eye(n)
    B = rng.standard_normal((n, vec))
    a, b = _dev(A), _dev(B)
    task = [hc.TrsmTask(side=141, uplo=122, trans=111, diag=131, M=n, N=vec, alpha=1.0, A=a.data_ptr(), lda=n,
                        B=b.data_ptr(), ldb=n)]
    with short_waits, pytest.raises(hc.HcoreError, match="gave up"):
        hc.trsm_batched(task)
    b.copy_(_dev(B))
    hc.trsm_batched(task)
    assert np.abs(b.cpu().numpy().T - np.linalg.solve(A, B)).max() < 1e-11


def test_compression(hc, short_waits):
    import torch

    M = 300
    p = np.random.default_rng(3).random((M, 2))
    D = np.exp(-((p[:, None] - p[None] - [0.7, 0.1]) ** 2).sum(-1) / 0.05)
    d = _dev(D)
    u, v = (torch.zeros((M, M), dtype=torch.float64, device="cuda") for _ in range(2))
    task = [hc.CompressTask(M=M, D=d.data_ptr(), ldd=M, acc=1e-8, relative=1, maxrank=M, U=u.data_ptr(),
                            V=v.data_ptr(), ldo=M)]
    with short_waits, pytest.raises(hc.HcoreError, match="gave up"):
        hc.compress_batched(task)
    ranks, status = hc.compress_batched(task)
    r = int(ranks[0])
    assert status[0] == 0 and np.abs((u[:r].T @ v[:r]).cpu().numpy() - D).max() < 1e-6 * np.abs(D).max()
