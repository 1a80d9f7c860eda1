"""Triangular solves by blocks and Cholesky updates as products (hc_tlr.cu), from
the orders where they take over: all 16 solve cases with ragged last blocks,
padded leading dimensions and NaN in every entry that must not be read; tiles
whose early updates are products and whose late ones are not, both triangles, a
failing pivot beside them.  Against the oracle, with the bounds of the smaller
solves and factorizations' tests (1e-12 of the largest entry)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NOTRANS, TRANS, UPPER, LOWER, NONUNIT, UNIT, LEFT, RIGHT = 111, 112, 121, 122, 131, 132, 141, 142


def _close(x, y, tol):
    assert np.array_equal(np.isnan(x), np.isnan(y))
    ok = ~np.isnan(y)
    assert np.abs(x[ok] - y[ok]).max() <= tol * np.abs(y[ok]).max()


def _dev(x, ld):
    import torch

    d = torch.full((x.shape[1], ld), float("nan"), dtype=torch.float64, device="cuda")
    d[:, :x.shape[0]] = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    return d


def _triangle(rng, n, uplo, unit):
    A = rng.standard_normal((n, n)) / n
    A[np.arange(n), np.arange(n)] = np.nan if unit else 1.0 + rng.random(n)
    mask = np.triu(np.ones((n, n), bool), 1) if uplo == LOWER else np.tril(np.ones((n, n), bool), -1)
    A[mask] = np.nan
    return np.asfortranarray(A)


@pytest.mark.parametrize("n", [448, 513])
def test_every_solve_by_blocks(hc, port, n):
    rng = np.random.default_rng(n)
    tasks, keep = [], []
    for side in (LEFT, RIGHT):
        for uplo in (UPPER, LOWER):
            for tr in (NOTRANS, TRANS):
                for dg in (NONUNIT, UNIT):
                    M, N = (n, 21) if side == LEFT else (45, n)
                    A = _triangle(rng, n, uplo, dg == UNIT)
                    B = np.asfortranarray(rng.standard_normal((M, N)))
                    ref, _ = port.dtrsm(side, uplo, tr, dg, M, N, -0.75, A, B)
                    dA, dB = _dev(A, n + 2), _dev(B, M + 5)
                    keep.append((dA, dB, M, ref))
                    tasks.append(hc.TrsmTask(side=side, uplo=uplo, trans=tr, diag=dg, M=M, N=N, alpha=-0.75,
                                             A=dA.data_ptr(), lda=n + 2, B=dB.data_ptr(), ldb=M + 5))
    hc.trsm_batched(tasks)
    for _, dB, M, ref in keep:
        out = dB.cpu().numpy()
        _close(out[:, :M].T, ref, 1e-12)
        assert np.isnan(out[:, M:]).all()   # the padding is not touched


def test_factorizations_with_products(hc, port):
    rng = np.random.default_rng(5)
    keep, tasks = [], []
    for up, n, fail in (("L", 700, None), ("U", 700, None), ("L", 645, 450), ("U", 640, None), ("L", 65, None)):
        X = rng.standard_normal((n, n))
        S = X @ X.T / n + np.eye(n)
        if fail:
            S[fail - 1, fail - 1] = -1.0
        other = np.tril(np.ones((n, n), bool), -1) if up == "U" else np.triu(np.ones((n, n), bool), 1)
        S = np.asfortranarray(np.where(other, np.nan, S))
        ref, info, _ = port.dpotrf(ord(up), n, S)
        d = _dev(S, n + 3)
        keep.append((d, n, up, ref, info))
        tasks.append(hc.PotrfTask(uplo=ord(up), n=n, A=d.data_ptr(), lda=n + 3))
    infos = hc.potrf_batched(tasks)
    for (d, n, up, ref, info), got in zip(keep, infos):
        assert got == info
        out = d.cpu().numpy()[:, :n].T
        j = n if info == 0 else info - 1
        tri = np.tril if up == "L" else np.triu
        _close(tri(np.nan_to_num(out[:j, :j])), tri(np.nan_to_num(ref[:j, :j])), 1e-12)
        if info:
            assert abs(out[j, j] - ref[j, j]) <= 1e-12 * abs(ref[j, j])
        assert np.array_equal(np.isnan(out), np.isnan(ref)) or info
