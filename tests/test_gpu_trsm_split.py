"""Triangular solves with one to eight vectors a CTA, with both chunk heights, and by
blocks where the vectors are many: all 16 cases, orders around the blocks' and
chunks' edges, padded leading dimensions, NaN in every entry that must not be read.
Against the oracle, 1e-12 of the largest entry, as the other solves' tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NOTRANS, TRANS, UPPER, LOWER, NONUNIT, UNIT, LEFT, RIGHT = 111, 112, 121, 122, 131, 132, 141, 142


def _dev(x, ld):
    import torch

    d = torch.full((x.shape[1], ld), float("nan"), dtype=torch.float64, device="cuda")
    d[:, :x.shape[0]] = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    return d


@pytest.mark.parametrize("n,vec", [(31, 1), (33, 3), (128, 9), (161, 13), (300, 20), (97, 40), (450, 9), (448, 77),
                                   (513, 78), (1030, 31)])
def test_every_case(hc, port, n, vec):
    rng = np.random.default_rng(n)
    tasks, keep = [], []
    for side in (LEFT, RIGHT):
        for uplo in (UPPER, LOWER):
            for tr in (NOTRANS, TRANS):
                for dg in (NONUNIT, UNIT):
                    M, N = (n, vec) if side == LEFT else (vec, n)
                    A = rng.standard_normal((n, n)) / n
                    A[np.arange(n), np.arange(n)] = np.nan if dg == UNIT else 1.0 + rng.random(n)
                    unread = np.triu_indices(n, 1) if uplo == LOWER else np.tril_indices(n, -1)
                    A[unread] = np.nan
                    A = np.asfortranarray(A)
                    B = np.asfortranarray(rng.standard_normal((M, N)))
                    ref, _ = port.dtrsm(side, uplo, tr, dg, M, N, 1.25, A, B)
                    dA, dB = _dev(A, n + 2), _dev(B, M + 5)
                    keep.append((dA, dB, M, ref))
                    tasks.append(hc.TrsmTask(side=side, uplo=uplo, trans=tr, diag=dg, M=M, N=N, alpha=1.25,
                                             A=dA.data_ptr(), lda=n + 2, B=dB.data_ptr(), ldb=M + 5))
    hc.trsm_batched(tasks)
    for _, dB, M, ref in keep:
        out = dB.cpu().numpy()
        assert np.abs(out[:, :M].T - ref).max() <= 1e-12 * np.abs(ref).max()
        assert np.isnan(out[:, M:]).all()
