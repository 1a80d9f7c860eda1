"""The diagonal block of the batched Cholesky factorization (sub-blocks of 16 columns,
the rest of a sub-block's update beside the next factorization) and its panel: orders
around the sub-blocks' and blocks' edges, both triangles, pivots that fail in the first,
a middle and the last column of a sub-block (info, the leading part, the pivot left in
place), tiny and huge scales.  Against the oracle, 1e-12 of the largest entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("up", ["L", "U"])
def test_orders_and_failing_pivots(hc, port, up):
    import torch

    rng = np.random.default_rng(11)
    cases = [(n, None, 1.0) for n in (1, 2, 15, 16, 17, 31, 33, 48, 49, 63, 64, 65, 79, 80, 96, 127, 128, 129, 200)]
    cases += [(n, f, 1.0) for n, f in ((1, 1), (16, 16), (17, 17), (40, 1), (40, 24), (64, 33), (64, 64), (70, 48),
                                       (100, 65), (130, 90), (130, 129))]
    cases += [(50, None, 1e-290), (90, None, 1e290)]
    keep, tasks = [], []
    for n, fail, scale in cases:
        X = rng.standard_normal((n, n))
        S = (X @ X.T / n + np.eye(n)) * scale
        if fail:
            S[fail - 1, fail - 1] = -1.0
        other = np.tril(np.ones((n, n), bool), -1) if up == "U" else np.triu(np.ones((n, n), bool), 1)
        S = np.asfortranarray(np.where(other, np.nan, S))
        ref, info, _ = port.dpotrf(ord(up), n, S)
        d = torch.full((n, n + 3), float("nan"), dtype=torch.float64, device="cuda")
        d[:, :n] = torch.from_numpy(np.ascontiguousarray(S.T)).cuda()
        keep.append((d, n, fail, ref, info))
        tasks.append(hc.PotrfTask(uplo=ord(up), n=n, A=d.data_ptr(), lda=n + 3))
    infos = hc.potrf_batched(tasks)
    for (d, n, fail, ref, info), got in zip(keep, infos):
        assert got == info == (fail or 0)
        out = d.cpu().numpy()[:, :n].T
        j = n if not fail else fail - 1
        tri = np.tril if up == "L" else np.triu
        x, y = (tri(np.nan_to_num(v[:j, :j])) for v in (out, ref))
        assert j == 0 or np.abs(x - y).max() <= 1e-12 * np.abs(y).max()
        if fail:
            assert abs(out[j, j] - ref[j, j]) <= 1e-12 * max(abs(ref[j, j]), 1.0)
        assert np.isnan(d.cpu().numpy()[:, n:]).all()
        other = np.tril_indices(n, -1) if up == "U" else np.triu_indices(n, 1)
        assert np.isnan(out[other]).all()
