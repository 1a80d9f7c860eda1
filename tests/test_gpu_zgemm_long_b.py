"""A complex update whose B has more columns than a grid's y axis takes blocks of eight
for (8 * 65535): order 1, so that F = AV^T BV is one row of that many products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b", [8 * 65535, 8 * 65535 + 1, 8 * 65535 + 9])
def test_more_columns_than_blocks(hc, b):
    import torch

    rng = np.random.default_rng(b)
    z = lambda n: rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))  # noqa: E731
    M = 2   # (a + c = 2)
    AU, AV, CU, CV = z(1), z(1), z(1), z(1)
    BU, BV = z(b) / np.sqrt(b), z(b)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (AU, AV, BU, BV)]
    c = [torch.from_numpy(np.vstack([x, np.zeros_like(x)])).cuda() for x in (CU, CV)]
    ranks, status = hc.zgemm_batched([hc.ZlrTask(
        M=M, a=1, b=b, c=1, rk=2, maxrk=2, alpha=hc.DComplex(-1.0, 0.0), beta=hc.DComplex(1.0, 0.0), acc=1e-8,
        AU=d[0].data_ptr(), AV=d[1].data_ptr(), lda=M, BU=d[2].data_ptr(), BV=d[3].data_ptr(), ldb=M,
        CU=c[0].data_ptr(), CV=c[1].data_ptr(), ldc=M)])
    assert status[0] == 0 and ranks[0] == 2
    F = BV @ AV[0]                     # (b,) = sum over rows of AV(l) BV(l, q)
    want = CU.T @ CV - np.outer(AU[0], F @ BU)
    got = (c[0].T @ c[1]).cpu().numpy()
    # sums of b terms of order 1 / sqrt(b) in any order: sqrt(b) eps and a margin of 100
    assert np.abs(got - want).max() <= 100 * np.sqrt(b) * 2.0 ** -53 * np.abs(want).max()
