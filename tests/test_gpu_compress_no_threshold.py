"""Compression without a threshold (acc 0, absolute or relative): the rank is that of the
range, found column by column to 64 eps of the norm, on both sides of the order from
which blocks of test vectors find the range: the tile's exact rank, since its singular
values lie in [1, 2].  A negative acc is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [100, 128, 256])
@pytest.mark.parametrize("relative", [0, 1])
def test_rank_of_the_range(hc, M, relative):
    import torch

    rng = np.random.default_rng(M)
    U, V = (np.linalg.qr(rng.standard_normal((M, 10)))[0] for _ in range(2))
    D = (U * np.linspace(2, 1, 10)) @ V.T
    d = torch.from_numpy(np.ascontiguousarray(D.T)).cuda()
    u, v = (torch.zeros((M, M), dtype=torch.float64, device="cuda") for _ in range(2))
    task = lambda acc: hc.CompressTask(M=M, D=d.data_ptr(), ldd=M, acc=acc, relative=relative, maxrank=M,  # noqa: E731
                                       U=u.data_ptr(), V=v.data_ptr(), ldo=M)
    with pytest.raises(hc.HcoreError):
        hc.compress_batched([task(-1e-300)])
    ranks, status = hc.compress_batched([task(0.0)])
    assert status[0] == 0 and ranks[0] == 10
    assert np.abs((u[:10].T @ v[:10]).cpu().numpy() - D).max() <= 1e-12
