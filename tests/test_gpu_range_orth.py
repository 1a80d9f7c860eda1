"""The range finder's orthonormalization on clusters of one to eight CTAs per tile
(the number of tiles and their order decide), mixed orders in one call: the ranks of
the tiles' full SVDs, products within the compressor's contract, orthonormal U."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tile(rng, M, rank):
    U, _ = np.linalg.qr(rng.standard_normal((M, rank)))
    V, _ = np.linalg.qr(rng.standard_normal((M, rank)))
    s = 10.0 ** (-14.0 * np.arange(rank) / rank)
    return (U * s) @ V.T, s


@pytest.mark.parametrize("orders,n", [((1025,), 1), ((130, 400), 2), ((300,), 20), ((129, 1024), 60), ((256,), 160)])
def test_ranks_products_and_factors(hc, orders, n):
    import torch

    rng = np.random.default_rng(n)
    acc, rank = 1e-8, 45   # no singular value within 5% of the threshold
    base = {M: _tile(rng, M, rank) for M in orders}
    tasks, keep = [], []
    for t in range(n):
        M = orders[t % len(orders)]
        d = torch.from_numpy(np.ascontiguousarray(base[M][0].T)).cuda()
        u, v = (torch.full((64, M), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
        keep.append((M, d, u, v))
        tasks.append(hc.CompressTask(M=M, D=d.data_ptr(), ldd=M, acc=acc, relative=1, maxrank=64, U=u.data_ptr(),
                                     V=v.data_ptr(), ldo=M))
    ranks, status = hc.compress_batched(tasks)
    assert (status == 0).all()
    for (M, d, u, v), r in zip(keep, ranks):
        D, s = base[M]
        assert np.abs(s / s[0] - acc).min() > 0.05 * acc
        assert r == (s >= acc * s[0]).sum()
        P = (u[:r].T @ v[:r]).cpu().numpy()
        # the dropped values, and the contract's margin of 1e-3 of the threshold
        assert np.linalg.norm(P - D) <= np.linalg.norm(s[r:]) + 1e-3 * acc * s[0]
        G = (u[:r] @ u[:r].T).cpu().numpy()
        assert np.abs(G - np.eye(r)).max() <= 1e-12
