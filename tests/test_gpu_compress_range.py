"""The compressor's range finder (find_ranges, hc_compress.cu) where its rules
change: orders around the smallest that it takes (128), a range wider than its
cap and squares outside FP64's range (both go to the pivoted QR), leading
dimensions above the order; against the full SVD's ranks and products, with the
margin and tolerance of the compressor's other tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tile(rng, M, shift):
    X = rng.uniform(0, 0.25, (M, 2))
    Y = rng.uniform(0, 0.25, (M, 2)) + np.array([shift, 0.1])
    d2 = ((X[:, None, :] - Y[None, :, :]) ** 2).sum(-1)
    return np.asfortranarray(np.exp(-d2 / 0.01))


def _run(hc, tiles, acc, relative, pad=0):
    import torch

    keep, tasks = [], []
    for D in tiles:
        M = D.shape[0]
        d = torch.full((M, M + pad), float("nan"), dtype=torch.float64, device="cuda")
        d[:, :M] = torch.from_numpy(np.ascontiguousarray(D.T)).cuda()
        u, v = (torch.full((M, M), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
        keep.append((d, u, v))
        tasks.append(hc.CompressTask(M=M, D=d.data_ptr(), ldd=M + pad, acc=acc, relative=int(relative), maxrank=M,
                                     U=u.data_ptr(), V=v.data_ptr(), ldo=M))
    ranks, status = hc.compress_batched(tasks)
    prods = [(u[:r].T @ v[:r]).cpu().numpy() for (_, u, v), r in zip(keep, ranks)]
    return ranks, status, prods


@pytest.mark.parametrize("M", [127, 128, 129, 160, 257])
@pytest.mark.parametrize("relative", [True, False])
def test_ranks_and_products(hc, port, M, relative):
    rng = np.random.default_rng(M)
    acc = 1e-8 if relative else 1e-6
    tiles = [_tile(rng, M, 0.2), _tile(rng, M, 0.35), np.asfortranarray(1e-3 * _tile(rng, M, 0.25))]
    ranks, status, prods = _run(hc, tiles, acc, relative, pad=3)
    assert (status == 0).all()
    for D, r, P in zip(tiles, ranks, prods):
        rr, U, V, sig = port.dcompress(D, acc, M, relative=relative)
        thr = acc * sig[0] if relative else acc
        assert np.all(np.abs(sig - thr) > 2e-3 * thr)
        assert r == rr
        # the compressor's contract: rounding, and the margin of 1e-3 of the threshold
        assert np.abs(P - U @ V.T).max() <= (1e-10 * sig[0] if relative else 1e-12 * np.abs(D).max() + 1e-3 * acc)


def test_tiles_left_to_the_pivoted_qr(hc):
    rng = np.random.default_rng(9)
    M = 200
    Q, _ = np.linalg.qr(rng.standard_normal((M, M)))
    full = np.asfortranarray(Q @ np.diag(np.linspace(1.0, 2.0, M)) @ Q.T)   # range wider than the cap
    nan = _tile(rng, M, 0.2)
    nan[5, 7] = np.nan
    zero = np.zeros((M, M), order="F")
    far = _tile(rng, M, 0.2)
    ranks, status, prods = _run(hc, [full, nan, zero, far], 1e-9, True)
    assert list(status) == [0, 6, 0, 0]
    assert ranks[0] == M and ranks[2] == 0 and 0 < ranks[3] < M
    assert np.abs(prods[0] - full).max() < 1e-12
    # the squares' sum is below 1e-280; the truncation drops singular values below 1e-9 sigma_max
    ranks2, status2, prods2 = _run(hc, [np.asfortranarray(far * 2.0 ** -480)], 1e-9, True)
    assert status2[0] == 0 and ranks2[0] > 0
    assert np.linalg.norm(prods2[0] * 2.0 ** 480 - far) <= 1e-8 * np.linalg.norm(far)
