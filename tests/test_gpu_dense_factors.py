"""The factors of syrk and gemmcd tasks formed as products on the tensor cores (lists
of more than 40 million multiply-adds): a above, equal to and below b, ranks 1, 17, 64,
130 (two chunks), orders that are no multiple of a tile, padded leading dimensions of
the syrk's inputs, tasks of rank 0 between them, several tasks on one tile; against the
same sums in numpy, and a short list (factors in FP64) of the same tasks.  1e-12 of the
largest entry, the dense tiles' gate; the triangle that syrk zeroes is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(x, ld=None):
    import torch

    d = torch.full((x.shape[1], ld or x.shape[0]), 3.0, dtype=torch.float64, device="cuda")
    d[:, :x.shape[0]] = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    return d


@pytest.mark.parametrize("M,copies", [(777, 5), (513, 9), (128, 60)])
def test_factors_as_products(hc, M, copies):
    import torch

    rng = np.random.default_rng(M)
    ranks = [(1, 17), (17, 1), (64, 64), (40, 33), (33, 40), (100, 110), (0, 5), (5, 0)]
    gem = []
    for a, b in ranks:
        f = [rng.standard_normal((M, max(r, 1))) * 10.0 ** rng.uniform(-4, 0, max(r, 1)) for r in (a, a, b, b)]
        gem.append((a, b, f, [_dev(x) for x in f]))
    syr = []
    for a in (1, 17, 64, 110):
        f = [rng.standard_normal((M, a)) for _ in range(2)]
        syr.append((a, f, [_dev(x, M + 2) for x in f]))
    C0 = rng.standard_normal((M, M))
    want_g = C0.copy()
    for a, b, (Au, Av, Bu, Bv), _ in gem:
        if a and b:
            want_g -= (Au @ (Av.T @ Bv)) @ Bu.T
    want_s = C0.copy()
    for a, (U, V), _ in syr:
        # (the reference sums the inner product over the leading dimension's rows)
        pad = np.full((2, a), 3.0)
        W = np.vstack([V, pad])
        want_s += -0.5 * (U @ (W.T @ W)) @ U.T
    want_s = np.tril(want_s)

    def run(n):
        tasks, outs = [], []
        for _ in range(n):
            g, s = _dev(C0), _dev(C0)
            outs.append((g, s))
            for a, b, _, d in gem:
                tasks.append(hc.DenseTask(kind=1, M=M, a=a, b=b, Au=d[0].data_ptr(), Av=d[1].data_ptr(),
                                          Bu=d[2].data_ptr(), Bv=d[3].data_ptr(), CD=g.data_ptr(), ldcd=M))
            for a, _, d in syr:
                tasks.append(hc.DenseTask(kind=0, M=M, a=a, alpha=-0.5, Au=d[0].data_ptr(), Av=d[1].data_ptr(),
                                          lda=M + 2, CD=s.data_ptr(), ldcd=M))
        hc.dense_batched(tasks)
        torch.cuda.synchronize()
        return [(g.cpu().numpy().T, s.cpu().numpy().T) for g, s in outs]

    many = run(copies)
    for g, s in many:
        assert np.array_equal(g, many[0][0]) and np.array_equal(s, many[0][1])
    for got, want in zip(many[0], (want_g, want_s)):
        assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
    assert (np.triu(many[0][1], 1) == 0).all()
