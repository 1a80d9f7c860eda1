"""The shared-memory SVD with a cluster of CTAs per update: the cluster's size
depends on how many updates share the GPU, the result does not.  Every size from
eight CTAs (one update) to four, and one, odd and even k, a deflated core (the tail far below
acc), a core of equal singular values; the bits of one CTA per update."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _run(hc, d, out, n, a, b, c, M, acc, rk, lanes):
    t = [hc.LrTask(M=M, a=a, b=b, c=c, rk=rk, maxrk=a + c, ld_newv=0, storage_maxrank=0, alpha=-1.0, beta=1.0,
                   acc=acc, AU=d[0].data_ptr(), AV=d[1].data_ptr(), lda=M, BU=d[2].data_ptr(), BV=d[3].data_ptr(),
                   ldb=M, Bdense=None, CU=d[4].data_ptr(), CV=d[5].data_ptr(), ldc=M, CUo=out[0][q].data_ptr(),
                   CVo=out[1][q].data_ptr(), ldco=M) for q in range(n)]
    batch = hc.Batch(t, tuning=hc.make_tuning(svd_lanes=lanes) if lanes else None)
    batch.execute()
    r, st = batch.results()
    sig = batch.sigma(n - 1)
    batch.close()
    return r, st, sig


@pytest.mark.parametrize("n,a,c,kind", [(1, 60, 59, ""), (1, 24, 25, ""), (2, 32, 32, "tail"), (21, 40, 40, ""),
                                        (30, 24, 27, "equal"), (38, 32, 31, "rk"), (39, 32, 31, "")])
def test_same_bits_as_one_cta(hc, n, a, c, kind):
    import torch
    from hcore_gb300 import devmem

    M, acc = 160, 1e-8
    b = a if kind == "" else 9
    rng = np.random.default_rng(17 * n + a)
    arr = [list(O.graded_lowrank(rng, M, r, 60.0 if kind == "tail" else 8.0)) for r in (a, b, c)]
    if kind == "equal":
        arr[2][0], _ = np.linalg.qr(arr[2][0])
        arr[0][0] *= 1e-13
    d = [devmem.to_device(np.asfortranarray(x)) for pair in arr for x in pair]
    res = []
    for lanes in (None, [8, 8, 8]):
        out = [torch.zeros((n, a + c, M), dtype=torch.float64, device="cuda") for _ in range(2)]
        res.append((_run(hc, d, out, n, a, b, c, M, acc, a + c if kind == "rk" else 0, lanes), out))
    (r, st, sig), out = res[0]
    (r1, st1, sig1), out1 = res[1]
    assert not st.any() and not st1.any() and np.array_equal(r, r1) and np.array_equal(sig, sig1)
    assert len(set(r)) == 1
    for x, y in zip(out, out1):
        assert torch.equal(x, y) and torch.equal(x, x[:1].expand_as(x))
    (AU, AV), (BU, BV), (CU, CV) = arr
    exact = CU @ CV.T - (AU @ (AV.T @ BV)) @ BU.T
    U, V = out[0][0, :r[0]].cpu().numpy().T, out[1][0, :r[0]].cpu().numpy().T
    assert np.linalg.norm(U @ V.T - exact) <= acc * np.sqrt(a + c) + 1e-11 * np.linalg.norm(exact)
