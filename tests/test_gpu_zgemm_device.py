"""Complex updates whose factors stay in device memory (written in place by the
last kernel) beside the same updates in host memory and with one output factor
on each side: the same bits, nothing outside the new factors touched, a rejected
update's factors left alone.  Sizes at the edges of the stack phase's groups (four
columns of AV, eight of BV, 64 rows)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _factor(rng, M, k):
    Q, _ = np.linalg.qr(rng.standard_normal((M, k)) + 1j * rng.standard_normal((M, k)))
    return np.asfortranarray(Q * 10.0 ** (-8.0 * np.arange(k) / k))


@pytest.mark.parametrize("M,a,b,c", [(64, 4, 8, 5), (65, 1, 9, 3), (200, 13, 40, 24), (33, 5, 1, 28)])
def test_device_and_host_outputs(hc, M, a, b, c):
    import torch

    rng = np.random.default_rng(M + a)
    k, ld = a + c, M + 3
    f = {n: _factor(rng, M, r) for n, r in (("AU", a), ("AV", a), ("BU", min(b, M)), ("BV", min(b, M)),
                                            ("CU", c), ("CV", c))}
    b = min(b, M)
    rr, P, S = O.zgemm_dense_truncation(-0.5 + 1j, f["AU"], f["AV"], f["BU"], f["BV"], 1.0, f["CU"], f["CV"], acc=1e-6)
    assert np.all(np.abs(S - 1e-6) > 1e-9)

    def dev(x, cols):
        d = torch.full((cols, ld), 7.0, dtype=torch.complex128, device="cuda")
        d[:x.shape[1], :M] = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
        return d

    def host(x, cols):
        h = np.full((cols, ld), 7.0, dtype=np.complex128)
        h[:x.shape[1], :M] = x.T
        return h

    at = lambda x: x.data_ptr() if hasattr(x, "data_ptr") else x.ctypes.data  # noqa: E731
    tasks, outs = [], []
    # (the last: its rank sum is above maxrk, refused)
    for place_u, place_v, maxrk in ((dev, dev, k), (host, host, k), (dev, host, k), (host, dev, k), (dev, dev, k - 1)):
        ins = {n: dev(f[n], f[n].shape[1]) for n in ("AU", "AV", "BU", "BV")}
        cu, cv = place_u(f["CU"], k), place_v(f["CV"], k)
        t = hc.ZlrTask(M=M, a=a, b=b, c=c, rk=0, maxrk=maxrk, alpha=hc.DComplex(-0.5, 1.0), beta=hc.DComplex(1.0, 0.0),
                       acc=1e-6, AU=at(ins["AU"]), AV=at(ins["AV"]), lda=ld, BU=at(ins["BU"]), BV=at(ins["BV"]), ldb=ld,
                       CU=at(cu), CV=at(cv), ldc=ld)
        tasks.append(t)
        outs.append((cu, cv, ins))
    ranks, status = hc.zgemm_batched(tasks)
    assert list(status[:4]) == [0] * 4 and status[4] != 0 and list(ranks[:4]) == [rr] * 4
    get = lambda x: x.cpu().numpy() if hasattr(x, "cpu") else x  # noqa: E731
    first = [get(x) for x in outs[0][:2]]
    for cu, cv, _ in outs[:4]:
        for got, want in zip((cu, cv), first):
            assert np.array_equal(get(got), want)
    for x in first:
        assert np.all(x[:, M:] == 7.0)
    for x, n in zip(first, ("CU", "CV")):   # columns past the new rank: as they were
        keep = np.full((k, M), 7.0 + 0j)
        keep[:c] = f[n].T
        assert np.array_equal(x[rr:, :M], keep[rr:])
    for got, n in zip(outs[4][:2], ("CU", "CV")):
        assert np.array_equal(get(got)[:c, :M], f[n].T)
    prod = first[0][:rr, :M].T @ first[1][:rr, :M]
    assert np.linalg.norm(prod - P) <= 1e-11 * np.linalg.norm(P)
