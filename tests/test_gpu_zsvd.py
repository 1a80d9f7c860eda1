"""The complex SVD over its launch shapes: a cluster of eight to two CTAs per update,
one CTA with 16 or eight lanes a column pair; odd and even k up to the shared-memory
limit, a core whose tail lies far below acc, one of equal
singular values, a zero update, a fixed rank.  Against the dense truncation (product
1e-11, orthonormal factor 1e-12, as in the other complex tests; the singular values to
1e-12 of the largest); the copies of one update in a batch have the same bits."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _factor(rng, M, k, decades=8.0):
    Q, _ = np.linalg.qr(rng.standard_normal((M, k)) + 1j * rng.standard_normal((M, k)))
    return np.asfortranarray(Q * 10.0 ** (-decades * np.arange(k) / k))


@pytest.mark.parametrize("n,a,c,kind", [(1, 41, 42, ""), (1, 8, 8, ""), (1, 8, 9, ""), (2, 16, 17, "tail"), (19, 32, 31, ""),
                                        (50, 30, 34, "equal"), (60, 30, 34, "rk"), (76, 24, 25, ""), (90, 25, 24, ""),
                                        (153, 30, 34, ""), (153, 9, 8, ""), (3, 20, 20, "zero")])
def test_complex_svd(hc, n, a, c, kind):
    import torch

    M, acc, k = 96, 1e-6, a + c
    rng = np.random.default_rng(31 * n + a)
    AU, AV, BU, BV = (_factor(rng, M, a, 60.0 if kind == "tail" else 8.0) for _ in range(4))
    CU, CV = _factor(rng, M, c), _factor(rng, M, c)
    if kind == "equal":
        CU, CV = (np.asfortranarray(np.linalg.qr(x)[0]) for x in (CU, CV))
        AU *= 1e-13
    if kind == "zero":
        AU *= 0
        CU[:, 1:] *= 0
    exact = CU @ CV.T - (AU @ (AV.T @ BV)) @ BU.T
    S = np.linalg.svd(exact, compute_uv=False)[:k]
    rr = k if kind == "rk" else max(1, int((S >= acc).sum()))
    assert np.all(np.abs(S - acc) > 1e-9)
    dev = {m: torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for m, x in
           (("AU", AU), ("AV", AV), ("BU", BU), ("BV", BV))}
    cu, cv = (torch.zeros((n, k, M), dtype=torch.complex128, device="cuda") for _ in range(2))
    cu[:, :c], cv[:, :c] = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (CU, CV))
    tasks = [hc.ZlrTask(M=M, a=a, b=a, c=c, rk=k if kind == "rk" else 0, maxrk=k, alpha=hc.DComplex(-1.0, 0.0),
                        beta=hc.DComplex(1.0, 0.0), acc=acc, AU=dev["AU"].data_ptr(), AV=dev["AV"].data_ptr(), lda=M,
                        BU=dev["BU"].data_ptr(), BV=dev["BV"].data_ptr(), ldb=M, CU=cu[q].data_ptr(),
                        CV=cv[q].data_ptr(), ldc=M) for q in range(n)]
    ranks, status = hc.zgemm_batched(tasks)
    assert not status.any() and set(ranks) == {rr}
    assert torch.equal(cu, cu[:1].expand_as(cu)) and torch.equal(cv, cv[:1].expand_as(cv))
    U, V = cu[0, :rr].cpu().numpy().T, cv[0, :rr].cpu().numpy().T
    _, P, _ = O.zgemm_dense_truncation(-1.0, AU, AV, BU, BV, 1.0, CU, CV, acc=acc) if kind != "rk" else (0, exact, 0)
    assert np.linalg.norm(U @ V.T - P) <= 1e-11 * np.linalg.norm(P)
    assert np.abs(U.conj().T @ U - np.eye(rr)).max() <= 1e-12
    assert np.abs(np.linalg.norm(V, axis=0) - S[:rr]).max() <= 1e-12 * S[0]
