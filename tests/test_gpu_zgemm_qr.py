"""The complex QR on clusters of CTAs: every cluster size, rows that are no multiple
of a CTA's share, rank sums equal to the order and at the shared-memory limit, a zero
column, real data (reflectors with a zero tau at the last row).  Against the dense
truncation, with the bounds of the other complex updates (product 1e-11, orthonormal
factor 1e-12); the copies of one update in a batch have the same bits."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _factor(rng, M, k, real):
    X = rng.standard_normal((M, k)) + (0 if real else 1j) * rng.standard_normal((M, k))
    Q, _ = np.linalg.qr(X)
    return np.asfortranarray((Q * 10.0 ** (-8.0 * np.arange(k) / k)).astype(np.complex128))


@pytest.mark.parametrize("M,a,c,copies,kind", [(1024, 41, 42, 1, ""), (513, 20, 30, 3, ""), (31, 8, 23, 2, "real"),
                                               (97, 1, 1, 5, "zero"), (200, 16, 30, 90, ""), (160, 30, 40, 170, "")])
def test_complex_qr(hc, M, a, c, copies, kind):
    import torch

    rng = np.random.default_rng(M + copies)
    AU, AV, BU, BV, CU, CV = (_factor(rng, M, r, kind == "real") for r in (a, a, a, a, c, c))
    if kind == "zero":
        AU[:, 0] = 0
    rr, P, S = O.zgemm_dense_truncation(-1.0, AU, AV, BU, BV, 1.0, CU, CV, acc=1e-6)
    assert np.all(np.abs(S - 1e-6) > 1e-9)
    dev = {n: torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for n, x in
           (("AU", AU), ("AV", AV), ("BU", BU), ("BV", BV))}
    k = a + c
    cu, cv = (torch.zeros((copies, k, M), dtype=torch.complex128, device="cuda") for _ in range(2))
    cu[:, :c], cv[:, :c] = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (CU, CV))
    tasks = [hc.ZlrTask(M=M, a=a, b=a, c=c, rk=0, maxrk=k, alpha=hc.DComplex(-1.0, 0.0), beta=hc.DComplex(1.0, 0.0),
                        acc=1e-6, AU=dev["AU"].data_ptr(), AV=dev["AV"].data_ptr(), lda=M, BU=dev["BU"].data_ptr(),
                        BV=dev["BV"].data_ptr(), ldb=M, CU=cu[q].data_ptr(), CV=cv[q].data_ptr(), ldc=M)
             for q in range(copies)]
    ranks, status = hc.zgemm_batched(tasks)
    assert not status.any() and set(ranks) == {rr}
    assert torch.equal(cu, cu[:1].expand_as(cu)) and torch.equal(cv, cv[:1].expand_as(cv))
    U, V = cu[0, :rr].cpu().numpy().T, cv[0, :rr].cpu().numpy().T
    assert np.linalg.norm(U @ V.T - P) <= 1e-11 * np.linalg.norm(P)
    assert np.abs(U.conj().T @ U - np.eye(rr)).max() <= 1e-12
