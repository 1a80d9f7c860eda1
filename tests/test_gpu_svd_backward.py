"""Backward error of the core SVD's QR on graded cores, whose columns below the pivot are
small beside it: there a reflector changes a row's sign and little else, which is
one rounding if its parameters are formed as tau = 2 and v = (1, small), and four
if v is left unscaled.

The factors are chosen so that everything before the SVD is exact: CU the first
columns of the identity, CV upper triangular, A B^T = 0, so that T is CV^T in its
top block.  A float32 restatement of the kernel's steps (same order, same sums)
gives errors ||U S V^T - T|| / ||T|| of 1.0 (k = 12) and 1.5 (24) units roundoff on
average with the scaled parameters and 4.0 and 3.6 with the others; the limit, 2.6 on
the root mean square over the updates, lies between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [12, 24])
def test_graded_fp32_core(hc, c):
    import torch

    n, M, dt, limit = 64, 192, np.float32, 2.6
    rng = np.random.default_rng(c)
    grade = 10.0 ** (-4.0 * np.arange(c) / c)
    z = torch.zeros((1, M), dtype=torch.float32, device="cuda")
    cu = np.zeros((c, M), dt)
    cu[np.arange(c), np.arange(c)] = 1
    cvs = []
    for _ in range(n):
        r = grade[:, None] * (np.eye(c) + 1e-3 * np.triu(rng.standard_normal((c, c)), 1))
        cv = np.zeros((c, M), dt)
        cv[:, :c] = r.T   # (row j of the array is column j of CV)
        cvs.append(cv)
    dcu, dcv = torch.from_numpy(cu).cuda(), torch.from_numpy(np.stack(cvs)).cuda()
    cuo, cvo = (torch.zeros((n, c + 1, M), dtype=z.dtype, device="cuda") for _ in range(2))
    tasks = [hc.LrTask(M=M, a=1, b=1, c=c, rk=c, maxrk=c + 1, ld_newv=0, storage_maxrank=0, alpha=-1.0, beta=1.0,
                       acc=1e-30, AU=z.data_ptr(), AV=z.data_ptr(), lda=M, BU=z.data_ptr(), BV=z.data_ptr(), ldb=M,
                       Bdense=None, CU=dcu.data_ptr(), CV=dcv[q].data_ptr(), ldc=M, CUo=cuo[q].data_ptr(),
                       CVo=cvo[q].data_ptr(), ldco=M) for q in range(n)]
    batch = hc.Batch(tasks, precision=hc.F32)
    batch.execute()
    ranks, status = batch.results()
    batch.close()
    assert not status.any() and (ranks == c).all()
    err = []
    for q in range(n):
        u, v = (x[q, :c, :c].cpu().numpy().astype(np.float64) for x in (cuo, cvo))
        t = cvs[q][:, :c].astype(np.float64)   # its transpose is T, and CU the identity
        d = u.T @ v - t
        err.append(float(np.sqrt((d ** 2).sum() / (t ** 2).sum())) / (np.finfo(dt).eps / 2))
    assert np.sqrt(np.mean(np.square(err))) <= limit
