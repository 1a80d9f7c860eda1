"""The cluster SVD (hc_svd.cu) at the edges of its range: k = a + c just above
shared memory (119 in FP64, 168 in FP32), around the 256 columns where the lanes
per pair change, and at the largest k; alone (eight CTAs an update) and in a
batch that leaves one CTA each; graded, deflated and fixed-rank updates; a NaN
beside them.  The blocked QR of the same updates takes several column groups a
panel.  Against the oracle, with the plan's usual gates."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _tasks(hc, arrays, acc, rk=0):
    import torch
    from hcore_gb300 import devmem

    keep, tasks = [], []
    for (AU, AV), (BU, BV), (CU, CV) in arrays:
        M, a, b, c = AU.shape[0], AU.shape[1], BU.shape[1], CU.shape[1]
        d = [devmem.to_device(x) for x in (AU, AV, BU, BV, CU, CV)]
        out = [torch.zeros((a + c, M), dtype=d[0].dtype, device="cuda") for _ in range(2)]
        keep.append((d, out))
        tasks.append(hc.LrTask(M=M, a=a, b=b, c=c, rk=rk, maxrk=a + c, ld_newv=0, storage_maxrank=0, alpha=-1.0,
                               beta=1.0, acc=acc, AU=d[0].data_ptr(), AV=d[1].data_ptr(), lda=M, BU=d[2].data_ptr(),
                               BV=d[3].data_ptr(), ldb=M, Bdense=None, CU=d[4].data_ptr(), CV=d[5].data_ptr(), ldc=M,
                               CUo=out[0].data_ptr(), CVo=out[1].data_ptr(), ldco=M))
    return keep, tasks


def _run(hc, arrays, acc, rk=0, precision=0):
    from hcore_gb300 import devmem

    keep, tasks = _tasks(hc, arrays, acc, rk)
    b = hc.Batch(tasks, precision=precision)
    b.execute()
    r, st = b.results()
    b.close()
    return r, st, [devmem.to_host(o[0], int(q)) @ devmem.to_host(o[1], int(q)).T for (_, o), q in zip(keep, r)]


def _arrays(rng, M, a, c, decades):
    return tuple(O.graded_lowrank(rng, M, r, decades) for r in (a, max(1, a // 2), c))


def _check(port, arr, r, P, acc, rk=0):
    (AU, AV), (BU, BV), (CU, CV) = arr
    a, b, c = AU.shape[1], BU.shape[1], CU.shape[1]
    ref = port.gemm(AU.shape[0], -1.0, AU, AV, a, BU, BV, b, 1.0, CU, CV, c, rk=rk, maxrk=a + c, acc=acc)
    assert r == ref["rank"]
    assert O.rel_fro(P, ref["CU"] @ ref["CV"].T) < 1e-11


@pytest.mark.parametrize("a,c,decades", [(60, 60, 8.0), (60, 61, 30.0), (127, 128, 8.0), (128, 128, 12.0),
                                         (129, 128, 8.0), (256, 256, 8.0)])
def test_alone(hc, port, a, c, decades):
    rng = np.random.default_rng(a + c)
    arr = _arrays(rng, 600, a, c, decades)
    r, st, P = _run(hc, [arr], 1e-8)
    assert st[0] == 0
    _check(port, arr, int(r[0]), P[0], 1e-8)


def test_batch_of_many_and_a_nan(hc, port):
    rng = np.random.default_rng(11)
    arrays = [_arrays(rng, 260, 60 + q % 5, 61 + q % 7, 10.0) for q in range(12)] * 14   # one CTA each
    bad = _arrays(rng, 260, 70, 70, 8.0)
    bad[0][1][3, 4] = np.nan
    r, st, P = _run(hc, arrays + [bad], 1e-8)
    assert (st[:-1] == 0).all() and st[-1] == 6
    for q in (0, 5, 11, len(arrays) - 1):
        _check(port, arrays[q], int(r[q]), P[q], 1e-8)


def test_fixed_rank(hc, port):
    rng = np.random.default_rng(12)
    arr = _arrays(rng, 300, 75, 70, 20.0)
    r, st, P = _run(hc, [arr], 1e-8, rk=40)
    assert st[0] == 0 and r[0] == 40
    _check(port, arr, 40, P[0], 1e-8, rk=40)


def test_fp32(hc):
    rng = np.random.default_rng(13)
    arr = tuple(tuple(x.astype(np.float32) for x in p) for p in _arrays(rng, 400, 85, 84, 3.0))
    r, st, P = _run(hc, [arr], 1e-6, precision=hc.F32)
    assert st[0] == 0
    (AU, AV), (BU, BV), (CU, CV) = (tuple(x.astype(np.float64) for x in p) for p in arr)
    exact = CU @ CV.T - AU @ (AV.T @ BV) @ BU.T
    assert np.linalg.norm(P[0] - exact) < 1e-6 * 13 + 5e-5 * np.linalg.norm(exact)
