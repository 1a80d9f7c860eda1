"""The shared-memory SVD (hc_svd.cu) at the edges of its range: k = a + c at
the boundaries of a warp, of eight rows and of shared memory (119 in FP64, 168
in FP32), against the oracle.  The lanes per column pair change no bit of the
result: the kernel adds in one fixed order."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _run(hc, rng_seed, a, b, c, acc, precision, lanes):
    import torch
    from hcore_gb300 import devmem

    M, dt = 200, np.float64 if precision == hc.F64 else np.float32
    rng = np.random.default_rng(rng_seed)
    arr = [tuple(x.astype(dt) for x in O.graded_lowrank(rng, M, r, 8.0 if dt == np.float64 else 3.0))
           for r in (a, b, c)]
    d = [devmem.to_device(x) for pair in arr for x in pair]
    out = [torch.zeros((a + c, M), dtype=d[0].dtype, device="cuda") for _ in range(2)]
    t = hc.LrTask(M=M, a=a, b=b, c=c, rk=0, maxrk=a + c, ld_newv=0, storage_maxrank=0, alpha=-1.0, beta=1.0, acc=acc,
                  AU=d[0].data_ptr(), AV=d[1].data_ptr(), lda=M, BU=d[2].data_ptr(), BV=d[3].data_ptr(), ldb=M,
                  Bdense=None, CU=d[4].data_ptr(), CV=d[5].data_ptr(), ldc=M, CUo=out[0].data_ptr(),
                  CVo=out[1].data_ptr(), ldco=M)
    batch = hc.Batch([t], precision=precision,
                     tuning=None if lanes is None else hc.make_tuning(svd_lanes=[lanes] * 3))
    batch.execute()
    r, st = batch.results()
    batch.close()
    assert st[0] == 0
    return arr, int(r[0]), [devmem.to_host(x, int(r[0])) for x in out]


@pytest.mark.parametrize("a,c", [(1, 1), (1, 2), (4, 4), (4, 5), (15, 16), (16, 16), (16, 17), (31, 32), (32, 33),
                                 (48, 49), (59, 59), (59, 60)])
def test_fp64_edges_and_lanes(hc, port, a, c):
    M, b = 200, max(1, a - 1)
    arr, r0, out0 = _run(hc, 100 + a + c, a, b, c, 1e-8, hc.F64, None)
    (AU, AV), (BU, BV), (CU, CV) = arr
    ref = port.gemm(M, -1.0, AU, AV, a, BU, BV, b, 1.0, CU, CV, c, maxrk=a + c, acc=1e-8)
    assert r0 == ref["rank"]
    assert O.rel_fro(out0[0] @ out0[1].T, ref["CU"] @ ref["CV"].T) < 1e-11
    for lanes in (1, 2, 4, 8):
        _, r, out = _run(hc, 100 + a + c, a, b, c, 1e-8, hc.F64, lanes)
        assert r == r0 and np.array_equal(out[0], out0[0]) and np.array_equal(out[1], out0[1]), lanes


@pytest.mark.parametrize("a,c", [(1, 1), (16, 17), (64, 65), (84, 84)])
def test_fp32_edges(hc, a, c):
    arr, r, out = _run(hc, 300 + a + c, a, a, c, 1e-6, hc.F32, None)
    (AU, AV), (BU, BV), (CU, CV) = (tuple(x.astype(np.float64) for x in p) for p in arr)
    exact = CU @ CV.T - AU @ (AV.T @ BV) @ BU.T
    # truncation: fewer than a + c values below acc; FP32 rounding: the FP32 gate of the other tests
    tol = 1e-6 * np.sqrt(a + c) + 5e-5 * np.linalg.norm(exact)
    assert np.linalg.norm(out[0].astype(np.float64) @ out[1].astype(np.float64).T - exact) < tol
