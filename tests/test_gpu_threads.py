"""Calls from several threads at once, each thread with sizes of its own, so that a
kernel is launched with more shared memory by one thread than by another: every
call succeeds and returns what it returns alone.  (The GIL is released in a call.)"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _together(jobs, calls):
    """run every job `calls` times, each in a thread of its own; their results"""
    res, err, gate = [[] for _ in jobs], [], threading.Barrier(len(jobs))

    def work(q):
        import torch

        try:
            stream = torch.cuda.Stream().cuda_stream
            gate.wait()
            for _ in range(calls):
                res[q].append(jobs[q](stream))
        except Exception as e:   # reported by the test's own thread
            err.append(e)
            gate.abort()

    th = [threading.Thread(target=work, args=(q,)) for q in range(len(jobs))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not err, err
    return res


def test_triangular_solves(hc):
    import torch

    rng = np.random.default_rng(1)

    def job(n, vec):
        a = torch.from_numpy(np.triu(rng.standard_normal((n, n)) / n) + np.eye(n)).cuda()   # (column-major: lower)
        b = torch.from_numpy(rng.standard_normal((vec, n))).cuda()
        x = torch.empty_like(b)
        t = [hc.TrsmTask(side=141, uplo=121, trans=111, diag=131, M=n, N=vec, alpha=1.0, A=a.data_ptr(), lda=n,
                         B=x.data_ptr(), ldb=n)]

        def run(stream):
            with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
                x.copy_(b)
            hc.trsm_batched(t, stream)
            return x.cpu().numpy(), a

        return run

    jobs = [job(1000, 8), job(40, 8), job(700, 4), job(100, 300)]
    alone = [j(0) for j in jobs]
    for got, want in zip(_together(jobs, 150), alone):
        assert all(np.array_equal(x[0], want[0]) for x in got)


def test_compression(hc):
    import torch

    rng = np.random.default_rng(2)

    def job(M):
        p = rng.random((M, 2))
        D = np.exp(-((p[:, None] - p[None] - [0.7, 0.1]) ** 2).sum(-1) / 0.05)
        d, u, v = (torch.from_numpy(D).cuda(), torch.zeros(M, M, dtype=torch.float64, device="cuda"),
                   torch.zeros(M, M, dtype=torch.float64, device="cuda"))
        t = [hc.CompressTask(M=M, D=d.data_ptr(), ldd=M, acc=1e-8, relative=1, maxrank=M, U=u.data_ptr(),
                             V=v.data_ptr(), ldo=M)]

        def run(stream):
            r, st = hc.compress_batched(t, stream)
            return int(r[0]), int(st[0]), u[:r[0]].cpu().numpy(), d

        return run

    jobs = [job(M) for M in (128, 700, 300, 1000)]
    alone = [j(0) for j in jobs]
    for got, want in zip(_together(jobs, 40), alone):
        assert all(x[:2] == want[:2] and x[1] == 0 and np.array_equal(x[2], want[2]) for x in got)


def test_complex_updates(hc):
    import torch

    rng = np.random.default_rng(3)

    def job(M, r):
        f = [torch.from_numpy(rng.standard_normal((r, M)) + 1j * rng.standard_normal((r, M))).cuda() for _ in range(4)]
        c0 = [torch.from_numpy(rng.standard_normal((2 * r, M)) + 0j).cuda() for _ in range(2)]
        c = [torch.empty_like(x) for x in c0]
        t = [hc.ZlrTask(M=M, a=r, b=r, c=r, rk=0, maxrk=2 * r, alpha=hc.DComplex(-1.0, 0.0), beta=hc.DComplex(1.0, 0.0),
                        acc=1e-8, AU=f[0].data_ptr(), AV=f[1].data_ptr(), lda=M, BU=f[2].data_ptr(),
                        BV=f[3].data_ptr(), ldb=M, CU=c[0].data_ptr(), CV=c[1].data_ptr(), ldc=M)]

        def run(stream):
            with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
                for x, y in zip(c, c0):
                    x.copy_(y)
            rk, st = hc.zgemm_batched(t, stream)
            return int(rk[0]), int(st[0]), c[0].cpu().numpy(), f

        return run

    jobs = [job(M, r) for M, r in ((64, 4), (512, 32), (300, 40), (100, 12))]
    alone = [j(0) for j in jobs]
    for got, want in zip(_together(jobs, 60), alone):
        assert all(x[:2] == want[:2] and x[1] == 0 and np.array_equal(x[2], want[2]) for x in got)
