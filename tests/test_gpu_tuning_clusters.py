"""A plan with the default tuning, with one field of it changed, or with an autotuned one
runs few wide updates as fast as a plan without a tuning: their SVDs on a cluster of CTAs
each (one update of a + c = 116: 3.6 ms of SVD so, 6.2 with one CTA), the small ones with
eight lanes a pair.  Medians of replays, with a margin of a quarter."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,a,c", [(1, 58, 58), (16, 9, 9)])
def test_no_slower_with_a_tuning(hc, n, a, c):
    import torch
    from hcore_gb300 import devmem

    M = 400
    rng = np.random.default_rng(a)
    d = [devmem.to_device(x) for r in (a, a, c) for x in O.graded_lowrank(rng, M, r, 8.0)]
    out = [torch.zeros((n, a + c, M), dtype=torch.float64, device="cuda") for _ in range(2)]
    tasks = [hc.LrTask(M=M, a=a, b=a, c=c, rk=0, maxrk=a + c, ld_newv=0, storage_maxrank=0, alpha=-1.0, beta=1.0,
                       acc=1e-8, AU=d[0].data_ptr(), AV=d[1].data_ptr(), lda=M, BU=d[2].data_ptr(),
                       BV=d[3].data_ptr(), ldb=M, Bdense=None, CU=d[4].data_ptr(), CV=d[5].data_ptr(), ldc=M,
                       CUo=out[0][q].data_ptr(), CVo=out[1][q].data_ptr(), ldco=M) for q in range(n)]

    def median(tuning):
        batch = hc.Batch(tasks, tuning=tuning)
        s, ev, t = torch.cuda.Stream(), [torch.cuda.Event(enable_timing=True) for _ in range(2)], []
        for q in range(25):
            ev[0].record(s)
            batch.execute(s.cuda_stream)
            ev[1].record(s)
            s.synchronize()
            t.append(ev[0].elapsed_time(ev[1]))
        batch.close()
        return float(np.median(t[5:]))

    plain = median(None)
    best, _ = hc.autotune(tasks, reps=3)
    for tuning in (hc.make_tuning(), hc.make_tuning(bucket_width=16), best):
        assert median(tuning) <= 1.25 * plain, tuning.as_dict()
