"""A plan's captured execute (stream groups, on as many streams) against its
direct one (one group): the same bits, whatever the groups, also when outputs
overlap other updates' inputs."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _setup(hc, n, in_place_of_next):
    import torch
    from hcore_gb300 import devmem

    rng = np.random.default_rng(41)
    M, keep, tasks = 200, [], []
    for _ in range(n):
        a, b, c = (int(x) for x in rng.integers(1, 30, size=3))
        keep.append(([devmem.to_device(x, 64) for r in (a, b, c) for x in O.graded_lowrank(rng, M, r)], (a, b, c)))
    out = [[torch.zeros((64, M), dtype=torch.float64, device="cuda") for _ in range(2)] for _ in range(n)]
    for q, (d, (a, b, c)) in enumerate(keep):
        # outputs over the next update's A factors, or into buffers of their own
        o = keep[(q + 1) % n][0][:2] if in_place_of_next else out[q]
        tasks.append(hc.LrTask(M=M, a=a, b=b, c=c, rk=0, maxrk=a + c, ld_newv=0, storage_maxrank=0, alpha=-1.0, beta=1.0,
                               acc=1e-8, AU=d[0].data_ptr(), AV=d[1].data_ptr(), lda=M, BU=d[2].data_ptr(),
                               BV=d[3].data_ptr(), ldb=M, Bdense=None, CU=d[4].data_ptr(), CV=d[5].data_ptr(), ldc=M,
                               CUo=o[0].data_ptr(), CVo=o[1].data_ptr(), ldco=M))
    outs = [keep[(q + 1) % n][0][:2] if in_place_of_next else out[q] for q in range(n)]
    return keep, tasks, outs


def _execute(hc, in_place, captured, **tuning):
    import torch

    keep, tasks, outs = _setup(hc, 20, in_place)
    b = hc.Batch(tasks, tuning=tuning or None)
    if captured:
        g, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            with torch.cuda.graph(g, stream=side):
                b.execute(side.cuda_stream)
        g.replay()
        torch.cuda.synchronize()
    else:
        b.execute()
    r, st = b.results()
    b.close()
    assert (st == 0).all()
    return [int(x) for x in r], [(u[:q].cpu().numpy(), v[:q].cpu().numpy()) for (u, v), q in zip(outs, r)]


@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("tuning", [{"stream_groups": 1}, {"stream_groups": 3}, {"stream_groups": 16},
                                    {"stream_groups": 5, "phase_sync": 1}])
def test_captured_equals_direct(hc, in_place, tuning):
    r0, o0 = _execute(hc, in_place, False)
    r1, o1 = _execute(hc, in_place, True, **tuning, qr_warps=4)
    assert r0 == r1
    for (u0, v0), (u1, v1) in zip(o0, o1):
        assert np.array_equal(u0, u1) and np.array_equal(v0, v1)
