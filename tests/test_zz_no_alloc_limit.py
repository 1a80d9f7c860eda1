"""hcore_gpu_dgemm_noalloc right below its workspace limit: a rank sum and an F = AV^T BV
that leave fewer doubles free than the SVD's small arrays take (4 (a + c) + 16), which
do not count; one more column of B is refused."""
import ctypes as C

import pytest

from test_zz_no_alloc import NOALLOC_WS_ELEMS, _bind, _case, _check_against_plan, _ws_need

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,a,c", [(1024, 73, 72), (1000, 72, 70), (1024, 60, 70), (1000, 75, 75)])
def test_full_workspace(hc, M, a, c):
    from hcore_gb300 import devmem

    f = _bind(hc.lib())
    b = max(b for b in range(1, M + 1) if _ws_need(M, a, b, a + c) <= NOALLOC_WS_ELEMS)
    assert NOALLOC_WS_ELEMS - _ws_need(M, a, b, a + c) < 4 * (a + c) + 16 and b < M
    _check_against_plan(f, hc, 46, M, a, b, c, a + c)
    d = [devmem.to_device(x) for x in _case(47, M, a, b + 1, c)]
    r, st = C.c_int(-1), C.c_int(-1)
    rc = f(M, -1.0, d[0].data_ptr(), d[1].data_ptr(), a, M, d[2].data_ptr(), d[3].data_ptr(), b + 1, M, 1.0,
           d[4].data_ptr(), d[5].data_ptr(), c, M, 0, a + c, 1e-8, C.byref(r), C.byref(st), None)
    assert rc == -1 and "scratch" in hc.last_error()
