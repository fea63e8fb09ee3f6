"""The allocation-free pressure solve on few SMs: one block, one row per thread
with more than 512 threads a block, eight rows per thread with a remainder in
the rows, the threads and the blocks, and the largest eight rows reach; against
the context's solve, and the statuses that the kernel finds for itself."""
import ctypes as C

import numpy as np
import pytest

import cfdl
from test_gpu_noalloc_sizes import _ref
from test_zz_no_alloc import INVALID, NONFINITE, OK, RTOL_PC, TOO_LARGE, _assembled_case, _Device

CELLS = 131072          # CFDL_NOALLOC_MAX_CELLS


class _Few(_Device):
    def few(self, sms, rtol=1e-13, maxit=20000):
        x = self.torch.full((self.ne,), float("nan"), dtype=self.torch.float64, device=self.dev)
        self.torch.cuda.synchronize()
        iters, rnorm = C.c_int(-1), C.c_double(-1.0)
        status = cfdl.lib().cfdl_solve_pc_noalloc_sms(
            self.ne, self.nh, self.ef1.data_ptr(), self.idx.data_ptr(), self.ap.data_ptr(), self.anb.data_ptr(),
            self.b.data_ptr(), x.data_ptr(), rtol, maxit, sms, C.byref(iters), C.byref(rnorm))
        return status, x.cpu().numpy(), iters.value, rnorm.value


# 17^3 = 4913 rows: 1 and 3 SMs take eight rows per thread (615 threads), 5 one;
# 43^3 = 79507: eight rows reach with 10 SMs and not with 9
@pytest.mark.gpu
@pytest.mark.parametrize("n,sms", [(2, 1), (9, 1), (17, 1), (17, 3), (17, 5), (43, 10), (43, 60), (43, 1000)])
def test_few_sms(need_gpu, n, sms):
    torch = pytest.importorskip("torch")
    z, s, g = _assembled_case(n)
    d = _Few(torch, s, g.get("ap"), g.get("anb"), g.get("b"))
    ref = _ref(g)
    status, x, iters, rnorm = d.few(sms)
    assert status == OK, cfdl.STATUS.get(status, status)
    again = d.few(sms)
    assert again[2] == iters and np.array_equal(again[1], x)
    x = x - x[0]
    assert np.linalg.norm(x - ref) < RTOL_PC * np.linalg.norm(ref)


@pytest.mark.gpu
def test_rows_of_the_eight(need_gpu):
    """Wide rows (18 half-faces) and what the kernel reports, with eight rows per thread."""
    torch = pytest.importorskip("torch")
    z, s, g = _assembled_case(17)
    ap, anb, b = g.get("ap"), g.get("anb"), g.get("b")
    ref = _ref(g)
    ef1, idx = s.get_int("ef2nb1"), s.get_int("ef2nb_idx")
    d = _Few(torch, s, ap, np.repeat(anb / 3.0, 3), b, ef1=np.repeat(ef1, 3), idx=(1 + 3 * (idx - 1)).astype(np.int32))
    d.nh = 3 * s.H
    status, x, iters, rnorm = d.few(2)
    assert status == OK, cfdl.STATUS.get(status, status)
    x = x - x[0]
    assert np.linalg.norm(x - ref) < RTOL_PC * np.linalg.norm(ref)
    bad = ef1.copy()
    bad[np.flatnonzero(bad & 31)[-1]] = ((s.ne + 1) << 5) | 1
    assert _Few(torch, s, ap, anb, b, ef1=bad).few(2)[0] == INVALID
    ap0 = ap.copy()
    ap0[4900] = 0.0
    assert _Few(torch, s, ap0, anb, b).few(2)[0] == NONFINITE


@pytest.mark.gpu
def test_too_few_sms(need_gpu):
    torch = pytest.importorskip("torch")
    z, s, g = _assembled_case(43)
    d = _Few(torch, s, g.get("ap"), g.get("anb"), g.get("b"))
    assert d.few(9)[0] == TOO_LARGE


def test_sms_are_checked_before_the_device():
    buf, ibuf = (C.c_double * 8)(), (C.c_int * 8)()
    p, ip = C.cast(buf, C.c_void_p), C.cast(ibuf, C.c_void_p)
    L = cfdl.lib()
    for sms in (0, -1):
        assert L.cfdl_solve_pc_noalloc_sms(4, 8, ip, ip, p, p, p, p, 1e-8, 10, sms, None, None) == INVALID
    assert L.cfdl_solve_pc_noalloc_sms(CELLS + 1, 8, ip, ip, p, p, p, p, 1e-8, 10, 4, None, None) == TOO_LARGE
