"""The allocation-free pressure solve at the sizes where its launch changes
shape -- one block, a few blocks, one block per SM with at most and with more
than 512 rows -- against the context's solve of the same system, and with rows
of more couplings than a thread keeps in registers."""
import numpy as np
import pytest

import cfdl
from test_zz_no_alloc import OK, RTOL_PC, _assembled_case, _Device

pytestmark = pytest.mark.gpu


def _ref(g):
    assert g.solve_pc().status == 0
    x = g.get("phic")[:g.ne]
    return x - x[0]


@pytest.mark.parametrize("n", [2, 5, 6, 17, 43, 50])
def test_sizes(need_gpu, n):
    torch = pytest.importorskip("torch")
    z, s, g = _assembled_case(n)
    d = _Device(torch, s, g.get("ap"), g.get("anb"), g.get("b"))
    ref = _ref(g)
    status, x, iters, rnorm = d.solve()
    assert status == OK, cfdl.STATUS.get(status, status)
    x = x - x[0]
    assert np.linalg.norm(x - ref) < RTOL_PC * np.linalg.norm(ref)
    again = d.solve()
    assert again[2] == iters and np.array_equal(again[1] - again[1][0], x)   # the same call, the same answer


def test_wide_rows(need_gpu):
    """Each coupling given as three thirds: rows of up to 18 half-faces."""
    torch = pytest.importorskip("torch")
    z, s, g = _assembled_case(9)
    ap, anb, b = g.get("ap"), g.get("anb"), g.get("b")
    ref = _ref(g)
    ef1, idx = np.repeat(s.get_int("ef2nb1"), 3), 1 + 3 * (s.get_int("ef2nb_idx") - 1)
    d = _Device(torch, s, ap, np.repeat(anb / 3.0, 3), b, ef1=ef1, idx=idx.astype(np.int32))
    d.nh = 3 * s.H
    status, x, iters, rnorm = d.solve()
    assert status == OK, cfdl.STATUS.get(status, status)
    x = x - x[0]
    assert np.linalg.norm(x - ref) < RTOL_PC * np.linalg.norm(ref)
