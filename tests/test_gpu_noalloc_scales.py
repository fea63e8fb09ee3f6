"""The allocation-free pressure solve at the ends of the number range: the steps
of CG do not depend on powers of two in the matrix and the right-hand side, so a
system scaled by them has the same iterations and the scaled solution."""
import numpy as np
import pytest

import cfdl
from test_zz_no_alloc import OK, _assembled_case, _Device

pytestmark = pytest.mark.gpu


def _system():
    """Couplings of 1..8 and a zero-sum right-hand side of small integers on a mesh's
    graph: exact at any scale, subnormal numbers included."""
    z, s, g = _assembled_case(9)
    idx = s.get_int("ef2nb_idx") - 1
    ef1 = s.get_int("ef2nb1").view(np.uint32)
    row = np.repeat(np.arange(s.ne), np.diff(idx))
    nb, inside = (ef1 >> 5).astype(np.int64) - 1, (ef1 & 31) != 0
    anb = np.where(inside, 1.0 + (row + nb) % 8, 0.0)
    ap = np.bincount(row, weights=anb, minlength=s.ne)
    b = np.random.default_rng(2).integers(-8, 9, s.ne).astype(np.float64)
    b[0] -= b.sum()
    return s, ap, anb, b


@pytest.mark.parametrize("matrix,rhs", [(-1060, -400), (900, 400), (0, -300), (-1000, 0)])
def test_scaled_system(need_gpu, matrix, rhs):
    torch = pytest.importorskip("torch")
    s, ap, anb, b = _system()
    status, x, iters, rnorm = _Device(torch, s, ap, anb, b).solve(rtol=1e-12)
    assert status == OK
    st2, x2, it2, rn2 = _Device(torch, s, np.ldexp(ap, matrix), np.ldexp(anb, matrix), np.ldexp(b, rhs)).solve(rtol=1e-12)
    assert st2 == OK, cfdl.STATUS.get(st2, st2)
    assert it2 == iters and rn2 == np.ldexp(rnorm, rhs)
    assert np.array_equal(x2, np.ldexp(x, rhs - matrix))

