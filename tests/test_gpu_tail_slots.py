"""The V-cycle's tail with less shared memory than its levels' slots take: the
last slots are read from global memory, in the same order, so the pressure
solve takes the same iterations to the same solution."""
import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

KB = 1024
TIGHT = 1e-12
# both solutions are within TIGHT times the condition number (below 1e3), with a
# decade left; the sums' order is the same, so in practice they are equal
RTOL = 1e-8


def _solved(g):
    g.update_boundaries()
    g.calc_coef_uvw()
    g.solve_momentum()
    g.calc_grad("uvw")
    g.calc_mip(True)
    g.calc_coef_p()
    st = g.solve_pc()
    assert st.status == 0
    x = g.get("phic")[:g.ne]
    return x - x[0], st.it_p


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind,n", [("hex", 24), ("tet", 14), ("mixed", 13), ("prism", 20)])
def test_slots_left_out(need_gpu, kind, n, precision):
    s = cfdl.Setup(cfdl.Zone(n, kind=kind, jitter=0.1, seed=6))
    cfg = cfdl.steady(solve_mode=1, tight_rtol=TIGHT, precision=precision)
    L = cfdl.lib()
    a, b = cfdl.Solver(s, cfg), cfdl.Solver(s, cfg)
    a.step(1, 0)
    start = {f: a.get(f) for f in ("u", "v", "w", "p", "u0", "v0", "w0", "gu", "gv", "gw", "gp", "mip", "mip0")}
    want, it = _solved(a)
    tried = 0
    for kb in range(200, 4, -8):                 # down to what the plan needs without any slot
        if L.cfdl_set_tail_smem(b._h, kb * KB):
            break
        for f, v in start.items():
            b.set(f, v)
        got, it_b = _solved(b)
        assert np.linalg.norm(got - want) <= RTOL * np.linalg.norm(want), kb
        assert abs(it_b - it) <= 1, kb
        tried += 1
    assert 1 < tried < 25                        # some limits held slots back, the last was refused
    assert L.cfdl_set_tail_smem(b._h, 0) == 0
