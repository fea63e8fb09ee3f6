"""The dense inverse of the coarsest multigrid level at its edges: a mesh that is
itself the coarsest level (8, 27, 64 rows, the last the largest there is), where
the preconditioner is exact, and meshes with one coarse level or more."""
import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

TIGHT = 1e-13
# TIGHT times the condition number of these systems (below 1e3), with a decade left
RTOL = 1e-9
# an exact preconditioner ends CG in one iteration but for rounding, which a
# second and a third take from the system's 1e-13 of condition times epsilon
EXACT_ITERS = 4


def _assembled(g):
    g.update_boundaries()
    g.calc_coef_uvw()
    g.solve_momentum()
    g.calc_grad("uvw")
    g.calc_mip(True)
    g.calc_coef_p()


@pytest.mark.parametrize("kind,n", [("hex", 2), ("hex", 3), ("hex", 4), ("hex", 5), ("hex", 9), ("hex", 20), ("tet", 2), ("tet", 6)])
def test_coarsest_inverse(need_gpu, kind, n):
    s = cfdl.Setup(cfdl.Zone(n, kind=kind, jitter=0.2, seed=4))
    a, b = (cfdl.Solver(s, cfdl.steady(solve_mode=1, tight_rtol=TIGHT, precond=p)) for p in (0, 1))
    a.step(3)
    for f in ("u", "v", "w", "p", "u0", "v0", "w0", "gu", "gv", "gw", "gp", "mip", "mip0", "d"):
        b.set(f, a.get(f))
    x, it = [], []
    for g in (a, b):
        _assembled(g)
        st = g.solve_pc()
        assert st.status == 0
        x.append(g.get("phic")[:g.ne] - g.get("phic")[0])
        it.append(st.it_p)
    assert np.linalg.norm(x[1] - x[0]) <= RTOL * np.linalg.norm(x[0])
    assert it[1] <= (EXACT_ITERS if s.ne <= 64 else it[0]), it
