"""d and dc of solve_uvwp's fused assembly against the single routine's, which
divides: correctly rounded quotients of the same operands, so the same bits
in every form."""
import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transient", [False, True])
@pytest.mark.parametrize("precision", [0, 1, 3])
@pytest.mark.parametrize("kind,n", [("hex", 3), ("hex", 21), ("tet", 13), ("prism", 7), ("mixed", 6)])
def test_quotients_of_the_assembly(need_gpu, kind, n, precision, transient):
    s = cfdl.Setup(cfdl.Zone(n, kind=kind, jitter=0.15, seed=n))
    kw = dict(precision=precision)
    cfg = cfdl.default_config(dt=0.02, alpha_u=0.9, **kw) if transient else cfdl.steady(mu=0.004, **kw)
    a, b = cfdl.Solver(s, cfg), cfdl.Solver(s, cfg)
    a.step(3, 2)
    for f in ("u", "v", "w", "p", "u0", "v0", "w0", "gu", "gv", "gw", "gp", "mip", "mip0", "d"):
        b.set(f, a.get(f))
    a.update_boundaries()
    a.solve_uvwp()
    b.update_boundaries()
    b.calc_coef_uvw()
    for f in ("d", "dc"):
        assert np.array_equal(a.get(f), b.get(f)), f
