"""solve_uvwp assembles the momentum equations and starts their solve in one pass
(and keeps calc_coef_p's flux factors for update_uvwp); the single routines do
not.  One outer iteration both ways from the same state: bit for bit in the
mixed forms, whose FP32 roundings would turn any difference into 1e-7; to
rounding in FP64, where the fused pass orders its sums another way."""
import math

import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

# FP64: each array is a few sums of a dozen terms (1e-15 each) and inner solves
# stopped at a fixed residual drop, whose two or three iterations amplify a
# difference of their input by less than the 1e3 of their condition number
RTOL = 1e-12


def _outer(g):
    g.update_boundaries()
    g.calc_coef_uvw()
    got = {f: g.get(f) for f in ("bu", "bv", "bw", "d", "dc")}
    g.solve_momentum()
    g.calc_grad("uvw")
    g.calc_mip(True)
    g.calc_coef_p()
    g.solve_pc()
    g.adjust_pc()
    g.calc_grad("phic")
    g.update_uvwp()
    return got


@pytest.mark.parametrize("transient", [False, True])
@pytest.mark.parametrize("precision", [0, 1, 2, 3])
@pytest.mark.parametrize("kind,n", [("hex", 3), ("hex", 9), ("hex", 21), ("tet", 4), ("tet", 13), ("prism", 7), ("pyramid", 6), ("mixed", 6)])
def test_fused_equals_routines(need_gpu, kind, n, precision, transient):
    s = cfdl.Setup(cfdl.Zone(n, kind=kind, jitter=0.15, seed=n))
    kw = dict(precision=precision, precond=1)
    cfg = cfdl.default_config(dt=0.02, alpha_u=0.9, **kw) if transient else cfdl.steady(mu=0.004, **kw)
    a, b = cfdl.Solver(s, cfg), cfdl.Solver(s, cfg)
    a.step(3, 2)
    for f in ("u", "v", "w", "p", "u0", "v0", "w0", "gu", "gv", "gw", "gp", "mip", "mip0", "d"):
        b.set(f, a.get(f))
    a.update_boundaries()
    a.solve_uvwp()
    got = _outer(b)
    got.update({f: b.get(f) for f in ("u", "v", "w", "p", "gp", "mip", "phic", "b")})
    for f, y in got.items():
        x = a.get(f)
        if precision == 0:
            assert np.linalg.norm(x - y) <= RTOL * np.linalg.norm(y), f
        else:
            assert np.array_equal(x, y), (f, float(np.linalg.norm(x - y)))


def test_unrelaxed_steady_form(need_gpu):
    """alpha_u = 1 and no time step: the SIMPLEC denominator of an inner cell is
    zero, so dc is infinite there, in the single routine and in solve_uvwp."""
    s = cfdl.Setup(cfdl.Zone(6, kind="hex", jitter=0.0, seed=1))
    g = cfdl.Solver(s, cfdl.steady(alpha_u=1.0, precision=0))
    assert math.isinf(g.config.dt)
    g.update_boundaries()
    g.calc_coef_uvw()
    want, d = g.get("dc"), g.get("d")
    try:
        g.solve_uvwp()
    except cfdl.CfdlError as e:
        assert e.status == cfdl.CFDL_ERR_NONFINITE
    assert np.array_equal(np.isinf(g.get("dc")), np.isinf(want)) and np.isinf(want).any()
    assert np.array_equal(g.get("d"), d) and np.all(np.isfinite(d))
