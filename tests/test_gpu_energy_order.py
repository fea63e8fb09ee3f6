"""With the energy equation set up, the FP64 flow passes keep the order of sums of
precision 1: the momentum half of an outer iteration equals precision 1's bit
for bit, and the pressure half agrees with the flow alone to rounding."""
import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

RTOL = 1e-11     # rounding (1e-15 a sum), amplified below 1e3 by the stopped solves, with a decade left

STATE = ("u", "v", "w", "p", "u0", "v0", "w0", "gu", "gv", "gw", "gp", "mip", "mip0")


@pytest.mark.parametrize("kind,n", [("hex", 2), ("hex", 13), ("hex", 33), ("tet", 9), ("prism", 12), ("pyramid", 7), ("mixed", 9)])
def test_order(need_gpu, kind, n):
    s = cfdl.Setup(cfdl.Zone(n, kind=kind, jitter=0.15, seed=n))
    g = {p: cfdl.Solver(s, cfdl.steady(mu=0.01, precision=p % 2)) for p in (0, 1, 2)}   # 2: precision 0 without the energy equation
    g[0].energy_init()
    g[0].step(3, 0)
    for p in (1, 2):
        for f in STATE:
            g[p].set(f, g[0].get(f))
    for x in g.values():
        x.update_boundaries()
        x.solve_uvwp()
    for f in ("u", "v", "w", "p"):
        a, b = g[0].get(f), g[2].get(f)
        assert np.linalg.norm(a - b) <= RTOL * np.linalg.norm(b), f
    for p in (0, 1):
        g[p].update_boundaries()
    for f in STATE:
        g[1].set(f, g[0].get(f))
    for p in (0, 1):
        g[p].calc_coef_uvw()
        g[p].solve_momentum()
        g[p].calc_grad("uvw")
        g[p].calc_mip(True)
    for f in ("bu", "bv", "bw", "d", "u", "v", "w", "gu", "gv", "gw", "mip"):
        assert np.array_equal(g[0].get(f), g[1].get(f)), f
