"""Quotients taken by Newton steps from an FP32 reciprocal (div_rn) against the
division: the temperature is a stored quotient of stored operands, so it is
compared with numpy's division, bit for bit, over ranges inside and outside the
fast one."""
import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-20, 1e20, 1e-29, 1e-31, 1e31, 1e-200, 1e200])
def test_temperature_quotient(need_gpu, scale):
    """calc_temperature is t = phi / cp: cp inside the fast range, at its ends
    (2^-100, 2^101) and far outside; phi with zeros, signs and extremes."""
    s = cfdl.Setup(cfdl.Zone(7, jitter=0.1, seed=3))
    g = cfdl.Solver(s, cfdl.steady(nit=0))           # no inner iteration: phi stays what it is
    g.energy_init()
    r = np.random.default_rng(int(abs(np.log10(scale))) + 1)
    cp = scale * np.exp(r.uniform(-3, 3, s.ne))
    e = g.get("e")
    e[:s.ne] = r.standard_normal(s.ne) * np.exp2(r.integers(-60, 60, s.ne))
    e[:4] = (0.0, 1.0, -1.0, 5e-324)
    g.set("cp", cp)
    g.set("e", e)
    try:
        g.solve_energy()
    except cfdl.CfdlError as err:        # tc/cp beyond the range: reported, and t is still phi / cp
        assert err.status == cfdl.CFDL_ERR_NONFINITE
    with np.errstate(all="ignore"):
        want = g.get("e")[:s.ne] / cp
    assert np.array_equal(g.get("t")[:s.ne], want)
