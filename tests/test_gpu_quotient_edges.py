"""div_rn at the divisors its correction can miss: significands of all ones and
next to it, on both sides of the line where the division takes over, and
numerators next to a power of two.  t = phi / cp as in test_gpu_quotients.py,
against numpy's division, bit for bit."""
import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -52


def _significands():
    line = 2.0 - 2.0 ** -20                                     # the first significand whose upper 20 bits are ones
    near_two = [2.0 - k * ULP for k in list(range(1, 40)) + [2 ** j + d for j in range(6, 34) for d in (-1, 0, 1)]]
    near_line = [line + k * ULP for k in (-3, -2, -1, 0, 1, 2, 3)]
    near_one = [1.0 + k * ULP for k in list(range(0, 12)) + [2 ** j - 1 for j in range(4, 30)]]
    return np.array(near_two + near_line + near_one)


@pytest.mark.parametrize("exponent", [0, -100, 100, -7])
def test_edge_divisors(need_gpu, exponent):
    s = cfdl.Setup(cfdl.Zone(9, jitter=0.1, seed=3))
    g = cfdl.Solver(s, cfdl.steady(nit=0))
    g.energy_init()
    a = _significands()
    b = np.concatenate([[1.0, 1.0 + ULP, 2.0 - ULP, 2.0 - 2 * ULP, 1.5], np.random.default_rng(1).uniform(1.0, 2.0, 4)])
    pairs = [(x, y) for y in b for x in a]
    for at in range(0, len(pairs), s.ne):
        some = pairs[at:at + s.ne]
        cp, e = np.ones(s.ne), g.get("e")
        cp[:len(some)] = [np.ldexp(x, exponent) for x, _ in some]
        e[:len(some)] = [y * (-1.0) ** k for k, (_, y) in enumerate(some)]
        g.set("cp", cp)
        g.set("e", e)
        try:
            g.solve_energy()
        except cfdl.CfdlError as err:    # tc/cp beyond the range: reported, and t is still phi / cp
            assert err.status == cfdl.CFDL_ERR_NONFINITE
        want = g.get("e")[:s.ne] / cp
        assert np.array_equal(g.get("t")[:s.ne], want)
