"""The mixed pressure solve's FP32 mesh-level kernels take rows in pairs: odd and
even cell counts, a last tile of one row, of one pair and a full one, four-,
five- and six-slot rows, with 16-bit offsets and with int32 indices, against
the FP64 solve of the same system."""
import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

# both solves stop at ||r|| <= 1e-11 ||b||; the systems (diagonal within a
# factor of ten, at most 30 cells across) have condition numbers below 2e3, so
# the solutions agree within 2 * 2e3 * 1e-11 and less in the 2-norm
RTOL = 4e-8


def _system(kind, n, precision):
    s = cfdl.Setup(cfdl.Zone(n, kind=kind, jitter=0.1, seed=n))
    g = cfdl.Solver(s, cfdl.steady(solve_mode=1, tight_rtol=1e-11, precision=precision))
    return s, g


@pytest.mark.parametrize("kind,n", [("hex", 5), ("hex", 6), ("hex", 7), ("hex", 8), ("hex", 9), ("hex", 13), ("tet", 3), ("tet", 5),
                                    ("prism", 5), ("prism", 8), ("pyramid", 4), ("mixed", 4), ("mixed", 5)])
def test_mixed_solve_matches_fp64(need_gpu, kind, n):
    s, ref = _system(kind, n, 0)
    ref.step(2, 0)
    ref.update_boundaries()
    ref.calc_coef_uvw()
    ref.solve_momentum()
    ref.calc_grad("uvw")
    ref.calc_mip(True)
    ref.calc_coef_p()
    assert ref.solve_pc().status == 0
    want = ref.get("phic")[:s.ne]
    want = want - want.mean()
    _, g = _system(kind, n, 1)
    got = []
    for on in (True, False):
        g.set_index16(on)
        for f in ("u", "v", "w", "p", "gu", "gv", "gw", "gp", "d", "dc", "mip"):
            g.set(f, ref.get(f))
        g.calc_coef_p()
        st = g.solve_pc()
        assert st.status == 0 and st.it_p > 0
        x = g.get("phic")[:s.ne]
        x = x - x.mean()
        assert np.linalg.norm(x - want) < RTOL * np.linalg.norm(want)
        got.append(x)
    assert np.array_equal(got[0], got[1])
