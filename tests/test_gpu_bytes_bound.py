"""cfdl_case_bytes_estimate bounds what a case holds on the device after its first
solve, down to meshes of one cell, where what does not grow with the mesh (the
coarsest inverse, the V-cycle tail's plans) is most of it."""
import pytest

import cfdl

pytestmark = pytest.mark.gpu

SLOTS = {"hex": 6, "tet": 4, "prism": 5, "pyramid": 5, "mixed": 6}


@pytest.mark.parametrize("precision", [0, 1, 3])
@pytest.mark.parametrize("kind,n", [(k, n) for k in ("hex", "tet") for n in (1, 2, 3, 4, 5, 9, 16)] +
                         [(k, n) for k in ("prism", "pyramid", "mixed") for n in (2, 6)])
def test_bound(need_gpu, kind, n, precision):
    s = cfdl.Setup(cfdl.Zone(n, kind=kind))
    b = cfdl.Batch([s, s], [cfdl.steady(precision=precision)] * 2)
    b.step(1, 0)
    for c in b.ids():
        assert b.case_info(c)[1] <= cfdl.case_bytes_estimate(s.ne, s.nf, s.nbf, SLOTS[kind])
