"""Meshes in which two cells share two faces (a face given as two halves, as
cut-cell and polyhedral meshes have them): rows with two slots for one
neighbour.  The multigrid solve of such a mesh against the Jacobi one."""
import ctypes as C

import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

TIGHT = 1e-13
# TIGHT times the condition of the systems (below 1e3), through a few outer
# iterations, with a decade left: as the coarsest level's own test
RTOL = 1e-9


class SplitSetup:
    """The set-up's mesh with every `step`-th interior face split in two halves;
    a cell takes one extra face at most."""

    def __init__(self, s, step):
        i32 = lambda name: s.get_int(name)
        ef1, ef2, idx = i32("ef2nb1"), i32("ef2nb2"), i32("ef2nb_idx") - 1
        cells = [[(int(ef1[h]), int(ef2[h])) for h in range(idx[e], idx[e + 1])] for e in range(s.ne)]
        aip, rip = s.get_dbl("aip").reshape(-1, 3).copy(), s.get_dbl("rip").reshape(-1, 3)
        s2g, grown, new = list(i32("s2g")), set(), []
        for e in range(s.ne):
            for c, f in list(cells[e]):
                nb = (c >> 5) - 1
                if f < 0 or nb >= s.ne or f % step or e in grown or nb in grown:
                    continue
                grown |= {e, nb}
                g = s.nf + len(new) + 1                      # the second half's face, 1-based
                new.append(f - 1)
                here, there = len(cells[e]) + 1, len(cells[nb]) + 1
                cells[e].append((((nb + 1) << 5) | there, g))
                cells[nb].append((((e + 1) << 5) | here, -g))
                s2g.append(((e + 1) << 5) | here)
        aip[new] *= 0.5
        self.split = len(new)
        self.ne, self.nf, self.nbf, self.H = s.ne, s.nf + len(new), s.nbf, s.H + 2 * len(new)
        flat = [h for c in cells for h in c]
        self.a = dict(ef2nb1=np.array([h[0] for h in flat], np.int32), ef2nb2=np.array([h[1] for h in flat], np.int32),
                      ef2nb_idx=(1 + np.concatenate([[0], np.cumsum([len(c) for c in cells])])).astype(np.int32),
                      s2g=np.array(s2g, np.int32), aip=np.concatenate([aip, aip[new]]).ravel(),
                      rip=np.concatenate([rip, rip[new]]).ravel())
        self.base = s

    def mesh(self, u_lid=1.0):
        m = self.base.mesh(u_lid)
        m.nf = self.nf
        for k, v in self.a.items():
            setattr(m, k, v.ctypes.data_as(C.c_void_p))
        return m


@pytest.mark.parametrize("n,step", [(2, 1), (2, 3), (4, 1)])
def test_split_faces(need_gpu, n, step):
    """48 tets (the mesh is the coarsest multigrid level) and 384 (it is not)."""
    s = cfdl.Setup(cfdl.Zone(n, kind="tet", jitter=0.1, seed=5))
    t = SplitSetup(s, step)
    assert t.split >= 3 and cfdl.lib().cfdl_mesh_check(C.byref(t.mesh())) == 0
    a, b, c = (cfdl.Solver(t, cfdl.steady(solve_mode=1, tight_rtol=TIGHT, precond=p)) for p in (0, 1, 1))
    for g in (a, b, c):
        st = g.step(4, 0)
        assert st.status == 0
    for f in ("u", "v", "w", "p"):
        x, y = a.get(f), b.get(f)
        assert np.linalg.norm(x - y) <= RTOL * np.linalg.norm(x), f
        assert np.array_equal(y, c.get(f)), f
    if t.ne <= 64:                           # the exact preconditioner's iterations (test_gpu_coarsest.py)
        assert st.it_p <= 4
