"""Small contexts share a solver tile among four blocks, one row per thread, with the
sums of the whole tile: a case has the same bits alone (split) and in a batch
whose cells are too many for it, in every precision, at row counts below, at and
above a tile and a quarter of one."""
import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

KINDS = [("hex", 2), ("hex", 6), ("hex", 10), ("hex", 11), ("hex", 16), ("hex", 23), ("tet", 9), ("prism", 11), ("pyramid", 7), ("mixed", 6)]
LARGE = 55      # cells of one more case (166375): with it whole tiles are used


@pytest.mark.parametrize("precision", [0, 1, 2, 3])
def test_alone_and_in_a_large_batch(need_gpu, precision):
    setups = [cfdl.Setup(cfdl.Zone(n, kind=k, jitter=0.1, seed=n)) for k, n in KINDS]
    cfg = cfdl.steady(mu=0.01, precision=precision)
    bt = cfdl.Batch(setups + [cfdl.Setup(cfdl.Zone(LARGE, seed=1))], [cfg] * (len(setups) + 1))
    bt.step(3, 0)
    for i, s, (k, n) in zip(bt.ids(), setups, KINDS):
        g = cfdl.Solver(s, cfg)
        g.step(3, 0)
        for f in ("u", "v", "w", "p", "mip"):
            assert np.array_equal(bt.case_get(i, f), g.get(f)), (k, n, f)


@pytest.mark.parametrize("precision", [0, 1])
def test_tight_solves(need_gpu, precision):
    """Solves to a tolerance, and the Jacobi preconditioner, against a tile shape that is not split."""
    s = cfdl.Setup(cfdl.Zone(13, kind="hex", jitter=0.1, seed=3))
    for precond in (0, 1):
        cfg = cfdl.steady(mu=0.01, precision=precision, precond=precond, solve_mode=1, tight_rtol=1e-12)
        a, b = cfdl.Solver(s, cfg), cfdl.Solver(s, cfg)
        b.set_tile(2)
        for g in (a, b):
            assert g.step(2, 0).status == 0
        for f in ("u", "p"):
            # both solved to 1e-12 of the right-hand side; two decades for the condition of the systems
            assert np.linalg.norm(a.get(f) - b.get(f)) <= 1e-9 * np.linalg.norm(b.get(f)), (precond, f)
