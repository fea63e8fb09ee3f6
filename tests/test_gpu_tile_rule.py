"""The FP64 solver tiles that go by the case's size: on both sides of each size
where the rows per thread change, against a tile shape given by the caller; and
contexts whose precision is changed or whose energy equation is set up."""
import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

# the tile shape only orders partial sums (1e-15 relative); the inner solves of
# an outer iteration amplify a difference by less than 1e3, and two of them and
# the fields' own cancellations leave a decade
RTOL = 1e-11


def _close(a, b, fields):
    for f in fields:
        x, y = a.get(f), b.get(f)
        assert np.linalg.norm(x - y) <= RTOL * np.linalg.norm(y), f


@pytest.mark.parametrize("n", [85, 86, 109])
def test_flow(need_gpu, n):
    s = cfdl.Setup(cfdl.Zone(n, jitter=0.1, seed=n))
    a, b = (cfdl.Solver(s, cfdl.steady()) for _ in range(2))
    b.set_tile(2)
    for g in (a, b):
        g.step(2, 0)
    _close(a, b, ("u", "v", "w", "p"))


def test_energy_keeps_its_tiles(need_gpu):
    """Setting the energy equation up takes the size rule back, as naming the tile shape does."""
    s = cfdl.Setup(cfdl.Zone(86, jitter=0.1, seed=1))
    a, b = (cfdl.Solver(s, cfdl.steady()) for _ in range(2))
    a.energy_init()
    b.set_tile(2)
    b.energy_init()
    b.set_tile(4)
    for g in (a, b):
        g.step(2, 0)
    for f in ("u", "p", "t"):
        assert np.array_equal(a.get(f), b.get(f)), f


def test_precision_changed(need_gpu):
    s = cfdl.Setup(cfdl.Zone(86, jitter=0.1, seed=1))
    a, b = cfdl.Solver(s, cfdl.steady()), cfdl.Solver(s, cfdl.steady(precision=3))
    b.set_config(cfdl.steady())
    for g in (a, b):
        g.step(2, 0)
    for f in ("u", "v", "w", "p"):
        assert np.array_equal(a.get(f), b.get(f)), f
