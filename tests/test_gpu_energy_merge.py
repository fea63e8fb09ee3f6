"""The energy solve's blocks take one to four tiles each, by the cells of the whole
context: a case has the same bits alone (one tile a block) and in batches where
blocks take two, three and four, with whole and part-filled last blocks."""
import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

STATE = ("u", "v", "w", "p", "gu", "gv", "gw", "gp", "mip", "mip0", "t", "e", "e0")

# cells of one more case, which set the tiles a block takes in the whole context (608 blocks of 256 cells a wave)
OTHERS = {2: 55, 3: 69, 4: 86}


@pytest.mark.parametrize("tiles", [2, 3, 4])
@pytest.mark.parametrize("precision", [0, 2])
def test_alone_and_merged(need_gpu, precision, tiles):
    zones = [cfdl.Zone(n, kind=k, jitter=0.1, seed=n) for k, n in (("hex", 2), ("hex", 10), ("tet", 9), ("prism", 11), ("hex", 23))]
    setups = [cfdl.Setup(z) for z in zones]
    cfg = cfdl.steady(precision=precision)
    bt = cfdl.Batch(setups + [cfdl.Setup(cfdl.Zone(OTHERS[tiles], seed=1))], [cfg] * (len(setups) + 1))
    bt.energy_init()
    bt.step(2, 0)
    alone = {}
    for i, s in zip(bt.ids(), setups):      # the flow and temperature of the batch: the energy solve alone is compared
        g = alone[i] = cfdl.Solver(s, cfg)
        g.energy_init()
        for f in STATE:
            g.set(f, bt.case_get(i, f))
    for g in (bt, *alone.values()):
        g.solve_energy()
    for i, g in alone.items():
        for f in ("t", "e"):
            assert np.array_equal(bt.case_get(i, f), g.get(f)), (g.ne, f)
