"""A schedule that was picked for a unit on one side of an on-chip kernel's size
limit is not applied to a unit on the other side of it, in the same size class."""
import numpy as np
import pytest

from test_gpu_grid_levels import _level
from tgvreconclaude_gb300 import api, scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beyond, within, cfg", [(3000, 2048, 23), (600_000, 530_000, 24)])
def test_picks_stay_on_their_side(beyond, within, cfg):
    """Too few iterations to tune: the unit within takes its own default."""
    ctx = api.context()
    ctx.set_schedule("inmem", -1, -1)
    got = []
    try:
        for n, iters in ((beyond, 500), (within, 8), (beyond, 8)):
            rng = np.random.default_rng(n)
            cubes = _level(rng, n)
            st = api.tgv_solve(cubes, S.random_histograms(rng, len(cubes)), None, "inmem", api.TGVParams(0.5, 0.5, iters))[1]
            got.append(st["schedule"][st["active"].index(n)])
        assert got[1] == cfg and got[2] == got[0]
    finally:
        ctx.set_schedule("inmem", -1, -1)
