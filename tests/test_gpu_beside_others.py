"""Levels that take the whole GPU beside another stream's kernel that stays on
one SM for longer than the grid barrier's limit: the solve waits for it where
there is no room beside it, and its own waits do not run out."""
import numpy as np
import pytest

from test_gpu_grid_levels import _level
from tgvreconclaude_gb300 import api, scenes as S

pytestmark = pytest.mark.gpu


# one cube a thread and two, all registers in use, shared memory
@pytest.mark.parametrize("n", [30_000, 1024 * 152, 250_000, 300_000])
def test_waits_for_a_resident_block(n):
    import torch
    rng = np.random.default_rng(n)
    cubes = _level(rng, n)
    h = S.random_histograms(rng, len(cubes))
    ctx, side, prm = api.context(), torch.cuda.Stream(), api.TGVParams(0.5, 0.5, 20)
    try:
        ctx.set_schedule("inmem", -1, 14)
        want = api.tgv_solve(cubes, h, None, "inmem", prm)[0].tobytes()
        ctx.set_schedule("inmem", -1, 24)
        with torch.cuda.stream(side):
            torch.cuda._sleep(5_000_000_000)  # about 2.5 s
        out, st = api.tgv_solve(cubes, h, None, "inmem", prm)
        assert st["schedule"][st["active"].index(n)] == 24 and out.tobytes() == want
    finally:
        ctx.set_schedule("inmem", -1, -1)
        side.synchronize()
