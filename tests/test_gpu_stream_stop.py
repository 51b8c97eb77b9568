"""Streaming solves to a tolerance on the on-chip schedules end when every leaf
has stopped, and not at the cap on iterations."""
import numpy as np
import pytest

from test_gpu_grid_levels import _level
from tgvreconclaude_gb300 import api, scenes as S

pytestmark = pytest.mark.gpu
CAP = 400_000


# one CTA, a cluster of 8 and of 16, one and two cubes a thread over the whole GPU, shared memory
@pytest.mark.parametrize("n, cfg", [(200, 23), (2000, 23), (9000, 24), (30_000, 24), (200_000, 24), (300_000, 24)])
def test_ends_with_its_last_leaf(oracle_lib, n, cfg):
    """Two barriers an iteration are at least 0.2 us, so a level run to the cap
    would take 80 ms and more; leaves that stop within 400 iterations, under 10."""
    rng = np.random.default_rng(n)
    cubes = _level(rng, n)
    h = S.random_histograms(rng, len(cubes))
    lv = S.split_leaves(len(cubes), 5, rng, cubes, aligned=True)
    ref, rst = oracle_lib.tgv_solve(cubes, h, lv, "stream", 0.5, 0.5, CAP, nthreads=8, tol=0.06, check_every=5)
    assert max(r["iters_run"] for r in rst) <= 400
    ctx = api.context()
    ctx.set_schedule("stream", n.bit_length() - 1, cfg)
    try:
        for _ in range(4):  # the last ones replay a captured level loop
            out, st = api.tgv_solve(cubes, h, lv, "stream", api.TGVParams(0.5, 0.5, CAP, tol=0.06, check_every=5))
            assert out.tobytes() == ref.tobytes()
            assert st["iters_run"] == [r["iters_run"] for r in rst]
            k = st["active"].index(n)
            assert st["schedule"][k] == cfg and st["level_ms"][k] < 10.0
    finally:
        ctx.set_schedule("stream", -1, -1)
