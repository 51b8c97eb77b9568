"""The whole-GPU register kernel at the edges of its sizes: one cube more than a
cluster holds, a last block with one cube, one and two cubes per thread, the
largest unit and one beyond it, against the oracle."""
import numpy as np
import pytest

from tgvreconclaude_gb300 import api, formats as F, scenes as S

pytestmark = pytest.mark.gpu
SM = 152


def _level(rng, n):
    """n cells of a slab three cells thick at one depth, and a few thousand of other depths."""
    d = 7 if n <= 30_000 else 9
    g = 1 << d
    i = rng.choice(3 * g * g, n, replace=False)
    x, y, z = i // 3 % g, i // (3 * g), g // 2 + i % 3
    sh = 21 - d
    key = F.morton_encode(*[(v << sh).astype(np.uint32) for v in (x, y, z)])
    c = F.make_cubes(key, np.full(n, d, np.int32), np.full(n, 0.01, np.float32))
    e = S.random_octree(rng, 2, 6, 4000)
    c = np.concatenate([c, e])
    key = F.cube_keys(c)
    return c[np.argsort(key, kind="stable")]


@pytest.mark.parametrize("mode", ["inmem", "oc", "stream"])
@pytest.mark.parametrize("tol", [0.0, 1e-3])
@pytest.mark.parametrize("n", [16 * 1024 + 1, SM * 160 - 1, SM * 160 + 1, SM * 1024, SM * 1024 + 1, SM * 1664, SM * 1664 + 1])
def test_units_over_the_whole_gpu(oracle_lib, n, mode, tol):
    """Bit for bit, as every schedule: the default of an untuned unit of this size."""
    rng = np.random.default_rng(n)
    cubes = _level(rng, n)
    h = S.random_histograms(rng, len(cubes))
    lv = None if mode == "inmem" else S.split_leaves(len(cubes), 1 if mode == "oc" else 5, rng, cubes, aligned=True)
    iters = 25 if tol else 8
    ref, rst = oracle_lib.tgv_solve(cubes, h, lv, mode, 0.5, 0.5, iters, nthreads=8,
                                    **(dict(tol=tol, check_every=5) if tol else {}))
    out, st = api.tgv_solve(cubes, h, lv, mode, api.TGVParams(0.5, 0.5, iters, tol=tol, check_every=5))
    assert out.tobytes() == ref.tobytes()
    if tol:
        assert st["iters_run"] == [r["iters_run"] for r in rst]


def test_graph_replays_follow_a_moved_scratch(oracle_lib):
    """A captured solve of a unit that ran on the whole GPU, then a larger one
    (the exchange buffer moves), then the first again: captured anew, same bits."""
    ctx = api.context()
    rng = np.random.default_rng(1)
    small, big = _level(rng, 20_000), _level(rng, 120_000)
    prm = api.TGVParams(0.5, 0.5, 6)
    hs, hb = S.random_histograms(rng, len(small)), S.random_histograms(rng, len(big))
    ref = oracle_lib.tgv_solve(small, hs, None, "inmem", 0.5, 0.5, 6)[0].tobytes()
    for _ in range(3):
        assert api.tgv_solve(small, hs, None, "inmem", prm)[0].tobytes() == ref
    assert api.tgv_solve(big, hb, None, "inmem", prm)[0].tobytes() == \
        oracle_lib.tgv_solve(big, hb, None, "inmem", 0.5, 0.5, 6)[0].tobytes()
    for _ in range(3):
        assert api.tgv_solve(small, hs, None, "inmem", prm)[0].tobytes() == ref


@pytest.mark.parametrize("mode", ["inmem", "oc", "stream"])
@pytest.mark.parametrize("tol", [0.0, 1e-3])
@pytest.mark.parametrize("n", [SM * 1664 + 1, 300_000, 520_001, 700_001])
def test_units_in_shared_memory(oracle_lib, n, mode, tol):
    """Schedule 24 beyond the registers: in shared memory while the unit fits,
    band order above, bit for bit the oracle's."""
    rng = np.random.default_rng(n)
    cubes = _level(rng, n)
    h = S.random_histograms(rng, len(cubes))
    lv = None if mode == "inmem" else S.split_leaves(len(cubes), 1 if mode == "oc" else 5, rng, cubes, aligned=True)
    iters = 25 if tol else 8
    ref, rst = oracle_lib.tgv_solve(cubes, h, lv, mode, 0.5, 0.5, iters, nthreads=8,
                                    **(dict(tol=tol, check_every=5) if tol else {}))
    ctx = api.context()
    ctx.set_schedule(mode, -1, 24)
    try:
        out, st = api.tgv_solve(cubes, h, lv, mode, api.TGVParams(0.5, 0.5, iters, tol=tol, check_every=5))
    finally:
        ctx.set_schedule(mode, -1, -1)
    assert set(st["schedule"]) == ({24} if n < 530_000 else {24, 14})
    assert out.tobytes() == ref.tobytes()
    if tol:
        assert st["iters_run"] == [r["iters_run"] for r in rst]
