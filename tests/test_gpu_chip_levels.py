"""Levels on chip where their rarer paths run: ghost tables beside the
shared-memory kernel, more foreign neighbours than a block has room to stage,
the schedules that untuned units take, and two contexts at once."""
import ctypes as C
import threading

import numpy as np
import pytest

from test_gpu_grid_levels import _level
from test_gpu_parity import _refined_slab
from tgvreconclaude_gb300 import _native as N, api, formats as F, scenes as S

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _against_oracle(oracle, cubes, mode, leaves, iters, n, cfg=24):
    """Fixed count and to a tolerance, bit for bit; the level of n cubes runs schedule cfg."""
    h = S.random_histograms(np.random.default_rng(n), len(cubes), empty_frac=0.05)
    ctx = api.context()
    ctx.set_schedule(mode, -1, cfg)
    try:
        for tol in (0.0, 0.02):
            kw = dict(tol=tol, check_every=5) if tol else {}
            ref, rst = oracle.tgv_solve(cubes, h, leaves, mode, 0.5, 0.5, iters, nthreads=8, **kw)
            out, st = api.tgv_solve(cubes, h, leaves, mode, api.TGVParams(0.5, 0.5, iters, tol=tol, check_every=5))
            assert st["schedule"][st["active"].index(n)] == cfg
            assert out.tobytes() == ref.tobytes(), (mode, tol)
            if tol:
                assert st["iters_run"] == [r["iters_run"] for r in rst]
    finally:
        ctx.set_schedule(mode, -1, -1)


@pytest.mark.parametrize("mode", ["inmem", "stream"])
def test_shared_memory_kernel_reads_coarser_ghosts(oracle_lib, mode):
    """A level beyond the registers' 1664 cubes an SM with coarser neighbours across its -x/-y/-z faces."""
    rng = np.random.default_rng(3)
    cubes = S.random_octree(rng, dmin=3, dmax=9, target=600_000, shape="sphere")
    n = int(np.bincount(cubes["depth"]).max())
    assert 1664 * _sms() < n < 3500 * _sms()
    fine = np.where(cubes["depth"] == cubes["depth"].max())[0]
    assert len(fine) == n
    nb = oracle_lib.neighbour_table(cubes)[fine][:, 1::2]
    assert ((nb >= 0) & (cubes["depth"][np.maximum(nb, 0)] < cubes["depth"].max())).mean() > 0.03
    _against_oracle(oracle_lib, cubes, mode, S.split_leaves(len(cubes), 4, rng, cubes, aligned=True), 40, n)


@pytest.mark.parametrize("mode", ["inmem", "stream"])
def test_shared_memory_kernel_reads_deeper_ghosts(oracle_lib, mode):
    """262,144 cubes with a deeper neighbour across every +z face, from the dual sweep's table."""
    cubes = _refined_slab()
    assert 1664 * _sms() < 262_144
    lv = S.split_leaves(len(cubes), 3, np.random.default_rng(17), cubes, aligned=True)
    _against_oracle(oracle_lib, cubes, mode, lv, 12, 262_144)


def _sparse_children(n, d=8):
    """n cells of depth d, three of the eight of each cell of depth d - 1, which
    are cubes too: nearly every neighbour of a deep cell is a coarser cube."""
    m = next(m for m in range(1, 200) if 3 * m ** 3 >= n)
    x, y, z = (v.ravel().astype(np.uint32) for v in np.meshgrid(*[np.arange(m)] * 3, indexing="ij"))
    sh = 21 - d
    up = F.morton_encode(*[v << (sh + 1) for v in (x, y, z)])
    down = np.sort(np.concatenate([F.morton_encode((2 * x + a) << sh, (2 * y + b) << sh, (2 * z + c) << sh)
                                   for a, b, c in ((1, 1, 0), (1, 0, 1), (0, 1, 1))]))[:n]
    key, depth = np.concatenate([up, down]), np.repeat(np.int32([d - 1, d]), [len(up), n])
    o = np.lexsort((depth, key))
    return F.make_cubes(key[o], depth[o], np.full(len(key), 0.01, np.float32))


@pytest.mark.parametrize("mode", ["inmem", "oc", "stream"])
def test_more_foreign_records_than_a_block_stages(oracle_lib, mode):
    """Two cubes a thread on nearly the most threads: of a block's 1,640 cubes'
    9,840 neighbours, all on the coarser level, shared memory has room for some
    5,300 records (231,424 bytes less 88 a cube, 16 each)."""
    n = 1640 * _sms()
    cubes = _sparse_children(n)
    nb = oracle_lib.neighbour_table(cubes)[cubes["depth"] == 8]
    assert ((nb >= 0) & (cubes["depth"][np.maximum(nb, 0)] == 7)).sum(1).mean() > 5.5
    lv = S.split_leaves(len(cubes), 1 if mode == "oc" else 3, np.random.default_rng(1), cubes, aligned=True)
    _against_oracle(oracle_lib, cubes, mode, lv, 20, n)


@pytest.mark.parametrize("mode", ["inmem", "oc", "stream"])
def test_schedules_of_untuned_units(mode):
    """Clusters up to 2,048 and 16 x 1,024 cubes, then the whole GPU up to what its shared memory holds, then
    band order; the states are band order's, bit for bit."""
    sm = _sms()
    ctx = api.context()
    for n, cfg in ((1, 23), (2048, 23), (2049, 24), (16_384, 24), (16_385, 24), (1664 * sm, 24), (1664 * sm + 1, 24),
                   (3500 * sm, 24), (3600 * sm, 14)):
        rng = np.random.default_rng(n)
        cubes = _level(rng, n)
        h = S.random_histograms(rng, len(cubes))
        lv = None if mode == "inmem" else S.split_leaves(len(cubes), 1 if mode == "oc" else 3, rng, cubes, aligned=True)
        got = []
        try:
            for fixed in (-1, 14):
                ctx.set_schedule(mode, -1, fixed)
                out, st = api.tgv_solve(cubes, h, lv, mode, api.TGVParams(0.5, 0.5, 6))
                got.append((out.tobytes(), st["schedule"][st["active"].index(n)]))
        finally:
            ctx.set_schedule(mode, -1, -1)
        assert got[0] == (got[1][0], cfg) and got[1][1] == 14, n


def test_two_contexts_at_once(oracle_lib):
    """Two threads, each with a context and stream of its own, solve levels that take the whole GPU (one and two
    cubes a thread, shared memory) at the same time."""
    work = []
    for n in (30_000, 1640 * _sms(), 300_000):
        rng = np.random.default_rng(n)
        cubes = _level(rng, n)
        h = S.random_histograms(rng, len(cubes))
        ref = oracle_lib.tgv_solve(cubes, h, None, "inmem", 0.5, 0.5, 30, nthreads=8)[0].tobytes()
        work.append((cubes, h, ref))
    prm = N.Params(0.5, 0.5, 30, 0, 0.0, 10, 0)
    bad = []

    def solves(first):
        ctx = api.Context(0)
        try:
            ctx.set_schedule("inmem", -1, 24)
            for k in range(12):
                cubes, h, ref = work[(first + k) % len(work)]
                out = np.zeros(len(cubes), F.STATE_DTYPE)
                rc = ctx.lib.tgvg_tgv_minimize(ctx.h, cubes.ctypes.data, h.ctypes.data, len(cubes), h.shape[1], None, 0,
                                               0, C.byref(prm), None, out.ctypes.data, None)
                if rc != 0 or out.tobytes() != ref:
                    bad.append((first, k, rc))
        finally:
            ctx.close()

    threads = [threading.Thread(target=solves, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
