"""The register-resident level kernels at the edges of their sizes: every CTA
count, a CTA that ends inside a warp, one that holds no cube, the largest unit."""
import numpy as np
import pytest

from tgvreconclaude_gb300 import api, scenes as S

pytestmark = pytest.mark.gpu


def _one_level(rng, n):
    """n cubes of one depth (and some of the depths beside it) around a plane."""
    d = 4 if n <= 500 else (5 if n <= 1100 else 7)
    c = S.random_octree(rng, d, d, 10 ** 9, shape="plane")
    c = c[np.sort(rng.choice(len(c), n, replace=False))]
    e = S.random_octree(rng, 2, d + 1, 300)
    c = np.concatenate([c, e[e["depth"] != d]])
    key = (c["hi"].astype(np.uint64) << np.uint64(32)) | c["lo"]
    return c[np.argsort(key, kind="stable")]


# one CTA: a lane, a warp, around it; 2, 4, 8 CTAs; schedule 23's end; the cluster's end and one beyond
SIZES = [1, 31, 32, 33, 255, 256, 257, 511, 513, 1023, 1025, 2047, 2048, 2049, 16 * 1024 - 1, 16 * 1024, 16 * 1024 + 1]


@pytest.mark.parametrize("mode", ["inmem", "oc", "stream"])
@pytest.mark.parametrize("tol", [0.0, 1e-3])
@pytest.mark.parametrize("n", SIZES)
def test_default_schedule_at_unit_sizes(oracle_lib, n, mode, tol):
    """States are the oracle's bit for bit (the arithmetic is the reference's,
    explicitly rounded), and so are the iteration counts of stopped solves."""
    rng = np.random.default_rng(n)
    cubes = _one_level(rng, n)
    h = S.random_histograms(rng, len(cubes))
    lv = None if mode == "inmem" else S.split_leaves(len(cubes), 1 if mode == "oc" else 3, rng, cubes, aligned=True)
    iters = 40 if tol else 12
    ref, rst = oracle_lib.tgv_solve(cubes, h, lv, mode, 0.5, 0.5, iters, **(dict(tol=tol, check_every=5) if tol else {}))
    out, st = api.tgv_solve(cubes, h, lv, mode, api.TGVParams(0.5, 0.5, iters, tol=tol, check_every=5))
    assert out.tobytes() == ref.tobytes()
    if tol:
        assert st["iters_run"] == [r["iters_run"] for r in rst]
