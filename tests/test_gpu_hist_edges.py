"""The binning kernel's quick pixel, level and bin values where they matter: pairs
that fall exactly on whole pixels, on level thresholds and on bin edges, a few
units in the last place beside them, and parameters outside the range in which
quick values are used.  Histograms equal the oracle's, bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import cams_from
from tgvreconclaude_gb300 import api, formats as F

pytestmark = pytest.mark.gpu
ORIGIN, R_ROOT = (-1.0, -1.0, -1.0), 1.0


def _nudge(x, rng):
    """x, or the float one, two or many units in the last place beside it."""
    x = np.asarray(x, np.float32)
    k = rng.choice([0, 0, 1, -1, 2, -2, 8, -8, 40, -40, 400, -400], x.shape)
    return (x.view(np.int32) + k).astype(np.int32).view(np.float32)


def _grid(rng, n=6000, d=5):
    """Cubes whose centres are dyadic numbers, radii around powers of two."""
    g = rng.integers(0, 1 << d, (n, 3)).astype(np.uint32) << (21 - d)
    key = np.sort(F.morton_encode(g[:, 0], g[:, 1], g[:, 2]))
    return F.make_cubes(key, np.full(n, d, np.int32), _nudge(2.0 ** rng.integers(-9, -1, n), rng))


def _map(rng, fx, fy, cx, cy, w=64, h=48, z0=-3.0, rt=None):
    """A camera on the z axis looking along it; depths at the cubes' own distances
    plus multiples of an eighth and a tenth of common deltas."""
    m = np.eye(4, dtype=np.float32)
    m[2, 3] = -z0
    if rt is not None:
        m = rt
    z = (np.arange(32) + 0.5) / 16 - 1.0 - z0
    depth = rng.choice(z, (h, w)) + rng.integers(-10, 11, (h, w)) * rng.choice([2 / 8, 2 / 10, 1 / 16], (h, w)) * 6.0 \
        * 2.0 ** rng.integers(-9, -4, (h, w))
    depth = _nudge(depth.astype(np.float32), rng)
    depth[rng.random((h, w)) < 0.1] = rng.choice([np.nan, 0.0, -1.0, np.inf], (depth.shape))[rng.random((h, w)) < 0.1][:1]
    return dict(depth=np.ascontiguousarray(depth, np.float32), rt_inv=m, rt=np.eye(4, dtype=np.float32), fx=fx, fy=fy,
                cx=cx, cy=cy, lidar=bool(rng.integers(2)))


def _check(oracle_lib, cubes, maps, nbins, origin=ORIGIN, r_root=R_ROOT):
    ref = oracle_lib.compute_histograms(cubes, maps, origin, r_root, nbins=nbins, nthreads=8)
    gpu = api.compute_histograms_from_maps(cubes, cams_from(maps), [m["depth"] for m in maps], origin, r_root,
                                           nbins=nbins)
    assert np.array_equal(gpu, ref)
    return int(ref.sum())


@pytest.mark.parametrize("nbins", [8, 10])
@pytest.mark.parametrize("seed", range(4))
def test_whole_pixels_levels_and_bin_edges(oracle_lib, nbins, seed):
    rng = np.random.default_rng(100 * nbins + seed)
    maps = [_map(rng, float(_nudge(f, rng)), float(_nudge(-f if seed == 3 else f, rng)), c, c - 8.0)
            for f in (16.0, 32.0, 64.0, 96.0, 128.0) for c in (32.0, 31.5, 0.0, 64.0)]
    assert _check(oracle_lib, _grid(rng), maps, nbins) > 1000


def test_large_images(oracle_lib):
    """The margin grows with the image: 4,100 columns, centres off to both sides."""
    rng = np.random.default_rng(5)
    maps = [_map(rng, float(f), 8.0, c, 8.0, w=4100, h=16) for f in (2048.0, 1500.0) for c in (0.0, 2050.0, 5000.0)]
    assert _check(oracle_lib, _grid(rng, 20000), maps, 10) > 1000


@pytest.mark.parametrize("kind", ["tiny f", "huge f", "inf f", "nan f", "zero f", "huge c", "nan row", "inf row", "tiny z",
                                  "huge z"])
def test_parameters_out_of_range(oracle_lib, kind):
    rng = np.random.default_rng(len(kind))
    m = [_map(rng, 32.0, 32.0, 32.0, 24.0) for _ in range(3)]
    rt = m[1]["rt_inv"].copy()
    if kind.endswith(" f"):
        m[1]["fx"] = {"tiny": 1e-5, "huge": 1e8, "inf": np.inf, "nan": np.nan, "zero": 0.0}[kind[:-2]]
    elif kind == "huge c":
        m[1]["cx"] = 1e7
    else:
        s = {"tiny z": 1e-30, "huge z": 1e30}.get(kind)
        if s:  # the whole camera space scaled: the same pixels, depths far out of range
            rt[:3] *= np.float32(s)
            m[1]["depth"] = (m[1]["depth"] * np.float32(s)).astype(np.float32)
        else:
            rt[0, 1] = np.nan if kind == "nan row" else np.inf
    m[1]["rt_inv"] = rt
    _check(oracle_lib, _grid(rng), m, 8)


def test_radii_out_of_range(oracle_lib):
    rng = np.random.default_rng(3)
    c = _grid(rng)
    odd = rng.random(len(c)) < 0.5
    c["r_c"][odd] = rng.choice(np.float32([0.0, -1.0, 1e-30, 1e-40, 1e28, 3e38, np.inf, np.nan]), odd.sum())
    _check(oracle_lib, c, [_map(rng, 32.0, 32.0, 32.0, 24.0) for _ in range(4)], 10)


def test_many_votes(oracle_lib):
    """More votes than 16 bits hold: 14,000 lidar cameras at five votes each."""
    rng = np.random.default_rng(4)
    m = _map(rng, 4.0, 4.0, 2.0, 2.0, w=4, h=4)
    m["lidar"] = True
    m["depth"][:] = 3.0
    ref = _check(oracle_lib, _grid(rng, 40, 2), [m] * 14000, 8)
    assert ref > 65535
