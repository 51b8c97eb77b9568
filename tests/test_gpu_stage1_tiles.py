"""Stage 1 at the edges of its pixel tiles and on both ways of sorting: codes
whose differing bits fit in one word with the record number, and codes of
depth 21 that do not."""
import numpy as np
import pytest

from tgvreconclaude_gb300 import api

pytestmark = pytest.mark.gpu


def _map(rng, w, h, f, holes):
    d = rng.uniform(0.9, 1.1, (h, w)).astype(np.float32)
    d[rng.random((h, w)) < holes] = np.nan
    return dict(depth=d, rt=np.eye(4, dtype=np.float32), fx=f, fy=f, cx=w / 2, cy=h / 2)


@pytest.mark.parametrize("w,h", [(2, 1), (31, 1), (32, 32), (341, 3), (1025, 1), (64, 32), (683, 3), (1024, 5)])
@pytest.mark.parametrize("holes", [0.0, 0.3, 0.97])
def test_tiles(oracle_lib, w, h, holes):
    m = _map(np.random.default_rng(w), w, h, 100.0, holes)
    assert api.build_cubes(m, (-3, -3, -3), 3.0).tobytes() == oracle_lib.build_cubes(m, (-3, -3, -3), 3.0).tobytes()


@pytest.mark.parametrize("r_root,deep", [(3.0, False), (1000.0, True), (3e5, True), (1e-3, False)])
def test_code_bits(oracle_lib, r_root, deep):
    """r_root 1000 and up: depth 21, all 63 bits; 1e-3: no pixel inside the box."""
    m = _map(np.random.default_rng(3), 160, 90, 2500.0, 0.1)
    m["depth"][np.isfinite(m["depth"])] = 1.0
    o = (-r_root,) * 3
    out = api.build_cubes(m, o, r_root)
    assert out.tobytes() == oracle_lib.build_cubes(m, o, r_root).tobytes()
    assert not deep or out["depth"].max() == 21
