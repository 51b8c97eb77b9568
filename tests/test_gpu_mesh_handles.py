"""Mesh handles: the newest mesh of a context is read from the device, older
ones and those of a destroyed context from host memory, with the same bytes."""
import ctypes as C
import threading

import numpy as np
import pytest

from tgvreconclaude_gb300 import api, formats as F, scenes as S

pytestmark = pytest.mark.gpu
ORIGIN = np.zeros(3, np.float32)


def _problem(seed, n=4000):
    rng = np.random.default_rng(seed)
    cubes = S.random_octree(rng, 2, 6, n)
    st = np.zeros(len(cubes), F.STATE_DTYPE)
    st["u"] = rng.uniform(-1, 1, len(cubes))
    return cubes, st


def _extract(ctx, cubes, st):
    h = C.c_void_p()
    ctx.check(ctx.lib.tgvg_extract_surface(ctx.h, cubes.ctypes.data, st.ctypes.data, len(cubes), None,
                                           ORIGIN.ctypes.data, 1.0, 1, C.byref(h)), "extract")
    return h


def _read(lib, h):
    nv, nf, hn = C.c_int64(), C.c_int64(), C.c_int32()
    assert lib.tgvg_mesh_size(h, C.byref(nv), C.byref(nf), C.byref(hn)) == 0 and hn.value == 1
    v, n = np.zeros((nv.value, 3), np.float32), np.zeros((nv.value, 3), np.float32)
    f = np.zeros((nf.value, 3), np.uint32)
    assert lib.tgvg_mesh_read(h, v.ctypes.data, f.ctypes.data, n.ctypes.data) == 0
    return v.tobytes(), f.tobytes(), n.tobytes()


def test_meshes_outlive_later_calls_and_their_context(oracle_lib):
    a, b = _problem(1), _problem(2, 9000)
    want = [tuple(x.tobytes() for x in oracle_lib.extract_surface(c, s, ORIGIN, 1.0, normals=True)) for c, s in (a, b)]
    ctx = api.Context(0)
    lib = ctx.lib
    ha = _extract(ctx, *a)
    hb = _extract(ctx, *b)  # moves the first mesh to the host
    assert _read(lib, ha) == want[0] and _read(lib, hb) == want[1]
    hc = _extract(ctx, *a)
    v = np.frombuffer(want[1][0], np.float32).reshape(-1, 3).copy()
    f = np.frombuffer(want[1][1], np.uint32).reshape(-1, 3).copy()
    n = np.zeros_like(v)
    ctx.check(lib.tgvg_compute_normals(ctx.h, v.ctypes.data, len(v), f.ctypes.data, len(f), n.ctypes.data), "normals")
    assert n.tobytes() == want[1][2]
    hd = _extract(ctx, *b)
    lib.tgvg_mesh_free(hb)
    ctx.close()
    assert _read(lib, hc) == want[0] and _read(lib, hd) == want[1]  # the context is gone
    for h in (ha, hc, hd):
        lib.tgvg_mesh_free(h)


def test_reads_beside_extractions(oracle_lib):
    """One thread reads a mesh while another extracts the next ones on the same context."""
    a, b = _problem(3), _problem(4)
    want = tuple(x.tobytes() for x in oracle_lib.extract_surface(*a, ORIGIN, 1.0, normals=True))
    ctx = api.context()
    h = _extract(ctx, *a)
    bad = []

    def reads():
        for _ in range(40):
            if _read(ctx.lib, h) != want:
                bad.append(1)

    t = threading.Thread(target=reads)
    t.start()
    for _ in range(20):
        ctx.lib.tgvg_mesh_free(_extract(ctx, *b))
    t.join()
    ctx.lib.tgvg_mesh_free(h)
    assert not bad
