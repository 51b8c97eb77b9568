"""The scratch that merges and balances leave in their context is given back:
by tgvg_trim, and to an eighth of a device budget when one is set."""
import ctypes as C

import numpy as np
import pytest

from tgvreconclaude_gb300 import api, formats as F

pytestmark = pytest.mark.gpu


def _merge(ctx, lists):
    n = sum(len(a) for a in lists)
    out, cnt = np.empty(n, F.CUBE_DTYPE), C.c_int64()
    ptrs = (C.c_void_p * len(lists))(*[a.ctypes.data for a in lists])
    sizes = (C.c_int64 * len(lists))(*[len(a) for a in lists])
    ctx.check(ctx.lib.tgvg_merge_cubes(ctx.h, ptrs, sizes, len(lists), out.ctypes.data, n, C.byref(cnt)), "merge")
    return out[:cnt.value].tobytes()


def test_scratch_is_given_back():
    """8 M cubes leave their two lists (256 MB) in the context's cache."""
    import torch
    key = np.arange(4_000_000, dtype=np.uint64)
    lists = [F.make_cubes(key * np.uint64(2) + np.uint64(k), np.full(len(key), 21, np.int32),
                          np.full(len(key), 0.5 + k, np.float32)) for k in (0, 1)]
    ctx = api.Context(0)
    free = lambda: torch.cuda.mem_get_info()[0]
    try:
        want = _merge(ctx, lists)
        held = free()
        ctx.check(ctx.lib.tgvg_set_device_budget(ctx.h, 8 << 20), "budget")  # keeps 1 MiB of it
        assert free() - held >= 250e6
        assert _merge(ctx, lists) == want and free() - held >= 250e6
        ctx.check(ctx.lib.tgvg_set_device_budget(ctx.h, 0), "budget")
        assert _merge(ctx, lists) == want and free() - held < 100e6
        ctx.trim()
        assert free() - held >= 250e6
        assert _merge(ctx, lists) == want
    finally:
        ctx.close()
