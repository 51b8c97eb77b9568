"""A wait of the network's kernel that runs out: the call it happens in says so,
no other one does, and the context goes on (the wait limit set to nothing)."""
import numpy as np
import pytest

from tgvreconclaude_gb300 import api, scenes as S, warmstart as WS

pytestmark = pytest.mark.gpu


def _limit(m, polls):
    m.ctx.check(m.lib.tgvg_mlp_set_wait_limit(m.h, polls), "wait limit")


# one row, a tile and a half, a tile for every group of every SM and more
@pytest.mark.parametrize("n", [1, 200, 400_000])
def test_a_call_that_waits_reports_its_own_wait(n):
    m = WS.WarmStartMLP(10, seed=3)
    X = np.random.default_rng(n).integers(0x3c00, 0x3f80, (n, 16)).astype(np.uint16)
    good = m.predict(X).tobytes()
    for _ in range(2):
        _limit(m, 0)
        with pytest.raises(RuntimeError, match="timed out"):
            m.predict(X)
        _limit(m, 1 << 30)
        assert m.predict(X).tobytes() == good


def test_the_device_form_is_reported_by_the_next_solve_only(oracle_lib):
    import torch
    rng = np.random.default_rng(0)
    cubes = S.random_octree(rng, 2, 6, 3000)
    hists = S.random_histograms(rng, len(cubes), 8)
    m = WS.WarmStartMLP(8, seed=3)
    want = m.warm_start(cubes, hists)
    c = torch.from_numpy(cubes.view(np.int32).reshape(-1, 4).copy()).cuda()
    h = torch.from_numpy(hists.view(np.int32)).cuda()
    u = torch.zeros(len(cubes), device="cuda")
    torch.cuda.synchronize()

    def dev():
        m.ctx.check(m.lib.tgvg_mlp_warm_start_dev(m.ctx.h, m.h, c.data_ptr(), h.data_ptr(), len(cubes), 8, None, 0,
                                                  u.data_ptr()), "warm start")
        torch.cuda.synchronize()
        return u.cpu().numpy()

    prm = api.TGVParams(0.5, 0.5, 5)
    ref = oracle_lib.tgv_solve(cubes, hists, None, "inmem", 0.5, 0.5, 5)[0].tobytes()
    _limit(m, 0)
    assert np.isnan(dev()).all()
    _limit(m, 1 << 15)
    assert m.warm_start(cubes, hists).tobytes() == want.tobytes()  # a good call of the same network
    assert m.predict(np.zeros((5, 16), np.uint16)).shape == (5,)
    assert dev().tobytes() == want.tobytes()
    with pytest.raises(RuntimeError, match="timed out"):
        api.tgv_solve(cubes, hists, None, "inmem", prm)
    assert api.tgv_solve(cubes, hists, None, "inmem", prm)[0].tobytes() == ref
    dev()
    assert api.tgv_solve(cubes, hists, None, "inmem", prm)[0].tobytes() == ref
