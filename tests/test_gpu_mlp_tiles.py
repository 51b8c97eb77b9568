"""The warm-start MLP kernels at the edges of their row tiles, against the FP64
numpy reference."""
import numpy as np
import pytest

import mlp_ref
from tgvreconclaude_gb300 import warmstart as WS

pytestmark = pytest.mark.gpu


def _rows(n, seed, nbins=10):
    rng = np.random.default_rng(seed)
    X = np.zeros((n, 16), np.float32)
    X[:, :nbins + 5] = rng.uniform(-1, 1, (n, nbins + 5))
    bits = (mlp_ref.bf16_round(X).view(np.uint32) >> 16).astype(np.uint16)
    return bits, rng.uniform(-1, 1, n).astype(np.float32)


# one row, a 16-row warp tile, a 64- and a 128-row step, the switch between them (128 rows per SM), a long ragged set
@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 128, 129, 128 * 152 - 1, 128 * 152, 128 * 152 + 1, 50_001])
def test_gradient_at_tile_edges(n):
    """Sums are FP32, so what can differ by more is a hidden activation that lies
    between two bf16 values and is rounded the other way: 2^-8 of it, seldom."""
    X, t = _rows(n, n)
    m = WS.WarmStartMLP(10, seed=5)
    loss, g = m.grad(X, t)
    lr, gr = mlp_ref.loss_and_grad(m.get_params(), mlp_ref.bf16_bits_to_float(X), t)
    assert abs(loss - lr) <= 2.0 ** -8 * lr
    for a, b in ((mlp_ref.P_W1, mlp_ref.P_B1), (mlp_ref.P_B1, mlp_ref.P_W2), (mlp_ref.P_W2, mlp_ref.P_B2),
                 (mlp_ref.P_B2, mlp_ref.P_W3), (mlp_ref.P_W3, mlp_ref.P_B3), (mlp_ref.P_B3, mlp_ref.P_N)):
        assert np.linalg.norm(g[a:b] - gr[a:b]) <= 2.0 ** -8 * np.linalg.norm(gr[a:b]), (a, b)


# one row, a warp, a 128-row tile, a tile on each SM, one on each of its eight groups, and their neighbours
@pytest.mark.parametrize("n", [1, 31, 32, 127, 128, 129, 128 * 152, 128 * 152 + 1, 1024 * 152 - 1, 1024 * 152 + 129])
def test_forward_at_tile_edges(n):
    """Sums are FP32, so what can differ by more is a hidden activation rounded to
    the other bf16 neighbour: 2^-8 of it, seldom.  The biases fill 24 bits."""
    X, _ = _rows(n, n)
    m = WS.WarmStartMLP(10, seed=5)
    p = np.array(m.get_params(), np.float32)
    b = np.random.default_rng(n).uniform(-0.5, 0.5, 129).astype(np.float32)
    p[mlp_ref.P_B1:mlp_ref.P_W2], p[mlp_ref.P_B2:mlp_ref.P_W3], p[mlp_ref.P_B3] = b[:64], b[64:128], b[128]
    m.set_params(p)
    y = m.predict(X)
    yr = np.asarray(mlp_ref.forward(p, mlp_ref.bf16_bits_to_float(X))[0]).reshape(-1)
    assert np.abs(y - yr).max() <= 2.0 ** -8 * np.abs(yr).max()
    assert np.linalg.norm(y - yr) <= 2.0 ** -8 * np.linalg.norm(yr)


@pytest.mark.parametrize("bias, want", [(np.inf, np.inf), (-np.inf, 0.0), (np.nan, 0.0), (3.4e38, 3.4e38)])
def test_forward_with_extreme_bias(bias, want):
    """ReLU of the bias alone: infinities stay, NaN counts as zero, as the FP32
    accumulator held them (3.4e38 rounds to a bf16 infinity there too)."""
    m = WS.WarmStartMLP(10, seed=5)
    p = np.zeros(mlp_ref.P_N, np.float32)
    p[mlp_ref.P_B2], p[mlp_ref.P_W3] = bias, 1.0
    m.set_params(p)
    y = m.predict(_rows(130, 1)[0])
    want = mlp_ref.bf16_round(np.array([want], np.float32))[0]
    assert np.all(y == want)


def _leaves(kind, n):
    """Chunk ranges over n cubes: a treetop's ascending ones, with gaps and an
    end beyond the cubes, out of order, overlapping, and with an empty one."""
    from tgvreconclaude_gb300 import formats as F
    e = np.linspace(0, n, 8).astype(int)
    r = {"none": [], "one": [(0, n - 1)], "ascending": [(a, b - 1) for a, b in zip(e, e[1:]) if b > a],
         "gaps": [(e[1], e[2] - 1), (e[3], e[4] - 1), (e[6], 2 * n + 5)], "reversed": [(e[4], n - 1), (0, e[4] - 1)],
         "overlap": [(0, e[5]), (e[2], n - 1)], "empty": [(5, 2), (0, n - 1)]}[kind]
    lv = np.zeros(len(r), F.LEAF_DTYPE)
    for k, (a, b) in enumerate(r):
        lv[k] = (k * 0x01000000, k * 0x10000, k % 5, max(0, a), max(0, b))
    return lv if len(lv) else None


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 5003])
@pytest.mark.parametrize("kind", ["none", "one", "ascending", "gaps", "reversed", "overlap", "empty"])
@pytest.mark.parametrize("nbins", [8, 10])
def test_fused_warm_start_is_features_then_network(n, kind, nbins):
    """The one-pass warm start equals median + predict(features), bit for bit,
    whatever the chunk ranges."""
    from tgvreconclaude_gb300 import scenes as S
    rng = np.random.default_rng(n)
    cubes = S.random_octree(rng, 2, 6, n, shape="plane")
    hists = S.random_histograms(rng, len(cubes), nbins)
    lv = _leaves(kind, len(cubes))
    m = WS.WarmStartMLP(nbins, seed=2)
    y = m.predict(m.features(cubes, hists, lv))
    assert m.warm_start(cubes, hists, lv).tobytes() == (WS.median_start(hists) + y).astype(np.float32).tobytes()


def test_fused_warm_start_takes_rows_at_any_word():
    """Device histogram rows that start on 4 bytes only (the wide loads need 8 or 16)."""
    import torch
    from tgvreconclaude_gb300 import scenes as S
    rng = np.random.default_rng(1)
    for nbins in (8, 10):
        cubes = S.random_octree(rng, 2, 6, 1000)
        hists = S.random_histograms(rng, len(cubes), nbins)
        m = WS.WarmStartMLP(nbins, seed=2)
        want = m.warm_start(cubes, hists)
        c = torch.from_numpy(cubes.view(np.int32).reshape(-1, 4).copy()).cuda()
        buf = torch.zeros(hists.size + 1, dtype=torch.int32, device="cuda")
        buf[1:] = torch.from_numpy(hists.view(np.int32).reshape(-1)).cuda()
        u = torch.empty(len(cubes), device="cuda")
        torch.cuda.synchronize()
        m.ctx.check(m.lib.tgvg_mlp_warm_start_dev(m.ctx.h, m.h, c.data_ptr(), buf[1:].data_ptr(), len(cubes), nbins,
                                                  None, 0, u.data_ptr()), "warm start")
        torch.cuda.synchronize()
        assert u.cpu().numpy().tobytes() == want.tobytes()
