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
