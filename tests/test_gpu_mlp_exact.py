"""The gradient keeps FP32 accuracy: every part of the split factors of the
backward products counts."""
import numpy as np
import pytest

import mlp_ref
from tgvreconclaude_gb300 import warmstart as WS

pytestmark = pytest.mark.gpu

BLOCKS = {"W1": (mlp_ref.P_W1, mlp_ref.P_B1), "b1": (mlp_ref.P_B1, mlp_ref.P_W2), "W2": (mlp_ref.P_W2, mlp_ref.P_B2),
          "b2": (mlp_ref.P_B2, mlp_ref.P_W3), "W3": (mlp_ref.P_W3, mlp_ref.P_B3), "b3": (mlp_ref.P_B3, mlp_ref.P_N)}


def problem(n, seed):
    """Rows and positive weights in eighths, so that the hidden layers' sums are
    exact in FP32 and round to the same bf16 values as the reference's, and
    targets below every output, so that no sum of the gradient cancels."""
    rng = np.random.default_rng(seed)
    X = rng.integers(0, 9, (n, 16)).astype(np.float32) / 8
    p = np.zeros(mlp_ref.P_N, np.float32)
    p[mlp_ref.P_W1:mlp_ref.P_B1] = rng.integers(1, 9, 16 * 64) / 8
    p[mlp_ref.P_W2:mlp_ref.P_B2] = rng.integers(1, 9, 64 * 64) / 8
    p[mlp_ref.P_W3:mlp_ref.P_B3] = rng.integers(1, 9, 64) / 8
    return X, p, -rng.uniform(1, 9000, n).astype(np.float32)


# half a step of 64 rows, a ragged one, many; the 128-row form, ragged
@pytest.mark.parametrize("n", [32, 100, 2000, 25_001])
def test_gradient_has_fp32_accuracy(n):
    """Twelve accumulating mma and the FP32 adds over rows and blocks each lose
    at most 2^-23, typically 2^-24, of a sum without cancellation: 2e-6 if all
    in one direction, and the bound is twice that.  Without the low part of the
    split the gradients of W2 and W1 are 1.0e-5 and 2.1e-5 off, without the
    middle part 2.7e-3."""
    X, p, t = problem(n, n)
    m = WS.WarmStartMLP(10, seed=5)
    m.set_params(p)
    loss, g = m.grad((X.view(np.uint32) >> 16).astype(np.uint16), t)
    lr, gr = mlp_ref.loss_and_grad(p, X, t)
    assert abs(loss - lr) <= 4e-6 * lr
    for name, (a, b) in BLOCKS.items():
        assert np.linalg.norm(g[a:b] - gr[a:b]) <= 4e-6 * np.linalg.norm(gr[a:b]), name
