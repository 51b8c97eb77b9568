"""A NaN bias is NaN whatever its payload: zero behind a ReLU, NaN as the output's."""
import numpy as np
import pytest

import mlp_ref
from tgvreconclaude_gb300 import warmstart as WS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [0x7fc00000, 0x7f800001, 0x7f80ffff, 0xff800001, 0xffc12345])
def test_nan_biases(bits):
    m = WS.WarmStartMLP(10, seed=5)
    for at in ("P_B1", "P_B2", "P_B3"):
        p = np.zeros(mlp_ref.P_N, np.float32)
        p[mlp_ref.P_W2:mlp_ref.P_B2:65] = 1.0  # each unit of layer 1 to its own of layer 2
        p[mlp_ref.P_W3] = 1.0
        p.view(np.uint32)[getattr(mlp_ref, at)] = bits
        m.set_params(p)
        y = m.predict(np.zeros((130, 16), np.uint16))
        assert np.isnan(y).all() if at == "P_B3" else np.all(y == 0), at
