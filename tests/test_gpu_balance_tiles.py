"""The balance where a window of queue entries ends at the edges of its tiles
(2,048 slots, six per entry) against the oracle."""
import numpy as np
import pytest

import octree_cases as OC
from tgvreconclaude_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 341, 342, 343, 682, 683, 1024, 1365, 1366])
@pytest.mark.parametrize("seed", [0, 1, 5])
def test_balance_at_tile_edges(oracle_lib, n, seed):
    c = OC.balance_inputs(seed)
    c = c[np.sort(np.random.default_rng(n).choice(len(c), min(n, len(c)), replace=False))]
    assert api.balance_cubes(c, 2.0).tobytes() == oracle_lib.balance_cubes(c, 2.0).tobytes()
