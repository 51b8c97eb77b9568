"""The merge at the edges of its passes: tile sizes, odd numbers of lists, empty
and unsorted lists, runs longer than a tile."""
import numpy as np
import pytest

from tgvreconclaude_gb300 import api, formats as F

pytestmark = pytest.mark.gpu
T = 2048  # outputs per block of a pass


def _want(lists):
    """Stable sort of the concatenation by code, then each run's mean in float32, in order."""
    c = np.concatenate([np.zeros(0, F.CUBE_DTYPE)] + list(lists))
    key = F.cube_keys(c)
    c = c[np.argsort(key, kind="stable")]
    if not len(c):
        return c
    new = np.ones(len(c), bool)
    new[1:] = (F.cube_keys(c)[1:] != F.cube_keys(c)[:-1]) | (c["depth"][1:] != c["depth"][:-1])
    s = np.flatnonzero(new)
    out = c[s].copy()
    for k, (a, b) in enumerate(zip(s, np.append(s[1:], len(c)))):
        t = c["r_c"][a]
        for x in c["r_c"][a + 1:b]:
            t = np.float32(t + x)
        out["r_c"][k] = np.float32(t / np.float32(b - a))
    return out


def _list(rng, n, span, sort=True):
    key = rng.integers(0, span, n).astype(np.uint64) << np.uint64(33)
    if sort:
        key = np.sort(key)
    return F.make_cubes(key, rng.integers(8, 10, n), rng.uniform(0.1, 1, n).astype(np.float32))


@pytest.mark.parametrize("sizes", [[1], [T - 1], [T], [T + 1], [1, 1], [T, T], [T - 1, 2], [0, T + 1, 0], [3 * T, 1],
                                   [1, 3 * T], [5, 0, 700, T, 1], [100] * 33, [T + 7, 900, 1, 2 * T, 31, 4 * T + 1, 8], [40, 41, 42], [1] * 40, [1] * 41, [1] * 42, [1] * 170])
@pytest.mark.parametrize("span", [1, 40, 1 << 20])
def test_merge_sizes(sizes, span):
    rng = np.random.default_rng(len(sizes) * 1000 + span)
    lists = [_list(rng, n, span) for n in sizes]
    assert api.merge_cubes(lists).tobytes() == _want(lists).tobytes()


@pytest.mark.parametrize("where", [0, 1, 2])
def test_unsorted_inputs_are_sorted(where):
    """What was taken before is taken still: a list out of order at its start, at
    a tile's edge or at its end only."""
    rng = np.random.default_rng(where)
    for at in (0, T - 1, 2 * T - 2, 3 * T - 2):
        lists = [_list(rng, 3 * T, 1 << 20) for _ in range(3)]
        c = lists[where]
        c[[at, at + 1]] = c[[at + 1, at]]
        assert api.merge_cubes(lists).tobytes() == _want(lists).tobytes()
    lists = [_list(rng, 2 * T + 5, 1 << 20, sort=False) for _ in range(where + 1)]
    assert api.merge_cubes(lists).tobytes() == _want(lists).tobytes()
