"""Cell plans of deep trees (a5g_debug_plans, no GPU needed): what a topology
upload builds on the host depends on the boxes there are, not on the columns
of the finest level."""
import time

import numpy as np
import pytest

from a5_streamer_b200 import _lib
from plan_emulator import Plans


def _chain(levels):
    """One box per level at the right end of the domain."""
    meta = np.zeros((levels + 1, 16), dtype=np.int32)
    geom = np.zeros((levels + 1, 4))
    lists = {}
    for l in range(1, levels + 1):
        n = 2 ** (l - 1)  # boxes per edge of the level
        low = -1 if l == 1 else 0
        meta[l] = [1, l, n, 1, 0, l - 1, 0, 0, 0, 0, low, -1, -1, low, 8, 0]
        if l < levels:
            meta[l, 7] = l + 1
        geom[l] = [(n - 1) / n, 0.0, 0.0, 1.0 / (8 * n)]
        lists[l] = ([l], [l] if l == levels else [], [l] if l < levels else [])
    return meta, geom, lists


def _plans(tree, levels):
    return Plans(*tree, 1, levels, 0.125)


@pytest.mark.parametrize("levels", [1, 8, 16, 23, 25, 30])
def test_plans_of_a_deep_chain(levels):
    tree = _chain(levels)
    _lib.lib()
    best = np.inf
    for _ in range(5):
        t = time.perf_counter()
        p = _plans(tree, levels)  # two builds
        best = min(best, time.perf_counter() - t)
        if best < 0.004:
            break
    assert p.bx_off[levels] == levels
    # two builds of under 2 ms each; a table over all columns of the finest
    # level doubles with every level and takes seconds at level 25
    assert best < 0.004, best
