"""The bytes the fused 3D step must move, on a uniform octree's census."""
from a5_streamer_b200 import metrics


def _census(level, n_base=1):
    cells, leaf, par = {}, {}, {}
    for l in range(-1, level + 1):
        edge = 8 * 2 ** (l - 1) if l >= 1 else 8 >> (1 - l)
        cells[l] = n_base * edge ** 3
        leaf[l] = cells[l] if l == level else 0
        par[l] = 0 if l == level else cells[l]
    return metrics.Census(3, 8, -1, level, cells, leaf, par)


def test_level_6_cube():
    c = _census(6)
    leaf = 64 ** 3 * 64
    assert c.n_leaf == leaf == 16777216
    moved = metrics.moved_bytes_per_step_3d(c) / 8 / leaf
    # by hand: 37 + 28 (1/8 + ... + 8^-5 = 1/7) for the transport; two solves,
    # each with the finest level visited once (restriction 2.375, correction
    # 1.375, 12 of half-sweeps, restriction 2.375, correction 1.375) and the
    # next ones 2, 3, ... times at 1/8, 1/64, ...
    finest = 2.375 + 2 * 1.375 + 12 + 2.375
    assert 37 + 28 / 7 + 2 * finest < moved < 37 + 28 / 7 + 2 * finest * (1 + 2.4 / 8 + 3.6 / 64 + 0.02)
    assert moved * 8 < metrics.bytes_per_step(c) / leaf  # the reference's operations move more


def test_cost_is_linear_in_the_boxes():
    a, b = (metrics.moved_bytes_per_step_3d(_census(4, n)) for n in (1, 6))
    assert abs(b - 6 * a) < 1e-6 * b
