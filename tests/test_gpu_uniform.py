"""The dense field solve of uniformly refined Cartesian runs in grid mode
(a5g_uniform.cu) against the oracle and against the box phases, bit for bit,
on base grids and levels where its pieces change."""
import numpy as np
import pytest

import a5ref
from a5_streamer_b200 import config
from parity import compare, device_from_oracle

pytestmark = pytest.mark.gpu

# n_base, level: one base box; odd counts (rows of odd length on the coarsest
# level); level 2 of 4 x 4 the largest one-block level; 9 x 9 with level 1 above
# a section of level 0, 33 x 32 (4,224 cells on the coarsest level) without one
SHAPES = [((1, 1), 2), ((4, 4), 2), ((4, 4), 3), ((3, 5), 3), ((9, 9), 2), ((1, 6), 4), ((33, 32), 2)]


def _cfg(n_base, level):
    return config.cartesian_uniform(level, n_base=n_base, domain_len=tuple(2e-3 * n for n in n_base))


def _pair(n_base, level, n_cta=148):
    cfg = _cfg(n_base, level)
    sim = a5ref.Sim(cfg, n_threads=8)
    sim.init()
    run = device_from_oracle(sim, cfg)
    run.set_ctas(min(n_cta, run.ctas()[1]))
    return cfg, sim, run


@pytest.mark.parametrize("n_base,level", SHAPES)
def test_steps_and_solve_parity(n_base, level):
    cfg, sim, run = _pair(n_base, level)
    rng = np.random.default_rng(5)
    for iv, scale in ((0, 1e15), (1, 1e15), (4, 1e3)):
        x = scale * (rng.random(sim.cc(iv).shape) - 0.5)
        sim.set_cc(iv, x)
        run.set_cc(iv, x)
    sim.op("compute_fld", 0)
    run.compute_fld(False)
    compare(sim, run, where="solve from a random state")
    sim = a5ref.Sim(cfg, n_threads=8)
    sim.init()
    device_from_oracle(sim, cfg, run)
    run.set_ctas(min(148, run.ctas()[1]))
    for k in range(3):
        dt = sim.get_max_dt()
        assert run.get_max_dt() == dt
        sim.step(dt)
        run.step(dt)
    compare(sim, run, where=f"{n_base} level {level}")


@pytest.mark.parametrize("n_base,level", SHAPES)
@pytest.mark.parametrize("schedule", [None, (0, 1, 1, 2, 2), (1, 3, 1, 5, 1)])
def test_mixed_equals_box_phases(n_base, level, schedule):
    cfg, sim, a = _pair(n_base, level)
    b = device_from_oracle(sim, cfg)  # one block: the box phases
    for r in (a, b):
        r.set_precision(True, schedule)
    dt = sim.get_max_dt()
    for _ in range(2):
        a.step(dt)
        b.step(dt)
    a.compute_fld(False)
    b.compute_fld(False)
    for iv in range(8):
        x, y = a.cc(iv), b.cc(iv)
        g = x.reshape(len(x), -1)
        n = sim.meta()[:, 14]
        for id_ in np.nonzero(sim.meta()[:, 0])[0]:
            m = n[id_] + 2
            u, v = g[id_, :m * m].reshape(m, m), y[id_, :m * m].reshape(m, m)
            assert np.array_equal(u[1:-1, 1:-1], v[1:-1, 1:-1]), (iv, id_)
            if iv in (0, 1, 4, 5):
                assert np.array_equal(u[1:-1], v[1:-1]) and np.array_equal(u[:, 1:-1], v[:, 1:-1]), (iv, id_)


def test_settings_reach_a_captured_solve():
    """Applied field, schedule and precision changed between solves."""
    cfg, sim, run = _pair((3, 5), 3)
    other = device_from_oracle(sim, cfg)
    for fld, mixed, sched in ((2.5e6, False, None), (3e6, False, None), (3e6, True, None), (1e6, True, (0, 2, 1, 3, 1)),
                              (1e6, False, None)):
        for r in (run, other):
            r.set_precision(mixed, sched)
            from a5_streamer_b200._lib import call
            call("a5g_set_applied_field", r.h, fld)
            r.compute_fld(False)
        assert np.array_equal(run.cc(4)[:, 11:89], other.cc(4)[:, 11:89]), (fld, mixed)
