"""The 3D form without its dense levels, which serves where they do not fit:
the box-slot solves and steps against the oracle (FP64) and against the dense
form (mixed), and what is left when one of the dense form's resources is not
to be had."""
import ctypes

import numpy as np
import pytest
import torch

from a5_streamer_b200 import _lib
from test_gpu_3d import _compare
from test_gpu_3d_dense import SHAPES, _pair

pytestmark = pytest.mark.gpu


def _info(run):
    out = (ctypes.c_int * 2)()
    _lib.call3("a5g3_debug_info", run.h, out)
    return bool(out[0]), bool(out[1])


def _slots(run):
    _lib.call3("a5g3_debug_set_dense", run.h, 0)
    assert _info(run) == (False, False)
    return run


def _same(a, b, where=""):
    for iv in range(9):
        assert np.array_equal(a.cc(iv), b.cc(iv)), (where, iv)
    for d in range(3):
        for f in range(2):
            assert np.array_equal(a.fc(d, f), b.fc(d, f)), (where, d, f)


@pytest.mark.parametrize("n_base,level", SHAPES)
def test_slot_form_against_the_oracle(n_base, level):
    """A solve from a random state, then whole steps."""
    cfg, sim, run = _pair(n_base, level, eps=False)
    assert _info(run) == (True, level > 1)
    _slots(run)
    rng = np.random.default_rng(6)
    for iv, scale in ((0, 1e15), (1, 1e15), (4, 1e3), (5, 1e6), (6, 1e8)):
        x = sim.cc(iv)
        x[:] = scale * (0.5 + rng.random(x.shape)) if iv < 2 else scale * (rng.random(x.shape) - 0.5)
        sim.set_cc(iv, x)
        run.set_cc(iv, sim.cc(iv))
    sim.op("compute_fld", 0)
    run.compute_fld(False)
    run.sync()
    _compare(sim, run, f"solve, {n_base} level {level}")
    dt = 0.1 * sim.get_max_dt()
    for _ in range(2):
        sim.step(dt)
        run.step(dt)
    run.sync()
    _compare(sim, run, f"steps, {n_base} level {level}")


@pytest.mark.parametrize("schedule", [(1, 2, 2, 8, 1), (0, 1, 1, 4, 2)])
@pytest.mark.parametrize("n_base,level", SHAPES)
def test_mixed_slot_form_equals_the_dense_form(n_base, level, schedule):
    """Cells of every box and side ghosts of the densities, potential and
    field. (The right-hand side and |E| entries of the parents that no
    operation reads are each form's own.)"""
    a, b = _pair(n_base, level)[2], _slots(_pair(n_base, level)[2])
    dt = a.get_max_dt()
    for r in (a, b):
        r.set_precision(True, schedule)
        r.compute_fld(False)
        for _ in range(2):
            r.step(dt)
        r.sync()
    meta = a.meta()
    for iv in (0, 1, 2, 3, 4, 5):
        x, y = a.cc(iv), b.cc(iv)
        for id_ in np.nonzero(meta[:, 0])[0]:
            g = meta[id_, 20] + 2
            u, v = x[id_, :g ** 3].reshape(g, g, g), y[id_, :g ** 3].reshape(g, g, g)
            assert np.array_equal(u[1:-1, 1:-1, 1:-1], v[1:-1, 1:-1, 1:-1]), (iv, id_)
    for d in range(3):
        for f in range(2):
            assert np.array_equal(a.fc(d, f), b.fc(d, f)), (d, f)


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_refused_resources_leave_the_slot_form():
    """Each resource of the dense form refused in turn: nothing of it stays
    allocated, and steps give the same values."""
    cfg, sim, run = _pair((1, 1, 1), 4, eps=False)
    ref = _pair((1, 1, 1), 4, eps=False)[2]
    dt = sim.get_max_dt()
    _slots(run)
    without = _free()
    k = 0
    while True:
        k += 1
        assert k < 32
        _lib.call3("a5g3_debug_fail_alloc", run.h, k)
        _lib.call3("a5g3_debug_set_dense", run.h, 1)
        _lib.call3("a5g3_debug_fail_alloc", run.h, 0)
        if _info(run)[0]:
            break
        assert _free() == without, k
        run.step(dt)
        ref.step(dt)
    assert k == 9  # places, arrays, five events, a stream
    assert _free() < without
    for r in (run, ref):
        r.step(dt)
        r.sync()
    _same(run, ref)


def test_mixed_form_without_room_for_the_dense_fp32_levels():
    """set_precision falls back to the box slots, and where those have no room
    either it reports that and leaves the FP64 form as it was."""
    runs = [_pair((1, 1, 1), 3, eps=False)[2] for _ in range(2)]
    a, b = runs
    dt = a.get_max_dt()
    _lib.call3("a5g3_debug_fail_alloc", a.h, 1)  # dense FP32 arrays refused
    a.set_precision(True)
    assert not _info(a)[0]
    b.set_precision(True)
    assert _info(b)[0]
    for r in runs:
        for _ in range(2):
            r.step(dt)
        r.sync()
    for iv in (0, 1, 4, 5):
        assert np.array_equal(a.cc(iv)[a.levels()[3][0]].reshape(-1, 10, 10, 10)[:, 1:-1, 1:-1, 1:-1],
                              b.cc(iv)[b.levels()[3][0]].reshape(-1, 10, 10, 10)[:, 1:-1, 1:-1, 1:-1]), iv
    c, d = (_pair((1, 1, 1), 3, eps=False)[2] for _ in range(2))
    _lib.call3("a5g3_debug_set_dense", c.h, 0)
    _lib.call3("a5g3_debug_fail_alloc", c.h, 1)  # slot FP32 arrays refused
    with pytest.raises(_lib.A5GError) as e:
        c.set_precision(True)
    assert e.value.code == _lib.A5G_ENOMEM
    assert _info(c)[0]
    for r in (c, d):
        r.step(dt)
        r.sync()
    _same(c, d)
