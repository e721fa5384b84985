"""Which form of the device code a call takes, and that the comparisons between
forms compare two: the cluster against one block, the dense solves against
the box phases, the adjoint's gather form against its tape."""
import ctypes
import gc

import numpy as np
import pytest
import torch

import a5ref
from a5_streamer_b200 import _lib, adjoint, config, device, streamer
from parity import compare, device_from_oracle

pytestmark = pytest.mark.gpu

BLOCK, CLUSTER, GROUP, DENSE = 1, 2, 3, 4
GATHER, TAPE = 1, 2


def _form(run):
    out = ctypes.c_int(0)
    _lib.call("a5g_debug_form", run.h, ctypes.byref(out))
    return out.value


def _equal(a, b, ivs, where):
    for iv in ivs:
        assert np.array_equal(a.cc(iv), b.cc(iv), equal_nan=True), (where, iv)


WIDE = dict(n_base=(12, 12), domain_len=(96e-3, 96e-3), lvls_max=6)
# configuration, precision; form of a step and a solve on an otherwise empty device
CLUSTERS = {
    "cart": (config.cartesian_8mm(), False),  # 96 boxes, solves in shared memory
    "cart_mixed": (config.cartesian_8mm(), True),
    "cyl_photoi": (config.cylindrical_16mm(photoi=True), False),  # 54
    "wide": (config.cylindrical_16mm(**WIDE), False),  # 484, in device memory
    "wide_mixed": (config.cylindrical_16mm(**WIDE), True),
    "wide_diel": (config.cylindrical_16mm(epsilon_diel=3.0, **WIDE), False),
}


@pytest.mark.parametrize("name", sorted(CLUSTERS))
def test_cluster_and_one_block(name):
    cfg, mixed = CLUSTERS[name]
    gc.collect()  # runs that earlier tests have dropped
    sim = streamer.Simulation(cfg)
    sim.init()
    a, b = device.clone_state(sim, mixed), device.clone_state(sim, mixed)
    crowd = []

    def advance(run, form):
        run.compute_fld(False)
        assert _form(run) == form
        for _ in range(3):
            run.step(run.get_max_dt())
            assert _form(run) == form
        run.compute_fld(True)
        assert _form(run) == form
        run.photoionization(1e-12) if cfg.photoi_enabled else run.gc_tree(0)
        run.sync()

    advance(a, CLUSTER)
    n = torch.cuda.get_device_properties(0).multi_processor_count // 8 + 1
    crowd = [device.DeviceRun(cfg) for _ in range(n)]
    advance(b, BLOCK)
    _equal(a, b, range(9), name)
    del crowd


def test_cluster_rule():
    """Forms by tree and operation on an otherwise empty device: few boxes, or
    few boxes a level where the phases go through device memory, take one
    block."""
    gc.collect()

    def forms(cfg, mixed=False):
        sim = streamer.Simulation(cfg)
        sim.init()
        r = device.clone_state(sim, mixed)
        out = []
        for f in (lambda: r.step(1e-15), lambda: r.compute_fld(False), lambda: r.fluxes_koren(1e-15),
                  lambda: r.gc_tree(0), lambda: r.restrict_tree(0), r.dt_reductions):
            f()
            out.append("-BC"[_form(r)])
        return "".join(out)

    uni = lambda level, n: config.cartesian_uniform(level, n_base=n, domain_len=tuple(2e-3 * k for k in n))
    # step, solve, fluxes, ghost cells, restriction, reductions
    assert forms(uni(2, (1, 1))) == "BBBBBB"  # 7 boxes
    assert forms(config.cylindrical_16mm()) == "CCCBBB"  # 54
    assert forms(config.cylindrical_16mm(), True) == "BBCBBB"
    assert forms(config.cartesian_8mm()) == "CCCBBB"  # 96
    assert forms(config.cartesian_8mm(), True) == "CCCBBB"
    assert forms(config.cylindrical_16mm(epsilon_diel=3.0)) == "BBCBBB"  # dielectric: solves in device memory
    assert forms(uni(2, (4, 4))) == "BBCBBB"  # 112: beyond shared memory in FP64, not in FP32
    assert forms(uni(2, (4, 4)), True) == "CCCBBB"
    assert forms(uni(2, (6, 6))) == "CCCCBB"  # 63 a level
    assert forms(uni(3, (4, 4))) == "CCCCCC"  # 73


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n_base,level", [((1, 1), 2), ((3, 5), 3), ((4, 4), 3)])
def test_dense_and_box_phases(n_base, level, mixed):
    cfg = config.cartesian_uniform(level, n_base=n_base, domain_len=tuple(2e-3 * n for n in n_base))
    sim = a5ref.Sim(cfg, n_threads=4)
    sim.init()
    a, b = device_from_oracle(sim, cfg), device_from_oracle(sim, cfg)
    a.set_ctas(min(148, a.ctas()[1]))
    for r in (a, b):
        r.set_precision(mixed)
    dt = sim.get_max_dt()
    for _ in range(2):
        a.step(dt)
        b.step(dt)
        a.compute_fld(False)
        b.compute_fld(False)
        assert _form(a) == DENSE and _form(b) in (BLOCK, CLUSTER)
    for iv in (0, 1, 4, 5):
        x, y = a.cc(iv).reshape(-1, 10, 10)[1:], b.cc(iv).reshape(-1, 10, 10)[1:]
        fine = sim.meta()[1:, 14] == 8
        assert np.array_equal(x[fine][:, 1:-1, 1:-1], y[fine][:, 1:-1, 1:-1]), iv
    a.compute_fld(True)  # a first solve
    assert _form(a) == GROUP


def test_runs_that_keep_the_box_phases():
    """Grid mode on what the dense levels do not cover."""
    def run_of(cfg):
        sim = a5ref.Sim(cfg, n_threads=4)
        sim.init()
        r = device_from_oracle(sim, cfg)
        r.set_ctas(16)
        return sim, r

    for cfg in (config.cartesian_8mm(), config.cylindrical_16mm()):  # refinement boundaries, axisymmetric
        sim, r = run_of(cfg)
        r.compute_fld(False)
        assert _form(r) == GROUP
    cfg = config.cartesian_uniform(2)
    sim, r = run_of(cfg)
    r.compute_fld(False)
    assert _form(r) == DENSE
    lsf = np.ones_like(r.cc(4))
    r.set_level_set(lsf, np.zeros_like(lsf))
    r.compute_fld(False)
    assert _form(r) == GROUP
    r.set_level_set(None, None)
    eps = r.cc(8)
    eps[:, 55] = 2.0
    r.set_cc(8, eps)
    r.compute_fld(False)
    assert _form(r) == GROUP
    eps[:, 55] = 1.0
    r.set_cc(8, eps)
    r.compute_fld(False)
    assert _form(r) == DENSE


def test_barrier_timeout_on_dense_levels():
    """A step whose transport runs out of its barrier budget reports it,
    although its solves are launches of their own; the run works again after."""
    cfg = config.cartesian_uniform(3)
    sim = a5ref.Sim(cfg, n_threads=4)
    sim.init()
    run = device_from_oracle(sim, cfg)
    run.set_ctas(4, 0)
    dt = sim.get_max_dt()
    run.step(dt)
    with pytest.raises(_lib.A5GError) as e:
        run.sync()
    assert e.value.code == _lib.A5G_TIMEOUT
    run.set_ctas(4)
    device_from_oracle(sim, cfg, run)
    sim.step(dt)
    run.step(dt)
    assert _form(run) == DENSE
    compare(sim, run, where="after a timeout")


# boxes of the trees: 48 (gather), 112 (gather, nearly all of shared memory), 368 (tape)
@pytest.mark.parametrize("level,form", [(1, GATHER), (2, GATHER), (3, TAPE)])
def test_adjoint_form(level, form):
    cfg = config.cartesian_uniform(level, n_base=(4, 4), domain_len=(8e-3, 8e-3))
    sim = streamer.Simulation(cfg)
    sim.init()
    adj = adjoint.HeadAdjoint(sim, adjoint.HeadProblem(n_steps=2, checkpoint_every=2))
    adj.schedule()
    adj.bind()
    try:
        out = ctypes.c_int(0)
        _lib.call("a5a_debug_form", adj.h, ctypes.byref(out))
        assert out.value == form
    finally:
        adj.close()
