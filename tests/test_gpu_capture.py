"""A caller's stream capture of single-run calls: a replay uses what the run
holds when it is replayed (applied field, schedule, data, tree), as the same
call made then would, whichever form that call takes outside a capture."""
import numpy as np
import pytest
import torch

import a5ref
from a5_streamer_b200 import _lib, config, device
from parity import device_from_oracle

pytestmark = pytest.mark.gpu

CELLS = (0, 1, 4, 5)


def _capture(run, fn):
    s = torch.cuda.ExternalStream(run.stream_ptr())
    run.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        fn()
    return g, s


def _replay(g, s):
    with torch.cuda.stream(s):
        g.replay()


def _inner(run, sim, iv):
    """Cells of the boxes in use, without their ghost cells."""
    meta, x = sim.meta(), run.cc(iv)
    out = []
    for b in np.nonzero(meta[:, 0])[0]:
        m = meta[b, 14] + 2
        out.append(x[b, :m * m].reshape(m, m)[1:-1, 1:-1].ravel())
    return np.concatenate(out)


@pytest.mark.parametrize("solved_before", [True, False])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("what", ["step", "compute_fld"])
def test_captured_grid_mode_call(what, mixed, solved_before):
    """Grid mode on a uniform tree: captured after an ordinary solve and as
    the first call on the tree; then the applied field and the schedule
    change, and the tree is uploaded again."""
    cfg = config.cartesian_uniform(3, n_base=(3, 5), domain_len=(6e-3, 10e-3))
    sim = a5ref.Sim(cfg, n_threads=4)
    sim.init()
    run, other = device_from_oracle(sim, cfg), device_from_oracle(sim, cfg)
    run.set_ctas(min(148, run.ctas()[1]))
    dt = sim.get_max_dt()

    def call(r):
        if what == "step":
            r.step(dt)
        else:
            r.compute_fld(False)

    for r in (run, other):
        r.set_precision(mixed, (0, 2, 2, 4, 1) if mixed else None)
        if solved_before:
            r.compute_fld(False)
    g, s = _capture(run, lambda: call(run))
    for fld, sched in ((2.5e6, (0, 2, 2, 4, 1)), (3e6, (1, 1, 2, 3, 2)), (None, None)):
        if fld is None:
            for r in (run, other):
                device_from_oracle(sim, cfg, r)
        else:
            for r in (run, other):
                _lib.call("a5g_set_applied_field", r.h, fld)
                if mixed:
                    r.set_precision(True, sched)
        _replay(g, s)
        call(other)
        run.sync()
        for iv in CELLS:
            assert np.array_equal(_inner(run, sim, iv), _inner(other, sim, iv)), (fld, iv)
    # an ordinary call afterwards
    call(run)
    call(other)
    for iv in CELLS:
        assert np.array_equal(_inner(run, sim, iv), _inner(other, sim, iv)), iv
    del g


@pytest.mark.parametrize("name", ["cart", "photoi"])
def test_captured_step_batch_outlives_larger_batches(name):
    """A batch captured as the run's first (its descriptor table is made
    during the capture), then larger batches that the run leads."""
    cfg = config.cartesian_8mm() if name == "cart" else config.cylindrical_16mm(photoi=True)
    sim = a5ref.Sim(cfg, n_threads=4)
    sim.init()
    runs = [device_from_oracle(sim, cfg) for _ in range(24)]
    one = device_from_oracle(sim, cfg)
    for r in runs + [one]:
        if cfg.photoi_enabled:
            r.set_photon_table(*sim.photon_table()[:2])
            r.set_rng_state(sim.rng_state())
    dt = [sim.get_max_dt()] * len(runs)
    g, s = _capture(runs[0], lambda: device.step_batch(runs[:1], dt[:1]))
    _replay(g, s)
    for n in (2, 3, 24):
        device.step_batch(runs[:n], dt[:n])
        _replay(g, s)
    for r in runs:
        r.sync()
    for _ in range(7):  # what the first run has done
        device.step_batch([one], dt[:1])
    one.sync()
    for iv in range(device.N_VAR_CELL):
        assert np.array_equal(runs[0].cc(iv), one.cc(iv)), iv
    del g
