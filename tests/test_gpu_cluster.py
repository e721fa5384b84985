"""A single run's operations on a cluster of blocks against the one-block form
(which serves where many runs are alive on the device), and step batches of
several sizes against single steps: the same bits."""
import numpy as np
import pytest
import torch

from a5_streamer_b200 import config, device, streamer

pytestmark = pytest.mark.gpu

CASES = {
    "cart": config.cartesian_8mm(),
    "cyl_photoi": config.cylindrical_16mm(photoi=True),
    "diel": config.cylindrical_16mm(epsilon_diel=3.0),
    "one_box": config.cartesian_uniform(2, n_base=(1, 1), domain_len=(2e-3, 2e-3)),
}


def _advance(run, n=4):
    run.compute_fld(False)
    for _ in range(n):
        run.step(run.get_max_dt())
    run.sync()


def _same(a, b, where):
    for iv in range(device.N_VAR_CELL):
        assert np.array_equal(a.cc(iv), b.cc(iv), equal_nan=True), f"{where}: cell variable {iv}"
    for d in range(2):
        for f in range(device.N_VAR_FACE):
            assert np.array_equal(a.fc(d, f), b.fc(d, f)), f"{where}: face {d} {f}"


# (the mixed form refuses dielectric runs)
@pytest.mark.parametrize("name,mixed", [(n, m) for n in sorted(CASES) for m in (False, True) if n != "diel" or not m])
def test_cluster_equals_one_block(name, mixed):
    cfg = CASES[name]
    sim = streamer.Simulation(cfg)
    sim.init()
    a = device.clone_state(sim, mixed)
    b = device.clone_state(sim, mixed)
    _advance(a)
    n = torch.cuda.get_device_properties(0).multi_processor_count // 8 + 1
    crowd = [device.DeviceRun(cfg) for _ in range(n)]
    _advance(b)
    _same(a, b, name)
    del crowd


def test_step_batch_sizes():
    """Batches that grow, shrink and change their first run, beyond one
    descriptor launch; between them single steps."""
    sim = streamer.Simulation(CASES["one_box"])
    sim.init()
    one = device.clone_state(sim)
    runs = [device.clone_state(sim) for _ in range(98)]
    dt = one.get_max_dt()
    for n, first in ((2, 0), (98, 0), (3, 1), (97, 1)):
        group = runs[first:first + n]
        device.step_batch(group, [dt] * n)
    done = [(k < 2) + 1 + (1 <= k < 4) + (1 <= k < 98) for k in range(98)]
    ref = {}
    for k in range(1, max(done) + 1):
        one.step(dt)
        one.sync()
        ref[k] = [one.cc(iv) for iv in range(device.N_VAR_CELL)]
    for k, r in enumerate(runs):
        r.sync()
        for iv in range(device.N_VAR_CELL):
            assert np.array_equal(r.cc(iv), ref[done[k]][iv]), (k, iv)
