"""Cylindrical trees by the number of their different columns (the weights of
the shared-memory solve are kept per column): against the oracle, bit for bit."""
import pytest

import a5ref
from a5_streamer_b200 import config
from parity import compare, device_from_oracle

pytestmark = pytest.mark.gpu

CASES = {
    # 86 boxes: the largest kind of tree that fits shared memory
    "fits": config.batch_cylindrical_runs(n=2, photoi=False)[1],
    # columns of three base boxes on every level
    "wide": config.cylindrical_16mm(n_base=(3, 2), domain_len=(24e-3, 16e-3), lvls_max=5),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_steps_equal_the_oracle(name):
    cfg = CASES[name]
    sim = a5ref.Sim(cfg, n_threads=8)
    sim.init()
    run = device_from_oracle(sim, cfg)
    sim.op("compute_fld", 0)
    run.compute_fld(False)
    compare(sim, run, where=f"{name}: compute_fld")
    for _ in range(3):
        dt = sim.get_max_dt()
        assert run.get_max_dt() == dt
        sim.step(dt)
        run.step(dt)
    compare(sim, run, where=name)
