"""A tree upload that fails for want of device memory, at each of its
allocations in turn: the call reports it, the run is left either with its old
tree, whole, or without a tree (calls that need one are refused), and the
next upload works as if nothing had been."""
import numpy as np
import pytest

import a5ref
from a5_streamer_b200 import _lib, config, device
from parity import compare, device_from_oracle

pytestmark = pytest.mark.gpu


def _sim(cfg):
    sim = a5ref.Sim(cfg, n_threads=4)
    sim.init()
    return sim


# (small tree, larger tree of the same problem); blocks per launch
CASES = {
    "cart": (config.cartesian_uniform(2), config.cartesian_uniform(3), 1),
    "grid": (config.cartesian_uniform(2), config.cartesian_uniform(3), 16),  # dense levels held by a captured solve
    "photoi": (config.cylindrical_16mm(photoi=True), config.batch_cylindrical_runs(n=2)[1], 1),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_failed_upload(name):
    cfg0, cfg1, n_cta = CASES[name]
    small, big = _sim(cfg0), _sim(cfg1)
    assert big.meta().shape[0] > small.meta().shape[0]
    failures, kept = 0, 0
    for k in range(1, 64):
        run = device.DeviceRun(cfg1)
        rc, xmin, inv = small.table()
        run.set_table(rc, xmin, inv)
        if cfg1.photoi_enabled:
            run.set_photon_table(*big.photon_table()[:2])
        device_from_oracle(small, cfg0, run)
        run.set_ctas(n_cta)
        run.compute_fld(False)
        before = [run.cc(iv) for iv in range(9)]
        _lib.call("a5g_debug_fail_alloc", run.h, k)
        try:
            run.upload_tree(big.meta(), big.geom(), big.min_lvl, big.max_lvl, big.levels())
            failed = False
        except _lib.A5GError as e:
            assert e.code in (_lib.A5G_ENOMEM, _lib.A5G_ECUDA)
            failed = True
        _lib.call("a5g_debug_fail_alloc", run.h, 0)
        if failed:
            failures += 1
            try:
                now = [run.cc(iv) for iv in range(9)]
            except _lib.A5GError as e:
                assert e.code == _lib.A5G_ESTATE
                for call in (lambda: run.step(1e-12), lambda: run.compute_fld(False), lambda: run.get_max_dt(),
                             lambda: device.step_batch([run], [1e-12])):
                    with pytest.raises(_lib.A5GError) as e2:
                        call()
                    assert e2.value.code == _lib.A5G_ESTATE
            else:
                kept += 1
                for a, b in zip(before, now):
                    assert np.array_equal(a, b, equal_nan=True)
                run.compute_fld(False)
        # the next upload and what follows it
        device_from_oracle(big, cfg1, run)
        ref = _sim(cfg1)
        ref.op("compute_fld", 0)
        run.compute_fld(False)
        dt = ref.get_max_dt()
        assert run.get_max_dt() == dt
        if not cfg1.photoi_enabled:
            ref.step(dt)
            run.step(dt)
        compare(ref, run, where=f"{name}, allocation {k}")
        run.close()
        if not failed:
            break
    assert not failed, "an upload with no failing allocation"
    # box storage fails with the old tree kept; lists and plans without one
    assert kept >= 7 and failures > kept
