"""Set-up calls are done with the caller's buffers when they return, page-locked
ones and behind queued work too."""
import ctypes

import numpy as np
import pytest
import torch

import a5ref
from a5_streamer_b200 import _lib, config, device as dv
from parity import device_from_oracle

pytestmark = pytest.mark.gpu


def test_photon_table_buffer_is_the_callers_again():
    cfg = config.cylindrical_16mm(photoi=True)
    ref = a5ref.Sim(cfg, n_threads=4)
    ref.init()
    dist, frac, _ = ref.photon_table()
    runs = [device_from_oracle(ref, cfg) for _ in range(2)]
    runs[0].set_photon_table(dist, frac)
    # the other run's first table, from page-locked memory, while its stream
    # has some 15 ms of solves ahead of it
    buf = torch.from_numpy(np.array(dist)).pin_memory()
    for _ in range(50):
        runs[1].compute_fld(False)
    _lib.call("a5g_set_photon_table", runs[1].h, len(buf), 0.0, float(len(buf) - 1),
              ctypes.cast(buf.data_ptr(), ctypes.POINTER(ctypes.c_double)), frac)
    buf.mul_(0.5)
    for _ in range(50):
        runs[0].compute_fld(False)
    for r in runs:
        r.set_rng_state(ref.rng_state())
        r.photoionization(None)
        r.sync()
    a, b = (r.cc(dv.I_PHO) for r in runs)
    assert np.abs(a).sum() > 0
    assert np.array_equal(a, b)
