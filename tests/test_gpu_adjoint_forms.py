"""The adjoint's two forms of the multigrid's transpose: in gather form with
its vector in shared memory, and by the tape where a tree is too large for
that. Each against the oracle's tangent-linear run, within the 1e-6 relative
that the 8 mm problem is held to."""
import numpy as np
import pytest

import a5ref
from a5_streamer_b200 import adjoint, config, streamer

pytestmark = pytest.mark.gpu

# boxes of the trees: 48 (gather), 112 (gather, nearly all of shared memory), 368 (tape)
CASES = [(1, (4, 4)), (2, (4, 4)), (3, (4, 4))]


@pytest.mark.parametrize("level,n_base", CASES)
def test_gradient_matches_the_oracle_tangent(level, n_base):
    cfg = config.cartesian_uniform(level, n_base=n_base, domain_len=tuple(2e-3 * n for n in n_base))
    prob = adjoint.HeadProblem(n_steps=5, checkpoint_every=3)
    sim = streamer.Simulation(cfg)
    sim.init()
    ref = a5ref.Sim(cfg, n_threads=8)
    ref.init()
    adj = adjoint.HeadAdjoint(sim, prob)
    p = prob.nominal()
    dts, T = adj.schedule()
    adj.bind()
    try:
        J, g = adj.gradient(p)
        _, again = adj.gradient(p)
    finally:
        adj.close()
    d, dV = adjoint.param_tangents(p, cfg.domain_len_z, cfg.lkptbl_size, cfg.lkptbl_max_fld)
    J_ref, g_ref = ref.tl_program(dts, prob.x0, T, d, dV)
    assert J == J_ref
    np.testing.assert_allclose(g, g_ref, rtol=1e-6, atol=0)
    np.testing.assert_allclose(again, g, rtol=1e-9, atol=0)
