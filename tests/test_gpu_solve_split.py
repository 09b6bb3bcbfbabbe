"""The triangular solves' split of the assembly tree by batch size: blocks of
256 to 2048 factor entries, top supernodes on CTAs alone (few scenarios) or on
warps below and CTAs above (many).  Mixed solves (FP32 factors, both passes)
within the mixed path's 1e-6 of the FP64 ones on the same scenarios, which a
batch of two reproduces."""
import numpy as np
import pytest

from helpers import DT, Case, synthetic_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    from gradpower_gb300 import build, gpu
    build.build()
    return gpu


@pytest.mark.parametrize("M_", [5, 40, 97, 258])
def test_batch_sizes(G, M_):
    c, w = synthetic_case("planar2k", M_)
    steps = 14
    gbl = G.GpuBatchedLayout(c.dp, c.ps, c.M)
    try:
        e = gbl.integrate(steps * DT, DT, scenario_faults=c.faults)
        gbl.restore_initial_state()
        x = gbl.integrate(steps * DT, DT, scenario_faults=c.faults, solver=G.LY.SOLVER_SCHUR_MIXED)
    finally:
        gbl.close()
    assert np.all(e["status"] == 0) and np.all(x["status"] == 0)
    assert np.max(np.abs(x["traj"] - e["traj"]) / np.maximum(1.0, np.abs(e["traj"]))) < 1e-6
    s = Case(w.ps, w.dp, c.faults[:2], 2)
    gbl = G.GpuBatchedLayout(s.dp, s.ps, 2)
    try:
        b = gbl.integrate(steps * DT, DT, scenario_faults=s.faults)
    finally:
        gbl.close()
    assert np.array_equal(e["iters"][:2], b["iters"])
    assert np.max(np.abs(e["traj"][:2] - b["traj"])) < 1e-9
