"""A call that asks for more memory than the device has (the checkpoints of
10^9 steps) ends with that error, and the calls after it are not told of it."""
import numpy as np
import pytest

from helpers import DT, synthetic_case

pytestmark = pytest.mark.gpu


def test_call_after_a_failed_allocation():
    from gradpower_gb300 import build, gpu
    build.build()
    c, _ = synthetic_case("planar2k", 6)
    gbl = gpu.GpuBatchedLayout(c.dp, c.ps, c.M)
    try:
        ref = gbl.adjoint(8 * DT, DT, scenario_faults=c.faults)
        gbl.restore_initial_state()
        for again in range(2):
            with pytest.raises(gpu.GradPowerError, match="cudaMalloc of"):
                gbl.adjoint(10 ** 9 * DT, DT, scenario_faults=c.faults, checkpoint_every=60)
            r = gbl.adjoint(8 * DT, DT, scenario_faults=c.faults)
            assert np.array_equal(r["grad_p"], ref["grad_p"]) and np.array_equal(r["J"], ref["J"])
            gbl.restore_initial_state()
            with pytest.raises(gpu.GradPowerError, match="cudaMalloc of"):
                gbl.adjoint(10 ** 9 * DT, DT, scenario_faults=c.faults, checkpoint_every=60)
            assert np.all(gbl.integrate(4 * DT, DT, scenario_faults=c.faults, want_traj=False)["status"] == 0)
            gbl.restore_initial_state()
    finally:
        gbl.close()
