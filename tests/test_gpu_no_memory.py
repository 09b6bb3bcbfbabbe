"""A call that asks for more memory than the device has (checkpoints,
trajectories or counts of 10^6 to 2 10^9 steps) ends with that error, and the
calls after it are not told of it."""
import ctypes as C

import numpy as np
import pytest

from helpers import DT, LY, synthetic_case

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


@pytest.mark.parametrize("name,M_,steps,want_traj", [("planar2k", 6, 10 ** 6, True),
                                                     ("two_bus", 40, 2 * 10 ** 9, False)])
def test_shorter_call_after_a_buffer_could_not_grow(name, M_, steps, want_traj):
    """The trajectory buffer (550 GB asked for) or the Newton counts' (640 GB)
    fails to grow; a call that had fitted before still has its buffer."""
    from gradpower_gb300 import build, gpu
    build.build()
    c, _ = synthetic_case(name, M_)
    gbl = gpu.GpuBatchedLayout(c.dp, c.ps, c.M)
    try:
        ref = gbl.integrate(6 * DT, DT, scenario_faults=c.faults)
        fa, nf = c.fault_array(DT)
        opt = LY.GpOptions(DT, steps, 1e-10, 30, LY.SOLVER_SCHUR_FP64)
        traj = np.zeros(16)
        gbl.restore_initial_state()
        rc = gpu.library().gp_integrate(gbl._h, C.byref(opt), nf, C.addressof(fa),
                                        traj.ctypes.data if want_traj else None, None, None)
        assert rc == -3 and np.all(traj == 0.0)
        r = gbl.integrate(6 * DT, DT, scenario_faults=c.faults)
    finally:
        gbl.close()
    assert np.array_equal(r["traj"], ref["traj"]) and np.array_equal(r["iters"], ref["iters"])
