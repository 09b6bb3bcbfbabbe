"""Layouts of different sizes alive at once: a kernel's shared-memory limit
belongs to the kernel, so a small layout made after a large one must leave the
large one's launches as they were (direct ones, and the graphs it captures
afterwards).  The same operations either way: equal bits."""
import numpy as np
import pytest

from helpers import DT, synthetic_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    from gradpower_gb300 import build, gpu
    build.build()
    return gpu


def _steps(G, gbl, c, n):
    """The calls of the large layout: the adjoint first (direct launches),
    then graphs captured anew (another tolerance, the other solvers)."""
    out = []
    for kw in (dict(newton_tol=1e-11), dict(solver=G.LY.SOLVER_SCHUR_MIXED),
               dict(solver=G.LY.SOLVER_SHARED_WOODBURY)):
        gbl.restore_initial_state()
        out.append(gbl.integrate(n * DT, DT, scenario_faults=c.faults, itermax=50, **kw))
    return out


@pytest.mark.parametrize("small", ["two_bus", "ring39"])
def test_small_layout_beside_a_large_one(G, small):
    c, _ = synthetic_case("planar2k", 6)
    b, _ = synthetic_case(small, 2)
    n = 16
    # alone
    gbl = G.GpuBatchedLayout(c.dp, c.ps, c.M)
    try:
        e0 = gbl.integrate(n * DT, DT, scenario_faults=c.faults)
        gbl.restore_initial_state()
        a0 = gbl.adjoint(n * DT, DT, scenario_faults=c.faults)
        r0 = _steps(G, gbl, c, n)
    finally:
        gbl.close()
    one = G.GpuBatchedLayout(b.dp, b.ps, b.M)
    try:
        s0 = one.integrate(n * DT, DT, scenario_faults=b.faults)
    finally:
        one.close()
    # the small one made between the large one's calls, and alive through them
    gbl = G.GpuBatchedLayout(c.dp, c.ps, c.M)
    one = None
    try:
        e1 = gbl.integrate(n * DT, DT, scenario_faults=c.faults)
        one = G.GpuBatchedLayout(b.dp, b.ps, b.M)
        gbl.restore_initial_state()
        a1 = gbl.adjoint(n * DT, DT, scenario_faults=c.faults)
        s1 = one.integrate(n * DT, DT, scenario_faults=b.faults)
        r1 = _steps(G, gbl, c, n)
    finally:
        gbl.close()
        if one is not None:
            one.close()
    for x, y in zip([e0, s0] + r0, [e1, s1] + r1):
        assert np.array_equal(x["status"], y["status"]) and np.array_equal(x["iters"], y["iters"])
        assert np.array_equal(x["traj"], y["traj"], equal_nan=True)
    for k in ("J", "grad_p"):
        assert np.array_equal(a0[k], a1[k])
