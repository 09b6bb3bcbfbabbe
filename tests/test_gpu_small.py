"""Small systems: the one-CTA Newton kernel against the batch kernels.

The device-driven loop of a small system runs on one CTA a scenario, the
host-driven one (gp_set_profiling) on the batch kernels; both apply the same
operations in the same order, so states, Newton counts and statuses are
equal bit for bit.  (The parity and failure tests compare the path with the
oracle.)"""
import numpy as np
import pytest

from helpers import DT, Case, M, psse_case, synthetic_case
from test_gpu_front_sizes import complete_grid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    from gradpower_gb300 import build, gpu
    build.build()
    return gpu


def _both(G, c, nsteps, **kw):
    gbl = G.GpuBatchedLayout(c.dp, c.ps, c.M)
    try:
        out = []
        for prof in (False, True):
            gbl.set_profiling(prof)
            gbl.restore_initial_state()
            r = gbl.integrate(nsteps * DT, DT, scenario_faults=c.faults, **kw)
            out.append((r, gbl.timing(), gbl.z))
    finally:
        gbl.close()
    (a, ta, za), (b, tb, zb) = out
    assert ta["launches"] < tb["launches"]      # the one-CTA path ran
    assert ta["linear_solves"] == tb["linear_solves"]
    assert np.array_equal(a["status"], b["status"]) and np.array_equal(a["iters"], b["iters"])
    assert np.array_equal(a["traj"], b["traj"], equal_nan=True)
    assert np.array_equal(za, zb, equal_nan=True)


@pytest.mark.parametrize("name,M_,nsteps", [("two_bus", 1, 70), ("ring39", 1, 20), ("ring39", 9, 30),
                                            ("ring39", 170, 16)])
def test_synthetic(G, name, M_, nsteps):
    _both(G, synthetic_case(name, M_)[0], nsteps)


@pytest.mark.parametrize("n", [1, 10, 11, 16])
def test_front_sizes(G, n):
    """Fronts up to the 32 rows a warp holds."""
    if n == 1:
        c, w = synthetic_case("two_bus", 3)
    else:
        c = complete_grid(n, 3)
    _both(G, c, 20)


def test_static_generators(G, golden_cases):
    """Algebraic states in the reduced system (PV and slack stand-ins)."""
    ps, dp = psse_case(golden_cases, "ieee9_v33.raw", "ieee9bus_gov.dyr", drop_dyr_gens=(1, 2))
    ev = [[M.ContingencyEvent(4, 0.05, 3 * DT, 6 * DT)], []]
    _both(G, Case(ps, dp, ev, 2), 15)


def test_trips_and_disconnections(G):
    c, w = synthetic_case("ring39", 4)
    br = c.ps.branches
    trips = [[M.trip_branch_event(br[k], 4 * DT, 9 * DT)] for k in (1, 5)] + [[], []]
    devs = c.ps.dynamic.devices
    exc = next(i for i, d in enumerate(devs) if d.dtype.kind == "sexs")
    zl = next(i for i, d in enumerate(devs) if d.dtype.kind == "zipload")
    disc = [[], [M.DisconnectDeviceEvent(exc, 6 * DT)], [M.DisconnectDeviceEvent(zl, 6 * DT)], []]
    c.faults = [[], [], [], [M.ContingencyEvent(3, 2.0, 2 * DT, 5 * DT)]]
    _both(G, c, 20, scenario_trips=trips, scenario_disconnects=disc)
