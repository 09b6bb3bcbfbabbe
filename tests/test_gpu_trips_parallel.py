"""Parallel circuits between two buses out in one scenario at once: their
off-diagonal terms fall on the same places of a front, and both have to
arrive.  A line is tripped as two circuits of half its admittance each (one
by the scenario, the other by the scenario or by every scenario), so that
the oracle's Newton counts hold only if neither is lost.  Each front size of
the FP64 factorisation, the one-CTA path and the FP32 factors; tolerances as
in the trip tests (1e-9 relative, mixed 1e-6)."""
import dataclasses

import numpy as np
import pytest

from helpers import DT, LY, M, run_oracle, synthetic_case
from test_gpu_front_sizes import complete_grid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    from gradpower_gb300 import build, gpu
    build.build()
    return gpu


def _halves(br, ton, toff=np.inf):
    t = M.trip_branch_event(br, ton, toff)
    return [dataclasses.replace(t, **{k: 0.5 * getattr(t, k) for k in ("yff", "yft", "ytf", "ytt")})] * 2


def parallel_trips(c):
    """Per scenario both circuits of a line; in every third scenario one
    circuit, whose twin trips with every scenario."""
    br = c.ps.branches
    shared = _halves(br[len(br) // 2], 3 * DT, 8 * DT)
    per = []
    for m in range(c.M):
        if m % 3 == 2:
            per.append(shared[:1])
        else:
            per.append(_halves(br[(7 * m + 3) % len(br)], 2 * DT, 6 * DT if m % 3 == 0 else np.inf))
    return per, shared[1:]


# (planar2k x 24 and x 60: the tiny fronts two and four scenarios a warp;
# complete graphs: one front of 2n rows)
@pytest.mark.parametrize("name,M_", [("ring39", 9), ("planar2k", 6), ("planar2k", 24), ("planar2k", 60),
                                     ("complete6", 3), ("complete14", 3), ("complete24", 3), ("complete40", 3)])
def test_parallel_circuits(G, orc, name, M_):
    c = complete_grid(int(name[8:]), M_) if name.startswith("complete") else synthetic_case(name, M_)[0]
    c.faults = [[] for _ in range(M_)]
    per, glob = parallel_trips(c)
    z, u, p = c.arrays()
    fa, nf = c.fault_array(DT)
    ta, nt = LY.trip_array(per, DT, glob)
    steps = 10
    o = orc.integrate(c.PA, z, u, p, fa, nf, DT, steps, solver=1, itermax=50, nthreads=8, trips=ta, n_trips=nt)
    assert np.all(o["status"] == 0)
    kw = dict(scenario_faults=c.faults, trip_events=glob, scenario_trips=per, itermax=50)
    gbl = G.GpuBatchedLayout(c.dp, c.ps, M_)
    try:
        g = gbl.integrate(steps * DT, DT, **kw)
        gbl.restore_initial_state()
        x = gbl.integrate(steps * DT, DT, solver=LY.SOLVER_SCHUR_MIXED, **kw)
    finally:
        gbl.close()
    scale = np.maximum(1.0, np.abs(o["traj"]))
    assert np.array_equal(g["status"], o["status"]) and np.array_equal(g["iters"], o["iters"])
    assert np.max(np.abs(g["traj"] - o["traj"]) / scale) <= 1e-9
    assert np.all(x["status"] == 0)
    assert np.max(np.abs(x["traj"] - o["traj"]) / scale) <= 1e-6
