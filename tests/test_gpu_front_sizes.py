"""The factorisation kernels at the edges of their front sizes: the reduced
matrix of a complete graph of n buses is one dense front of 2n rows, so n
picks the kernel (warp groups up to 20 rows, four warps in registers up to
32 and 64, the CTA kernel above).  FP64 against the oracle, with identical
Newton counts and the parity tests' 1e-9; mixed (the FP32 kernels) within
their 1e-6."""
import numpy as np
import pytest

from helpers import DT, Case, run_oracle, synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    from gradpower_gb300 import build, gpu
    build.build()
    return gpu


def complete_grid(n, M_):
    rng = np.random.default_rng(n)
    edges = [(a, b) for a in range(n) for b in range(a + 1, n)]
    gens = [0] if n < 4 else [0, n // 2]
    loads = [b for b in range(n) if b not in gens]
    machines = [[synthetic._genrou(rng, b + 1, "1", (3.0, 10.0), 0.2), synthetic._tgov1(b + 1, "1"),
                 synthetic._sexs(b + 1, "1"), None] for b in gens]
    w = synthetic._build("complete", rng, n, edges, gens, loads, rng.uniform(0.02, 0.05, size=len(loads)), machines,
                         (0.0, 0.0), M_scen=M_, tf=0.2, fault_buses=rng.integers(0, n, size=M_),
                         rf_range=(1.0, 2.0), ton=0.05, toff=0.1,
                         branch_params=[(0.005 * n, 0.05 * n * x, 0.0) for x in rng.uniform(0.5, 1.5, len(edges))])
    return Case(w.ps, w.dp, w.faults, M_)


@pytest.mark.parametrize("M_", [1, 3])
@pytest.mark.parametrize("n", [3, 10, 11, 16, 17, 24, 32, 33, 40])
def test_front_sizes_match_oracle(G, orc, n, M_):
    c = complete_grid(n, M_)
    steps = 20
    o = run_oracle(orc, c, steps, itermax=30)
    assert np.all(o["status"] == 0)
    gbl = G.GpuBatchedLayout(c.dp, c.ps, M_)
    try:
        assert gbl.stats()["max_front"] == 2 * n
        r = gbl.integrate(steps * DT, DT, scenario_faults=c.faults)
        assert np.array_equal(r["status"], o["status"]) and np.array_equal(r["iters"], o["iters"])
        assert np.max(np.abs(r["traj"] - o["traj"]) / np.maximum(1.0, np.abs(o["traj"]))) < 1e-9
        gbl.restore_initial_state()
        x = gbl.integrate(steps * DT, DT, scenario_faults=c.faults, solver=G.LY.SOLVER_SCHUR_MIXED)
        assert np.all(x["status"] == 0)
        assert np.max(np.abs(x["traj"] - o["traj"]) / np.maximum(1.0, np.abs(o["traj"]))) < 1e-6
    finally:
        gbl.close()
