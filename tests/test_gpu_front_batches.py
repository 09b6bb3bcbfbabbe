"""The FP64 factorisation of a batch with more than 6,000 fronts of 21 to 32
rows (9,001 buses have 38 a scenario): a launch of a warp a front for
those, and one of their own for the few above.  A few scenarios against
the same scenarios in a batch of three, which takes the register kernel for
both: identical Newton counts, trajectories within the parity tests' 1e-9.
And the same two launches under fronts above 64 rows, against the oracle."""
import numpy as np
import pytest

from helpers import DT, Case, M, run_oracle, synthetic

pytestmark = pytest.mark.gpu


def test_large_fp64_batch_against_a_small_one():
    from gradpower_gb300 import build, gpu
    build.build()
    w = synthetic._planar("planar", 5, 9001, 900, 0.55, 1, 1.0, "random")
    M_ = 200
    rng = np.random.default_rng(3)
    fault = [[M.ContingencyEvent(int(rng.integers(9001)), float(rng.uniform(0.05, 0.2)), 2 * DT, 4 * DT)]
             for _ in range(M_)]
    pick = [0, 111, 199]
    out = []
    for c in (Case(w.ps, w.dp, fault, M_), Case(w.ps, w.dp, [fault[m] for m in pick], len(pick))):
        gbl = gpu.GpuBatchedLayout(c.dp, c.ps, c.M)
        try:
            r = gbl.integrate(6 * DT, DT, scenario_faults=c.faults)
            t = gbl.timing()
        finally:
            gbl.close()
        out.append((r, t["factor_launches"] / t["linear_solves"]))
    (a, la), (b, lb) = out
    assert la == 3.0 and lb == 2.0
    assert np.all(a["status"] == 0) and np.all(b["status"] == 0)
    assert np.array_equal(a["iters"][pick], b["iters"])
    assert np.max(np.abs(a["traj"][pick] - b["traj"]) / np.maximum(1.0, np.abs(b["traj"]))) < 1e-9


def clique_grid(M_):
    """Forty buses, each joined to each (fronts of up to 82 rows), five
    groups of 13 hanging on them (fronts of 26 to 28) and paths of two on those."""
    rng = np.random.default_rng(5)
    edges, params = [], []

    def clique(nodes):
        for i, a in enumerate(nodes):
            for b in nodes[i + 1:]:
                edges.append((a, b))
                params.append((0.005 * len(nodes), 0.05 * len(nodes) * rng.uniform(0.5, 1.5), 0.0))

    def line(a, b):
        edges.append((a, b))
        params.append((0.002, 0.02, 0.0))
    clique(list(range(40)))
    n = 40
    for g in range(5):
        clique(list(range(n, n + 13)))
        line(7 * g, n)
        line(n + 5, n + 13)
        line(n + 13, n + 14)
        n += 15
    gens = [0, 20]
    loads = [b for b in range(n) if b not in gens]
    machines = [[synthetic._genrou(rng, b + 1, "1", (3.0, 10.0), 0.2), synthetic._tgov1(b + 1, "1"),
                 synthetic._sexs(b + 1, "1"), None] for b in gens]
    w = synthetic._build("cliques", rng, n, edges, gens, loads, rng.uniform(0.01, 0.02, size=len(loads)), machines,
                         (0.0, 0.0), M_scen=M_, tf=0.2, fault_buses=rng.integers(0, n, size=M_), rf_range=(1.0, 2.0),
                         ton=0.05, toff=0.1, branch_params=params)
    return Case(w.ps, w.dp, w.faults, M_)


@pytest.mark.parametrize("M_", [3, 1300])
def test_middle_fronts_under_large_ones(orc, M_):
    """Five fronts of 26 to 28 rows a scenario: 15 of them (four warps each),
    6,500 (a warp each)."""
    from gradpower_gb300 import build, gpu
    build.build()
    c = clique_grid(M_)
    steps = 15
    gbl = gpu.GpuBatchedLayout(c.dp, c.ps, M_)
    try:
        assert gbl.stats()["max_front"] > 64
        r = gbl.integrate(steps * DT, DT, scenario_faults=c.faults)
        t = gbl.timing()
    finally:
        gbl.close()
    assert t["factor_launches"] == 3.0 * t["linear_solves"]
    pick = [0, M_ // 2, M_ - 1]
    o = run_oracle(orc, Case(c.ps, c.dp, [c.faults[m] for m in pick], 3), steps, itermax=30)
    assert np.all(o["status"] == 0)
    assert np.array_equal(r["status"][pick], o["status"]) and np.array_equal(r["iters"][pick], o["iters"])
    assert np.max(np.abs(r["traj"][pick] - o["traj"]) / np.maximum(1.0, np.abs(o["traj"]))) < 1e-9
