"""gp_adjoint with every state kept and with checkpoints: the same numbers,
bit for bit (the steps between two checkpoints are recomputed by the same
operations), on the batch kernels and on the one-CTA path, with events inside
a segment and on its border and a horizon that the checkpoints do not divide;
and the memory that a layout holds on to."""
import numpy as np
import pytest

from helpers import DT, M, synthetic_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    from gradpower_gb300 import build, gpu
    build.build()
    return gpu


@pytest.mark.parametrize("name", ["ring39", "planar2k"])
def test_checkpoints_against_all_states(G, name):
    c, _ = synthetic_case(name, 3)
    ns = 26
    faults = [[M.ContingencyEvent(3, 2.0, 5 * DT, 10 * DT)], [M.ContingencyEvent(7, 1.5, 9 * DT, 14 * DT)], []]
    kw = dict(newton_tol=1e-11, scenario_faults=faults, w_volt=10.0)
    gbl = G.GpuBatchedLayout(c.dp, c.ps, c.M)
    try:
        ref = gbl.adjoint(ns * DT, DT, checkpoint_every=7, **kw)
        zref, launches = gbl.z, gbl.timing()["launches"]
        assert np.all(ref["status"] == 0) and np.any(ref["grad_p"] != 0.0)
        gbl.set_adjoint_memory(0)
        # (checkpoints take less than 26 + 4 states for each of these)
        for every in (1, 2, 5, 7, 13):
            if -(-ns // every) + 2 * every >= ns + 4:
                continue
            gbl.restore_initial_state()
            r = gbl.adjoint(ns * DT, DT, checkpoint_every=every, **kw)
            assert gbl.timing()["launches"] > launches      # steps were recomputed
            for k in ("J", "grad_p", "grad_z0", "status"):
                assert np.array_equal(r[k], ref[k]), (every, k)
            assert np.array_equal(gbl.z, zref)
        # the limit lifted, and one that the states fit
        for limit in (None, 1 << 30):
            gbl.set_adjoint_memory(limit)
            gbl.restore_initial_state()
            r = gbl.adjoint(ns * DT, DT, checkpoint_every=7, **kw)
            assert gbl.timing()["launches"] == launches
            assert np.array_equal(r["grad_p"], ref["grad_p"])
    finally:
        gbl.close()


def test_workspace_kept_and_given_back(G):
    import torch
    c, _ = synthetic_case("planar2k", 48)
    ns = 24
    kw = dict(scenario_faults=c.faults, checkpoint_every=4)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]
    gbl = G.GpuBatchedLayout(c.dp, c.ps, c.M)
    try:
        states = ns * c.M * gbl.n_sys * 8
        gbl.set_adjoint_memory(0)
        gbl.adjoint(ns * DT, DT, **kw)
        f0 = free()
        gbl.set_adjoint_memory(None)
        gbl.adjoint(ns * DT, DT, **kw)
        assert f0 - free() >= states            # the workspace stays with the layout
        gbl.set_adjoint_memory(0)
        assert f0 - free() < states // 4        # given back
        gbl.adjoint(ns * DT, DT, **kw)
        assert f0 - free() < states // 4        # and not taken again
    finally:
        gbl.close()
