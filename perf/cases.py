"""What this framework is measured by: batches of fault scenarios on power
grids, integrated (or differentiated) through the package's public entry
points.

A case is a grid, a number of scenarios, a horizon and one of the ways a
user runs it:

  fp64      GpuBatchedLayout.integrate, the exact FP64 Newton step
  mixed     the same call with the mixed-precision solver
  shared    integrate_gpu_shared_multi (one shared factorisation)
  adjoint   GpuBatchedLayout.adjoint (objective and gradients)

The grids are this repository's synthetic workloads (two_bus, ring39 and
planar2k .. planar70k) and planar grids of other sizes by the same recipe.
They play the part of the utility's network model: fixed, built once per
process.  What a seed changes is what a study changes from batch to batch:
which bus is faulted and how hard, and the machines' inertia and damping.

`exact` integrates the same equations in 64 bits with plain torch: its own
restatement of the device equations, Jacobian blocks by forward-mode
differentiation, a dense Schur complement on the buses, Newton iterations to
rounding level.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DT = 1.0 / 120.0


def _package():
    if "gradpower_gb300" not in sys.modules:
        pkg = os.path.join(ROOT, "gradpower.jl_gb300")
        spec = importlib.util.spec_from_file_location("gradpower_gb300", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["gradpower_gb300"] = mod
        spec.loader.exec_module(mod)
    from gradpower_gb300 import gpu, layout, model, synthetic
    return gpu, layout, model, synthetic


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _case(name, kind, grid, buses, machines, scenarios, steps, trips=False, traj="none", grid_seed=0):
    """traj: what the call brings back besides the final state: "none",
    "host" (a new array per call) or "pinned" (the user's page-locked
    buffer)."""
    c = dict(name=name, kind=kind, grid=grid, buses=buses, machines=machines, scenarios=scenarios, steps=steps,
             trips=trips, traj=traj, grid_seed=grid_seed)
    return {k: v for k, v in c.items() if not (k == "name" and v is None)}


def listed():
    return [
        # one contingency on the two-bus teaching case: every launch counts
        _case("fp64_2bus_x1", "fp64", "two_bus", 2, 1, 1, 60, traj="host"),
        # N-1 screening of a 39-bus system: 64 faults, a second each, the
        # trajectories kept (the benchmark's ring39 x 64)
        _case("fp64_39bus_x64", "fp64", "ring39", 39, 10, 64, 120, traj="host"),
        # a planner's batch on a 2,000-bus region, exact solver, the
        # trajectories streamed into page-locked memory
        _case("fp64_2kbus_x64", "fp64", "planar", 2000, 400, 64, 30, traj="pinned", grid_seed=2),
        # the benchmark's planar2k x 256 batch, mixed solver, the state at
        # the end of the window
        _case("mixed_2kbus_x256", "mixed", "planar", 2000, 400, 256, 30, grid_seed=2),
        # a handful of scenarios: faults cleared by tripping a line that
        # recloses, trajectories kept
        _case("mixed_2kbus_x7_trips", "mixed", "planar", 2000, 400, 7, 30, trips=True, traj="host", grid_seed=2),
        # the shared-factor integrator on the same region
        _case("shared_2kbus_x32", "shared", "planar", 2000, 400, 32, 24, grid_seed=2),
        # gradients of the speed and voltage objective for tuning, with
        # checkpoints as in the differentiation benchmark (every 60 steps at
        # most; here twice over the window)
        _case("adjoint_2kbus_x24", "adjoint", "planar", 2000, 400, 24, 24, grid_seed=2),
        # an odd-sized grid and batch between the benchmark's two sizes
        _case("mixed_9kbus_x5", "mixed", "planar", 9001, 900, 5, 30, grid_seed=5),
        _case("fp64_9kbus_x3", "fp64", "planar", 9001, 900, 3, 24, grid_seed=5),
        # the headline workload, planar70k x 8: a window that holds a fault
        # and its clearing, both solvers
        _case("mixed_70kbus_x8", "mixed", "planar", 70000, 5000, 8, 36, grid_seed=4),
        _case("fp64_70kbus_x8", "fp64", "planar", 70000, 5000, 8, 18, grid_seed=4),
    ]


def draw(rng):
    kind = rng.choice(["fp64", "fp64", "mixed", "mixed", "shared", "adjoint"])
    if kind in ("fp64", "adjoint") and rng.random() < 0.4:
        # small systems
        if rng.random() < 0.35:
            M, steps = int(round(2.0 ** rng.uniform(0, 6))), rng.randint(24, 120)
            return _case(None, kind, "two_bus", 2, 1, M, steps, traj=rng.choice(["none", "host"]))
        M, steps = int(round(2.0 ** rng.uniform(0, 7.5))), rng.randint(24, 120)
        return _case(None, kind, "ring39", 39, 10, M, steps, traj=rng.choice(["none", "host"]))
    # planar grids: 300 to 12,000 buses, a machine on every 5th to 14th
    buses = int(round(10.0 ** rng.uniform(math.log10(300), math.log10(12000))))
    machines = max(8, int(buses * rng.uniform(0.07, 0.2)))
    # the batch: up to 256 scenarios, less work than the largest listed case
    most = min(256.0, (400e3 if kind == "mixed" else 120e3) / buses)
    M = max(1, int(round(most ** rng.uniform(0.0, 1.0))))
    steps = rng.randint(18, 36)
    trips = kind in ("fp64", "mixed") and rng.random() < 0.3
    traj = "none" if kind == "adjoint" else rng.choice(["none", "none", "pinned", "host"])
    return _case(None, kind, "planar", buses, machines, M, steps, trips=trips, traj=traj,
                 grid_seed=rng.randint(3, 10 ** 6))


# ---------------------------------------------------------------------------
# what the user has in hand
# ---------------------------------------------------------------------------

_GRIDS = {}     # the last grids built, a few at most


def _grid(case):
    """(ps, dp, fault buses to choose from) of a case's network."""
    key = (case["grid"], case["buses"], case["machines"], case["grid_seed"])
    if key not in _GRIDS:
        S = _package()[3]
        if case["grid"] == "two_bus":
            w = S.two_bus()
            buses = [1]
        elif case["grid"] == "ring39":
            w = S.ring39()
            buses = list(range(39))
        else:
            w = S._planar("planar", case["grid_seed"], case["buses"], case["machines"], 0.55, 1, 1.0, "random")
            buses = list(range(case["buses"]))
        while len(_GRIDS) >= 4:
            _GRIDS.pop(next(iter(_GRIDS)))
        _GRIDS[key] = (w.ps, w.dp, buses)
    return _GRIDS[key]


def _inputs(case, seed):
    """The study: per scenario a bus fault (or, with trips, a fault cleared
    by tripping a line beside it, which recloses), and the machines' inertia
    and damping, drawn from the seed."""
    _, LY, Mdl, _ = _package()
    ps, dp, buses = _grid(case)
    rng = np.random.default_rng([int(seed), 77])
    M, steps = case["scenarios"], case["steps"]
    # fault on a third of the way in, off a third later (12 steps, 0.1 s, at
    # most, the benchmark's fault)
    on = max(1, min(12, steps // 3))
    off = min(2 * on, on + 12)
    # resistances as the workloads draw them; on the 39-bus ring, where
    # harder faults drive some buses into voltage collapse (no solution to
    # compare), high-impedance ones
    lo, hi = (1.2, 2.5) if case["grid"] == "ring39" else (0.05, 0.2)
    fb = rng.choice(buses, size=M, replace=M > len(buses))
    rf = rng.uniform(lo, hi, size=M)
    faults, trips = [], None
    for m in range(M):
        faults.append([Mdl.ContingencyEvent(int(fb[m]), float(rf[m]), on * DT, off * DT)])
    if case["trips"]:
        # lines on cycles only (their trip leaves the grid connected)
        lines = _cycle_lines(ps)
        trips = [[Mdl.trip_branch_event(ps.branches[int(rng.choice(lines))], off * DT, min(steps - 1, off + 6) * DT)]
                 for _ in range(M)]
    p = np.tile(dp.pvec, (M, 1))
    T = LY.ProblemArrays(ps).tables[LY.GP_GENROU]
    p[:, T.par_ptr + 6] *= rng.uniform(0.85, 1.15, size=(M, T.n))
    p[:, T.par_ptr + 7] = rng.uniform(0.0, 2.0, size=(M, T.n))
    return dict(ps=ps, dp=dp, faults=faults, trips=trips, p=p, fb=fb, rf=rf, on=on, off=off)


def _cycle_lines(ps):
    """Branches off the first spanning tree found: tripping one keeps the
    grid connected."""
    parent = list(range(ps.nbus))

    def find(a):
        while parent[a] != a:
            parent[a] = parent[parent[a]]
            a = parent[a]
        return a

    out = []
    for k, br in enumerate(ps.branches):
        a, b = find(br.fr), find(br.to)
        if a == b:
            out.append(k)
        else:
            parent[a] = b
    return out


def prepare(case, seed):
    G, LY, _, _ = _package()
    s = _inputs(case, seed)
    s["case"] = case
    s["gbl"] = G.GpuBatchedLayout(s["dp"], s["ps"], case["scenarios"], p=s["p"])
    s["buf"] = None
    if case["traj"] == "pinned":
        s["buf"] = torch.empty((case["scenarios"], case["steps"] + 1, s["gbl"].n_sys), dtype=torch.float64,
                               pin_memory=True).numpy()
    return s


def run(s):
    G, LY, _, _ = _package()
    case, gbl = s["case"], s["gbl"]
    tf = case["steps"] * DT
    gbl.restore_initial_state()
    kind = case["kind"]
    if kind == "shared":
        # (returns the trajectories whether wanted or not, as the reference's)
        _, trajs = G.integrate_gpu_shared_multi(gbl, s["ps"], tf, s["fb"], s["rf"], s["on"] * DT, s["off"] * DT)
        return {"traj": np.stack([t[:, -1] for t in trajs]) if case["traj"] == "none"
                else np.stack(trajs).transpose(0, 2, 1)}
    if kind == "adjoint":
        r = gbl.adjoint(tf, DT, scenario_faults=s["faults"], w_speed=1.0, w_volt=10.0, v_min=0.9,
                        checkpoint_every=max(1, min(60, case["steps"] // 2)))
        return {"J": r["J"], "grad_p": r["grad_p"], "grad_z0": r["grad_z0"], "status": r["status"]}
    r = gbl.integrate(tf, DT, scenario_faults=s["faults"], scenario_trips=s["trips"],
                      want_traj=case["traj"] != "none", traj_out=s["buf"],
                      solver=LY.SOLVER_SCHUR_MIXED if kind == "mixed" else LY.SOLVER_SCHUR_FP64)
    out = {"status": r["status"], "traj": r["traj"] if case["traj"] != "none" else gbl.z}
    if kind == "fp64":
        # Newton counts are part of the exact solver's contract (the
        # reference's); the mixed solver's depend on the rounding of its
        # FP32 factors and are a diagnostic there
        out["iters"] = r["iters"]
    return out


def work(case):
    """Bytes: the scenarios' states and parameters and the network read
    once, the outputs written once.  Operations: per scenario and step one
    evaluation of every device and bus and one solve with factors at hand
    (nnz(L + U) is about 18 per reduced unknown on these grids); an adjoint
    adds a transposed solve."""
    nb, ng, M, steps = case["buses"], case["machines"], case["scenarios"], case["steps"]
    n_sys = 2 * nb + 19 * ng
    n_par = 9 * int(0.6 * nb) + 35 * ng
    out = n_sys * (steps + 1 if case["traj"] != "none" else 1)
    if case["kind"] == "adjoint":
        out = n_sys + n_par
    by = 8.0 * M * (n_sys + n_par + out) + 16.0 * 4 * nb
    per = 60.0 * nb + 600.0 * ng + 2.0 * 18 * 2 * nb
    return {"bytes": by, "flops": M * steps * per * (2.0 if case["kind"] == "adjoint" else 1.0)}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------

def exact(case, seed):
    # dense (2 buses)^2 matrices per scenario: the small and middle sizes
    nb, M = case["buses"], case["scenarios"]
    solves = 2 if case["kind"] == "adjoint" else 1
    if nb > 2100 or M * float(nb) ** 3 * solves > 64 * 2000.0 ** 3:
        return None
    s = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return _Exact(case, s, dev).run()


class _Exact:
    def __init__(self, case, s, dev):
        LY = _package()[1]
        self.case, self.s, self.dev = case, s, dev
        A = LY.ProblemArrays(s["ps"])
        M = case["scenarios"]
        t = lambda a, dt=torch.float64: torch.as_tensor(np.asarray(a).copy(), dtype=dt, device=dev)  # noqa: E731
        i64 = torch.int64
        self.M, self.nb, self.net, self.n = M, A.n_bus, A.n_diff + A.n_alg, A.n_sys
        self.p0, self.u0 = t(s["p"]), t(np.tile(s["dp"].uvec, (M, 1)))
        self.z0 = t(np.tile(s["dp"].zvec, (M, 1)))
        self.is_diff = torch.zeros(self.n, dtype=torch.bool, device=dev)
        self.is_diff[:self.net] = t(A.is_diff, torch.bool)
        rows = np.repeat(np.arange(A.n_bus), np.diff(A.y_rowptr))
        self.Y = torch.zeros(A.n_bus, A.n_bus, dtype=torch.complex128, device=dev)
        self.Y[t(rows, i64), t(A.y_colidx, i64)] = torch.complex(t(A.y_re), t(A.y_im))
        self.T = []
        for T in A.tables:
            self.T.append({k: t(getattr(T, k), i64) for k in ("bus", "diff_ptr", "alg_ptr", "ctrl_ptr", "par_ptr",
                                                             "link0", "link1")})
        # clusters: their states, padded to the widest, and their bus
        W = int(A.cl_w_size.max())
        st = A.cl_w_start[:, None] + np.minimum(np.arange(W)[None], A.cl_w_size[:, None] - 1)
        self.cl, self.clw = t(st, i64), t(A.cl_w_size, i64)
        self.clbus = t(A.cl_bus, i64)
        assert len(set(A.cl_bus.tolist())) == len(A.cl_bus) and A.tables[LY.GP_STATIC_GEN].n == 0
        self.W = W
        self.yf = torch.zeros(M, A.n_bus, dtype=torch.float64, device=dev)
        self.dY = [None] * M      # line tripped in a scenario

    # -- equations: right-hand sides of the device rows, currents at the buses
    def local(self, z, p):
        M, net = z.shape[0], self.net
        vr_all, vi_all = z[:, net::2], z[:, net + 1::2]
        f = torch.zeros_like(z)
        cr, ci = torch.zeros_like(vr_all), torch.zeros_like(vi_all)
        g = self.T[0]
        if g["bus"].numel():
            P = lambda k: p[:, g["par_ptr"] + k]  # noqa: E731
            x_d, x_q, x_dp, x_qp, x_ddp, xl, H, D, Td0p, Tq0p, Td0dp, Tq0dp, S1, S2 = [P(k) for k in range(14)]
            dp_, ap = g["diff_ptr"], g["alg_ptr"]
            eq, ed, p1, p2, w, de = [z[:, dp_ + k] for k in range(6)]
            vq, vd, iq, id_ = [z[:, ap + k] for k in range(4)]
            vr, vi = vr_all[:, g["bus"]], vi_all[:, g["bus"]]
            efd = torch.where(g["link1"] >= 0, z[:, g["link1"].clamp(min=0)], self.u0[:M, g["ctrl_ptr"]])
            pm = torch.where(g["link0"] >= 0, z[:, g["link0"].clamp(min=0)], self.u0[:M, g["ctrl_ptr"] + 1])
            psd = (x_ddp - xl) / (x_dp - xl) * eq + (x_dp - x_ddp) / (x_dp - xl) * p1
            psq = -(x_ddp - xl) / (x_qp - xl) * ed + (x_qp - x_ddp) / (x_qp - xl) * p2
            has = (S1 > 0) & (S2 > 0)
            a = torch.sqrt(torch.where(has, S1 / (S2 * 1.2).clamp(min=1e-300), torch.full_like(S1, 0.25)))
            sa = 1.2 + 0.2 / (a - 1.0)
            sb = S2 * 1.2 * (a - 1.0) ** 2 / 0.04
            psi = torch.sqrt(psd * psd + psq * psq)
            Se = torch.where(has & (psi > sa), sb * (psi - sa) ** 2 / psi, torch.zeros_like(psi))
            kd = (x_dp - x_ddp) / (x_dp - xl) ** 2
            kq = (x_qp - x_ddp) / (x_qp - xl) ** 2
            r = [(-eq + efd - (id_ - kd * (-eq + id_ * (x_dp - xl) + p1)) * (x_d - x_dp) - Se * psd) / Td0p,
                 (-ed + (iq - kq * (ed + iq * (x_qp - xl) + p2)) * (x_q - x_qp)) / Tq0p,
                 (eq - id_ * (x_dp - xl) - p1) / Td0dp,
                 (-ed - iq * (x_qp - xl) - p2) / Tq0dp,
                 (pm - D * w - psd * iq + psq * id_) / (2.0 * H),
                 2.0 * math.pi * 60.0 * w]
            q = [id_ - (psd - vq) / x_ddp, iq - (psq + vd) / x_ddp,
                 vd - (vr * torch.sin(de) - vi * torch.cos(de)), vq - (vr * torch.cos(de) + vi * torch.sin(de))]
            f = f.index_copy(1, torch.cat([dp_ + k for k in range(6)] + [ap + k for k in range(4)]),
                             torch.cat(r + q, 1))
            cr = cr.index_add(1, g["bus"], torch.sin(de) * id_ + torch.cos(de) * iq)
            ci = ci.index_add(1, g["bus"], -torch.cos(de) * id_ + torch.sin(de) * iq)
        speed = lambda T: torch.where(T["link0"] >= 0, z[:, T["link0"].clamp(min=0)], torch.zeros((), dtype=z.dtype, device=z.device))  # noqa: E731,E501

        def put(f, T, d, a):
            ix = [T["diff_ptr"] + k for k in range(len(d))] + [T["alg_ptr"] + k for k in range(len(a))]
            return f.index_copy(1, torch.cat(ix), torch.cat(d + a, 1))

        T = self.T[1]
        if T["bus"].numel():       # IEESGO
            q = lambda k: p[:, T["par_ptr"] + k]  # noqa: E731
            x = [z[:, T["diff_ptr"] + k] for k in range(5)]
            pm = z[:, T["alg_ptr"]]
            r23 = q(1) / q(2)
            f = put(f, T, [(q(6) * speed(T) - x[0]) / q(0), ((1 - r23) * x[0] - x[1]) / q(2),
                           (q(11) - r23 * x[0] - x[1] - x[2]) / q(3), (q(7) * x[2] - x[3]) / q(4),
                           (q(8) * x[3] - x[4]) / q(5)],
                    [x[2] * (1 - q(7)) + x[3] * (1 - q(8)) + x[4] - pm])
        T = self.T[2]
        if T["bus"].numel():       # TGOV1
            q = lambda k: p[:, T["par_ptr"] + k]  # noqa: E731
            x1, x2, pm, w = z[:, T["diff_ptr"]], z[:, T["diff_ptr"] + 1], z[:, T["alg_ptr"]], speed(T)
            r23 = q(4) / q(5)
            f = put(f, T, [(-x1 + (1 - r23) * x2) / q(5), ((q(7) - w) / q(0) - x2) / q(1)],
                    [x1 + r23 * x2 - q(6) * w - pm])
        T = self.T[3]
        if T["bus"].numel():       # SEXS
            q = lambda k: p[:, T["par_ptr"] + k]  # noqa: E731
            x1, efd = z[:, T["diff_ptr"]], z[:, T["diff_ptr"] + 1]
            vm = torch.sqrt(vr_all[:, T["bus"]] ** 2 + vi_all[:, T["bus"]] ** 2)
            err = q(6) - vm + speed(T)
            f = put(f, T, [(-x1 + (1 - q(0)) * err) / q(1), (-efd + q(2) * (x1 + q(0) * err)) / q(3)], [])
        T = self.T[4]
        if T["bus"].numel():       # ESDC1A
            q = lambda k: p[:, T["par_ptr"] + k]  # noqa: E731
            v1, v2, efd = [z[:, T["diff_ptr"] + k] for k in range(3)]
            vm = torch.sqrt(vr_all[:, T["bus"]] ** 2 + vi_all[:, T["bus"]] ** 2)
            kft = q(2) / q(3)
            sat = torch.where((q(8) != 0) & (efd > q(7)), q(8) * (efd - q(7)) ** 2, torch.zeros_like(efd))
            f = put(f, T, [(q(0) * (q(9) - vm + speed(T) - v2 - kft * efd) - v1) / q(1), -(kft * efd + v2) / q(3),
                           (v1 - q(4) * efd - sat) / q(5)], [])
        T = self.T[5]
        if T["bus"].numel():       # IEEEST
            q = lambda k: p[:, T["par_ptr"] + k]  # noqa: E731
            s = [z[:, T["diff_ptr"] + k] for k in range(7)]
            vs = z[:, T["alg_ptr"]]
            A1, A2, A3, A4, A5, A6, T1, T2, T3, T4, T5, T6, KS = [q(k) for k in range(13)]
            qq = s[1] - s[3] - A3 * s[2]
            y2 = s[3] + A5 * s[2] + A6 / A4 * qq
            y3 = s[4] + T1 / T2 * (y2 - s[4])
            y4 = s[5] + T3 / T4 * (y3 - s[5])
            f = put(f, T, [(speed(T) - s[1] - A1 * s[0]) / A2, s[0], qq / A4, s[2], (y2 - s[4]) / T2,
                           (y3 - s[5]) / T4, (KS * y4 - s[6]) / T6], [vs - T5 / T6 * (KS * y4 - s[6])])
        T = self.T[6]
        if T["bus"].numel():       # ZIP loads
            q = lambda k: p[:, T["par_ptr"] + k]  # noqa: E731
            vr, vi = vr_all[:, T["bus"]], vi_all[:, T["bus"]]
            vm2 = (vr * vr + vi * vi).clamp(min=0.2)
            a = (1 - q(2)) * q(0) / vm2 + q(2) * q(7)
            c = (1 - q(2)) * q(1) / vm2 + q(2) * q(8)
            cr = cr.index_add(1, T["bus"], -vr * a + vi * c)
            ci = ci.index_add(1, T["bus"], -vi * a - vr * c)
        return f, cr, ci

    def residual(self, z, zold, dt, p, yf):
        """Backward-Euler residual; yf: the fault shunts."""
        f, cr, ci = self.local(z, p)
        net = self.net
        V = torch.complex(z[:, net::2], z[:, net + 1::2])
        I = -(V @ self.Y.T)
        for m, d in enumerate(self.dY):
            if d is not None:
                a, b, yff, yft, ytf, ytt = d
                e = torch.zeros_like(I)
                e[m, a] = yff * V[m, a].detach() + yft * V[m, b].detach()
                e[m, b] = ytf * V[m, a].detach() + ytt * V[m, b].detach()
                I = I + e
        cr = cr + I.real - yf * z[:, net::2]
        ci = ci + I.imag - yf * z[:, net + 1::2]
        bus = torch.stack([cr, ci], 2).reshape(z.shape[0], -1)
        F = torch.where(self.is_diff, z - zold - dt * f, f)
        return torch.cat([F[:, :net], bus], 1)

    # -- Jacobian blocks and the dense Schur complement on the buses
    def factor(self, z, dt, p, yf):
        M, net, W, nb = self.M, self.net, self.W, self.nb
        nc = self.cl.shape[0]

        def jvp(tan):
            _, (df, dr, di) = torch.func.jvp(lambda x: self.local(x, p), (z,), (tan,))
            rows = torch.where(self.is_diff[:net], tan[:, :net] - dt * df[:, :net], df[:, :net])
            return rows, dr, di

        A = torch.zeros(M, nc, W, W, dtype=z.dtype, device=z.device)
        B = torch.zeros(M, nc, W, 2, dtype=z.dtype, device=z.device)
        C = torch.zeros(M, nc, 2, W, dtype=z.dtype, device=z.device)
        real = torch.arange(W, device=z.device)[None] < self.clw[:, None]          # [nc, W]
        for j in range(W):
            tan = torch.zeros_like(z)
            tan[:, self.cl[real[:, j], j]] = 1.0
            rows, dr, di = jvp(tan)
            A[..., j] = torch.where(real, rows[:, self.cl], torch.zeros((), dtype=z.dtype, device=z.device))
            C[..., 0, j], C[..., 1, j] = dr[:, self.clbus], di[:, self.clbus]
            pad = ~real[:, j]
            A[:, pad, :, j] = 0.0
            A[:, pad, j, j] = 1.0
            C[:, pad, :, j] = 0.0
        D = torch.zeros(M, nb, 2, 2, dtype=z.dtype, device=z.device)
        for k in range(2):
            tan = torch.zeros_like(z)
            tan[:, net + k::2] = 1.0
            rows, dr, di = jvp(tan)
            B[..., k] = torch.where(real, rows[:, self.cl], torch.zeros((), dtype=z.dtype, device=z.device))
            D[..., 0, k], D[..., 1, k] = dr, di
        lu = torch.linalg.lu_factor(A)
        X = torch.linalg.lu_solve(*lu, B)
        D[:, self.clbus] -= C @ X
        ib = torch.arange(nb, device=z.device)
        D[:, ib, 0, 0] -= yf
        D[:, ib, 1, 1] -= yf
        Yr = torch.zeros(nb, 2, nb, 2, dtype=z.dtype, device=z.device)
        Yr[:, 0, :, 0] = -self.Y.real
        Yr[:, 0, :, 1] = self.Y.imag
        Yr[:, 1, :, 0] = -self.Y.imag
        Yr[:, 1, :, 1] = -self.Y.real
        out = []
        for m in range(M):
            S = Yr.clone()
            S[ib, :, ib, :] += D[m]
            if self.dY[m] is not None:
                a, b, yff, yft, ytf, ytt = self.dY[m]
                for i, j, y in ((a, a, yff), (a, b, yft), (b, a, ytf), (b, b, ytt)):
                    S[i, :, j, :] += torch.tensor([[y.real, -y.imag], [y.imag, y.real]], dtype=z.dtype,
                                                  device=z.device)
            out.append(torch.linalg.lu_factor(S.reshape(2 * nb, 2 * nb)))
        return dict(lu=lu, X=X, B=B, C=C, S=out, real=real)

    def solve(self, K, r, transpose=False):
        """J x = r with the blocks of factor (J^T x = r with transpose)."""
        M, net = self.M, self.net
        rc = torch.where(K["real"], r[:, self.cl], torch.zeros((), dtype=r.dtype, device=r.device))[..., None]
        rb = r[:, net:].reshape(M, -1, 2).clone()
        x = torch.zeros_like(r)
        if transpose:
            rb[:, self.clbus] -= (K["X"].transpose(-1, -2) @ rc)[..., 0]
        else:
            y = torch.linalg.lu_solve(*K["lu"], rc)
            rb[:, self.clbus] -= (K["C"] @ y)[..., 0]
        v = torch.stack([torch.linalg.lu_solve(*K["S"][m], rb[m].reshape(-1, 1), adjoint=transpose)[:, 0]
                         for m in range(M)])
        vb = v.reshape(M, -1, 2)[:, self.clbus][..., None]
        if transpose:
            w = torch.linalg.lu_solve(*K["lu"], rc - K["C"].transpose(-1, -2) @ vb, adjoint=True)
        else:
            w = y - K["X"] @ vb
        x[:, self.cl[K["real"]]] = w[..., 0][:, K["real"]]
        x[:, net:] = v
        return x

    def newton(self, z, zold, dt, p, yf, K):
        """To rounding level, with factors K as long as they contract well;
        returns the state and the factors last used."""
        last, fresh = math.inf, False
        for _ in range(60):
            F = self.residual(z, zold, dt, p, yf)
            nrm = float(F.abs().max())
            if nrm < 1e-11 and nrm > 0.3 * last or nrm == 0.0:
                break
            if K is None or (nrm > 0.1 * last and not fresh and nrm > 1e-11):
                K, fresh = self.factor(z, dt, p, yf), True
            else:
                fresh = False
            last = nrm
            z = z - self.solve(K, F)
        return z, K

    def events(self, k):
        """Toggles after step k; true when there were any."""
        s, hit = self.s, False
        for m in range(self.M):
            if k == s["on"] or k == s["off"]:
                self.yf[m, int(s["fb"][m])] = 1.0 / float(s["rf"][m]) if k == s["on"] else 0.0
                hit = True
            for t in (s["trips"] or [[]] * self.M)[m]:
                if k == int(round(t.ton / DT)):
                    self.dY[m], hit = (t.from_bus, t.to_bus, t.yff, t.yft, t.ytf, t.ytt), True
                elif math.isfinite(t.toff) and k == int(round(t.toff / DT)):
                    self.dY[m], hit = None, True
        return hit

    def run(self):
        with torch.no_grad():
            return self._run()

    def _run(self):
        case, p = self.case, self.p0
        z, traj, solves = self.z0, [self.z0], []
        K = None
        for k in range(1, case["steps"] + 1):
            zold = z
            z, K = self.newton(z, zold, DT, p, self.yf, K)
            traj.append(z)
            if case["kind"] == "adjoint":
                solves.append((z, DT, self.yf.clone(), True))
            if self.events(k):
                z, _ = self.newton(z, z, 0.0, p, self.yf, None)
                K = None
                if case["kind"] == "adjoint":
                    solves.append((z, 0.0, self.yf.clone(), False))
        if case["kind"] == "adjoint":
            return self.adjoint(solves)
        out = torch.stack(traj, 1) if case["traj"] != "none" else z
        if case["kind"] == "shared":
            return {"traj": out.cpu().numpy()}
        r = {"status": None, "traj": out.cpu().numpy()}
        if case["kind"] == "fp64":
            r["iters"] = None
        return r

    # -- adjoint of the solves, last to first
    def adjoint(self, solves):
        p, net = self.p0, self.net
        gw = self.T[0]["diff_ptr"] + 4
        diff = self.is_diff
        J = torch.zeros(self.M, dtype=torch.float64, device=self.dev)
        gp = torch.zeros_like(p)
        g = torch.zeros_like(self.z0)
        K, key = None, None
        for z, dt, yf, stored in reversed(solves):
            if stored:
                vr, vi = z[:, net::2], z[:, net + 1::2]
                vm = torch.sqrt(vr * vr + vi * vi)
                s = (0.9 - vm).clamp(min=0.0)
                J += DT * ((z[:, gw] ** 2).sum(1) + 10.0 * (s * s).sum(1))
                g[:, gw] += DT * 2.0 * z[:, gw]
                g[:, net::2] += -DT * 20.0 * s * vr / vm
                g[:, net + 1::2] += -DT * 20.0 * s * vi / vm
            now = (dt, yf.sum().item())
            if K is None or key != now:
                K, key = self.factor(z, dt, p, yf), now
            # J^T lambda = g at this state, refined with the factors at hand
            with torch.enable_grad():
                zz, pp = z.clone().requires_grad_(True), p.clone().requires_grad_(True)
                F = self.residual(zz, z, dt, pp, yf)
            jt = lambda lam: torch.autograd.grad(F, zz, lam, retain_graph=True)[0]  # noqa: E731
            # (states of scenarios that took no re-solve keep theirs: every
            # scenario's fault toggles at the same steps here)
            lam, last = self.solve(K, g, True), math.inf
            for _ in range(40):
                r = g - jt(lam)
                nrm = float((r.abs().amax(1) / g.abs().amax(1).clamp(min=1e-300)).max())
                if nrm < 1e-15 or (nrm < 1e-12 and nrm > 0.3 * last):
                    break
                if nrm > 0.2 * last:
                    K = self.factor(z, dt, p, yf)
                last = nrm
                lam = lam + self.solve(K, r, True)
            gp -= torch.autograd.grad(F, pp, lam)[0]
            g = torch.where(diff, lam, torch.zeros_like(lam))
        keep = torch.zeros(p.shape[1], dtype=torch.bool, device=self.dev)
        for t, ks in ((0, (6, 7)), (1, (6,)), (2, (0,)), (3, (2,)), (4, (0,))):
            for k in ks:
                keep[self.T[t]["par_ptr"] + k] = True
        gp = torch.where(keep, gp, torch.zeros_like(gp))
        return {"J": J.cpu().numpy(), "grad_p": gp.cpu().numpy(), "grad_z0": g.cpu().numpy(), "status": None}
