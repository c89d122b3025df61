"""The work this framework is used for, as timed cases: batched AC power flow through its public entry points.

A case is a dict of plain values; `prepare` makes what a program holds before the call (the
topology's solver and the call's inputs), `run` is one call, `exact` the same voltages from a
dense 64-bit Newton solve that uses none of this repository's code. Grids are the seeded
synthetic ones of `p3s_gb300.synthetic`; a topology's solver is kept for the life of the
program, as a user keeps it, and every seed gives other injections.

kind    entry point                                          what it stands for
solve   nr_klu.Solver.solve                                  one operating point, drop-in CPU surface
batch   PolarNewtonSolverCUDA.solve_batch                    steps or scenarios of one grid, host arrays
study   studies.calculate_timeseries_cpp (DC start)          a whole time-series study, host arrays
series  GpuSolver.solve_lanes_device                         an hourly series resident on the GPU
n1      contingency.solve_contingencies                      every single-branch outage of a grid
group   group.GpuGroup.solve                                 many grids of uneven size in one launch
"""

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "parallel-pandapower-solver_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

# pool grids left out of drawn outage sweeps: some outage of theirs has no AC solution
NO_N1 = (47, 59, 99, 105, 131, 148, 168, 190, 191, 241)
EXACT_MAX_BUS = 4000  # dense 64-bit solves up to this size (a 2 n x 2 n factorization)
EXACT_MAX_N1 = 300    # ... and one such system per outage case up to this size


def listed():
    return [
        # one operating point of a small grid: launches and latency
        {"name": "solve_118_double", "kind": "solve", "n": 118, "cases": 1, "precision": "double"},
        # one operating point of the 2,000-bus grid
        {"name": "solve_2000_mixed", "kind": "batch", "n": 2000, "cases": 1, "precision": "mixed"},
        # a day of quarter hours (96 steps): the serving loop's chunk, odd and round grid sizes
        {"name": "chunk_777x96_mixed", "kind": "batch", "n": 777, "cases": 96, "precision": "mixed"},
        {"name": "chunk_2000x96_double", "kind": "batch", "n": 2000, "cases": 96, "precision": "double"},
        # the largest single grid: a few load scenarios of a transmission model
        {"name": "scenarios_19999x16_mixed", "kind": "batch", "n": 19999, "cases": 16, "precision": "mixed"},
        # a month of hours as a study from its DC start
        {"name": "study_490x744_double", "kind": "study", "n": 490, "cases": 744, "precision": "double"},
        # a year of hours, each from the converged base case, both precisions
        {"name": "series_2000x8760_mixed", "kind": "series", "n": 2000, "cases": 8760, "lanes": 8760,
         "precision": "mixed"},
        {"name": "series_2000x8760_double", "kind": "series", "n": 2000, "cases": 8760, "lanes": 8760,
         "precision": "double"},
        # the same year in twelve-hour warm-start lanes (hour h from hour h - 1)
        {"name": "lanes_2000x8760_mixed", "kind": "series", "n": 2000, "cases": 8760, "lanes": 730,
         "precision": "mixed"},
        # the intact grid and every single-branch outage, islands found and re-slacked
        {"name": "n1_2000_mixed", "kind": "n1", "n": 2000, "cases": 3001, "precision": "mixed"},
        {"name": "n1_2000_double", "kind": "n1", "n": 2000, "cases": 3001, "precision": "double"},
        # grids of 30 to 20,000 buses, 16 load scenarios each, in one launch
        {"name": "group_20x16_mixed", "kind": "group", "n": 20000, "grids": 20, "cases": 16, "precision": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pool():
    """Bus counts of the uneven multi-grid batch's 256 grids, log-uniform in [30, 20,000]; grid i has seed 7000 + i."""
    rng = np.random.default_rng(7)
    return [int(x) for x in np.exp(rng.uniform(math.log(30), math.log(20000), 256)).astype(int)]


def _pick(rng, lo, hi, without=()):
    """A pool grid of lo to hi buses, sizes spread over their logarithm."""
    ok = [i for i, n in enumerate(_pool()) if lo <= n <= hi and i not in without]
    i = rng.choice(ok)
    return {"n": _pool()[i], "grid_seed": 7000 + i}


def draw(rng):
    """One more case: a grid of the multi-grid pool, n x cases within a year of the 2,000-bus grid."""
    kind = rng.choice(["solve", "batch", "batch", "study", "series", "series", "n1", "n1", "group"])
    precision = rng.choice(["mixed", "double"])
    if kind == "solve":
        return {"kind": kind, **_pick(rng, 30, 6000), "cases": 1, "precision": "double"}
    if kind == "batch":
        g = _pick(rng, 60, 20000)
        return {"kind": kind, **g, "cases": _log_int(rng, 1, min(400, 800000 // g["n"])), "precision": precision}
    if kind == "study":
        return {"kind": kind, **_pick(rng, 60, 1500), "cases": _log_int(rng, 24, 744), "precision": precision}
    if kind == "series":
        g = _pick(rng, 100, 3000)
        T = _log_int(rng, 300, min(8760, 8000000 // g["n"]))
        return {"kind": kind, **g, "cases": T, "lanes": rng.choice([T, max(1, T // rng.randint(2, 6))]),
                "precision": precision}
    if kind == "n1":
        g = _pick(rng, 60, 1500, NO_N1)
        return {"kind": kind, **g, "cases": int(round(1.5 * g["n"])) + 1, "precision": precision}
    return {"kind": kind, "n": _log_int(rng, 400, 12000), "grids": rng.randint(3, 16), "cases": rng.randint(3, 16),
            "precision": precision}


# ------------------------------------------------------------------------------ inputs
_kept = {}  # topologies and their solvers, kept for the life of the program


def _grid(n, seed=0):
    from p3s_gb300 import synthetic

    if ("grid", n, seed) not in _kept:
        if (n, seed) == (118, 0):
            g = synthetic.grid_118()
        elif (n, seed) == (2000, 0):
            g = synthetic.grid_2000()
        else:
            g = synthetic.make_grid(n, seed=seed, max_drop_pu=0.05)
        _kept["grid", n, seed] = g
    return _kept["grid", n, seed]


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _group_grids(case):
    """(n, seed) of a group's grids: the first pool grids of at most n buses, the largest of them first."""
    ok = [(n, 7000 + i) for i, n in enumerate(_pool()) if n <= case["n"]]
    return [max(ok)] + [g for g in ok if g != max(ok)][: case["grids"] - 1]


def _base_injections(g):
    return (g.p_gen - g.p_load) - 1j * g.q_load


def _host_injections(g, T, seed, spread=0.2):
    """(n, T) load scenarios: every load scaled by U(1 - spread, 1 + spread)."""
    rng = np.random.default_rng([seed, g.n])
    S = np.repeat(_base_injections(g)[:, None], T, axis=1)
    S[g.pq] *= rng.uniform(1.0 - spread, 1.0 + spread, (len(g.pq), T))
    return np.ascontiguousarray(S)


def _hourly_injections(g, T, seed):
    """(n, T, 2) float64 hourly injections on the GPU: loads base (1 + 0.3 sin(2 pi h / 24)) LogNormal(0, 0.1),
    generation base U(0.5, 1.2) dispatched to the hour's load."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    f64 = dict(dtype=torch.float64, device=dev)
    pq, pv = torch.as_tensor(g.pq, device=dev).long(), torch.as_tensor(g.pv, device=dev).long()
    h = torch.arange(T, **f64)
    lf = (1.0 + 0.3 * torch.sin(2.0 * math.pi * h / 24.0)) * torch.exp(0.1 * torch.randn(len(pq), T, generator=gen, **f64))
    pl = torch.as_tensor(g.p_load, **f64)[pq, None] * lf
    ql = torch.as_tensor(g.q_load, **f64)[pq, None] * lf
    pg = torch.as_tensor(g.p_gen, **f64)[pv, None] * (0.5 + 0.7 * torch.rand(len(pv), T, generator=gen, **f64))
    pg *= (float(g.p_gen.sum() / g.p_load.sum()) * pl.sum(0) / pg.sum(0))[None, :]
    S = torch.zeros(g.n, T, 2, **f64)
    S[pq, :, 0] = -pl
    S[pq, :, 1] = -ql
    S[pv, :, 0] = pg
    return S


def _base_voltage(g, solver):
    """The converged base case, as a file of it would hold it: magnitudes (set-points kept) and angles to nine decimals."""
    from p3s_gb300.solver import GpuSolver

    V = solver.solve_batch(_base_injections(g)[:, None], g.V0, GpuSolver.params())["V"][:, 0]
    vm = np.abs(g.V0)
    vm[g.pq] = np.round(np.abs(V[g.pq]), 9)
    return vm * np.exp(1j * np.round(np.angle(V), 9))


def prepare(case, seed):
    from p3s_gb300 import nr_klu
    from p3s_gb300.cuda.nr_polar_solver import PolarNewtonSolverCUDA
    from p3s_gb300.group import GpuGroup, GroupJob
    from p3s_gb300.solver import GpuSolver

    kind, T = case["kind"], case["cases"]
    st = {"kind": kind, "precision": case["precision"]}
    if kind == "group":
        jobs = []
        for n, grid_seed in _group_grids(case):
            g = _grid(n, grid_seed)
            s = _keep(("GpuSolver", n, grid_seed), lambda g=g: GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq))
            jobs.append(GroupJob(s, _host_injections(g, T, seed), g.V0))
        st.update(jobs=jobs, group=_keep("GpuGroup", GpuGroup), params=GpuSolver.params(precision=case["precision"]))
        return st
    g = st["grid"] = _grid(case["n"], case.get("grid_seed", 0))
    key = (g.n, case.get("grid_seed", 0))
    topology = (g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    if kind == "solve":
        st["solver"] = _keep(("nr_klu", *key), lambda: nr_klu.Solver(*topology))
        st["S"] = np.ascontiguousarray(_host_injections(g, 1, seed)[:, 0])
    elif kind in ("batch", "study"):
        st["solver"] = _keep(("cuda", *key), lambda: PolarNewtonSolverCUDA(*topology))
        st["S"] = _host_injections(g, T, seed)
    elif kind == "n1":
        st["solver"] = _keep(("cuda", *key), lambda: PolarNewtonSolverCUDA(*topology))
        st["S"] = np.ascontiguousarray(_host_injections(g, 1, seed, 0.1)[:, 0])
    elif kind == "series":
        s = st["solver"] = _keep(("GpuSolver", *key), lambda: GpuSolver(*topology))
        V0 = _keep(("base", *key), lambda: _base_voltage(g, s))
        st["S"] = _hourly_injections(g, T, seed)
        st["V0"] = torch.from_numpy(V0.view(np.float64).copy()).cuda()
        st["offsets"] = torch.linspace(0, T, case["lanes"] + 1, dtype=torch.float64).round().long().cuda()
        st["V"] = torch.empty(g.n, T, 2, dtype=torch.float64, device="cuda")
        st["iterations"] = torch.empty(T, dtype=torch.int32, device="cuda")
        st["converged"] = torch.empty(T, dtype=torch.uint8, device="cuda")
        st["params"] = GpuSolver.params(precision=case["precision"])
    else:
        raise ValueError("unknown kind %r" % kind)
    return st


# ------------------------------------------------------------------------------ one pass
def run(st):
    kind = st["kind"]
    if kind == "solve":
        r = st["solver"].solve(st["S"], st["grid"].V0)
    elif kind == "batch":
        st["solver"].precision = st["precision"]
        r = st["solver"].solve_batch(st["S"], st["grid"].V0)
    elif kind == "study":
        from p3s_gb300.studies import calculate_timeseries_cpp

        return {"V": calculate_timeseries_cpp(st["grid"], st["S"], init="dc", precision=st["precision"],
                                              solver=st["solver"])}
    elif kind == "n1":
        from p3s_gb300.contingency import solve_contingencies

        st["grid"].Sbus = st["S"]  # this snapshot's injections on the resident grid
        t = solve_contingencies(st["grid"], reslack_islands=True, precision=st["precision"], solver=st["solver"],
                                return_islands=False)
        return {"V": t.V, "iterations": t.iterations, "converged": t.converged, "served": t.served}
    elif kind == "group":
        return [{k: r[k] for k in ("V", "iterations", "converged")} for r in st["group"].solve(st["jobs"], st["params"])]
    else:
        T = st["S"].shape[1]
        st["solver"].solve_lanes_device(st["S"].data_ptr(), st["V0"].data_ptr(), st["offsets"].data_ptr(), T,
                                        len(st["offsets"]) - 1, st["params"], st["V"].data_ptr(),
                                        st["iterations"].data_ptr(), st["converged"].data_ptr())
        r = st
    return {k: r[k] for k in ("V", "iterations", "converged")}


def work(case):
    """Each case's injections read and voltages written once, its flags; and, per case, three Newton steps of a
    mismatch (8 per nonzero), a Jacobian (16 per nonzero) and a sparse factorization and solve with its fill
    (about 2.2 blocks of 2 x 2 multiply-adds per nonzero)."""
    sizes = [n for n, _ in _group_grids(case)] if case["kind"] == "group" else [case["n"]]
    T = case["cases"]
    per_case_in = 0 if case["kind"] == "n1" else 16
    nbytes = sum(n * (T * (16 + per_case_in) + 16 + 4 * 16) + 5 * T for n in sizes)
    return {"bytes": nbytes, "flops": sum(3.0 * T * 4 * n * (8 + 16 + 2.2 * 16) for n in sizes)}


# ------------------------------------------------------------------------------ the same in 64 bits, densely
def _injected(Yd, V):
    return V * torch.conj(Yd @ V)


def _dense_jacobian(Yd, V, fixed, pq):
    """d[P; Q] / d[angle; magnitude] for every bus (V (..., n)); identity rows and columns at fixed buses
    (angle and magnitude) and at PV buses (magnitude)."""
    n = V.shape[-1]
    I = (Yd @ V.unsqueeze(-1)).squeeze(-1)
    U = V / V.abs()
    D = torch.diag_embed
    dA = 1j * V.unsqueeze(-1) * torch.conj(D(I) - Yd * V.unsqueeze(-2))
    dM = V.unsqueeze(-1) * torch.conj(Yd * U.unsqueeze(-2)) + D(torch.conj(I) * U)
    J = torch.cat([torch.cat([dA.real, dM.real], -1), torch.cat([dA.imag, dM.imag], -1)], -2)
    keep = torch.cat([~fixed, pq & ~fixed], -1).double()
    return J * keep.unsqueeze(-1) * keep.unsqueeze(-2) + D(1.0 - keep), keep


def _dense_y(g, dev):
    Y = torch.zeros(g.n, g.n, dtype=torch.complex128, device=dev)
    rows = torch.as_tensor(np.repeat(np.arange(g.n), np.diff(g.Yp)), device=dev)
    Y[rows, torch.as_tensor(g.Yj, device=dev).long()] = torch.as_tensor(g.Yx, device=dev)
    return Y


def _step(V, dx, n):
    return (V.abs() + dx[n:]) * torch.exp(1j * (V.angle() + dx[:n]))


def _exact_columns(g, S):
    """(n, T) voltages of injections S (n, T): Newton on the base case, then its factored Jacobian for all
    columns until the worst mismatch is down to rounding; None where that does not converge."""
    dev, n = S.device, g.n
    Y = _dense_y(g, dev)
    sparse = Y.to_sparse_csr() if S.shape[1] > 1 else Y
    fixed = torch.ones(n, dtype=torch.bool, device=dev)
    pq = torch.zeros(n, dtype=torch.bool, device=dev)
    fixed[torch.as_tensor(np.r_[g.pv, g.pq], device=dev).long()] = False
    pq[torch.as_tensor(g.pq, device=dev).long()] = True
    V = torch.as_tensor(g.V0, device=dev)
    base = torch.as_tensor(_base_injections(g), device=dev)
    for _ in range(8):
        J, keep = _dense_jacobian(Y, V, fixed, pq)
        d = base - _injected(Y, V)
        V = _step(V, torch.linalg.solve(J, torch.cat([d.real, d.imag]) * keep), n)
    LU = torch.linalg.lu_factor(_dense_jacobian(Y, V, fixed, pq)[0])
    V = V[:, None].repeat(1, S.shape[1])
    best, stale = math.inf, 0
    for _ in range(100):
        d = S - _injected(sparse, V)
        b = torch.cat([d.real, d.imag]) * keep[:, None]
        worst = float(b.abs().max())
        stale = 0 if worst < 0.8 * best else stale + 1
        best = min(best, worst)
        if stale > 4 or not math.isfinite(worst):
            break
        V = _step(V, torch.linalg.lu_solve(*LU, b), n)
    return V if best < 1e-11 else None


def _exact_n1(g, S):
    """(n, L) voltages of the intact grid and every single-branch outage, NaN where unserved: components of
    the remaining branches by repeated label minimum; an island without the slack takes its generator of
    largest scheduled power (lowest index on ties) as a reference at |V0| + 0j."""
    dev, n, m = S.device, g.n, g.n_branch
    Y = _dense_y(g, dev)
    f, t = (torch.as_tensor(a, device=dev).long() for a in (g.f, g.t))
    pq = torch.zeros(n, dtype=torch.bool, device=dev)
    pq[torch.as_tensor(g.pq, device=dev).long()] = True
    slack = int(g.ref[0])
    prio = np.zeros(n)
    prio[g.pv] = np.maximum(g.p_gen[g.pv], np.finfo(float).tiny)
    Vs = []
    for lo in range(-1, m, 128):
        outs = list(range(lo, min(lo + 128, m)))
        L = len(outs)
        Yc = Y.repeat(L, 1, 1)
        fixed = torch.zeros(L, n, dtype=torch.bool, device=dev)
        V = torch.as_tensor(g.V0, device=dev).repeat(L, 1)
        dead = torch.zeros(L, n, dtype=torch.bool, device=dev)
        for c, b in enumerate(outs):
            if b >= 0:
                for (r, s), y in zip(((f[b], f[b]), (f[b], t[b]), (t[b], f[b]), (t[b], t[b])), g.stamp[b]):
                    Yc[c, r, s] -= complex(y)
            live = np.arange(m) != b
            lab = np.arange(n)
            while True:
                new = lab.copy()
                np.minimum.at(new, g.f[live], lab[g.t[live]])
                np.minimum.at(new, g.t[live], lab[g.f[live]])
                new = np.minimum(new, new[new])
                if np.array_equal(new, lab):
                    break
                lab = new
            for k in np.unique(lab):
                bus = np.nonzero(lab == k)[0]
                if slack in bus:
                    fixed[c, slack] = True
                elif prio[bus].max() > 0:
                    r = int(bus[np.argmax(prio[bus])])
                    fixed[c, r] = True
                    V[c, r] = abs(g.V0[r])
                else:
                    fixed[c, bus] = True
                    dead[c, bus] = True
                    V[c, bus] = 1.0
        pqc = pq.expand(L, n)
        for _ in range(12):
            J, keep = _dense_jacobian(Yc, V, fixed, pqc)
            d = S - V * torch.conj((Yc @ V.unsqueeze(-1)).squeeze(-1))
            dx = torch.linalg.solve(J, torch.cat([d.real, d.imag], -1) * keep)
            V = _step(V.T, dx.T, n).T
        if not float((torch.cat([d.real, d.imag], -1) * keep).abs().max()) < 1e-11:
            return None
        V[dead] = complex(math.nan, math.nan)
        Vs.append(V)
    return torch.cat(Vs).T.contiguous()


def exact(case, seed):
    kind, T = case["kind"], case["cases"]
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind == "group":
        out = []
        for n, grid_seed in _group_grids(case):
            g = _grid(n, grid_seed)
            V = None
            if n <= 2500:
                V = _exact_columns(g, torch.as_tensor(_host_injections(g, T, seed), device=dev))
            out.append({"V": None if V is None else V.cpu().numpy(), "iterations": None, "converged": None})
        return out if any(o["V"] is not None for o in out) else None
    g = _grid(case["n"], case.get("grid_seed", 0))
    if kind == "n1":
        if g.n > EXACT_MAX_N1:
            return None
        V = _exact_n1(g, torch.as_tensor(_host_injections(g, 1, seed, 0.1)[:, 0], device=dev))
        return None if V is None else {"V": V.cpu().numpy(), "iterations": None, "converged": None, "served": None}
    if g.n > EXACT_MAX_BUS:
        return None
    if kind == "series":
        V = _exact_columns(g, torch.view_as_complex(_hourly_injections(g, T, seed)))
        return None if V is None else {"V": torch.view_as_real(V), "iterations": None, "converged": None}
    V = _exact_columns(g, torch.as_tensor(_host_injections(g, T, seed), device=dev))
    if V is None:
        return None
    V = V.cpu().numpy()
    if kind == "study":
        return {"V": V}
    return {"V": V[:, 0] if kind == "solve" else V, "iterations": None, "converged": None}
