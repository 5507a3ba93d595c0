"""Performance cases of the LP solver: what its users run, at the sizes they run it.

A case is a dict of plain values:

  entry       "solve"     one LP through cupdlpx.solve (the drop-in solve, LP in host arrays)
              "resident"  one LP through DeviceProblem.solve (LP already in HBM)
              "batch"     `count` LPs of uneven sizes through cupdlpx.batch_solve
              "spmv"      y = A x through pdlp_spmv_noalloc on the caller's device buffers
  kind        structure of A: "random" (uniform positions), "powerlaw" (Zipf column degrees:
              columns of one entry up to columns of tens of thousands), "transport" (dense
              equal rows, two entries per column)
  m, n, nnz   rows, columns, non-zeros asked for (duplicates of the random positions are
              dropped, so a matrix holds slightly fewer); "transport" takes sources and sinks
  precision   "fp64", "fp32" (FP32 PDHG, then the FP64 finish) or "fp32m" (FP32 matrix only)
  iterations  the iteration limit.  A solve to 1e-4 takes from 1,000 (small random LPs) to
              55,000 iterations (the 20M-non-zero power-law LP); the limit makes the work of
              a pass known and keeps it short.  A mixed-precision solve keeps its last 600
              iterations for the FP64 finish.

LPs are made on the GPU from the seed alone and handed over as host arrays, as a caller has
them; all other parameters are the solver's defaults (presolve off: the library has none).
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "d-pdlp_gb300"))
import cupdlpx as cp  # noqa: E402

os.environ.setdefault("PDLP_QUIET", "1")  # no summary printed per solve

PRECISION = {"fp64": cp.PRECISION_FP64, "fp32": cp.PRECISION_FP32_REFINE,
             "fp32m": cp.PRECISION_FP32_MATRIX}
FINISH = 600       # iterations a mixed-precision solve keeps for its FP64 finish
PERIOD = 200       # evaluation and restart period (termination_evaluation_frequency)
L2_BYTES = 129e6


def listed():
    return [
        # An application's own loop around one small product: launches and the wait count.
        {"name": "spmv_random_20k", "entry": "spmv", "kind": "random",
         "m": 2000, "n": 5000, "nnz": 20000},
        # The same call on a matrix far larger than L2, rows of about 20.
        {"name": "spmv_powerlaw_20m", "entry": "spmv", "kind": "powerlaw",
         "m": 1000000, "n": 2000000, "nnz": 20000000},
        # ... and with every row thousands of non-zeros long (an assignment-type matrix).
        {"name": "spmv_transport_20m", "entry": "spmv", "kind": "transport",
         "sources": 2000, "sinks": 5000},
        # The smallest LP a caller sends: set-up and launches are all of it.
        {"name": "solve_tiny_fp64", "entry": "solve", "kind": "random",
         "m": 200, "n": 500, "nnz": 2000, "precision": "fp64", "iterations": 1000},
        # The small random LP the documentation solves, in both arithmetics.
        {"name": "solve_2k_fp64", "entry": "solve", "kind": "random",
         "m": 2000, "n": 5000, "nnz": 20000, "precision": "fp64", "iterations": 2000},
        {"name": "solve_2k_fp32", "entry": "solve", "kind": "random",
         "m": 2000, "n": 5000, "nnz": 20000, "precision": "fp32", "iterations": 1600},
        # An ordinary LP of a request stream, with odd sizes.
        {"name": "solve_40k_fp64", "entry": "solve", "kind": "random",
         "m": 39997, "n": 99991, "nnz": 999913, "precision": "fp64", "iterations": 1000},
        # The large LP of a request stream: its matrices (120 MB with A^T) just fit in L2.
        {"name": "solve_200k_fp32", "entry": "solve", "kind": "random",
         "m": 200000, "n": 500000, "nnz": 5000000, "precision": "fp32", "iterations": 1600},
        # The large power-law LP kept in HBM and solved again, as after a change of
        # tolerance or from a service that holds its model: both arithmetics.
        {"name": "resident_powerlaw_fp64", "entry": "resident", "kind": "powerlaw",
         "m": 1000000, "n": 2000000, "nnz": 20000000, "precision": "fp64", "iterations": 1000},
        {"name": "resident_powerlaw_fp32", "entry": "resident", "kind": "powerlaw",
         "m": 1000000, "n": 2000000, "nnz": 20000000, "precision": "fp32", "iterations": 1600},
        # The transportation LP: 10M columns of two entries, 7,000 long rows.
        {"name": "resident_transport_fp64", "entry": "resident", "kind": "transport",
         "sources": 2000, "sinks": 5000, "precision": "fp64", "iterations": 1000},
        # Uneven independent LPs solved side by side.
        {"name": "batch_16_fp32", "entry": "batch", "kind": "random", "count": 16,
         "m_min": 1000, "m_max": 100000, "precision": "fp32", "iterations": 1200},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["spmv", "spmv", "solve", "solve", "resident", "resident", "batch"])
    if entry == "batch":
        lo = _log(rng, 500, 3000)
        return {"entry": entry, "kind": "random", "count": rng.randint(3, 16), "m_min": lo,
                "m_max": _log(rng, 2 * lo, 100000), "precision": rng.choice(["fp64", "fp32"]),
                "iterations": 1200}
    case = {"entry": entry, "kind": rng.choice(["random", "random", "powerlaw", "transport"])}
    big = 20000000 if entry != "solve" else 5000000
    if case["kind"] == "transport":
        a = _log(rng, 20, 2000)
        case.update(sources=a, sinks=_log(rng, 20, min(5000, big // (2 * a))))
    else:
        nnz = _log(rng, 2000, big)
        # 3 to 40 non-zeros per column, 0.3 to 4 columns per row
        n = max(20, int(nnz / _log(rng, 3, 40)))
        case.update(m=max(10, int(n / rng.uniform(0.3, 4.0))), n=n, nnz=nnz)
        case["nnz"] = min(nnz, case["m"] * n // 4)
    if entry != "spmv":
        # a transportation LP's duals are free up to one constant, which drifts with the
        # rounding of FP32 iterates: its y says nothing there, so it is solved in FP64
        case["precision"] = ("fp64" if case["kind"] == "transport" else
                             rng.choice(["fp64", "fp32", "fp64", "fp32", "fp32m"]))
        case["iterations"] = PERIOD * rng.randint(3, 5)
        if case["precision"] != "fp64":
            case["iterations"] += FINISH
    return case


# ------------------------------------------------------------------- inputs
def _zipf_degrees(n, nnz, cap):
    """Column degrees clip(round(C rank^-1.2), 1, cap) that sum to about nnz."""
    base = np.arange(1, n + 1, dtype=np.float64) ** -1.2
    lo, hi = 0.0, 4.0 * nnz
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        if np.clip(np.round(mid * base), 1, cap).sum() < nnz:
            lo = mid
        else:
            hi = mid
    return np.clip(np.round(hi * base), 1, cap).astype(np.int64)


def _matrix(case, g):
    """(m, n, row pointers, columns, values) on the GPU, columns of a row ascending."""
    dev = "cuda"
    if case["kind"] == "transport":
        s, d = case["sources"], case["sinks"]
        m, n = s + d, s * d
        arcs = torch.arange(n, device=dev).reshape(s, d)
        col = torch.cat([arcs.reshape(-1), arcs.t().reshape(-1)]).int()
        row = torch.cat([torch.arange(s, device=dev).repeat_interleave(d),
                         s + torch.arange(d, device=dev).repeat_interleave(s)])
        val = torch.ones(2 * n, dtype=torch.float64, device=dev)
    else:
        m, n, nnz = case["m"], case["n"], case["nnz"]
        if case["kind"] == "powerlaw":
            deg = torch.from_numpy(_zipf_degrees(n, nnz, max(2, min(50000, m // 20)))).to(dev)
            deg = deg[torch.randperm(n, generator=g, device=dev)]
            c = torch.arange(n, device=dev).repeat_interleave(deg)
            r = torch.randint(m, (c.numel(),), generator=g, device=dev)
        else:
            c = torch.randint(n, (nnz,), generator=g, device=dev)
            r = torch.randint(m, (nnz,), generator=g, device=dev)
        key = torch.unique(r * n + c)
        row, col = key // n, (key % n).int()
        val = torch.randn(key.numel(), generator=g, device=dev, dtype=torch.float64)
        if case["kind"] == "powerlaw":
            ones = torch.rand(key.numel(), generator=g, device=dev) < 0.05
            val = torch.where(ones, torch.sign(val), val)
    ptr = torch.zeros(m + 1, dtype=torch.int32, device=dev)
    ptr[1:] = torch.bincount(row, minlength=m).cumsum(0)
    return m, n, ptr, col, val


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, size, lo, hi):
    return lo + (hi - lo) * torch.rand(size, generator=g, device="cuda", dtype=torch.float64)


def _lp(case, seed):
    """An LP with a feasible point, as host arrays: A in CSR, objective, bounds."""
    g = _generator(seed)
    m, n, ptr, col, val = _matrix(case, g)
    lp = {"m": m, "n": n, "ptr": ptr.cpu().numpy(), "col": col.cpu().numpy(),
          "val": val.cpu().numpy()}
    inf = math.inf
    if case["kind"] == "transport":
        supply = _uniform(g, case["sources"], 1.0, 100.0)
        demand = _uniform(g, case["sinks"], 1.0, 100.0)
        demand = demand * (supply.sum() / demand.sum())
        b = torch.cat([supply, demand]).cpu().numpy()
        lp.update(lc=b, uc=b.copy(), c=_uniform(g, n, 0.0, 1.0).cpu().numpy(),
                  lv=np.zeros(n), uv=np.full(n, inf))
        return lp
    x0 = _uniform(g, n, 0.0, 1.0).cpu().numpy()
    act = np.concatenate([lp["val"] * x0[lp["col"]], [0.0]])
    act = np.where(np.diff(lp["ptr"]) > 0, np.add.reduceat(act, lp["ptr"][:-1]), 0.0)
    eq = torch.rand(m, generator=g, device="cuda").cpu().numpy() < 0.3
    slack = _uniform(g, m, 0.0, 1.0).cpu().numpy()
    lp.update(lc=np.where(eq, act, act - slack), uc=np.where(eq, act, inf),
              c=_uniform(g, n, -1.0, 1.0).cpu().numpy(), lv=np.zeros(n), uv=np.full(n, 10.0))
    return lp


def _members(case, seed):
    """The LPs of a batch: rows spread evenly in log over [m_min, m_max], largest last."""
    k, r = case["count"], case["m_max"] / case["m_min"]
    sizes = [int(case["m_min"] * r ** (i / (k - 1))) for i in range(k)]
    return [({"kind": "random", "m": m, "n": 5 * m // 2, "nnz": 25 * m}, seed * 1000 + i)
            for i, m in enumerate(sizes)]


def _problem(lp):
    return cp.Problem.from_csr(lp["ptr"], lp["col"], lp["val"], lp["n"], c=lp["c"], lc=lp["lc"],
                               uc=lp["uc"], lv=lp["lv"], uv=lp["uv"])


def prepare(case, seed):
    if case["entry"] == "spmv":
        g = _generator(seed)
        m, n, ptr, col, val = _matrix(case, g)
        call = cp.lib().pdlp_spmv_noalloc
        call.restype = ctypes.c_int
        call.argtypes = [ctypes.c_int] * 3 + [ctypes.c_void_p] * 6
        return {"entry": "spmv", "call": call, "m": m, "n": n, "ptr": ptr, "col": col,
                "val": val, "x": torch.randn(n, generator=g, device="cuda", dtype=torch.float64),
                "y": torch.empty(m, device="cuda", dtype=torch.float64)}
    params = cp.default_parameters()
    params.presolve = False
    params.termination_criteria.iteration_limit = case["iterations"]
    state = {"entry": case["entry"], "params": params, "precision": PRECISION[case["precision"]]}
    if case["entry"] == "batch":
        state["problems"] = [_problem(_lp(c, s)) for c, s in _members(case, seed)]
    else:
        problem = _problem(_lp(case, seed))
        state["problem"] = problem if case["entry"] == "solve" else cp.DeviceProblem(problem)
    return state


# ------------------------------------------------------------------ a pass
def _outputs(r, precision):
    # the point of a mixed-precision solve carries the FP32 rounding of its rounds (the API
    # widens it to double), so it is returned in the precision it has
    kind = np.float64 if precision == cp.PRECISION_FP64 else np.float32
    return {"x": r["x"].astype(kind, copy=False), "y": r["y"].astype(kind, copy=False),
            "reduced_cost": r["rc"].astype(kind, copy=False),
            "primal_objective": kind(r["primal_objective_value"]),
            "dual_objective": kind(r["dual_objective_value"])}


def run(state):
    if state["entry"] == "spmv":
        s = state
        rc = s["call"](s["m"], s["n"], s["val"].numel(), s["ptr"].data_ptr(), s["col"].data_ptr(),
                       s["val"].data_ptr(), s["x"].data_ptr(), s["y"].data_ptr(),
                       torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError("pdlp_spmv_noalloc returned %d" % rc)
        return s["y"]
    p = state["precision"]
    if state["entry"] == "solve":
        out = cp.solve(state["problem"], state["params"], precision=p)
        return dict(_outputs(out.result, p), iterations=out.result["total_count"])
    if state["entry"] == "resident":
        out = state["problem"].solve(state["params"], precision=p)
        return dict(_outputs(out.result, p), iterations=out.result["total_count"])
    results, _ = cp.batch_solve(state["problems"], state["params"], precision=p)
    # three vectors per LP; their objectives together
    return {"points": [[o["x"], o["y"], o["reduced_cost"]]
                       for o in (_outputs(r, p) for r in results)],
            "objectives": np.array([r["primal_objective_value"] for r in results],
                                   np.float64 if p == cp.PRECISION_FP64 else np.float32),
            "iterations": np.array([r["total_count"] for r in results])}


# ------------------------------------------------------------------- work
def _sizes(case):
    if case["kind"] == "transport":
        s, d = case["sources"], case["sinks"]
        return s + d, s * d, 2 * s * d
    return case["m"], case["n"], case["nnz"]


def _solve_work(m, n, nnz, precision, iterations):
    """Host arrays in and results out once; beyond that, an iteration streams A and A^T, the
    other side's iterate twice and 7 n + 5 m vector entries -- from HBM where the matrices
    exceed L2, and on chip where they do not.  Set-up is left out (a few sweeps)."""
    low = max(0, iterations - FINISH) if precision != "fp64" else 0
    moved, flops = 12.0 * nnz + 4.0 * (m + 1) + 8.0 * (5 * n + 3 * m), 0.0
    for count, v, s in ((low, 4, 8 if precision == "fp32m" else 4), (iterations - low, 8, 8)):
        if 2.0 * nnz * (v + 4) > L2_BYTES:
            moved += count * (2.0 * nnz * (v + 4) + 4.0 * (m + n + 2) + s * (8.0 * n + 6.0 * m))
        flops += count * (4.0 * nnz + 10.0 * n + 9.0 * m)
    return moved, flops


def work(case):
    if case["entry"] == "spmv":
        m, n, nnz = _sizes(case)
        return {"bytes": 12.0 * nnz + 4.0 * (m + 1) + 8.0 * (m + n), "flops": 2.0 * nnz}
    members = [c for c, _ in _members(case, 0)] if case["entry"] == "batch" else [case]
    both = [_solve_work(*_sizes(c), case["precision"], case["iterations"]) for c in members]
    return {"bytes": sum(b for b, _ in both), "flops": sum(f for _, f in both)}


# ------------------------------------------------- the same in plain 64 bits
class _Lp64:
    """The LP on the GPU in FP64: matrices, vectors and their scalings."""

    def __init__(self, lp, scaled):
        t = lambda a: torch.from_numpy(a).to("cuda")  # noqa: E731
        self.m, self.n = lp["m"], lp["n"]
        self.ptr, self.col, self.val = t(lp["ptr"]).long(), t(lp["col"]).long(), t(lp["val"])
        self.row = torch.arange(self.m, device="cuda").repeat_interleave(self.ptr.diff())
        self.c, self.lv, self.uv, self.lc, self.uc = (t(lp[k])
                                                      for k in ("c", "lv", "uv", "lc", "uc"))
        b = torch.where(self.lc.isfinite() & (self.lc != self.uc), self.lc, 0.0)
        u = torch.where(self.uc.isfinite(), self.uc, 0.0)
        self.bnorm, self.cnorm = math.sqrt(float(b @ b + u @ u)), float(self.c.norm())
        self.Dr = torch.ones_like(self.lc)
        self.Dc = torch.ones_like(self.c)
        self.cb = self.ob = 1.0
        if scaled:
            self._scale()
        order = torch.argsort(self.col, stable=True)
        tptr = torch.zeros(self.n + 1, dtype=torch.long, device="cuda")
        tptr[1:] = torch.bincount(self.col, minlength=self.n).cumsum(0)
        self.A = torch.sparse_csr_tensor(self.ptr, self.col, self.val, (self.m, self.n))
        self.AT = torch.sparse_csr_tensor(tptr, self.row[order], self.val[order],
                                          (self.n, self.m))

    def _scale(self):
        for sweep in range(11):  # ten of Ruiz in the max norm, one of Pock-Chambolle
            a = self.val.abs()
            r, s = torch.zeros_like(self.lc), torch.zeros_like(self.c)
            if sweep < 10:
                r.scatter_reduce_(0, self.row, a, "amax")
                s.scatter_reduce_(0, self.col, a, "amax")
            else:
                r.index_add_(0, self.row, a)
                s.index_add_(0, self.col, a)
            r = torch.where(r < 1e-12, 1.0, r.sqrt())
            s = torch.where(s < 1e-12, 1.0, s.sqrt())
            self.val = self.val / (r[self.row] * s[self.col])
            self.c, self.lv, self.uv, self.Dc = self.c / s, self.lv * s, self.uv * s, self.Dc * s
            self.lc, self.uc, self.Dr = self.lc / r, self.uc / r, self.Dr * r
        b = torch.where(self.lc.isfinite() & (self.lc != self.uc), self.lc, 0.0)
        u = torch.where(self.uc.isfinite(), self.uc, 0.0)
        self.cb = 1.0 / (math.sqrt(float(b @ b + u @ u)) + 1.0)
        self.ob = 1.0 / (float(self.c.norm()) + 1.0)
        self.lc, self.uc = self.lc * self.cb, self.uc * self.cb
        self.lv, self.uv, self.c = self.lv * self.cb, self.uv * self.cb, self.c * self.ob

    def kkt(self, x, y, lam):
        """(relative primal and dual residuals and gap, primal and dual objectives)."""
        ax = self.A @ x
        p = float(((ax - ax.clamp(self.lc, self.uc)) * self.Dr).norm()) / self.cb
        d = float(((self.c - self.AT @ y - lam) * self.Dc).norm()) / self.ob
        zero = torch.zeros((), dtype=torch.float64, device="cuda")
        lo = torch.where(self.lc.isfinite(), self.lc, zero)
        up = torch.where(self.uc.isfinite(), self.uc, zero)
        po = float(self.c @ x) / (self.cb * self.ob)
        do = float(lam @ x + y.clamp(min=0.0) @ lo + y.clamp(max=0.0) @ up) / (self.cb * self.ob)
        return (p / (1.0 + self.bnorm), d / (1.0 + self.cnorm),
                abs(po - do) / (1.0 + abs(po) + abs(do)), po, do)


def _normals(count):
    """The solver's start vector of its power method: N(0,1) by Marsaglia's polar method from
    the Mersenne Twister with seed 1, two 32-bit words a uniform."""
    bits = np.random.MT19937()
    bits._legacy_seeding(1)
    have, out = 0, []
    while have < count:
        w = bits.random_raw(4 * (count + 64)).astype(np.float64).reshape(-1, 4)
        u = 2.0 * ((w[:, 0::2] + w[:, 1::2] * 2.0 ** 32) / 2.0 ** 64) - 1.0
        r2 = u[:, 0] ** 2 + u[:, 1] ** 2
        ok = (r2 <= 1.0) & (r2 != 0.0)
        u, r2 = u[ok], r2[ok]
        out.append((u[:, ::-1] * np.sqrt(-2.0 * np.log(r2) / r2)[:, None]).reshape(-1))
        have += out[-1].size
    return np.concatenate(out)[:count]


def _sigma(P):
    v = torch.from_numpy(_normals(P.m)).to("cuda")
    v = v / v.norm()
    for _ in range(5000):
        w = P.A @ (P.AT @ v)
        s = float(v @ w)
        if float((w - s * v).norm()) < 1e-4:
            break
        v = w / w.norm()
    return math.sqrt(s)


def _cadence(t):
    step = 10
    while t >= 100 * step:
        step *= 10
    return step


def _pdhg(P, limit, sigma, start=None, keep_best=False):
    """Restarted Halpern PDHG in FP64 for `limit` iterations or to 1e-4.  Returns the final
    (or, with keep_best, the best evaluated) x, y and dual slack, scaled, and the count."""
    z = lambda v: torch.zeros_like(v)  # noqa: E731
    x, y = (z(P.c), z(P.lc)) if start is None else (start[0] * P.Dc * P.cb,
                                                    start[1] * P.Dr * P.ob)
    x0, y0, xh, yh, lam = x, y, x, y, z(P.c)
    eta, omega = 0.998 / sigma, 1.0
    best_gap, best_omega, err_sum, err_last = math.inf, 1.0, 0.0, 0.0
    fpe, fpe0, trial, since = 0.0, 0.0, math.inf, 0
    best, t = (math.inf, xh, yh, lam), 0
    while True:
        top, restart = t > 0 and t % PERIOD == 0, False
        if t == limit or top or t % _cadence(t) == 0:
            rp, rd, rg, _, _ = P.kkt(xh, yh, lam)
            if t < limit and max(rp, rd, rg) < best[0]:
                best = (max(rp, rd, rg), xh, yh, lam)
            if t == limit or max(rp, rd, rg) < 1e-4:
                break
            if top:
                restart = (t == PERIOD or fpe <= 0.2 * fpe0 or
                           (fpe <= 0.5 * fpe0 and fpe > trial) or t - since >= 0.36 * t)
            if top or t == 0:
                trial = fpe
        if restart:
            pd, dd = float((xh - x0).norm()), float((yh - y0).norm())
            ratio = rd / rp if rp > 0.0 else math.inf
            if 1e-16 < pd < 1e12 and 1e-16 < dd < 1e12 and 1e-8 < ratio < 1e8:
                e = math.log(dd) - math.log(pd) - math.log(omega)
                err_sum = 0.3 * err_sum + e
                omega *= math.exp(0.99 * e + 0.01 * err_sum)
                err_last = e
            else:
                omega, err_sum, err_last = best_omega, 0.0, 0.0
            gap = abs(math.log10(ratio)) if 0.0 < ratio < math.inf else math.inf
            if gap < best_gap:
                best_gap, best_omega = gap, omega
            x = x0 = xh
            y = y0 = yh
            since, trial = t, math.inf
        tau, step = eta / omega, eta * omega
        w = (t - since + 1) / (t - since + 2)
        g = x - tau * (P.c - P.AT @ y)
        xn = g.clamp(P.lv, P.uv)
        ref = 2.0 * xn - x
        h = y / step - P.A @ ref
        yn = step * (h - h.clamp(-P.uc, -P.lc))
        yref = 2.0 * yn - y
        ends = (t + 1) % PERIOD == 0
        if ends or (t + 2) % _cadence(t + 2) == 0:
            xh, yh, lam = xn, yn, (xn - g) / tau
        if ends or restart:
            dx, dy = ref - x, yref - y
            fpe = math.sqrt(float(dx @ dx) * omega + float(dy @ dy) / omega
                            + 2.0 * eta * float((P.AT @ dy) @ dx))
            if restart:
                fpe0 = fpe
        x, y = w * ref + (1.0 - w) * x0, w * yref + (1.0 - w) * y0
        t += 1
    return (best[1:] if keep_best else (xh, yh, lam)) + (t, max(rp, rd, rg) < 1e-4)


def _solve64(lp, precision, limit):
    P = _Lp64(lp, True)
    sigma = _sigma(P)
    if precision == "fp64":
        xh, yh, lam, t, _ = _pdhg(P, limit, sigma)
        po, do = P.kkt(xh, yh, lam)[3:]
        return {"x": xh / P.Dc / P.cb, "y": yh / P.Dr / P.ob,
                "reduced_cost": (P.c - P.AT @ yh) * P.Dc / P.ob,
                "primal_objective": np.float64(po), "dual_objective": np.float64(do),
                "iterations": t}
    # the FP32 round's best point, then the FP64 finish from there
    U = _Lp64(lp, False)
    first = limit - min(3 * PERIOD, limit // 2)
    xh, yh, lam, t, met = _pdhg(P, first, sigma, keep_best=True)
    x, y = xh / P.Dc / P.cb, yh / P.Dr / P.ob
    if not met:
        xh, yh, lam, t2, _ = _pdhg(P, limit - t, sigma, start=(x, y))
        x, y, t = xh / P.Dc / P.cb, yh / P.Dr / P.ob, t + t2
    rc = U.c - U.AT @ y
    lo, up = U.lv.isfinite(), U.uv.isfinite()
    slack = torch.where(lo & up, rc, torch.where(lo, rc.clamp(min=0.0),
                                                 torch.where(up, rc.clamp(max=0.0), 0.0)))
    k = U.kkt(x, y, slack)
    if not met and max(k[:3]) >= 1e-4:
        k2 = U.kkt(x, y, lam * P.Dc / P.ob)
        k = k2 if max(k2[:3]) < max(k[:3]) else k
    return {"x": x, "y": y, "reduced_cost": rc, "primal_objective": np.float64(k[3]),
            "dual_objective": np.float64(k[4]), "iterations": t}


def exact(case, seed):
    if case["entry"] == "spmv":
        g = _generator(seed)
        m, n, ptr, col, val = _matrix(case, g)
        x = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
        return torch.sparse_csr_tensor(ptr.long(), col.long(), val, (m, n)) @ x
    if case["entry"] != "batch":
        return _solve64(_lp(case, seed), case["precision"], case["iterations"])
    all64 = [_solve64(_lp(c, s), case["precision"], case["iterations"])
             for c, s in _members(case, seed)]
    return {"points": [[r["x"], r["y"], r["reduced_cost"]] for r in all64],
            "objectives": np.array([r["primal_objective"] for r in all64]),
            "iterations": np.array([r["iterations"] for r in all64])}
