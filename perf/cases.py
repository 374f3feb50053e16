"""Performance cases: the calls that a calibration makes of this framework.

Every flow case goes through ``ForwardBatch.evaluate`` (one mesh class),
``evaluate_fields`` (rows plus final fields) or ``evaluate_multi`` (several classes in
one call): coefficients from host memory in, rows and predictions back in host memory.
The outer iterations are capped (except in the smallest case, which runs to its
verdict): a whole Re_tau 1000 solve takes about a minute, and its outer iterations are
alike. The caps of the channels also end before the cold start's unsteady phase, which
amplifies last-digit differences of the sums a millionfold before the steady state
damps them again: up to there two orders of the same sums agree to 1e-12. Linear cases
go through ``LinearBatch.solve``, whose operators and hierarchies stay on the device
between solves.

The mixed form of the flow solve is left out: it measured slower than FP64 on every
mesh class, so FP64 is the default and what a calibration runs. The mixed form of the
linear solves is in.
"""
import math

import numpy as np
import torch

from rans_uq_b200 import core, linear, workloads

LINEAR_TOL = 1e-10
LINEAR_MAX_ITER = 500


def listed():
    return [
        # one draw on the smallest mesh, solved to its verdict: a notebook's first call
        {"name": "small_to_verdict", "kind": "channel", "re_tau": 182.088, "ny": 24, "draws": 1,
         "iters": 60000, "yplus": 1.0, "tol": 1e-8, "alpha_u": 0.7},
        # the sequential model: one draw of the calibration's own class
        {"name": "re182_one", "kind": "channel", "re_tau": 182.088, "ny": 128, "draws": 1,
         "iters": 40, "yplus": 0.5, "tol": 1e-10, "alpha_u": 0.8},
        # the uniform design that opens a calibration (24 draws)
        {"name": "re182_design", "kind": "channel", "re_tau": 182.088, "ny": 128, "draws": 24,
         "iters": 60, "yplus": 0.5, "tol": 1e-8, "alpha_u": 0.5},
        # the 5 x 5 Laplace grid on the middle class
        {"name": "re550_grid", "kind": "channel", "re_tau": 550.0, "ny": 256, "draws": 25,
         "iters": 200, "yplus": 0.5, "tol": 1e-8, "alpha_u": 0.8},
        # an importance sample of 64 draws on the largest channel class
        {"name": "re1000_importance", "kind": "channel", "re_tau": 1000.0, "ny": 512, "draws": 64,
         "iters": 200, "yplus": 0.5, "tol": 1e-8, "alpha_u": 0.8},
        # the benchmark's ensemble: 256 draws over the three classes in one call
        {"name": "ensemble", "kind": "ensemble", "draws": 256, "iters": 40},
        # odd sizes: a poll of the 3 x 3 pattern search on a mesh of odd width and height
        {"name": "odd_poll", "kind": "channel", "re_tau": 395.0, "ny": 181, "nx": 5, "draws": 9,
         "iters": 60, "yplus": 0.7, "tol": 1e-8, "alpha_u": 0.8},
        # bump-wall channel, coarse, with the final fields (plots, snapshots)
        {"name": "bump_coarse_fields", "kind": "bump", "nx": 24, "ny": 16, "draws": 9,
         "iters": 100},
        # bump-wall channel of the serving mix
        {"name": "bump_medium", "kind": "bump", "nx": 100, "ny": 50, "draws": 8, "iters": 40},
        # bump-wall channel of the batched benchmark: 32 draws on 200 x 100 cells
        {"name": "bump_full", "kind": "bump", "nx": 200, "ny": 100, "draws": 32, "iters": 14},
        # Poisson systems of uneven size, AMG-preconditioned PCG in FP64
        {"name": "linear_batch", "kind": "linear", "systems": 16, "n_min": 64, "n_max": 512,
         "precision": "fp64"},
        # one system at a time, FP32 corrections inside FP64 refinement
        {"name": "linear_mixed_one", "kind": "linear", "systems": 1, "n_min": 128, "n_max": 128,
         "precision": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["verdict", "channel", "channel", "channel", "ensemble", "bump", "bump",
                       "linear"])
    if kind == "verdict":
        return {"kind": "channel", "re_tau": rng.uniform(175.0, 190.0), "nx": 3, "ny": 24,
                "draws": _log_int(rng, 1, 32), "iters": 60000, "yplus": 1.0, "tol": 1e-5,
                "alpha_u": 0.7}
    if kind == "channel":
        nx, ny = rng.choice([3, 3, 3, 4, 5]), _log_int(rng, 40, 512)
        while nx * ny > 1536:
            ny = _log_int(rng, 40, 512)
        return {"kind": "channel", "re_tau": rng.uniform(150.0, 1000.0), "nx": nx, "ny": ny,
                "draws": _log_int(rng, 1, 256), "yplus": rng.uniform(0.5, 1.0), "tol": 1e-8,
                "iters": rng.randint(20, 40), "alpha_u": 0.5}
    if kind == "ensemble":
        return {"kind": "ensemble", "draws": _log_int(rng, 12, 256), "iters": rng.randint(15, 40)}
    if kind == "bump":
        nx = _log_int(rng, 20, 200)
        ny = max(12, int(nx * rng.uniform(0.4, 0.7)))
        return {"kind": "bump", "nx": nx, "ny": ny, "draws": _log_int(rng, 1, 32),
                "iters": max(6, min(100, int(120000 / (nx * ny + 600))))}
    lo = _log_int(rng, 48, 256)
    return {"kind": "linear", "systems": _log_int(rng, 1, 12), "n_min": lo,
            "n_max": rng.randint(lo, min(512, 2 * lo)), "precision": rng.choice(["fp64", "mixed"])}


# ---------------------------------------------------------------- inputs
def _profile(re_tau, yplus):
    """A smooth mean-velocity profile in wall units (Reichardt), as observed data."""
    y = np.asarray(yplus)
    return (np.log(1 + 0.41 * y) / 0.41 +
            7.8 * (1 - np.exp(-y / 11.0) - y / 11.0 * np.exp(-y / 3.0)))


def _channel(case, rng):
    re_tau = case["re_tau"]
    mesh = core.Mesh.make_periodic_channel_2d(case.get("nx", 3), case["ny"], 1.0, 1.0, re_tau,
                                              case["yplus"])
    mesh.compute_wall_distance()
    yp = np.geomspace(2.0, 0.8 * min(re_tau, 175.0 / 0.8), 30)
    u = _profile(re_tau, yp) * (1 + 0.0014 * rng.standard_normal(len(yp)))
    obs = core.ObservationOperator()
    for y, ui in zip(yp / re_tau, u):
        obs.add_velocity_profile(core.Vec3(0.5, float(y), 0.0), 0, float(ui), 0.0014 * abs(ui))
    st = core.SolverSettings(max_iterations=case["iters"], convergence_tol=case["tol"],
                             alpha_u=case["alpha_u"], body_force=core.Vec3(1.0, 0.0, 0.0),
                             verbose=False)
    bcs = core.FlowBoundaryConditions.channel_defaults(mesh, 1.0, 1.0, 10.0)
    return core.ForwardBatch(mesh, core.InferenceParameterSet.a1_betaStar(), obs, bcs,
                             1.0 / re_tau, st, core.Vec3(15.0, 0.0, 0.0), 0.0, 1.0, 10.0)


def _theta(rng, n):
    return rng.uniform(workloads.BOX_LO, workloads.BOX_HI, (n, 2))


def _sizes(case, rng):
    """Grid sides of a linear case: the largest first, the rest spread over the range."""
    lo, hi = case["n_min"], case["n_max"]
    rest = np.exp(rng.uniform(math.log(lo), math.log(hi), case["systems"] - 1))
    return [hi] + [int(round(v)) for v in rest]


def _systems(case, seed):
    # the grid sides belong to the case (equal work for every seed), the coefficients
    # and right-hand sides to the seed
    sizes = _sizes(case, np.random.default_rng(case["systems"] * 1000 + case["n_max"]))
    return [workloads.poisson_system(n, seed * 1000 + k) for k, n in enumerate(sizes)]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "channel":
        return {"kind": kind, "batch": _channel(case, rng), "theta": _theta(rng, case["draws"])}
    if kind == "ensemble":
        batches = []
        for c, (re_tau, ny) in enumerate(workloads.CLASSES):
            u = workloads.stored_truth(c)
            u = u * (1 + workloads.NOISE * rng.standard_normal(len(u)))
            batches.append(workloads.channel_batch(re_tau, ny, u, workloads.NOISE * np.abs(u),
                                                   max_iter=case["iters"]))
        return {"kind": kind, "batches": batches, "theta": _theta(rng, case["draws"]),
                "cls": np.arange(case["draws"]) % len(batches)}
    if kind == "bump":
        return {"kind": kind, "batch": workloads.bump_batch(case["nx"], case["ny"], case["iters"]),
                "theta": _theta(rng, case["draws"])}
    return {"kind": kind,
            "batch": linear.LinearBatch(_systems(case, seed), "AMG", case["precision"])}


# ---------------------------------------------------------------- one pass
def _rows(res):
    return {"loglik": np.asarray(res.log_likelihoods), "pred": np.asarray(res.predictions),
            "status": np.array([int(s) for s in res.statuses]),
            "iterations": np.asarray(res.iteration_counts)}


def run(state):
    kind = state["kind"]
    if kind == "channel":
        return _rows(state["batch"].evaluate(state["theta"]))
    if kind == "ensemble":
        return _rows(core.evaluate_multi(state["batches"], state["cls"], state["theta"]))
    if kind == "bump":
        res, fields, _ = state["batch"].evaluate_fields(state["theta"])
        return {**_rows(res), "fields": fields}
    results, xs = state["batch"].solve(LINEAR_MAX_ITER, LINEAR_TOL)
    return {"x": np.concatenate(xs), "iterations": np.array([r.iterations for r in results]),
            "converged": np.array([int(r.converged) for r in results])}


# ---------------------------------------------------------------- least work
def _flow_work(cells, draws, iters):
    # one outer iteration reads and writes, per cell, about 200 arrays outside the inner
    # solvers, and its inner solvers pass about 9 BiCGSTAB iterations of 45 arrays and 2
    # AMG-PCG iterations of 50; a multiply and an add per value
    values = float(cells) * draws * iters * (200 + 9 * 45 + 2 * 50)
    return {"bytes": 8.0 * values, "flops": 2.0 * values}


def work(case):
    kind = case["kind"]
    if kind == "channel":
        iters = min(case["iters"], 3000)
        return _flow_work(case.get("nx", 3) * case["ny"], case["draws"], iters)
    if kind == "ensemble":
        parts = [_flow_work(3 * ny, len(range(c, case["draws"], len(workloads.CLASSES))),
                            case["iters"])
                 for c, (_, ny) in enumerate(workloads.CLASSES)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "bump":
        return _flow_work(case["nx"] * case["ny"], case["draws"], case["iters"])
    sizes = _sizes(case, np.random.default_rng(case["systems"] * 1000 + case["n_max"]))
    rows = float(sum(n * n for n in sizes))
    # per PCG iteration: five passes of a 5-point matrix (12 bytes an entry, 1.6 over the
    # levels) and about 32 vector passes; about 30 iterations
    return {"bytes": 30 * rows * (5 * 5 * 12 * 1.6 + 32 * 8), "flops": 30 * rows * (50 * 1.6 + 32)}


# ---------------------------------------------------------------- 64-bit solution
def _line_solve(system, n):
    """Direct solution of an n x n grid system (block elimination along grid lines, FP64)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    diag = torch.from_numpy(system.diag).reshape(n, n).to(dev)
    rhs = torch.from_numpy(system.source).reshape(n, n).to(dev)
    cx = torch.from_numpy(system.upper[:n * (n - 1)].copy()).reshape(n, n - 1).to(dev)
    cy = torch.from_numpy(system.upper[n * (n - 1):].copy()).reshape(n - 1, n).to(dev)
    inv, carry = [], []
    for j in range(n):
        block = torch.diag(diag[j]) + torch.diag(cx[j], 1) + torch.diag(cx[j], -1)
        r = rhs[j]
        if j:
            block = block - cy[j - 1][:, None] * inv[-1] * cy[j - 1][None, :]
            r = r - cy[j - 1] * carry[-1]
        inv.append(torch.linalg.inv(block))
        carry.append(inv[-1] @ r)
    x = [carry[-1]]
    for j in range(n - 2, -1, -1):
        x.append(carry[j] - inv[j] @ (cy[j] * x[-1]))
    return torch.cat(x[::-1]).cpu().numpy()


def exact(case, seed):
    """The direct solutions of a linear case; a flow solve has no plain 64-bit value within
    a few seconds."""
    if case["kind"] != "linear":
        return None
    sizes = _sizes(case, np.random.default_rng(case["systems"] * 1000 + case["n_max"]))
    if sum(sizes) > 6000:
        return None
    xs = [_line_solve(s, n) for s, n in zip(_systems(case, seed), sizes)]
    return {"x": np.concatenate(xs), "iterations": None, "converged": None}
