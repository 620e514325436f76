"""The work that users of the framework have it do, as cases that can be timed.

Every case goes through the package's public entry points: `Solver` and
`BatchSolver` (the steady iteration in its precisions, the unsteady stage, the
chemistry integrator) and `surrogate.MLP` (inference and training).  Meshes,
physics and sizes are those of the presets of `rocketcombustor_gb300.cases`, of
the benchmark and of the tests.

A steady pass is what a driver does between two looks at the residual: the
state goes in from page-locked host memory, some iterations run, the norms are
read and the state comes back.  Solvers take the launch configuration that they
have by default, as the steady driver `Case.run_steady` does.  Case directories
are written once per machine, cases and solvers opened once per process, as a
program that runs many states on one mesh does; the states come from the seed.
"""
from __future__ import annotations

import functools
import hashlib
import json
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import rocketcombustor_gb300 as rc
from rocketcombustor_gb300 import cases as nozzles
from rocketcombustor_gb300 import surrogate

PRECISION = {"fp64": rc.RC_PREC_FP64, "mixed": rc.RC_PREC_MIXED, "mixed_dc": rc.RC_PREC_MIXED_DC}


def listed():
    return [
        # the smallest steady case of the tests, 720 quadrilaterals: launches and latency
        {"name": "steady_720", "kind": "steady", "preset": "s2t", "nx": 60, "ny": 12, "order": "natural",
         "precision": "fp64", "iters": 10},
        # one perfect gas without viscosity or chemistry, 20,000 triangles
        {"name": "steady_gas_20k", "kind": "steady", "preset": "c1", "nx": 250, "ny": 40, "order": "natural",
         "precision": "fp64", "iters": 10},
        # the reacting viscous nozzle at its usual size, plain and mixed precision
        {"name": "steady_120k", "kind": "steady", "preset": "c2", "nx": 600, "ny": 100, "order": "natural",
         "precision": "fp64", "iters": 10},
        {"name": "mixed_120k", "kind": "steady", "preset": "c2", "nx": 600, "ny": 100, "order": "natural",
         "precision": "mixed", "iters": 10},
        # the benchmark's mesh of two million triangles, plain and mixed precision
        {"name": "steady_2m", "kind": "steady", "preset": "c4", "nx": 2500, "ny": 400, "order": "natural",
         "precision": "fp64", "iters": 10},
        {"name": "mixed_2m", "kind": "steady", "preset": "c4", "nx": 2500, "ny": 400, "order": "natural",
         "precision": "mixed", "iters": 10},
        # a design study: 64 uneven nozzles in one context with the integrated chemistry
        {"name": "batch_64", "kind": "batch", "n": 64, "ne_min": 2000, "ne_max": 60000, "precision": "fp64",
         "iters": 5},
        {"name": "batch_64_mixed", "kind": "batch", "n": 64, "ne_min": 2000, "ne_max": 60000, "precision": "mixed",
         "iters": 5},
        # the shipped unsteady scheme: two physical steps of dual-time BDF2
        {"name": "bdf2_120k", "kind": "bdf2", "nx": 600, "ny": 100, "steps": 2},
        # labelling training states with the integrator at the data set's tolerance
        {"name": "chem_256k", "kind": "chem", "n": 262144, "tol": 0.005, "max_substeps": 2000},
        # surrogate inference over a large set of states
        {"name": "mlp_forward_4m", "kind": "mlp_forward", "n": 4194304},
        # surrogate training at the benchmark's batch size
        {"name": "mlp_train_8192", "kind": "mlp_train", "n": 1048576, "steps": 200, "batch": 8192},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["steady"] * 5 + ["batch", "bdf2", "chem", "mlp_forward", "mlp_train"])
    if kind == "steady":
        preset = rng.choice(["c2", "c2", "c4", "c1", "s2"])
        cells = _log(rng, 300, 1.2e6 if preset == "s2" else 2.0e6)
        ny = max(3, round(math.sqrt(cells / (6.0 * (1 if preset == "s2" else 2)) * rng.uniform(0.5, 2.0))))
        nx = max(8, int(cells / ((1 if preset == "s2" else 2) * ny)))
        precision = rng.choice(["fp64", "fp64", "mixed", "mixed", "mixed_dc"])
        # the mesh generators of the presets order cells column by column; other
        # generators do not ("colored" is written cell by cell: small meshes only)
        orders = ["natural"] * 4 + ["random"] + (["colored"] if preset != "s2" and cells < 1e5 else [])
        return {"kind": "steady", "preset": preset, "nx": nx, "ny": ny, "order": rng.choice(orders),
                "precision": precision, "iters": rng.choice([1, 10])}
    if kind == "batch":
        lo = int(_log(rng, 300, 6000))
        return {"kind": "batch", "n": rng.randint(2, 40), "ne_min": lo, "ne_max": int(lo * rng.uniform(1.5, 10.0)),
                "precision": rng.choice(["fp64", "mixed"]), "iters": 5}
    if kind == "bdf2":
        cells = _log(rng, 300, 1.2e5)
        ny = max(3, round(math.sqrt(cells / 12.0 * rng.uniform(0.5, 1.5))))
        return {"kind": "bdf2", "nx": max(8, int(cells / (2 * ny))), "ny": ny, "steps": rng.choice([1, 2])}
    if kind == "chem":
        tol, most = rng.choice([(0.05, 200), (0.005, 2000)])
        return {"kind": "chem", "n": int(_log(rng, 1, 262144)), "tol": tol, "max_substeps": most}
    if kind == "mlp_forward":
        return {"kind": "mlp_forward", "n": int(_log(rng, 1, 4194304))}
    return {"kind": "mlp_train", "n": int(_log(rng, 20000, 1048576)), "steps": rng.randint(50, 200),
            "batch": 128 * int(_log(rng, 1, 128))}


# ------------------------------------------------------------ cases, solvers ---
def _directory(what, write):
    """The case directory (or directories) that `write(path)` makes, kept on this machine's disk by what it holds."""
    key = hashlib.sha256(json.dumps(what, sort_keys=True).encode()).hexdigest()[:20]
    root = os.path.join(tempfile.gettempdir(), "nozzle_cases_%d" % os.getuid())
    os.makedirs(root, mode=0o700, exist_ok=True)
    path = os.path.join(root, key)
    if not os.path.isdir(path):
        new = tempfile.mkdtemp(dir=root)
        write(new)
        try:
            os.rename(new, path)
        except OSError:  # another process was first
            shutil.rmtree(new)
    return path


@functools.lru_cache(maxsize=None)
def _one(preset, nx, ny, order):
    over = {"nx": nx, "ny": ny, "order": order}
    return rc.Case(_directory([preset, over], lambda d: nozzles.make_case(d, preset, **over)))


@functools.lru_cache(maxsize=None)
def _many(n, ne_min, ne_max):
    over = {"ne_min": ne_min, "ne_max": ne_max}
    d = _directory(["batch", n, over], lambda d: nozzles.make_batch(d, n, **over))
    return [rc.Case(os.path.join(d, name)) for name in sorted(os.listdir(d))]


@functools.lru_cache(maxsize=None)
def _solver(preset, nx, ny, order, precision):
    return rc.Solver(_one(preset, nx, ny, order), precision=PRECISION[precision])


@functools.lru_cache(maxsize=None)
def _batch_solver(n, ne_min, ne_max, precision):
    s = rc.BatchSolver(_many(n, ne_min, ne_max), precision=PRECISION[precision])
    s.set_chemistry(rc.RC_CHEM_INTEGRATED)
    return s


# ------------------------------------------------------------------- inputs ---
def _pinned(shape):
    """Page-locked host memory as an array."""
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _state(case_list, seed):
    """The cases' initial states with smooth pressure waves of up to 1 % at constant temperature, which scale
    every conserved variable by the same factor."""
    rng = np.random.default_rng(seed)
    ne = sum(c.NE for c in case_list)
    P, W = (_pinned((ne, case_list[0].NVar)) for _ in range(2))
    at = 0
    for c in case_list:
        xy, sl = c.array("CELLXY"), slice(at, at + c.NE)
        f = np.ones(c.NE)
        for _ in range(3):
            k = rng.uniform(-1.0, 1.0, 2) * 2.0 * math.pi * np.array([8.0, 25.0])
            f += 0.0033 * np.sin(xy @ k + rng.uniform(0.0, 2.0 * math.pi))
        np.copyto(P[sl], c.array("PA"))
        P[sl, 0] *= f
        np.multiply(c.array("WA"), f[:, None], out=W[sl])
        at += c.NE
    return P, W


def _samples(n, seed):
    """n states (pool of the tiny reacting nozzle's, T, p and dt over the surrogate's domain) and their dt."""
    P = torch.tensor(_one("t2", 24, 6, "natural").array("PA").T.copy(), device="cuda")
    return surrogate.sample_states(P, n, seed)


def _features(n, seed):
    """Raw network inputs (T, p, Y_1..Y_4, dt)."""
    P, dt = _samples(n, seed)
    last = 1.0 - P[4:].sum(0)
    return torch.stack([P[3], P[0], P[4], P[5], P[6], last, dt], 1).float().contiguous()


def _features64(x):
    """1000/T, log10 p, log10(Y + 1e-10), log10 dt in 64 bits."""
    x = x.double()
    return torch.cat([1000.0 / x[:, :1].clamp_min(1.0), x[:, 1:2].clamp_min(1e-30).log10(),
                      (x[:, 2:6].clamp_min(0.0) + 1e-10).log10(), x[:, 6:].clamp_min(1e-30).log10()], 1)


@functools.lru_cache(maxsize=None)
def _norm():
    """The training set's feature mean and standard deviation."""
    f = _features64(_features(65536, 1))
    std = f.std(0)
    return f.mean(0).cpu().numpy(), torch.where(std > 1e-6, std, torch.ones_like(std)).cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("steady", "batch"):
        if kind == "steady":
            key = (case["preset"], case["nx"], case["ny"], case["order"])
            solver, cs = _solver(*key, case["precision"]), [_one(*key)]
        else:
            key = (case["n"], case["ne_min"], case["ne_max"])
            solver, cs = _batch_solver(*key, case["precision"]), _many(*key)
        P, W = _state(cs, seed)
        return {"kind": kind, "solver": solver, "P": P, "W": W, "out": (_pinned(P.shape), _pinned(P.shape)),
                "iters": case["iters"]}
    if kind == "bdf2":
        key = ("c2u", case["nx"], case["ny"], "natural")
        c = _one(*key)
        P, W = _state([c], seed)
        u = c.unsteady
        return {"kind": kind, "solver": _solver(*key, "fp64"), "P": P, "W": W,
                "out": (_pinned(P.shape), _pinned(P.shape)), "steps": case["steps"], "dt": u["dt"],
                "inner_loop": u["inner_loop"], "rel_tol": u["rel_tol"]}
    if kind == "chem":
        P, dt = _samples(case["n"], seed)
        return {"kind": kind, "solver": _solver("t2", 24, 6, "natural", "fp64"), "P": P, "dt": dt,
                "tol": case["tol"], "max_substeps": case["max_substeps"]}
    x = _features(case["n"], seed)
    net = surrogate.MLP(seed=seed)
    net.set_norm(*_norm())
    if kind == "mlp_forward":
        return {"kind": kind, "net": net, "x": x}
    # targets near those of the integrator: z close to 1, falling where the Damkoehler number is large
    t = torch.sigmoid(3.0 - _features64(x)[:, [0, 1, 6]].float().sum(1, keepdim=True) * 0.25)
    return {"kind": kind, "net": net, "x": x, "t": t.repeat(1, 4).contiguous(), "p": surrogate.init_params(seed),
            "steps": case["steps"], "batch": case["batch"], "seed": seed}


def run(state):
    kind = state["kind"]
    if kind in ("steady", "batch"):
        s = state["solver"]
        s.set_state(state["P"], state["W"])
        for it in range(1, state["iters"] + 1):
            s.lu_sgs_stage(it)
        res, romax = s.residual()
        P, W = s.get_state(*state["out"])
        return {"P": P, "W": W, "res": res, "romax": romax}
    if kind == "bdf2":
        s = state["solver"]
        s.set_state(state["P"], state["W"])
        inner = [s.bdf2_stage(k, state["dt"], state["inner_loop"], state["rel_tol"])
                 for k in range(1, state["steps"] + 1)]
        res, romax = s.residual()
        P, W = s.get_state(*state["out"])
        return {"P": P, "W": W, "res": res, "romax": romax, "inner": inner}
    if kind == "chem":
        P, nsub = state["solver"].chem_integrate(state["P"], state["dt"], state["tol"], state["max_substeps"])
        return {"P": P, "substeps": nsub}
    if kind == "mlp_forward":
        return state["net"].forward(state["x"])
    net = state["net"]
    net.set_params(state["p"])
    loss = net.train(state["x"], state["t"], state["steps"], state["batch"], seed=state["seed"], log_every=1)
    return {"loss": np.array([v for _, v in loss], dtype=np.float32), "params": net.get_params()}


# --------------------------------------------------------------- work, exact ---
def work(case):
    kind = case["kind"]
    if kind in ("steady", "batch", "bdf2"):
        if kind == "batch":
            over = {"ne_min": case["ne_min"], "ne_max": case["ne_max"]}
            cells, nvar, faces = sum(c.n_cells for c in nozzles.batch_configs(case["n"], **over)), 7, 1.5
        else:
            preset = nozzles.PRESETS[case.get("preset", "c2u")]
            quads = preset.quads
            cells = (1 if quads else 2) * case["nx"] * case["ny"]
            nvar, faces = 3 + preset.nsp, 2.0 if quads else 1.5
        # per iteration and cell: the state read and written, and the geometry read once (volume, length scales,
        # least-squares and limiter coefficients, indices; per face the vectors and the Gauss-point basis)
        byte = 4 * 8 * nvar + 8 * (3 + 8 + 8 + 4) + 32 + faces * (8 * 16 + 8)
        # floating-point operations of one iteration per cell: about 4,000 for the four reacting viscous species (a
        # third of them in exp, log and pow), 500 for the perfect gas; the unsteady cell solves add 1,500
        flop = (4000 if nvar > 4 else 500) + (1500 if kind == "bdf2" else 0)
        n = case["iters"] if kind != "bdf2" else 3 * case["steps"]
        return {"bytes": float(n * cells * byte + 4 * 8 * nvar * cells), "flops": float(n * cells * flop)}
    if kind == "chem":
        # about 45 (tolerance 0.005) or 6 (0.05) substeps of 600 operations
        return {"bytes": 124.0 * case["n"], "flops": 600.0 * (45 if case["tol"] < 0.01 else 6) * case["n"]}
    if kind == "mlp_forward":
        return {"bytes": 44.0 * case["n"], "flops": 101120.0 * case["n"]}
    k = case["steps"] * min(case["batch"], case["n"])
    return {"bytes": 44.0 * k + 6 * 4 * 51076.0 * case["steps"], "flops": 3 * 101120.0 * k}


def _forward64(p, x, mean, std):
    f = (_features64(x) - mean) / std
    for k in range(5):
        w, b = p["W%d" % k], p["b%d" % k]
        f = f @ w.T + b
        if k < 4:
            f = 0.5 * f * (1.0 + torch.tanh(0.7978845608 * (f + 0.044715 * f ** 3)))
    return f


def exact(case, seed):
    """The network in 64 bits, tanh form of GELU.  The solver's passes have none: they are themselves 64-bit
    iterations of a whole nonlinear solver (or, mixed, held to them), the integrator chooses its own steps, and
    training draws its batches on the device."""
    if case["kind"] != "mlp_forward":
        return None
    x = _features(case["n"], seed)
    mean, std = (torch.tensor(np.asarray(v, dtype=np.float32), device=x.device).double() for v in _norm())
    flat = torch.tensor(surrogate.init_params(seed), device=x.device).double()
    p, at = {}, 0
    for k, (o, i) in enumerate([(128, 7), (128, 128), (128, 128), (128, 128), (4, 128)]):
        p["W%d" % k] = flat[at:at + o * i].reshape(o, i)
        p["b%d" % k] = flat[at + o * i:at + o * i + o]
        at += o * i + o
    return torch.cat([_forward64(p, part, mean, std) for part in x.split(1 << 19)])
