"""The workloads this framework is timed on: what its users run, through its public entry points.

  single        the command line's call: one small Van der Pol problem (101 nodes, m = 4, zero guess), batch object and all
  constrained   the same call on a control-constrained problem: the continuation in the smoothing parameter, hundreds of
                dependent Newton steps on one small mesh
  batch         thousands of Van der Pol instances with uneven meshes (32 .. 2048 intervals) from the plain guess, guesses and
                solutions in page-locked host memory (what the benchmark calls end to end)
  warm          the same, started from predicted trajectories on the device (the learned warm start's solve)
  direction     one Newton direction of a batch: the stage entry point behind construct / reduce Jacobian, the BABD solve and
                the recovery
  pend_batch    a batch of pendulum chains, K = 8 (medium stage systems: s = 72)
  pend          one long pendulum chain, K = 16 or 32, in FP64 or with the TF32 / BF16 condensation
  train         an epoch of the warm-start network's training on solved trajectories
  predict       its forward pass for a batch of instances, device to device
  files         the solution files of a solved batch as text
  babd          one bordered almost-block-diagonal system in device memory

The Van der Pol batches draw the control weight from [0.1, 1] and otherwise use the family's full ranges: with larger weights a
few instances iterate to the limit of 200 steps from the plain guess, and there the last bits decide the counts.
"""
import ctypes
import functools
import importlib
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
cs = importlib.import_module("collocation-solver-cuda_gb300")
WS = cs.warmstart

COUNTS = ("status", "N", "newton_steps", "residual_evals", "segment_evals", "remeshes", "continuation_steps", "singular",
          "fail_reason")


# ------------------------------------------------------------------ cases ---
def listed():
    return [
        {"name": "single", "kind": "single", "m": 4, "nodes": 101},
        {"name": "constrained", "kind": "constrained", "m": 4, "nodes": 21},
        {"name": "batch m5", "kind": "batch", "m": 5, "instances": 1024, "n_lo": 32, "n_hi": 2048},
        {"name": "warm m3", "kind": "warm", "m": 3, "instances": 2048, "n_lo": 32, "n_hi": 2048},
        {"name": "direction m4", "kind": "direction", "m": 4, "instances": 333, "nodes": 801},
        {"name": "pend8 batch", "kind": "pend_batch", "m": 4, "instances": 96, "n_lo": 32, "n_hi": 128},
        {"name": "pend16 fp64", "kind": "pend", "K": 16, "m": 5, "nodes": 2049, "precision": "fp64"},
        {"name": "pend32 bf16", "kind": "pend", "K": 32, "m": 4, "nodes": 1025, "precision": "bf16"},
        {"name": "train", "kind": "train", "samples": 4133, "batch": 1024, "n_in": 4, "width": 256, "n_out": 322},
        {"name": "predict", "kind": "predict", "samples": 8192, "n_in": 4, "width": 256, "n_out": 322},
        {"name": "files", "kind": "files", "m": 4, "instances": 512, "n_lo": 32, "n_hi": 2048},
        {"name": "babd", "kind": "babd", "ny": 6, "np": 2, "intervals": 1500},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "constrained", "batch", "batch", "warm", "warm", "direction", "pend_batch", "pend", "pend",
                       "train", "predict", "files", "babd"])
    if kind == "single":
        return {"kind": kind, "m": rng.choice([3, 4, 5]), "nodes": _log_int(rng, 33, 1025)}
    if kind == "constrained":
        return {"kind": kind, "m": 4, "nodes": rng.randint(17, 41)}
    if kind in ("batch", "warm", "files"):
        hi = _log_int(rng, 64, 2048)
        most = min(1024 if kind == "batch" else 2048 if kind == "warm" else 512, 2200000 // (32 + hi))
        return {"kind": kind, "m": rng.choice([3, 4, 5]), "instances": _log_int(rng, 3, most), "n_lo": 32, "n_hi": hi}
    if kind == "direction":
        nodes = _log_int(rng, 33, 2049)
        return {"kind": kind, "m": rng.choice([3, 4, 5]), "instances": _log_int(rng, 1, max(1, 266000 // nodes)),
                "nodes": nodes}
    if kind == "pend_batch":
        return {"kind": kind, "m": 4, "instances": _log_int(rng, 1, 96), "n_lo": 32, "n_hi": rng.randint(40, 128)}
    if kind == "pend":
        K, precision = rng.choice([16, 32]), rng.choice(["fp64", "tf32", "bf16"])
        most = 2049 if K == 16 else 385 if precision == "fp64" else 1025
        return {"kind": kind, "K": K, "m": 5 if K == 16 else 4, "nodes": _log_int(rng, 65, most), "precision": precision}
    if kind == "train":
        batch = _log_int(rng, 128, 1024)
        return {"kind": kind, "samples": rng.randint(batch, 4 * batch + batch // 2), "batch": batch, "n_in": rng.choice([4, 10]),
                "width": rng.choice([64, 128, 256]), "n_out": rng.choice([130, 322])}
    if kind == "predict":
        return {"kind": kind, "samples": _log_int(rng, 1, 8192), "n_in": rng.choice([4, 10]), "width": rng.choice([64, 128, 256]),
                "n_out": rng.choice([130, 322])}
    ny, npar = rng.randint(2, 20), rng.randint(0, 4)
    return {"kind": "babd", "ny": ny, "np": npar, "intervals": _log_int(rng, 20, min(6000, 36000 // ny))}


# ------------------------------------------------- problems, compiled once ---
@functools.lru_cache(maxsize=None)
def _family(name):
    """Van der Pol ("vdp"), or the pendulum chain of K ("pend8", ...)."""
    return WS.vdp_family() if name == "vdp" else WS.pendulum_family(int(name[4:]))


@functools.lru_cache(maxsize=None)
def _constrained_problem():
    return cs.ocp.Problem.from_file(os.path.join(ROOT, "tests", "golden", "ocp", "vdp_ineq.ocp"))


@functools.lru_cache(maxsize=None)
def _compiled(name, m, precision="fp64"):
    return cs.CompiledProblem(_family(name).problem, m, precision=precision)


# ----------------------------------------------------------------- inputs ---
def _meshes(case):
    """Intervals per instance: the program's meshes stay while the instances on them change."""
    return np.random.default_rng(case["instances"]).integers(case["n_lo"], case["n_hi"] + 1, case["instances"])


def _vdp_instances(case, rng, wide=True):
    """Instances of the Van der Pol family; wide: over its ranges, else near one nominal instance."""
    B, N = case["instances"], _meshes(case)
    if wide:
        x0 = rng.uniform(-2.0, 2.0, (B, 2))
        T = rng.uniform(2.0, 8.0, B)
        r = np.exp(rng.uniform(np.log(0.1), 0.0, B))
    else:
        x0 = rng.uniform(-1.5, 1.5, 2) + 0.1 * rng.uniform(-1.0, 1.0, (B, 2))
        T = rng.uniform(3.0, 6.0) * rng.uniform(0.95, 1.05, B)
        r = np.exp(rng.uniform(np.log(0.2), 0.0)) * rng.uniform(0.95, 1.05, B)
    V = cs.workloads.VdpInstance
    return [V(x0[b], float(T[b]), float(r[b]), int(N[b]), case["m"]) for b in range(B)]


def _pinned(shape, dtype=np.float64):
    """A page-locked array (it keeps its memory alive by itself)."""
    return torch.zeros(shape, dtype=torch.from_numpy(np.zeros(0, dtype)).dtype, pin_memory=True).numpy()


def _pinned_copy(a):
    p = _pinned(a.shape, a.dtype)
    p[...] = a
    return p


def _batch_state(cp, packed, opts):
    """A batch with its guesses in page-locked host memory, and page-locked room for solutions on the meshes a solve may refine
    them to (short meshes to five times their nodes)."""
    N, t, y, z, p, th = packed
    cap = int((N + np.minimum(4 * N, 512)).sum())
    host = [_pinned_copy(a) for a in (N, t, y, z, p, th)]
    out = [_pinned(s) for s in ((cap,), (cap, cp.ny), (cap, max(cp.nz, 1)), (len(N), max(cp.np, 1)))]
    return {"batch": cs.Batch(cp, len(N), node_capacity=int(N.sum())), "host": host, "out": out, "opts": opts}


def _solve_batch(s):
    """Guesses in, solve, solutions out."""
    bt = s["batch"]
    bt.set_guess_packed(*s["host"])
    if "traj" in s:
        bt.warm_start(s["traj"].data_ptr(), WS.N_NODES, s["traj"].shape[1])
    bt.solve(s["opts"])
    N, T = bt.sizes()
    t, y, z, p = s["out"]
    if T > t.shape[0]:
        raise RuntimeError("solution larger than the host buffers")
    st = (cs._lib.Stats * bt.B)()
    cs._lib.check(bt._lib.cs_get_solution(bt.handle, cs._lib.dptr(t), cs._lib.dptr(y), cs._lib.dptr(z), cs._lib.dptr(p), st),
                  "cs_get_solution")
    rec = np.ctypeslib.as_array(st)
    # the caller's buffers: an instance's nodes follow the previous instance's, counts N of them
    return {"t": t, "y": y, "z": z, "p": p, "counts": [rec[k] for k in COUNTS]}


def _network(case, rng):
    """The warm-start network of the case's sizes, freshly initialised, with the normalisation of its data."""
    net = WS.Mlp(case["n_in"], case["n_out"], width=case["width"], depth=4, seed=int(rng.integers(1 << 31)))
    mean = rng.uniform(-1.0, 1.0, case["n_out"])
    net.set_normalization(rng.uniform(-0.5, 0.5, case["n_in"]), rng.uniform(0.5, 2.0, case["n_in"]), mean,
                          rng.uniform(0.3, 1.5, case["n_out"]))
    return net


def _direction_guess(case, rng):
    """Smooth trajectories of the size solutions have, one mesh size for all instances, uneven steps."""
    B, N = case["instances"], case["nodes"]
    h = rng.uniform(0.5, 1.5, (B, N - 1))
    t = np.concatenate([np.zeros((B, 1)), np.cumsum(h, axis=1)], axis=1)
    t *= (rng.uniform(2.0, 8.0, (B, 1)) / t[:, -1:])
    amp, w, ph = (rng.uniform(lo, hi, (B, 1, 5)) for lo, hi in ((0.1, 1.5), (0.5, 1.5), (0.0, 6.28)))
    v = amp * np.cos(w * t[:, :, None] + ph) * np.exp(-0.2 * t[:, :, None])
    x0 = rng.uniform(-2.0, 2.0, (B, 2))
    th = np.concatenate([x0, np.exp(rng.uniform(np.log(0.1), np.log(10.0), (B, 1)))], axis=1)
    return t, v[:, :, :4].copy(), v[:, :, 4:].copy(), rng.uniform(-1.0, 1.0, (B, 2)), th


def _babd_system(case, rng):
    """Block rows as the condensation leaves them (C = I, A = -I + something), full boundary rows."""
    ny, npar, n = case["ny"], case["np"], case["intervals"]
    A = -np.eye(ny)[None] + 0.2 * rng.standard_normal((n, ny, ny))
    C = np.broadcast_to(np.eye(ny), (n, ny, ny)).copy()
    H = 0.1 * rng.standard_normal((n, ny, npar))
    b = rng.standard_normal((n, ny))
    return [A, C, H, b, rng.standard_normal((ny + npar, ny)), rng.standard_normal((ny + npar, ny)),
            rng.standard_normal((ny + npar, npar)), rng.standard_normal(ny + npar)]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "single":
        pr, N = _family("vdp").problem, case["nodes"]
        T, theta = rng.uniform(2.0, 8.0), np.array([*rng.uniform(-2.0, 2.0, 2), np.exp(rng.uniform(np.log(0.1), 0.0))])
        cs.solver.compiled(pr, case["m"])
        return {"kind": kind, "problem": pr, "m": case["m"], "T0": np.linspace(0.0, T, N), "Y0": np.zeros((N, 4)),
                "Z0": np.zeros((N, 1)), "P0": np.ones(2), "theta": theta, "opts": cs.default_opts(pr)}
    if kind == "constrained":
        pr, N = _constrained_problem(), case["nodes"]
        cs.solver.compiled(pr, case["m"])
        Y0 = np.tile(np.asarray(pr.Y0)[0], (N, 1)) + 0.05 * rng.uniform(-1.0, 1.0, 4) * np.linspace(1.0, 0.0, N)[:, None]
        return {"kind": kind, "problem": pr, "m": case["m"], "T0": np.linspace(0.0, 3.0, N), "Y0": Y0,
                "Z0": np.tile(np.asarray(pr.Z0)[0], (N, 1)), "P0": np.asarray(pr.P0, float), "theta": None,
                "opts": cs.default_opts(pr)}
    if kind in ("batch", "warm"):
        fam, cp = _family("vdp"), _compiled("vdp", case["m"])
        insts = _vdp_instances(case, rng, wide=kind == "batch")
        opts = cs.default_opts(fam.problem)
        s = _batch_state(cp, cs.workloads.pack_vdp(insts), opts)
        if kind == "warm":
            # the network's answer for instances near one it knows: the nominal solution
            mid = cs.workloads.VdpInstance(np.mean([i.x0 for i in insts], axis=0), float(np.mean([i.T for i in insts])),
                                           float(np.mean([i.r for i in insts])), 128, case["m"])
            sol = WS.BatchSolver(fam, opts=opts).solve([mid])[0]
            v = WS.trajectory_vector(sol["t"], sol["y"], sol["z"], sol["p"], mid.T)
            traj = np.tile(v, (len(insts), 1)) * (1.0 + 0.01 * rng.standard_normal((len(insts), 1)))
            s["traj"] = torch.tensor(traj, dtype=torch.float32, device="cuda")
        return dict(s, kind=kind)
    if kind in ("pend_batch", "pend"):
        K = case.get("K", 8)
        fam = _family("pend%d" % K)
        cp = _compiled("pend%d" % K, case["m"], case.get("precision", "fp64"))
        if kind == "pend":
            insts = [cs.workloads.PendulumInstance(rng.uniform(-0.5, 0.5, K), 10.0, 0.5, case["nodes"] - 1, case["m"])]
        else:
            insts = [cs.workloads.PendulumInstance(rng.uniform(-0.5, 0.5, K), rng.uniform(5.0, 15.0), rng.uniform(0.2, 1.0),
                                                   int(n), case["m"]) for n in _meshes(case)]
        # the long chains' own tolerances: 1e-6 for K = 16, 1e-8 for K = 32
        opts = cs.default_opts(fam.problem, tol=1e-8 if K == 32 else 1e-6)
        return dict(_batch_state(cp, WS.pack_family(fam, insts), opts), kind=kind)
    if kind == "direction":
        cp = _compiled("vdp", case["m"])
        B, N, m = case["instances"], case["nodes"], case["m"]
        t, y, z, p, th = _direction_guess(case, rng)
        bt = cs.Batch(cp, B, node_capacity=B * N)
        bt.set_guess_packed(np.full(B, N, np.int32), t.ravel(), y.reshape(-1, 4), z.reshape(-1, 1), p, th)
        out = [_pinned(s) for s in ((B * N, 4), (B * N, m, 4), (B * N, m, 1), (B, 2))]
        return {"kind": kind, "batch": bt, "out": out, "shape": (B, N, m)}
    if kind == "train":
        net = _network(case, rng)
        X = rng.uniform(-2.0, 2.0, (case["samples"], case["n_in"]))
        Y = np.tanh(X @ rng.standard_normal((case["n_in"], 24))) @ rng.standard_normal((24, case["n_out"]))
        return {"kind": kind, "net": net, "X": X.astype(np.float32), "Y": Y.astype(np.float32), "batch": case["batch"]}
    if kind == "predict":
        net = _network(case, rng)
        X = torch.tensor(rng.uniform(-2.0, 2.0, (case["samples"], case["n_in"])), dtype=torch.float32, device="cuda")
        return {"kind": kind, "net": net, "X": X, "Y": torch.empty(case["samples"], case["n_out"], device="cuda")}
    if kind == "files":
        fam, cp = _family("vdp"), _compiled("vdp", case["m"])
        N, t, y, z, p, th = cs.workloads.pack_vdp(_vdp_instances(case, rng))
        y, z = 0.7 * rng.standard_normal(y.shape), 0.5 * rng.standard_normal(z.shape)
        bt = cs.Batch(cp, len(N), node_capacity=int(N.sum()))
        bt.set_guess_packed(N, t, y, z, rng.standard_normal(p.shape), th)
        # a number takes at most 24 characters and a blank
        text = _pinned(25 * 6 * int(N.sum()) + 300 * len(N), np.uint8)
        return {"kind": kind, "batch": bt, "text": text, "offsets": np.zeros(len(N) + 1, np.int64)}
    if kind == "babd":
        ins = [torch.tensor(a if a.size else np.zeros(1), dtype=torch.float64, device="cuda") for a in _babd_system(case, rng)]
        dims = (case["ny"], case["np"], case["intervals"])
        return {"kind": kind, "dims": dims, "ins": ins,
                "dy": torch.zeros(dims[2] + 1, dims[0], dtype=torch.float64, device="cuda"),
                "dp": torch.zeros(max(dims[1], 1), dtype=torch.float64, device="cuda")}
    raise ValueError(kind)


# -------------------------------------------------------------------- run ---
def run(state):
    kind = state["kind"]
    if kind in ("single", "constrained"):
        sol = cs.solver.solve_single(state["problem"], state["m"], state["T0"], state["Y0"], state["Z0"], state["P0"],
                                     state["theta"], state["opts"])
        # (the residual norms a solve ends on are rounding: not among the outputs)
        return {"t": sol["t"], "y": sol["y"], "z": sol["z"], "p": sol["p"], "counts": [sol[k] for k in COUNTS]}
    if kind in ("batch", "warm", "pend_batch", "pend"):
        return _solve_batch(state)
    if kind == "direction":
        bt = state["batch"]
        dy, dyd, dz, dp = state["out"]
        cs._lib.check(bt._lib.cs_stage_newton_direction(bt.handle, 0.1, None, cs._lib.dptr(dy), cs._lib.dptr(dyd),
                                                        cs._lib.dptr(dz), cs._lib.dptr(dp)), "cs_stage_newton_direction")
        B, N, m = state["shape"]
        # stage steps: one row per interval (an instance's last slot has none)
        return {"dy": dy.reshape(B, N, 4), "dydot": dyd.reshape(B, N, m, 4)[:, :-1], "dzt": dz.reshape(B, N, m)[:, :-1],
                "dp": dp}
    if kind == "train":
        loss = state["net"].train(state["X"], state["Y"], epochs=1, batch=state["batch"], lr=1e-3, seed=1)
        return {"loss": loss, "params": state["net"].params()}
    if kind == "predict":
        state["net"].predict_device(state["X"].data_ptr(), state["X"].shape[0], state["Y"].data_ptr())
        return state["Y"]
    if kind == "files":
        # sizes first, then the text into the caller's buffer (as Batch.solution_text does, which allocates it)
        bt, text, off = state["batch"], state["text"], state["offsets"]
        cs._lib.check(bt._lib.cs_format_solutions(bt.handle, None, 0, off.ctypes.data), "cs_format_solutions")
        if off[-1] > text.size:
            raise RuntimeError("text larger than the host buffer")
        cs._lib.check(bt._lib.cs_format_solutions(bt.handle, text.ctypes.data, text.size, off.ctypes.data), "cs_format_solutions")
        return {"text": text, "offsets": off}
    if kind == "babd":
        ptr = [ctypes.c_void_p(a.data_ptr()) for a in (*state["ins"], state["dy"], state["dp"])]
        singular = ctypes.c_int()
        cs._lib.check(cs._lib.load().cs_babd_solve(*state["dims"], *ptr, ctypes.byref(singular), None), "cs_babd_solve")
        return {"dy": state["dy"], "dp": state["dp"][:state["dims"][1]], "singular": singular.value}
    raise ValueError(kind)


# ------------------------------------------------------------------- work ---
def _step_work(ny, nz, m, intervals):
    """One Newton step: stage systems condensed (LU without the explicit first stage), block rows eliminated by QR of
    (2 ny) x ny blocks, the iterate and the direction read and written once."""
    s1, r = (m - 1) * (ny + nz), ny + 1
    condense = 2.0 / 3.0 * s1 ** 3 + 2.0 * s1 * s1 * r + 2.0 * s1 * r * ny
    tree = sum(4.0 * (2 * ny - k) * (3 * ny + 1 - k) for k in range(ny))
    per = ny + m * (ny + nz)
    return {"flops": intervals * (condense + tree), "bytes": 8.0 * intervals * (3 * per + 1)}


def work(case):
    kind = case["kind"]
    if kind in ("single", "constrained", "direction"):
        nz = 5 if kind == "constrained" else 1
        w = _step_work(4, nz, case["m"], (case["nodes"] - 1) * case.get("instances", 1))
        steps = {"single": 6, "constrained": 300, "direction": 1}[kind]
    elif kind in ("batch", "warm", "pend_batch", "pend"):
        K = case.get("K", 8)
        ny, nz = (4, 1) if kind in ("batch", "warm") else (4 * K, K // 4)
        n = case["nodes"] - 1 if kind == "pend" else case["instances"] * (case["n_lo"] + case["n_hi"]) / 2.0
        w = _step_work(ny, nz, case["m"], n)
        steps = {"batch": 6, "warm": 4, "pend_batch": 3, "pend": 3}[kind]
    elif kind in ("train", "predict"):
        w0 = case["width"]
        weights = case["n_in"] * w0 + 2 * w0 * w0 + w0 * case["n_out"]
        n = case["samples"] if kind == "predict" else (case["samples"] // case["batch"] + 1) * case["batch"]
        return {"flops": (2.0 if kind == "predict" else 6.0) * n * weights,
                "bytes": 4.0 * n * (case["n_in"] + case["n_out"]) + 4.0 * weights}
    elif kind == "files":
        values = case["instances"] * ((case["n_lo"] + case["n_hi"]) / 2.0 + 1) * 6
        return {"flops": 0.0, "bytes": values * (8.0 + 20.0)}
    else:
        ny, npar, n = case["ny"], case["np"], case["intervals"]
        tree = sum(4.0 * (2 * ny - k) * (3 * ny + npar + 1 - k) for k in range(ny))
        return {"flops": n * tree, "bytes": 8.0 * n * ny * (2 * ny + npar + 2)}
    return {k: v * steps for k, v in w.items()}


# ------------------------------------------------------------------ exact ---
def _lobatto(m):
    """Lobatto IIIA: nodes on [0, 1], A[j][k] = integral of the k-th basis polynomial to node j, weights b."""
    P = np.polynomial.legendre.Legendre.basis(m - 1)
    c = np.concatenate([[0.0], np.sort(P.deriv().roots().real) / 2 + 0.5, [1.0]])
    V = np.vander(c, m, increasing=True)
    powers = np.arange(1, m + 1)
    A = np.linalg.solve(V.T, (c[:, None] ** powers / powers).T).T
    return c, A, A[-1]


def _exact_direction(case, seed):
    """Newton direction of the collocation equations, stage systems and block rows by plain batched linear algebra."""
    t, y, z, p, th = _direction_guess(case, np.random.default_rng(seed))
    B, N, m = case["instances"], case["nodes"], case["m"]
    if B * N > 300000:
        return None
    c, A, b = _lobatto(m)
    r = th[:, 2][:, None, None]

    def f(v, u):
        x1, x2, l1, l2 = (v[..., k] for k in range(4))
        q = x1 * x1 - 1.0
        return np.stack([x2, -q * x2 - x1 + u, -x1 + l2 * (2 * x1 * x2 + 1.0), q * l2 - x2 - l1], axis=-1)

    mid = (1 - c)[:, None] * y[:, :-1, None] + c[:, None] * y[:, 1:, None]
    u = ((1 - c)[:, None] * z[:, :-1, None] + c[:, None] * z[:, 1:, None])[..., 0]
    yd = f(mid, u)
    h = np.diff(t, axis=1)
    v = y[:, :-1, None] + h[:, :, None, None] * np.einsum("jk,bnka->bnja", A, yd)
    x1, x2, l2 = v[..., 0], v[..., 1], v[..., 3]
    F = np.zeros((B, N - 1, m, 5, 5))  # d[f; g] / d[y; u]
    F[..., 0, 1] = 1.0
    F[..., 1, 0], F[..., 1, 1], F[..., 1, 4] = -(2 * x1 * x2 + 1.0), -(x1 * x1 - 1.0), 1.0
    F[..., 2, 0], F[..., 2, 1], F[..., 2, 3] = 2 * l2 * x2 - 1.0, 2 * x1 * l2, 2 * x1 * x2 + 1.0
    F[..., 3, 0], F[..., 3, 1], F[..., 3, 2], F[..., 3, 3] = 2 * x1 * l2, -1.0, -1.0, x1 * x1 - 1.0
    F[..., 4, 3], F[..., 4, 4] = 1.0, r
    res = np.concatenate([f(v, u) - yd, (r * u + l2)[..., None]], axis=-1).reshape(B, N - 1, 5 * m)
    W = np.zeros((B, N - 1, m, 5, m, 5))
    W[..., :4] = np.einsum("bn,jk,bnjac->bnjakc", h, A, F[..., :4])
    for j in range(m):
        W[:, :, j, :, j, 4] = F[:, :, j, :, 4]
        W[:, :, j, :4, j, :4] -= np.eye(4)
    rhs = np.concatenate([F[..., :4].reshape(B, N - 1, 5 * m, 4), res[..., None]], axis=-1)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X = torch.linalg.solve(torch.tensor(W.reshape(B, N - 1, 5 * m, 5 * m), device=dev), torch.tensor(rhs, device=dev)).cpu().numpy()
    D = h[:, :, None, None] * np.einsum("j,bnjac->bnac", b, X.reshape(B, N - 1, m, 5, 5)[..., :4, :])
    fb = np.diff(y, axis=1) - h[:, :, None] * np.einsum("j,bnja->bna", b, yd)
    # block rows  L dy_i + dy_{i+1} = d, eliminated from the left: the row kept couples dy_0 and dy_{i+1}
    L, d = D[..., :4] - np.eye(4), -fb - D[..., 4]
    keep, tops = None, []
    for i in range(N - 1):
        if keep is None:
            keep = np.concatenate([L[:, i], np.broadcast_to(np.eye(4), (B, 4, 4)), d[:, i, :, None]], axis=2)  # y0, y1, d
            continue
        M = np.zeros((B, 8, 13))  # y_i | y_0 | y_{i+1} | d
        M[:, :4, :4], M[:, :4, 4:8], M[:, :4, 12] = keep[:, :, 4:8], keep[:, :, :4], keep[:, :, 8]
        M[:, 4:, :4], M[:, 4:, 8:12], M[:, 4:, 12] = L[:, i], np.eye(4), d[:, i]
        Q = np.linalg.qr(M[:, :, :4], mode="complete")[0]
        M = Q.transpose(0, 2, 1) @ M
        tops.append(M[:, :4])
        keep = np.concatenate([M[:, 4:, 4:12], M[:, 4:, 12:]], axis=2)
    top, g = np.zeros((B, 10, 10)), np.zeros((B, 10))
    top[:, :4, :8], g[:, :4] = keep[:, :, :8], keep[:, :, 8]
    top[:, 4, 0] = top[:, 5, 1] = top[:, 6, 2] = top[:, 7, 3] = top[:, 6, 8] = top[:, 7, 9] = 1.0
    top[:, 8, 6] = top[:, 9, 7] = 1.0
    g[:, 4:6], g[:, 6:8], g[:, 8:] = th[:, :2] - y[:, 0, :2], -y[:, 0, 2:] - p, -y[:, -1, 2:]
    x = np.linalg.solve(top, g[..., None])[..., 0]
    dy = np.zeros((B, N, 4))
    dy[:, 0], dy[:, -1] = x[:, :4], x[:, 4:8]
    for i in range(N - 2, 0, -1):
        M = tops[i - 1]
        q = M[:, :, 12] - np.einsum("bac,bc->ba", M[:, :, 4:8], dy[:, 0]) - np.einsum("bac,bc->ba", M[:, :, 8:12], dy[:, i + 1])
        dy[:, i] = np.linalg.solve(M[:, :, :4], q[..., None])[..., 0]
    k = -(X[..., 4] + np.einsum("bnsc,bnc->bns", X[..., :4], dy[:, :-1])).reshape(B, N - 1, m, 5)
    return {"dy": dy, "dydot": k[..., :4], "dzt": k[..., 4], "dp": x[:, 8:]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "direction":
        return _exact_direction(case, seed)
    if kind == "predict":
        s = prepare(case, seed)
        net = s["net"]
        xm, xs, ym, ys = (torch.tensor(a, dtype=torch.float64, device="cuda") for a in net.norm)
        w, at = torch.tensor(net.params(), dtype=torch.float64, device="cuda"), 0
        v = (s["X"].double() - xm) / xs
        for layer, (n_in, n_out) in enumerate(net.sizes):
            v = v @ w[at:at + n_in * n_out].reshape(n_out, n_in).T + w[at + n_in * n_out:at + (n_in + 1) * n_out]
            at += (n_in + 1) * n_out
            if layer < net.depth - 1:
                v = torch.nn.functional.gelu(v)
        return v * ys + ym
    if kind == "babd":
        ny, npar, n = case["ny"], case["np"], case["intervals"]
        size = (n + 1) * ny + npar
        if size > 12000:
            return None
        A, C, H, b, B0, Bn, Vn, r = _babd_system(case, np.random.default_rng(seed))
        M, g = np.zeros((size, size)), np.zeros(size)
        for i in range(n):
            rows = slice(i * ny, (i + 1) * ny)
            M[rows, i * ny:(i + 1) * ny], M[rows, (i + 1) * ny:(i + 2) * ny] = A[i], C[i]
            M[rows, (n + 1) * ny:], g[rows] = H[i], b[i]
        M[n * ny:, :ny], M[n * ny:, n * ny:(n + 1) * ny], M[n * ny:, (n + 1) * ny:], g[n * ny:] = B0, Bn, Vn, -r
        x = torch.linalg.solve(torch.tensor(M, device="cuda"), torch.tensor(g, device="cuda")).cpu().numpy()
        return {"dy": x[:(n + 1) * ny].reshape(n + 1, ny), "dp": x[(n + 1) * ny:], "singular": None}
    return None  # a whole solve stops where its own Newton does, an epoch shuffles by the library's own rule, text has no error
