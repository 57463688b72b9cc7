"""The work that programs built on this library have it do, as measurable cases.

A time-stepping program opens a deck, sets its start field, then advances the
flow and reads the fields and the history rows at every output interval
(``tframef`` of the decks: 100 to 200 steps).  The single-flow cases are one
such interval, over the grids from the smallest test deck to the largest
benchmark grid; the others are the loops of hosts that keep the rigid body
themselves, that let dt follow the CFL number, that couple strongly, that use
the split-precision Poisson form or that advance many flows at once, the
training of the coupling predictor, and the CFL check on a caller's own device
arrays.  Sizes are cells (z x y).
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

MAX_CELLS = 2048 * 1536


def listed():
    return [
        # the smallest test deck: a step is launches and their latencies only
        {"name": "cylinder_48x32", "kind": "flow", "body": "tiny_cylinder", "n3m": 48, "n2m": 32, "nlm": 40,
         "steps": 100},
        # vortex-induced vibration at the resolution of a parameter study
        {"name": "cylinder_384x256", "kind": "flow", "body": "viv_cylinder_384x256", "n3m": 384, "n2m": 256,
         "nlm": 302, "steps": 100},
        # the benchmark's flow: rotational galloping of a rectangle
        {"name": "rectangle_1024x768", "kind": "flow", "body": "galloping_rectangle_1024x768", "n3m": 1024,
         "n2m": 768, "nlm": 1200, "steps": 100},
        # the largest benchmark grid
        {"name": "cylinder_2048x1536", "kind": "flow", "body": "viv_cylinder_2048x1536", "n3m": 2048, "n2m": 1536,
         "nlm": 604, "steps": 50},
        # a ragged grid near the reference's galloping deck (731 x 561 nodes,
        # 798 markers), with the end-of-step diagnostics its report file needs
        {"name": "rectangle_731x561_report", "kind": "flow", "body": "rectangle", "n3m": 731, "n2m": 561, "nlm": 798,
         "steps": 100, "report": True},
        # Adams-Bashforth with dt following the CFL number: steps launch
        # eagerly, the host reads the CFL number of each
        {"name": "adaptive_cylinder_501x333", "kind": "flow", "body": "cylinder", "n3m": 501, "n2m": 333, "nlm": 300,
         "steps": 60, "adaptive": True},
        # the Poisson transforms in split precision with refinement sweeps
        {"name": "precision_1024x768", "kind": "flow", "body": "galloping_rectangle_1024x768", "n3m": 1024,
         "n2m": 768, "nlm": 1200, "steps": 50, "poisson": "tf32x3"},
        # strong fluid-structure coupling iterated on the device
        {"name": "coupled_384x256", "kind": "flow", "body": "viv_cylinder_384x256", "n3m": 384, "n2m": 256,
         "nlm": 302, "steps": 50, "coupled": True},
        # a host that keeps the rigid body: markers in, fluid step, rigid
        # update, markers out, every step (the size of the reference's
        # cylinder deck: 811 x 673 nodes, 377 markers)
        {"name": "host_loop_810x672", "kind": "host", "body": "cylinder", "n3m": 810, "n2m": 672, "nlm": 377,
         "steps": 50},
        # a parameter study advanced as one batch (grids 256x192 .. 768x512)
        {"name": "batch_20", "kind": "batch", "count": 20, "draw": 0, "steps": 50},
        # training the coupling predictor on samples of coupled steps
        {"name": "predictor_training", "kind": "train", "samples": 8192, "batch": 128, "epochs": 2},
        # the CFL check of a caller that owns its device arrays
        {"name": "cfl_1024x768", "kind": "cfl", "n3m": 1024, "n2m": 768},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["flow", "adaptive", "precision", "coupled", "host", "batch", "train", "cfl"],
                       [8, 2, 2, 2, 2, 2, 1, 1])[0]
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(3, 20), "draw": rng.randint(1, 10000), "steps": 20}
    if kind == "train":
        return {"kind": "train", "samples": _log_int(rng, 1000, 16384), "batch": rng.choice([64, 100, 128, 256, 512]),
                "epochs": rng.randint(1, 3)}
    n3m = _log_int(rng, 48, 2048)
    n2m = min(1536, max(32, int(n3m * rng.uniform(0.6, 0.8))))
    if kind == "cfl":
        return {"kind": "cfl", "n3m": n3m, "n2m": n2m}
    if kind == "coupled" and n3m > 700:   # a coupled step takes two to three fluid solves
        n3m, n2m = n3m // 2, n2m // 2
    body = "rectangle" if n3m >= 256 and rng.random() < 0.4 else "cylinder"
    # one to two markers per grid spacing on the outline
    perimeter = 10.0 if body == "rectangle" else math.pi
    nlm = max(24, int(perimeter / _spacing(body, n3m) * rng.uniform(1.0, 2.0)))
    case = {"kind": "host" if kind == "host" else "flow", "body": body, "n3m": n3m, "n2m": n2m, "nlm": nlm,
            "steps": rng.choice([20, 30, 40])}
    if kind == "adaptive":
        case["adaptive"] = True
    elif kind == "precision":
        case["poisson"] = "tf32x3"
    elif kind == "coupled":
        case["coupled"] = True
    elif rng.random() < 0.25:
        case["nsst"] = 1   # Adams-Bashforth at fixed dt
    return case


# ------------------------------------------------------------------ decks

def _spacing(body, n3m):
    """Window spacing: half of the z cells lie in the uniform window."""
    window = 9.0 if body == "rectangle" else (6.0 if n3m >= 160 else 3.0)
    return window / (n3m // 2)


def _deck(case):
    """The deck of a single flow: the repository's own ones by name, or the
    same families on any grid."""
    n3m, n2m, nlm, body = case["n3m"], case["n2m"], case["nlm"], case["body"]
    if body == "tiny_cylinder":
        c = cases.tiny_cylinder(n3m=n3m, n2m=n2m, nlm=nlm)
    elif body in cases.WORKLOADS:
        c = cases.WORKLOADS[body]()
    else:
        h = _spacing(body, n3m)
        wz, wy = (n3m // 2) * h, (n2m // 2) * h
        kw = dict(n3m=n3m, n2m=n2m, h=h, ywin=(-0.5 * wy, 0.5 * wy), nlm=nlm, dt=0.1 * h, name="deck")
        if body == "rectangle":
            c = cases.galloping_rectangle(zwin=(-0.3 * wz, 0.7 * wz), **kw)
        elif n3m >= 160:
            c = cases.viv_cylinder(zwin=(-0.3 * wz, 0.7 * wz), **kw)
        else:
            c = cases.viv_cylinder(zwin=(-wz / 3.0, 2.0 * wz / 3.0), zdom=(-3.0, 9.0), ydom=(-3.0, 3.0), **kw)
    if case.get("adaptive"):
        c.params.idtv = False
        c.params.nsst = 1
        c.params.dtmax = 4.0 * c.params.dt
    if "nsst" in case:
        c.params.nsst = case["nsst"]
    return c


def _open(c, rng):
    """A context on the deck, its start field disturbed: a few smooth modes of
    5 % of the free stream and Gaussian noise of 1e-3."""
    with tempfile.TemporaryDirectory(prefix="fbdeck_") as root:
        s = fb.Solver(c.write(os.path.join(root, "deck")))
    z = np.linspace(0.0, 1.0, c.n3m)[:, None]
    y = np.linspace(0.0, 1.0, c.n2m)[None, :]
    for name, cols in (("q2", slice(1, c.n2m)), ("q3", slice(0, c.n2m))):
        yy = y[:, cols.start:]
        f = 1e-3 * rng.standard_normal((c.n3m, yy.shape[1]))
        for _ in range(3):
            a, m, n, p = rng.normal(), rng.integers(1, 6), rng.integers(1, 4), rng.uniform(0.0, 2.0 * math.pi)
            f += 0.03 * a * np.sin(math.pi * z) * np.sin(2.0 * math.pi * m * z + p) * np.sin(math.pi * n * yy)
        q = s.get(name)
        q[1:c.n3m + 1, cols] += f
        s.set(name, q)
    return s


# ------------------------------------------------------------------ a pass

def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("flow", "host"):
        s = _open(_deck(case), rng)
        if case.get("poisson") == "tf32x3":
            s.set_poisson(fb.POISSON_TF32X3)
        if case.get("report"):
            s.set_report(True)
        if case.get("coupled"):
            s.set_coupling(fb.COUPLING_STRONG, tol=1e-10)
        state = {"case": case, "solver": s, "ns": 0}
        if kind == "host":
            state["markers"] = s.get_markers()
        return state
    if kind == "batch":
        decks = cases.viv_batch(case["count"], seed=case["draw"])
        return {"case": case, "batch": fb.Batch([_open(c, rng) for c in decks])}
    if kind == "train":
        x = rng.standard_normal((case["samples"], 27)).astype(np.float32)
        w = rng.standard_normal((27, 2)).astype(np.float32) / 27 ** 0.5
        t = (np.tanh(x @ w) + 0.1 * rng.standard_normal((case["samples"], 2))).astype(np.float32)
        return {"case": case, "mlp": fb.MLP(27, 2, seed=seed), "x": x, "t": t, "pass": 0}
    # cfl: the caller's own device arrays
    dev = {k: torch.from_numpy(v).cuda() for k, v in _cfl_arrays(case, rng).items()}
    f = fb.lib().fb_cfl_noalloc
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int] + \
        [ctypes.c_void_p] * 4 + [ctypes.c_double] * 3 + [ctypes.c_void_p] * 2
    return {"case": case, "arrays": dev, "out": torch.zeros(2, dtype=torch.float64, device="cuda"), "call": f}


def _cfl_arrays(case, rng):
    """Velocities (dense rows, k = 0 .. n3), stretched node coordinates of a
    40 x 30 domain and their inverse spacings."""
    n2m, n3m = case["n2m"], case["n3m"]
    q2 = 0.1 * rng.standard_normal((n3m + 2, n2m + 1))
    q3 = 1.0 + 0.1 * rng.standard_normal((n3m + 2, n2m + 1))
    rc = 30.0 * (0.7 * np.linspace(0.0, 1.0, n2m + 1) + 0.3 * np.linspace(0.0, 1.0, n2m + 1) ** 3)
    zz = 40.0 * (0.7 * np.linspace(0.0, 1.0, n3m + 1) + 0.3 * np.linspace(0.0, 1.0, n3m + 1) ** 3)
    return dict(q2=q2, q3=q3, rc=rc, zz=zz, udx2m=1.0 / np.diff(rc), udx3m=1.0 / np.diff(zz))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "flow":
        s, n = state["solver"], case["steps"]
        coupled = bool(case.get("coupled"))
        hist = s.advance(state["ns"], n, history=not coupled)
        state["ns"] += n
        out = {"q2": s.get("q2"), "q3": s.get("q3"), "pr": s.get("pr")}
        # a coupled interval reports the converged body; its per-step rows
        # count iterations
        out["rows"] = s.get("rigid") if coupled else hist
        return out
    if kind == "host":
        s, rows = state["solver"], []
        for _ in range(case["steps"]):
            s.set_markers(*state["markers"])
            s.fluid_tsch(state["ns"])
            rows.append(s.rigid(state["ns"]))
            state["markers"] = s.get_markers()
            state["ns"] += 1
        return {"rows": np.stack(rows), "markers": state["markers"], "q2": s.get("q2"), "q3": s.get("q3")}
    if kind == "batch":
        b = state["batch"]
        b.advance(case["steps"])
        return [{"q2": s.get("q2"), "q3": s.get("q3"), "row": s.last_history()} for s in b.solvers]
    if kind == "train":
        m = state["mlp"]
        loss = m.train(state["x"], state["t"], epochs=case["epochs"], batch=case["batch"], lr=2e-3, seed=state["pass"])
        state["pass"] += 1
        return {"params": m.params(), "loss": loss}
    a, n2, n3 = state["arrays"], case["n2m"] + 1, case["n3m"] + 1
    st = state["call"](a["q2"].data_ptr(), a["q3"].data_ptr(), n2, n2, n3, a["rc"].data_ptr(), a["zz"].data_ptr(),
                       a["udx2m"].data_ptr(), a["udx3m"].data_ptr(), 1e-3, 30.0, 40.0, state["out"].data_ptr(),
                       torch.cuda.current_stream().cuda_stream)
    if st:
        raise RuntimeError(f"fb_cfl_noalloc: {st}")
    return state["out"]


# ------------------------------------------------------------------ what a pass cannot do without

def _step_work(n3m, n2m, substeps):
    """One step: velocities, pressure and the two convective histories read
    and written once, the eigenvectors read once; two dense eigen transforms
    per substep, and about 200 operations per cell in the stencils and line
    solves."""
    cells = n3m * n2m
    return (10 * 8.0 * cells + 2 * 8.0 * n3m * n3m,
            substeps * (4.0 * n2m * n3m * n3m + 200.0 * cells))


def work(case):
    kind = case["kind"]
    if kind in ("flow", "host"):
        sub = 1 if case.get("adaptive") or case.get("nsst") == 1 else 3
        b, f = _step_work(case["n3m"], case["n2m"], sub)
        return {"bytes": case["steps"] * b, "flops": case["steps"] * f}
    if kind == "batch":
        w = [_step_work(c.n3m, c.n2m, 3) for c in cases.viv_batch(case["count"], seed=case["draw"])]
        return {"bytes": case["steps"] * sum(b for b, _ in w), "flops": case["steps"] * sum(f for _, f in w)}
    if kind == "train":
        n = case["epochs"] * (case["samples"] // min(case["batch"], case["samples"])) * case["batch"]
        weights = 64 * 27 + 64 * 64 + 2 * 64
        return {"bytes": 4.0 * (n * 29 + 6 * weights), "flops": 6.0 * n * weights}
    cells = case["n3m"] * case["n2m"]
    return {"bytes": 16.0 * cells, "flops": 10.0 * cells}


# ------------------------------------------------------------------ values in 64 bits

def exact(case, seed):
    """The CFL case.  A whole time step (or a training run, whose minibatch
    order the library draws) has no short restatement in plain numpy."""
    if case["kind"] != "cfl":
        return None
    c = _cfl_arrays(case, np.random.default_rng(seed))
    n2m, n3m, q2, q3 = case["n2m"], case["n3m"], c["q2"], c["q3"]
    v = 0.5 * (q2[1:n3m + 1, :n2m] + q2[1:n3m + 1, 1:])
    w = 0.5 * (q3[1:n3m + 1, :n2m] + q3[2:, :n2m])
    cfl = np.max(np.abs(v * c["udx2m"][None, :]) + np.abs(w * c["udx3m"][:, None])) * 1e-3
    area = np.diff(c["rc"])[None, :] * np.diff(c["zz"])[:, None]
    return torch.tensor([cfl, np.sum(q3[1:n3m + 1, :n2m] * area) / (30.0 * 40.0)], dtype=torch.float64)
