"""The stencil work a user of this package has it do, as timed cases.

Every case goes through a public entry point (``DeviceGrid.run``,
``kernel_stencil``, ``Batch.run``, ``time_loop``, ``forward_batch`` /
``backward_batch``). Grids are synthetic: every cell, halo included, i.i.d.
U[0,1); coefficients U[0,1) normalised so that the update is an average.

``exact`` restates each path in plain torch at 64 bits.
"""
from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "an5d-artifact_gb300"))

from gbstencil import adjoint, capi  # noqa: E402
from gbstencil.grid import DeviceGrid  # noqa: E402

NAMES_2D = [s["name"] for s in capi.TABLE if s["dim"] == 2]
NAMES_3D = [s["name"] for s in capi.TABLE if s["dim"] == 3]
# the stencils of the batched mix (as in the benchmark's batched workload)
MIX = ["star2d1r", "star2d2r", "star2d3r", "star2d4r", "box2d1r", "box2d2r", "box2d3r", "box2d4r", "j2d5pt", "j2d9pt"]
TORCH = {"f32": torch.float32, "f64": torch.float64}
NUMPY = {"f32": np.float32, "f64": np.float64}


def _loop(name, stencil, dtype, n, T, mode="fma", path="loop"):
    n = list(n) + [0] * (3 - len(n))
    c = {"path": path, "stencil": stencil, "dtype": dtype, "n0": n[0], "n1": n[1], "n2": n[2], "T": T, "mode": mode}
    return dict(c, name=name) if name else c


def _grad(name, stencil, dtype, n, T, every, want_coef):
    return dict(_loop(name, stencil, dtype, n, T, path="grad"), every=every, want_coef=want_coef)


def _batch(name, count, lo, hi, tmax, mix, schedule):
    c = {"path": "batch", "count": count, "lo": lo, "hi": hi, "tmax": tmax, "mix": mix, "schedule": schedule, "mode": "fma"}
    return dict(c, name=name) if name else c


def _gradbatch(name, count, lo, hi, T, every, mix):
    c = {"path": "gradbatch", "stencil": "j3d27pt", "dtype": "f32", "count": count, "lo": lo, "hi": hi, "T": T,
         "every": every, "mix": mix}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a few steps on a grid that a test or a coupled
        # code advances between other work; latency is what it pays
        _loop("tiny_star2d1r_f32", "star2d1r", "f32", (128, 96), 16),
        # the plain 2-D sweep the benchmark quotes (4096^2, T=100)
        _loop("star2d1r_f32_4096", "star2d1r", "f32", (4096, 4096), 100),
        # an odd, ragged grid and a stencil of many terms
        _loop("box2d2r_f32_ragged", "box2d2r", "f32", (3001, 2217), 50),
        # the artifact's own 2-D benchmark size, far beyond the L2
        _loop("j2d5pt_f32_16384", "j2d5pt", "f32", (16384, 16384), 50),
        # a 2-D double run
        _loop("j2d9pt_f64_ragged", "j2d9pt", "f64", (1777, 2500), 40),
        # the 3-D sweeps the benchmark quotes (512^3), fewer steps
        _loop("star3d2r_f32_512", "star3d2r", "f32", (512, 512, 512), 20),
        _loop("box3d1r_f64_512", "box3d1r", "f64", (512, 512, 512), 10),
        # the drop-in call: host grid in and out, the bit-exact default mode
        _loop("dropin_gol_f32_exact", "j2d9pt-gol", "f32", (1500, 1500), 100, mode="exact", path="host"),
        # many uneven grids advanced by one graph launch
        _batch("batch_layered_48", 48, 128, 2048, 128, 7, "layered"),
        # training through the loop: gradients of u_0 and the coefficients
        _grad("grad_j2d5pt_f32_2048", "j2d5pt", "f32", (2048, 2048), 128, 32, True),
        # the nonlinear stencil in double, forward with checkpoints and back
        _grad("grad_gradient2d_f64", "gradient2d", "f64", (1024, 1100), 64, 16, False),
        # 3-D gradients of several uneven instances side by side
        _gradbatch("grad_j3d27pt_batch4", 4, 96, 192, 32, 16, 3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choices(["loop2", "loop3", "host", "batch", "grad", "gradbatch"], [5, 4, 2, 2, 3, 1])[0]
    if kind == "batch":
        return _batch(None, rng.randint(6, 48), _log(rng, 48, 160), _log(rng, 300, 2048), rng.randint(20, 128),
                      rng.randrange(1 << 20), rng.choices(["layered", "persistent", "streams"], [3, 1, 1])[0])
    if kind == "gradbatch":
        return _gradbatch(None, rng.randint(2, 6), _log(rng, 32, 96), _log(rng, 97, 192), rng.randint(8, 32),
                          rng.randint(4, 16), rng.randrange(1 << 20))
    three = kind == "loop3" or (kind != "loop2" and rng.random() < 0.3)
    dtype = rng.choice(["f32", "f32", "f64"])
    mode = "exact" if kind == "host" else rng.choices(["fma", "exact"], [4, 1])[0]
    names = NAMES_3D if three else NAMES_2D
    if mode == "exact":
        names = [x for x in names if capi.info(x)["exact"]]
    if kind == "grad":
        # symmetric offset sets; the double-counted tap and the big boxes are
        # not differentiated in earnest
        names = [x for x in names if capi.info(x)["nterms"] <= 27 and x != "star2d4r"]
        mode = "fma"
    name = rng.choice(names)
    fpp = capi.info(name)["fpp"]
    top = {"loop2": 8192, "loop3": 448, "host": 160 if three else 2048, "grad": 160 if three else 2048}[kind]
    n = [_log(rng, 24 if three else 48, top) for _ in range(3 if three else 2)]
    if kind == "host":
        n = [n[0]] * len(n)  # the drop-in call takes one extent for all axes
    budget = 2e10 if dtype == "f64" or mode == "exact" or kind == "grad" else 5e10
    while fpp * math.prod(n) * 2 > budget:
        n = [max(16, int(x * 0.9)) for x in n]
    T = max(2, min(_log(rng, 4, 128), int(budget / (fpp * math.prod(n)))))
    if kind == "grad":
        return _grad(None, name, dtype, n, T, rng.randint(3, 32),
                     rng.random() < 0.5 and not (three and capi.info(name)["nterms"] > 13))
    return _loop(None, name, dtype, n, T, mode, "host" if kind == "host" else "loop")


def _n(case):
    return [case[k] for k in ("n0", "n1", "n2") if case[k]]


def _specs(case):
    """(stencil, extents, T) of each grid of a batch: the plan a program keeps."""
    rng = random.Random(case["mix"])
    if case["path"] == "gradbatch":
        return [(case["stencil"], [_log(rng, case["lo"], case["hi"]) for _ in range(3)], case["T"])
                for _ in range(case["count"])]
    return [(rng.choice(MIX), [_log(rng, case["lo"], case["hi"]) for _ in range(2)], rng.randint(8, case["tmax"]))
            for _ in range(case["count"])]


def _coef(name, dtype, seed):
    """Random coefficients of an average (None for the nonlinear stencil)."""
    s = capi.info(name)
    if s["kind"] != "linear":
        return None
    c = np.random.default_rng(seed).random(s["nterms"])
    return (c / c.sum() * (s["divisor"] or 1)).astype(NUMPY[dtype])


def _u0(name, dtype, n, seed):
    """One plane, halo included, U[0,1)."""
    r = capi.info(name)["rad"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand([x + 2 * r for x in n], generator=g, device="cuda", dtype=TORCH[dtype])


def _lam(name, dtype, n, seed):
    """dL/du_T: weights on the interior."""
    r = capi.info(name)["rad"]
    lam = torch.zeros([x + 2 * r for x in n], device="cuda", dtype=TORCH[dtype])
    g = torch.Generator(device="cuda").manual_seed(seed)
    lam[_inner(r, lam.dim())] = torch.rand(n, generator=g, device="cuda", dtype=TORCH[dtype]) - 0.5
    return lam


def _inner(r, dim, off=None):
    off = off or [0] * dim
    return tuple(slice(r + o, -r + o if o < r else None) for o in off)


def prepare(case, seed):
    path = case["path"]
    if path in ("loop", "host", "grad"):
        name, dtype, n = case["stencil"], case["dtype"], _n(case)
        coef = _coef(name, dtype, seed + 1)
        if path == "grad":
            u0 = _u0(name, dtype, n, seed).requires_grad_(True)
            c = None
            if coef is not None:
                c = torch.tensor(coef, device="cuda", requires_grad=case["want_coef"])
            return {"case": case, "u0": u0, "coef": c, "lam": _lam(name, dtype, n, seed + 2)}
        if path == "host":
            u0 = _u0(name, dtype, n, seed).cpu().numpy()
            return {"case": case, "A": np.stack([u0, u0]), "coef": coef}
        g = DeviceGrid(name, NUMPY[dtype], n)
        g.plane(0).copy_(_u0(name, dtype, n, seed))
        g.plane(1).copy_(g.plane(0))
        return {"case": case, "grid": g, "coef": coef}
    if path == "batch":
        entries = []
        for i, (name, n, T) in enumerate(_specs(case)):
            g = DeviceGrid(name, np.float32, n)
            g.plane(0).copy_(_u0(name, "f32", n, seed + 3 * i))
            g.plane(1).copy_(g.plane(0))
            entries.append((g, T, _coef(name, "f32", seed + 3 * i + 1)))
        return {"case": case, "entries": entries, "plan": capi.Batch(entries, case["mode"], case["schedule"])}
    specs = _specs(case)
    return {"case": case,
            "u0": [_u0(name, "f32", n, seed + 3 * i) for i, (name, n, _) in enumerate(specs)],
            "lam": [_lam(name, "f32", n, seed + 3 * i + 2) for i, (name, n, _) in enumerate(specs)]}


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "loop":
        g = state["grid"]
        g.run(case["T"], case["mode"], coef=state["coef"])
        return g.plane(case["T"] % 2)
    if path == "host":
        capi.kernel_stencil(state["A"], case["n0"], case["T"], stencil=case["stencil"], fp_mode=case["mode"],
                            coef=state["coef"])
        return state["A"][case["T"] % 2]
    if path == "batch":
        state["plan"].run(torch.cuda.current_stream().cuda_stream)
        return [g.plane(T % 2) for g, T, _ in state["entries"]]
    if path == "grad":
        u0, coef = state["u0"], state["coef"]
        u0.grad = None
        if coef is not None:
            coef.grad = None
        uT = adjoint.time_loop(u0, coef, case["stencil"], case["T"], case["every"])
        uT.backward(state["lam"])
        return [uT.detach(), u0.grad, coef.grad if coef is not None and case["want_coef"] else None]
    runs = adjoint.forward_batch([(case["stencil"], u) for u in state["u0"]], case["T"], case["every"])
    uT = [r.u_T for r in runs]
    grads, _ = adjoint.backward_batch(runs, state["lam"])
    return {"u_T": uT, "grad_u0": grads}


def work(case):
    def one(name, n, T, es, grad=False, coef=False):
        s = capi.info(name)
        cells = math.prod(n)
        flops = s["fpp"] * cells * T
        if grad:  # forward, the transposed steps and the products for the coefficients
            flops = 2 * flops + (2 * s["nterms"] * cells * T if coef else 0)
        return (4 if grad else 2) * es * cells, flops

    if case["path"] in ("batch", "gradbatch"):
        each = [one(name, n, T, 4, case["path"] == "gradbatch") for name, n, T in _specs(case)]
    else:
        each = [one(case["stencil"], _n(case), case["T"], 8 if case["dtype"] == "f64" else 4, case["path"] == "grad",
                    case.get("want_coef", False))]
    return {"bytes": float(sum(b for b, _ in each)), "flops": float(sum(f for _, f in each))}


def _step(name, u, coef):
    """One Jacobi step of the interior, halo fixed, in the type of u."""
    s = capi.info(name)
    r, d = s["rad"], u.dim()
    out = u.clone()
    c = u[_inner(r, d)]
    if s["kind"] != "linear":
        acc = torch.full_like(c, s["eps"])
        for o in s["neighbours"]:
            acc = acc + (c - u[_inner(r, d, o)]) ** 2
        out[_inner(r, d)] = c + s["numerator"] / acc.sqrt()
        return out
    acc = torch.zeros_like(c)
    for k, t in enumerate(s["terms"]):
        acc = acc + coef[k] * u[_inner(r, d, t["off"])]
    out[_inner(r, d)] = acc / s["divisor"] if s["divisor"] else acc
    return out


def _advance(name, u0, coef, T):
    u = u0.double()
    for _ in range(T):
        u = _step(name, u, coef)
    return u


def _reverse(name, u0, coef, lam, T, want_coef):
    """u_T, dL/du_0 and dL/dcoef (or None) at 64 bits, every state kept."""
    states = [u0.double()]
    for _ in range(T):
        states.append(_step(name, states[-1], coef))
    lam = lam.double()
    gc = torch.zeros_like(coef) if want_coef else None
    for t in range(T - 1, -1, -1):
        u = states[t].detach().requires_grad_(True)
        with torch.enable_grad():
            c = coef.detach().requires_grad_(True) if want_coef else coef
            got = torch.autograd.grad(_step(name, u, c), [u, c] if want_coef else [u], lam)
        lam = got[0]
        if want_coef:
            gc = gc + got[1]
    return states[-1], lam, gc


def exact(case, seed):
    def on_gpu(c):
        return None if c is None else torch.tensor(c, dtype=torch.float64, device="cuda")

    path = case["path"]
    with torch.no_grad():
        if path in ("loop", "host"):
            name, dtype, n = case["stencil"], case["dtype"], _n(case)
            if capi.info(name)["nterms"] * math.prod(n) * case["T"] > 4e11:
                return None
            got = _advance(name, _u0(name, dtype, n, seed), on_gpu(_coef(name, dtype, seed + 1)), case["T"])
            return got.cpu().numpy() if path == "host" else got
        if path == "batch":
            return [_advance(name, _u0(name, "f32", n, seed + 3 * i), on_gpu(_coef(name, "f32", seed + 3 * i + 1)), T)
                    for i, (name, n, T) in enumerate(_specs(case))]
        if path == "grad":
            name, dtype, n = case["stencil"], case["dtype"], _n(case)
            return list(_reverse(name, _u0(name, dtype, n, seed), on_gpu(_coef(name, dtype, seed + 1)),
                                 _lam(name, dtype, n, seed + 2), case["T"],
                                 case["want_coef"] and capi.info(name)["kind"] == "linear"))
        u, g = [], []
        for i, (name, n, T) in enumerate(_specs(case)):
            literals = torch.tensor([np.float32(t["value"]) for t in capi.info(name)["terms"]], dtype=torch.float64,
                                    device="cuda")
            a, b, _ = _reverse(name, _u0(name, "f32", n, seed + 3 * i), literals, _lam(name, "f32", n, seed + 3 * i + 2),
                               T, False)
            u.append(a)
            g.append(b)
        return {"u_T": u, "grad_u0": g}
