"""Timed cases of the engine's public entry points.

Each case is one call as a host code makes it: ``react`` on flat host or
device arrays, on species-major device arrays or on a box with a mask, with
each integrator and equation of state; the adjoint of ``react``; and the
transport coefficients of a box.  Fields and tolerances are those of
``pelephysics_b200/workloads.py``, the tests and the benchmark, at sizes from
a single cell to the 64^3 field.

The outputs are the state and energies after the call (and gradients, and
transport coefficients).  The work counters that calls report beside them
(right-hand sides per cell or in sum) are not results and are left out.
"""

import math
import os
import re

import numpy as np
import torch

import pelephysics_b200
from pelephysics_b200 import _lib, adjoint, transport, workloads
from pelephysics_b200.reactor import Reactor

TIGHT = dict(rtol=1e-10, atol=1e-10, max_order=5)  # the accuracy configurations
LOOSE = dict(rtol=1e-6, atol=1e-10, max_order=2)  # the defaults of ode.* and cvode.*
HEPTANE = dict(rtol=1e-8, atol=1e-12, max_order=5)

# per kind: mechanism, smallest and largest number of cells (or box edge)
RANGES = {
    "react": ("drm19", 1, 262144),
    "box": ("LiDryer", 3, 18),
    "large": ("dodecane_lu", 32, 24576),
    "heptane": ("heptane_lu_88sk", 32, 6144),
    "qss": ("CH4_lean_qss", 32, 65536),
    "srk": ("drm19", 32, 8192),
    "adjoint": ("drm19", 32, 16384),
    "arkode": ("drm19", 3, 32),
    "transport": ("", 3, 64),
}

# Mean integrator work per cell of each kind: right-hand sides, Jacobians,
# factorisations and Newton solves of a call (per-cell counters of the fields
# below); one right-hand side takes about 143 and one analytical Jacobian 273
# FP64 operations per reaction (drm19: 12,023 and 22,908).
COUNTS = {
    "react": (54.6, 1.09, 9.8, 51.6),
    "react loose": (17.9, 1.0, 5.4, 14.9),
    "box": (826.0, 14.8, 79.1, 823.6),
    "large": (38.0, 1.0, 9.7, 35.0),
    "heptane": (46.7, 1.07, 10.7, 43.7),
    "qss": (57.8, 0.0, 8.4, 40.7),  # the difference quotients' right-hand sides among the first
    "srk": (588.6, 0.0, 56.4, 496.7),
    "adjoint": (69.3, 1.24, 11.8, 66.3),
    "arkode": (321.0, 0.0, 0.0, 0.0),
}


def listed():
    return [
        # a zero-dimensional reactor: one cell on host arrays, default tolerances
        {"name": "one_cell_host", "kind": "react", "mech": "drm19", "cells": 1, "path": "host", "tight": False},
        # a small rank's leftover cells, an odd count, on device arrays
        {"name": "ragged_997", "kind": "react", "mech": "drm19", "cells": 997, "path": "flat", "tight": True},
        # an ordinary patch handed over on host arrays at the default tolerances
        {"name": "host_32768", "kind": "react", "mech": "drm19", "cells": 32768, "path": "host", "tight": False},
        # the 64^3 field of the benchmark
        {"name": "drm19_64cubed", "kind": "react", "mech": "drm19", "cells": 262144, "path": "flat", "tight": True},
        # a box of an adaptive mesh with covered (masked) cells: hydrogen ignition
        {"name": "lidryer_box", "kind": "box", "mech": "LiDryer", "nx": 16, "ny": 16, "nz": 16, "masked": 0.1},
        # a large mechanism at engine pressure with advective sources, species-major arrays
        {"name": "dodecane_16384", "kind": "large", "mech": "dodecane_lu", "cells": 16384, "fp32": False},
        # the largest mechanism, with the FP32 factor
        {"name": "heptane_4096_fp32", "kind": "heptane", "mech": "heptane_lu_88sk", "cells": 4096, "fp32": True},
        # a quasi-steady-state mechanism (difference-quotient Jacobian)
        {"name": "qss_16384", "kind": "qss", "mech": "CH4_lean_qss", "cells": 16384},
        # the real-gas reactor at 50 atm
        {"name": "srk_4097", "kind": "srk", "mech": "drm19", "cells": 4097},
        # gradients of a loss on the final state with respect to rates and initial state
        {"name": "adjoint_8192", "kind": "adjoint", "mech": "drm19", "cells": 8192},
        # the batch-coupled explicit integrator on a ragged box
        {"name": "arkode_box", "kind": "arkode", "mech": "drm19", "nx": 28, "ny": 24, "nz": 20},
        # transport coefficients of a box, the Soret option on
        {"name": "transport_box", "kind": "transport", "mech": "heptane_lu_88sk", "nx": 40, "ny": 36, "nz": 28,
         "soret": True},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["react", "react", "react", "box", "large", "heptane", "qss", "srk", "adjoint", "arkode",
                       "transport"])
    mech, lo, hi = RANGES[kind]
    if kind == "react":
        return {"kind": kind, "mech": mech, "cells": _spread(rng, lo, hi), "path": rng.choice(["host", "flat", "soa"]),
                "tight": rng.random() < 0.5}
    if kind == "transport":
        mech = rng.choice(["LiDryer", "drm19", "dodecane_lu", "heptane_lu_88sk"])
    if kind in ("box", "arkode", "transport"):
        case = {"kind": kind, "mech": mech}
        for d in ("nx", "ny", "nz"):
            case[d] = _spread(rng, lo, hi)
        if kind == "box":
            case["masked"] = rng.choice([0.0, 0.1, 0.5])
        if kind == "transport":
            case["soret"] = rng.random() < 0.5
        return case
    case = {"kind": kind, "mech": mech, "cells": _spread(rng, lo, hi)}
    if kind in ("large", "heptane"):
        case["fp32"] = rng.random() < 0.5
    return case


def _ncells(case):
    return case["cells"] if "cells" in case else case["nx"] * case["ny"] * case["nz"]


def _slice(cells, n):
    """The first n cells of a field: a contiguous range, as a rank owns one."""
    return cells.rY[:n].copy(), cells.rYsrc[:n].copy(), cells.rX[:n].copy(), cells.rX_src[:n].copy()


def _drm19(n, seed):
    edge = max(2, math.ceil(round(n ** (1.0 / 3.0), 9)))
    return _slice(workloads.drm19_field(edge, seed=seed + 1), n)


def _fields(case, seed):
    """rY, rYsrc, rX, rX_src of the case on the host, and dt."""
    kind, n = case["kind"], _ncells(case)
    if kind == "react":
        return _drm19(n, seed) + (1e-5,)
    if kind == "arkode":
        return _drm19(n, seed) + (1e-6,)
    if kind == "srk":  # the field compressed to 50 atm; the energies scale with the density
        rY, src, rX, rXs = _drm19(n, seed)
        rY[:, :-1] *= 50.0
        return rY, src, rX * 50.0, rXs, 1e-5
    if kind == "box":
        c = workloads.premix_cells("LiDryer", n, seed, 1000.0, 400.0, 0.5, 1.5, dt=1e-4)
    elif kind == "large":
        edge = max(4, math.ceil(round(n ** (1.0 / 3.0), 9)))
        c = workloads.dodecane_field((edge, edge, edge), seed=seed + 2)
    elif kind == "heptane":
        c = workloads.heptane_cells(n, seed=seed + 5)
    elif kind == "qss":
        c = workloads.premix_cells("CH4_lean_qss", n, seed, 1100.0, 1000.0, 0.5, 0.5, dt=1e-5)
    elif kind == "adjoint":
        c = workloads.premix_cells("drm19", n, seed, 1100.0, 500.0, 0.5, 1.5, reactor_type=2, dt=5e-4)
    return _slice(c, n) + (c.dt,)


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _transport_inputs(case, seed):
    """Y [N, nz, ny, nx], T and rho [1, nz, ny, nx]: flame-like states of all species."""
    g = torch.Generator(device="cuda").manual_seed(seed + 11)
    N, shape = _lib.mechanism_info(case["mech"])[0], (case["nz"], case["ny"], case["nx"])
    rand = lambda *s: torch.rand(*s, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    Y = rand(N, *shape) ** 3 * (rand(N, *shape) > 0.2)
    Y[-1] += 0.5  # a bath gas
    return Y / Y.sum(0), 300.0 + 2500.0 * rand(1, *shape), 10.0 ** (-4.0 + 2.0 * rand(1, *shape))


def prepare(case, seed):
    kind, n = case["kind"], _ncells(case)
    s = {"case": dict(case), "lo": (0, 0, 0)}
    if "nx" in case:
        s["hi"] = (case["nx"] - 1, case["ny"] - 1, case["nz"] - 1)
    if kind == "transport":
        s["Y"], s["T"], s["rho"] = _transport_inputs(case, seed)
        empty = lambda m: torch.zeros((m,) + tuple(s["T"].shape[1:]), dtype=torch.float64, device="cuda")  # noqa: E731
        s["out"] = [empty(s["Y"].shape[0]) for _ in range(2)] + [empty(1) for _ in range(3)]
        return s
    rY, src, rX, rXs, dt = _fields(case, seed)
    s["dt"] = dt
    opts = dict(HEPTANE if kind == "heptane" else TIGHT if case.get("tight", kind != "arkode") else LOOSE)
    if case.get("fp32"):
        opts.update(lu_fp32=1)
    if kind == "srk":
        opts.update(eos=1)
    s["reactor"] = Reactor(case["mech"], "ReactorArkode" if kind == "arkode" else "ReactorCvode")
    s["reactor"].init(2 if kind == "adjoint" else 1, n, **opts)
    if case.get("path") == "host":
        s["host"] = [np.ascontiguousarray(a) for a in (rY, src, rX, rXs)]
        s["y"], s["x"] = np.empty_like(s["host"][0]), np.empty_like(s["host"][2])
        return s
    if kind in ("box", "arkode"):
        shape = (case["nz"], case["ny"], case["nx"])
        comp = lambda a: _dev(a.reshape(n, -1).T).reshape((-1,) + shape)  # noqa: E731
        s["rY0"], s["T0"], s["rYsrc"] = comp(rY[:, :-1]), comp(rY[:, -1:]), comp(src)
        s["rE0"], s["rEs"] = comp(rX), comp(rXs)
        s["rY"], s["T"], s["rE"] = (torch.empty_like(s[k]) for k in ("rY0", "T0", "rE0"))
        s["FC"] = torch.zeros((1,) + shape, dtype=torch.float64, device="cuda")
        s["mask"] = None
        if case.get("masked"):
            covered = np.random.default_rng(seed + 21).uniform(size=(1,) + shape) < case["masked"]
            s["mask"] = torch.as_tensor(np.where(covered, -1, 1).astype(np.int32), device="cuda")
        return s
    if case.get("path") == "soa" or kind in ("large", "heptane"):
        s["path"] = "soa"
        rY, src = rY.T, src.T
    s["y0"], s["src"], s["x0"], s["xs"] = _dev(rY), _dev(src), _dev(rX), _dev(rXs)
    if kind == "adjoint":
        w = np.random.default_rng(seed + 4).normal(size=(2, n))
        i_oh = [k.lower() for k in _lib.species_names(case["mech"])].index("oh")
        # the seed dL/dy of L = sum(w_T T + w_OH Y_OH), as a caller's loss gives it
        s["lam"] = adjoint.loss_T_OH(s["y0"], i_oh, _dev(w[0]), _dev(w[1]))[1].contiguous()
    else:
        s["y"], s["x"] = torch.empty_like(s["y0"]), torch.empty_like(s["x0"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "transport":
        D, chi, mu, xi, lam = s["out"]
        transport.transport_box(case["mech"], s["lo"], s["hi"], s["Y"], s["T"], s["rho"], D, chi, mu, xi, lam,
                                use_soret=case["soret"])
        return {"D": D, "chi": chi, "mu": mu, "xi": xi, "lam": lam}
    r = s["reactor"]
    # react() advances in place: each pass starts from the prepared state
    if case.get("path") == "host":
        y0, src, x0, xs = s["host"]
        s["y"][...] = y0
        s["x"][...] = x0
        r.react(s["y"], src, s["x"], xs, s["dt"])
        return {"rY": s["y"], "rX": s["x"]}
    if kind in ("box", "arkode"):
        s["rY"].copy_(s["rY0"])
        s["T"].copy_(s["T0"])
        s["rE"].copy_(s["rE0"])
        r.react_box(s["lo"], s["hi"], s["rY"], s["rYsrc"], s["T"], s["rE"], s["rEs"], s["FC"], mask=s["mask"],
                    dt_react=s["dt"])
        return {"rY": s["rY"], "T": s["T"], "rE": s["rE"]}
    if kind == "adjoint":
        y, lam_y0, lam_e, grad = r.adjoint(s["y0"], s["src"], s["x0"], s["xs"], s["dt"], s["lam"])
        return {"y": y, "lam_y0": lam_y0, "lam_e": lam_e, "grad": grad}
    s["y"].copy_(s["y0"])
    s["x"].copy_(s["x0"])
    if s.get("path") == "soa":
        r.react_soa(s["y"], s["src"], s["x"], s["xs"], s["dt"])
    else:
        r.react(s["y"], s["src"], s["x"], s["xs"], s["dt"])
    return {"rY": s["y"], "rX": s["x"]}


def work(case):
    kind, n = case["kind"], _ncells(case)
    N, R = _lib.mechanism_info(case["mech"])
    m = N + 1
    if kind == "transport":
        pairs = N * (N - 1) / 2
        return {"bytes": 8.0 * n * (N + 2 + N + 3 + (N if case["soret"] else 0)),
                "flops": n * (pairs * 55.0 + N * 160.0)}
    rhs, jac, lu, solve = COUNTS["react loose" if kind == "react" and not case["tight"] else kind]
    flops = rhs * 143.0 * R + jac * 273.0 * R + lu * (2.0 / 3.0 * m ** 3 + m * m) + solve * 2.0 * m * m
    # state and energies in and out, sources in
    size = 8.0 * n * (2 * m + N + 3)
    if kind == "adjoint":  # forward, and the reverse sweep's solves with the transposed matrices
        return {"bytes": size + 8.0 * n * (2 * m + 1) + 24.0 * R, "flops": 3.0 * n * flops}
    return {"bytes": size, "flops": n * flops}


def _table(text, mech, name):
    body = re.search(r"ppbt_%s_%s\[\] = \{(.*?)\}" % (re.escape(mech), name), text, re.S).group(1)
    return np.array([float(v) for v in body.replace("\n", " ").split(",") if v.strip()])


def _nasa_cv(mech, path, T):
    """cv/R of each species [N, cells] from the mechanism's NASA-7 table."""
    with open(path) as f:
        text = f.read()
    arr = {}
    for name in ("tmid", "th_cv"):
        body = re.search(r"\w*_%s\[\] = \{(.*?)\}" % name, text, re.S).group(1)
        arr[name] = np.array([float(v) for v in body.replace("\n", " ").split(",") if v.strip()])
    tmid = arr["tmid"]
    c = arr["th_cv"].reshape(len(tmid), 2, 5)
    low = (tmid[:, None] >= 0.0) & (T[None] < tmid[:, None])
    p = np.stack([T ** k for k in range(5)])
    return np.where(low, c[:, 0] @ p, c[:, 1] @ p)


def exact(case, seed):
    """The mixture-averaged transport formulas in plain numpy, from the tables'
    values.  None for the integrations: a converged stiff integration of a
    batch in plain torch or numpy takes minutes."""
    if case["kind"] != "transport":
        return None
    mech = case["mech"]
    N = _lib.mechanism_info(mech)[0]
    n = _ncells(case)
    Y, T, _ = _transport_inputs(case, seed)
    shape = tuple(T.shape[1:])
    Y, T = Y.reshape(N, n).cpu().numpy(), T.reshape(n).cpu().numpy()
    folder = os.path.join(list(pelephysics_b200.__path__)[0], "csrc", "mech")
    with open(os.path.join(folder, "trans_%s.h" % mech)) as f:
        text = f.read()
    tab = {k: _table(text, mech, k) for k in ("wt", "eps", "zrot", "nlin", "fitmu", "fitlam", "fitdbin", "ktdif",
                                              "fittdrat", "cvms")}
    ru, patm = 8.31446261815324e7, 1.01325e6
    wt = tab["wt"][:, None]
    L = np.log(T)
    logs = np.stack([np.ones_like(L), L, L * L, L * L * L])
    yl = Y + 1e-15 * (Y.sum(0) / N - Y)
    X = yl / wt / (yl / wt).sum(0)
    mus = np.exp(tab["fitmu"].reshape(N, 4) @ logs)
    mu = (X * mus ** 6).sum(0) ** (1.0 / 6.0)
    lam = (X * np.exp(tab["fitlam"].reshape(N, 4) @ logs) ** 0.25).sum(0) ** 4
    # bulk viscosity
    cvk = _nasa_cv(mech, os.path.join(folder, "mech_%s.h" % mech), T) * tab["cvms"][:, None]
    cint = cvk * wt / ru - 1.5
    crot = np.where(tab["nlin"] == 1, 1.0, 1.5)[:, None]
    fn = lambda e: 1 + 0.5 * np.pi ** 1.5 * np.sqrt(e) + (2 + 0.5 * np.pi ** 2) * e + (np.pi * e) ** 1.5  # noqa: E731
    eps = tab["eps"][:, None]
    xs = 0.25 * np.pi * (cint / (cint + 1.5)) ** 2 * tab["zrot"][:, None] / crot * fn(eps / 298.0) / fn(eps / T) * mus
    xs = np.where(tab["nlin"][:, None] == 0, 0.0, xs)
    xi = (X * xs ** 0.75).sum(0) ** (4.0 / 3.0)
    # mixture-averaged diffusion: sum over the others of X_j / D_ij
    fit = tab["fitdbin"].reshape(N, N, 4)  # [j, i]
    den = np.zeros((N, n))
    for i in range(N):
        e = np.exp(-(fit[:, i] @ logs)) * X
        den[i] = e.sum(0) - e[i]
    D = wt * (yl.sum(0) - yl) / den * patm / (ru * T)
    chi = np.zeros((N, n))
    if case["soret"]:
        powers = np.stack([T ** k for k in range(4)])
        for m, i in enumerate(tab["ktdif"].astype(int)):
            t = X * (tab["fittdrat"].reshape(-1, N, 4)[m] @ powers)
            chi[i] = (t.sum(0) - t[i]) * X[i]
    return {"D": D.reshape((N,) + shape), "chi": chi.reshape((N,) + shape), "mu": mu.reshape((1,) + shape),
            "xi": xi.reshape((1,) + shape), "lam": lam.reshape((1,) + shape)}
