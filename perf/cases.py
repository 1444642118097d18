"""The work a user has the provider do, as cases that can be timed and checked.

Every case goes through the public entry points: a solver (or a batch) made
once, and per pass the state handed over, advanced, and read back.

  grid      one grid: sfg_upload_device, sfg_advance over `steps` CFL steps,
            sfg_download_device
  residual  the spatial operator alone on caller-owned device arrays
            (sfg_residual_noalloc), as a host time integrator calls it
  batch     many grids of uneven sizes and two recipes: sfg_batch_add with host
            arrays, sfg_batch_step, sfg_batch_download, sfg_batch_remove

Grid keys: dim, nx, ny, nz (nodes), bc ("periodic" | "transmissive"), flow,
recipe, time (time recipe), prec ("fp64" | "fp32"), variant (the kernel variant
the autotuner picks; -1: the library's default), curved (wavy mesh with
per-node metrics), steps.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from sonicsolver_b200 import capi, cases as wl

GAMMA = 1.4


# ------------------------------------------------------------------ the cases

def _grid(name, dim, n, bc, flow, recipe, prec, steps, time="SSPRK3", variant=-1, curved=False):
    n = tuple(n) + (1,) * (3 - len(n))
    c = {"kind": "grid", "dim": dim, "nx": n[0], "ny": n[1], "nz": n[2], "bc": bc, "flow": flow, "recipe": recipe,
         "time": time, "prec": prec, "variant": variant, "curved": curved, "steps": steps}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the 1-D Sod tube of the reference's own golden case, at its 1000 cells: one short run, all latency
        _grid("sod1d_1000", 1, (1001,), "transmissive", "tube", "weno5Rusanov", "fp64", 256),
        # a small 2-D study, where a step's launches count
        _grid("vortex2d_64", 2, (64, 64), "periodic", "vortex", "teno5Rusanov", "fp64", 64),
        # a mid-size shock problem on an odd, non-square grid, Roe faces
        _grid("tube2d_257x193", 2, (257, 193), "transmissive", "tube", "weno5Roe", "fp64", 48),
        # the isentropic vortex at 1024^2, plain precision
        _grid("vortex2d_1024_fp64", 2, (1024, 1024), "periodic", "vortex", "teno5Rusanov", "fp64", 12),
        # the same with FP32 fluxes: the headline workload
        _grid("vortex2d_1024_fp32", 2, (1024, 1024), "periodic", "vortex", "teno5Rusanov", "fp32", 24),
        # Taylor-Green 256^3 in plain precision (the autotuner keeps the axis sweeps there)
        _grid("tgv3d_256_fp64", 3, (256, 256, 256), "periodic", "taylor_green", "weno5Rusanov", "fp64", 3),
        # and with FP32 fluxes on the 3-D tiles the autotuner picks
        _grid("tgv3d_256_fp32", 3, (256, 256, 256), "periodic", "taylor_green", "weno5Rusanov", "fp32", 4, variant=1),
        # a 3-D shock box with ragged extents, the high-order scheme and classical RK4
        _grid("tube3d_97x83x61", 3, (97, 83, 61), "transmissive", "tube", "weno7Rusanov", "fp64", 8,
              time="classicalRK4"),
        # a curved (wavy) mesh with per-node metrics, both precisions
        _grid("wavy2d_768_fp64", 2, (768, 768), "periodic", "vortex", "teno5Rusanov", "fp64", 10, curved=True),
        _grid("wavy2d_1024_fp32", 2, (1024, 1024), "periodic", "vortex", "teno5Rusanov", "fp32", 12, curved=True),
        # the operator alone on a caller's arrays: the smallest call there is
        {"name": "residual2d_160x120", "kind": "residual", "dim": 2, "nx": 160, "ny": 120, "nz": 1, "bc": "periodic",
         "flow": "vortex", "recipe": "weno5Rusanov", "prec": "fp64"},
        # many small jobs side by side, as a served mix has them: shock tubes (1-D, 2-D) with vortices among them
        {"name": "batch_64_mixed_fp32", "kind": "batch", "count": 64, "max_1d": 16384, "max_2d": 384,
         "prec": "fp32", "steps": 96},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["g1", "g2", "g2", "g2", "g3", "g3", "curved", "residual", "batch"])
    time = rng.choice(["SSPRK3", "SSPRK3", "SSPRK3", "forwardEuler", "classicalRK4"])
    prec = rng.choice(["fp64", "fp32"])
    bc = "periodic" if kind == "curved" else "transmissive" if kind == "g1" else rng.choice(["periodic", "transmissive"])
    flow = "vortex" if bc == "periodic" else "tube"
    # TENO5 on the smooth flows, as the project's own workloads have it: beside a shock its cut-off turns the
    # round-off ahead of the front into whole sub-stencils, so that no two correct runs agree there.  WENO3 (the
    # reference's four-point form) loses positivity at strong shocks.
    schemes = ["weno5", "weno5", "weno7"] + (["weno3"] + ["teno5"] * 4 if flow == "vortex" else [])
    recipe = rng.choice(schemes) + rng.choice(["Rusanov", "Rusanov", "Roe"])
    if kind == "g1":
        nx = _log_int(rng, 200, 8000)
        return _grid(None, 1, (nx,), bc, flow, recipe, "fp64", min(rng.randint(48, 200), nx // 4), time)
    if kind == "g2":
        nx = _log_int(rng, 48, 1024)
        ny = min(1024, max(32, int(nx * rng.uniform(0.5, 1.6))))
        steps = max(6, min(64, nx // 3, ny // 3, 10_000_000 // (nx * ny)))
        return _grid(None, 2, (nx, ny), bc, flow, recipe, prec, steps, time)
    if kind == "g3":
        n = [_log_int(rng, 24, 200) for _ in range(3)]
        steps = max(2, min(16, min(n) // 4, 8_000_000 // (n[0] * n[1] * n[2])))
        return _grid(None, 3, n, bc, "taylor_green" if bc == "periodic" else "tube", recipe, prec, steps, time,
                     variant=1 if prec == "fp32" else -1)
    if kind == "curved":
        nx, ny = _log_int(rng, 64, 900), _log_int(rng, 64, 900)
        steps = max(4, min(32, 4_000_000 // (nx * ny)))
        return _grid(None, 2, (nx, ny), "periodic", "vortex", recipe, prec, steps, curved=True)
    if kind == "residual":
        d = rng.choice([1, 2, 3])
        n = ([_log_int(rng, 100, 100_000), 1, 1] if d == 1 else [_log_int(rng, 40, 500), _log_int(rng, 40, 500), 1]
             if d == 2 else [_log_int(rng, 16, 62) for _ in range(3)])
        return {"kind": "residual", "dim": d, "nx": n[0], "ny": n[1], "nz": n[2], "bc": bc,
                "flow": flow if d < 3 or bc == "transmissive" else "taylor_green", "recipe": recipe, "prec": prec}
    return {"kind": "batch", "count": rng.randint(8, 80), "max_1d": _log_int(rng, 1024, 16384),
            "max_2d": _log_int(rng, 96, 384), "prec": prec, "steps": rng.randint(24, 96)}


# ------------------------------------------------------------------ inputs

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _spacing(case):
    """Node spacing: unit length (tubes), [0, 10]^d (vortex), [0, 2 pi]^3 (Taylor-Green) along x."""
    length = {"tube": 1.0, "vortex": 10.0, "taylor_green": 2 * math.pi}[case["flow"]]
    n = (case["nx"], case["ny"], case["nz"])
    h = [1.0, 1.0, 1.0]
    for d in range(case["dim"]):
        cells = n[d] if case["bc"] == "periodic" else n[d] - 1
        h[d] = length / cells
    return n, h


def _mesh(case):
    """Node coordinates (X, Y, Z) and, on a curved mesh, the ten metrics per node."""
    n, h = _spacing(case)
    ax = [torch.arange(n[d], dtype=torch.float64, device=_device()) for d in range(3)]
    K, J, I = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    X, Y, Z = I * h[0], J * h[1], K * h[2]
    if not case.get("curved"):
        return (X, Y, Z), None
    # x = i hx + A sin(2 pi j / ny), y = j hy + A sin(2 pi i / nx)
    A = 0.3 * 10.0 / (2 * math.pi)
    kx, ky = 2 * math.pi / n[0], 2 * math.pi / n[1]
    X, Y = X + A * torch.sin(ky * J), Y + A * torch.sin(kx * I)
    xj, yi = A * ky * torch.cos(ky * J), A * kx * torch.cos(kx * I)
    det = h[0] * h[1] - xj * yi
    one, zero = torch.ones_like(X), torch.zeros_like(X)
    M = torch.stack([1 / det, h[1] / det, -xj / det, zero, -yi / det, h[0] / det, zero, zero, zero, one], -1)
    return (X, Y, Z), M


def _state(case, seed):
    """Conserved state [nz][ny][nx][5] of the case's flow, its parameters from the seed."""
    r = np.random.default_rng([int(seed), case["nx"], case["ny"], case["nz"]])
    (X, Y, Z), metrics = _mesh(case)
    w = torch.zeros_like(X)
    if case["flow"] == "tube":
        # two states, the diaphragm through the middle at an angle
        rl, pl = r.uniform(0.8, 1.2), r.uniform(0.8, 1.2)
        rr, pr = r.uniform(0.15, 0.3), r.uniform(0.12, 0.25)
        ul, ur = r.uniform(-0.1, 0.1, 2)
        th, ph = (r.uniform(0, math.pi) if case["dim"] > 1 else 0.0), (r.uniform(0.3, 1.2) if case["dim"] > 2 else math.pi / 2)
        nv = (math.cos(th) * math.sin(ph), math.sin(th) * math.sin(ph), math.cos(ph) if case["dim"] > 2 else 0.0)
        s = (X - 0.5) * nv[0]
        if case["dim"] > 1:
            s = s + (Y - 0.5) * nv[1]
        if case["dim"] > 2:
            s = s + (Z - 0.5) * nv[2]
        left = (s < 0).double()
        rho, p, un = rr + (rl - rr) * left, pr + (pl - pr) * left, ur + (ul - ur) * left
        u, v, w = un * nv[0], un * nv[1], un * nv[2]
    elif case["flow"] == "vortex":
        xc, yc = r.uniform(3, 7, 2)
        ui, vi = r.uniform(0.6, 1.3, 2)
        beta = r.uniform(4.0, 5.5)
        if case["dim"] == 1:
            yc, Y = 0.0, torch.zeros_like(X)
        dx, dy = (X - xc + 5) % 10 - 5, (Y - yc + 5) % 10 - 5
        e = torch.exp(0.5 * (1 - dx * dx - dy * dy))
        u = ui - beta / (2 * math.pi) * e * dy
        v = vi + beta / (2 * math.pi) * e * dx
        T = 1 - (GAMMA - 1) * beta ** 2 / (8 * GAMMA * math.pi ** 2) * e * e
        rho = T ** (1 / (GAMMA - 1))
        p = rho ** GAMMA
    else:
        a, b, c = r.uniform(0, 2 * math.pi, 3)
        X, Y, Z = X + a, Y + b, Z + c
        u = torch.sin(X) * torch.cos(Y) * torch.cos(Z)
        v = -torch.cos(X) * torch.sin(Y) * torch.cos(Z)
        rho = torch.ones_like(X)
        p = 1 / (GAMMA * 0.01) + (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2) / 16
    E = p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v + w * w)
    return torch.stack([rho, rho * u, rho * v, rho * w, E], -1).contiguous(), metrics


def _cfl(case):
    if case.get("time") == "forwardEuler":
        return 0.2
    return 0.4 if case["flow"] == "vortex" else 0.5


def _bc(case):
    b = capi.BC_PERIODIC if case["bc"] == "periodic" else capi.BC_TRANSMISSIVE
    return tuple(b if d < case["dim"] else capi.BC_TRANSMISSIVE for d in range(3))


def _prec(case):
    return capi.PREC_FP64 if case["prec"] == "fp64" else capi.PREC_FP32_FLUX


def _tube2d(side, angle, left, right):
    """Two states (rho, u_n, p) on the unit square, the diaphragm through the centre at an angle."""
    x = np.arange(side + 1) / side
    X, Y = np.meshgrid(x, x, indexing="xy")
    c, s = math.cos(angle), math.sin(angle)
    at = (X - 0.5) * c + (Y - 0.5) * s < 0
    rho, un, p = (np.where(at, a, b) for a, b in zip(left, right))
    q = wl.conserved(rho, un * c, un * s, 0.0, p, GAMMA)[None]
    return wl.Case("tube2d", 2, (side + 1, side + 1, 1), (1.0 / side, 1.0 / side, 1.0), (0, 0, 0), (0, 0, 0), q, GAMMA,
                   1e9, 0.5, "weno5Rusanov")


def _batch_grids(case, seed):
    """The batch's grids: shock tubes, 1-D and 2-D, and every fourth grid a periodic vortex.  The sizes are
    the case's, the states the seed's."""
    rng = np.random.default_rng([int(seed), case["count"]])
    sizes = np.random.default_rng([case["count"], case["max_1d"], case["max_2d"]])

    def size(lo, hi):
        return int(round(math.exp(sizes.uniform(math.log(lo), math.log(hi)))))

    grids = []
    for k in range(case["count"]):
        left = (rng.uniform(0.6, 2.0), rng.uniform(-0.2, 0.2), rng.uniform(0.6, 2.0))
        right = (rng.uniform(0.1, 0.5), rng.uniform(-0.2, 0.2), rng.uniform(0.1, 0.5))
        if k % 4 == 3:
            grids.append(wl.isentropic_vortex(size(48, case["max_2d"]), beta=float(rng.uniform(4.0, 5.5)), t_end=1e9))
        elif k % 2:
            grids.append(_tube2d(size(64, case["max_2d"]), rng.uniform(0, math.pi), left, right))
        else:
            grids.append(wl.sod_1d(size(256, case["max_1d"]), GAMMA, left, right, t_end=1e9))
    return grids


def prepare(case, seed):
    if case["kind"] == "batch":
        grids = _batch_grids(case, seed)
        b = capi.Batch(sum(200 * g.nodes + 4096 for g in grids) + (1 << 21), len(grids), recipe="weno5Rusanov",
                       precision=_prec(case))
        return {"case": case, "batch": b, "grids": grids}
    q, metrics = _state(case, seed)
    n, h = _spacing(case)
    bc = _bc(case)
    if case["kind"] == "residual":
        soa = q.reshape(-1, 5).t().contiguous()
        r = torch.empty_like(soa)
        torch.cuda.synchronize()
        return {"case": case, "n": n, "h": h, "bc": bc, "q": soa, "r": r}
    s = capi.Solver(case["dim"], n, h, bc, bc, recipe=case["recipe"], time_recipe=case["time"], precision=_prec(case),
                    gamma=GAMMA, cfl=_cfl(case))
    if metrics is not None:
        s.set_metrics(metrics.cpu().numpy())
    if case["variant"] >= 0:
        s.variant = case["variant"]
    out = torch.empty_like(q)
    torch.cuda.synchronize()
    return {"case": case, "solver": s, "q": q, "out": out}


# ------------------------------------------------------------------ one pass

def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        slots = [b.add(g, recipe=g.recipe, cfl=g.cfl) for g in state["grids"]]
        b.step(case["steps"])
        out = [b.download(s) for s in slots]
        times = np.array([b.status(s)["time"] for s in slots])
        for s in slots:
            b.remove(s)
        flat = np.concatenate([x.reshape(-1) for x in out])
        return {"states": flat, "tube": out[0], "vortex": out[3], "times": times}
    if case["kind"] == "residual":
        capi.residual_noalloc(case["dim"], state["n"], state["h"], state["bc"], state["bc"], state["q"].data_ptr(),
                              state["r"].data_ptr(), recipe=case["recipe"], precision=_prec(case), gamma=GAMMA)
        return state["r"]
    s, lib = state["solver"], capi.lib()
    capi.check(lib.sfg_upload_device(s.handle, ctypes.c_void_p(state["q"].data_ptr()), 0.0))
    st, dts = s.advance(1e9, max_steps=case["steps"], dt_capacity=case["steps"])
    capi.check(lib.sfg_download_device(s.handle, ctypes.c_void_p(state["out"].data_ptr())))
    return {"q": state["out"], "dt": dts}


# ------------------------------------------------------------------ what a pass cannot do without

_STAGES = {"forwardEuler": 1, "SSPRK3": 3, "classicalRK4": 4}
# floating-point operations of one face: basis of the face state, five
# stencils' differences projected, five reconstructions on both sides, back to
# conserved variables, the flux
_CORE = {"weno3": 50, "weno5": 115, "teno5": 95, "weno7": 260}


def _face_flops(recipe):
    scheme = recipe[:5]
    points = {"weno3": 3, "weno7": 7}.get(scheme, 5)
    return 45 + points * 26 + 5 * _CORE[scheme] + 45 + (110 if recipe.endswith("Rusanov") else 210)


def _stage_flops(dim, nodes, recipe, curved=False):
    return nodes * (dim * (_face_flops(recipe) + (90 if curved else 0)) + 40)


def work(case):
    if case["kind"] == "batch":
        # sizes are log-uniform: their means stand for the seeded draw
        def mean(lo, hi, p):
            return (hi ** p - lo ** p) / (p * math.log(hi / lo)) if hi > lo else lo ** p
        v, n1 = case["count"] // 4, (case["count"] + 1) // 2
        one, two, vor = mean(256, case["max_1d"], 1), mean(64, case["max_2d"], 2), mean(48, case["max_2d"], 2)
        n2 = case["count"] - v - n1
        cells = n1 * one + n2 * two + v * vor
        per = n1 * _stage_flops(1, one, "weno5Rusanov") + n2 * _stage_flops(2, two, "weno5Rusanov") + \
            v * _stage_flops(2, vor, "teno5Rusanov")
        return {"bytes": 80.0 * cells, "flops": 3.0 * case["steps"] * per}
    nodes = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "residual":
        return {"bytes": 80.0 * nodes, "flops": float(_stage_flops(case["dim"], nodes, case["recipe"]))}
    return {"bytes": (80.0 + (80.0 if case["curved"] else 0.0)) * nodes,
            "flops": float(case["steps"]) * _STAGES[case["time"]] *
            _stage_flops(case["dim"], nodes, case["recipe"], case["curved"])}


def tolerance(case):
    # About four times what was seen against exact() over the ranges.  FP64:
    # round-off (1e-15 on WENO5 states, 2e-11 of a residual, which is the
    # small difference of large fluxes); where TENO5 runs, the cut-offs that
    # turn on that round-off in a coarse vortex's far field (2e-8).  FP32
    # fluxes on an FP64 state: 3e-7 of the state, 4e-4 of a residual.
    if case["prec"] == "fp64":
        teno = case["kind"] == "batch" or case["recipe"].startswith("teno5")
        return {"rel": 8e-8, "max": 8e-6} if teno else {"rel": 1e-10, "max": 1e-8}
    if case["kind"] == "residual":
        return {"rel": 1.6e-3, "max": 2.6e-2}
    return {"rel": 1e-6, "max": 5e-5}


# ------------------------------------------------------------------ the same in 64 bits, in plain torch

def _weno3(v):
    p = [(-v[0] + 5 * v[1] + 2 * v[2]) / 6, (2 * v[1] + 5 * v[2] - v[3]) / 6]
    a = [d / (1e-6 + b * b) ** 2 for d, b in ((1 / 3, v[2] - v[0]), (2 / 3, v[3] - v[1]))]
    return (a[0] * p[0] + a[1] * p[1]) / (a[0] + a[1])


def _polys5(v):
    return [(2 * v[0] - 7 * v[1] + 11 * v[2]) / 6, (-v[1] + 5 * v[2] + 2 * v[3]) / 6, (2 * v[2] + 5 * v[3] - v[4]) / 6]


def _betas5(v):
    return [13 / 12 * (v[0] - 2 * v[1] + v[2]) ** 2 + 0.25 * (v[0] - 4 * v[1] + 3 * v[2]) ** 2,
            13 / 12 * (v[1] - 2 * v[2] + v[3]) ** 2 + 0.25 * (v[1] - v[3]) ** 2,
            13 / 12 * (v[2] - 2 * v[3] + v[4]) ** 2 + 0.25 * (3 * v[2] - 4 * v[3] + v[4]) ** 2]


def _weno5(v):
    p, b = _polys5(v), _betas5(v)
    a = [d / (1e-6 + x) ** 2 for d, x in zip((0.1, 0.6, 0.3), b)]
    return (a[0] * p[0] + a[1] * p[1] + a[2] * p[2]) / (a[0] + a[1] + a[2])


def _teno5(v):
    p, b = _polys5(v), _betas5(v)
    tau = (b[0] - b[2]).abs()
    g = [(1 + tau / (x + 1e-40)) ** 6 for x in b]
    s = g[0] + g[1] + g[2]
    a = [d * (x >= 1e-5 * s).to(x.dtype) for x, d in zip(g, (0.1, 0.6, 0.3))]
    return (a[0] * p[0] + a[1] * p[1] + a[2] * p[2]) / (a[0] + a[1] + a[2])


def _weno7(v):
    p = [(-3 * v[0] + 13 * v[1] - 23 * v[2] + 25 * v[3]) / 12, (v[1] - 5 * v[2] + 13 * v[3] + 3 * v[4]) / 12,
         (-v[2] + 7 * v[3] + 7 * v[4] - v[5]) / 12, (3 * v[3] + 13 * v[4] - 5 * v[5] + v[6]) / 12]
    num = den = 0.0
    for k, d in enumerate((1 / 35, 12 / 35, 18 / 35, 4 / 35)):
        lo, hi = 2.5 - k, 3.5 - k
        w = v[k:k + 4]
        d1, d2, d3 = w[1] - w[0], (w[2] - 2 * w[1] + w[0]) / 2, (w[3] - 3 * w[2] + 3 * w[1] - w[0]) / 6
        A, B, C = d1 - d2 + 2 * d3, 2 * d2 - 6 * d3, 3 * d3   # first derivative A + B x + C x^2
        m = [hi - lo] + [(hi ** j - lo ** j) / j for j in range(2, 6)]
        b = A * A * m[0] + 2 * A * B * m[1] + (B * B + 2 * A * C) * m[2] + 2 * B * C * m[3] + C * C * m[4]
        E = 6 * d3
        b = b + B * B * m[0] + 2 * B * E * m[1] + E * E * m[2] + 36 * d3 * d3 * m[0]
        a = d / (1e-6 + b) ** 2
        num, den = num + a * p[k], den + a
    return num / den


_RECON = {"weno3": (2, 4, _weno3), "weno5": (3, 5, _weno5), "teno5": (3, 5, _teno5), "weno7": (4, 7, _weno7)}


def _pressure(q):
    return (GAMMA - 1) * (q[4] - 0.5 * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2) / q[0])


def _basis(q, n):
    """Rows of L and columns of R of the flux Jacobian along the unit normal n."""
    u = [q[k] / q[0] for k in (1, 2, 3)]
    p = _pressure(q)
    q2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
    c = torch.sqrt(GAMMA * p / q[0])
    H = (q[4] + p) / q[0]
    swap = n[2].abs() > n[1].abs()
    ss = torch.where(swap, torch.sqrt(n[0] ** 2 + n[2] ** 2), torch.sqrt(n[0] ** 2 + n[1] ** 2))
    zero = torch.zeros_like(ss)
    l = [torch.where(swap, -n[2], -n[1]) / ss, torch.where(swap, zero, n[0]) / ss, torch.where(swap, n[0], zero) / ss]
    m = [n[1] * l[2] - n[2] * l[1], n[2] * l[0] - n[0] * l[2], n[0] * l[1] - n[1] * l[0]]
    dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2]  # noqa: E731
    un, ul, um = dot(u, n), dot(u, l), dot(u, m)
    b1 = (GAMMA - 1) / c ** 2
    b2, x1 = b1 / 2, 1 / (2 * c)
    L = [[1 - b2 * q2, b1 * u[0], b1 * u[1], b1 * u[2], -b1],
         [-ul, l[0], l[1], l[2], zero], [-um, m[0], m[1], m[2], zero],
         [0.5 * b2 * q2 + x1 * un] + [-x1 * n[k] - b2 * u[k] for k in range(3)] + [b2],
         [0.5 * b2 * q2 - x1 * un] + [x1 * n[k] - b2 * u[k] for k in range(3)] + [b2]]
    one = zero + 1
    R = [[one, u[0], u[1], u[2], 0.5 * q2], [zero, l[0], l[1], l[2], ul], [zero, m[0], m[1], m[2], um],
         [one] + [u[k] - c * n[k] for k in range(3)] + [H - c * un],
         [one] + [u[k] + c * n[k] for k in range(3)] + [H + c * un]]
    return L, R


def _flux(q, n):
    un = (q[1] * n[0] + q[2] * n[1] + q[3] * n[2]) / q[0]
    p = _pressure(q)
    return [q[0] * un] + [q[1 + k] * un + p * n[k] for k in range(3)] + [(q[4] + p) * un], un, p


def _face_flux(st, n, scheme, roe):
    """Flux through the faces with stencil st (points x 5 fields) and unit normals n."""
    reach, width, core = _RECON[scheme]
    mid = [0.5 * (a + b) for a, b in zip(st[reach - 1], st[reach])]
    L, R = _basis(mid, n)
    qL, qR = [0.0] * 5, [0.0] * 5
    for k in range(5):
        ch = [sum(L[k][v] * s[v] for v in range(5)) for s in st]
        wl_, wr = core(ch[:width]), core(ch[::-1][:width])
        for v in range(5):
            qL[v], qR[v] = qL[v] + R[k][v] * wl_, qR[v] + R[k][v] * wr
    del L, R
    fL, unL, pL = _flux(qL, n)
    fR, unR, pR = _flux(qR, n)
    if not roe:
        lam = torch.maximum(unL.abs() + torch.sqrt(GAMMA * pL / qL[0]), unR.abs() + torch.sqrt(GAMMA * pR / qR[0]))
        return [0.5 * (a + b) - 0.5 * lam * (y - x) for a, b, x, y in zip(fL, fR, qL, qR)]
    sL, sR = torch.sqrt(qL[0]), torch.sqrt(qR[0])
    avg = lambda a, b: (sL * a + sR * b) / (sL + sR)  # noqa: E731
    u = [avg(qL[k] / qL[0], qR[k] / qR[0]) for k in (1, 2, 3)]
    h = avg((qL[4] + pL) / qL[0], (qR[4] + pR) / qR[0])
    q2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
    a2 = (GAMMA - 1) * (h - 0.5 * q2)
    rho = sL * sR
    L, R = _basis([rho, rho * u[0], rho * u[1], rho * u[2], rho * (0.5 * q2 + a2 / (GAMMA - 1))], n)
    a = torch.sqrt(a2)
    un = u[0] * n[0] + u[1] * n[1] + u[2] * n[2]
    eps = 0.1 * a
    dq = [y - x for x, y in zip(qL, qR)]
    diss = [0.0] * 5
    for k, lam in enumerate((un, un, un, un + a, un - a)):  # the reference's pairing of speeds and waves
        x = lam.abs()
        x = torch.where(x < 2 * eps, 0.5 * (x * x / (2 * eps) + eps), x)
        s = x * sum(L[k][v] * dq[v] for v in range(5))
        diss = [diss[v] + R[k][v] * s for v in range(5)]
    return [0.5 * (x + y - d) for x, y, d in zip(fL, fR, diss)]


class _Exact:
    """The explicit scheme on one grid: five fields of shape (nz, ny, nx)."""

    def __init__(self, dim, n, h, periodic, recipe, time, cfl, q, metrics=None):
        self.dim, self.n, self.h, self.per, self.cfl, self.time = dim, n, h, periodic, cfl, time
        self.scheme, self.roe = recipe[:5], recipe.endswith("Roe")
        self.q = [q[..., v].contiguous() for v in range(5)]
        self.lo = [0 if periodic or d >= dim else 1 for d in range(3)]
        self.hi = [n[d] if periodic or d >= dim else n[d] - 1 for d in range(3)]
        self.jac = 1.0 / (h[0] * h[1] * h[2])
        self.m = None if metrics is None else [metrics[..., k].contiguous() for k in range(10)]

    def _index(self, d, lo, hi):
        i = torch.arange(lo, hi, device=self.q[0].device)
        return i % self.n[d] if self.per else i.clamp(1, self.n[d] - 2)

    def _solved(self, x, skip=-1):
        for d in range(3):
            if d != skip:
                x = x.narrow(2 - d, self.lo[d], self.hi[d] - self.lo[d])
        return x

    def residual(self, q):
        total = [0.0] * 5
        for d in range(self.dim):
            ax, reach = 2 - d, _RECON[self.scheme][0]
            nf = self.hi[d] - self.lo[d] + 1
            pad = [self._solved(x, d).index_select(ax, self._index(d, self.lo[d] - reach, self.hi[d] + reach)) for x in q]
            st = [[x.narrow(ax, s, nf) for x in pad] for s in range(2 * reach)]
            if self.m is None:
                area = self.h[0] * self.h[1] * self.h[2] / self.h[d]
                nv = [torch.full((1, 1, 1), 1.0 if k == d else 0.0, dtype=torch.float64, device=q[0].device) for k in range(3)]
            else:  # periodic: face f between nodes f - 1 and f
                cof = []
                for k in range(3):
                    c = (self.m[1 + 3 * d + k] / self.m[0]).index_select(ax, self._index(d, self.lo[d] - 1, self.hi[d] + 1))
                    cof.append(0.5 * (c.narrow(ax, 0, nf) + c.narrow(ax, 1, nf)))
                area = torch.sqrt(cof[0] ** 2 + cof[1] ** 2 + cof[2] ** 2)
                nv = [c / area for c in cof]
            F = _face_flux(st, nv, self.scheme, self.roe)
            total = [t + (f * area).diff(dim=ax) for t, f in zip(total, F)]
        jac = self.jac if self.m is None else self.m[0]
        return [jac * t for t in total]

    def dt(self):
        q = [self._solved(x) for x in self.q]
        c = torch.sqrt(GAMMA * _pressure(q) / q[0])
        s = 0.0
        for d in range(self.dim):
            if self.m is None:
                s = s + ((q[1 + d] / q[0]).abs() + c) / self.h[d]
            else:
                m = self.m[1 + 3 * d:4 + 3 * d]
                s = s + ((q[1] * m[0] + q[2] * m[1] + q[3] * m[2]) / q[0]).abs() + \
                    c * torch.sqrt(m[0] ** 2 + m[1] ** 2 + m[2] ** 2)
        return self.cfl / float(s.max())

    def _with(self, solved):
        out = [x.clone() for x in self.q]
        for o, x in zip(out, solved):
            self._solved(o).copy_(x)
        return out

    def step(self):
        dt = self.dt()
        q0 = [self._solved(x) for x in self.q]
        if self.time == "forwardEuler":
            new = [a - dt * r for a, r in zip(q0, self.residual(self.q))]
        elif self.time == "SSPRK3":
            new = [a - dt * r for a, r in zip(q0, self.residual(self.q))]
            for a0, a1 in ((0.75, 0.25), (1 / 3, 2 / 3)):
                r = self.residual(self._with(new))
                new = [a0 * a + a1 * (b - dt * x) for a, b, x in zip(q0, new, r)]
        else:
            k1 = self.residual(self.q)
            k2 = self.residual(self._with([a - 0.5 * dt * r for a, r in zip(q0, k1)]))
            k3 = self.residual(self._with([a - 0.5 * dt * r for a, r in zip(q0, k2)]))
            k4 = self.residual(self._with([a - dt * r for a, r in zip(q0, k3)]))
            new = [a - dt / 6 * (w + 2 * x + 2 * y + z) for a, w, x, y, z in zip(q0, k1, k2, k3, k4)]
        self.q = self._with(new)
        return dt

    def state(self):
        out = torch.stack(self.q, -1)
        for d in range(self.dim):  # unsolved boundary nodes copy their inner neighbours
            if not self.per:
                out = out.index_select(2 - d, self._index(d, 0, self.n[d]))
        return out


def exact(case, seed):
    if case["kind"] == "batch":
        grids = _batch_grids(case, seed)
        ends = []
        for g in (grids[0], grids[3]):
            x = _Exact(g.dim, g.n, g.h, g.bc_lo[0] == capi.BC_PERIODIC, g.recipe, "SSPRK3", g.cfl,
                       torch.from_numpy(g.q).to(_device()))
            t = 0.0
            for _ in range(case["steps"]):
                t += x.step()
            ends.append(x.state())
        return {"states": None, "tube": ends[0], "vortex": ends[1], "times": None}
    q, metrics = _state(case, seed)
    n, h = _spacing(case)
    x = _Exact(case["dim"], n, h, case["bc"] == "periodic", case["recipe"], case.get("time", "SSPRK3"), _cfl(case), q,
               metrics)
    if case["kind"] == "residual":
        out = torch.zeros((5,) + tuple(q.shape[:3]), dtype=torch.float64, device=q.device)
        for v, r in enumerate(x.residual(x.q)):
            x._solved(out[v]).copy_(r)
        return out.reshape(5, -1)
    dts = [x.step() for _ in range(case["steps"])]
    return {"q": x.state(), "dt": np.array(dts)}
