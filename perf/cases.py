"""The work users of this framework have it do, as measurable cases.

Every case goes through the public entry points: PoissonContext / SolveBatch
(curvib_old_gb300.solver) where the arrays stay on the device, and the C ABI
(include/cvb.h, through curvib_old_gb300._lib) where a CURVIB program hands
over host arrays, which are pinned here as in bench.py.  Kinds:

``solve``   one pressure solve of a right-hand side that is resident on the
            device, into the resident pressure: PoissonSolver_MG's KSPSolve as a
            time loop repeats it.  On the distorted box with a sphere (19-point
            operator) or on the periodic channel (7-point operator); FP32
            V-cycles inside FP64 FGMRES ("mixed") or FP64 throughout.
``warm``    a follow-up solve on a problem the caller keeps: host right-hand
            side in, pressure in as the initial guess and out.
``batch``   many uneven problems in one batch (several blocks, a parameter
            study, a served queue).
``step``    the projection part of a time step on host arrays:
            PoissonSolver_MG, UpdatePressure, Projection.
``body``    the step of a moving body: the cells classified against its mesh,
            the operators rebuilt, then PoissonSolver_MG.
``rhs``     the momentum right-hand side CalcRHS on host arrays (other momentum
            solvers of CURVIB call it directly).
``imprk``   ImpRK, the momentum equation's pseudo-time iteration, on a box with
            an inlet and an outlet.

Grids are the repository's own (workload.py): a [0,1]^3 box with tanh
stretching 2.0 in y and sine distortion, and the 2 pi x 2 x pi channel with
tanh stretching 2.5.  A case's seed gives the body, the fluxes and the noise on
them; a grid's metrics are uploaded once per process and shared, as a run keeps
its grid.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from curvib_old_gb300 import _lib
from curvib_old_gb300 import workload as W
from curvib_old_gb300.solver import PoissonContext, SolveBatch

DT, ST, REN = 1e-3, 1.0, 300.0  # time step, pseudo-time factor, Reynolds number
CHANNEL = (2 * np.pi, 2.0, np.pi)  # its lengths in x, y, z
BATCH_SIZES = W.CONFIG3_SIZES  # the five sizes of the batched workload
PRECISION = {"mixed": _lib.MIXED, "fp64": _lib.FP64}


def listed():
    return [
        # the smallest problem of the batched and served workloads, alone: a
        # few hundred launches of a few microseconds
        {"name": "solve-32", "kind": "solve", "grid": "box", "nx": 32, "ny": 32, "nz": 32, "levels": 0,
         "precision": "mixed", "rtol": 1e-8},
        # the 64^3 box with its stated 3 levels, in plain FP64 as the reference
        # runs it
        {"name": "solve-64-fp64", "kind": "solve", "grid": "box", "nx": 64, "ny": 64, "nz": 64, "levels": 3,
         "precision": "fp64", "rtol": 1e-8},
        # uneven sides that coarsen to odd ones
        {"name": "solve-88x56x72", "kind": "solve", "grid": "box", "nx": 88, "ny": 56, "nz": 72, "levels": 0,
         "precision": "mixed", "rtol": 1e-8},
        # a served follow-up request at an ordinary size: host arrays in and out
        {"name": "warm-128", "kind": "warm", "grid": "box", "nx": 128, "ny": 128, "nz": 128, "levels": 0,
         "precision": "mixed", "rtol": 1e-8},
        # the channel of the headline benchmark in both precisions
        {"name": "channel", "kind": "solve", "grid": "channel", "nx": 256, "ny": 128, "nz": 128, "levels": 5,
         "precision": "mixed", "rtol": 1e-10},
        {"name": "channel-fp64", "kind": "solve", "grid": "channel", "nx": 256, "ny": 128, "nz": 128, "levels": 5,
         "precision": "fp64", "rtol": 1e-10},
        # half of the batched workload's 64 problems
        {"name": "batch-32", "kind": "batch", "count": 32, "precision": "mixed", "rtol": 1e-8},
        # a moving body at the batched workload's largest cube
        {"name": "body-96", "kind": "body", "nx": 96, "ny": 96, "nz": 96, "rtol": 1e-8, "triangles": 5120},
        # the inlet/outlet momentum step: small, and at an ordinary size
        {"name": "imprk-32", "kind": "imprk", "nx": 32, "ny": 32, "nz": 32, "central": 0},
        {"name": "imprk-96", "kind": "imprk", "nx": 96, "ny": 96, "nz": 96, "central": 0},
        # the full time step's size, 192^3: its momentum right-hand side and its
        # projection part
        {"name": "rhs-192", "kind": "rhs", "nx": 192, "ny": 192, "nz": 192, "central": 0},
        {"name": "step-192", "kind": "step", "nx": 192, "ny": 192, "nz": 192, "rtol": 1e-8},
    ]


def _side(rng, lo, hi, unit):
    """A multiple of ``unit`` in [lo, hi], spread over the logarithm."""
    return unit * max(1, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / unit))


def draw(rng):
    """One more case: pressure problems of 32^3 to 192^3 cells with sides of
    multiples of 8 (three halvings at least, odd coarse sides among them),
    momentum boxes with any sides."""
    kind = rng.choices(["solve", "warm", "batch", "body", "imprk", "rhs", "step"], [8, 2, 1, 2, 2, 2, 2])[0]
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(2, 32), "precision": rng.choice(["mixed", "fp64"]),
                "rtol": 10.0 ** -rng.uniform(7.0, 8.0)}
    if kind in ("imprk", "rhs"):
        lo, hi = (24, 80) if kind == "imprk" else (32, 176)
        nx, ny, nz = (_side(rng, lo, hi, 1) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "central": int(rng.random() < 0.3)}
    lo, hi = {"solve": (32, 160), "warm": (48, 128), "body": (32, 96), "step": (48, 160)}[kind]
    nx, ny, nz = (_side(rng, lo, hi, 8) for _ in range(3))
    case = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "rtol": 10.0 ** -rng.uniform(7.5, 8.5)}
    if kind in ("solve", "warm"):
        case |= {"grid": rng.choice(["box", "channel"]) if kind == "solve" else "box", "levels": 0,
                 "precision": rng.choice(["mixed", "fp64"])}
    if kind == "body":
        case["triangles"] = rng.choice([1280, 5120, 20480])
    return case


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=8)
def _grid(grid, cells, levels, faces):
    """A grid's donor context (its metrics resident once) and the arrays the
    inputs are made from: cell centres, face areas and the base fluxes on the
    GPU, boundary types from ``faces``."""
    channel = grid == "channel"
    P = W.make_problem(cells, CHANNEL if channel else (1.0, 1.0, 1.0), 2.5 if channel else 2.0, not channel,
                       (True, False, True) if channel else (False,) * 3, nlevels=levels or None)
    if faces == "inout":
        P.bctype = [1, 1, 1, 1, 5, 4]
    m = P.metrics[-1]
    areas = torch.stack([torch.from_numpy(m[a]).cuda().square().sum(-1).sqrt() for a in ("Csi", "Eta", "Zet")], -1)
    base = None if channel else torch.from_numpy(P.ucont).cuda()
    cent = np.ascontiguousarray(m["Cent"])
    return {"donor": PoissonContext().setup_geometry(P), "cent": torch.from_numpy(cent).cuda(), "cent_host": cent,
            "areas": areas, "base": base, "shape": P.nvert.shape}


def _grid_of(case, faces="walls"):
    return _grid(case.get("grid", "box"), (case["nx"], case["ny"], case["nz"]), case.get("levels", 0), faces)


def _sphere(rng, lo=0.1, hi=0.2):
    """A seeded body: centre in [0.3, 0.7]^3 and radius in [lo, hi]."""
    return [float(v) for v in rng.uniform(0.3, 0.7, 3)], float(rng.uniform(lo, hi))


def _nvert(cent, centre, radius):
    """Codes of the cells for a sphere: solid inside it, one immersed-boundary
    layer around it, fluid elsewhere and on the ring."""
    c = torch.tensor(centre, dtype=torch.float64, device=cent.device)
    solid = (cent - c).square().sum(-1) < radius * radius
    inner = torch.zeros_like(solid)
    inner[1:-1, 1:-1, 1:-1] = True
    solid &= inner
    near = torch.nn.functional.max_pool3d(solid[None, None].float(), 3, 1, 1)[0, 0] > 0
    nv = torch.zeros(solid.shape, dtype=torch.float64, device=cent.device)
    nv[near & inner] = W.IB_CODE
    nv[solid] = W.SOLID_CODE
    return nv


def _noise(shape, seed):
    """Seeded uniform values in [-1, 1), the same on every machine."""
    g = torch.Generator().manual_seed(seed)
    return (2 * torch.rand(shape, generator=g, dtype=torch.float64) - 1).cuda()


def _walled_ucont(G, seed, amp=1e-2):
    """The box's fluxes: the Taylor-Green field and uniform noise on the inner faces."""
    n = _noise(G["base"].shape, seed) * amp * G["areas"]
    uc = G["base"].clone()
    mz, my, mx = G["shape"]
    for c, (ex, ey, ez) in enumerate(((1, 0, 0), (0, 1, 0), (0, 0, 1))):
        sl = (slice(1, mz - 1 - ez), slice(1, my - 1 - ey), slice(1, mx - 1 - ex))
        uc[sl + (c,)] += n[sl + (c,)]
    return uc


def _channel_y(ny):
    """The channel's y nodes and the widths the metrics use: of the cells, of
    the x and z faces, of the inner y faces."""
    eta = np.arange(ny + 1) / ny
    y = 2.0 * (0.5 * (1.0 + np.tanh(2.5 * (2.0 * eta - 1.0)) / math.tanh(2.5)))
    yc = 0.5 * (y[1:] + y[:-1])
    face = np.empty(ny)
    face[1:-1] = 0.5 * (yc[2:] - yc[:-2])
    face[0], face[-1] = yc[1] - yc[0], yc[-1] - yc[-2]
    return y[1:] - y[:-1], face, 0.5 * (y[2:] - y[:-2])


def _channel_ucont(cells, seed):
    """The channel's fluxes: a seeded Gaussian cell velocity (sigma 0.1), three
    damped Jacobi passes, averaged to the faces; periodic in x and z, no flux
    through the walls.  [nz+2][ny+2][nx+2][3]."""
    nx, ny, nz = cells
    g = torch.Generator().manual_seed(seed)
    v = (0.1 * torch.randn((nz, ny, nx, 3), generator=g, dtype=torch.float64)).cuda()

    def ring(v):
        v = torch.cat([v[-1:], v, v[:1]], 0)
        v = torch.cat([v[:, :1], v, v[:, -1:]], 1)
        return torch.cat([v[:, :, -1:], v, v[:, :, :1]], 2)

    for _ in range(3):
        p = ring(v)
        nb = (p[2:, 1:-1, 1:-1] + p[:-2, 1:-1, 1:-1] + p[1:-1, 2:, 1:-1] + p[1:-1, :-2, 1:-1] + p[1:-1, 1:-1, 2:]
              + p[1:-1, 1:-1, :-2]) / 6.0
        v = v + (2.0 / 3.0) * (nb - v)
    p = ring(v)
    dx, dz = CHANNEL[0] / nx, CHANNEL[2] / nz
    dy = torch.from_numpy(_channel_y(ny)[0]).cuda()
    uc = torch.zeros_like(p)
    uc[1:-1, 1:-1, :-1, 0] = 0.5 * (p[1:-1, 1:-1, :-1, 0] + p[1:-1, 1:-1, 1:, 0]) * (dy * dz)[None, :, None]
    uc[1:-1, 1:-2, 1:-1, 1] = 0.5 * (p[1:-1, 1:-2, 1:-1, 1] + p[1:-1, 2:-1, 1:-1, 1]) * (dx * dz)
    uc[:-1, 1:-1, 1:-1, 2] = 0.5 * (p[:-1, 1:-1, 1:-1, 2] + p[1:, 1:-1, 1:-1, 2]) * (dx * dy)[None, :, None]
    return uc


def _host(t):
    """The same values in pinned host memory."""
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out


def _zeros(shape):
    return torch.zeros(shape, dtype=torch.float64).pin_memory()


class _Phi:
    """A context's resident pressure as torch sees it; holds the context, which
    owns the memory."""

    def __init__(self, ctx):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"data": (ctx.device_phi(), False), "shape": tuple(ctx.shapes[-1]),
                                         "typestr": "<f8", "version": 3}


def _phi(ctx):
    return torch.as_tensor(_Phi(ctx), device="cuda")


def _problem(case, seed, faces="walls"):
    """(context, fluxes) of one block with the seed's body, on the case's grid."""
    G = _grid_of(case, faces)
    ctx = PoissonContext()
    if case.get("grid") == "channel":
        ctx.setup_like(G["donor"], np.zeros(G["shape"]))
        return ctx, _channel_ucont((case["nx"], case["ny"], case["nz"]), seed)
    big = case["kind"] in ("step", "rhs")
    nv = _nvert(G["cent"], *_sphere(np.random.default_rng(seed), *((0.2, 0.25) if big else (0.1, 0.2))))
    ctx.setup_like(G["donor"], nv.cpu().numpy())
    return ctx, _walled_ucont(G, seed)


def _resident(case, seed):
    """A context whose resident right-hand side is PoissonRHS of the seed's fluxes."""
    ctx, uc = _problem(case, seed)
    uc, _, _ = ctx.volume_flux_rev(uc.cpu().numpy())
    return ctx, ctx.poisson_rhs(uc, DT, ST)[0]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return {"case": case, "ctx": _resident(case, seed)[0]}
    if kind == "warm":
        # the caller's last pressure, and a right-hand side 1 % away from its own
        ctx, b = _resident(case, seed)
        phi, _ = ctx.solve(b, precision=_lib.MIXED, rtol=1e-8)
        b = torch.from_numpy(b).cuda()
        b += 0.01 * b.abs().mean() * _noise(b.shape, seed + 1) * (b != 0)
        opts = _lib.default_opts(precision=PRECISION[case["precision"]], rtol=case["rtol"], warm_start=1)
        return {"case": case, "ctx": ctx, "b": _host(b), "guess": _host(torch.from_numpy(phi)),
                "phi": _zeros(phi.shape), "opts": opts}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        ctxs = []
        for q in range(case["count"]):
            # the sizes in turn: the seed moves the bodies and the fluxes
            nx, ny, nz = BATCH_SIZES[q % len(BATCH_SIZES)]
            one = {"kind": "solve", "grid": "box", "nx": nx, "ny": ny, "nz": nz}
            ctxs.append(_resident(one, int(rng.integers(1 << 30)))[0])
        return {"case": case, "ctxs": ctxs,
                "batch": SolveBatch(precision=PRECISION[case["precision"]], rtol=case["rtol"])}
    if kind in ("step", "body"):
        ctx, uc = _problem(case, seed)
        vec = tuple(uc.shape)
        s = {"case": case, "ctx": ctx, "u_star": _host(uc), "ucont": _zeros(vec), "phi": _zeros(vec[:3]),
             "opts": _lib.default_opts(precision=_lib.MIXED, rtol=case["rtol"])}
        if kind == "step":
            s |= {"p0": _host(_noise(vec[:3], seed + 1)), "p": _zeros(vec[:3]), "ubcs": _zeros(vec), "ucat": _zeros(vec)}
        else:
            # the body's previous place, and its mesh one hundredth of a radius on
            G = _grid_of(case)
            centre, r = _sphere(np.random.default_rng(seed))
            mesh = W.sphere_mesh(centre, r, {1280: 3, 5120: 4, 20480: 5}[case["triangles"]])
            old = ctx.ibm_search(G["cent_host"], *mesh, 0, 1, np.zeros(vec[:3]), np.zeros(vec[:3]))
            s |= {"xyz": mesh[0] + [0.01 * r, 0.0, 0.0], "tri": mesh[1], "nf": mesh[2], "nvert": old}
        return s
    if kind == "rhs":
        ctx, uc = _problem(case, seed)
        vec = tuple(uc.shape)
        return {"case": case, "ctx": ctx, "ucont": _host(uc), "ucont_o": _host(0.999 * uc),
                "ucont_rm1": _host(0.998 * uc), "ucat": _zeros(vec), "p": _host(_noise(vec[:3], seed + 1)),
                "rhs": _zeros(vec)}
    # imprk: a uniform stream from the inlet, slightly disturbed, around the body
    ctx, _ = _problem(case, seed, "inout")
    G = _grid_of(case, "inout")
    nv = torch.from_numpy(ctx.get_nvert(ctx.nlevels - 1)[0]).cuda()
    u0 = torch.zeros(G["base"].shape, dtype=torch.float64, device="cuda")
    fluid = (nv[:-1] < 0.1) & (nv[1:] < 0.1)
    stream = 2.0 * G["areas"][:-1, :, :, 2] * (1.0 + 1e-3 * _noise(fluid.shape, seed))
    u0[:-1, 1:-1, 1:-1, 2] = torch.where(fluid, stream, 0.0)[:, 1:-1, 1:-1]
    vec = tuple(u0.shape)
    opts = _lib.imp_rk_opts(ren=REN, dt=2e-3, st=1.0, cfl=0.1, ti=1, tistart=0, central=case["central"])
    return {"case": case, "ctx": ctx, "u0": _host(u0), "ucont": _zeros(vec), "ucat": _zeros(vec), "p": _zeros(vec[:3]),
            "ubcs": _zeros(vec), "opts": opts}


# --------------------------------------------------------------------- run
def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _ok(ctx, rc):
    if rc:
        raise _lib.CvbError(rc, _lib.lib().cvb_last_error(ctx._ctx).decode())


def _solver_mg(s):
    """PoissonSolver_MG on this step's u*, host arrays."""
    s["ucont"].copy_(s["u_star"])
    st = _lib.SolveStats()
    _ok(s["ctx"], _lib.lib().cvb_poisson_solver_mg(s["ctx"]._ctx, _p(s["ucont"]), 0.0, 1, DT, ST, _p(s["phi"]),
                                                   ctypes.byref(s["opts"]), ctypes.byref(st)))


def run(state):
    s, case = state, state["case"]
    kind, L = case["kind"], _lib.lib()
    if kind == "solve":
        s["ctx"].solve_resident(precision=PRECISION[case["precision"]], rtol=case["rtol"])
        return {"phi": _phi(s["ctx"])}
    if kind == "warm":
        s["phi"].copy_(s["guess"])
        st = _lib.SolveStats()
        _ok(s["ctx"], L.cvb_poisson_solve(s["ctx"]._ctx, _p(s["b"]), _p(s["phi"]), ctypes.byref(s["opts"]),
                                          ctypes.byref(st)))
        return {"phi": s["phi"]}
    if kind == "batch":
        s["batch"].solve(s["ctxs"])
        return {"phi": [_phi(c) for c in s["ctxs"]]}
    if kind == "step":
        _solver_mg(s)
        s["p"].copy_(s["p0"])
        _ok(s["ctx"], L.cvb_update_pressure(s["ctx"]._ctx, _p(s["p"]), _p(s["phi"])))
        _ok(s["ctx"], L.cvb_projection_cart(s["ctx"]._ctx, _p(s["phi"]), DT, ST, _p(s["ucont"]), _p(s["ubcs"]),
                                            _p(s["ucat"])))
        return {k: s[k] for k in ("phi", "p", "ucont", "ubcs", "ucat")}
    if kind == "body":
        nvert = s["ctx"].ibm_search(None, s["xyz"], s["tri"], s["nf"], 0, 1, s["nvert"], s["nvert"])
        s["ctx"].set_nvert(nvert)
        _solver_mg(s)
        return {"nvert": nvert, "phi": s["phi"], "ucont": s["ucont"]}
    if kind == "rhs":
        _ok(s["ctx"], L.cvb_calc_rhs(s["ctx"]._ctx, _p(s["ucont"]), _p(s["ucont_o"]), _p(s["ucont_rm1"]),
                                     _p(s["ucat"]), _p(s["p"]), REN, 2e-3, 5, 0, case["central"], _p(s["rhs"])))
        return {"rhs": s["rhs"], "ucat": s["ucat"]}
    s["ucont"].copy_(s["u0"])
    for k in ("ucat", "p", "ubcs"):
        s[k].zero_()
    st = _lib.ImpRKStats()
    _ok(s["ctx"], L.cvb_imp_rk(s["ctx"]._ctx, _p(s["ucont"]), _p(s["u0"]), _p(s["u0"]), _p(s["ucat"]), _p(s["p"]),
                               _p(s["ubcs"]), ctypes.byref(s["opts"]), ctypes.byref(st)))
    return {"ucont": s["ucont"], "ucat": s["ucat"], "p": s["p"], "ubcs": s["ubcs"],
            "iterations": st.pseudo_iterations, "undone": st.rejected}


def work(case):
    """Bytes of the inputs and the outputs once, and the operations of one pass
    over them: a solve's operator (its face coefficients, 1/aj and the cell
    codes) with the right-hand side and the pressure, one operator apply; the
    momentum's fields with the nine face metrics, their products and Jacobians,
    one evaluation of the right-hand side."""
    if case["kind"] == "batch":
        cells = sum(math.prod(BATCH_SIZES[q % len(BATCH_SIZES)]) for q in range(case["count"]))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    orthogonal = case.get("grid") == "channel"
    solve = (44 if orthogonal else 92) + 16, 14 if orthogonal else 38
    fields = {"solve": (0, 0), "batch": (0, 0), "warm": (8, 0),
              # Ucont in and out; P in and out, Ucat and Ubcs in and out, the metrics
              "step": (48 + 16 + 96 + 72, 60), "body": (48 + 16 + 24, 0),
              # Ucont, its two previous values, Ucat in and out, P, Rhs in and out, metrics
              "rhs": (24 * 3 + 48 + 8 + 48 + 328, 700), "imprk": (48 + 48 + 48 + 48 + 16 + 328, 700)}[case["kind"]]
    if case["kind"] in ("rhs", "imprk"):
        solve = 0, 0
    return {"bytes": cells * (solve[0] + fields[0]), "flops": cells * (solve[1] + fields[1])}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """The channel's pressure to 64 bits: its operator is a sum of differences
    in x, y and z whose coefficients depend on y alone, so Fourier transforms
    in the periodic directions leave one tridiagonal system in y per wave
    number.  The boxes' operators (distorted grid, a body) have no such direct
    form and a sparse factorisation takes minutes: none there.  The momentum
    equation's results are those of its written order of roundings."""
    if case.get("grid") != "channel":
        return None
    nx, ny, nz = cells = case["nx"], case["ny"], case["nz"]
    uc = _channel_ucont(cells, seed).cpu().numpy()
    c = uc[1:-1, 1:-1, 1:-1]
    div = (c[..., 0] - uc[1:-1, 1:-1, :-2, 0] + c[..., 1] - uc[1:-1, :-2, 1:-1, 1] + c[..., 2] - uc[:-2, 1:-1, 1:-1, 2])
    dx, dz = CHANNEL[0] / nx, CHANNEL[2] / nz
    dy, face, node = _channel_y(ny)
    # A phi = b with A = -aj (sum of face fluxes) and b = -1.5 aj div / (dt st):
    # the sum of the fluxes is 1.5 div / (dt st), its mean removed
    q = 1.5 / (DT * ST) * div
    q = np.fft.fft(np.fft.rfft(q - q.mean(), axis=2), axis=0)
    lam = ((2 * np.cos(2 * np.pi * np.arange(nz) / nz) - 2) * dx / dz)[:, None] \
        + ((2 * np.cos(2 * np.pi * np.arange(nx // 2 + 1) / nx) - 2) * dz / dx)[None, :]
    up = np.append(dx * dz / node, 0.0)
    low = np.insert(dx * dz / node, 0, 0.0)
    diag = face[:, None, None] * lam[None] - (up + low)[:, None, None]
    diag[0, 0, 0] *= 2  # wave number 0 is known up to a constant: fix it in the first row
    d = np.moveaxis(q, 1, 0).copy()
    cp = np.empty(diag.shape)
    cp[0] = up[0] / diag[0]
    d[0] /= diag[0]
    for j in range(1, ny):
        m = diag[j] - low[j] * cp[j - 1]
        cp[j] = up[j] / m
        d[j] = (d[j] - low[j] * d[j - 1]) / m
    for j in range(ny - 2, -1, -1):
        d[j] -= cp[j] * d[j + 1]
    x = np.fft.irfft(np.fft.ifft(np.moveaxis(d, 0, 1), axis=0), nx, axis=2)
    phi = np.zeros(uc.shape[:3])
    phi[1:-1, 1:-1, 1:-1] = x - x.mean()
    return {"phi": phi}
