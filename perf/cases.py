"""Performance cases of the library: what a solver run asks of it, through its public entry points.

A case is a plain dict; `prepare` makes the inputs (from the seed alone) and the handles that a program keeps,
`run` is one pass through the public calls, `work` the bytes and operations it cannot do without, and `exact`
the same result in plain 64-bit torch.  Kinds of pass:

  noalloc   rts_scattering_noalloc on the caller's device arrays
  update    rts_scattering_update: host Illum in, integral and source update, host S out
  calls     the solver's own sequence: one Illum copy per direction, the pair of integral calls on the two
            scattering streams with their copies back, the wait
  solve     a source iteration: set-up, relaxed steps, S and the residuals read back
  batch     several problems set up from host intensities, one captured graph of relaxed steps, results read
  serve     a burst of requests through the serving loop
  sweep     a new medium, then the device source iteration (transport sweep + scattering integral)
  moments   energy and flux, then every illumination parameter with the divergences
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import relativistic_solver_hllc_gb300 as pkg
from relativistic_solver_hllc_gb300 import _native as native


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest call: a solver that owns its device memory, a coarse mesh and direction set
        {"name": "noalloc_2000x64", "kind": "noalloc", "cells": 2000, "dirs": 64, "sigma": 1.5},
        # configuration 1: one integral and source update at the default precision
        {"name": "update_fp64_10368x200", "kind": "update", "cells": 10368, "dirs": 200, "sigma": 1.0,
         "precision": "fp64", "lam": 0.5},
        # a fine mesh with configuration 2's direction set, the default precision
        {"name": "update_fp64_162000x1000", "kind": "update", "cells": 162000, "dirs": 1000, "sigma": 1.5,
         "precision": "fp64", "lam": 0.9},
        # the unchanged solver's sequence of calls, default precision and a tensor precision
        {"name": "calls_fp64_82944x400", "kind": "calls", "cells": 82944, "dirs": 400, "sigma": 1.0,
         "precision": "fp64"},
        {"name": "calls_fp16x3_82944x400", "kind": "calls", "cells": 82944, "dirs": 400, "sigma": 1.0,
         "precision": "fp16x3"},
        # source iterations with relaxation: a ragged mesh in FP64, and configuration 2's kind of problem with the
        # Illum already on the device
        {"name": "solve_fp64_30011x302", "kind": "solve", "cells": 30011, "dirs": 302, "sigma": 1.0,
         "precision": "fp64", "lam": 0.9, "steps": 6, "resident": False},
        {"name": "solve_fp16x3_162000x1000", "kind": "solve", "cells": 162000, "dirs": 1000, "sigma": 1.5,
         "precision": "fp16x3", "lam": 0.9, "steps": 20, "resident": True},
        # multigroup anisotropic problems (configuration 3's kernel), set up and solved together
        {"name": "batch_tf32x3_3x_hg_590", "kind": "batch", "cells": 15000, "dirs": 590, "groups": 4, "problems": 3,
         "g": 0.7, "precision": "tf32x3", "steps": 10},
        # a burst of requests (configuration 5's mix, smaller meshes)
        {"name": "serve_fp16x3_12", "kind": "serve", "requests": 12, "median_cells": 15000, "mix": 5,
         "precision": "fp16x3"},
        # device source iterations from a new medium: a small mesh in FP64, a larger one at a tensor precision
        {"name": "sweep_fp64_6000x48", "kind": "sweep", "cube": 10, "dirs": 48, "precision": "fp64", "iters": 5},
        {"name": "sweep_fp16x3_82944x400", "kind": "sweep", "cube": 24, "dirs": 400, "precision": "fp16x3",
         "iters": 5},
        # the illumination parameters of a solved field
        {"name": "moments_82944x400", "kind": "moments", "cells": 82944, "dirs": 400, "sigma": 1.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: sizes log-uniform and mostly odd, bounded by the largest listed work."""
    kind = rng.choice(["noalloc", "update", "update", "calls", "calls", "solve", "solve", "batch", "serve", "sweep",
                       "moments"])
    tensor = rng.choice(["fp16x3", "tf32x3", "bf16x3"])
    any_precision = rng.choice(["fp64", "fp64", tensor])
    sigma = round(rng.uniform(0.5, 1.5), 3)
    lam = round(rng.uniform(0.2, 0.95), 3)
    if kind == "noalloc":
        return {"kind": kind, "cells": _log_int(rng, 1000, 60000), "dirs": _log_int(rng, 24, 512), "sigma": sigma}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(2, 12), "median_cells": _log_int(rng, 3000, 15000),
                "mix": rng.randint(0, 10**6), "precision": tensor}
    if kind == "sweep":
        return {"kind": kind, "cube": rng.randint(6, 24), "dirs": _log_int(rng, 24, 400), "precision": any_precision,
                "iters": rng.randint(2, 5)}
    if kind == "batch":
        return {"kind": kind, "cells": _log_int(rng, 2000, 15000), "dirs": rng.choice([110, 146, 302, 590]),
                "groups": rng.randint(1, 4), "problems": rng.randint(2, 6), "g": round(rng.uniform(0.0, 0.8), 3),
                "precision": tensor, "steps": rng.randint(4, 20)}
    dirs = _log_int(rng, 48, 1000)
    cells = min(_log_int(rng, 2000, 162000), 60_000_000 // dirs)
    case = {"kind": kind, "cells": cells, "dirs": dirs, "sigma": sigma}
    if kind in ("update", "calls", "solve"):
        case["precision"] = any_precision
    if kind in ("update", "solve"):
        case["lam"] = lam
    if kind == "solve":
        case["steps"] = rng.randint(3, 20) if any_precision != "fp64" else rng.randint(2, 5)
        case["resident"] = any_precision != "fp64"
    return case


# ----------------------------------------------------------------------------------------------- inputs
def _directions(M):
    """Spherical Fibonacci points with equal weights (host FP64)."""
    i = np.arange(M, dtype=np.float64)
    z = 1.0 - (2.0 * i + 1.0) / M
    r = np.sqrt(np.maximum(0.0, 1.0 - z * z))
    phi = math.pi * (3.0 - math.sqrt(5.0)) * i
    xyz = np.ascontiguousarray(np.stack([r * np.cos(phi), r * np.sin(phi), z], axis=1))
    return xyz, np.full(M, 4 * math.pi / M), 4 * math.pi


def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 64 + stream)


def _uniform(seed, stream, shape, lo, hi, dtype=torch.float64):
    return torch.rand(shape, generator=_generator(seed, stream), device="cuda", dtype=dtype) * (hi - lo) + lo


def _illum(case, seed):
    """Illum [M][N][4]: a lognormal intensity per cell and direction, the faces within 10 % of it."""
    shape = (case["dirs"], case["cells"])
    gen = _generator(seed, 1)
    mean = torch.exp(torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64) * case["sigma"])
    il = torch.rand(shape + (4,), generator=gen, device="cuda", dtype=torch.float64)
    return il.mul_(0.2).add_(0.9).mul_(mean[:, :, None])


def _source(case, seed):
    return _uniform(seed, 2, (case["cells"],), 0.1, 1.0)


def _geometry(case, seed):
    n = case["cells"]
    nrm = torch.randn((n, 4, 3), generator=_generator(seed, 3), device="cuda", dtype=torch.float64)
    nrm /= nrm.norm(dim=2, keepdim=True)
    return nrm, _uniform(seed, 4, (n, 4), 0.5, 1.0), _uniform(seed, 5, (n,), 0.5, 1.0)


def _problems(case):
    """(cells, directions, groups, phase, g, albedos, iterations) of each problem of a batch or request of a burst."""
    if case["kind"] == "batch":
        out = []
        for i in range(case["problems"]):
            lams = [0.3 + 0.08 * k for k in range(case["groups"])]
            phase = pkg.PHASE_THOMSON if i % 3 == 2 else pkg.PHASE_HG
            out.append((max(1, case["cells"] * 2 // (i + 2)), case["dirs"], case["groups"], phase,
                        case["g"] if phase == pkg.PHASE_HG else 0.0, lams, case["steps"]))
        return out
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["requests"]):
        cells = int(np.clip(round(case["median_cells"] * math.exp(rng.normal(0.0, 1.0))), 2000,
                            4 * case["median_cells"]))
        dirs = int(rng.choice([110, 302, 590, 1202]))
        out.append((cells, dirs, 1, pkg.PHASE_HG, float(rng.uniform(0.0, 0.8)), [float(rng.uniform(0.2, 0.95))],
                    int(rng.integers(5, 41))))
    return out


def _problem_inputs(problem, seed, i):
    """FP32 Ibar [groups][M][N] and B [groups][N] on the GPU."""
    cells, dirs, groups = problem[:3]
    gen = _generator(seed, 8 + i)
    ibar = torch.exp(torch.randn((groups, dirs, cells), generator=gen, device="cuda", dtype=torch.float32))
    B = torch.rand((groups, cells), generator=gen, device="cuda", dtype=torch.float32) * 0.9 + 0.1
    return ibar, B


# ------------------------------------------------------------------------------------- handles and views
class _Host(np.ndarray):
    """An array over memory that `owner` frees."""


def _host_view(array, owner):
    v = array.view(_Host)
    v.owner = owner
    return v


class _DeviceArray:
    def __init__(self, ptr, shape, owner):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}
        self.owner = owner


def _device_illum(ctx):
    return torch.as_tensor(_DeviceArray(ctx.device_arrays()[0], (ctx.M, ctx.N, 4), ctx), device="cuda")


def _pinned(owner_list, shape, dtype):
    count = int(np.prod(shape))
    buf = native.PinnedBuffer(max(count, 1) * np.dtype(dtype).itemsize)
    owner_list.append(buf)
    return _host_view(buf.array(dtype, count).reshape(shape), buf)


def _context(case, host_illum=None, device_illum=None):
    xyz, area, full = _directions(case["dirs"])
    ctx = pkg.Context(0)
    ctx.init(xyz, area, full, case["cells"])
    if host_illum is not None:
        torch.from_numpy(ctx.host_illum()).copy_(host_illum.reshape(-1))
    if device_illum is not None:
        _device_illum(ctx).copy_(device_illum)
    return ctx


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": dict(case), "kind": kind}
    if kind == "noalloc":
        xyz, area, full = _directions(case["dirs"])
        s["illum"] = _illum(case, seed)
        s["xyz"], s["area"] = torch.from_numpy(xyz).cuda(), torch.from_numpy(area).cuda()
        s["full"] = full
        s["out"] = torch.empty((case["dirs"], case["cells"]), dtype=torch.float64, device="cuda")
        fn = native.load_library().rts_scattering_noalloc
        fn.restype = C.c_int
        fn.argtypes = [C.c_void_p] * 3 + [C.c_int64] * 2 + [C.c_double] + [C.c_void_p] * 2
        s["fn"] = fn
    elif kind in ("update", "calls", "solve"):
        il = _illum(case, seed)
        if case.get("resident"):
            ctx = _context(case, device_illum=il)
        else:
            ctx = _context(case, host_illum=il)
        s["ctx"] = ctx
        s["host"] = ctx.host_illum()
        s["out"] = _host_view(ctx.host_scattering(), ctx)
        if kind != "calls":
            s["B"] = _source(case, seed).cpu().numpy()
        else:
            ctx.set_precision(case["precision"])
    elif kind in ("batch", "serve"):
        ctx = s["ctx"] = pkg.Context(0)
        s["keep"], s["problems"] = [], []
        for i, p in enumerate(_problems(case)):
            cells, dirs, groups, phase, g, lams, steps = p
            ibar, B = _problem_inputs(p, seed, i)
            h_ibar = _pinned(s["keep"], (groups, dirs, cells), np.float32)
            h_B = _pinned(s["keep"], (groups, cells), np.float32)
            torch.from_numpy(h_ibar.view(np.ndarray)).copy_(ibar)
            torch.from_numpy(h_B.view(np.ndarray)).copy_(B)
            out = _pinned(s["keep"], (groups, dirs, cells), np.float32)
            desc = native.problem_desc(cells, dirs, groups, phase, g, case["precision"])
            s["problems"].append((desc, h_ibar.view(np.ndarray), h_B.view(np.ndarray), np.array(lams), steps, out))
        if kind == "serve":
            fp = C.POINTER(C.c_float)
            s["requests"] = [native.Request(0.0, d, it, i.ctypes.data_as(fp), b.ctypes.data_as(fp),
                                            l.ctypes.data_as(native._dp), o.ctypes.data_as(fp))
                             for d, i, b, l, it, o in s["problems"]]
    elif kind == "sweep":
        vert, pairs, normals = pkg.mesh_cube(case["cube"], 1, True)
        n = vert.shape[0]
        ctx = s["ctx"] = _context({"dirs": case["dirs"], "cells": n})
        ctx.sweep_set_mesh(vert, pairs, normals)
        ctx.sweep_build()
        s["scattering"] = ctx.host_scattering()
        s["scattering"][:] = 0.0  # the iteration starts without scattered light
        s["medium"] = [_uniform(seed, 2 + k, (n,), lo, hi).cpu().numpy()
                       for k, (lo, hi) in enumerate(((0.5, 1.5), (0.5, 1.5), (0.1, 1.0)))]
        s["illum"] = _device_illum(ctx)
        s["illum"].zero_()
    elif kind == "moments":
        ctx = s["ctx"] = _context(case, device_illum=_illum(case, seed))
        ctx.set_geometry(*(x.cpu().numpy() for x in _geometry(case, seed)))
    return s


# ------------------------------------------------------------------------------------------------- run
def _batch_pass(s):
    ctx, steps = s["ctx"], s["case"]["steps"]
    with pkg.Batch(ctx) as b:
        ids = [b.add(desc, ibar, B, lam) for desc, ibar, B, lam, _, _ in s["problems"]]
        b.capture(steps, True)
        b.replay()
        residuals = []
        for pid, problem in zip(ids, s["problems"]):
            r = C.c_double()
            out = problem[-1]
            ctx._check(ctx.lib.rts_batch_read(b.h, pid, out.ctypes.data_as(C.POINTER(C.c_float)), C.byref(r)),
                       "rts_batch_read")
            residuals.append(r.value)
    return [p[-1] for p in s["problems"]], residuals


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "noalloc":
        rc = s["fn"](s["illum"].data_ptr(), s["xyz"].data_ptr(), s["area"].data_ptr(), case["cells"], case["dirs"],
                     s["full"], s["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if rc != native.OK:
            raise pkg.RtsError(rc, "rts_scattering_noalloc")
        return s["out"]
    ctx = s["ctx"]
    if kind == "update":
        return ctx.scattering_update(case["precision"], s["host"], s["B"], case["lam"], s["out"])
    if kind == "calls":
        N, M = case["cells"], case["dirs"]
        for j in range(M):
            ctx.send_illum_async(4 * N, 4 * N * j, 4 * N * j, s["host"])
        ctx.scattering_async(0, M // 3, pkg.STREAM_SCATTERING_1, s["out"])
        ctx.scattering_async(0, M, pkg.STREAM_SCATTERING_2, s["out"])
        ctx.wait()
        return s["out"]
    if kind == "solve":
        if not case["resident"]:
            ctx.copy_illum(s["host"])
        ctx.solve_setup(case["precision"], s["B"], case["lam"])
        for _ in range(case["steps"]):
            ctx.solve_step_async(True)
        ctx._check(ctx.lib.rts_solve_read(ctx.h, s["out"].ctypes.data_as(native._dp)), "rts_solve_read")
        return {"S": s["out"], "residuals": ctx.solve_residual_history(case["steps"])}
    if kind == "batch":
        S, residuals = _batch_pass(s)
        return {"S": S, "residuals": np.array(residuals, dtype=np.float32)}
    if kind == "serve":
        native.serve(ctx, s["requests"], 120 * 10**9)
        return [p[-1] for p in s["problems"]]
    if kind == "sweep":
        ctx.send_scattering(s["scattering"])
        ctx.sweep_set_medium(pkg.medium(), *s["medium"])
        norms = ctx.illum_solve(case["precision"], max_iter=case["iters"], accuracy=0.0)
        return {"illum": s["illum"], "norms": norms[1:]}  # the first compares with what was there before
    energy, flux = ctx.moments()
    return {"moments": [energy, flux], "params": list(ctx.illum_params())}


# ------------------------------------------------------------------------------------------------ work
def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        nbytes = flops = 0.0
        for cells, dirs, groups, _, _, _, steps in _problems(case):
            rows = cells * groups
            nbytes += rows * (8.0 * dirs + 4)
            flops += 2.0 * rows * dirs * dirs * steps
        return {"bytes": nbytes, "flops": flops}
    if kind == "sweep":
        pairs = 6.0 * case["cube"] ** 3 * case["dirs"]
        # per sweep: Illum read (for its change) and written, S read, two out-faces of three nodes per cell and
        # direction with a distance each; per integral Illum read, S written
        return {"bytes": pairs * (128 + 40) * case["iters"], "flops": 2.0 * pairs * case["dirs"] * case["iters"]}
    N, M = case["cells"], case["dirs"]
    if kind == "moments":
        return {"bytes": 2 * 32.0 * N * M + 8.0 * 38 * N, "flops": 71.0 * N * M}
    steps = case.get("steps", 1)
    return {"bytes": 40.0 * N * M + 8.0 * N, "flops": 2.0 * N * M * M * steps}


# ----------------------------------------------------------------------------------------------- exact
def _weights(M, phase=0, g=0.0):
    xyz, area, full = _directions(M)
    x = torch.from_numpy(xyz).cuda()
    mu = x @ x.T
    if phase == pkg.PHASE_THOMSON:
        return 3.0 * (1.0 + mu * mu) / 4.0 * (4 * math.pi / M) / full
    den = 1.0 + g * g - 2.0 * g * mu
    w = (1.0 - g * g) / (4.0 * math.pi * den * torch.sqrt(den)) * (4 * math.pi / M)
    return w / w.sum(dim=0, keepdim=True)


def _iterate(W, ibar, B, lam, steps):
    """Relaxed steps from ibar [M][N]: S and the residual of each step."""
    S = torch.zeros_like(ibar)
    residuals = []
    for _ in range(steps):
        new = (1.0 - lam) * B[None, :] + lam * (W.T @ ibar)
        residuals.append(float((new - S).abs().max()))
        S = new
        ibar = 0.5 * ibar + 0.5 * S
    return S, residuals


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        return None
    if kind in ("batch", "serve"):
        out, residuals = [], []
        for i, p in enumerate(_problems(case)):
            cells, dirs, groups, phase, g, lams, steps = p
            ibar, B = _problem_inputs(p, seed, i)
            W = _weights(dirs, phase, g)
            S, last = torch.empty(ibar.shape, dtype=torch.float64, device="cuda"), 0.0
            for k in range(groups):
                S[k], r = _iterate(W, ibar[k].double(), B[k].double(), lams[k], steps)
                last = max(last, r[-1])
            out.append(S)
            residuals.append(last)
        return out if kind == "serve" else {"S": out, "residuals": np.array(residuals)}
    il = _illum(case, seed)
    if kind == "moments":
        xyz, area, full = (torch.from_numpy(v).cuda() if isinstance(v, np.ndarray) else v
                           for v in _directions(case["dirs"]))
        nrm, face, vol = _geometry(case, seed)
        a = area[:, None]
        T = torch.cat([a, a * xyz, (a[:, :, None] * xyz[:, :, None] * xyz[:, None, :]).reshape(-1, 9)], dim=1)
        G = torch.einsum("jk,jcf->cfk", T, il)  # per face: sums with 1, w and w w^T
        mean = G.sum(dim=1) / (4.0 * full)
        nS = nrm * face[:, :, None]
        divs = torch.einsum("cfd,cfd->c", nS, G[:, :, 1:4]) / (full * vol)
        divi = torch.einsum("cfd,cfde->ce", nS, G[:, :, 4:].reshape(-1, 4, 3, 3)) / (full * vol[:, None])
        e, f = mean[:, 0], mean[:, 1:4]
        return {"moments": [e, f], "params": [e, f, mean[:, 4:].reshape(-1, 3, 3), divs, divi]}
    W = _weights(case["dirs"])
    ibar = il.sum(dim=2) / 4.0
    del il
    if kind == "noalloc":
        return W.T @ ibar
    if kind == "calls":
        return (W.T @ ibar).reshape(-1)
    B = _source(case, seed)
    if kind == "update":
        return ((1.0 - case["lam"]) * B[None, :] + case["lam"] * (W.T @ ibar)).reshape(-1)
    S, residuals = _iterate(W, ibar, B, case["lam"], case["steps"])
    return {"S": S.reshape(-1), "residuals": np.array(residuals)}
