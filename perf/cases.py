"""Performance cases: the work that programs of this framework have it do,
through its public entry points, from the smallest calls to the largest.

A case is a dict of plain values; ``prepare`` makes what a program holds
before the call (inputs from a seed, handles, host buffers), ``run`` is one
pass of the program, ``exact`` gives the same outputs in 64 bits from plain
torch. ``listed`` names the fixed cases, ``draw`` gives more of the same
ranges.

Kinds of cases:
  solve    one Jacobi2d problem: grid in from the host, run, grid out
  stream   several grids through charming_jacobi2d_solve_stream
  batch    many uneven Jacobi2d problems in one scheduler launch
  serve    requests through the solve server, results fetched
  noalloc  charming_jacobi2d_sweeps_noalloc on the caller's device grids
  jacobi3d charming_jacobi3d on the caller's host grid, stepped in place
  fanout   seeded message fan-out, FIFO or with refnums
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

from charming_b200 import _lib
from charming_b200.batch import uneven_set
from charming_b200.jacobi import Jacobi2D, Problem
from charming_b200.runtime import Runtime
from charming_b200.serve import Server

MIB16 = 16 << 20


def listed() -> list[dict]:
    return [
        # The reference's example size, 512^2 in 4 x 4 chares, 100 sweeps: a
        # grid that stays in L2, where messages and launches are the time.
        dict(name="solve_512_f64", kind="solve", dtype="f64", nx=512, ny=512, px=4, py=4, side=0, sweeps=100,
             check=0, depth=0, pipeline=False, halo_mode=0),
        # The headline problem and decomposition (8192^2, 4 x 37 chares),
        # grid in and out, over the sweeps of a longer solve.
        dict(name="solve_8192_f64", kind="solve", dtype="f64", nx=8192, ny=8192, px=4, py=37, side=0, sweeps=1000,
             check=0, depth=0, pipeline=False, halo_mode=0),
        # A mid-size FP32 solve that watches its FP64 residual every 10 sweeps.
        dict(name="solve_4096_f32_residual", kind="solve", dtype="f32", nx=4096, ny=4096, px=4, py=37, side=0,
             sweeps=500, check=10, depth=0, pipeline=False, halo_mode=0),
        # An odd-sized solve on the default decomposition, one halo exchange
        # per sweep as in the reference's example.
        dict(name="solve_1999x1501_depth1", kind="solve", dtype="f64", nx=1999, ny=1501, px=0, py=0, side=256,
             sweeps=100, check=0, depth=1, pipeline=False, halo_mode=0),
        # A stream of host grids through one handle, copies beside the solves.
        dict(name="stream_2048_f64", kind="stream", dtype="f64", nx=2048, ny=2048, px=0, py=0, side=256, sweeps=300,
             n=6, depth=0),
        # The batched set: 64 uneven problems, 500 sweeps, one graph launch
        # on the default runtime.
        dict(name="batch64_f64", kind="batch", dtype="f64", set_seed=0xC3, n=64, lo=64, hi=2048, sweeps=500, check=0,
             side=256, pes_per_sm=1, graph=True),
        # The same set in FP32 with the FP64 residual, on the small PEs (4
        # per SM) that the autotuner of the batched set considers.
        dict(name="batch64_f32_residual", kind="batch", dtype="f32", set_seed=0xC3, n=64, lo=64, hi=2048, sweeps=300,
             check=10, side=256, pes_per_sm=4, graph=True),
        # The solve server: a burst of requests of mixed sizes, each result
        # fetched, start and stop included.
        dict(name="serve_16_f32", kind="serve", dtype="f32", set_seed=0xC5, n=16, lo=128, hi=2048, sweeps=500,
             check=10, side=512),
        # The smallest call: a grid of a few hundred points a side on the
        # caller's own device buffers.
        dict(name="noalloc_254_f64", kind="noalloc", dtype="f64", nx=254, ny=254, sweeps=20),
        # The largest grid of that entry point in FP32 (16 MiB).
        dict(name="noalloc_2046_f32", kind="noalloc", dtype="f32", nx=2046, ny=2046, sweeps=100),
        # 3-D sweeps of a grid a little larger than L2.
        dict(name="jacobi3d_256", kind="jacobi3d", nx=256, ny=256, nz=256, sweeps=300),
        # Messaging: 4096 chares send 16 messages of 64 bytes with refnums.
        dict(name="fanout_4096x16x64_refnum", kind="fanout", n=4096, msgs=16, payload=64, mode=1),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["solve", "solve", "solve", "stream", "batch", "batch", "serve", "noalloc", "noalloc",
                       "jacobi3d", "fanout", "fanout"])
    dtype = rng.choice(["f64", "f32"])
    if kind == "solve":
        nx, ny = _log_int(rng, 64, 3500), _log_int(rng, 64, 3500)
        return dict(kind=kind, dtype=dtype, nx=nx, ny=ny, px=0, py=0, side=rng.choice([100, 128, 256, 500, 1024]),
                    sweeps=_log_int(rng, 20, 400), check=rng.choice([0, 0, 10, 7]),
                    depth=rng.choice([0, 0, 0, 0, 1, 3, 8]), pipeline=rng.random() < 0.1,
                    halo_mode=1 if rng.random() < 0.1 else 0)
    if kind == "stream":
        nx, ny = _log_int(rng, 128, 3000), _log_int(rng, 128, 3000)
        return dict(kind=kind, dtype=dtype, nx=nx, ny=ny, px=0, py=0, side=rng.choice([128, 256, 400]),
                    sweeps=_log_int(rng, 20, 300), n=rng.randint(2, 6), depth=0)
    if kind == "batch":
        hi = rng.choice([300, 800, 2048])
        return dict(kind=kind, dtype=dtype, set_seed=rng.randrange(1 << 20), n=rng.randint(4, 64), lo=64, hi=hi,
                    sweeps=_log_int(rng, 30, 500 if hi < 2048 else 300), check=rng.choice([0, 10, 16]),
                    side=rng.choice([64, 128, 256, 512] if hi < 2048 else [128, 256, 512]), pes_per_sm=rng.choice([1, 1, 2, 4]),
                    graph=rng.random() < 0.7)
    if kind == "serve":
        return dict(kind=kind, dtype=dtype, set_seed=rng.randrange(1 << 20), n=rng.randint(3, 16), lo=128,
                    hi=rng.choice([500, 1500, 2048]), sweeps=_log_int(rng, 50, 500), check=rng.choice([0, 10, 25]),
                    side=rng.choice([256, 512, 1024]))
    if kind == "noalloc":
        esz = 8 if dtype == "f64" else 4
        nx = _log_int(rng, 16, 4000)
        ny = _log_int(rng, 16, min(4000, MIB16 // esz // (nx + 2) - 2))
        return dict(kind=kind, dtype=dtype, nx=nx, ny=ny, sweeps=_log_int(rng, 1, 200))
    if kind == "jacobi3d":
        return dict(kind=kind, nx=_log_int(rng, 16, 300), ny=_log_int(rng, 16, 300), nz=_log_int(rng, 16, 250),
                    sweeps=_log_int(rng, 10, 300))
    return dict(kind="fanout", n=_log_int(rng, 100, 6000), msgs=_log_int(rng, 4, 32),
                payload=8 * _log_int(rng, 2, 128), mode=rng.choice([0, 1]))


# ---- inputs -----------------------------------------------------------------
def _np_type(case: dict):
    return np.float64 if case["dtype"] == "f64" else np.float32


def _torch_type(case: dict):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _uniform(shape, dtype, seed: int, k: int = 0) -> torch.Tensor:
    """Seeded values in [0, 1) on the GPU (grids with their boundary ring)."""
    gen = torch.Generator(device="cuda").manual_seed((seed * 1000003 + k) & 0x7FFFFFFF)
    return torch.rand(shape, dtype=dtype, device="cuda", generator=gen)


def _pinned(shape, dtype) -> torch.Tensor:
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _runtime(pes_per_sm: int = 1) -> Runtime:
    """The process's runtime with this many PEs per SM."""
    threads = 512 // pes_per_sm
    rt = Runtime._active
    if rt is None or rt.config.pes_per_sm != pes_per_sm or rt.config.threads_per_pe != threads:
        rt = Runtime(pes_per_sm=pes_per_sm, threads_per_pe=threads)
    return rt


def _problems(case: dict, seed: int) -> list[Problem]:
    """The case's uneven sizes, with boundary values of the seed."""
    probs = uneven_set(case["set_seed"], case["n"], case["lo"], case["hi"], case["sweeps"], case["check"],
                       1e-5 if case["check"] else 0.0)
    rng = random.Random(seed)
    for p in probs:
        p.bc = tuple(rng.random() for _ in range(4))
    return probs


def _views(flat, probs: list[Problem]) -> list:
    """One grid per problem inside a flat array."""
    out, at = [], 0
    for p in probs:
        n = (p.nx + 2) * (p.ny + 2)
        out.append(flat[at:at + n].reshape(p.ny + 2, p.nx + 2))
        at += n
    return out


def _cells(probs: list[Problem]) -> int:
    return sum((p.nx + 2) * (p.ny + 2) for p in probs)


def _one_problem(case: dict) -> Problem:
    check = case.get("check", 0)
    return Problem(case["nx"], case["ny"], case["sweeps"], px=case["px"], py=case["py"], check_every=check,
                   tol=1e-5 if check else 0.0)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    s = {"case": case, "seed": seed}
    if kind in ("solve", "stream"):
        _runtime()
        dt, shape = _torch_type(case), (case["ny"] + 2, case["nx"] + 2)
        n = case.get("n", 1)
        s["in"], s["out"] = [], []
        for k in range(n):
            h = _pinned(shape, dt)
            h.copy_(_uniform(shape, dt, seed, k))
            s["in"].append(h.numpy())
            s["out"].append(_pinned(shape, dt).numpy())
        s["jac"] = Jacobi2D([_one_problem(case)], dtype=case["dtype"], chare_side=case["side"], depth=case["depth"],
                            pipeline=case.get("pipeline", False), halo_mode=case.get("halo_mode", 0))
    elif kind == "batch":
        _runtime(case["pes_per_sm"])
        s["probs"] = _problems(case, seed)
        s["flat"] = _pinned(_cells(s["probs"]), _torch_type(case)).numpy()
        s["out"] = _views(s["flat"], s["probs"])
        s["jac"] = Jacobi2D(s["probs"], dtype=case["dtype"], chare_side=case["side"], use_graph=case["graph"])
    elif kind == "serve":
        _runtime()
        s["probs"] = _problems(case, seed)
        s["flat"] = _pinned(_cells(s["probs"]), _torch_type(case)).numpy()
        s["out"] = _views(s["flat"], s["probs"])
    elif kind == "noalloc":
        s["lib"] = _lib.load()
        s["in"] = _uniform((case["ny"] + 2, case["nx"] + 2), _torch_type(case), seed)
        s["out"] = torch.empty_like(s["in"])
    elif kind == "jacobi3d":
        s["lib"] = _runtime().lib
        shape = (case["nz"] + 2, case["ny"] + 2, case["nx"] + 2)
        h = _pinned(shape, torch.float64)
        h.copy_(_uniform(shape, torch.float64, seed))
        s["grid"] = h.numpy()
    else:
        s["rt"] = _runtime()
    return s


# ---- one pass ---------------------------------------------------------------
def run(s: dict):
    case = s["case"]
    kind = case["kind"]
    if kind == "solve":
        j = s["jac"]
        j.load(0, s["in"][0])
        j.run()
        out = {"grid": j.store(0, s["out"][0])}
        if case["check"]:
            r = j.result(0)
            out.update(sweeps=r.sweeps, checks=r.checks, norms=np.array([r.res0, r.res_last]))
        return out
    if kind == "stream":
        s["jac"].solve_stream(0, s["in"], s["out"])
        return s["out"]
    if kind == "batch":
        j = s["jac"]
        j.init()
        j.run()
        for p, o in enumerate(s["out"]):
            j.store(p, o)
        if not case["check"]:
            return {"grids": s["flat"]}
        rs = [j.result(p) for p in range(len(s["probs"]))]
        return {"grids": s["flat"], "sweeps": np.array([r.sweeps for r in rs]),
                "norms": np.array([(r.res0, r.res_last) for r in rs])}
    if kind == "serve":
        probs = s["probs"]
        with Server(2 << 30, max_inflight=64, chare_side=case["side"], dtype=case["dtype"]) as srv:
            for k, p in enumerate(probs):
                srv.submit(p, k)
            done = srv.wait(range(len(probs)))
            for k in range(len(probs)):
                srv.fetch(k, s["out"][k])
                srv.release(k)
        return {"grids": s["flat"], "sweeps": np.array([done[k].sweeps for k in range(len(probs))])}
    if kind == "noalloc":
        _lib.check(s["lib"].charming_jacobi2d_sweeps_noalloc(
            _lib.F64 if case["dtype"] == "f64" else _lib.F32, case["nx"], case["ny"], case["sweeps"],
            s["in"].data_ptr(), s["out"].data_ptr()), "sweeps_noalloc")
        return s["out"]
    if kind == "jacobi3d":
        ms = C.c_double(0.0)
        _lib.check(s["lib"].charming_jacobi3d(case["nx"], case["ny"], case["nz"], case["sweeps"],
                                              s["grid"].ctypes.data_as(C.POINTER(C.c_double)), C.byref(ms)), "jacobi3d")
        return s["grid"]
    # fan-out: the deliveries' records by message (receiver, sender, number,
    # refnum, checksum, receiver's refnum); their order among each other is
    # not fixed, so the sequence number at the receiver is left out
    n, msgs = case["n"], case["msgs"]
    log, _ms = s["rt"].fanout(n, msgs, case["payload"], s["seed"], case["mode"])
    out = np.zeros((n * msgs, 8), dtype=np.uint32)
    out[log[:, 1].astype(np.int64) * msgs + log[:, 2]] = log
    out[:, 4] = 0
    return out.view(np.int32)


# ---- what a pass cannot do without, and its exact outputs -------------------
def work(case: dict) -> dict:
    kind = case["kind"]
    esz = 4 if case.get("dtype") == "f32" else 8
    if kind in ("solve", "stream", "noalloc"):
        n = case.get("n", 1)
        cells = (case["nx"] + 2) * (case["ny"] + 2)
        return {"bytes": 2.0 * n * cells * esz, "flops": 5.0 * n * case["nx"] * case["ny"] * case["sweeps"]}
    if kind in ("batch", "serve"):
        probs = _problems(case, 0)
        return {"bytes": 1.0 * _cells(probs) * esz, "flops": 5.0 * sum(p.nx * p.ny for p in probs) * case["sweeps"]}
    if kind == "jacobi3d":
        cells = (case["nx"] + 2) * (case["ny"] + 2) * (case["nz"] + 2)
        return {"bytes": 16.0 * cells, "flops": 7.0 * case["nx"] * case["ny"] * case["nz"] * case["sweeps"]}
    total = case["n"] * case["msgs"]
    return {"bytes": total * (2.0 * (case["payload"] + 32) + 32), "flops": 0.0}


def _sweep2d(src: torch.Tensor, dst: torch.Tensor) -> None:
    t = dst[1:-1, 1:-1]
    torch.add(src[1:-1, 1:-1], src[1:-1, :-2], out=t)
    t.add_(src[1:-1, 2:]).add_(src[:-2, 1:-1]).add_(src[2:, 1:-1]).mul_(0.2)


def _exact2d(u: torch.Tensor, sweeps: int, check: int = 0):
    """The grid after `sweeps` sweeps, and the norms of S(u) - u at the first
    and the last check."""
    a, b = u.double().clone(), u.double().clone()
    norms = []
    last = (sweeps - 1) // check * check if check else -1
    for k in range(sweeps):
        _sweep2d(a, b)
        if check and k in (0, last):
            norms.append(float((b - a)[1:-1, 1:-1].norm()))
        a, b = b, a
    return a, ([norms[0], norms[-1]] if check else None)


def _exact3d(u: torch.Tensor, sweeps: int) -> torch.Tensor:
    a, b = u.clone(), u.clone()
    c = slice(1, -1)
    for _ in range(sweeps):
        t = b[c, c, c]
        torch.add(a[c, c, c], a[c, c, :-2], out=t)
        t.add_(a[c, c, 2:]).add_(a[c, :-2, c]).add_(a[c, 2:, c]).add_(a[:-2, c, c]).add_(a[2:, c, c]).mul_(0.142857)
        a, b = b, a
    return a


def _initial(p: Problem) -> torch.Tensor:
    g = torch.zeros((p.ny + 2, p.nx + 2), dtype=torch.float64, device="cuda")
    g[:, 0], g[:, -1] = p.bc[2], p.bc[3]
    g[0, :], g[-1, :] = p.bc[0], p.bc[1]
    return g


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "fanout":
        return None
    if kind == "jacobi3d":
        u = _uniform((case["nz"] + 2, case["ny"] + 2, case["nx"] + 2), torch.float64, seed)
        return _exact3d(u, case["sweeps"])
    if kind in ("batch", "serve"):
        probs = _problems(case, seed)
        f32 = case["dtype"] == "f32"
        got = [_exact2d(_initial(p).float() if f32 else _initial(p), p.max_sweeps, p.check_every) for p in probs]
        out = {"grids": torch.cat([g.reshape(-1) for g, _ in got])}
        if kind == "serve":
            out["sweeps"] = None
        elif case["check"]:
            out.update(sweeps=None, norms=np.array([n for _, n in got]))
        return out
    shape = (case["ny"] + 2, case["nx"] + 2)
    dt = _torch_type(case)
    if kind == "stream":
        return [_exact2d(_uniform(shape, dt, seed, k), case["sweeps"])[0] for k in range(case["n"])]
    grid, norms = _exact2d(_uniform(shape, dt, seed), case["sweeps"], case.get("check", 0))
    if kind == "noalloc":
        return grid
    return {"grid": grid, "sweeps": None, "checks": None, "norms": np.array(norms)} if norms else {"grid": grid}
