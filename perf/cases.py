"""The work that programs have this library do, as measurable cases.

A circuit simulator calls the library in a few ways, and each is here:

  newton     one step of a Newton or Monte-Carlo loop: fresh matrix values and
             right-hand sides come from host memory, the batch is refactored
             and solved, and the solutions go back to the host
  corners    the same for many circuits of uneven sizes and patterns in one
             launch, the values already in the batch's device buffers
  factor     the refactorization alone of one large circuit, its factor read
             on the device
  transient  solves alone: new right-hand sides against factors that stay
  spmv       the standalone SELL sparse matrix-vector product
  classic    the single-matrix kernels of lu_gpu_par.h: factorization with
             pivoting on the device, then the triangular solve
  serve      requests of concurrent simulations to the serving loop

Circuits come from the generators of luspice_b200.mna (analog netlists, power
grids, netlists with supply nets) and, for the large products, from a mesh.
A case is a dict of plain values; "circuit" seeds the netlist, and the seed of
prepare() gives the element values and right-hand sides.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from luspice_b200 import _lib, api, mna

PREC = {"mixed": api.MIXED, "fp64": api.FP64}


# ---------------------------------------------------------------------------
# Circuits and inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=256)
def circuit(kind: str, n: int, seed: int):
    """A netlist's matrix: an analog circuit, a power grid or a netlist with
    supply nets of about n unknowns."""
    return mna.serving_class(kind, n, seed)


def corner_sizes(case) -> list[int]:
    """The uneven sizes of a corner run, uniform in [lo, hi]."""
    return [int(v) for v in mna.batch_sizes(case["patterns"], case["lo"], case["hi"], case["circuit"])]


def serve_kinds(case) -> list[tuple[str, int]]:
    """(kind, n) of the served circuits: sizes log-uniform in [lo, hi]."""
    ns = np.exp(np.random.default_rng(case["circuit"]).uniform(math.log(case["lo"]), math.log(case["hi"]),
                                                               case["patterns"])).astype(int)
    return [(("analog", "grid")[i % 2], int(n)) for i, n in enumerate(ns)]


def systems(case, seed: int):
    """[(matrix, values [count, nnz], rhs [count, n])] of a case: the element
    values of each Newton step or corner differ by a log-normal factor."""
    rng = np.random.default_rng([seed, case["circuit"]])
    if case["op"] == "corners":
        mats = [(circuit("analog", n, case["circuit"] + i), case["corners"]) for i, n in enumerate(corner_sizes(case))]
    elif case["op"] == "serve":
        mats = [(circuit(k, n, case["circuit"] + i), case["requests"] // case["patterns"])
                for i, (k, n) in enumerate(serve_kinds(case))]
    else:
        mats = [(circuit(case["kind"], case["n"], case["circuit"]), case.get("systems", 1))]
    out = []
    for m, count in mats:
        vals = m.perturbed(count, int(rng.integers(1 << 31)))
        rhs = m.b * np.exp(0.1 * rng.standard_normal((count, m.n)))
        out.append((m, vals, rhs))
    return out


def mesh(case, seed: int):
    """CSR arrays of a mesh of conductances in [0.1, 10] with a grounded
    capacitor companion at each node (the power grid's stamps)."""
    side = max(2, int(math.sqrt(case["n"])))
    cols = max(2, case["n"] // side)
    n = side * cols
    rng = np.random.default_rng([seed, case["circuit"]])
    idx = np.arange(n, dtype=np.int64).reshape(side, cols)
    gh = np.exp(rng.uniform(math.log(0.1), math.log(10.0), (side, cols - 1)))
    gv = np.exp(rng.uniform(math.log(0.1), math.log(10.0), (side - 1, cols)))
    dia = np.exp(rng.uniform(math.log(1e-2), math.log(1.0), (side, cols)))
    dia[:, :-1] += gh
    dia[:, 1:] += gh
    dia[:-1] += gv
    dia[1:] += gv
    col = np.full((side, cols, 5), -1, dtype=np.int64)      # up, left, self, right, down
    val = np.zeros((side, cols, 5))
    col[1:, :, 0], val[1:, :, 0] = idx[:-1], -gv
    col[:, 1:, 1], val[:, 1:, 1] = idx[:, :-1], -gh
    col[:, :, 2], val[:, :, 2] = idx, dia
    col[:, :-1, 3], val[:, :-1, 3] = idx[:, 1:], -gh
    col[:-1, :, 4], val[:-1, :, 4] = idx[1:], -gv
    keep = col >= 0
    rowptr = np.zeros(n + 1, dtype=np.int32)
    rowptr[1:] = np.cumsum(keep.reshape(n, 5).sum(1))
    return n, rowptr, col[keep].astype(np.int32), val[keep]


def sell_matrix(case, seed: int):
    """CSR arrays of a product's matrix."""
    if case["kind"] == "mesh":
        return mesh(case, seed)
    m = circuit(case["kind"], case["n"], case["circuit"])
    a = m.csr(m.perturbed(1, seed)[0])
    return m.n, a.indptr, a.indices, a.data


class _Device:
    """Device memory of a batch, for torch; keeps the batch that owns it alive."""

    def __init__(self, owner, ptr: int, count: int, kind: str):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": kind, "data": (ptr, False), "version": 3}


def device_view(owner, ptr: int, count: int, kind: str = "<f8") -> torch.Tensor:
    return torch.as_tensor(_Device(owner, ptr, count, kind), device="cuda")


def pinned(a: np.ndarray) -> np.ndarray:
    return torch.from_numpy(np.ascontiguousarray(a).ravel()).pin_memory().numpy()


def on_gpu(a, dtype) -> torch.Tensor:
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest circuit of the serving workload, one Newton step: the
        # inner loop of a single simulation, where launches and latency count.
        dict(name="newton_analog113_x1", op="newton", kind="analog", n=113, circuit=42, systems=1, prec="mixed"),
        # Monte-Carlo samples of the reference's n = 989 analog circuit.
        dict(name="newton_analog989_x50", op="newton", kind="analog", n=989, circuit=42, systems=50, prec="mixed"),
        # One Newton step of one power grid: the request latency of a single simulation.
        dict(name="newton_grid4050_x1", op="newton", kind="grid", n=4050, circuit=42, systems=1, prec="mixed"),
        # The headline batch: 50 value sets of the n = 4050 power grid, in the
        # mixed precision and in plain fp64.
        dict(name="newton_grid4050_x50", op="newton", kind="grid", n=4050, circuit=42, systems=50, prec="mixed"),
        dict(name="newton_grid4050_x50_fp64", op="newton", kind="grid", n=4050, circuit=42, systems=50, prec="fp64"),
        # Corners of many circuits with their own patterns and sizes in one launch.
        dict(name="corners_48x16", op="corners", patterns=48, corners=16, lo=100, hi=5000, circuit=42, prec="mixed"),
        # The largest circuit: 40,000 unknowns, dense supply rows.
        dict(name="factor_supply40000", op="factor", kind="supply", n=40000, circuit=42, prec="fp64"),
        # Time steps of a linear circuit: the factors stay, the sources change.
        dict(name="transient_analog3001_x100", op="transient", kind="analog", n=3001, circuit=7, systems=100,
             prec="fp64"),
        # Products of the large circuit (long supply rows beside short ones)
        # and of a mesh larger than the cache.
        dict(name="spmv_supply40000_fp32", op="spmv", kind="supply", n=40000, circuit=42, values="fp32"),
        dict(name="spmv_mesh2m_fp64", op="spmv", kind="mesh", n=2000000, circuit=42, values="fp64"),
        # The reference's own single-matrix calls on its n = 989 circuit.
        dict(name="classic_analog989", op="classic", kind="analog", n=989, circuit=42),
        # Concurrent simulations of six circuits through the serving loop.
        dict(name="serve_6x16", op="serve", patterns=6, requests=96, lo=113, hi=4050, circuit=42, prec="mixed"),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["newton", "newton", "newton", "newton", "corners", "factor", "transient", "transient", "spmv",
                     "spmv", "classic", "serve"])
    seed, prec = rng.randrange(1, 10000), rng.choice(["mixed", "fp64"])
    kind = rng.choice(["analog", "grid"])
    if op in ("newton", "transient"):
        n = _log(rng, 113, 5000) if kind == "analog" else _log(rng, 200, 4100)
        count = _log(rng, 1, 128) if op == "newton" else _log(rng, 8, 256)
        return dict(op=op, kind=kind, n=n, circuit=seed, systems=count, prec=prec)
    if op == "corners":
        return dict(op=op, patterns=rng.randrange(16, 49), corners=rng.randrange(4, 17), lo=100,
                    hi=rng.randrange(1000, 5001), circuit=seed, prec=prec)
    if op == "factor":
        return dict(op=op, kind="supply", n=_log(rng, 8000, 40000), circuit=seed, prec=prec)
    if op == "spmv":
        if rng.random() < 0.5:
            return dict(op=op, kind="supply", n=_log(rng, 4000, 40000), circuit=seed,
                        values=rng.choice(["fp64", "fp32"]))
        return dict(op=op, kind="mesh", n=_log(rng, 10000, 2000000), circuit=seed,
                    values=rng.choice(["fp64", "fp32", "fp16"]))
    if op == "classic":
        return dict(op=op, kind="analog", n=_log(rng, 113, 989), circuit=seed)
    patterns = rng.randrange(3, 7)
    return dict(op=op, patterns=patterns, requests=patterns * rng.randrange(6, 17), lo=113,
                hi=rng.randrange(989, 4051), circuit=seed, prec=prec)


# ---------------------------------------------------------------------------
# What a program has in hand, and one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    op = case["op"]
    if op == "spmv":
        n, rowptr, col, val = sell_matrix(case, seed)
        sell = api.Sell(n, rowptr, col, val, 32, 256, case["values"])
        x = on_gpu(np.random.default_rng(seed).uniform(-1.0, 1.0, n), torch.float64)
        return dict(op=op, sell=sell, x=x, y=torch.zeros(n, dtype=torch.float64, device="cuda"))
    sets = systems(case, seed)
    if op == "classic":
        m, vals, rhs = sets[0]
        q = api.colamd(m.n, m.Ap, m.Ai)
        order = np.concatenate([np.arange(m.Ap[c], m.Ap[c + 1]) for c in q])
        ap = np.concatenate([[0], np.cumsum(np.diff(m.Ap)[q])])
        f = api.pivot_factor(m.n, m.Ap, m.Ai, m.Ax, q)
        cap = 2 * int(max(f["lnnz"], f["unnz"])) + 1024
        i32, f64 = torch.int32, torch.float64

        def zeros(k, t):
            return torch.zeros(k, dtype=t, device="cuda")
        return dict(op=op, n=m.n, cap=cap, Ap=on_gpu(ap, i32), Ai=on_gpu(m.Ai[order], i32),
                    Ax=on_gpu(vals[0][order], f64), q=on_gpu(q, i32), b=on_gpu(rhs[0], f64), Lp=zeros(m.n + 1, i32),
                    Li=zeros(cap, i32), Lx=zeros(cap, f64), Up=zeros(m.n + 1, i32), Ui=zeros(cap, i32),
                    Ux=zeros(cap, f64), pinv=zeros(m.n, i32), xi=zeros(m.n + 2048, i32), info=zeros(3, i32),
                    x=zeros(m.n, f64), wi=zeros(m.n, i32), wd=zeros(2 * m.n, f64), lib=_lib.load())
    if op == "serve":
        # The simulations run already: their patterns are analysed and cached.
        server = api.Server(prec=PREC[case["prec"]], arena_gb=1.0, staging_mb=64.0)
        for m, vals, rhs in sets:
            server.poll(server.submit(m.n, m.Ap, m.Ai, m.Ax, m.b))
        # Requests of the simulations interleaved, as they arrive.
        reqs = [(m, vals[t], rhs[t]) for t in range(sets[0][1].shape[0]) for m, vals, rhs in sets]
        return dict(op=op, server=server, reqs=reqs)
    pats = []
    for m, vals, _ in sets:
        pats += [api.Pattern.from_matrix(m)] * vals.shape[0]
    batch = api.Batch(pats, prec=PREC[case["prec"]])
    vals = pinned(np.concatenate([v.ravel() for _, v, _ in sets]))
    rhs = pinned(np.concatenate([b.ravel() for _, _, b in sets]))
    state = dict(op=op, batch=batch, vals=vals, rhs=rhs, out=pinned(np.zeros(rhs.size)))
    state["x"] = device_view(batch, batch.device_ptrs(0)[2], rhs.size)
    batch.upload(vals, rhs)
    if op == "transient":
        batch.run(api.RUN_REFACTOR)
    if op == "factor":
        state["cap"] = pats[0].info["cap"]
        state["kind"] = "<f8" if case["prec"] == "fp64" else "<f4"
    torch.cuda.synchronize()
    # The corners' solutions come back circuit by circuit.
    state["split"] = [v.shape[0] * m.n for m, v, _ in sets]
    return state


def run(state):
    op = state["op"]
    if op == "spmv":
        state["sell"].spmv(state["x"].data_ptr(), state["y"].data_ptr())
        return state["y"]
    if op == "classic":
        s, n, cap = state, state["n"], state["cap"]
        p = lambda k: C.c_void_p(s[k].data_ptr())  # noqa: E731
        info = s["info"].data_ptr()
        rc = s["lib"].lusp_lu_factor_par_launch(n, p("Ap"), p("Ai"), p("Ax"), p("q"), p("Lp"), p("Li"), p("Lx"), cap,
                                                p("Up"), p("Ui"), p("Ux"), cap, p("pinv"), p("xi"), None,
                                                C.c_void_p(info), C.c_void_p(info + 4), C.c_void_p(info + 8), None)
        rc |= s["lib"].lusp_trisolve_par_launch(n, p("Lp"), p("Li"), p("Lx"), p("Up"), p("Ui"), p("Ux"), p("pinv"),
                                                p("q"), p("b"), p("x"), p("wi"), p("wd"), None)
        if rc != 0:
            raise RuntimeError(f"classic: rc={rc}")
        return {k: s[k] for k in ("x", "Lp", "Li", "Lx", "Up", "Ui", "Ux", "pinv", "info")}
    if op == "serve":
        server = state["server"]
        ids = [server.submit(m.n, m.Ap, m.Ai, v, b) for m, v, b in state["reqs"]]
        return np.concatenate([server.poll(i)[0] for i in ids])
    batch = state["batch"]
    if op == "newton":
        batch.upload(state["vals"], state["rhs"])
        batch.run(api.RUN_BOTH, graph=True)
        return batch.download(state["out"])
    if op == "corners":
        batch.run(api.RUN_BOTH, graph=True)
        return list(torch.split(state["x"], state["split"]))
    if op == "transient":
        batch.run(api.RUN_SOLVE, graph=True)
        return state["x"]
    batch.run(api.RUN_REFACTOR, graph=True)
    ptr = C.c_void_p()
    api._check(_lib.load().lusp_batch_factor_device_ptr(batch.handle, 0, C.byref(ptr)), "factor_device_ptr")
    return device_view(batch, ptr.value, state["cap"], state["kind"])


# ---------------------------------------------------------------------------
# What a pass cannot do without, and its exact result
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=256)
def _factor_counts(kind: str, n: int, seed: int):
    """(multiply-subtract pairs of the factorization, entries of L and U)."""
    m = circuit(kind, n, seed)
    f = api.pivot_factor(m.n, m.Ap, m.Ai, m.Ax, api.colamd(m.n, m.Ap, m.Ai))
    below = np.diff(f["Lp"]) - 1
    return int(below[f["Ui"]].sum() - below.sum()), f["lnnz"] + f["unnz"]


def work(case):
    op = case["op"]
    if op == "spmv":
        if case["kind"] == "mesh":
            side = max(2, int(math.sqrt(case["n"])))
            cols = max(2, case["n"] // side)
            n, nnz = side * cols, 5 * side * cols - 2 * (side + cols)
        else:
            m = circuit(case["kind"], case["n"], case["circuit"])
            n, nnz = m.n, m.nnz
        size = {"fp64": 8, "fp32": 4, "fp16": 2}[case["values"]]
        return {"bytes": nnz * (size + 4) + 4 * (n + 1) + 16 * n, "flops": 2 * nnz}
    if op == "corners":
        keys = [("analog", n, case["circuit"] + i, case["corners"]) for i, n in enumerate(corner_sizes(case))]
    elif op == "serve":
        keys = [(k, n, case["circuit"] + i, case["requests"] // case["patterns"])
                for i, (k, n) in enumerate(serve_kinds(case))]
    else:
        keys = [(case["kind"], case["n"], case["circuit"], case.get("systems", 1))]
    size = 4 if case.get("prec") == "mixed" else 8
    total, flops = 0, 0
    for kind, n, seed, count in keys:
        m = circuit(kind, n, seed)
        pairs, entries = _factor_counts(kind, n, seed)
        # The pattern's indices once; per system the values, the factor and
        # the vectors.
        total += 4 * (m.nnz + entries + 2 * n)
        vectors = 0 if op == "factor" else 16 * m.n
        values = 0 if op == "transient" else 8 * m.nnz
        total += count * (values + vectors + size * entries)
        flops += count * ((0 if op == "transient" else 2 * pairs) + (0 if op == "factor" else 2 * entries))
    return {"bytes": total, "flops": flops}


def _dense(m, vals) -> torch.Tensor:
    cols = np.repeat(np.arange(m.n), np.diff(m.Ap))
    a = torch.zeros((m.n, m.n), dtype=torch.float64, device="cuda")
    a.index_put_((on_gpu(m.Ai, torch.int64), on_gpu(cols, torch.int64)), on_gpu(vals, torch.float64), accumulate=True)
    return a


def _solve(m, vals, rhs) -> torch.Tensor:
    """The solution in 64 bits by dense LU, with one step of refinement."""
    a, b = _dense(m, vals), on_gpu(rhs, torch.float64)[:, None]
    lu, piv = torch.linalg.lu_factor(a)
    x = torch.linalg.lu_solve(lu, piv, b)
    return (x + torch.linalg.lu_solve(lu, piv, b - a @ x))[:, 0]


def exact(case, seed):
    op = case["op"]
    if op == "spmv":
        n, rowptr, col, val = sell_matrix(case, seed)
        if case["values"] == "fp32":
            val = val.astype(np.float32).astype(np.float64)
        elif case["values"] == "fp16":
            return None
        x = np.random.default_rng(seed).uniform(-1.0, 1.0, n)
        return on_gpu(np.add.reduceat(val * x[col], rowptr[:-1]), torch.float64)
    if op == "factor":
        return None
    sets = systems(case, seed)
    if op == "classic":
        m, vals, rhs = sets[0]
        return {"x": _solve(m, vals[0], rhs[0]), "Lp": None, "Li": None, "Lx": None, "Up": None, "Ui": None,
                "Ux": None, "pinv": None, "info": None}
    if op == "serve":
        return torch.cat([_solve(m, vals[t], rhs[t]) for t in range(sets[0][1].shape[0]) for m, vals, rhs in sets])
    if op == "corners":
        # The smaller circuits: a dense solution of all would take too long.
        return [torch.cat([_solve(m, v, b) for v, b in zip(vals, rhs)]) if m.n <= 1000 else None
                for m, vals, rhs in sets]
    m, vals, rhs = sets[0]
    return torch.cat([_solve(m, v, b) for v, b in zip(vals, rhs)])
