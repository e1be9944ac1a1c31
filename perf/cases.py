"""The partitioner's measured workloads: what a program has this package do,
through its public entry points (the Context and Server classes and the C ABI
behind them), on inputs drawn from a seed.

The graph families are the ones this package is configured, tested and
benchmarked with: 2D and 3D grids (finite-difference meshes), random
geometric graphs of mean degree 10 and R-MAT graphs of edge factor 16.  A
grid's seed closes one face in a hundred, so that two seeds give two graphs;
the other families are random by nature.

A program keeps one Context (or Server) for all of its graphs, so the states
made here share one, as they share the GPU.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import horkxg_b200 as hb
from horkxg_b200 import graphs

_KEPT = {}


def _context() -> hb.Context:
    if "context" not in _KEPT:
        _KEPT["context"] = hb.Context(0)
    return _KEPT["context"]


def _server() -> hb.Server:
    if "server" not in _KEPT:
        _KEPT["server"] = hb.Server(slots=8)
    return _KEPT["server"]


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # The smallest call: the 64x64 grid of the smoke run.  All latency.
        {"name": "partition_grid_64x64_k4", "do": "partition", "graph": "grid", "nx": 64, "ny": 64, "nz": 1,
         "width": "standard", "weighted": False, "parts": 4, "deterministic": True, "host": False},
        # A typical graph of the batched and serving mixes, taken alone.
        {"name": "partition_rgg_20000_k8", "do": "partition", "graph": "rgg", "n": 20000, "width": "standard",
         "weighted": False, "parts": 8, "deterministic": True, "host": False},
        # The configured 256x256 grid with edge and vertex weights (the weights
        # option: a mesh whose cells cost differently).
        {"name": "partition_grid_256x256_w_k4", "do": "partition", "graph": "grid", "nx": 256, "ny": 256, "nz": 1,
         "width": "standard", "weighted": True, "parts": 4, "deterministic": True, "host": False},
        # A power-law graph handed over from host memory in the file format's
        # int64 arrays, labels back on the host: the drop-in driver's call.
        {"name": "partition_rmat_20_host_k32", "do": "partition", "graph": "rmat", "scale": 20, "width": "standard",
         "weighted": False, "parts": 32, "deterministic": True, "host": True},
        # The headline benchmark: R-MAT 24, k = 32, default (not
        # bit-reproducible) mode, the CSR resident on the device.
        {"name": "partition_rmat_24_k32", "do": "partition", "graph": "rmat", "scale": 24, "width": "standard",
         "weighted": False, "parts": 32, "deterministic": False, "host": False},
        # The full-scale 3D grid in the big (64-bit) width.
        {"name": "partition_grid_320x320x320_big_k8", "do": "partition", "graph": "grid", "nx": 320, "ny": 320,
         "nz": 320, "width": "big", "weighted": False, "parts": 8, "deterministic": True, "host": False},
        # A packed batch of small graphs on the server's slots.
        {"name": "batch_rgg_48", "do": "batch", "count": 48, "n_lo": 1000, "n_hi": 60000},
        # Refinement of a partition that a program already has (an old one,
        # disturbed where the graph changed).
        {"name": "refine_grid_1000x997_k16", "do": "refine", "nx": 1000, "ny": 997, "nz": 1, "parts": 16},
        # The spectral partition of a graph of coarsest-level size, weighted as
        # contraction leaves it.
        {"name": "initial_rgg_3001_k32", "do": "initial", "n": 3001, "parts": 32},
        # One coarsening step of a power-law graph: the aggregation alone.
        {"name": "aggregate_rmat_20_k32", "do": "aggregate", "scale": 20, "parts": 32},
        # The report on a finished partition.
        {"name": "analyze_rmat_22_k32", "do": "analyze", "scale": 22, "parts": 32},
        # Preparing a directed link graph: both directions, no duplicates.
        {"name": "symmetrize_1000003_16m", "do": "symmetrize", "n": 1000003, "m": 16000000},
    ]


def _log_uniform(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    do = rng.choice(["partition", "partition", "partition", "batch", "refine", "initial", "aggregate", "analyze",
                     "symmetrize"])
    parts = rng.randint(2, 32)
    if do == "partition":
        c = {"do": do, "graph": rng.choice(["grid", "grid3", "rgg", "rmat"]), "parts": parts,
             "width": rng.choice(["standard", "standard", "big"]), "weighted": rng.random() < 0.25,
             "deterministic": True, "host": rng.random() < 0.25}
        if c["graph"] == "grid":
            n = _log_uniform(rng, 4e3, 4e6)
            nx = _log_uniform(rng, 0.5 * n ** 0.5, 2 * n ** 0.5)
            c.update(nx=nx, ny=max(2, n // nx), nz=1)
        elif c["graph"] == "grid3":
            n = _log_uniform(rng, 4e3, 2e7)
            nx = _log_uniform(rng, 0.6 * n ** (1 / 3), 1.6 * n ** (1 / 3))
            ny = _log_uniform(rng, 0.6 * n ** (1 / 3), 1.6 * n ** (1 / 3))
            c.update(graph="grid", nx=nx, ny=ny, nz=max(2, n // (nx * ny)))
        elif c["graph"] == "rgg":
            c.update(n=_log_uniform(rng, 1e3, 1e6))
        else:
            c.update(scale=rng.randint(12, 22))
            # at this size and above the cut of the default mode repeats well
            # enough to be compared
            c.update(deterministic=c["scale"] < 18 or rng.random() < 0.5)
        # enough vertices in a part for 3% of it to hold a heavy vertex
        c["weighted"] = c["weighted"] and _size(c)[0] >= 200 * parts
        return c
    if do == "batch":
        count = rng.randint(8, 48)
        return {"do": do, "count": count, "n_lo": 1000, "n_hi": _log_uniform(rng, 1e4, 1e5)}
    if do == "refine":
        n = _log_uniform(rng, 1e4, 4e6)
        nx = _log_uniform(rng, 0.5 * n ** 0.5, 2 * n ** 0.5)
        return {"do": do, "nx": nx, "ny": max(2, n // nx), "nz": 1, "parts": parts}
    if do == "initial":
        return {"do": do, "n": parts * rng.randint(90, 190), "parts": parts}
    if do == "aggregate":
        return {"do": do, "scale": rng.randint(14, 22), "parts": parts}
    if do == "analyze":
        return {"do": do, "scale": rng.randint(14, 22), "parts": parts}
    n = _log_uniform(rng, 1e4, 4e6)
    return {"do": do, "n": n, "m": min(30_000_000, n * rng.randint(4, 24))}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
class DeviceGraph:
    """A CSR on the GPU in the width's own types, passed in place."""

    def __init__(self, off, nbr, width: int, ew=None, vw=None):
        self.width = width
        wdt = torch.int32 if width == hb.STANDARD else torch.int64   # the bits of uint32 / uint64
        self.off = off.to(torch.int32 if width == hb.STANDARD else torch.int64)
        self.nbr = nbr.to(torch.int32)
        self.ew = None if ew is None else ew.to(wdt)
        self.vw = None if vw is None else vw.to(wdt)
        self.n, self.m = len(self.off) - 1, len(self.nbr)

    def desc(self) -> hb.GraphDesc:
        d = hb.GraphDesc()
        d.n, d.m, d.width, d.memory, d.index64 = self.n, self.m, self.width, hb.DEVICE, 0
        d.offsets, d.neighbors = self.off.data_ptr(), self.nbr.data_ptr()
        d.edge_weights = None if self.ew is None else self.ew.data_ptr()
        d.vertex_weights = None if self.vw is None else self.vw.data_ptr()
        return d


def _generator(seed: int) -> torch.Generator:
    return torch.Generator("cuda").manual_seed(seed)


def _grid(nx: int, ny: int, nz: int, seed: int):
    """Grid of nx * ny * nz cells (5-point for nz = 1, else 7-point), rows in
    ascending order, with one face in a hundred closed."""
    gen = _generator(seed)
    v = torch.arange(nx * ny * nz, dtype=torch.int32, device="cuda").view(nz, ny, nx)
    columns = []   # (id offset of the neighbour, whether the face is open)
    for axis, step in ((0, nx * ny), (1, nx), (2, 1)):
        face = torch.rand(v.shape, generator=gen, device="cuda") >= 0.01   # the face towards the next cell
        face.select(axis, v.shape[axis] - 1).fill_(False)
        columns += [(step, face), (-step, torch.roll(face, 1, axis))]
    columns.sort(key=lambda c: c[0])
    has = torch.stack([f.reshape(-1) for _, f in columns], 1)
    off = torch.zeros(v.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(has.sum(1), 0, out=off[1:])
    nbr = torch.stack([v.reshape(-1) + step for step, _ in columns], 1)[has]
    return off, nbr


def _rgg(n: int, seed: int):
    off, nbr = graphs.rgg_csr(n, 10.0, seed)
    return torch.from_numpy(off).cuda(), torch.from_numpy(nbr).cuda()


def _rmat(scale: int, seed: int):
    """R-MAT of edge factor 16, made on the GPU by the package's generator."""
    n = 1 << scale
    off = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    nbr = torch.empty(32 * n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    info = hb.SymmetrizeInfo()
    ctx = _context()
    ctx._check(hb.lib().gp_generate_rmat(ctx._h, scale, 16, 0.57, 0.19, 0.19, seed, hb.DEVICE, off.data_ptr(),
                                         nbr.data_ptr(), 4, len(nbr), ctypes.byref(info)))
    return off, nbr[:info.output_directed_edges]


def _csr(case: dict, seed: int):
    if case.get("graph", "grid") == "grid":
        return _grid(case["nx"], case["ny"], case["nz"], seed)
    if case["graph"] == "rgg":
        return _rgg(case["n"], seed)
    return _rmat(case["scale"], seed)


def _weights(off, nbr, seed: int):
    """Symmetric edge weights in [1, 16] and vertex weights in [1, 8]."""
    n = len(off) - 1
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), off[1:] - off[:-1])
    lo, hi = torch.minimum(row, nbr.long()), torch.maximum(row, nbr.long())
    ew = 1 + ((lo * 2654435761 + hi * 40503 + seed * 69069) % 1000003) % 16
    vw = torch.randint(1, 9, (n,), generator=_generator(seed + 1), device="cuda")
    return ew, vw


def _width(case: dict) -> int:
    return hb.BIG if case.get("width") == "big" else hb.STANDARD


def prepare(case: dict, seed: int) -> dict:
    do = case["do"]
    state = {"case": case, "seed": seed, "ctx": _context()}
    if do == "partition":
        off, nbr = _csr(case, seed)
        ew = vw = None
        if case["weighted"]:
            ew, vw = _weights(off, nbr, seed)
        if case["host"]:
            pinned = [x.to(torch.int64).cpu().pin_memory().numpy() for x in (off, nbr)]
            state["graph"] = hb.HostGraph(*pinned, None if ew is None else ew.cpu().numpy(),
                                          None if vw is None else vw.cpu().numpy(), _width(case), index64=True)
        else:
            state["graph"] = DeviceGraph(off, nbr, _width(case), ew, vw)
            state["labels"] = torch.empty(state["graph"].n, dtype=torch.int32, device="cuda")
        state["options"] = hb.default_options(parts=case["parts"], seed=seed % 5,
                                              deterministic=int(case["deterministic"]))
    elif do == "batch":
        # sizes spread evenly over their logarithm, in no order
        rng = np.random.default_rng(case["count"])
        ns = rng.permutation(np.geomspace(case["n_lo"], case["n_hi"], case["count"]).astype(np.int64))
        ks = rng.choice(np.array([2, 4, 8, 16, 32]), case["count"])
        state["packed"] = hb.PackedGraph.pack(graphs.rgg_csr(int(n), 10.0, seed * 1_000_003 + i)
                                              for i, n in enumerate(ns))
        state["options"] = [hb.default_options(parts=int(k), deterministic=1) for k in ks]
        state["server"] = _server()
    elif do == "refine":
        g = DeviceGraph(*_csr(case, seed), hb.STANDARD)
        # stripes of equal size in the grid's order, one vertex in twenty
        # exchanged with another such vertex
        labels = (torch.arange(g.n, device="cuda") * case["parts"] // g.n).int()
        gen = _generator(seed + 2)
        moved = (torch.rand(g.n, generator=gen, device="cuda") < 0.05).nonzero().view(-1)
        labels[moved] = labels[moved[torch.randperm(len(moved), generator=gen, device="cuda")]]
        state.update(graph=g, labels=labels.cpu().numpy())
    elif do == "initial":
        off, nbr = _rgg(case["n"], seed)
        state["graph"] = DeviceGraph(off, nbr, hb.STANDARD, *_weights(off, nbr, seed))
    elif do == "aggregate":
        state["graph"] = DeviceGraph(*_rmat(case["scale"], seed), hb.STANDARD)
    elif do == "analyze":
        g = DeviceGraph(*_rmat(case["scale"], seed), hb.STANDARD)
        labels = torch.empty(g.n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        state["ctx"].partition_desc(g.desc(), labels.data_ptr(),
                                    hb.default_options(parts=case["parts"], deterministic=1))
        state.update(graph=g, labels=labels)
    elif do == "symmetrize":
        # links whose ends are skewed towards popular vertices, grouped by
        # source, targets unsorted; some are self loops and duplicates
        n, m, gen = case["n"], case["m"], _generator(seed)
        name = torch.randperm(n, generator=gen, device="cuda")
        src, dst = (name[(n * torch.rand(m, generator=gen, device="cuda", dtype=torch.float64) ** 2).long()]
                    for _ in range(2))
        src, order = torch.sort(src)
        off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        torch.cumsum(torch.bincount(src, minlength=n), 0, out=off[1:])
        state["graph"] = DeviceGraph(off, dst[order], hb.STANDARD)
        state["off_out"] = torch.empty(n + 1, dtype=torch.int64, device="cuda")
        state["nbr_out"] = torch.zeros(2 * m, dtype=torch.int64, device="cuda")   # the tail stays zero
    torch.cuda.synchronize()   # the library works on its own stream
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state: dict):
    case, ctx = state["case"], state["ctx"]
    do = case["do"]
    if do == "partition":
        if case["host"]:
            labels, report = ctx.partition(state["graph"], state["options"])
        else:
            labels = state["labels"]
            report = ctx.partition_desc(state["graph"].desc(), labels.data_ptr(), state["options"])
        if not case["deterministic"]:
            # the default mode's labels differ from run to run by design; its
            # cut, its heaviest part and the hierarchy's shape are its result
            return {"cut": float(report.cut), "heaviest": float(max(report.part_weights)), "levels": report.levels,
                    "coarsest": report.coarsest_n}
        return {"labels": labels, "cut": report.cut, "weights": np.array(report.part_weights[:case["parts"]], np.int64)}
    if do == "batch":
        labels, reports = state["server"].partition_batch(state["packed"], state["options"])
        return {"labels": labels, "cuts": np.array([r.cut for r in reports], np.int64)}
    if do == "refine":
        labels, stats = ctx.refine(state["graph"], state["labels"], case["parts"])
        return {"labels": labels, "cut": stats.final_cut}
    if do == "initial":
        return {"labels": ctx.initial_partition(state["graph"], case["parts"], seed=state["seed"] % 5)}
    if do == "aggregate":
        cluster, count, cap = ctx.aggregate(state["graph"], case["parts"], state["seed"] % 5, 0)
        return {"map": cluster, "count": count, "cap": cap}
    if do == "analyze":
        parts = (hb.PartStats * case["parts"])()
        summary = hb.Analysis()
        ctx._check(hb.lib().gp_analyze(ctx._h, ctypes.byref(state["graph"].desc()), state["labels"].data_ptr(),
                                       case["parts"], parts, ctypes.byref(summary)))
        return {"parts": np.array([[getattr(p, f) for f, _ in hb.PartStats._fields_] for p in parts], np.int64),
                "summary": np.array([summary.vertex_imbalance, summary.vertex_max_deviation,
                                     summary.edge_set_imbalance, summary.edge_set_max_deviation])}
    info = hb.SymmetrizeInfo()
    ctx._check(hb.lib().gp_symmetrize(ctx._h, ctypes.byref(state["graph"].desc()), state["off_out"].data_ptr(),
                                      state["nbr_out"].data_ptr(), 8, len(state["nbr_out"]), ctypes.byref(info)))
    return {"offsets": state["off_out"], "neighbors": state["nbr_out"],
            "entries": info.output_directed_edges, "loops": info.self_loops_removed}


# ---------------------------------------------------------------------------
# Bytes, tolerances, reference values
# ---------------------------------------------------------------------------
def _size(case: dict) -> tuple[float, float]:
    """Vertices and (about) directed entries."""
    if "nx" in case:
        x, y, z = case["nx"], case["ny"], case["nz"]
        return x * y * z, 2 * 0.99 * (3 * x * y * z - x * y - y * z - x * z)
    if "scale" in case:
        return 1 << case["scale"], 0.95 * 32 * (1 << case["scale"])
    if "count" in case:
        n = case["count"] * (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])
        return n, 9.8 * n
    return case["n"], case.get("m", 9.8 * case["n"])


def work(case: dict) -> dict:
    n, m = _size(case)
    o = w = 8 if case.get("width") == "big" else 4
    do = case["do"]
    if do == "partition" and case["host"]:
        bytes_ = (n + m) * 8 + n * 4
    elif do == "batch":
        bytes_ = n * 8 + m * 4 + n * 4
    else:
        bytes_ = n * o + m * 4 + n * 4
    if case.get("weighted") or do == "initial":
        bytes_ += (n + m) * w
    if do == "refine":
        bytes_ += n * 4
    if do == "symmetrize":
        bytes_ = n * 12 + m * 4 + 2 * m * 8   # int32 CSR in, int64 CSR out
    return {"bytes": bytes_, "flops": 0}


def tolerance(case: dict):
    if case["do"] == "partition" and not case["deterministic"]:
        # run-to-run spread of the default mode's cut: below 0.5% on R-MAT
        return {"rel": 0.02, "max": 0.02, "differ": 0.0}
    if case["do"] == "analyze":
        return {"rel": 1e-14, "max": 1e-13, "differ": 0.0}   # ratios of exact counts
    return "exact"


def exact(case: dict, seed: int):
    """Only the analyzer's ratios are computed floating-point numbers; every
    other output is whole numbers (or a default-mode cut, which has no single
    right value)."""
    if case["do"] != "analyze":
        return None
    s = prepare(case, seed)
    g, lab, k = s["graph"], s["labels"].long(), case["parts"]
    src = torch.repeat_interleave(lab, (g.off[1:] - g.off[:-1]).long())
    dst = lab[g.nbr.long()]
    cross = src != dst
    vertices = torch.bincount(lab, minlength=k)
    inside = torch.bincount(src[~cross], minlength=k)
    leaving, entering = torch.bincount(src[cross], minlength=k), torch.bincount(dst[cross], minlength=k)
    parts = torch.stack([vertices, inside, leaving, entering, inside, leaving, entering], 1)
    ratios = []
    for x, mean in ((vertices, g.n / k), (inside + leaving + entering, (g.m + int(leaving.sum())) / k)):
        x = x.double()
        ratios += [float(x.max()) / mean, float((x - mean).abs().max()) / mean]
    return {"parts": parts.cpu().numpy(), "summary": np.array(ratios)}
