"""The engine's workloads as a user's program runs them, for timing.

A step is one graph (or one batch of graphs, or one burst of served requests) taken from its
edge list to its triangle count through the package's public entry points.  The handle that
is rebuilt step after step, the batch and the server are what such a program keeps, so
``prepare`` makes them (from other graphs of the same kind: a program's next graph is never
the one its handle already holds), and ``run`` takes the step.

  listed()            the named cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) inputs (made from the seed) and the kept handle
  run(state)          one step; returns its outputs
  work(case)          bytes one step cannot do without
  exact(case, seed)   the same outputs computed plainly in 64 bits, where that is quick
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "btc-tc-artifact_b200"))

from btc_b200 import api as A  # noqa: E402
from btc_b200 import graphs as G  # noqa: E402


def listed():
    return [
        # the smallest graphs of the mixed batches, one at a time: a step is its latency
        dict(name="er_256", mode="wait", graph="er", n=256, degree=24.0),
        # a plain random graph, one blocking rebuild + count per graph
        dict(name="er_16384", mode="wait", graph="er", n=16384, degree=16.0),
        # a banded mesh in natural order, steps enqueued without waiting (a stream of graphs)
        dict(name="mesh27_64", mode="enqueue", graph="mesh27", k=64),
        # a wide sparse grid, whose cell bitmap is too large for its edges (sort-based build)
        dict(name="mesh7_144", mode="wait", graph="mesh7", k=144),
        # a one-off graph: a new handle built, counted and freed (a command-line run)
        dict(name="rmat16_once", mode="once", graph="rmat", scale=16, ef=8, by_degree=False),
        # communities: dense neighbourhoods, the heaviest kind of the mixed batches
        dict(name="sbm_32768", mode="wait", graph="sbm", n=32768, p_in=0.2),
        # a large request that arrives in host memory: copy, degree-ordered build and count
        dict(name="rmat20_host", mode="host", graph="rmat", scale=20, ef=16, by_degree=True),
        # the headline graph: degree-ordered R-MAT of 67M draws, steps enqueued
        dict(name="rmat22", mode="enqueue", graph="rmat", scale=22, ef=16, by_degree=True),
        # the reference-shaped calls: preprocess, convert, adaptive count, free
        dict(name="reference_rmat18", mode="reference", graph="rmat", scale=18, ef=16,
             by_degree=False, tile_cols=128),
        dict(name="reference_er_65000", mode="reference", graph="er", n=65000, degree=24.0,
             by_degree=False, tile_cols=32),
        # many graphs of mixed kinds and sizes in one build and one count, sizes new each time
        dict(name="batch_256", mode="batch", graphs=256, n_max=16384),
        # a burst of requests to the continuous-batching server
        dict(name="serve_128", mode="serve", graphs=128, n_max=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    mode = rng.choice(["wait", "wait", "enqueue", "enqueue", "once", "host", "reference", "batch",
                       "serve"])
    if mode == "batch":
        return dict(mode=mode, graphs=_log_int(rng, 8, 256), n_max=_log_int(rng, 512, 16384))
    if mode == "serve":
        return dict(mode=mode, graphs=_log_int(rng, 8, 160), n_max=_log_int(rng, 512, 4096))
    kind = rng.choice(["er", "mesh27", "mesh7", "rmat", "rmat", "sbm"])
    case = dict(mode=mode, graph=kind)
    if kind == "er":
        case.update(n=_log_int(rng, 256, 200000), degree=round(rng.uniform(16, 32), 2))
    elif kind == "mesh27":
        case.update(k=_log_int(rng, 8, 80))
    elif kind == "mesh7":
        case.update(k=_log_int(rng, 20, 150))
    elif kind == "sbm":
        case.update(n=_log_int(rng, 256, 32768), p_in=round(rng.uniform(0.05, 0.3), 4))
    else:
        by_degree = mode != "reference" and rng.random() < 0.6
        case.update(scale=rng.randint(10, 21 if by_degree else 18), ef=rng.randint(6, 16),
                    by_degree=by_degree)
    if mode == "reference":
        case.update(tile_cols=rng.choice([32, 128]))
    return case


# ---- inputs ---------------------------------------------------------------------------

def _vertices(case):
    if case["graph"] in ("mesh27", "mesh7"):
        return case["k"] ** 3
    if case["graph"] == "rmat":
        return 1 << case["scale"]
    return case["n"]


def _community_draws(n, p_in):
    per = n // 8
    inside = int(round(8 * per * (per - 1) / 2 * p_in))
    outside = int(round(n * (n - per) / 2 * 0.001))
    return inside, outside


def _mesh(kind, k, gen):
    """Edges of a k^3 grid in natural vertex order, listed in random order and direction.
    27-point: 98% of the neighbour pairs (a mesh with a few open faces); 7-point: every axis
    pair and 1% of the face diagonals (a grid with a few refined cells)."""
    idx = torch.arange(k ** 3, device="cuda")
    x, y, z = idx // (k * k), (idx // k) % k, idx % k
    us, vs = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                if (dx, dy, dz) <= (0, 0, 0):
                    continue
                axis = abs(dx) + abs(dy) + abs(dz)
                keep = 0.98 if kind == "mesh27" else (1.0 if axis == 1 else 0.01)
                if kind == "mesh7" and axis == 3:
                    continue
                ok = ((x + dx >= 0) & (x + dx < k) & (y + dy >= 0) & (y + dy < k)
                      & (z + dz >= 0) & (z + dz < k))
                if keep < 1.0:
                    ok &= torch.rand(k ** 3, generator=gen, device="cuda") < keep
                u = idx[ok]
                us.append(u)
                vs.append(u + dx * k * k + dy * k + dz)
    u, v = torch.cat(us), torch.cat(vs)
    p = torch.randperm(u.numel(), generator=gen, device="cuda")
    u, v = u[p], v[p]
    flip = torch.rand(u.numel(), generator=gen, device="cuda") < 0.5
    return torch.where(flip, v, u).int(), torch.where(flip, u, v).int()


def _edges(case, seed):
    """(src, dst, n): raw draws on the GPU; duplicates and self-loops are the engine's to drop."""
    n, kind = _vertices(case), case["graph"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if kind in ("mesh27", "mesh7"):
        return (*_mesh(kind, case["k"], gen), n)
    if kind == "rmat":
        return G.rmat_raw_torch(case["scale"], case["ef"], seed=seed)
    if kind == "er":
        m = int(round(n * case["degree"] / 2))
        e = torch.randint(0, n, (2, m), generator=gen, device="cuda", dtype=torch.int32)
        return e[0].contiguous(), e[1].contiguous(), n
    # eight equal communities, then pairs between any two vertices
    inside, outside = _community_draws(n, case["p_in"])
    per = n // 8
    base = torch.randint(0, 8, (inside,), generator=gen, device="cuda", dtype=torch.int32) * per
    e = torch.randint(0, per, (2, inside), generator=gen, device="cuda", dtype=torch.int32) + base
    o = torch.randint(0, n, (2, outside), generator=gen, device="cuda", dtype=torch.int32)
    p = torch.randperm(inside + outside, generator=gen, device="cuda")
    e = torch.cat([e, o], dim=1)[:, p]
    return e[0].contiguous(), e[1].contiguous(), n


def _mix(case, seed):
    """Graphs of mixed kinds (Erdos-Renyi, communities, R-MAT of scale 10..), concatenated."""
    plan = G.batch_mix_plan(case["graphs"], 256, case["n_max"], seed % (1 << 31))
    top = max(10, int(math.log2(case["n_max"])))
    graphs = []
    for i, (kind, n, segs) in enumerate(plan):
        if kind == "er":
            c = dict(graph="er", n=n, degree=2.0 * segs[0][-1] / n)
        elif kind == "sbm":
            c = dict(graph="sbm", n=n, p_in=0.05 + 0.25 * ((seed + 7 * i) % 16) / 16)
        else:
            c = dict(graph="rmat", scale=min(segs[0][1], top), ef=8)
        graphs.append(_edges(c, (seed * 1000003 + i) % (1 << 62)))
    offsets = np.zeros(len(graphs) + 1, np.int64)
    offsets[1:] = np.cumsum([g[0].numel() for g in graphs])
    nv = np.array([g[2] for g in graphs], np.int32)
    return torch.cat([g[0] for g in graphs]), torch.cat([g[1] for g in graphs]), offsets, nv


def _other(seed):
    return (int(seed) + 500009) % (1 << 31)


def prepare(case, seed):
    seed = int(seed) % (1 << 31)
    mode = case["mode"]
    s = dict(mode=mode, by_degree=bool(case.get("by_degree", False)))
    if mode == "batch":
        src, dst, offsets, nv = _mix(case, _other(seed))
        s["batch"] = A.Batch(src=src, dst=dst, offsets=offsets, num_vertices=nv)
        s["src"], s["dst"], s["offsets"], s["nv"] = _mix(case, seed)
        return s
    if mode == "serve":
        src, dst, offsets, nv = _mix(case, seed)
        hs, hd = src.cpu().numpy(), dst.cpu().numpy()
        s["requests"] = [(hs[a:b].copy(), hd[a:b].copy(), int(n))
                         for a, b, n in zip(offsets[:-1], offsets[1:], nv)]
        s["server"] = A.Server()
        return s
    src, dst, n = _edges(case, seed)
    s.update(src=src, dst=dst, n=n, tile_cols=int(case.get("tile_cols", 0)))
    if mode == "host":
        s["src"], s["dst"] = src.cpu().pin_memory(), dst.cpu().pin_memory()
    if mode in ("wait", "enqueue", "host"):
        s["graph"] = A.BitBSR(*_edges(case, _other(seed)), orient_degree=s["by_degree"])
        # the kept handle has counted its first graph
        s["graph"].count()
    if mode == "enqueue":
        s["count"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    return s


# ---- one step -------------------------------------------------------------------------

def run(s):
    mode = s["mode"]
    if mode in ("wait", "host"):
        s["graph"].rebuild(s["src"], s["dst"], s["n"], orient_degree=s["by_degree"])
        return {"count": s["graph"].count()}
    if mode == "enqueue":
        s["graph"].rebuild(s["src"], s["dst"], s["n"], orient_degree=s["by_degree"],
                           asynchronous=True)
        s["graph"].count_async(d_out=s["count"].data_ptr())
        return {"count": s["count"]}
    if mode == "once":
        g = A.BitBSR(s["src"], s["dst"], s["n"], orient_degree=s["by_degree"])
        count = g.count()
        g.free()
        return {"count": count}
    if mode == "reference":
        coo = A.CooMatrix(s["src"].clone(), s["dst"].clone(), s["n"])
        A.preprocess_for_triangle_counting(coo)
        wide = s["tile_cols"] == 128
        bcsr = A.BCSR_16x128_Device() if wide else A.BCSR_16x32_Device()
        if wide:
            A.convert_coo_to_bcsr_16x128_gpu(bcsr, coo)
            count = A.count_triangles_16x128_adaptive(bcsr)
        else:
            A.convert_coo_to_bcsr_16x32_gpu(bcsr, coo)
            count = A.count_triangles_16x32_adaptive(bcsr)
        tiles = int(bcsr.num_blocks)
        bcsr.free()
        return {"count": count, "rows": coo.num_rows, "edges": coo.num_entries, "tiles": tiles}
    if mode == "batch":
        s["batch"].rebuild(src=s["src"], dst=s["dst"], offsets=s["offsets"],
                           num_vertices=s["nv"])
        return {"counts": s["batch"].count().astype(np.int64)}
    server, requests = s["server"], s["requests"]
    place = {server.submit(u, v, n, borrow=True): i for i, (u, v, n) in enumerate(requests)}
    counts = np.zeros(len(requests), np.int64)
    left = len(requests)
    while left:
        for r in server.poll(wait_ms=1000):
            counts[place[r["id"]]] = r["count"] if r["status"] == 0 else -1
            left -= 1
    return {"counts": counts}


# ---- what a step cannot do without ------------------------------------------------------

def _draws(case):
    kind = case["graph"]
    if kind == "er":
        return int(round(case["n"] * case["degree"] / 2))
    if kind == "rmat":
        return case["ef"] << case["scale"]
    if kind == "sbm":
        return sum(_community_draws(case["n"], case["p_in"]))
    k = case["k"]
    if kind == "mesh7":
        return 3 * k * k * (k - 1) + int(0.01 * 6 * k * (k - 1) ** 2)
    return int(0.98 * ((3 * k - 2) ** 3 - k ** 3) / 2)


def work(case):
    """The edge list read once (8 bytes an edge) and the row pointers and the count written;
    the tiles, whose number depends on the draw, are left out.  Mixed batches: the mean over
    their kinds and log-uniform sizes."""
    if case["mode"] in ("batch", "serve"):
        lo, hi = math.log(256), math.log(max(case["n_max"], 257))
        mean_n = (math.exp(hi) - math.exp(lo)) / (hi - lo)
        mean_n2 = (math.exp(2 * hi) - math.exp(2 * lo)) / (2 * (hi - lo))
        scales = range(10, 17)
        top = max(10, int(math.log2(case["n_max"])))
        er, sbm = 10.0 * mean_n, 0.175 * mean_n2 / 16
        rmat = sum(8 << min(x, top) for x in scales) / len(scales)
        m = case["graphs"] * (er + sbm + rmat) / 3
        return {"bytes": 8.0 * m + 8.0 * case["graphs"], "flops": 0.0}
    m = _draws(case)
    return {"bytes": 8.0 * m + 4.0 * (_vertices(case) // 16 + 1) + 8.0, "flops": 0.0}


# ---- the same in plain 64-bit arithmetic --------------------------------------------------

def _lower(src, dst, n):
    """Unique (row, column) pairs with row > column, in row order."""
    r = torch.maximum(src, dst).long()
    c = torch.minimum(src, dst).long()
    key = torch.unique((r * n + c)[r != c])
    return key // n, key % n


def _triangles(r, c, n):
    """Triangles of a sorted unique lower triangle, or None where it takes too long: dense
    64-bit products for small or dense graphs, else every pair of a row looked up."""
    m = r.numel()
    deg = torch.bincount(r, minlength=n)
    pairs = int((deg * (deg - 1) // 2).sum())
    if n <= 4096 or (n <= 33000 and pairs > 100_000_000):
        low = torch.zeros((n, n), dtype=torch.float64, device=r.device)
        low[r, c] = 1.0
        total = 0
        for a in range(0, n, 4096):
            rows = low[a:a + 4096]
            total += int(((rows @ low.T) * rows).sum().item())
        return total
    if pairs > 2_000_000_000:
        return None
    key = r * n + c
    start = torch.cumsum(deg, 0) - deg
    before = torch.arange(m, device=r.device) - start[r]  # lower neighbours listed before it
    ends = torch.cumsum(before, 0)
    total, a = 0, 0
    while a < m:
        done = int(ends[a - 1]) if a else 0
        b = int(torch.searchsorted(ends, torch.tensor(done + 50_000_000, device=r.device)))
        b = min(max(b, a + 1), m)
        reps = before[a:b]
        e = torch.repeat_interleave(torch.arange(a, b, device=r.device), reps)
        first = torch.cumsum(reps, 0) - reps
        w = c[start[r[e]] + torch.arange(e.numel(), device=r.device)
              - torch.repeat_interleave(first, reps)]
        want = c[e] * n + w
        at = torch.searchsorted(key, want).clamp_(max=m - 1)
        total += int((key[at] == want).sum())
        a = b
    return total


def exact(case, seed):
    seed = int(seed) % (1 << 31)
    mode = case["mode"]
    if mode in ("batch", "serve"):
        src, dst, offsets, nv = _mix(case, seed)
        counts = []
        for a, b, n in zip(offsets[:-1], offsets[1:], nv):
            r, c = _lower(src[a:b], dst[a:b], int(n))
            counts.append(_triangles(r, c, int(n)))
        return None if None in counts else {"counts": np.array(counts, np.int64)}
    if case["graph"] == "rmat" and case["scale"] > 20:
        return None  # over two billion pairs
    src, dst, n = _edges(case, seed)
    r, c = _lower(src, dst, n)
    if mode != "reference":
        count = _triangles(r, c, n)
        return None if count is None else {"count": count}
    used = torch.zeros(n, dtype=torch.int64, device=r.device)
    used[r] = 1
    used[c] = 1
    new = torch.cumsum(used, 0) - 1
    rows = int(used.sum())
    r, c = new[r], new[c]
    width = case["tile_cols"]
    cells = torch.unique((r // 16) * (rows // width + 1) + c // width).numel()
    return {"count": _triangles(r, c, rows), "rows": rows, "edges": r.numel(), "tiles": cells}
