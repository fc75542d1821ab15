"""The framework's calls as its users make them, for measuring.

A user of the framework has an edge list (an R-MAT, grid or other graph),
builds a Graph from it once and runs toolkits on it: BFS, PageRank, CC, SSSP
and BC, one root at a time or 64 roots in one batch.  A state here is the
resident graph and the root or roots; a pass is one toolkit call (for the
"build" cases, the build itself from the records in hand).

Results stay on the device where the case says "out": "device", as for a
program that goes on with them there (to_host=False and
gg_result_device_ptr), or come back as the host arrays the Python calls return.
"""
import ctypes
import math
import random

import torch

import geminigraph_gb300 as gg

INF = 1e9          # SSSP's distance of a vertex that is not reached
ITERATIONS = 20    # PageRank iterations of every PageRank case
DEV = "cuda"


# ---------------------------------------------------------------- cases
def _case(do, shape, v, ef, weighted=False, symmetric=False, **more):
    """shape "rmat" / "uniform": v vertices, v * ef records; "grid": v = rows * cols, 4-neighbour, both directions."""
    return {"do": do, "shape": shape, "v": v, "ef": ef, "weighted": weighted, "symmetric": symmetric, **more}


def listed():
    return [
        # the smallest interactive query: one BFS of a graph that fits in cache, parents to the host
        {"name": "bfs-4k", **_case("bfs", "rmat", 1 << 12, 16, out="host")},
        # the headline workload: one BFS of the largest resident graph
        {"name": "bfs-rmat26", **_case("bfs", "rmat", 1 << 26, 16, out="device")},
        # PageRank in float, the plain configuration of the toolkit
        {"name": "pagerank-f32-rmat20", **_case("pagerank", "rmat", 1 << 20, 16, f32=True, out="device")},
        # PageRank in double, the drop-in toolkit's precision, on an odd number of vertices
        {"name": "pagerank-f64-7m", **_case("pagerank", "rmat", 7340033, 16, f32=False, out="device")},
        # PageRank on the largest resident graph
        {"name": "pagerank-f32-rmat26", **_case("pagerank", "rmat", 1 << 26, 16, f32=True, out="device")},
        # connected components of a symmetrised graph
        {"name": "cc-rmat24", **_case("cc", "rmat", 1 << 24, 16, symmetric=True, out="device")},
        # shortest paths over a power-law graph with weights in [0, 1)
        {"name": "sssp-rmat24", **_case("sssp", "rmat", 1 << 24, 16, weighted=True, out="device")},
        # shortest paths over a road-like graph: thousands of small frontiers, distances to the host
        {"name": "sssp-grid", **_case("sssp", "grid", 1500 * 701, 0, weighted=True, cols=701, out="host")},
        # betweenness of one root: forward and backward sweeps in double
        {"name": "bc-rmat22", **_case("bc", "rmat", 1 << 22, 16, out="device")},
        # 64 BFS queries answered in one batch, every level to the host
        {"name": "bfs-batch64-600k", **_case("bfs_batched", "rmat", 600011, 16, roots=64)},
        # 64 SSSP queries answered in one batch, every distance to the host
        {"name": "sssp-batch64-100k", **_case("sssp_batched", "rmat", 100003, 16, weighted=True, roots=64)},
        # the load: adjacency in both directions from weighted records in device memory
        {"name": "build-rmat23", **_case("build", "rmat", 1 << 23, 16, weighted=True)},
    ]


#: log2 of the vertices a drawn case of each kind has
RANGES = {"bfs": (10, 25.5), "pagerank": (10, 25), "cc": (10, 24), "sssp": (10, 24), "bc": (10, 23),
          "bfs_batched": (10, 20), "sssp_batched": (10, 17), "build": (10, 23.5)}


def draw(rng: random.Random):
    do = rng.choice(sorted(RANGES))
    lo, hi = RANGES[do]
    v = int(2 ** rng.uniform(lo, hi)) | 1
    ef = rng.choice([8, 12, 16, 16, 16, 24])
    if v * ef > 16 << int(hi):
        ef = 8
    shape = rng.choice(["rmat", "rmat", "rmat", "uniform"])
    more = {"weighted": do in ("sssp", "sssp_batched"), "symmetric": do == "cc"}
    if do in ("cc", "sssp") and v < 1 << 18 and rng.random() < 0.5:
        cols = rng.randint(24, int(math.sqrt(v)) + 8)
        return _case(do, "grid", max(2, v // cols) * cols, 0, cols=cols, out="host", **more)
    if do == "build":
        more = {"weighted": rng.random() < 0.5, "symmetric": rng.random() < 0.4}
        v = v if not more["symmetric"] else (v // 2) | 1
        return _case(do, shape, v, ef, **more)
    if do in ("bfs_batched", "sssp_batched"):
        return _case(do, shape, v, ef, roots=rng.choice([5, 33, 64]), **more)
    if do == "pagerank":
        more["f32"] = rng.random() < 0.5
    return _case(do, shape, v, ef, out="host" if v < 1 << 18 else "device", **more)


# ---------------------------------------------------------------- inputs
def _edges(case, seed):
    """(src, dst, weights or None) on the GPU and the generator, drawn from the seed alone."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)
    v = case["v"]
    if case["shape"] == "grid":
        ids = torch.arange(v, device=DEV, dtype=torch.int32)
        cols = case["cols"]
        right, down = ids[ids % cols != cols - 1], ids[: v - cols]
        a = torch.cat([right, right + 1, down, down + cols])
        b = torch.cat([right + 1, right, down + cols, down])
        order = torch.randperm(a.numel(), device=DEV, generator=gen)
        src, dst = a[order], b[order]
    else:
        e = v * case["ef"]
        src = torch.empty(e, device=DEV, dtype=torch.int32)
        dst = torch.empty(e, device=DEV, dtype=torch.int32)
        bits = max(1, (v - 1).bit_length())
        step = 1 << 26
        for at in range(0, e, step):
            n = min(step, e - at)
            if case["shape"] == "uniform":
                src[at:at + n] = torch.randint(0, v, (n,), device=DEV, generator=gen, dtype=torch.int32)
                dst[at:at + n] = torch.randint(0, v, (n,), device=DEV, generator=gen, dtype=torch.int32)
                continue
            s = torch.zeros(n, device=DEV, dtype=torch.int32)
            d = torch.zeros(n, device=DEV, dtype=torch.int32)
            for _ in range(bits):  # R-MAT quadrants .57 .19 .19 .05
                u = torch.rand(n, device=DEV, generator=gen)
                low = u >= 0.76
                s.mul_(2).add_(low)
                d.mul_(2).add_(((u >= 0.57) ^ low) | (u >= 0.95))
            if v & (v - 1):
                s.remainder_(v)
                d.remainder_(v)
            src[at:at + n] = s
            dst[at:at + n] = d
    w = torch.rand(src.numel(), device=DEV, generator=gen) if case["weighted"] else None
    return src, dst, w, gen


def _roots(case, src, gen, count):
    """`count` vertices with out-edges, uniformly drawn."""
    has = torch.zeros(case["v"], device=DEV, dtype=torch.bool)
    has[src] = True
    if case["symmetric"]:
        return [0] * count
    cand = has.nonzero().flatten()
    return cand[torch.randint(0, cand.numel(), (count,), device=DEV, generator=gen)].tolist()


def _records(src, dst, w):
    """The packed records of the framework's edge list: {u32 src, u32 dst[, f32 weight]}."""
    cols = [src, dst] + ([w.view(torch.int32)] if w is not None else [])
    return torch.stack(cols, 1).contiguous()


def _build(case, rec):
    h = ctypes.c_void_p()
    rc = gg.library().gg_graph_from_device_records(rec.data_ptr(), rec.numel() * 4, case["v"], int(case["weighted"]),
                                                   int(case["symmetric"]), torch.cuda.current_device(),
                                                   ctypes.byref(h))
    if rc:
        raise RuntimeError(gg.library().gg_last_error().decode())
    return gg.Graph(h)


def prepare(case, seed):
    src, dst, w, gen = _edges(case, seed)
    state = {"case": case}
    if case["do"] == "build":
        state["rec"] = _records(src, dst, w)
    else:
        if case["do"] not in ("pagerank", "cc"):
            roots = _roots(case, src, gen, case.get("roots", 1))
            state["roots"], state["root"] = roots, roots[0]
        rec = _records(src, dst, w)
        torch.cuda.synchronize()
        state["g"] = _build(case, rec)
        del rec
    del src, dst, w
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return state


# ---------------------------------------------------------------- passes
class _View:
    """A device array of the graph `owner`, for torch (which keeps it, and so the graph, alive)."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(owner, ptr, n, typestr):
    return torch.as_tensor(_View(owner, ptr, n, typestr), device=DEV)


def _device_result(g, which, n, typestr):
    return _view(g, gg.library().gg_result_device_ptr(g.h, which), n, typestr)


class _DeviceAdj(ctypes.Structure):
    """gg_device_adj of the C interface."""
    _fields_ = [("offsets", ctypes.c_void_p), ("neighbours", ctypes.c_void_p), ("weights", ctypes.c_void_p),
                ("degree", ctypes.c_void_p), ("vertices", ctypes.c_uint32), ("entries", ctypes.c_uint64),
                ("edges", ctypes.c_uint64), ("device", ctypes.c_int32)]


def _adjacency(g, incoming):
    a = _DeviceAdj()
    if gg.library().gg_graph_device_view(g.h, incoming, ctypes.byref(a)):
        raise RuntimeError(gg.library().gg_last_error().decode())
    got = {"offsets": _view(g, a.offsets, a.vertices + 1, "<i8"), "neighbours": _view(g, a.neighbours, a.entries, "<i4"),
           "degree": _view(g, a.degree, a.vertices, "<i4")}
    if a.weights:
        got["weights"] = _view(g, a.weights, a.entries, "<f4")
    return got


def run(state):
    case = state["case"]
    do, v = case["do"], case["v"]
    if do == "build":
        g = _build(case, state["rec"])
        return {"out": _adjacency(g, 0), "in": _adjacency(g, 1)}
    g = state["g"]
    if do == "bfs_batched":
        levels, _, reached, edges, _ = gg.bfs_batched(g, state["roots"])
        return {"levels": levels, "reached": reached, "edges": edges}
    if do == "sssp_batched":
        dist, reached, _ = gg.sssp_batched(g, state["roots"])
        return {"distances": dist, "reached": reached}
    host = case["out"] == "host"
    if do == "bfs":
        parent, _ = g.bfs(state["root"], to_host=host)
        return {"parent": parent if host else _device_result(g, 0, v, "<i4")}
    if do == "pagerank":
        ranks, deltas, _ = g.pagerank(ITERATIONS, to_host=host, f32=case["f32"])
        deltas = torch.as_tensor(deltas, dtype=torch.float32 if case["f32"] else torch.float64)  # as exact as the ranks
        return {"ranks": ranks if host else _device_result(g, 0, v, "<f4" if case["f32"] else "<f8"), "deltas": deltas}
    if do == "cc":
        label, _ = g.cc(to_host=host)
        return {"label": label if host else _device_result(g, 0, v, "<i4")}
    if do == "sssp":
        dist, _ = g.sssp(state["root"], to_host=host)
        return {"distance": dist if host else _device_result(g, 0, v, "<f4")}
    dep, inv, _ = g.bc(state["root"], to_host=host)
    return {"dependencies": dep if host else _device_result(g, 0, v, "<f8"),
            "inv_num_paths": inv if host else _device_result(g, 1, v, "<f8")}


# ---------------------------------------------------------------- work
def work(case):
    do, v = case["do"], case["v"]
    e = 4 * v - 2 * case["cols"] - 2 * (v // case["cols"]) if case["shape"] == "grid" else v * case["ef"]
    entries = e * (2 if case["symmetric"] else 1)
    side = 8 * (v + 1) + entries * (8 if case["weighted"] else 4)  # one direction of the adjacency
    if do == "build":
        return {"bytes": e * (12 if case["weighted"] else 8) + (side + 4 * v) * (1 if case["symmetric"] else 2),
                "flops": 0}
    if do == "pagerank":
        t = 4 if case["f32"] else 8
        return {"bytes": ITERATIONS * (side + 4 * v + 2 * t * v), "flops": ITERATIONS * (entries + 5 * v)}
    if do == "bc":
        return {"bytes": 2 * side + 16 * v, "flops": 2 * entries + 4 * v}
    if do in ("bfs_batched", "sssp_batched"):
        return {"bytes": side + 4 * v * case["roots"], "flops": 0 if do == "bfs_batched" else entries * case["roots"]}
    return {"bytes": side + 4 * v, "flops": entries if do == "sssp" else 0}


# ---------------------------------------------------------------- 64-bit results
def _exact_pagerank(case, src, dst):
    v = case["v"]
    key = dst.long().mul_(1 << 32).add_(src)
    del src, dst
    key = key.sort().values
    row = torch.searchsorted(key, torch.arange(v + 1, device=DEV) * (1 << 32))
    key &= 0xFFFFFFFF
    od = torch.zeros(v, device=DEV, dtype=torch.float64)
    for at in range(0, key.numel(), 1 << 27):
        od += torch.bincount(key[at:at + (1 << 27)], minlength=v)
    a = torch.sparse_csr_tensor(row, key, torch.ones(key.numel(), device=DEV, dtype=torch.float64), (v, v))
    share = torch.where(od > 0, od, 1.0)
    curr, deltas = 1.0 / share, [1.0]
    for i in range(ITERATIONS):
        new = 0.15 + 0.85 * (a @ curr)
        if i < ITERATIONS - 1:
            new /= share
            deltas.append(float(((new - curr).abs() * share).sum() / v))
        curr = new
    return {"ranks": curr, "deltas": torch.tensor(deltas, dtype=torch.float64)}


def _exact_sssp(v, src, dst, w, root):
    dist = torch.full((v,), INF, device=DEV, dtype=torch.float64)
    dist[root] = 0.0
    changed = torch.zeros(v, device=DEV, dtype=torch.bool)
    changed[root] = True
    while True:
        k = changed[src].nonzero().flatten()
        d, cand = dst[k], dist[src[k]] + w[k]
        k = (cand < dist[d]).nonzero().flatten()
        if k.numel() == 0:
            return dist
        d, cand = d[k], cand[k]
        cand, order = cand.sort()
        d, order = d[order].sort(stable=True)
        first = torch.ones_like(d, dtype=torch.bool)
        first[1:] = d[1:] != d[:-1]
        d, cand = d[first], cand[order[first]]
        changed.zero_()
        dist[d] = cand
        changed[d] = True


def _exact_bc(v, src, dst, root):
    level = torch.full((v,), -1, device=DEV, dtype=torch.int32)
    paths = torch.zeros(v, device=DEV, dtype=torch.float64)
    level[root] = 0
    paths[root] = 1.0
    steps = []
    while True:
        k = ((level[src] == len(steps)) & (level[dst] == -1)).nonzero().flatten()
        if k.numel() == 0:
            break
        s, d = src[k], dst[k]
        level[d] = len(steps) + 1
        paths.index_add_(0, d, paths[s])
        steps.append((s, d))
    inv = 1.0 / paths
    dep = torch.where(level >= 0, inv, torch.nan)
    for s, d in reversed(steps):
        dep.index_add_(0, s, dep[d])
    return {"dependencies": (dep - inv) / inv, "inv_num_paths": inv}


def _exact_side(v, major, minor, w):
    order = major.long().mul_(1 << 32).add_(minor).sort(stable=True).indices
    return w[order].double()


def exact(case, seed):
    do, v = case["do"], case["v"]
    if do in ("bfs", "cc", "bfs_batched") or (do == "build" and not case["weighted"]):
        return None
    src, dst, w, gen = _edges(case, seed)
    if do == "pagerank":
        return _exact_pagerank(case, src, dst)
    if do == "build":
        none = {"offsets": None, "neighbours": None, "degree": None}
        if case["symmetric"]:
            both = _exact_side(v, torch.cat([src, dst]), torch.cat([dst, src]), torch.cat([w, w]))
            return {"out": {**none, "weights": both}, "in": {**none, "weights": both}}
        return {"out": {**none, "weights": _exact_side(v, src, dst, w)},
                "in": {**none, "weights": _exact_side(v, dst, src, w)}}
    roots = _roots(case, src, gen, case.get("roots", 1))
    if do == "bc":
        return _exact_bc(v, src, dst, roots[0])
    w = w.double()
    if do == "sssp":
        return {"distance": _exact_sssp(v, src, dst, w, roots[0])}
    return {"distances": torch.stack([_exact_sssp(v, src, dst, w, r) for r in roots]), "reached": None}
