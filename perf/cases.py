"""Timed cases of the BFS engine: what a program asks of it, through its Python
binding (and, for the allocation-free call, the C ABI underneath).

A case is a graph family with its size, the entry point and its options.  The
graph and the roots come from the seed alone; the graph is on the device and
the handle exists before the pass, as in a program that searches one graph
from many roots.  One pass is one call of the entry point.

Level arrays, edge counts and reached counts are whole numbers with one right
value.  Any shortest-path parent is right, and which one a run records depends
on which edge is claimed first; so the case that records parents returns the
level of every vertex's parent, which is unique.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "bfs-gpu-sycl_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import bfs_gb300 as B  # noqa: E402

BLOCKS = (128, 256, 512)


def case(graph, entry, name=None, **kw):
    c = {"graph": graph, "entry": entry, "scale": 0, "edge_factor": 16, "symmetrize": True,
         "n": 0, "degree": 0, "width": 0, "height": 0, "rows_less": 0, "lb": "learned",
         "block": 256, "parents": False, "roots": 1, "graphs": 0, "scale_lo": 0, "scale_hi": 0,
         "ipt": 4, "cluster": 1}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a graph of a few thousand vertices, where the
        # launches and the levels' latencies are the whole time
        case("rmat", "device", "rmat12_learned", scale=12),
        # the reference's own program: one root, its default form (LLB, 256
        # threads), the level array back in host memory
        case("rmat", "host", "rmat19_llb_host", scale=19, lb="llb"),
        # a caller without device allocation, on a directed graph whose last
        # vertices have no row (the reference's dataset has rows < cols)
        case("rmat", "noalloc", "rmat18_rows_noalloc", scale=18, symmetrize=False, rows_less=1001),
        # a BFS tree: levels and parents
        case("rmat", "device", "rmat21_parents", scale=21, parents=True),
        # the default options on a large power-law graph
        case("rmat", "device", "rmat23_llb", scale=23, lb="llb"),
        # a loop over roots whose level arrays the program reads on the host
        case("rmat", "roots", "rmat23_roots8", scale=23, roots=8),
        # the largest: R-MAT scale 25, about a billion edges, learned schedule
        case("rmat", "device", "rmat25_learned", scale=25),
        # a flat-degree graph of an odd size
        case("er", "device", "er3000017_learned", n=3000017, degree=16),
        # road-like graphs: thousands of levels with few vertices each
        case("grid", "device", "grid4096_learned", width=4096, height=4096),
        case("grid", "device", "grid1023x1537_llb", width=1023, height=1537, lb="llb", block=128),
        # all-pairs style work: 64 roots share one pass
        case("rmat", "batch", "rmat22_batch64", scale=22, roots=64),
        # a dataset of many small graphs, one root each, in one launch
        case("rmat", "multi", "multi256", graphs=256, scale_lo=10, scale_hi=16, block=512, ipt=4,
             cluster=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rmat", "rmat", "rmat", "er", "grid", "noalloc", "batch", "multi"])
    lb = rng.choice(["learned", "learned", "llb", "glb", "slb"])
    kw = {"lb": lb, "block": rng.choice(BLOCKS)}
    entry = rng.choice(["device", "device", "host", "roots"])
    if entry == "roots":
        kw["roots"] = rng.randint(2, 9)
    if entry == "device":
        kw["parents"] = rng.random() < 0.25
    if kind == "multi":
        lo = rng.randint(8, 12)
        cluster = rng.choice([1, 2, 4, 8])
        return case("rmat", "multi", graphs=_log_int(rng, 16, 256), scale_lo=lo,
                    scale_hi=lo + rng.randint(1, 4), block=rng.choice([256, 512]),
                    ipt=rng.choice([2, 4]), cluster=cluster)
    if kind == "noalloc":
        n = _log_int(rng, 1000, 1 << 20)
        return case("er", "noalloc", n=n, degree=rng.randint(4, 24), rows_less=rng.randint(0, n // 8))
    if kind == "batch":
        roots = _log_int(rng, 2, 130)
        if rng.random() < 0.3:
            return case("grid", "batch", width=_log_int(rng, 40, 300), height=_log_int(rng, 40, 300),
                        roots=roots)
        if rng.random() < 0.5:
            return case("er", "batch", n=_log_int(rng, 5000, 2000000), degree=rng.randint(4, 24),
                        roots=roots)
        return case("rmat", "batch", scale=rng.randint(12, 21), edge_factor=rng.choice([8, 16, 32]),
                    roots=roots)
    if kind == "rmat":
        scale = rng.randint(11, 21 if entry == "roots" else 24)
        n = 1 << scale
        return case("rmat", entry, scale=scale, edge_factor=rng.choice([8, 16, 16, 31]),
                    symmetrize=rng.random() < 0.8,
                    rows_less=rng.randint(1, n // 16) if rng.random() < 0.2 else 0, **kw)
    if kind == "er":
        return case("er", entry, n=_log_int(rng, 2000, 6000000), degree=rng.randint(3, 30), **kw)
    side = 900 if entry == "roots" else 3000
    return case("grid", entry, width=_log_int(rng, 50, side), height=_log_int(rng, 50, side), **kw)


def _rmat_density(scale):
    """Share of an R-MAT stream's edges left after self-loops and duplicates."""
    return 1.0 - 0.19 * math.exp(-0.18 * (scale - 14.0)) if scale >= 10 else 0.6


def _size(c):
    """(vertices, directed edges) of a case's graph, the edges to a few percent."""
    if c["graph"] == "rmat":
        n = 1 << c["scale"]
        e = c["edge_factor"] * n * _rmat_density(c["scale"]) * (2 if c["symmetrize"] else 1)
    elif c["graph"] == "er":
        n = c["n"]
        e = c["degree"] * n
    else:
        n = c["width"] * c["height"]
        e = 4 * 0.95 * n
    return n, e


def work(c):
    if c["entry"] == "multi":
        scales = [s for s, _, _ in B.multi_batch_specs(c["graphs"], 1, (c["scale_lo"], c["scale_hi"]))]
        b = sum(4.0 * (2 * 16 * (1 << s) * _rmat_density(s)) + 8.0 * (1 << s) for s in scales)
        return {"bytes": b, "flops": 0}
    n, e = _size(c)
    out = 4.0 * n * (2 if c["parents"] else 1)  # levels (and parents) of one root
    graph = 4.0 * e + 4.0 * n                   # edges and offsets
    if c["entry"] == "batch":                   # one pass of the graph serves 64 roots
        return {"bytes": graph * math.ceil(c["roots"] / 64) + out * c["roots"], "flops": 0}
    return {"bytes": (graph + out) * c["roots"], "flops": 0}


def _csc(src, dst, n):
    """Device CSC (int32 tensors) of the symmetric closure of src -> dst,
    without self-loops and duplicates."""
    keep = src != dst
    src, dst = src[keep], dst[keep]
    key = torch.unique_consecutive(torch.sort(torch.cat([src * n + dst, dst * n + src]))[0])
    inds = (key % n).to(torch.int32)
    deg = torch.bincount(torch.div(key, n, rounding_mode="floor"), minlength=n)
    indptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(deg, 0, out=indptr[1:])
    return indptr.to(torch.int32), inds


def _er(c, gen):
    n = c["n"]
    m = n * c["degree"] // 2
    return _csc(torch.randint(0, n, (m,), generator=gen, device="cuda"),
                torch.randint(0, n, (m,), generator=gen, device="cuda"), n)


def _grid(c, gen):
    """4-neighbour grid, every edge deleted with probability 0.05."""
    w, h = c["width"], c["height"]
    v = torch.arange(w * h, device="cuda").view(h, w)
    pairs = [(v[:, :-1], v[:, 1:]), (v[:-1], v[1:])]
    src = torch.cat([a.reshape(-1) for a, _ in pairs])
    dst = torch.cat([b.reshape(-1) for _, b in pairs])
    keep = torch.rand(src.numel(), generator=gen, device="cuda") >= 0.05
    return _csc(src[keep], dst[keep], w * h)


class _DeviceArray:
    """A device array owned by a graph handle, as torch sees it."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False),
                                         "version": 2}


def prepare(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if c["entry"] == "multi":
        graphs, roots = B.multi_batch_graphs(B.multi_batch_specs(
            c["graphs"], 1 + 1000 * (seed % 100003), (c["scale_lo"], c["scale_hi"])))
        batch = B.MultiBatch(graphs)
        levels = torch.empty(batch.total_cols, dtype=torch.int32, device="cuda")
        return {"case": c, "batch": batch, "roots": roots, "levels": levels}
    s = {"case": c}
    if c["graph"] == "rmat":
        full = B.Graph.gen_rmat_device(c["scale"], c["edge_factor"], seed=1 + seed,
                                       symmetrize=c["symmetrize"])
        n, nnz = full.n_cols, full.nnz
        ip, ix = full.device_csc()
        indptr = torch.as_tensor(_DeviceArray(ip, n + 1), device="cuda")
    else:
        indptr, inds = (_er if c["graph"] == "er" else _grid)(c, gen)
        torch.cuda.synchronize()
        n, nnz = indptr.numel() - 1, inds.numel()
        ip, ix = indptr.data_ptr(), inds.data_ptr()
        full = None
        s["csc"] = (indptr, inds)
    rows = n - c["rows_less"]
    # roots: distinct vertices with out-edges, as the engine's sampler draws them
    able = torch.nonzero(indptr[1:rows + 1] != indptr[:rows]).view(-1)
    at = torch.randint(0, able.numel(), (8 * c["roots"],), generator=gen, device="cuda")
    drawn = [int(r) for r in able[at].tolist()]
    roots = list(dict.fromkeys(drawn))[:c["roots"]]
    s["roots"] = (roots + drawn)[:c["roots"]]
    del indptr, able, at
    s["n"], s["rows"], s["nnz"], s["ptrs"] = n, rows, nnz, (ip, ix)
    s["full"] = full
    if c["entry"] == "noalloc":
        f = B.lib().bfs_run_device_noalloc
        vp, u32 = ctypes.c_void_p, ctypes.c_uint32
        f.argtypes = [vp, vp, u32, u32, ctypes.c_uint64, u32, vp, ctypes.POINTER(ctypes.c_uint64), vp]
        f.restype = ctypes.c_int
        s["call"] = f
        s["levels"] = torch.empty(n, dtype=torch.int32, device="cuda")
        return s
    if full is None or c["rows_less"]:
        s["handle"] = B.Graph.wrap_device(ip, ix, rows, n, nnz)
    else:
        s["handle"] = full
    if c["entry"] == "batch":
        s["levels"] = torch.empty(c["roots"], n, dtype=torch.int32, device="cuda")
        return s
    if c["lb"] == "learned":
        s["handle"].sched_attach(np.fromfile(os.path.join(PKG, "sched_weights.f32"), np.float32))
    s["opts"] = B.options(c["lb"], c["block"])
    if c["entry"] == "roots":
        s["levels"] = [torch.empty(n, dtype=torch.int32, pin_memory=True) for _ in s["roots"]]
        s["out"] = [t.data_ptr() for t in s["levels"]]
    else:
        s["levels"] = torch.empty(n, dtype=torch.int32, pin_memory=c["entry"] == "host",
                                  device="cpu" if c["entry"] == "host" else "cuda")
        if c["parents"]:
            s["parents"] = torch.empty(n, dtype=torch.int32, device="cuda")
    return s


def run(s):
    c = s["case"]
    entry, levels = c["entry"], s["levels"]
    if entry == "multi":
        edges, _ = s["batch"].run(s["roots"], levels.data_ptr(), c["block"], c["ipt"], c["cluster"])
        return {"levels": levels, "edges": edges.view(np.int64)}
    if entry == "noalloc":
        edges = ctypes.c_uint64(0)
        B.check(s["call"](*s["ptrs"], s["rows"], s["n"], s["nnz"], s["roots"][0],
                          levels.data_ptr(), ctypes.byref(edges), None))
        return {"levels": levels, "edges": edges.value}
    g = s["handle"]
    if entry == "batch":
        edges, _ = g.run_batch(s["roots"], levels.data_ptr())
        return {"levels": levels, "edges": edges.view(np.int64)}
    if entry == "roots":
        sts = g.run_roots(s["roots"], s["out"], opts=s["opts"])
        return {"levels": levels, "edges": [int(t.edges_count) for t in sts]}
    if entry == "host":
        st = g.run_into(s["roots"][0], levels.data_ptr(), opts=s["opts"])
    else:
        st = g.run_device(s["roots"][0], levels.data_ptr(),
                          s["parents"].data_ptr() if c["parents"] else None, opts=s["opts"])
    out = {"levels": levels, "edges": int(st.edges_count), "reached": int(st.reached)}
    if c["parents"]:
        out["parent_levels"] = torch.index_select(levels, 0, s["parents"].clamp_(min=0))
    return out


def exact(c, seed):
    """Every output is a whole number: there is no rounding to measure."""
    return None
