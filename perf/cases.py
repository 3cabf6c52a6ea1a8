"""The work that users of this library have it do, as cases that can be timed.

A case is a dict of plain values. `prepare` makes a program's inputs and the handles it keeps (context, device
graph, batch) on the GPU, `run` is one pass through the public entry points, `work` says what a pass cannot do
without, and `exact` gives the computed numbers in 64 bits with plain torch.

The graphs are those of the library's own configurations: R-MAT(0.57, 0.19, 0.19, 0.05) with shuffled vertex ids
(vertex counts that are no powers of two among them), 4-neighbour grids, and batches of R-MAT graphs of uneven size.
"""
import importlib.util
import math
import sys
from pathlib import Path

import torch

ROOT = Path(__file__).resolve().parent.parent


def _package():
    """The package directory's name is no identifier, so it is loaded by path (as its own entry points do)."""
    name = "smdp_gb300"
    if name not in sys.modules:
        pkg = ROOT / "show-me-dynamic-parallelism_gb300"
        spec = importlib.util.spec_from_file_location(name, pkg / "__init__.py", submodule_search_locations=[str(pkg)])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


def listed():
    return [
        # The smallest configuration: one shortest-path query on a graph that fits in L2. Latency and launches.
        {"name": "sssp_rmat14", "kind": "sssp", "graph": "rmat", "V": 1 << 14, "ef": 16, "wmax": 100},
        # Shortest paths at scale, the largest single-source configuration.
        {"name": "sssp_rmat24", "kind": "sssp", "graph": "rmat", "V": 1 << 24, "ef": 16, "wmax": 255},
        # Shortest paths on a high-diameter graph (roads, grids): thousands of small frontiers.
        {"name": "sssp_grid4096", "kind": "sssp", "graph": "grid", "rows": 4096, "cols": 4096, "wmax": 1000},
        # Levels of a power-law graph: direction-optimizing traversal.
        {"name": "bfs_rmat22", "kind": "bfs", "graph": "rmat", "V": 1 << 22, "ef": 16},
        # Levels of a high-diameter graph with ragged sides.
        {"name": "bfs_grid1501x2003", "kind": "bfs", "graph": "grid", "rows": 1501, "cols": 2003},
        # One sparse product with a vector, at the size of the plain SpMV configuration.
        {"name": "spmv_rmat22", "kind": "spmv", "V": 1 << 22, "ef": 16},
        # The forward of a few right-hand sides (no multiple of 32) on a ragged mid-size matrix.
        {"name": "spmm_200003x20", "kind": "spmm", "V": 200_003, "ef": 16, "nrhs": 20},
        # The backward of 64 right-hand sides: both gradients, dX = A^T G and the one per nonzero.
        {"name": "spmv_bwd_rmat22x64", "kind": "spmv_bwd", "V": 1 << 22, "ef": 16, "nrhs": 64},
        # The headline: 20 PageRank sweeps on a resident graph.
        {"name": "pagerank_rmat22", "kind": "pagerank", "V": 1 << 22, "ef": 16, "iterations": 20},
        # One call with host arrays, as the command-line program makes it: upload, sweeps until no rank
        # moves, download. Ragged and mid-size.
        {"name": "pagerank_host_700001", "kind": "pagerank_host", "V": 700_001, "ef": 16, "iterations": 100,
         "epsilon": 1e-9},
        # Weighted PageRank and its gradient with respect to the edge weights, both to a tolerance.
        {"name": "prgrad_rmat20", "kind": "prgrad", "V": 1 << 20, "ef": 16},
        # Many graphs of uneven size in one launch: 8 shortest-path sources and 20 PageRank sweeps each.
        {"name": "batch_48", "kind": "batch", "graphs": 48, "vmax": 1 << 20, "nsrc": 8, "iterations": 20, "spec": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sssp", "sssp_grid", "bfs", "bfs_grid", "spmv", "spmm", "spmv_bwd", "pagerank", "pagerank_host",
                       "prgrad", "batch"])
    ef = rng.choice([8, 16, 32])
    if kind in ("sssp", "bfs"):
        c = {"kind": kind, "graph": "rmat", "V": _log_int(rng, 1 << 12, (1 << 27) // ef), "ef": ef}
    elif kind in ("sssp_grid", "bfs_grid"):
        c = {"kind": kind[:-5], "graph": "grid", "rows": _log_int(rng, 50, 3000), "cols": _log_int(rng, 50, 3000)}
    elif kind in ("spmm", "spmv_bwd"):
        c = {"kind": kind, "V": _log_int(rng, 1 << 11, (1 << 25) // ef), "ef": ef,
             "nrhs": rng.choice([1, 3, 8, 20, 32, 64, 96, 100, 128])}
    elif kind == "pagerank_host":
        c = {"kind": kind, "V": _log_int(rng, 1 << 11, (1 << 24) // ef), "ef": ef, "iterations": 100, "epsilon": 1e-9}
    elif kind == "prgrad":
        c = {"kind": kind, "V": _log_int(rng, 1 << 11, (1 << 24) // ef), "ef": ef}
    elif kind == "batch":
        c = {"kind": kind, "graphs": rng.randint(2, 40), "vmax": _log_int(rng, 1 << 12, 1 << 20),
             "nsrc": rng.choice([1, 3, 4, 8, 16]), "iterations": 20, "spec": rng.randint(1, 1 << 30)}
    else:
        c = {"kind": kind, "V": _log_int(rng, 1 << 12, (1 << 26) // ef), "ef": ef}
        if kind == "pagerank":
            c["iterations"] = rng.choice([1, 5, 20])
    if c["kind"] == "sssp":
        c["wmax"] = rng.choice([100, 255, 1000])
    return c


# ---- inputs ------------------------------------------------------------------------------------------------------

def _rmat(V, ef, gen):
    """Arc list (tail, head) of an R-MAT graph of V vertices and ef * V arcs, ids shuffled."""
    scale = max(1, math.ceil(math.log2(V)))
    n = V * ef
    src = torch.empty(n, dtype=torch.int32, device="cuda")
    dst = torch.empty(n, dtype=torch.int32, device="cuda")
    shuffle = torch.randperm(V, generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    for a in range(0, n, 1 << 26):
        m = min(1 << 26, n - a)
        s = torch.zeros(m, dtype=torch.int32, device="cuda")
        d = torch.zeros(m, dtype=torch.int32, device="cuda")
        for _ in range(scale):
            u = torch.rand(m, generator=gen, device="cuda")
            down = u >= 0.76
            right = ((u >= 0.57) & (u < 0.76)) | (u >= 0.95)
            s = (s << 1) | down.to(torch.int32)
            d = (d << 1) | right.to(torch.int32)
        if V != 1 << scale:  # squeeze [0, 2^scale) onto [0, V)
            s = (s.to(torch.int64) * V >> scale).to(torch.int32)
            d = (d.to(torch.int64) * V >> scale).to(torch.int32)
        src[a:a + m] = shuffle[s.long()]
        dst[a:a + m] = shuffle[d.long()]
    return src, dst


def _csr(V, row, col):
    """CSR of the arcs by `row`; each row keeps its arcs in drawn order."""
    row, idx = torch.sort(row, stable=True)
    col = col[idx]
    off = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(row.long(), minlength=V), 0)
    return off.to(torch.int32), col, row


def _grid(rows, cols):
    """CSR of the 4-neighbour grid: every adjacency as two arcs."""
    V = rows * cols
    v = torch.arange(V, dtype=torch.int64, device="cuda")
    r, c = v // cols, v % cols
    ok = torch.stack([r > 0, c > 0, c + 1 < cols, r + 1 < rows], 1)
    nb = torch.stack([v - cols, v - 1, v + 1, v + cols], 1)
    off = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(ok.sum(1), 0)
    return off.to(torch.int32), nb[ok].to(torch.int32)


def _gen(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _uniform(n, lo, hi, gen):
    return torch.rand(n, generator=gen, device="cuda") * (hi - lo) + lo


def _specs(case):
    """(V, edge factor) of each graph of a batch: vertex counts log-uniform, edge factors 8, 16 or 32; the
    same for every seed, so that a case stays one amount of work."""
    return _package().rmat_batch_specs(case["graphs"], seed=case["spec"], vmin=1024, vmax=case["vmax"])


def _inputs(case, seed):
    """The plain tensors of a case, from the seed alone."""
    gen = _gen(seed)
    kind = case["kind"]
    if kind in ("sssp", "bfs"):
        if case["graph"] == "rmat":
            off, col, row = _csr(case["V"], *_rmat(case["V"], case["ef"], gen))
            # A query's source has out-arcs: the tail of a random arc.
            source = int(row[torch.randint(len(row), (1,), generator=gen, device="cuda")])
        else:
            off, col = _grid(case["rows"], case["cols"])
            source = int(torch.randint(len(off) - 1, (1,), generator=gen, device="cuda"))
        w = None
        if kind == "sssp":
            w = torch.randint(1, case["wmax"] + 1, (len(col),), generator=gen, device="cuda", dtype=torch.int32)
        return {"off": off, "col": col, "w": w, "source": source}
    if kind in ("spmv", "spmm", "spmv_bwd"):
        V = case["V"]
        off, col, row = _csr(V, *_rmat(V, case["ef"], gen))
        d = {"off": off, "col": col, "row": row}
        if kind == "spmv":
            d["vals"] = 1.0 - torch.rand(len(col), generator=gen, device="cuda")  # uniform in (0, 1]
            d["x"] = _uniform(V, -1.0, 1.0, gen)
        else:
            d["vals"] = torch.randn(len(col), generator=gen, device="cuda").exp()  # lognormal(0, 1)
            d["X"] = torch.randn(V, case["nrhs"], generator=gen, device="cuda")
            if kind == "spmv_bwd":
                d["G"] = torch.randn(V, case["nrhs"], generator=gen, device="cuda")
        return d
    if kind in ("pagerank", "pagerank_host"):
        src, dst = _rmat(case["V"], case["ef"], gen)
        off, col, row = _csr(case["V"], dst, src)  # in-arcs
        outdeg = torch.bincount(src.long(), minlength=case["V"]).to(torch.int32)
        return {"off": off, "col": col, "row": row, "outdeg": outdeg}
    if kind == "prgrad":
        V = case["V"]
        off, col, row = _csr(V, *_rmat(V, case["ef"], gen))
        w = torch.randn(len(col), generator=gen, device="cuda").exp()
        dr = torch.zeros(V, device="cuda")
        dr[torch.randperm(V, generator=gen, device="cuda")[:max(1, V // 100)]] = 1.0  # loss: ranks of 1 % of the vertices
        return {"off": off, "col": col, "row": row, "w": w, "dr": dr}
    graphs, sources = [], []
    for V, ef in _specs(case):
        off, col, row = _csr(V, *_rmat(V, ef, gen))
        w = torch.randint(1, 101, (len(col),), generator=gen, device="cuda", dtype=torch.int32)
        graphs.append((V, off, col, row, w))
        sources.append(row[torch.randint(len(row), (case["nsrc"],), generator=gen, device="cuda")])
    return {"graphs": graphs, "sources": torch.stack(sources)}


PR = {"damping": 0.85, "total_rank": 1.0}
GRAD = {"iterations": 400, "epsilon": 3e-7, "adjoint_epsilon": 3e-7}


def prepare(case, seed):
    dpg = _package()
    kind = case["kind"]
    d = _inputs(case, seed)
    ctx = dpg.Context(0)
    s = {"case": case, "ctx": ctx}

    def graph(w=None):
        torch.cuda.synchronize()  # the context's stream reads what torch's stream made
        return dpg.Graph.from_device(ctx, len(d["off"]) - 1, len(d["col"]), d["off"].data_ptr(), d["col"].data_ptr(),
                                     None if w is None else w.data_ptr())

    if kind in ("sssp", "bfs"):
        s.update(graph=graph(d["w"]), source=d["source"],
                 out=torch.empty(len(d["off"]) - 1, dtype=torch.int32, device="cuda"))
    elif kind == "spmv":
        s.update(graph=graph(), vals=d["vals"], x=d["x"], y=torch.empty_like(d["x"]))
    elif kind == "spmm":
        s.update(graph=graph(), vals=d["vals"], X=d["X"], Y=torch.empty_like(d["X"]))
    elif kind == "spmv_bwd":
        s.update(graph=graph(), vals=d["vals"], X=d["X"], G=d["G"], dX=torch.empty_like(d["X"]),
                 dA=torch.empty_like(d["vals"]))
    elif kind == "pagerank":
        s.update(graph=graph(), outdeg=d["outdeg"], rank=torch.empty(case["V"], device="cuda"))
    elif kind == "pagerank_host":
        for name in ("off", "col", "outdeg"):
            s[name] = d[name].cpu().pin_memory().numpy()
    elif kind == "prgrad":
        s.update(graph=graph(), w=d["w"], dr=d["dr"], rank=torch.empty(case["V"], device="cuda"),
                 grad=torch.empty_like(d["w"]))
    else:
        csrs = [dpg.CSR(V, len(col), 0, off.cpu().numpy(), col.cpu().numpy(), w.cpu().numpy())
                for V, off, col, row, w in d["graphs"]]
        s["batch"] = dpg.Batch(ctx, csrs)
        s["sources"] = d["sources"].cpu().numpy()
        s["dist"] = torch.empty(s["batch"].V * case["nsrc"], dtype=torch.int32, device="cuda")
        s["rank"] = torch.empty(s["batch"].V, device="cuda")
    torch.cuda.synchronize()
    return s


def run(s):
    dpg = _package()
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "pagerank_host":
        return dpg.pagerank_host(ctx, s["off"], s["col"], s["outdeg"], iterations=case["iterations"],
                                 epsilon=case["epsilon"], **PR)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    if kind == "sssp":
        dpg.sssp_dev(ctx, s["graph"], s["source"], s["out"].data_ptr())
        return s["out"]
    if kind == "bfs":
        dpg.bfs_dev(ctx, s["graph"], s["source"], s["out"].data_ptr())
        return s["out"]
    if kind == "spmv":
        dpg.spmv_dev(ctx, s["graph"], s["vals"].data_ptr(), s["x"].data_ptr(), s["y"].data_ptr())
        return s["y"]
    if kind == "spmm":
        dpg.spmm_dev(ctx, s["graph"], s["vals"].data_ptr(), case["nrhs"], s["X"].data_ptr(), s["Y"].data_ptr())
        return s["Y"]
    if kind == "spmv_bwd":
        dpg.spmv_bwd_dev(ctx, s["graph"], s["vals"].data_ptr(), case["nrhs"], s["X"].data_ptr(), s["G"].data_ptr(),
                         s["dX"].data_ptr(), s["dA"].data_ptr())
        return {"dX": s["dX"], "dA": s["dA"]}
    if kind == "pagerank":
        dpg.pagerank_dev(ctx, s["graph"], s["outdeg"].data_ptr(), s["rank"].data_ptr(), iterations=case["iterations"],
                         **PR)
        return s["rank"]
    if kind == "prgrad":
        dpg.pagerank_grad_dev(ctx, s["graph"], s["w"].data_ptr(), s["dr"].data_ptr(), s["rank"].data_ptr(),
                              s["grad"].data_ptr(), **GRAD, **PR)
        return {"rank": s["rank"], "grad": s["grad"]}
    s["batch"].run(s["sources"], s["dist"].data_ptr(), s["rank"].data_ptr(), {}, dict(PR, iterations=case["iterations"]))
    return {"dist": s["dist"], "rank": s["rank"]}


def work(case):
    """Each input read once and each output written once (4-byte values), per sweep where there are sweeps."""
    kind = case["kind"]
    if kind == "batch":
        V = sum(v for v, _ in _specs(case))
        E = sum(v * ef for v, ef in _specs(case))
        k, it = case["nsrc"], case["iterations"]
        return {"bytes": 4 * V + 8 * E + 4 * k * V + it * (4 * V + 4 * E + 12 * V), "flops": k * E + it * (E + 3 * V)}
    if case.get("graph") == "grid":
        V = case["rows"] * case["cols"]
        E = 4 * V - 2 * case["rows"] - 2 * case["cols"]
    else:
        V, E = case["V"], case["V"] * case["ef"]
    if kind == "sssp":
        return {"bytes": 4 * (V + 1) + 8 * E + 4 * V, "flops": E}
    if kind == "bfs":
        return {"bytes": 4 * (V + 1) + 4 * E + 4 * V, "flops": E}
    if kind == "spmv":
        return {"bytes": 4 * (V + 1) + 8 * E + 8 * V, "flops": 2 * E}
    if kind == "spmm":
        return {"bytes": 4 * (V + 1) + 8 * E + 8 * case["nrhs"] * V, "flops": 2 * E * case["nrhs"]}
    if kind == "spmv_bwd":
        return {"bytes": 4 * (V + 1) + 12 * E + 12 * case["nrhs"] * V, "flops": 4 * E * case["nrhs"]}
    if kind == "pagerank":
        it = case["iterations"]
        return {"bytes": it * (4 * (V + 1) + 4 * E + 12 * V), "flops": it * (E + 3 * V)}
    if kind == "pagerank_host":  # the arrays cross the host link once; at least one sweep
        return {"bytes": 4 * (V + 1) + 4 * E + 8 * V, "flops": E + 3 * V}
    # prgrad: at least one forward and one adjoint sweep (offsets, columns, weights, vectors), and the gradient
    return {"bytes": 2 * (4 * (V + 1) + 8 * E + 12 * V) + 4 * E, "flops": 7 * E}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------

def _pull(V, row, col, x, vals=None):
    g = x[col.long()]
    if vals is not None:
        g = g * vals
    return torch.zeros(V, dtype=torch.float64, device="cuda").index_add_(0, row, g)


def _pagerank64(V, row, col, outdeg, iterations, epsilon=0.0):
    d, total = PR["damping"], PR["total_rank"]
    od = outdeg.double()
    live = od > 0
    r = torch.full((V,), total / V, dtype=torch.float64, device="cuda")
    for _ in range(iterations):
        contrib = torch.where(live, r / od.clamp(min=1.0), torch.zeros_like(r))
        new = (1 - d) * total / V + d * r[~live].sum() / V + d * _pull(V, row, col, contrib)
        done = epsilon > 0 and bool(((new - r).abs() <= epsilon).all())
        r = new
        if done:
            break
    return r


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sssp", "bfs"):
        return None  # whole numbers
    d = _inputs(case, seed)
    if kind == "batch":
        ranks = [_pagerank64(V, col.long(), row, off[1:] - off[:-1], case["iterations"])
                 for V, off, col, row, w in d["graphs"]]  # in-arcs: the arcs turned round
        return {"dist": None, "rank": torch.cat(ranks)}
    V = case["V"]
    row, col = d["row"].long(), d["col"]
    if kind in ("pagerank", "pagerank_host"):
        r = _pagerank64(V, row, col, d["outdeg"], case["iterations"], case.get("epsilon", 0.0))
        return r if kind == "pagerank" else r.cpu().numpy()
    if kind == "spmv":
        return _pull(V, row, col, d["x"].double(), d["vals"].double())
    if kind == "spmm":
        Y = torch.zeros(V, case["nrhs"], dtype=torch.float64, device="cuda")
        for a in range(0, len(col), 1 << 22):
            e = slice(a, a + (1 << 22))
            Y.index_add_(0, row[e], d["X"][col[e].long()].double() * d["vals"][e, None].double())
        return Y
    if kind == "spmv_bwd":
        dX = torch.zeros(V, case["nrhs"], dtype=torch.float64, device="cuda")
        dA = torch.empty(len(col), dtype=torch.float64, device="cuda")
        for a in range(0, len(col), 1 << 22):
            e = slice(a, a + (1 << 22))
            c, g = col[e].long(), d["G"][row[e]].double()
            dX.index_add_(0, c, g * d["vals"][e, None].double())
            dA[e] = (g * d["X"][c].double()).sum(1)
        return {"dX": dX, "dA": dA}
    # The weighted PageRank's fixed point and its adjoint's, far past the tolerance of the timed call.
    damping, w = PR["damping"], d["w"].double()
    W = torch.zeros(V, dtype=torch.float64, device="cuda").index_add_(0, row, w)
    live = W > 0
    inv = torch.where(live, 1.0 / W.clamp(min=1e-300), torch.zeros_like(W))
    r = torch.full((V,), PR["total_rank"] / V, dtype=torch.float64, device="cuda")
    for _ in range(160):
        r = ((1 - damping) * PR["total_rank"] / V + damping * r[~live].sum() / V
             + damping * _pull(V, col.long(), row, r * inv, w))
    seed64 = d["dr"].double()
    lam = seed64.clone()
    for _ in range(220):
        lam = seed64 + torch.where(live, damping * inv * _pull(V, row, col, lam, w), damping / V * lam.sum())
    q = inv * _pull(V, row, col, lam, w)
    grad = damping * (r * inv)[row] * (lam[col.long()] - q[row])
    return {"rank": r, "grad": grad}
