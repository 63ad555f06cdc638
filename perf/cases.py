"""The calls whose speed this framework is judged by.

Every case is one call through the public Python API, on inputs a program
has in hand: a CSR, an oriented graph, an edge list or a batch of graphs.
One engine serves all of them, as in a program that counts one graph after
another.  Graphs come from the seeded generators, so a seed gives the same
input everywhere.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import hetegeneous_parallel_programming_gb300 as tc

_engine = None


def engine() -> tc.Engine:
    """The engine a program keeps for all of its calls."""
    global _engine
    if _engine is None:
        _engine = tc.Engine(0)
        if not _engine.load_shipped_selector():
            raise RuntimeError("the shipped selector weights are missing")
    return _engine


def listed():
    return [
        # a small graph in an interactive loop: launches and host latency are all there is
        dict(name="tiny_er", op="count", graph="er", n=300, degree=5.0, edges=True),
        # the plain small workload: Erdos-Renyi n = 16384, degree 16
        dict(name="er_16k", op="count", graph="er", n=16384, degree=16.0),
        # a graph held in numpy arrays, its vertices' counts wanted back in numpy
        dict(name="host_chung_lu_50k", op="vertices_host", graph="chung_lu", n=50000, degree=24.0),
        # labelled intersections over a middling skewed graph
        dict(name="labelled_rmat_18", op="labelled", graph="rmat", scale=18, degree=32.0, a=0.57, b=0.19, c=0.19,
             classes=4),
        # a skewed graph of the size most users have, with every edge's count
        dict(name="rmat_20_edges", op="count", graph="rmat", scale=20, degree=32.0, a=0.57, b=0.19, c=0.19,
             edges=True),
        # triangles through every vertex, what clustering coefficients are made of
        dict(name="vertices_rmat_20", op="vertices", graph="rmat", scale=20, degree=32.0, a=0.57, b=0.19, c=0.19),
        # a graph its owner oriented already (the solver's own contract), flatter skew
        dict(name="dag_rmat_20", op="dag", graph="rmat", scale=20, degree=32.0, a=0.45, b=0.25, c=0.15),
        # an edge list with duplicates made into a clean symmetric CSR
        dict(name="build_rmat_21", op="build", graph="rmat", scale=21, degree=32.0, a=0.57, b=0.19, c=0.19),
        # a thousand small graphs of three families and uneven sizes in one call
        dict(name="batch_1024", op="batch", graphs=1024, n_min=64, n_max=16384, deg_min=4.0, deg_max=64.0),
        # power-law graph of odd size, learned selector
        dict(name="chung_lu_8m_learned", op="count", graph="chung_lu", n=8000009, degree=32.0, selector="learned"),
        # end to end from page-locked host memory
        dict(name="pinned_rmat_22", op="count_pinned", graph="rmat", scale=22, degree=32.0, a=0.57, b=0.19, c=0.19),
        # the headline workload: R-MAT scale 24, edge factor 16
        dict(name="rmat_24", op="count", graph="rmat", scale=24, degree=32.0, a=0.57, b=0.19, c=0.19),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_graph(rng, most):
    """A graph of at most `most` adjacency entries or so."""
    kind = rng.choice(("er", "rmat", "rmat", "chung_lu", "rgg"))
    degree = round(_log(rng, 4.0, 64.0), 2)
    entries = _log(rng, 2000.0, min(most, 4e6) if kind == "rgg" else most)
    n = max(32, int(entries / degree))
    degree = min(degree, n / 4.0)
    if kind == "rmat":
        return dict(graph=kind, scale=max(6, int(round(math.log2(n) - 0.5))), degree=degree,
                    a=round(rng.uniform(0.45, 0.6), 3), b=round(rng.uniform(0.1, 0.2), 3),
                    c=round(rng.uniform(0.1, 0.2), 3))
    return dict(graph=kind, n=n, degree=degree)


def draw(rng):
    op = rng.choice(("count", "count", "count", "count_host", "vertices_host", "count_pinned", "labelled", "vertices",
                     "dag", "build", "batch"))
    if op == "batch":
        n_min = int(_log(rng, 16, 256))
        n_max = int(_log(rng, n_min * 4, 16384))
        deg_min = round(rng.uniform(2.0, 8.0), 2)
        return dict(op=op, graphs=int(_log(rng, 3, 1024)), n_min=n_min, n_max=n_max, deg_min=deg_min,
                    deg_max=round(rng.uniform(deg_min + 2.0, 64.0), 2))
    case = dict(op=op, **_draw_graph(rng, {"count": 1.2e8, "count_pinned": 1.2e8, "count_host": 4e6,
                                               "vertices_host": 4e6}.get(op, 3e7)))
    if op == "labelled":
        case["classes"] = rng.randint(2, 16)
    if op == "count":
        case["edges"] = rng.random() < 0.5
    if op in ("count", "count_host"):
        case["selector"] = rng.choice(("fixed", "learned"))
    if op == "dag":
        lo = round(rng.uniform(0.0, 0.5), 3)
        case["from"], case["to"] = rng.choice(((0.0, 1.0), (lo, round(rng.uniform(lo + 0.1, 1.0), 3))))
    return case


# ---- inputs --------------------------------------------------------------------------

def _spec(case, seed):
    if case["graph"] == "rmat":
        return tc.GenSpec("rmat", scale=case["scale"], edge_factor=case["degree"] / 2, a=case["a"], b=case["b"],
                          c=case["c"], seed=seed)
    return tc.GenSpec(case["graph"], n=case["n"], avg_degree=case["degree"], gamma=2.1, seed=seed)


def _room(case):
    """Edges to make room for, whatever the seed (a geometric graph's number depends on it: twice the mean)."""
    if case["graph"] == "rgg":
        return int(case["n"] * case["degree"]) + 1024
    return max(_spec(case, 0).num_samples, 1)


def _edge_list(case, seed):
    """(n, src, dst) on the GPU: the generator's samples, duplicates and loops among them."""
    spec = _spec(case, seed)
    if case["graph"] == "rgg":  # drawn on the host
        n, s, d = tc.gen_edges_host(spec)
        return n, torch.from_numpy(s.copy()).cuda(), torch.from_numpy(d.copy()).cuda()
    k = spec.num_samples
    s = torch.empty(max(k, 1), dtype=torch.int32, device="cuda")
    d = torch.empty(max(k, 1), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    k = engine().gen_edges_device(spec, s.data_ptr(), d.data_ptr(), k)
    return spec.num_vertices, s[:k], d[:k]


def _csr(case, seed):
    """(n, rowptr, colidx) on the GPU."""
    n, s, d = _edge_list(case, seed)
    rowptr = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    colidx = torch.empty(max(2 * s.numel(), 1), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    nnz = engine().csr_from_edges_device(n, s.numel(), s.data_ptr(), d.data_ptr(), rowptr.data_ptr(),
                                         colidx.data_ptr(), colidx.numel())
    return n, rowptr, colidx[:nnz].clone()


def _orient(n, rowptr, colidx):
    """The degree-ordered DAG of a symmetric CSR in original ids."""
    deg = rowptr[1:] - rowptr[:-1]
    u = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
    v = colidx.long()
    keep = (deg[v] > deg[u]) | ((deg[v] == deg[u]) & (v > u))
    out = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    out[1:] = torch.cumsum(torch.bincount(u[keep], minlength=n), 0)
    return out, colidx[keep].contiguous()


def prepare(case, seed):
    engine()
    op = case["op"]
    st = dict(op=op, selector=case.get("selector", "fixed"))
    if op == "batch":
        vtx, rowptr, colidx = tc.gen_batch_host(case["graphs"], n_min=case["n_min"], n_max=case["n_max"],
                                                deg_min=case["deg_min"], deg_max=case["deg_max"], seed=seed)
        st.update(graphs=case["graphs"], vtx=torch.from_numpy(vtx).cuda(), rowptr=torch.from_numpy(rowptr).cuda(),
                  colidx=torch.from_numpy(colidx).cuda())
    elif op == "build":
        n, s, d = _edge_list(case, seed)
        st.update(n=n, src=s, dst=d, rowptr=torch.empty(n + 1, dtype=torch.int64, device="cuda"),
                  colidx=torch.zeros(2 * _room(case), dtype=torch.int32, device="cuda"))
    else:
        n, rowptr, colidx = _csr(case, seed)
        st.update(n=n)
        if op == "dag":
            rowptr, colidx = _orient(n, rowptr, colidx)
            st.update(first=int(case.get("from", 0.0) * n), last=int(math.ceil(case.get("to", 1.0) * n)))
        if op in ("count_host", "vertices_host"):
            rowptr, colidx = rowptr.cpu().numpy(), colidx.cpu().numpy()
        elif op == "count_pinned":
            rowptr, colidx = (torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for t in (rowptr, colidx))
        if case.get("edges"):
            st["per_edge"] = torch.zeros(_room(case), dtype=torch.int32, device="cuda")
        if op == "vertices":
            st["per_vertex"] = torch.zeros(n, dtype=torch.int64, device="cuda")
        if op == "labelled":
            gen = torch.Generator(device="cuda").manual_seed(seed)
            st["labels"] = torch.randint(case["classes"], (n,), dtype=torch.uint8, device="cuda", generator=gen)
        st.update(rowptr=rowptr, colidx=colidx)
    torch.cuda.synchronize()
    return st


# ---- one pass ------------------------------------------------------------------------

def run(st):
    eng, op = engine(), st["op"]
    if op == "batch":
        totals, stats = eng.batch_count_device(st["graphs"], st["vtx"].data_ptr(), st["rowptr"].data_ptr(),
                                               st["colidx"].data_ptr(), selector=st["selector"])
        return {"triangles": totals.view(np.int64), "edges": stats["m"]}
    if op == "build":
        nnz = eng.csr_from_edges_device(st["n"], st["src"].numel(), st["src"].data_ptr(), st["dst"].data_ptr(),
                                        st["rowptr"].data_ptr(), st["colidx"].data_ptr(), st["colidx"].numel())
        return {"entries": nnz, "rowptr": st["rowptr"], "colidx": st["colidx"]}
    if op == "count_host":
        total, _, stats = eng.count(st["rowptr"], st["colidx"], selector=st["selector"])
        return {"triangles": total, "edges": stats["m"]}
    if op == "vertices_host":
        total, per_vertex, stats = eng.count_vertices(st["rowptr"], st["colidx"])
        return {"triangles": total, "edges": stats["m"], "per_vertex": per_vertex.view(np.int64)}
    rowptr, colidx = st["rowptr"], st["colidx"]
    graph = (st["n"], colidx.numel(), rowptr.data_ptr(), colidx.data_ptr())
    if op == "count_pinned":
        total, stats = eng.count_host_ptr(*graph, selector=st["selector"])
        return {"triangles": total, "edges": stats["m"]}
    if op == "dag":
        total, stats = eng.count_dag_range_device(*graph, st["first"], st["last"], selector=st["selector"])
        return {"triangles": total, "edges": stats["m"]}
    if op == "labelled":
        total, stats = eng.count_labelled_device(*graph, st["labels"].data_ptr(), 1)
        return {"triangles": total, "edges": stats["m"]}
    if op == "vertices":
        total, stats = eng.count_vertices_device(*graph, st["per_vertex"].data_ptr())
        return {"triangles": total, "edges": stats["m"], "per_vertex": st["per_vertex"]}
    if op == "count":
        out = st.get("per_edge")
        total, stats = eng.count_device(*graph, selector=st["selector"],
                                        edge_counts_ptr=0 if out is None else out.data_ptr(),
                                        edge_capacity=0 if out is None else out.numel())
        got = {"triangles": total, "edges": stats["m"]}
        if out is not None:
            got["per_edge"] = out
        return got
    raise ValueError(op)


# ---- what a pass cannot do without ------------------------------------------------------

def work(case):
    """Bytes of the inputs read once and the outputs written once (counts are
    comparisons, not floating-point work; sizes before duplicates go)."""
    op = case["op"]
    if op == "batch":
        lo, hi = math.log(case["n_min"]), math.log(max(case["n_max"], case["n_min"] + 1))
        n = case["graphs"] * (math.exp(hi) - math.exp(lo)) / (hi - lo)  # mean of a log-uniform size
        return {"bytes": 8 * n + 4 * n * (case["deg_min"] + case["deg_max"]) / 2 + 16 * case["graphs"], "flops": 0}
    n = 1 << case["scale"] if case["graph"] == "rmat" else case["n"]
    entries = n * case["degree"]
    if op == "build":
        return {"bytes": 4 * entries + 8 * n + 4 * entries, "flops": 0}
    if op == "dag":
        return {"bytes": 8 * n + 4 * entries / 2 * (case.get("to", 1.0) - case.get("from", 0.0)), "flops": 0}
    out = {"vertices": 8 * n, "vertices_host": 8 * n, "labelled": n}.get(op, 0) + (4 * entries / 2 if case.get("edges") else 0)
    return {"bytes": 8 * n + 4 * entries + out + 8, "flops": 0}


def exact(case, seed):
    """Triangles and edges by a dense product, where the graph is small enough."""
    if case["op"] not in ("count", "count_host", "count_pinned"):
        return None
    n = 1 << case["scale"] if case["graph"] == "rmat" else case["n"]
    if n > 8192:
        return None
    n, s, d = _edge_list(case, seed)
    adj = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    adj[s.long(), d.long()] = 1.0
    adj = ((adj + adj.T) > 0).double()
    adj.fill_diagonal_(0.0)
    total = int(round(float(((adj @ adj) * adj).sum()))) // 6
    out = {"triangles": total, "edges": int(round(float(adj.sum()))) // 2}
    if case.get("edges"):
        out["per_edge"] = None
    return out
