"""Performance cases: the calls that users of graphblox_gb300 make, over the sizes they make them at.

listed() names twelve, draw() gives more of the same ranges. prepare() makes a
case's inputs on the GPU from a seed with torch alone (graph families and value
distributions below) and the handles a program keeps (DeviceGraph, GraphBatch,
output buffers); run() is one pass through the public entry points; exact() is
the same result in 64 bits from plain torch.

Graph families
  rmat   R-MAT quadrants .57/.19/.19/.05: the social-network shape with hubs.
         A vertex count that is no power of two scales the ids down to it.
  crawl  Chung-Lu, out-degree power law with exponent 2.1, 70% of the edges
         inside 4,096-id windows: the web-crawl shape with local ids.
"""
import ctypes
import math

import numpy as np
import torch

import graphblox_gb300 as gbx

DEVICE = "cuda"
DAMPING = 0.85

M = 1 << 20


def listed():
    return [
        # A traversal of a graph of test size, as an interactive query makes it:
        # launches and host latency are all there is.
        {"name": "bfs_1k", "kind": "bfs", "family": "rmat", "vertices": 1000, "edges": 10_000, "directed": True, "roots": 1},
        # The benchmark graph (RMAT-22) traversed from random roots, levels and parents kept per root.
        {"name": "bfs_rmat22", "kind": "bfs", "family": "rmat", "vertices": 4 * M, "edges": 64 * M, "directed": True, "roots": 8},
        # The small configuration: RMAT-16, 20 iterations, each a few microseconds.
        {"name": "pagerank_rmat16", "kind": "pagerank", "family": "rmat", "vertices": 65_536, "edges": M, "directed": True, "iterations": 20},
        # The benchmark graph, 20 iterations: the gather of 65M contributions per iteration.
        {"name": "pagerank_rmat22", "kind": "pagerank", "family": "rmat", "vertices": 4 * M, "edges": 64 * M, "directed": True, "iterations": 20},
        # One y = A x over a crawl graph: the gather with local ids, each edge value read once.
        {"name": "spmv_crawl", "kind": "spmv", "family": "crawl", "vertices": 5_000_011, "edges": 150_000_000, "directed": True},
        # Weighted shortest paths on the benchmark graph, integer weights in [1, 255].
        {"name": "sssp_rmat22", "kind": "sssp", "family": "rmat", "vertices": 4 * M, "edges": 64 * M, "directed": True},
        # Components of the benchmark graph's symmetric form (128M edges).
        {"name": "cc_rmat22", "kind": "cc", "family": "rmat", "vertices": 4 * M, "edges": 64 * M, "directed": False},
        # Triangles of a degree-ordered undirected graph.
        {"name": "triangles_rmat20", "kind": "triangles", "family": "rmat", "vertices": M, "edges": 16 * M, "directed": False},
        # Graph load: edge list -> sorted, deduplicated CSR -> degree order -> CSR again, weights carried along.
        {"name": "preprocess_rmat22", "kind": "preprocess", "family": "rmat", "vertices": 4 * M, "edges": 64 * M, "weighted": True},
        # 64 personalised PageRank columns and their gradients for weights and teleport.
        {"name": "ppr_train_rmat20", "kind": "ppr", "family": "rmat", "vertices": M, "edges": 16 * M, "directed": True, "columns": 64},
        # 2,048 uneven graphs (2^8 to 2^15 vertices): BFS and 30 PageRank iterations of each, one launch per algorithm.
        {"name": "batch_2048", "kind": "batch", "family": "rmat", "graphs": 2048, "scale_lo": 8.0, "scale_hi": 15.0, "iterations": 30},
        # 256 BFS sources in one sweep (closeness and landmark sketches).
        {"name": "multisource_rmat20", "kind": "multisource", "family": "rmat", "vertices": M, "edges": 16 * M, "directed": True, "sources": 256},
    ]


def draw(rng):
    def log_uniform(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["bfs", "bfs", "pagerank", "pagerank", "spmv", "sssp", "cc", "triangles", "preprocess", "preprocess", "ppr", "batch",
                       "multisource"])
    if kind == "batch":
        lo = rng.uniform(6.0, 10.0)
        return {"kind": kind, "family": "rmat", "graphs": log_uniform(16, 1200), "scale_lo": round(lo, 2),
                "scale_hi": round(rng.uniform(lo + 1.0, 14.9), 2), "iterations": rng.randint(10, 30)}
    most = {"triangles": M, "ppr": M // 2, "multisource": M}.get(kind, 3 * M)
    vertices = log_uniform(700, most)
    case = {"kind": kind, "family": rng.choice(["rmat", "rmat", "crawl"]), "vertices": vertices,
            "edges": int(vertices * rng.uniform(4.0, 20.0))}
    if kind == "preprocess":
        return dict(case, weighted=rng.random() < 0.5)
    case["directed"] = kind == "ppr" or (kind not in ("cc", "triangles") and rng.random() < 0.75)
    if kind == "bfs":
        case["roots"] = rng.choice([1, 1, 2, 5, 8])
    elif kind == "pagerank":
        case["iterations"] = rng.randint(10, 30)
    elif kind == "ppr":
        case["columns"] = rng.choice([32, 64, 128])
    elif kind == "multisource":
        case["sources"] = rng.randint(20, 256)
    return case


# ---------------------------------------------------------------------------
# inputs


def _rng(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _rmat_bits(count, levels, g, level_of=None):
    """R-MAT (src, dst) ids of `levels` bits; level_of[e]: edge e stops after that many levels."""
    s = torch.zeros(count, dtype=torch.int64, device=DEVICE)
    d = torch.zeros(count, dtype=torch.int64, device=DEVICE)
    for i in range(levels):
        r = torch.rand(count, device=DEVICE, generator=g)
        sb = (r >= 0.76).long()
        db = (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).long()
        if level_of is None:
            s.mul_(2).add_(sb)
            d.mul_(2).add_(db)
        else:
            live = level_of > i
            s = torch.where(live, s * 2 + sb, s)
            d = torch.where(live, d * 2 + db, d)
    return s, d


def _crawl(V, E, g):
    a = 1.0 / 1.1  # weight (i + i0)^-a: out-degree exponent 2.1
    b = 1.0 - a
    lo, hi = 1e-3, float(V)
    for _ in range(60):  # i0: the largest expected degree is sqrt(E)
        i0 = math.sqrt(lo * hi)
        top = i0 ** -a * E * b / ((V + i0) ** b - i0 ** b)
        lo, hi = (i0, hi) if top > math.sqrt(E) else (lo, i0)

    def by_weight(u):
        x = (u * (V + i0) ** b + (1.0 - u) * i0 ** b) ** (1.0 / b) - i0
        return x.long().clamp_(0, V - 1)

    def uniform(n):
        return torch.rand(n, device=DEVICE, dtype=torch.float64, generator=g)

    s = by_weight(uniform(E))
    window = 4096
    base = s - s % window
    near = base + (uniform(E) * (V - base).clamp(max=window)).long()
    d = torch.where(torch.rand(E, device=DEVICE, generator=g) < 0.7, near, by_weight(uniform(E)))
    return s, d


def _edges(case, g):
    """The edge list as a file would hold it: repeated edges and self loops included."""
    V, E = case["vertices"], case["edges"]
    if case["family"] == "crawl":
        return _crawl(V, E, g)
    levels = max(1, math.ceil(math.log2(V)))
    s, d = _rmat_bits(E, levels, g)
    if V != 1 << levels:
        s, d = (s * V) >> levels, (d * V) >> levels
    return s, d


def _rows(sorted_rows, V):
    return torch.searchsorted(sorted_rows, torch.arange(V + 1, device=DEVICE)).int()


class _Csr:
    """Deduplicated CSR without self loops; the inverse CSR when directed; both edge orders' permutation."""

    def __init__(self, case, g, degree_order=False):
        V = self.V = case["vertices"]
        s, d = _edges(case, g)
        if not case["directed"]:
            s, d = torch.cat([s, d]), torch.cat([d, s])
        key = torch.unique((s * V + d)[s != d])
        s, d = key // V, key % V
        if degree_order:  # label 0 = the highest degree, as gbx_degree_reorder's lmode 1 gives it
            order = torch.sort(torch.bincount(s, minlength=V), stable=True).indices
            new = torch.empty(V, dtype=torch.int64, device=DEVICE)
            new[order] = torch.arange(V - 1, -1, -1, device=DEVICE)
            key = torch.sort(new[s] * V + new[d]).values
            s, d = key // V, key % V
        del key
        self.E = int(s.numel())
        self.offsets, self.dest = _rows(s, V), d.int()
        self.in_offsets = self.in_src = self.in_order = None
        if case["directed"]:
            back, self.in_order = torch.sort(d * V + s)
            self.in_offsets, self.in_src = _rows(back // V, V), (back % V).int()

    def device_graph(self, weight=None):
        in_weight = weight[self.in_order] if weight is not None and self.in_order is not None else None
        return gbx.DeviceGraph.from_offsets(self.V, self.offsets, self.dest, weight, self.in_offsets, self.in_src, in_weight)

    def pull(self):
        return (self.offsets, self.dest) if self.in_src is None else (self.in_offsets, self.in_src)


def _some_vertices(csr, n, g):
    """n random vertices that have out-edges, as a benchmark draws its roots."""
    live = torch.nonzero(torch.diff(csr.offsets)).flatten()
    return live[torch.randint(0, live.numel(), (n,), device=DEVICE, generator=g)].tolist()


def _int_weights(n, g):
    return torch.randint(1, 256, (n,), device=DEVICE, generator=g).float()


def _spmv_inputs(csr, g):
    values = 1.0 - torch.rand(csr.E, device=DEVICE, generator=g)  # (0, 1]
    x = torch.rand(csr.V, device=DEVICE, generator=g) * 2 - 1
    return values, x


def _ppr_inputs(csr, K, g):
    weights = torch.randn(csr.E, device=DEVICE, generator=g).exp_()
    seeds = torch.randint(0, csr.V, (32, K), device=DEVICE, generator=g)
    teleport = torch.zeros(csr.V, K, device=DEVICE).scatter_(0, seeds, 1.0)
    teleport /= teleport.sum(0)
    loss_weights = torch.randn(csr.V, K, device=DEVICE, generator=g)
    return weights, teleport, loss_weights


def _batch_sizes(case):
    """Vertices and generated edges per graph: scale and edge factor uniform, the same for every seed."""
    host = np.random.default_rng(case["graphs"])
    n = case["graphs"]
    sizes = np.floor(2.0 ** host.uniform(case["scale_lo"], case["scale_hi"], n)).astype(np.int64)
    return sizes, np.round(host.uniform(4.0, 32.0, n) * sizes).astype(np.int64)


def _packed(case, g):
    """Back-to-back CSR and in-edge CSR of uneven graphs."""
    sizes, counts = _batch_sizes(case)
    n = case["graphs"]
    base = torch.from_numpy(np.concatenate([[0], np.cumsum(sizes)])).to(DEVICE)
    of = torch.repeat_interleave(torch.arange(n, device=DEVICE), torch.from_numpy(counts).to(DEVICE))
    levels = torch.from_numpy(np.ceil(np.log2(sizes)).astype(np.int8)).to(DEVICE)
    s, d = _rmat_bits(of.numel(), int(levels.max()), g, levels[of])
    size = torch.from_numpy(sizes).to(DEVICE)[of]
    keep = (s < size) & (d < size)
    first = base[of[keep]]
    s, d = s[keep] + first, d[keep] + first
    V = int(base[-1])

    def csr(a, b):
        key = torch.sort(a * V + b).values
        rows = key // V
        local = key % V - base[torch.searchsorted(base, rows, right=True) - 1]
        return _rows(rows, V), local.int()

    (off, dest), (in_off, in_src) = csr(s, d), csr(d, s)
    return base, off, dest, in_off, in_src


def _host(t):
    return t.cpu().numpy().astype(np.uint32)


def prepare(case, seed):
    kind, g = case["kind"], _rng(seed)
    if kind == "batch":
        base, off, dest, in_off, in_src = _packed(case, g)
        V = int(base[-1])
        packed = gbx.PackedGraphs(_host(base), _host(off), _host(dest), _host(in_off), _host(in_src))
        return {"kind": kind, "batch": gbx.GraphBatch(packed), "sources": np.zeros(case["graphs"], np.uint32),
                "iterations": case["iterations"], "distances": torch.empty(V, dtype=torch.int32, device=DEVICE),
                "parents": torch.empty(V, dtype=torch.int32, device=DEVICE), "ranks": torch.empty(V, device=DEVICE)}
    V = case["vertices"]
    ints = lambda n: torch.empty(n, dtype=torch.int32, device=DEVICE)  # noqa: E731
    if kind == "preprocess":
        s, d = _edges(case, g)
        E = case["edges"]
        w = _int_weights(E, g) if case["weighted"] else None
        # room for every edge; what lies past the edges kept is never written
        room = lambda: torch.zeros(E, dtype=torch.int32, device=DEVICE)  # noqa: E731
        lists = lambda: {"deg": ints(V), "idx": ints(V), "src": room(), "dst": room(),  # noqa: E731
                         "w": torch.zeros(E, device=DEVICE) if case["weighted"] else None}
        return {"kind": kind, "V": V, "src": s.int(), "dst": d.int(), "w": w, "first": lists(), "second": lists(),
                "labels": ints(V), "inverse": ints(V), "identity": torch.arange(V, dtype=torch.int32, device=DEVICE)}
    csr = _Csr(case, g, degree_order=kind == "triangles")
    st = {"kind": kind}
    if kind == "bfs":
        st.update(roots=_some_vertices(csr, case["roots"], g), distances=ints(case["roots"] * V), parents=ints(case["roots"] * V))
    elif kind == "pagerank":
        st.update(iterations=case["iterations"], ranks=torch.empty(V, device=DEVICE))
    elif kind == "spmv":
        st["values"], st["x"] = _spmv_inputs(csr, g)
        st["y"] = torch.empty(V, device=DEVICE)
    elif kind == "sssp":
        st.update(root=_some_vertices(csr, 1, g)[0], distances=ints(V))
    elif kind == "cc":
        st["components"] = ints(V)
    elif kind == "ppr":
        st["weights"], st["teleport"], st["loss_weights"] = _ppr_inputs(csr, case["columns"], g)
        st.update(ranks=torch.empty(V, case["columns"], device=DEVICE), grad_weights=torch.zeros(case["edges"], device=DEVICE), edges=csr.E,
                  grad_teleport=torch.empty(V, case["columns"], device=DEVICE))
    elif kind == "multisource":
        st.update(sources=_some_vertices(csr, case["sources"], g), distances=ints(V * case["sources"]).view(V, case["sources"]))
    st["graph"] = csr.device_graph(_int_weights(csr.E, g) if kind == "sssp" else None)
    return st


# ---------------------------------------------------------------------------
# one pass


def _abi(name, *args):
    lib = gbx.load()
    status = getattr(lib, name)(*args)
    if status:
        raise gbx.GbxError(name, status, lib.gbx_last_error().decode())


def _p(t):
    return None if t is None else t.data_ptr()


def run(st):
    kind = st["kind"]
    if kind == "bfs":
        # which of a vertex's valid parents is written is a race, as in the
        # reference: the parents are computed and not compared
        V = st["graph"].num_vertices
        if len(st["roots"]) == 1:
            r = [gbx.breadth_first_search(st["graph"], st["roots"][0], distances=st["distances"], parents=st["parents"])]
        else:
            r = gbx.breadth_first_search_trials(st["graph"], st["roots"], distances=st["distances"], parents=st["parents"], out_stride=V)
        return {"distances": st["distances"], "processed": [x.processed_nodes for x in r]}
    if kind == "pagerank":
        return gbx.page_rank(st["graph"], st["iterations"], 0.0, ranks=st["ranks"]).pageRanks
    if kind == "spmv":
        return gbx.spmv(st["graph"], st["x"], values=st["values"], y=st["y"].zero_())
    if kind == "sssp":
        r = gbx.sssp(st["graph"], st["root"], distances=st["distances"])
        return {"distances": r.distances, "reached": r.reached, "edges_traversed": r.edges_traversed}
    if kind == "cc":
        return gbx.connected_components(st["graph"], components=st["components"])[0]
    if kind == "triangles":
        return gbx.triangle_count(st["graph"])
    if kind == "ppr":
        f = gbx.ppr_forward(st["graph"], st["weights"], st["teleport"], ranks=st["ranks"])
        b = gbx.ppr_adjoint(st["graph"], st["weights"], f.ranks, st["loss_weights"],
                            grad_weights=st["grad_weights"][:st["edges"]], grad_teleport=st["grad_teleport"])
        return {"ranks": f.ranks, "loss": b.loss, "grad_weights": st["grad_weights"], "grad_teleport": b.grad_teleport}
    if kind == "multisource":
        d, r = gbx.bfs_multisource(st["graph"], st["sources"], distances=st["distances"])
        return {"distances": d, "processed": r["processed_nodes"]}
    if kind == "batch":
        d, _, r = st["batch"].bfs(st["sources"], distances=st["distances"], parents=st["parents"])
        ranks, _ = st["batch"].page_rank(st["iterations"], 0.0, ranks=st["ranks"])
        return {"distances": d, "processed": r["processed_nodes"], "ranks": ranks}
    # preprocess: the steps of graph_csr_preprocessing with dedup and degree
    # order on edge arrays that are already on the GPU (the C interface takes
    # device pointers)
    V, a, b = st["V"], st["first"], st["second"]
    n, n2 = ctypes.c_uint32(), ctypes.c_uint32()
    _abi("gbx_csr_build", st["src"].numel(), _p(st["src"]), _p(st["dst"]), _p(st["w"]), 0, 1, 1, V, _p(a["deg"]), _p(a["idx"]),
         _p(a["src"]), _p(a["dst"]), _p(a["w"]), ctypes.byref(n), None)
    labels, inverse = st["labels"].copy_(st["identity"]), st["inverse"].copy_(st["identity"])
    _abi("gbx_degree_reorder", V, n.value, _p(a["src"]), _p(a["dst"]), 1, _p(labels), _p(inverse), None)
    _abi("gbx_csr_build", n.value, _p(a["src"]), _p(a["dst"]), _p(a["w"]), 0, 0, 1, V, _p(b["deg"]), _p(b["idx"]), _p(b["src"]),
         _p(b["dst"]), _p(b["w"]), ctypes.byref(n2), None)
    return {"labels": labels, "inverse": inverse, "edges": n2.value, **b}


# ---------------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    """Bytes: the graph arrays the call needs and its inputs read once, its outputs written once (an iterative
    solver reads its graph once per iteration). Edge counts are those generated, before removal of repeats."""
    kind = case["kind"]
    if kind == "batch":
        V, E = (int(x.sum()) for x in _batch_sizes(case))
        it = case["iterations"]
        return {"bytes": 4 * V + 4 * E + 8 * V + it * (4 * V + 4 * E + 8 * V), "flops": it * (E + 3 * V)}
    V, E = case["vertices"], case["edges"]
    if kind != "preprocess" and not case["directed"]:
        E *= 2
    graph = 4 * (V + 1) + 4 * E
    if kind == "bfs":
        return {"bytes": case["roots"] * (graph + 8 * V), "flops": 0}
    if kind == "pagerank":
        # per iteration: the in-edges, out-degrees and ranks in, ranks out
        return {"bytes": case["iterations"] * (graph + 12 * V), "flops": case["iterations"] * (E + 3 * V)}
    if kind == "spmv":
        return {"bytes": graph + 4 * E + 8 * V, "flops": 2 * E}
    if kind == "sssp":
        return {"bytes": graph + 4 * E + 4 * V, "flops": E}
    if kind == "cc":
        return {"bytes": graph + 4 * V, "flops": 0}
    if kind == "triangles":
        # each undirected edge once; at least one comparison per edge end
        return {"bytes": 4 * (V + 1) + 2 * E, "flops": 0}
    if kind == "ppr":
        # 1e-7 at damping .85 takes about 90 sweeps per solve for these
        # graphs; a sweep reads the edges with weights and the teleport block
        # and reads and writes the rank block, two operations per edge and column
        K, sweeps = case["columns"], 2 * 90
        return {"bytes": sweeps * (graph + 4 * E + 12 * V * K) + 8 * E, "flops": sweeps * 2 * E * K}
    if kind == "multisource":
        return {"bytes": graph + 4 * V * case["sources"], "flops": 0}
    w = 4 if case["weighted"] else 0
    # preprocess: read the edge list, write the CSR and both label arrays
    return {"bytes": 2 * E * (8 + w) + 16 * V, "flops": 0}


# ---------------------------------------------------------------------------
# the same in 64 bits


def _row_of_edge(offsets):
    n = torch.diff(offsets).long()
    return torch.repeat_interleave(torch.arange(n.numel(), device=DEVICE), n)


def _row_sums(terms, offsets):
    """Sums of consecutive runs of a 64-bit vector."""
    return torch.segment_reduce(terms, "sum", offsets=offsets.long(), initial=0.0)


def _exact_pagerank(V_of_row, out_degree, offsets, src, iterations):
    base, damp = 1.0 - float(np.float32(0.85)), float(np.float32(0.85))
    inverse = torch.where(out_degree > 0, 1.0 / out_degree.double().clamp(min=1), 0.0)
    r = torch.full((out_degree.numel(),), base, dtype=torch.float64, device=DEVICE)
    for _ in range(iterations):
        r = base + damp * _row_sums((r * inverse)[src], offsets)
    return r / V_of_row


def _exact_ppr(csr, case, g):
    w, T, W = (t.double() for t in _ppr_inputs(csr, case["columns"], g))
    V, K = csr.V, case["columns"]
    row, dest = _row_of_edge(csr.offsets), csr.dest.long()
    total = _row_sums(w, csr.offsets)
    P = w / total[row]
    # rows of `back` are destinations, of `forth` sources
    back = torch.sparse_csr_tensor(csr.in_offsets.long(), csr.in_src.long(), P[csr.in_order], size=(V, V))
    forth = torch.sparse_csr_tensor(csr.offsets.long(), dest, P, size=(V, V))
    R, Lam = T.clone(), W.clone()
    for _ in range(140):  # .85^140 = 1e-10
        R = (1 - DAMPING) * T + DAMPING * (back @ R)
        Lam = W + DAMPING * (forth @ Lam)
    inner = torch.empty(csr.E, dtype=torch.float64, device=DEVICE)
    step = max(1, (1 << 27) // K)
    for i in range(0, csr.E, step):
        j = slice(i, i + step)
        inner[j] = DAMPING * (Lam[dest[j]] * R[row[j]]).sum(1)
    mean = _row_sums(inner * P, csr.offsets)
    grad = torch.zeros(case["edges"], dtype=torch.float64, device=DEVICE)
    grad[:csr.E] = (inner - mean[row]) / total[row]
    return {"ranks": R, "loss": float((W * R).sum()), "grad_weights": grad, "grad_teleport": (1 - DAMPING) * Lam}


def exact(case, seed):
    kind, g = case["kind"], _rng(seed)
    if kind == "batch":
        base, off, _, in_off, in_src = _packed(case, g)
        of = torch.repeat_interleave(torch.arange(case["graphs"], device=DEVICE), torch.diff(base))
        first = base[of]
        src = in_src.long() + first[_row_of_edge(in_off)]
        ranks = _exact_pagerank(torch.diff(base)[of].double(), torch.diff(off), in_off, src, case["iterations"])
        return {"distances": None, "processed": None, "ranks": ranks}
    if kind not in ("pagerank", "spmv", "ppr"):
        return None
    csr = _Csr(case, g)
    if kind == "ppr":
        return _exact_ppr(csr, case, g)
    offsets, src = csr.pull()
    src = src.long()
    if kind == "pagerank":
        return _exact_pagerank(float(csr.V), torch.diff(csr.offsets), offsets, src, case["iterations"])
    values, x = _spmv_inputs(csr, g)
    return _row_sums(values.double() * x.double()[src], offsets)
