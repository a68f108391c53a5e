"""Performance cases of the graph engine, measured through its public Python API.

listed() names fixed cases, draw(rng) makes one more of the same ranges;
prepare / run / work / exact take a case's dict.  Graphs are seeded R-MAT
graphs (a, b, c = .57, .19, .19; duplicates and self-loops removed, u32
weights uniform in [1, 63]) of any vertex count, drawn here with torch, so a
case's inputs depend on its seed alone.
"""
import math

import numpy as np
import torch

import hytgraph_b200 as hyt
from hytgraph_b200 import capi

DEVICE = "cuda"
RMAT_AB, RMAT_ABC, RMAT_A = 0.76, 0.95, 0.57


def listed():
    return [
        # The engine's headline workload: R-MAT scale 24, edge factor 16, kept
        # on the GPU in hub order; ranks to an L1 change of 1e-6.
        {"name": "pagerank_s24", "op": "rank", "vertices": 1 << 24, "edge_factor": 16, "hub": True, "weights": "u32",
         "personalized": False, "host": False},
        # The other half of that workload: one SSSP source on the same graph.
        {"name": "sssp_s24", "op": "sssp", "vertices": 1 << 24, "edge_factor": 16, "hub": True, "weights": "u32",
         "host": False},
        # The smallest calls: a graph the size of the unit tests' (scale 12), built
        # in input order with default options, the result in a numpy array.  Time
        # goes to launches and the host path.
        {"name": "pagerank_small", "op": "rank", "vertices": 4099, "edge_factor": 16, "hub": False, "weights": "none",
         "personalized": False, "host": True},
        {"name": "sssp_small", "op": "sssp", "vertices": 4099, "edge_factor": 16, "hub": False, "weights": "f32",
         "host": True},
        # An ordinary query in input order: float weights, ragged vertex count.
        {"name": "sssp_f32_mid", "op": "sssp", "vertices": 500009, "edge_factor": 16, "hub": False, "weights": "f32",
         "host": True},
        # Eight queries sharing each pass over one graph (what the server packs).
        {"name": "sssp_pack8", "op": "sssp_multi", "vertices": 1 << 20, "edge_factor": 16, "hub": True,
         "weights": "u32", "queries": 8},
        {"name": "ppr_pack8", "op": "ppr_multi", "vertices": 1 << 21, "edge_factor": 16, "hub": True,
         "weights": "u32", "queries": 8},
        # A batch of uneven queries (60 % SSSP, else personalized PageRank) over
        # several resident graphs of scales 12 to 18, one call.
        {"name": "batch_48", "op": "batch", "graphs": 12, "low": 12, "high": 18, "queries": 48, "hub": True,
         "weights": "u32"},
        # A whole job from host arrays, as pagerank_gpu / sssp_gpu callers have it:
        # upload, graph build in hub order, PageRank, one SSSP, results on the host.
        {"name": "job_from_host", "op": "job", "vertices": 1 << 20, "edge_factor": 16, "hub": True, "weights": "u32"},
        # Hub sort and renumbering of a CSR on the GPU (scale 22).
        {"name": "reorder_s22", "op": "reorder", "vertices": 1 << 22, "edge_factor": 16, "weights": "u32"},
        # Contribution scheduling of every vertex: PageRank contributions of the
        # current ranks, SSSP contributions of a round and their schedule.
        {"name": "contrib_s22", "op": "contrib", "vertices": 1 << 22, "edge_factor": 16, "weights": "none"},
        # A graph whose edges stay in pinned host memory, under a device budget of
        # a sixth of them, in 33 to 64 partitions: PageRank and one SSSP over the link.
        {"name": "hybrid_s20", "op": "hybrid", "vertices": 1 << 20, "edge_factor": 16, "weights": "u32",
         "budget_mib": 32},
    ]


def _log_int(rng, low, high):
    """An integer of [low, high], uniform over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    op = rng.choice(["rank", "rank", "sssp", "sssp", "sssp_multi", "ppr_multi", "batch", "job", "reorder", "contrib",
                     "hybrid"])
    ef = rng.choice([4, 8, 16, 16, 16])
    kind = rng.choice(["u32", "u32", "f32", "none"])
    hub = rng.random() < 0.5
    if op in ("rank", "sssp"):
        c = {"op": op, "vertices": _log_int(rng, 1000, 1 << 24), "edge_factor": ef, "hub": hub, "weights": kind,
             "host": rng.random() < 0.5}
        if op == "rank":
            c["personalized"] = rng.random() < 0.5
        return c
    if op in ("sssp_multi", "ppr_multi"):
        return {"op": op, "vertices": _log_int(rng, 1 << 14, 1 << 21), "edge_factor": ef, "hub": hub,
                "weights": kind, "queries": rng.randint(2, 8)}
    if op == "batch":
        low = rng.randint(10, 13)
        return {"op": op, "graphs": rng.randint(3, 12), "low": low, "high": low + rng.randint(2, 5),
                "queries": rng.randint(8, 48), "hub": hub, "weights": kind}
    if op == "job":
        return {"op": op, "vertices": _log_int(rng, 1000, 1 << 20), "edge_factor": ef, "hub": hub, "weights": kind}
    if op == "reorder":
        return {"op": op, "vertices": _log_int(rng, 1000, 1 << 22), "edge_factor": ef, "weights": kind}
    if op == "contrib":
        return {"op": op, "vertices": _log_int(rng, 1000, 1 << 22), "edge_factor": ef, "weights": "none"}
    return {"op": op, "vertices": _log_int(rng, 1 << 16, 1 << 20), "edge_factor": rng.choice([8, 16]),
            "weights": rng.choice(["u32", "none"]), "budget_mib": rng.choice([8, 16, 32])}


# ---- inputs ----------------------------------------------------------------

def _edges(vertices, edge_factor, weights, seed):
    """(source, destination, weights) of an R-MAT graph, int32 on the GPU,
    ordered by (source, destination)."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    n = vertices * edge_factor
    bits = max(1, math.ceil(math.log2(vertices)))
    keys = []
    step = 1 << 26
    for first in range(0, n, step):
        m = min(step, n - first)
        src = torch.zeros(m, dtype=torch.int64, device=DEVICE)
        dst = torch.zeros(m, dtype=torch.int64, device=DEVICE)
        for _ in range(bits):
            u = torch.rand(m, generator=gen, device=DEVICE)
            src.mul_(2).add_(u >= RMAT_AB)
            dst.mul_(2).add_(((u >= RMAT_A) & (u < RMAT_AB)) | (u >= RMAT_ABC))
        # vertex counts that are no power of two: scale the ids into the range
        src = (src * vertices) >> bits
        dst = (dst * vertices) >> bits
        keys.append((src * vertices + dst)[src != dst])
        del src, dst, u
    key = torch.unique(torch.cat(keys))
    del keys
    src = (key // vertices).to(torch.int32)
    dst = (key % vertices).to(torch.int32)
    w = None
    if weights == "u32":
        w = torch.randint(1, 64, (key.numel(),), generator=gen, device=DEVICE, dtype=torch.int32)
    elif weights == "f32":
        w = torch.rand(key.numel(), generator=gen, device=DEVICE) * 10.0 + 0.05
    return src, dst, w


def _reorder_edges(case):
    """Edges kept for a reorder: below what duplicates leave at any seed
    (0.96 of the draws at scale 20, 0.7 at a thousand vertices)."""
    n = case["vertices"] * case["edge_factor"]
    return n * 9 // 10 if case["vertices"] >= 1 << 18 else n // 2


def _sources(src, seed, count):
    """`count` vertices with out-edges (host ints), spread over the ids."""
    u = torch.unique_consecutive(src)
    gen = torch.Generator().manual_seed(seed + 17)
    at = torch.randint(0, u.numel(), (count,), generator=gen)
    return [int(v) for v in u[at.to(DEVICE)].cpu()]


def _device_csr(case, seed):
    src, dst, w = _edges(case["vertices"], case["edge_factor"], case["weights"], seed)
    if case["op"] == "reorder":  # a fixed edge count, so that every seed's arrays have one shape
        keep = _reorder_edges(case)
        gen = torch.Generator(device=DEVICE).manual_seed(seed + 7)
        at = torch.randperm(src.numel(), generator=gen, device=DEVICE)[:keep].sort().values
        if at.numel() < keep:
            raise ValueError("the R-MAT draw left fewer edges than the case keeps")
        src, dst, w = src[at], dst[at], None if w is None else w[at]
    torch.cuda.synchronize()  # the library works on streams of its own
    csr = hyt.csr_from_edges(src, dst, case["vertices"], w, device=True)
    return src, dst, csr


def _flags(case):
    return capi.HYT_GRAPH_ALL | (capi.HYT_GRAPH_HUB_ORDER if case.get("hub") else 0)


def _batch_specs(case, seed):
    """Vertex counts and edge factors of the batch's graphs, and its queries
    as (graph, is_sssp); sources are picked per graph."""
    rng = np.random.default_rng(seed)
    # the mix of sizes is the case's own, the edges are the seed's
    fixed = np.random.default_rng(case["graphs"] * 1000 + case["low"] * 100 + case["high"])
    specs = [(int(2 ** fixed.uniform(case["low"], case["high"])), int(fixed.integers(8, 17)),
              int(rng.integers(1, 1 << 30))) for _ in range(case["graphs"])]
    queries = [(i % case["graphs"], bool(fixed.random() < 0.6)) for i in range(case["queries"])]
    return specs, queries


def _current_ranks(src, vertices, seed):
    """Ranks between two iterations of a solve: uneven, summing to about 1."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed + 3)
    deg = torch.bincount(src, minlength=vertices).float()
    r = (deg + 1.0) * (0.5 + torch.rand(vertices, generator=gen, device=DEVICE))
    return (r / r.double().sum()).float()


class _View:
    """Device memory of a library-owned array as a tensor's storage (the
    owner lives as long as the tensor does)."""

    def __init__(self, owner, ptr, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (count,), "typestr": typestr, "version": 3}


def _views(csr):
    """Offsets, ids and weights of a DeviceCSR as tensors."""
    c = csr.to_c()
    out = [torch.as_tensor(_View(csr, c.row_offsets, csr.num_vertices + 1, "<i8"), device=DEVICE),
           torch.as_tensor(_View(csr, c.column_indices, csr.num_edges, "<i4"), device=DEVICE)]
    if c.weights:
        out.append(torch.as_tensor(_View(csr, c.weights, csr.num_edges, "<i4"), device=DEVICE))
    return out


def prepare(case, seed):
    state = _state(case, seed)
    torch.cuda.synchronize()
    return state


def _state(case, seed):
    op = case["op"]
    if op == "batch":
        specs, queries = _batch_specs(case, seed)
        graphs, sources = [], []
        for v, ef, gseed in specs:
            src, _, csr = _device_csr(dict(case, vertices=v, edge_factor=ef), gseed)
            graphs.append(hyt.Graph(csr, flags=_flags(case)))
            sources.append(_sources(src, gseed, case["queries"]))
        qs = []
        for i, (g, is_sssp) in enumerate(queries):
            out = torch.empty(specs[g][0], dtype=torch.int32 if is_sssp else torch.float32, device=DEVICE)
            qs.append({"graph": g, "kind": "sssp" if is_sssp else "ppr", "source": sources[g][i], "restart": 0.15,
                       "tolerance": 1e-6, "out": out})
        return {"op": op, "batch": hyt.Batch(graphs), "queries": qs, "graphs": graphs}

    V = case["vertices"]
    src, dst, csr = _device_csr(case, seed)
    state = {"op": op}
    if op in ("rank", "sssp", "sssp_multi", "ppr_multi"):
        state["graph"] = hyt.Graph(csr, flags=_flags(case))
        state["personalized"] = case.get("personalized", False)
        state["sources"] = _sources(src, seed, case.get("queries", 1))
        dt = torch.float32 if op in ("rank", "ppr_multi") else torch.int32
        if op in ("rank", "sssp"):
            host = np.empty(V, np.float32 if op == "rank" else np.uint32)
            state["out"] = host if case["host"] else torch.empty(V, dtype=dt, device=DEVICE)
        else:
            state["out"] = torch.empty(case["queries"], V, dtype=dt, device=DEVICE)
    elif op == "job":
        state["csr"] = csr.download()
        state["flags"] = _flags(case)
        state["sources"] = _sources(src, seed, 1)
    elif op == "reorder":
        state["csr"] = csr
        state["order"] = torch.empty(V, dtype=torch.int32, device=DEVICE)
        state["scores"] = torch.empty(V, dtype=torch.float64, device=DEVICE)
    elif op == "contrib":
        state["graph"] = hyt.Graph(csr)
        state["ranks"] = _current_ranks(src, V, seed)
        gen = torch.Generator(device=DEVICE).manual_seed(seed + 5)
        # labels of a round: half unchanged, some reached for the first time
        cur = torch.rand(V, generator=gen, device=DEVICE) * 100.0
        u = torch.rand(V, generator=gen, device=DEVICE)
        cand = torch.where(u < 0.5, cur, cur * torch.rand(V, generator=gen, device=DEVICE))
        cur = torch.where(u > 0.9, torch.full_like(cur, math.inf), cur)
        state["current"], state["candidate"] = cur, cand
        state["items"] = torch.arange(V, dtype=torch.int64, device=DEVICE)
        state["out"] = torch.empty(V, dtype=torch.float64, device=DEVICE)
        state["gain"] = torch.empty(V, dtype=torch.float64, device=DEVICE)
        state["order"] = torch.empty(V, dtype=torch.int64, device=DEVICE)
    elif op == "hybrid":
        h = csr.download()
        order = torch.sort(dst, stable=True)
        in_off = torch.zeros(V + 1, dtype=torch.int64, device=DEVICE)
        in_off[1:] = torch.cumsum(torch.bincount(dst, minlength=V), 0)
        in_src = src[order.indices]
        state["graph"] = hyt.HybridGraph(h.row_offsets, h.column_indices, h.weights,
                                         in_off.cpu().numpy().view(np.uint64), in_src.cpu().numpy().view(np.uint32),
                                         budget_bytes=case["budget_mib"] << 20,
                                         partition_vertices=1 << ((V - 1).bit_length() - 6))
        state["sources"] = _sources(src, seed, 1)
        state["ranks"] = torch.empty(V, dtype=torch.float32, device=DEVICE)
        state["dist"] = torch.empty(V, dtype=torch.int32, device=DEVICE)
    return state


# ---- one pass --------------------------------------------------------------

def run(state):
    op = state["op"]
    if op == "rank":
        g = state["graph"]
        if state["personalized"]:
            return g.ppr(state["sources"][0], out=state["out"])[0]
        return g.pagerank(out=state["out"])[0]
    if op == "sssp":
        return state["graph"].sssp(state["sources"][0], out=state["out"])[0]
    if op == "sssp_multi":
        return state["graph"].sssp_multi(state["sources"], out=state["out"])[0]
    if op == "ppr_multi":
        return state["graph"].ppr_multi(state["sources"], out=state["out"])[0]
    if op == "batch":
        return state["batch"].run(state["queries"])[0]
    if op == "job":
        with hyt.Graph(state["csr"], flags=state["flags"]) as g:
            return g.pagerank()[0], g.sssp(state["sources"][0])[0]
    if op == "reorder":
        order, scores, hubs = hyt.hub_sort(state["csr"], order_out=state["order"], scores_out=state["scores"])
        return [order, scores, hubs] + _views(hyt.reorder(state["csr"], order, device=True))
    if op == "contrib":
        ranks = state["graph"].pagerank_contributions(state["ranks"], out=state["out"])
        gain = hyt.sssp_contributions(state["current"], state["candidate"], out=state["gain"])
        return ranks, gain, hyt.contribution_schedule(state["items"], gain, out=state["order"])[0]
    ranks = state["graph"].pagerank(out=state["ranks"])[0]
    return ranks, state["graph"].sssp(state["sources"][0], out=state["dist"])[0]


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    """Each input array read once and the result written once (edge counts as
    the draws before duplicates go, which is within a few percent)."""
    op = case["op"]
    wb = 0 if case["weights"] == "none" else 4
    if op == "batch":
        specs, queries = _batch_specs(case, 0)
        nbytes = flops = 0
        for g, is_sssp in queries:
            v, e = specs[g][0], specs[g][0] * specs[g][1]
            nbytes += 12 * v + (4 + (wb if is_sssp else 0)) * e
            flops += e if is_sssp else 2 * e
        return {"bytes": nbytes, "flops": flops}
    V = case["vertices"]
    E = V * case["edge_factor"]
    csr = 8 * V + 4 * E
    if op == "rank":
        return {"bytes": csr + 4 * V, "flops": 2 * E}
    if op == "sssp":
        return {"bytes": csr + wb * E + 4 * V, "flops": E}
    if op == "sssp_multi":
        return {"bytes": csr + wb * E + 4 * V * case["queries"], "flops": E * case["queries"]}
    if op == "ppr_multi":
        return {"bytes": csr + 4 * V * case["queries"], "flops": 2 * E * case["queries"]}
    if op == "job":
        return {"bytes": csr + wb * E + 8 * V, "flops": 3 * E}
    if op == "reorder":
        E = _reorder_edges(case)
        csr = 8 * V + 4 * E
        return {"bytes": 2 * (csr + wb * E) + 12 * V, "flops": 2 * E}
    if op == "contrib":
        return {"bytes": csr + (4 + 8) * V + (4 + 4 + 8) * V + (8 + 8 + 8) * V, "flops": 2 * E}
    return {"bytes": 2 * csr + wb * E + 8 * V, "flops": 3 * E}


# ---- the same results in 64 bits ----------------------------------------------

def _ranks_f64(src, dst, vertices, sources):
    """PageRank (sources None) or personalized PageRank of each source, by
    the engine's definition: Jacobi steps until the L1 change is at most 1e-6
    or 100 iterations; columns stop on their own."""
    deg = torch.bincount(src, minlength=vertices).double()
    inv = torch.where(deg > 0, 1.0 / deg.clamp(min=1.0), torch.zeros_like(deg))
    dead = deg == 0
    order = torch.sort(dst, stable=True).indices
    at = torch.zeros(vertices + 1, dtype=torch.int64, device=DEVICE)
    at[1:] = torch.cumsum(torch.bincount(dst, minlength=vertices), 0)
    m = torch.sparse_csr_tensor(at, src[order].long(), torch.ones(src.numel(), dtype=torch.float64, device=DEVICE),
                                size=(vertices, vertices), check_invariants=False)
    out = []
    d = float(np.float32(0.85)) if sources is None else float(np.float32(1.0) - np.float32(0.15))
    tol = float(np.float32(1e-6))
    for s in ([None] if sources is None else sources):
        x = torch.zeros(vertices, dtype=torch.float64, device=DEVICE)
        if s is None:
            x += 1.0 / vertices
        else:
            x[s] = 1.0
        for _ in range(100):
            lost = float(x[dead].sum())
            y = d * (m @ (x * inv).unsqueeze(1)).squeeze(1)
            if s is None:
                y += (1.0 - d) / vertices + d * lost / vertices
            else:
                y[s] += (1.0 - d) + d * lost
            change = float((y - x).abs().sum())
            x = y
            if change <= tol:
                break
        out.append(x)
    return out


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        specs, queries = _batch_specs(case, seed)
        out = [None] * len(queries)
        for g, (v, ef, gseed) in enumerate(specs):
            src, dst, _ = _edges(v, ef, case["weights"], gseed)
            sources = _sources(src, gseed, case["queries"])
            mine = [i for i, q in enumerate(queries) if q[0] == g and not q[1]]
            for i, x in zip(mine, _ranks_f64(src, dst, v, [sources[i] for i in mine])):
                out[i] = x
        return out
    if op in ("sssp", "sssp_multi", "reorder"):
        return None  # whole numbers, and scores defined by their rounding
    V = case["vertices"]
    src, dst, _ = _edges(V, case["edge_factor"], case["weights"], seed)
    if op == "rank":
        return _ranks_f64(src, dst, V, _sources(src, seed, 1) if case["personalized"] else None)[0]
    if op == "ppr_multi":
        return torch.stack(_ranks_f64(src, dst, V, _sources(src, seed, case["queries"])))
    if op == "contrib":
        x = _current_ranks(src, V, seed).double()
        deg = torch.bincount(src, minlength=V).double()
        y = torch.zeros_like(x).index_add_(0, dst, (x / deg.clamp(min=1.0))[src])
        d = float(np.float32(0.85))
        y = d * y + (1.0 - d) / V + d * float(x[deg == 0].sum()) / V
        return (y - x).abs(), None, None
    return _ranks_f64(src, dst, V, None)[0], None
