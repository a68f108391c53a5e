"""SSSP rounds that run as pull sweeps, at the row lengths where the sweep's
groups of lanes, wide rows and chunks of long rows change, for every form of the
weights: packed up to exactly 32 bits, one bit more, saturating, float and none.

A source reaches a layer of vertices whose out-edges are most of the graph's, so
the round after the first is a sweep; vertices that no source reaches feed the
same rows, so that a sweep (which reads every in-edge of a row) relaxes more
edges than any schedule of pushes."""
import heapq

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# group sizes end at 2, 4, 8, 16, 32 and 64 in-edges; tiles at 512, chunks at
# 1024 on graphs of this size
DEGREES = [0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513,
           1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097]
INF = 0xFFFFFFFF


def _graph(hyt, order, weights, seed, high=None, chain=0):
    """0: the source.  1 .. M: the first layer.  Then the rows, of all DEGREES
    and many of a few in-edges (two in-edges in three from the first layer, the
    others from vertices that nothing reaches), each with an edge to the next row;
    chain: that many vertices between the source and the first layer, edges of
    the largest weight."""
    rng = np.random.default_rng(seed)
    M = 3000
    rows = np.array(DEGREES + list(rng.integers(0, 40, 700)))
    rows = np.sort(rows)[::-1] if order == "sorted" else rng.permutation(rows)
    first = 1 + M
    V = first + rows.size + 3000 + chain  # 3000 that nothing reaches, then the chain
    lost, link = first + rows.size, V - chain
    src, dst = [], []
    for i, d in enumerate(rows):
        pool = np.concatenate([np.arange(1, first), np.arange(lost, link)])
        pick = rng.choice(pool, d, replace=False) if d <= pool.size else pool
        src.append(pick)
        dst.append(np.full(pick.size, first + i))
    src += [np.arange(first, first + rows.size - 1)]
    dst += [np.arange(first + 1, first + rows.size)]
    hops = [0] + list(range(link, V))
    src += [np.array(hops[:-1], np.int64), np.full(M, hops[-1])]
    dst += [np.array(hops[1:], np.int64), np.arange(1, first)]
    src, dst = np.concatenate(src), np.concatenate(dst)
    o = np.argsort(src, kind="stable")
    src, dst = src[o], dst[o].astype(np.uint32)
    off = np.zeros(V + 1, np.uint64)
    np.cumsum(np.bincount(src, minlength=V), out=off[1:])
    w = None
    if weights == "f32":
        w = (rng.random(src.size) * 10 + 0.05).astype(np.float32)
    elif weights == "u32":
        w = rng.integers(1, high, src.size, endpoint=True).astype(np.uint32)
        w[0] = high
        w[np.isin(src, hops[:-1])] = high
    return hyt.CSR(off, dst, w)


def _dijkstra(g, source):
    """Labels in 64 bits (floats: in the order of a path's edges, in 32)."""
    off, cols, w = g.row_offsets.astype(np.int64), g.column_indices, g.weights
    f32 = w is not None and w.dtype == np.float32
    dist = {source: np.float32(0) if f32 else 0}
    heap = [(dist[source], source)]
    while heap:
        d, u = heapq.heappop(heap)
        if d != dist[u]:
            continue
        for e in range(off[u], off[u + 1]):
            v = int(cols[e])
            n = np.float32(d + w[e]) if f32 else d + (1 if w is None else int(w[e]))
            if v not in dist or n < dist[v]:
                dist[v] = n
                heapq.heappush(heap, (n, v))
    if f32:
        out = np.full(g.num_vertices, np.inf, np.float32)
        for v, d in dist.items():
            out[v] = d
        return out.view(np.uint32)
    out = np.full(g.num_vertices, INF, np.uint32)
    for v, d in dist.items():
        out[v] = min(d, INF - 1)  # saturated, not unreached
    return out


CASES = [("none", None), ("u32", 63), ("u32", (1 << 19) - 1), ("u32", 1 << 19), ("u32", (1 << 19) + 1), ("u32", 1 << 31),
         ("u32", INF), ("f32", None)]


@pytest.mark.parametrize("order", ["sorted", "mixed"])
@pytest.mark.parametrize("weights,high", CASES)
@pytest.mark.parametrize("hub", [False, True])
def test_sweeps_match_dijkstra(hyt, gpu, order, weights, high, hub):
    g = _graph(hyt, order, weights, 11, high)
    assert 1 << 12 < g.num_vertices <= 1 << 13  # 13 bits of an id: weights of 19 bits pack, of 20 do not
    want = _dijkstra(g, 0)
    f = hyt.capi.HYT_GRAPH_HUB_ORDER if hub else 0
    with hyt.Graph(g, flags=hyt.capi.HYT_GRAPH_ALL | f) as a, hyt.Graph(g, flags=hyt.capi.HYT_GRAPH_PUSH | f) as p:
        got, st = a.sssp(0)
        assert np.array_equal(got, want)
        pushed, sp = p.sssp(0)
        assert np.array_equal(pushed, want)
        assert st["edges_processed"] > sp["edges_processed"]  # sweeps ran
        looped, _ = a.sssp(0, flags=hyt.capi.HYT_RUN_NO_GRAPH)
        assert np.array_equal(looped, want)
        # eight lanes, the first layer's vertices and the source among them
        sources = [0, 1, 2, 0, 3001, g.num_vertices - 1, 1500, 3000]
        many, sm = a.sssp_multi(sources)
        assert np.array_equal(many[0], want) and np.array_equal(many[3], want)
        for l in (1, 4, 7):
            assert np.array_equal(many[l], _dijkstra(g, sources[l])), l
        assert sm["edges_processed"] > p.sssp_multi(sources)[1]["edges_processed"]


@pytest.mark.parametrize("vertices_bits,high", [(13, (1 << 19) - 1), (13, 1 << 19)])
def test_labels_up_to_the_packed_infinity(hyt, gpu, vertices_bits, high):
    """A chain of the largest weight fills the id bits, so that labels come as
    near to the packed sweep's infinity as a path can bring them; sweeps follow."""
    short = _graph(hyt, "mixed", "u32", 13, high).num_vertices
    g = _graph(hyt, "mixed", "u32", 13, high, chain=(1 << vertices_bits) - short)
    assert g.num_vertices == 1 << vertices_bits
    want = _dijkstra(g, 0)
    with hyt.Graph(g) as a, hyt.Graph(g, flags=hyt.capi.HYT_GRAPH_PUSH) as p:
        got, st = a.sssp(0)
        assert np.array_equal(got, want)
        assert st["edges_processed"] > p.sssp(0)[1]["edges_processed"]
        assert np.array_equal(a.sssp_multi([0, 5])[0][0], want)


@pytest.mark.parametrize("edges", [9_000_000, 68_000_000])  # chunks of 2048 and of 4096 edges
@pytest.mark.parametrize("weights,high", [("none", None), ("u32", (1 << 12) - 1), ("u32", 1 << 12), ("f32", None)])
def test_chunk_limits_on_larger_graphs(hyt, gpu, edges, weights, high):
    """Long rows at the limits of the longer chunks, against a solve that only
    pushes.  Unweighted pushes relax every edge within reach once, which sweeps
    (whole rows, settled ones left out) do not."""
    import torch

    V, n = 1 << 20, 0
    gen = torch.Generator(device="cuda").manual_seed(edges & 1023)
    src = [torch.randint(0, V, (edges,), generator=gen, device="cuda", dtype=torch.int32)]
    dst = [torch.randint(1000, V - 5000, (edges,), generator=gen, device="cuda", dtype=torch.int32)]
    for d in (2047, 2048, 2049, 4095, 4096, 4097, 8191, 8192, 8193, 12289):
        for _ in range(3):
            src.append(torch.randint(0, V, (d,), generator=gen, device="cuda", dtype=torch.int32))
            dst.append(torch.full((d,), n, device="cuda", dtype=torch.int32))
            n += 1
    src, dst = torch.cat(src), torch.cat(dst)
    w = None
    if weights == "u32":
        w = torch.randint(1, high + 1, (src.numel(),), generator=gen, device="cuda", dtype=torch.int32)
        w[0] = high
    elif weights == "f32":
        w = torch.rand(src.numel(), generator=gen, device="cuda") * 10.0 + 0.05
    torch.cuda.synchronize()
    csr = hyt.csr_from_edges(src, dst, V, w, device=True)
    with hyt.Graph(csr) as a, hyt.Graph(csr, flags=hyt.capi.HYT_GRAPH_PUSH) as p:
        got, st = a.sssp(7)
        want, sp = p.sssp(7)
        assert np.array_equal(got, want)
        if weights == "none":
            assert st["edges_processed"] != sp["edges_processed"]
        many = a.sssp_multi([7, 40000, V - 1])[0]
        assert np.array_equal(many[0], want)
        assert np.array_equal(many[2], p.sssp(V - 1)[0])
