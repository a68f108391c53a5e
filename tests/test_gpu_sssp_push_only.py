"""SSSP on graphs without a CSC: whole solves that only push, at the sizes where
the edges a warp keeps in flight change, labels against Dijkstra and against a
solve with sweeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _labels(oracle, g, source):
    if g.weights is None:
        g = type(g)(g.row_offsets, g.column_indices, np.ones(g.num_edges, np.uint32))
    if g.weights.dtype == np.float32:
        d = oracle.sssp(g.row_offsets, g.column_indices, g.weights, source)[0]
        return d.astype(np.float32).view(np.uint32)
    d = oracle.dijkstra(g.row_offsets, g.column_indices, g.weights, source)
    return np.where(d == np.iinfo(np.uint64).max, 0xFFFFFFFF, d).astype(np.uint32)


@pytest.mark.parametrize("kind", ["none", "u32", "f32"])
@pytest.mark.parametrize("hub", [False, True])
def test_push_only_matches_dijkstra(hyt, oracle, gpu, kind, hub):
    # rows of 63, 64, 65 (the hub threshold), 511 to 513 and 2000 out-edges, a
    # chain that needs a round per vertex, and vertices that are not reached
    rng = np.random.default_rng(8)
    degrees = [63, 64, 65, 511, 512, 513, 2000, 1, 0, 31, 32, 33]
    V = 4000
    src = np.concatenate([np.full(d, i) for i, d in enumerate(degrees)] +
                         [np.arange(20, 2999), rng.integers(0, 3000, 4000)])
    dst = np.concatenate([rng.choice(3000, d, replace=False) for d in degrees] +
                         [np.arange(21, 3000), rng.integers(0, 3000, 4000)])
    order = np.argsort(src, kind="stable")
    off = np.zeros(V + 1, np.uint64)
    np.cumsum(np.bincount(src, minlength=V), out=off[1:])
    w = None if kind == "none" else rng.integers(1, 1 << 20, src.size).astype(np.uint32)
    if kind == "f32":
        w = (w / 1000.0).astype(np.float32)
    g = hyt.CSR(off, dst[order].astype(np.uint32), w)
    flags = hyt.capi.HYT_GRAPH_PUSH | (hyt.capi.HYT_GRAPH_HUB_ORDER if hub else 0)
    with hyt.Graph(g, flags=flags) as dg:
        for s in (6, 20, 3999):
            got = dg.sssp(s)[0]
            assert np.array_equal(got, _labels(oracle, g, s)), s
            assert np.array_equal(dg.sssp(s, flags=hyt.capi.HYT_RUN_NO_GRAPH)[0], got), s


@pytest.mark.parametrize("E", [(1 << 27) - 1, 1 << 27])
def test_push_only_at_the_wide_frontier_limit(hyt, gpu, E):
    import torch

    V = 1 << 20
    gen = torch.Generator(device="cuda").manual_seed(E & 7)
    src = torch.randint(0, V, (E,), generator=gen, device="cuda", dtype=torch.int32)
    dst = torch.randint(0, V - 1000, (E,), generator=gen, device="cuda", dtype=torch.int32)
    w = torch.randint(1, 1000, (E,), generator=gen, device="cuda", dtype=torch.int32)
    torch.cuda.synchronize()
    csr = hyt.csr_from_edges(src, dst, V, w, device=True)
    with hyt.Graph(csr, flags=hyt.capi.HYT_GRAPH_PUSH) as a, hyt.Graph(csr) as b:
        assert np.array_equal(a.sssp(5)[0], b.sssp(5)[0])
