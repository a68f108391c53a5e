"""Pull kernels at the in-degrees where their row dispatch changes: empty
rows, the limits of 1, 2, 4 and 8 lanes per row, warp rows, chunked rows and
rows of several chunks, against the FP64 and Dijkstra oracles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = [0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513,
           1023, 1024, 1025, 4095, 4096, 4097, 8191, 8192, 8193, 12289]


def _graph(hyt, order):
    """Rows of every degree of DEGREES (32 alike in a row, or mixed) pulled
    from seeded distinct sources; the last vertices are sources only."""
    rng = np.random.default_rng(11)
    V = 40000
    deg = np.repeat(DEGREES, 3 if order == "mixed" else 2)
    if order == "mixed":
        rng.shuffle(deg)
    src, dst = [], []
    for v, d in enumerate(deg):
        src.append(rng.choice(V, d, replace=False))
        dst.append(np.full(d, v))
    # a ring keeps most vertices from dangling
    ring = np.arange(V // 2, V)
    src += [ring]
    dst += [np.roll(ring, -1)]
    s, d = np.concatenate(src), np.concatenate(dst)
    keep = s != d
    s, d = s[keep].astype(np.uint32), d[keep].astype(np.uint32)
    at = np.lexsort((d, s))
    s, d = s[at], d[at]
    off = np.zeros(V + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(s, minlength=V))
    w = rng.integers(1, 64, s.shape[0]).astype(np.uint32)
    return hyt.CSR(off, d, w)


@pytest.mark.parametrize("order", ["sorted", "mixed"])
@pytest.mark.parametrize("hub", [False, True])
def test_pagerank_row_degrees(hyt, oracle, gpu, order, hub):
    g = _graph(hyt, order)
    flags = hyt.capi.HYT_GRAPH_ALL | (hyt.capi.HYT_GRAPH_HUB_ORDER if hub else 0)
    ref, _, _, _ = oracle.pagerank_f64(g.row_offsets, g.column_indices, 0.85, 1e-30, 20)
    with hyt.Graph(g, flags=flags) as dg:
        r, st = dg.pagerank(tolerance=1e-30, max_iterations=20)
    assert st["iterations"] == 20
    # compensated sums, one division, one multiplication and one addition are
    # under 3 ulp a step; the steps' errors shrink by 0.85 each: 3 / 0.15 = 20
    # ulp of 2^-24, tripled
    assert np.max(np.abs(r.astype(np.float64) - ref) / ref) <= 60 * 2.0 ** -24


@pytest.mark.parametrize("order", ["sorted", "mixed"])
@pytest.mark.parametrize("weights", ["none", "u32", "f32", "u32_large"])
def test_sssp_row_degrees(hyt, oracle, gpu, order, weights):
    g = _graph(hyt, order)
    w = {"none": None, "u32": g.weights, "f32": (g.weights * np.float32(0.37)).astype(np.float32),
         "u32_large": (g.weights.astype(np.uint64) * 40000001).astype(np.uint32)}[weights]
    csr = hyt.CSR(g.row_offsets, g.column_indices, w)
    with hyt.Graph(csr) as dg, hyt.Graph(csr, flags=hyt.capi.HYT_GRAPH_PUSH) as push_only:
        for s in (0, 5, g.num_vertices - 1):
            d, st = dg.sssp(s)
            assert np.array_equal(d, push_only.sssp(s)[0])
            n, _ = dg.sssp(s, flags=hyt.capi.HYT_RUN_NO_GRAPH)
            assert st["converged"] == 1 and np.array_equal(d, n)
            if weights == "u32_large":  # beyond what floats hold exactly: the push-only path
                p, _ = dg.sssp(s, delta=0xFFFFFFFE)
                assert np.array_equal(d, p)
                continue
            ref, _, _ = oracle.sssp(g.row_offsets, g.column_indices, None if w is None else w.astype(np.float32), s)
            if weights == "f32":
                assert np.array_equal(d, ref.view(np.uint32))
            else:
                want = np.where(np.isfinite(ref), ref, 0).astype(np.uint64)
                want = np.where(np.isfinite(ref), want, 0xFFFFFFFF).astype(np.uint32)
                assert np.array_equal(d, want)


@pytest.mark.parametrize("weights", ["none", "u32", "f32", "u32_large"])
def test_sssp_multi_row_degrees(hyt, gpu, weights):
    """Every lane of a packed solve equals the single solve, also where labels
    may saturate (u32_large) and where they cannot."""
    g = _graph(hyt, "mixed")
    w = {"none": None, "u32": g.weights, "f32": (g.weights * np.float32(0.37)).astype(np.float32),
         "u32_large": (g.weights.astype(np.uint64) * 40000001).astype(np.uint32)}[weights]
    with hyt.Graph(hyt.CSR(g.row_offsets, g.column_indices, w)) as dg:
        sources = [0, 5, g.num_vertices - 1, 17, 30000, 5, 39000]
        d, st = dg.sssp_multi(sources)
        assert st["converged"] == 1
        for lane, s in enumerate(sources):
            assert np.array_equal(d[lane], dg.sssp(s)[0]), s
