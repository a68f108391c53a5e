"""Long rows at the limits of their chunks, for each chunk length that a
graph's size (rows + edges) selects."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMITS = [511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097, 6145, 8193]


def _graph(hyt, vertices):
    """Rows of LIMITS in-edges from seeded distinct sources among the first
    40000 vertices and a ring over half of them; the other vertices stand
    alone and only make the graph larger."""
    rng = np.random.default_rng(23)
    near = 40000
    ring = np.arange(near // 2, near)
    s = np.concatenate([rng.choice(near, d, replace=False) for d in LIMITS] + [ring])
    d = np.concatenate([np.full(n, v) for v, n in enumerate(LIMITS)] + [np.roll(ring, -1)])
    s, d = s[s != d], d[s != d]
    at = np.lexsort((d, s))
    s, d = s[at], d[at].astype(np.uint32)
    off = np.zeros(vertices + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(s, minlength=vertices))
    return hyt.CSR(off, d, rng.integers(1, 64, d.shape[0]).astype(np.uint32))


@pytest.mark.parametrize("vertices", [40000, (1 << 23) + 3, 1 << 26])
def test_chunk_limits(hyt, oracle, gpu, vertices):
    g = _graph(hyt, vertices)
    ref, _, _, _ = oracle.pagerank_f64(g.row_offsets, g.column_indices, 0.85, 1e-30, 3)
    source = int(np.flatnonzero(np.diff(g.row_offsets.astype(np.int64)))[0])
    with hyt.Graph(g) as dg, hyt.Graph(g, flags=hyt.capi.HYT_GRAPH_PUSH) as push_only:
        r, st = dg.pagerank(tolerance=1e-30, max_iterations=3)
        d = dg.sssp(source)[0]
        m = dg.sssp_multi([source, 20000])[0]
        assert st["iterations"] == 3
        assert np.array_equal(d, push_only.sssp(source)[0])
        assert np.array_equal(m[0], d) and np.array_equal(m[1], push_only.sssp(20000)[0])
    # under 3 ulp a step (compensated sums, a division, a multiplication and
    # an addition), three steps, of 2^-24, tripled
    assert np.max(np.abs(r.astype(np.float64) - ref) / ref) <= 27 * 2.0 ** -24
