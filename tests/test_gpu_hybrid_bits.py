"""Out-of-HBM PageRank sums every row as the in-HBM solve does: the ranks are
the same bits at any budget, partition size and engine, though the pieces that
travel cut the tiles of rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csc(g):
    V = g.num_vertices
    src = np.repeat(np.arange(V, dtype=np.uint32), np.diff(g.row_offsets.astype(np.int64)))
    order = np.argsort(g.column_indices, kind="stable")
    in_off = np.zeros(V + 1, np.uint64)
    np.cumsum(np.bincount(g.column_indices, minlength=V), out=in_off[1:])
    return in_off, src[order]


# scale 20 takes 1024-unit tiles and 2048-edge chunks, the others 512 and 1024
@pytest.mark.parametrize("scale,ef,part_bits", [(10, 8, 5), (14, 16, 3), (16, 16, 10), (17, 4, 17), (20, 16, 14)])
@pytest.mark.parametrize("budget_kib", [1, 4096, 1 << 20])
def test_ranks_are_the_in_hbm_bits(hyt, gpu, scale, ef, part_bits, budget_kib):
    g = hyt.rmat(scale, ef, 31 + scale)
    in_off, in_src = _csc(g)
    with hyt.Graph(g) as dg:
        want, st = dg.pagerank()
        p = int(hyt.pick_sources(g.row_offsets, 3, 1)[0])
        want_p = dg.ppr(p)[0]
    for engine in ("AUTO", "FILTER", "ZERO_COPY"):
        if g.num_vertices >> part_bits > 1024:
            part_bits = (g.num_vertices >> 10).bit_length() - 1
        with hyt.HybridGraph(g.row_offsets, g.column_indices, None, in_off, in_src,
                             flags=hyt.capi.HYT_GRAPH_PULL, budget_bytes=budget_kib << 10,
                             partition_vertices=1 << part_bits,
                             force_engine=getattr(hyt.capi, "HYT_ENGINE_" + engine)) as hg:
            r, sh = hg.pagerank()[:2]
            assert sh["iterations"] == st["iterations"], engine
            assert np.array_equal(r.view(np.uint32), want.view(np.uint32)), (engine, np.count_nonzero(r != want))
            if hasattr(hg, "ppr"):
                assert np.array_equal(hg.ppr(p)[0].view(np.uint32), want_p.view(np.uint32)), engine
