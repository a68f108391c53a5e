"""Whole solves in one cooperative launch: the same ranks, bit for bit, as the
loop of launches, at sizes on both sides of the limit where the sums of an
iteration are shared out among the CTAs; and solves of several graphs on several
streams at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (rows + edges) / 512 slots, 1024 to a group, up to 4 groups summed by every CTA
@pytest.mark.parametrize("scale,ef", [(1, 1), (8, 4), (12, 16), (16, 16), (17, 15), (17, 18), (18, 16), (20, 16)])
@pytest.mark.parametrize("hub", [False, True])
def test_ranks_have_the_bits_of_the_loop(hyt, gpu, scale, ef, hub):
    g = hyt.rmat(scale, ef, 90 + scale, device=True)
    flags = hyt.capi.HYT_GRAPH_ALL | (hyt.capi.HYT_GRAPH_HUB_ORDER if hub else 0)
    loop = hyt.capi.HYT_RUN_NO_GRAPH
    with hyt.Graph(g, flags=flags) as dg:
        for max_iterations in (1, 2, 3, 100):
            a, sa = dg.pagerank(max_iterations=max_iterations)
            b, sb = dg.pagerank(max_iterations=max_iterations, flags=loop)
            assert sa["iterations"] == sb["iterations"] and sa["residual"] == sb["residual"]
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        a, sa = dg.ppr(1)
        b, sb = dg.ppr(1, flags=loop)
        assert sa["iterations"] == sb["iterations"]
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_solves_of_several_graphs_at_once(hyt, gpu):
    graphs = [hyt.rmat(s, 16, 70 + s) for s in (12, 17, 19)]
    handles = [hyt.Graph(g) for g in graphs]
    sources = [int(hyt.pick_sources(g.row_offsets, 4, 1)[0]) for g in graphs]
    want = [(h.pagerank()[0], h.sssp(s)[0], h.sssp_multi([s, 0])[0]) for h, s in zip(handles, sources)]
    wrong = []

    def work(i):
        try:
            for _ in range(20):
                got = (handles[i].pagerank()[0], handles[i].sssp(sources[i])[0], handles[i].sssp_multi([sources[i], 0])[0])
                for a, b in zip(got, want[i]):
                    if not np.array_equal(a.view(np.uint32), b.view(np.uint32)):
                        wrong.append(i)
        except Exception as e:  # a thread's exception fails the test
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(handles))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for h in handles:
        h.close()
    assert not wrong
