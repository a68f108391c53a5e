"""Packed personalized PageRank at the limits of its row classes (short, wide and
long rows, their rounds and the pieces of chunks) and for every set of classes
that run side by side, against the FP64 oracle; the same bits alone and packed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMITS = [31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 129, 192, 193, 511]
LONG = [512, 513, 639, 640, 641, 1023, 1024, 1025, 1151, 1152, 1153, 5000]


def _csr(hyt, V, degrees, extra, seed):
    """Rows of the given in-degrees, then rows of 0 to 3 in-edges (extra in all)."""
    rng = np.random.default_rng(seed)
    src = [rng.choice(V, d, replace=False) for d in degrees]
    dst = [np.full(d, i) for i, d in enumerate(degrees)]
    src.append(rng.integers(0, V, extra))
    dst.append(rng.integers(len(degrees), V, extra) if extra else np.zeros(0, np.int64))
    src, dst = np.concatenate(src), np.concatenate(dst)
    order = np.argsort(src, kind="stable")
    off = np.zeros(V + 1, np.uint64)
    np.cumsum(np.bincount(src, minlength=V), out=off[1:])
    w = rng.integers(1, 64, src.size).astype(np.uint32)
    return hyt.CSR(off, dst[order].astype(np.uint32), w)


CASES = {
    "short": (6000, [], 9000),
    "wide": (1500, [100] * 1490, 0),
    "wide_few": (6000, LIMITS, 9000),
    "wide_short": (6000, LIMITS * 3, 9000),
    "long": (5200, LONG, 0),
    "long_short": (6000, LONG, 9000),
    "long_wide": (5200, LONG + LIMITS * 8 + [40] * 4900, 0),
    "all": (9000, LONG * 2 + LIMITS * 4, 15000),
    "star": (70000, [69999], 1000),
}


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("weighted", [False, True])  # tagged ids, ids of packed words
def test_row_classes(hyt, oracle, gpu, case, weighted):
    V, degrees, extra = CASES[case]
    g = _csr(hyt, V, degrees, extra, len(degrees) + V)
    if not weighted:
        g = hyt.CSR(g.row_offsets, g.column_indices, None)
    sources = np.flatnonzero(np.diff(g.row_offsets.astype(np.int64)))[[0, 3, 17, 40, 99]].astype(np.uint32)
    with hyt.Graph(g) as dg:
        got, st = dg.ppr_multi(sources, tolerance=1e-7, max_iterations=300)
        again, _ = dg.ppr_multi(sources, tolerance=1e-7, max_iterations=300)
        alone, _ = dg.ppr_multi(sources[2:3], tolerance=1e-7, max_iterations=300)
    assert np.array_equal(got.view(np.uint32), again.view(np.uint32))
    assert np.array_equal(got[2].view(np.uint32), alone[0].view(np.uint32))
    for l, s in enumerate(sources):
        want = oracle.ppr_f64(g.row_offsets, g.column_indices, int(s), 0.15, 1e-12, 600)[0]
        assert np.abs(got[l].astype(np.float64) - want).sum() <= 1e-5, l
        assert st[l]["converged"] == 1
