"""Hub sort on both sides of the size up to which all vertices are sorted at once,
with none, some and all of the vertices scored, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 2, 2047, 2048, 2049])
@pytest.mark.parametrize("scored", ["none", "some", "all"])
@pytest.mark.parametrize("fraction", [0.0, 0.08, 1.0])
def test_sizes_around_the_whole_sort(hyt, oracle, gpu, V, scored, fraction):
    rng = np.random.default_rng(V)
    if scored == "none":  # edges from one half to the other: no vertex has both degrees
        src, dst = rng.integers(0, max(V // 2, 1), 4 * V), rng.integers(V // 2, V, 4 * V)
        if V < 2:
            src = dst = np.zeros(0, np.int64)
    elif scored == "some":
        src, dst = rng.integers(0, (V + 2) // 3, 4 * V), rng.integers(0, (V + 1) // 2, 4 * V)
    else:
        src = np.concatenate([np.arange(V), rng.integers(0, V, 4 * V)])
        dst = np.concatenate([np.roll(np.arange(V), 1), rng.integers(0, V, 4 * V)])
    order = np.argsort(src, kind="stable")
    off = np.zeros(V + 1, np.uint64)
    np.cumsum(np.bincount(src, minlength=V), out=off[1:])
    g = hyt.CSR(off, dst[order].astype(np.uint32), None)
    got, scores, hubs = hyt.hub_sort(g, fraction)
    want, want_scores, want_hubs = oracle.hub_sort(off, g.column_indices, fraction)
    assert hubs == want_hubs
    assert np.array_equal(got, want)
    assert np.array_equal(np.asarray(scores).view(np.uint64), np.asarray(want_scores).view(np.uint64))


@pytest.mark.parametrize("V", [2048, 2049])
def test_bad_destinations_are_rejected(hyt, gpu, V):
    off = np.arange(V + 1, dtype=np.uint64)
    cols = np.zeros(V, np.uint32)
    cols[V // 2] = V
    with pytest.raises(hyt.HytError) as e:
        hyt.hub_sort(hyt.CSR(off, cols, None), 0.1)
    assert e.value.code == hyt.capi.HYT_E_INVALID
