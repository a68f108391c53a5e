"""Contribution schedules where the sorts take other routes: items that ascend
(not sorted), ascend but for one, hold duplicates; contributions whose keys
share their high or low bits, or all of them; and PageRank contributions at the
in-degrees where a row's lanes change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("items", ["ascending", "one_descent", "duplicates", "large"])
@pytest.mark.parametrize("values", ["all_equal", "signed_zeros", "floats", "doubles", "negative"])
@pytest.mark.parametrize("n", [1, 2, 33, 4097])
def test_schedule_routes(hyt, gpu, items, values, n):
    rng = np.random.default_rng(n)
    it = np.arange(n, dtype=np.uint64) * 3
    if items == "one_descent" and n > 1:
        it[-1] = 0
    elif items == "duplicates":
        it = rng.integers(0, max(1, n // 2), n).astype(np.uint64)
    elif items == "large":
        it = np.uint64(2 ** 63) + np.arange(n, dtype=np.uint64)
    c = {"all_equal": np.full(n, 2.5), "signed_zeros": rng.choice([0.0, -0.0], n),
         "floats": rng.random(n).astype(np.float32).astype(np.float64).round(2),
         "doubles": rng.standard_normal(n), "negative": -rng.integers(1, 4, n).astype(np.float64)}[values]
    for tie in (True, False):
        got, m = hyt.contribution_schedule(it, c, deterministic_tie_break=tie)
        order = np.lexsort((np.arange(n), it, -c)) if tie else np.argsort(-c, kind="stable")
        assert np.array_equal(got, it[order]), tie
        assert m["reordered_item_count"] == int((order != np.arange(n)).sum())
        assert m["redundant_work_count"] == n - len(np.unique(it))
        assert m["zero_contribution_count"] == int((c == 0).sum())


@pytest.mark.parametrize("degrees", [[0, 1, 2, 4, 5, 8, 9, 16, 17], [32, 33, 63, 64, 65, 127, 128, 129, 256, 257],
                                     [511, 512, 513, 1023, 1024, 4095, 4096, 4097, 8193]])
def test_contribution_row_degrees(hyt, gpu, degrees):
    rng = np.random.default_rng(5)
    V = 20000
    src = np.concatenate([np.sort(rng.choice(V, d, replace=False)) for d in degrees for _ in range(2)])
    dst = np.repeat(np.arange(2 * len(degrees)), np.repeat(degrees, 2))
    at = np.lexsort((dst, src))
    src, dst = src[at].astype(np.uint32), dst[at].astype(np.uint32)
    off = np.zeros(V + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(src, minlength=V))
    rank = (rng.random(V) / V).astype(np.float32)
    with hyt.Graph(hyt.CSR(off, dst)) as g:
        got = g.pagerank_contributions(rank, 0.85)
    x = rank.astype(np.float64)
    deg = np.diff(off).astype(np.float64)
    share = np.divide(x, deg, out=np.zeros(V), where=deg > 0)
    d = float(np.float32(0.85))
    nxt = (1 - d) / V + d * x[deg == 0].sum() / V + d * np.bincount(dst, share[src], minlength=V)
    # sums of at most 8193 terms in FP64, every term and partial sum below nxt
    assert np.all(np.abs(got - np.abs(nxt - x)) <= 8193 * 2.0 ** -53 * (nxt + x))
