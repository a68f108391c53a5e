"""The bulk-staged task pass of packed personalized PageRank (HYT_STAGED=1) runs
at every graph size, the largest hot table included, and gives the oracle's
ranks.  The switch is read once per process, so each case is a process."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import json, sys
import numpy as np
import hytgraph_b200 as hyt
z = np.load(sys.argv[1])
with hyt.Graph(hyt.CSR(z["off"], z["cols"], None)) as g:
    r, st = g.ppr_multi(z["sources"], tolerance=1e-7, max_iterations=300)
np.save(sys.argv[2], r)
print(json.dumps({"launches": st[0]["total_launches"], "iterations": max(s["iterations"] for s in st)}))
"""


def _graph(V, seed):
    """Rows of every class: none or a few in-edges, 32 to 200, and 255, 256, 257,
    700, 1024 and 5000 around the tile and the chunk."""
    rng = np.random.default_rng(seed)
    degrees = [32, 63, 64, 65, 200, 255, 256, 257, 700, 1024, 1025, 5000]
    dst = np.concatenate([np.full(d, 7 * i + 1) for i, d in enumerate(degrees)] + [rng.integers(0, V, 60000)])
    src = rng.integers(0, min(V, 30000), dst.size)
    keep = np.unique(src * np.int64(V) + dst)
    src, dst = keep // V, (keep % V).astype(np.uint32)
    off = np.zeros(V + 1, np.uint64)
    np.cumsum(np.bincount(src, minlength=V), out=off[1:])
    return off, dst


@pytest.mark.parametrize("V", [30011, (1 << 22) - 1, 1 << 22, (1 << 22) + 12345])
def test_staged_pass(hyt, gpu, oracle, tmp_path, V):
    off, cols = _graph(V, V)
    sources = np.flatnonzero(np.diff(off.astype(np.int64)))[[0, 10, 999]].astype(np.uint32)
    np.savez(tmp_path / "g.npz", off=off, cols=cols, sources=sources)
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(tmp_path / "g.npz"), str(tmp_path / "r.npy")],
                       env=dict(os.environ, HYT_STAGED="1", PYTHONPATH=str(ROOT)), capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr
    st = json.loads(r.stdout.splitlines()[-1])
    # a step is five launches: shares, their sums, the staged tasks, the long
    # rows, the closing sums (seven when each row class has a kernel)
    assert st["launches"] == 1 + 5 * st["iterations"], st
    got = np.load(tmp_path / "r.npy")
    for l, s in enumerate(sources):
        want = oracle.ppr_f64(off, cols, int(s), 0.15, 1e-12, 600)[0]
        assert np.abs(got[l].astype(np.float64) - want).sum() <= 1e-5, l
