"""Host side of the pinned-chunk copies over a made-up CUDA runtime (no GPU, and
so no second one, is needed): which copies they take."""
from __future__ import annotations

import subprocess

from conftest import BUILD, ROOT, run_cpp


def test_staged_copies_over_a_fake_runtime():
    BUILD.mkdir(parents=True, exist_ok=True)
    obj, exe = BUILD / "staging.o", BUILD / "staging_tests"
    csrc = ROOT / "hytgraph_b200" / "csrc"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-cudart", "none", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", str(ROOT / "include"), "-I", str(csrc),
                    "--expt-relaxed-constexpr", "-c", str(csrc / "staging.cu"), "-o", str(obj)], check=True)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(csrc), "-I", "/usr/local/cuda/include",
                    str(ROOT / "tests" / "cpp" / "staging_tests.cpp"), str(obj), "-o", str(exe), "-lpthread"],
                   check=True)
    r = run_cpp(exe)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "staging tests passed" in r.stdout
