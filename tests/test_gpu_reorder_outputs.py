"""Device arrays handed to the caller by the renumbering: cudaMalloc memory (a
caller may export it), not handed on while work that reads it is queued, reused
at other sizes with the right contents, and returned on request."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(hyt, V, E, seed):
    rng = np.random.default_rng(seed)
    src = np.sort(rng.integers(0, V, E, dtype=np.uint32))
    off = np.zeros(V + 1, np.uint64)
    np.cumsum(np.bincount(src, minlength=V), out=off[1:])
    return hyt.CSR(off, rng.integers(0, V, E, dtype=np.uint32), rng.integers(1, 64, E, dtype=np.uint32))


def _order(V, seed):
    return np.random.default_rng(seed + 1).permutation(V).astype(np.uint32)


def _same(dev, host):
    d = dev.download()
    return (np.array_equal(d.row_offsets, host.row_offsets) and
            np.array_equal(d.column_indices, host.column_indices) and np.array_equal(d.weights, host.weights))


@pytest.mark.parametrize("V,E", [(1, 0), (100, 1000), (1 << 16, 1 << 20)])
def test_outputs_can_be_exported(hyt, gpu, V, E):
    d = hyt.reorder(_graph(hyt, V, E, 3), _order(V, 3), device=True)
    cuda = ctypes.CDLL("libcuda.so.1")
    c = d.to_c()
    for p in [c.row_offsets] + ([c.column_indices, c.weights] if E else []):
        pool = ctypes.c_void_p()
        # CU_POINTER_ATTRIBUTE_MEMPOOL_HANDLE: null for cudaMalloc memory
        assert cuda.cuPointerGetAttribute(ctypes.byref(pool), 17, ctypes.c_uint64(p)) == 0 and not pool.value
        handle = (ctypes.c_char * 64)()
        assert cuda.cuIpcGetMemHandle(handle, ctypes.c_uint64(p)) == 0


def test_free_waits_for_readers(hyt, gpu):
    """A stream of the caller's own still copies the arrays when they are freed,
    and another renumbering of the same sizes follows at once."""
    import torch

    V, E = 1 << 16, 1 << 24
    a, b, order = _graph(hyt, V, E, 5), _graph(hyt, V, E, 6), _order(V, 5)
    want = hyt.reorder(a, order).column_indices
    d = hyt.reorder(a, order, device=True)
    view = type("View", (), {"__cuda_array_interface__": {"data": (d.to_c().column_indices, False), "shape": (E,),
                                                          "typestr": "<i4", "version": 3}})()
    src = torch.as_tensor(view, device="cuda")
    dst = torch.zeros(E, dtype=torch.int32, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for _ in range(1500):  # 64 MiB each, longer on the GPU than to queue: tens of milliseconds in all
            dst.copy_(src)
    queued = not s.query()
    d.free()
    e = hyt.reorder(b, order, device=True)
    s.synchronize()
    assert queued
    assert np.array_equal(dst.cpu().numpy().view(np.uint32), want)
    assert _same(e, hyt.reorder(b, order))


def test_blocks_are_reused_at_other_sizes(hyt, gpu):
    for i, E in enumerate([1 << 20, (1 << 20) - 1, 1000, 900, 1 << 20, 0, 5, 1 << 21, 1 << 20]):
        V = 1 + E // 16
        g, order = _graph(hyt, V, E, i), _order(V, i)
        d = hyt.reorder(g, order, device=True)
        if E:
            assert _same(d, hyt.reorder(g, order)), E
        d.free()


def test_many_small_results_at_once(hyt, gpu):
    g, order = _graph(hyt, 1000, 8000, 2), _order(1000, 2)
    want = hyt.reorder(g, order)
    for _ in range(2):
        held = [hyt.reorder(g, order, device=True) for _ in range(100)]  # 300 blocks
        assert all(_same(d, want) for d in held)
        for d in held[::2] + held[1::2]:
            d.free()


def test_kept_blocks_are_bounded_and_returned(hyt, gpu):
    import torch

    g = hyt.rmat(20, 64, 9, device=True)  # 8 bytes an edge: about 0.45 GB a result
    order = torch.arange(g.num_vertices, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    hyt.reorder(g, order, device=True).free()
    hyt.capi.check(hyt.capi.lib.hyt_trim_device_memory(0))
    free = torch.cuda.mem_get_info()[0]
    for d in [hyt.reorder(g, order, device=True) for _ in range(14)]:
        d.free()
    # 4 GiB of results are kept, and the scratch of one call
    assert torch.cuda.mem_get_info()[0] >= free - (5 << 30)
    hyt.capi.check(hyt.capi.lib.hyt_trim_device_memory(0))
    assert torch.cuda.mem_get_info()[0] >= free - (64 << 20)
