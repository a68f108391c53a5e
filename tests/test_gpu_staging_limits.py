"""Pageable copies on both sides of the sizes from which they go through pinned
chunks (4 MiB to the device and into host memory that nothing has touched, 16 MiB
into host memory that has its pages), at odd addresses."""
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


@pytest.mark.parametrize("n", [4 * MIB - 1, 4 * MIB, 9 * MIB + 17, 16 * MIB - 1, 16 * MIB, 41 * MIB + 4099])
@pytest.mark.parametrize("shift", [0, 3])
def test_round_trip(hyt, gpu, n, shift):
    import torch

    host = np.random.default_rng(n + shift).integers(0, 256, n + shift, dtype=np.uint8)[shift:]
    dev = torch.zeros(n + shift, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    hyt.capi.copy(dev.data_ptr() + shift, host.ctypes.data, n)
    back = np.full(n + 2 * shift, 7, np.uint8)
    hyt.capi.copy(back.ctypes.data + shift, dev.data_ptr() + shift, n)
    assert np.array_equal(back[shift:shift + n], host)
    assert np.all(back[:shift] == 7) and np.all(back[shift + n:] == 7)
    assert np.array_equal(dev[shift:].cpu().numpy(), host)
    fresh = mmap.mmap(-1, n + 2 * shift)
    back = np.frombuffer(fresh, np.uint8)
    hyt.capi.copy(back.ctypes.data + shift, dev.data_ptr() + shift, n)
    assert np.array_equal(back[shift:shift + n], host)
    assert not back[:shift].any() and not back[shift + n:].any()
