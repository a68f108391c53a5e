"""Copies between pageable host memory and the device through pinned chunks:
sizes around the threshold and the chunk, odd addresses, several threads at
once, and after the chunks were given back."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _round_trip(hyt, torch, n, shift):
    rng = np.random.default_rng(n + shift)
    host = rng.integers(0, 256, n + shift, dtype=np.uint8)[shift:]
    dev = torch.zeros(n + shift, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    hyt.capi.copy(dev.data_ptr() + shift, host.ctypes.data, n)
    back = np.zeros(n + shift, np.uint8)
    hyt.capi.copy(back.ctypes.data + shift, dev.data_ptr() + shift, n)
    return np.array_equal(back[shift:], host) and np.array_equal(dev[shift:].cpu().numpy(), host)


@pytest.mark.parametrize("n", [1, MIB, 4 * MIB - 1, 4 * MIB, 4 * MIB + 1, 17 * MIB + 12345])
@pytest.mark.parametrize("shift", [0, 1, 13])
def test_pageable_round_trip(hyt, gpu, n, shift):
    import torch

    assert _round_trip(hyt, torch, n, shift)


def test_pageable_threads_and_trim(hyt, gpu):
    import torch

    torch.zeros(1, device="cuda")
    ok = []
    ts = [threading.Thread(target=lambda i=i: ok.append(_round_trip(hyt, torch, 9 * MIB + i, i))) for i in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert ok == [True] * 6
    hyt.capi.check(hyt.capi.lib.hyt_trim_device_memory(0))
    assert _round_trip(hyt, torch, 8 * MIB, 3)
