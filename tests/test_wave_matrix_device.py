"""Waves handed to a job as device tensors are held until they are copied, not for the job's lifetime."""
import weakref

import numpy as np
import torch

from dwba_b200.engine import WaveMatrix


def test_rows_from_a_tensor_are_released_after_their_copy():
    n = 40
    waves = WaveMatrix(n)
    t = torch.arange(3.0 * n, dtype=torch.float64).reshape(3, n)
    want = t.clone()
    host = np.linspace(0.0, 1.0, n)
    assert waves.add(host) == 0 and waves.add_device(t) == 1
    held = weakref.ref(waves._device[0][1])
    out = waves.upload("cpu")
    assert torch.equal(out[1:4], want) and np.array_equal(out[0].numpy(), host) and waves.n_host == 1
    assert held() is None  # the detached tensor, which shares the caller's memory
    t.fill_(7.0)
    waves.add(2.0 * host)  # a row more: uploaded again, from what was uploaded
    again = waves.upload("cpu")
    assert torch.equal(again[1:4], want) and np.array_equal(again[4].numpy(), 2.0 * host) and waves.n_host == 2
