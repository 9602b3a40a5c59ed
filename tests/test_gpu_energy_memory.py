"""What a batch of group energies leaves behind on the device.

The workspace of a batch of up to 1 GiB stays with the context; a larger one gives its memory back
when the call returns.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(groups: int, size: int):
    rng = np.random.default_rng(groups)
    n = groups * size
    off = np.arange(groups + 1, dtype=np.uint64) * np.uint64(size)
    return rng.random((n, 3), dtype=np.float32), rng.random((n, 3), dtype=np.float32), rng.random(n, dtype=np.float32), off


def test_large_batch_gives_its_memory_back(built):
    import torch

    p = built.params()
    built.lib().plan_params_derive(C.byref(p))
    f = built.Finder(0)
    small, large = _batch(16, 100), _batch(130000, 200)
    want = f.group_energies(*small, p)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    first = f.group_energies(*large, p)  # 26 million particles: 1.6 GB
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= free - (64 << 20)
    for a, b in zip(f.group_energies(*large, p), first):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(f.group_energies(*small, p), want):
        np.testing.assert_array_equal(a, b)
    f.close()
