"""The scratch arena's size against what the stages take from it, on the CPU (no GPU).

scratch_bytes_for(T) must hold all that one stage holds at a time: the octree's sort and its
level tables, HOP's member sort and group table, and the clumps' sort, each at its largest, for
any number of tree points. The sizes of the sorts and scans are the library's own.
"""
from __future__ import annotations

import ctypes as C

import pytest


def _fn(lib, name, args):
    f = getattr(lib, name)
    f.restype, f.argtypes = C.c_uint64, [C.c_uint64] * args
    return f


@pytest.mark.parametrize("T", [1, 2, 255, 4097, 16385, 100003, 1 << 20, 26_000_000, 28_000_123, 400_000_000])
def test_holds_every_stage(T, built):
    lib = built.lib()
    sort = _fn(lib, "_ZN4plan26radix_sort96_scratch_bytesEm", 1)
    scan = _fn(lib, "_ZN4plan22scan_u32_scratch_bytesEm", 1)
    size = _fn(lib, "_ZN4plan17scratch_bytes_forEm", 1)

    def takes(*sizes):
        return sum((s + 255) // 256 * 256 for s in sizes)

    blocks = (T + 255) // 256
    octree = takes(max(sort(T), scan(T)), *[4 * (T + 1)] * 3, T, T, T, 128 * blocks, 128)
    ghosts = takes(max(sort(T), scan(T)), 48 * 152 * 4)
    hop = takes(scan(T), *[4 * (T + 1)] * 3, sort(T), *[4 * (T + 1)] * 2, scan(T + 1))
    density = takes(*[4 * (T + 1)] * 2, 16, 4 * T, 4 * T)
    # the largest sort of clump members: every tree point, in clumps of more than 2,048
    clumps = takes(*[4 * T] * 4, *[4 * (T // 2049 + 1)] * 2, sort(T))
    for name, need in (("octree", octree), ("ghosts", ghosts), ("hop", hop), ("density", density), ("clumps", clumps)):
        assert need <= size(T), (name, need, size(T))
