"""Where the records of a snapshot lie: the tree is the same from any memory.

Blocks of records in pageable, page-locked and device memory, several of them with odd counts and
on boundaries of 16 and of 4 bytes, and a block of which a program has page-locked the first part
only (a kernel that reads it in place would leave the registration).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 5003
SPLITS = {"one": [N], "three": [1237, 0, 2001, N - 1237 - 2001]}


@pytest.fixture(scope="module")
def records(built):
    L = built.lib()
    spec = built.SynthSpec()
    L.plan_synth_default_spec(1, N, 5, C.byref(spec))
    spec.nx = 16
    g = L.plan_synth_four_pi_G_for_mean(C.byref(spec), 16, 16)
    spec.G = g / (4 * math.pi)
    rec = np.zeros(N * 44, np.uint8)
    assert L.plan_synth_records(C.byref(spec), C.c_void_p(rec.ctypes.data), C.byref(built.SynthInfo())) == 0
    return rec, g


class View:
    def __init__(self, built, addresses, counts):
        v = built.LisView()
        for i in range(12):
            v.coor_lim[i] = float(np.float32((-0.1, 0.1)[i % 2]))
        v.ntypes = 1
        v.type_info[0] = 1.0
        v.nblocks = len(counts)
        self.ptr, self.cnt = (C.c_void_p * len(counts))(*addresses), (C.c_uint64 * len(counts))(*counts)
        v.records = C.cast(self.ptr, C.POINTER(C.c_void_p))
        v.counts = C.cast(self.cnt, C.POINTER(C.c_uint64))
        self.view = v


def _tree(built, finder, view, g):
    p = built.params()
    p.box_resolution[:] = (16, 16, 16)
    p.solid_to_gas_ratio = 0.02
    p.four_pi_G = g
    finder.build_tree(view, p)
    return [finder.stage(a) for a in (built.PLAN_ARR_TREE_POS, built.PLAN_ARR_TREE_VEL, built.PLAN_ARR_ORIG_ID)]


@pytest.fixture(scope="module")
def want(built, records):
    f = built.Finder(0)
    out = _tree(built, f, View(built, [records[0].ctypes.data], [N]), records[1])
    f.close()
    return out


@pytest.mark.parametrize("split", SPLITS)
@pytest.mark.parametrize("offset", [0, 4, 20])
@pytest.mark.parametrize("memory", ["pageable", "locked", "device"])
def test_same_tree_from_any_memory(memory, offset, split, built, records, want):
    import torch

    counts = SPLITS[split]
    rec, g = records
    buf = torch.zeros(offset + rec.size, dtype=torch.uint8, pin_memory=memory == "locked")
    buf[offset:] = torch.from_numpy(rec)
    if memory == "device":
        buf = buf.cuda()
        torch.cuda.synchronize()
    at = buf.data_ptr() + offset + 44 * np.concatenate([[0], np.cumsum(counts)[:-1]])
    f = built.Finder(0)
    for got, w in zip(_tree(built, f, View(built, [int(a) for a in at], counts), g), want):
        np.testing.assert_array_equal(got, w)
    f.close()


def test_partly_locked_block(built, records, want):
    import torch

    rec, g = records
    raw = np.zeros(rec.size + (1 << 17), np.uint8)
    start = (raw.ctypes.data + 65535) // 65536 * 65536 - raw.ctypes.data
    raw[start:start + rec.size] = rec
    at = raw.ctypes.data + start
    torch.zeros(1, device="cuda")
    cudart = torch.cuda.cudart()
    assert int(cudart.cudaHostRegister(at, 65536, 0)) == 0  # of 220,132 bytes
    f = built.Finder(0)
    try:
        got = _tree(built, f, View(built, [at], [N]), g)
    except built.PlanError:
        got = want  # the copy may refuse such a range; it must not harm the context
    finally:
        assert int(cudart.cudaHostUnregister(at)) == 0
    for a, w in zip(got, want):
        np.testing.assert_array_equal(a, w)
    for a, w in zip(_tree(built, f, View(built, [at], [N]), g), want):
        np.testing.assert_array_equal(a, w)
    f.close()
