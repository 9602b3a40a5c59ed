"""A box narrower than the ghost zone: every particle has three ghosts.

The scratch memory is first sized from the particles alone. Seven million of them in such a box
make 28 million tree points, which need more than that.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

N = 7_000_000
HALF = 0.02


def test_tree_of_four_points_per_particle(built):
    rng = np.random.default_rng(1)
    rec = np.zeros(N, dtype=cases.REC)
    rec["pos"] = rng.random((N, 3), dtype=np.float32) * np.float32(2 * HALF * 0.999) - np.float32(HALF * 0.999)
    rec["id_in_run"] = np.arange(N)
    v = built.LisView()
    for i in range(12):
        v.coor_lim[i] = float(np.float32((-HALF, HALF)[i % 2]))
    v.ntypes = 1
    v.type_info[0] = 1.0
    v.nblocks = 1
    ptr, cnt = (C.c_void_p * 1)(rec.ctypes.data), (C.c_uint64 * 1)(N)
    v.records, v.counts = C.cast(ptr, C.POINTER(C.c_void_p)), C.cast(cnt, C.POINTER(C.c_uint64))

    class Snap:
        view = v

    p = built.params()
    p.box_resolution[:] = (64, 64, 64)
    p.solid_to_gas_ratio = 0.02
    p.four_pi_G = 0.05
    f = built.Finder(0)
    f.build_tree(Snap, p)
    orig, sinks = f.stage(built.PLAN_ARR_ORIG_ID), f.stage(built.PLAN_ARR_SINK_COUNT)
    inside = int((rec["pos"][:, :2] != 0).all(axis=1).sum())  # a ghost in x, one in y and one in both
    assert 4 * inside <= int(sinks.sum()) <= 4 * N
    assert len(np.unique(orig[orig < N])) > 0.99 * N
    f.close()
