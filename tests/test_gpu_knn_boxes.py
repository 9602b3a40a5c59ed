"""Neighbour lists at a program's own positions in boxes of any size, against the oracle.

The warp kernels decide in FP32 on float pairs, whose absolute errors grow with the coordinates:
boxes of half widths 0.1, 4 and 300 at a time with sheared ghosts, tight clusters on the planes
between the root's octants, positions a hair from a point and first radii far below the large
nodes' size.
"""
from __future__ import annotations

import struct

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

N = 6000


@pytest.fixture(scope="module", params=[0.1, 4.0, 300.0])
def tree(request, built, tmp_path_factory):
    import oracle

    X = request.param
    rng = np.random.default_rng(17)
    rec = np.zeros(N, dtype=cases.REC)
    pos = rng.uniform(-0.99, 0.99, (N, 3))
    at = 0
    for i in range(12):
        c = np.where(rng.random(3) < 0.6, 0.0, rng.uniform(-0.7, 0.7, 3))
        pos[at:at + 300] = c + 10.0 ** rng.uniform(-6, -3) * rng.standard_normal((300, 3))
        at += 300
    rec["pos"] = (pos * X).astype(np.float32)
    rec["id_in_run"] = np.arange(N)
    d = tmp_path_factory.mktemp("box")
    lim = [float(np.float32(-X)), float(np.float32(X))] * 6
    (d / "s.lis").write_bytes(struct.pack("<12fi1fffq", *lim, 1, 1.0, 0.37, 0.0, N) + rec.tobytes())
    (d / "p.txt").write_text("Nx1 = 16\nNx2 = 16\nNx3 = 16\nZ = 0.02\nfour_pi_G_par = 0.05\nknn = 32\nhop = 16\nnum_threads = 4\n")
    f = built.Finder(0)
    f.build_tree(built.Snapshot(str(d / "s.lis")), built.params(str(d / "p.txt")))
    yield X, f, oracle.Oracle(str(d / "s.lis"), str(d / "p.txt"), threads=4, pow_mode=1)
    f.close()


@pytest.mark.parametrize("k", [1, 8, 32, 100])
def test_lists(k, tree):
    X, f, o = tree
    rng = np.random.default_rng(k)
    pos = f.stage(1)[:, :3]
    at = pos[rng.integers(0, len(pos), 400)]
    near = at + X * 10.0 ** rng.uniform(-14, -2, (400, 1)) * rng.uniform(-1, 1, (400, 3))
    # (without a first radius a position must have a leaf of its own: the points')
    for q, est in ((at, 0.0), (near, 1e-6 * X), (near, 1e-4 * X), (near, 0.01 * X), (near, 0.5 * X)):
        gi, gd = f.knn(q, k, est)
        oi, od = o.knn(q, k, est)
        np.testing.assert_array_equal(gd, od)
        np.testing.assert_array_equal(gi, oi)
