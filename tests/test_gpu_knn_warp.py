"""The warp-per-query neighbour kernels where they can go wrong, against the oracle.

Neighbour lists for every k around the kernels' limits (lanes, buffers, the largest k) with the
reference's first radius, a far too small and a far too large one; a lattice, where every
distance ties and the library's heap order decides; two species, whose masses differ inside the
neighbourhoods, so that the density sums run in distance order.
"""
from __future__ import annotations

import struct

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracle_mod(built):
    import oracle

    return oracle


def _write(path, rec, ntypes=1, fractions=(1.0,)):
    lim = [-0.1, 0.1] * 6
    path.write_bytes(struct.pack(f"<12fi{ntypes}fffq", *lim, ntypes, *fractions, 0.0, 0.0, len(rec)) + rec.tobytes())


def _param(path, four_pi_G, knn=32, hop=16, nx=16):
    path.write_text(f"Nx1 = {nx}\nNx2 = {nx}\nNx3 = {nx}\nZ = 0.02\nfour_pi_G_par = {four_pi_G!r}\nknn = {knn}\nhop = {hop}\nnum_threads = 4\n")


@pytest.fixture(scope="module")
def snapshots(built, tmp_path_factory):
    """name -> (lis, param): the 20k snapshot, a lattice, a two-species snapshot."""
    d = tmp_path_factory.mktemp("knnw")
    out = {}
    rec, g = cases._records(cases.BY_NAME["w1_20k"])
    # every third particle of another species
    two = rec.copy()
    two["type"] = (np.arange(len(two)) % 3 == 0).astype(np.int32)
    n = 20
    lat = np.zeros(n**3, dtype=cases.REC)
    at = (np.arange(n, dtype=np.float32) - np.float32(9.5)) * np.float32(0.0078125)
    lat["pos"] = np.stack(np.meshgrid(at, at, at, indexing="ij"), -1).reshape(-1, 3)
    lat["id_in_run"] = np.arange(n**3)
    for name, r, nt, fr in (("plain", rec, 1, (1.0,)), ("two", two, 2, (0.7, 0.3)), ("lattice", lat, 1, (1.0,))):
        _write(d / f"{name}.lis", r, nt, fr)
        _param(d / f"{name}.txt", g)
        out[name] = (str(d / f"{name}.lis"), str(d / f"{name}.txt"))
    return out


@pytest.fixture(scope="module")
def trees(built, oracle_mod, snapshots):
    made = {}

    def get(name):
        if name not in made:
            lis, par = snapshots[name]
            f = built.Finder(0)
            f.build_tree(built.Snapshot(lis), built.params(par))
            made[name] = (f, oracle_mod.Oracle(lis, par, threads=4, pow_mode=1))
        return made[name]

    yield get
    for f, _ in made.values():
        f.close()


@pytest.mark.parametrize("name", ["plain", "lattice"])
@pytest.mark.parametrize("k", [1, 2, 31, 32, 33, 64, 65, 127, 128])
def test_knn_lists(name, k, trees):
    f, o = trees(name)
    pos = f.stage(1)[:, :3]
    q = pos[np.random.default_rng(k).integers(0, len(pos), 37)]
    for est in (0.0, 1e-6, 0.3):
        gi, gd = f.knn(q, k, est)
        oi, od = o.knn(q, k, est)
        np.testing.assert_array_equal(gd, od)
        np.testing.assert_array_equal(gi, oi)


@pytest.mark.parametrize("name", ["two", "lattice"])
def test_densities_and_densest(name, built, oracle_mod, snapshots):
    lis, par = snapshots[name]
    f = built.Finder(0)
    f.find_clumps(built.Snapshot(lis), built.params(par))
    o = oracle_mod.Oracle(lis, par, threads=4, pow_mode=1)
    o.find()
    np.testing.assert_array_equal(f.stage(built.PLAN_ARR_DENSITY), o.points()[0][:, 8])
    np.testing.assert_array_equal(f.stage(built.PLAN_ARR_DENSEST), o.densest())
    f.close()
