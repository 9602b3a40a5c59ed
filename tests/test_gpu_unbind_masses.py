"""Finds with particles of very unequal masses, against the oracle.

Two species of which one is a few hundred times as heavy, a few heavy particles in every clump
and some of them far out: unbinding then takes members that hold most of what is left of a clump's
mass, where its FP32 test must leave the decision to FP64.
"""
from __future__ import annotations

import struct

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ratio,heavy", [(1.0, 0.1), (60.0, 0.003), (400.0, 0.001)])
def test_find_matches_oracle(ratio, heavy, built, tmp_path):
    import oracle

    n = 20000
    rng = np.random.default_rng(int(ratio))
    rec, g = cases._records(cases.BY_NAME["w1_20k"])
    rec = np.resize(rec, n)
    rec["pos"] = rng.uniform(-0.099, 0.099, (n, 3)).astype(np.float32)
    rec["vel"] = (1e-4 * rng.standard_normal((n, 3))).astype(np.float32)
    rec["id_in_run"] = np.arange(n)
    rec["type"] = 0
    at = 0
    for i in range(27):  # spheres with a heavy member at the edge, one in the middle and some at random
        m = int(rng.integers(40, 700))
        x = rng.standard_normal((m, 3))
        x *= (0.002 * rng.random((m, 1)) ** (2 / 3)) / np.linalg.norm(x, axis=1, keepdims=True)
        x[0] *= 0.0021 / np.linalg.norm(x[0])
        c = np.array([i % 3 - 1, i // 3 % 3 - 1, i // 9 - 1]) * 0.06 + rng.uniform(-0.005, 0.005, 3)
        rec["pos"][at:at + m] = (c + x).astype(np.float32)
        if i % 2:
            rec["vel"][at:at + m] *= 30
        rec["type"][at:at + 2] = 1
        at += m
    rec["type"][rng.random(n) < heavy] = 1
    rec = rec[rng.permutation(n)]
    nh = int((rec["type"] == 1).sum())
    # a particle's mass is its species' share of all mass over the number of all particles: light ones as with one species
    lim = [-0.1, 0.1] * 6
    lis, par = str(tmp_path / "s.lis"), str(tmp_path / "p.txt")
    (tmp_path / "s.lis").write_bytes(struct.pack("<12fi2fffq", *lim, 2, 1.0, ratio, 0.0, 0.0, n) + rec.tobytes())
    (tmp_path / "p.txt").write_text(f"Nx1 = 16\nNx2 = 16\nNx3 = 16\nZ = {0.02 * (1 + ratio)}\nfour_pi_G_par = {g!r}\nknn = 32\nhop = 16\nnum_threads = 4\n")
    f = built.Finder(0)
    cat = f.find_clumps(built.Snapshot(lis), built.params(par))
    o = oracle.Oracle(lis, par, threads=4, pow_mode=1)
    o.find()
    pn, _, _ = o.clumps()
    assert nh > 27 and len(pn)
    assert cat.summary().strip() == o.summary().strip()
    for d in ("here", "there"):
        (tmp_path / d).mkdir()
    cat.write_peaks(str(tmp_path / "here" / "res.txt"))
    o.write_outputs(str(tmp_path / "there" / "res.txt"))
    names = sorted(e.name for e in (tmp_path / "there").iterdir() if e.name.startswith("peaks_at_"))
    assert names
    for x in names:
        assert (tmp_path / "here" / x).read_bytes() == (tmp_path / "there" / x).read_bytes(), x
    f.close()
