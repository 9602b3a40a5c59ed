"""Whole finds at sizes around the limits of the small kernels, against the oracle.

A scan of up to 16,384 values is one block: snapshots of 16,383 to 16,385 particles (one value
per leaf flag). Clumps of up to 512 members sum in a warp, larger ones in a block: spheres of 500
to 525 particles and one of 1,537. The neighbouring clumps of a merge sweep are found by brute
force while there are few, which all of these use.
"""
from __future__ import annotations

import struct

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _spheres(n: int, seed: int):
    rec, g = cases._records(cases.BY_NAME["w1_20k"])
    rng = np.random.default_rng(seed)
    rec = np.resize(rec, n)
    rec["pos"] = rng.uniform(-0.099, 0.099, (n, 3)).astype(np.float32)
    rec["vel"] = (1e-4 * rng.standard_normal((n, 3))).astype(np.float32)
    rec["id_in_run"] = np.arange(n)
    at = 0
    for i, m in enumerate([1537, *range(500, 526)]):
        x = rng.standard_normal((m, 3))
        x *= (0.002 * rng.random((m, 1)) ** (2 / 3)) / np.linalg.norm(x, axis=1, keepdims=True)
        c = np.array([i % 3 - 1, i // 3 % 3 - 1, i // 9 - 1]) * 0.06 + rng.uniform(-0.005, 0.005, 3)
        rec["pos"][at:at + m] = (c + x).astype(np.float32)
        at += m
    return rec[rng.permutation(n)], g


@pytest.mark.parametrize("n", [16383, 16384, 16385])
def test_find_matches_oracle(n, built, tmp_path):
    import oracle

    rec, g = _spheres(n, n)
    lim = [-0.1, 0.1] * 6
    lis, par = str(tmp_path / "s.lis"), str(tmp_path / "p.txt")
    (tmp_path / "s.lis").write_bytes(struct.pack("<12fi1fffq", *lim, 1, 1.0, 0.0, 0.0, n) + rec.tobytes())
    (tmp_path / "p.txt").write_text(f"Nx1 = 16\nNx2 = 16\nNx3 = 16\nZ = 0.02\nfour_pi_G_par = {g!r}\nknn = 32\nhop = 16\nnum_threads = 4\n")
    f = built.Finder(0)
    cat = f.find_clumps(built.Snapshot(lis), built.params(par))
    o = oracle.Oracle(lis, par, threads=4, pow_mode=1)
    o.find()
    pn, _, _ = o.clumps()
    assert pn[:, 1].min() <= 512 < pn[:, 1].max()
    assert cat.summary().strip() == o.summary().strip()
    for d in ("here", "there"):
        (tmp_path / d).mkdir()
    cat.write_peaks(str(tmp_path / "here" / "res.txt"))
    o.write_outputs(str(tmp_path / "there" / "res.txt"))
    for e in (tmp_path / "there").iterdir():
        if (tmp_path / "here" / e.name).exists():
            assert (tmp_path / "here" / e.name).read_bytes() == e.read_bytes(), e.name
    assert list((tmp_path / "here").iterdir())
    f.close()
