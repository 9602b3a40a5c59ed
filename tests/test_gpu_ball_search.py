"""The merge sweeps' two ball searches give one catalogue.

Up to a limit the clumps around a clump are found by brute force in FP32 with the nodes' FP64
tests near the ball's surface, above it by walking the clump tree in FP64. PLAN_BRUTE_CLUMPS moves
the limit, on snapshots of up to 1,890 clumps with many merges, plain and sheared.
"""
from __future__ import annotations

import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["w1_20k", "w1_20k_sheared", "w1_50k_spline", "config1_262k"])
def test_same_catalogue(name, built, case_dir, tmp_path, monkeypatch):
    c = case_dir(name)
    monkeypatch.setenv("PLAN_BRUTE_CLUMPS", "")
    got = []
    for limit in ("0", "4000000000", ""):  # the walk alone, brute force alone, the limit as it is
        monkeypatch.setenv("PLAN_BRUTE_CLUMPS", limit)
        f = built.Finder(0)
        cat = f.find_clumps(built.Snapshot(c["lis"]), built.params(c["param"]))
        out = tmp_path / f"limit{limit}"
        out.mkdir()
        cat.write_peaks(str(out / "res.txt"))
        got.append((cat.summary(), cases.find_peaks_file(out).read_bytes(), cat.clumps()))
        f.close()
    assert got[0] == got[1] == got[2]
