"""The queue items of the pair pass, and the energies where its fast rows do not apply.

On the CPU, every item of every row tile count decodes to a strip of its own and all strips
cover the upper triangle once. On the GPU, groups whose sizes lie at the edges of the tiles, the
size classes and the strips, with ordinary masses, coincident particles, negative and zero
masses, and coordinates whose squared distances underflow, against FP64 direct sums.
"""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HARNESS = r"""
#include <cstdio>
#include <vector>
#include "energy.cuh"
using namespace plan;
int main() {
    for (uint64_t T = 1; T < 150; ++T) {
        std::vector<int> seen(T * T, 0);
        for (uint64_t i = 0; i < strip_items(T); ++i) {
            uint64_t ti, tj, te;
            strip_of_item(i, T, ti, tj, te);
            if (ti >= T || tj < ti || te <= tj || te > T || te - tj > strip_of(T)) { printf("T %lu item %lu\n", (unsigned long)T, (unsigned long)i); return 1; }
            for (uint64_t k = tj; k < te; ++k) ++seen[ti * T + k];
        }
        for (uint64_t a = 0; a < T; ++a)
            for (uint64_t b = 0; b < T; ++b)
                if (seen[a * T + b] != (b >= a ? 1 : 0)) { printf("T %lu tile %lu %lu\n", (unsigned long)T, (unsigned long)a, (unsigned long)b); return 1; }
    }
    return 0;
}
"""


def test_items_cover_the_triangle(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "plan_gb300" / "csrc"), str(tmp_path / "h.cpp"), "-o", str(tmp_path / "h")],
                   check=True)
    r = subprocess.run([str(tmp_path / "h")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _direct(x, m, squares32=False):
    """Sum and size of the pair terms, and the coincident pairs; squares32: the squared distances
    in FP32, as the pass forms them, where they are so small that this decides their value."""
    m = m.astype(np.float64)
    tot, size, zeros = 0.0, 0.0, 0
    for i in range(len(m) - 1):
        if squares32:
            q = (x[i + 1:] - x[i]) ** 2
            d = np.sqrt(((q[:, 0] + q[:, 1]) + q[:, 2]).astype(np.float64))
        else:
            d = np.sqrt(((x[i + 1:].astype(np.float64) - x[i]) ** 2).sum(1))
        near = d == 0
        zeros += int(near.sum())
        t = m[i] * m[i + 1:][~near] / d[~near]
        tot += t.sum()
        size += np.abs(t).sum()
    return tot, size, zeros


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "coincident", "signed", "tiny"])
def test_energies_at_the_edges(kind, built):
    rng = np.random.default_rng(3)
    sizes = [0, 1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1025, 8191, 8193]
    if kind != "plain":
        sizes = sizes[:-2]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    n = int(off[-1])
    pos = rng.normal(scale=1e-3, size=(n, 3)).astype(np.float32)
    mass = (4e-8 * (0.5 + rng.random(n))).astype(np.float32)
    if kind == "coincident":
        for a, b in zip(off[:-1].astype(int), off[1:].astype(int)):
            if b - a >= 31:
                pos[b - 1] = pos[a]
                pos[a + 7] = pos[a + 3]
                pos[a + 8] = pos[a + 3]
    if kind == "signed":
        mass[::3] *= -1
        mass[1::5] = 0
    if kind == "tiny":
        pos[::2] *= np.float32(1e-19)
    vel = np.zeros((n, 3), np.float32)
    p = built.params()
    built.lib().plan_params_derive(C.byref(p))
    f = built.Finder(0)
    ek, ep, zeros = f.group_energies(pos, vel, mass, off, p)
    again = f.group_energies(pos, vel, mass, off, p)
    f.close()
    np.testing.assert_array_equal(ep, again[1])
    want_zeros = 0
    for g, (a, b) in enumerate(zip(off[:-1].astype(int), off[1:].astype(int))):
        w, size, z = _direct(pos[a:b], mass[a:b], kind == "tiny")
        want_zeros += z
        # the stated 1e-6 of the sum of the terms' magnitudes
        assert abs(ep[g] + p.grav_constant * w) <= 1e-6 * p.grav_constant * size, (sizes[g], ep[g], w)
    assert zeros == want_zeros
