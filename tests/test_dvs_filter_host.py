"""The FP32 node classes of --Density_Vs_Scale against the FP64 ones, on the CPU (no GPU).

dvs_class_f may say -1 (too close to call), never another class than dvs_class: over boxes of
several sizes and aspect ratios, shears of either sign up to many box lengths, balls from half a
cell to the box, nodes from the root to single points, and pairs placed at the edges of every
test (the periodic limits, the sphere through the node's corners, its faces).
"""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r"""
#include <cstdio>
#include <random>
#include "dvs.cuh"
using namespace plan;

int main() {
    std::mt19937_64 rng(5);
    auto u = [&](double a, double b) { return a + (b - a) * ((double)(rng() >> 11) * 0x1p-53); };
    long n = 0, unsure = 0, bad = 0, seen[3] = {0, 0, 0};
    for (int box = 0; box < 24; ++box) {
        DvsParams p{};
        const double L = box % 3 == 0 ? 0.2 : box % 3 == 1 ? 8.0 : 1e-3;
        for (int d = 0; d < 3; ++d) {
            p.box_length[d] = L * (box % 2 ? 1.0 : 0.5 + 0.5 * (d == 0));
            p.box_center[d] = box % 4 == 3 ? 0.3 * L : 0.0;
            p.box_min[d] = p.box_center[d] - p.box_length[d] / 2;
            p.box_max[d] = p.box_center[d] + p.box_length[d] / 2;
            p.cell_length[d] = p.box_length[d] / 32;
        }
        p.box_half_width0 = p.box_length[0] / 2;
        p.max_half_width = L / 2;
        p.shear_speed = 1.5 * p.box_length[0];
        p.mass_per_particle0 = 1e-8;
        const double times[6] = {0.0, 0.37, 1.0, 12.25, -0.6, 700.0};
        DvsGeom g;
        std::vector<double> xs, ys, zs;
        if (dvs_setup(p, times[box % 6], p.box_min[2], p.box_max[2], g, xs, ys, zs)) return 3;
        const DvsGeomF gf = dvs_geom_f(g, 2 * L + std::fabs(p.box_center[0]));
        for (int i = 0; i < 200000; ++i) {
            const int lev = (int)(rng() % g.nlev);
            const double r = g.radius[lev], hw = L * std::pow(0.5, (double)(rng() % 22));
            double c[3], nc[3];
            for (int d = 0; d < 3; ++d) {
                c[d] = p.box_center[d] + u(-0.52, 0.52) * p.box_length[d];
                nc[d] = p.box_center[d] + u(-1.0, 1.0) * p.box_length[d];
            }
            const int edge = (int)(rng() % 6);
            const double jit = u(-1.0, 1.0) * std::pow(10.0, -(double)(rng() % 17)) * L;
            const int ax = (int)(rng() % 3);
            if (edge >= 2)
                for (int d = 0; d < 3; ++d) nc[d] = c[d] + u(-1.0, 1.0) * (r + 2 * hw);
            if (edge == 1) nc[ax] = c[ax] + (rng() & 1 ? 1 : -1) * g.maxd[lev][ax == 2 ? 1 : ax] + jit;  // the periodic limit
            if (edge == 3) for (int d = 0; d < 3; ++d) nc[d] = c[d] + (d == ax ? r + hw : 0.0) + jit;  // a face
            if (edge == 4) for (int d = 0; d < 3; ++d) nc[d] = c[d] + (d == ax ? r + hw * g.diag : 0.0) + jit;
            if (edge == 5) for (int d = 0; d < 3; ++d) nc[d] = c[d] + (r / g.diag - hw * g.diag) + jit;  // just inside
            if (rng() % 50 == 0) c[0] = 0.0;
            const int want = dvs_class(c, nc, hw, r, g.maxd[lev], g);
            const float cf[3] = {(float)c[0], (float)c[1], (float)c[2]}, nf[3] = {(float)nc[0], (float)nc[1], (float)nc[2]};
            const int got = dvs_class_f(cf, nf, (float)hw, lev, gf);
            ++n;
            if (got < 0) ++unsure;
            else if (got != want) { if (bad++ < 5) printf("box %d lev %d edge %d: %d, want %d\n", box, lev, edge, got, want); }
            else if (box % 6 != 5) ++seen[want];
        }
    }
    printf("%ld pairs, %ld unsure, %ld wrong, classes %ld %ld %ld\n", n, unsure, bad, seen[0], seen[1], seen[2]);
    return bad || !seen[0] || !seen[1] || !seen[2] || unsure * 2 > n;
}
"""


def test_fp32_node_class_never_contradicts_fp64(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "plan_gb300" / "csrc"), str(tmp_path / "h.cpp"), "-o",
                    str(tmp_path / "h")], check=True)
    r = subprocess.run([str(tmp_path / "h")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    print(r.stdout)
