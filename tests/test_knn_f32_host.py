"""The FP32 node tests and distances of the neighbour searches against FP64, on the CPU (no GPU).

f_contained and f_intersects (knn_f32.cuh) may say -1 (too close to call), never another answer
than the FP64 tests of src/tree.hpp:3001-3049: for nodes from the root to single points and
spheres from far below a node's size to far above it, at random and placed at the edges of every
comparison, among them spheres that end just before or behind the faces of a node many times
their size, in root boxes of half widths from 0.01 to 10^6. f_lo and f_hi must enclose the FP64
squared distance of a position as close as 10^-12 of the box to a sheared point.
"""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r"""
#define __device__
#define __forceinline__ inline
struct float4 { float x, y, z, w; };
#include <cmath>
#include <cstdio>
#include <random>
#include "knn_f32.cuh"
using namespace plan;

static float4 hi4(const double *p, double w) { return {(float)p[0], (float)p[1], (float)p[2], (float)w}; }
static float4 lo4(const double *p, double w) {
    const float4 h = hi4(p, w);
    return {(float)(p[0] - (double)h.x), (float)(p[1] - (double)h.y), (float)(p[2] - (double)h.z), (float)(w - (double)h.w)};
}

static bool contained(const double *c, double hw, const double *q, double r) {
    const double t = hw * 1.7320508075688772;
    double s = 0;
    for (int d = 0; d < 3; ++d) s = s + (std::fabs(c[d] - q[d]) + t) * (std::fabs(c[d] - q[d]) + t);
    return s < r * r;
}
static bool intersects(const double *c, double hw, const double *q, double r) {
    double c2c = 0;
    for (int d = 0; d < 3; ++d) c2c = c2c + (c[d] - q[d]) * (c[d] - q[d]);
    const double t = hw * 1.7320508075688772 + r;
    if (c2c > t * t) return false;
    if (c2c < r || c2c < hw) return true;
    double m2 = 0;
    for (int d = 0; d < 3; ++d) {
        const double lo = c[d] - hw, hi = c[d] + hw;
        if (q[d] < lo) m2 = m2 + (q[d] - lo) * (q[d] - lo);
        else if (q[d] > hi) m2 = m2 + (q[d] - hi) * (q[d] - hi);
    }
    return m2 <= r * r;
}

int main() {
    std::mt19937_64 rng(7);
    auto u = [&](double a, double b) { return a + (b - a) * ((double)(rng() >> 11) * 0x1p-53); };
    long bad = 0, n = 0, unsure = 0, said[2][2] = {{0, 0}, {0, 0}};
    const double boxes[] = {0.125, 0.013, 4.0, 0.7, 300.0, 1e6};  // half widths of the root
    for (double X : boxes) {
        const Tol tol = tol_of(X);
        for (int i = 0; i < 1000000; ++i) {
            // a node of the tree: the root's corners halved
            const int depth = (int)(rng() % 20);
            const double hw = std::ldexp(X, -depth);
            double c[3], q[3];
            for (int d = 0; d < 3; ++d) c[d] = depth ? -X + hw * (1.0 + 2.0 * (double)(rng() & ((1ull << depth) - 1))) : 0.0;
            // the sphere: any size against the node's; its centre an FP64 position
            const double r = hw * std::exp(u(std::log(1e-5), std::log(1e3)));
            const double jit = u(-1.0, 1.0) * std::pow(10.0, -(double)(rng() % 14));
            const int edge = (int)(rng() % 5), ax = (int)(rng() % 3);
            for (int d = 0; d < 3; ++d) q[d] = edge == 0 ? u(-1.0, 1.0) * X : c[d] + u(-1.0, 1.0) * hw;
            const double side = rng() & 1 ? 1.0 : -1.0;
            if (edge >= 1 && edge <= 2) q[ax] = c[ax] + side * (hw + r * (1.0 + jit));         // tangent to a face
            if (edge == 2) {                                                                   // to an edge of the node
                const int ay = (ax + 1) % 3;
                const double a = u(0.0, 1.5707);
                q[ax] = c[ax] + side * (hw + r * std::cos(a) * (1.0 + jit));
                q[ay] = c[ay] - side * (hw + r * std::sin(a) * (1.0 + jit));
            }
            if (edge == 3) for (int d = 0; d < 3; ++d) q[d] = c[d] + (d == ax ? side * (hw * 1.7320508075688772 + r) * (1.0 + jit) : 0.0);
            if (edge == 4)  // the sphere through the containment test's corner
                for (int d = 0; d < 3; ++d) q[d] = c[d] + side * (r / 1.7320508075688772 - hw * 1.7320508075688772) * (1.0 + jit);
            const float4 nh = hi4(c, hw), nl = lo4(c, hw), qh = hi4(q, 0), ql = lo4(q, 0);
            const int cf = f_contained(nh, nl, qh, ql, (float)r, tol), mf = f_intersects(nh, nl, qh, ql, (float)r, tol);
            const int cd = contained(c, hw, q, r), md = intersects(c, hw, q, r);
            ++n;
            if (cf < 0 || mf < 0) ++unsure;
            if (cf >= 0) ++said[0][cf];
            if (mf >= 0) ++said[1][mf];
            if ((cf >= 0 && cf != cd) || (mf >= 0 && mf != md)) {
                if (bad++ < 8) printf("box %g hw %g r %g edge %d: contained %d (%d), met %d (%d)\n", X, hw, r, edge, cf, cd, mf, md);
            }
            // a point near a query: a record's float position, moved by a shear as ghosts are
            double p[3], near[3], s = 0;
            const double by = X * std::pow(10.0, -(double)(rng() % 13));
            for (int d = 0; d < 3; ++d) p[d] = (double)(float)(u(-1.0, 1.0) * X);
            if (rng() & 1) p[1] = p[1] + u(-0.5, 0.5) * X;
            for (int d = 0; d < 3; ++d) {
                near[d] = p[d] + u(-1.0, 1.0) * by;
                s = s + (near[d] - p[d]) * (near[d] - p[d]);
            }
            const float v = f_dr2(hi4(near, 0), lo4(near, 0), hi4(p, 0), lo4(p, 0));
            if (!((double)f_lo(v, tol) <= s && s <= (double)f_hi(v, tol))) {
                if (bad++ < 8) printf("box %g: distance %g not in [%g, %g]\n", X, s, (double)f_lo(v, tol), (double)f_hi(v, tol));
            }
        }
    }
    printf("%ld pairs, %ld unsure, %ld wrong; contained %ld/%ld, met %ld/%ld\n", n, unsure, bad, said[0][0], said[0][1], said[1][0], said[1][1]);
    return bad != 0 || unsure * 2 > n || !said[0][0] || !said[0][1] || !said[1][0] || !said[1][1];
}
"""


def test_fp32_never_contradicts_fp64(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "plan_gb300" / "csrc"), str(tmp_path / "h.cpp"), "-o",
                    str(tmp_path / "h")], check=True)
    r = subprocess.run([str(tmp_path / "h")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    print(r.stdout)
