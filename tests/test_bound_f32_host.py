"""The FP32 boundness tests of the rebinding against FP64, on the CPU (no GPU).

bound_hilo and bound_hilo_fast (bound_f32.cuh) may say -1 (too close to call), never another answer
than the FP64 test of src/tree.hpp:4686-4694: for candidates from the box's extent down to 10^-11 of
it from the clump's centre, plain and sheared points, masses from 10^-8 to 100 times the clump's,
energies at every distance from zero and velocities far below the shear's. The fast reciprocal and
reciprocal root are off by up to two units in the last place, in either direction.
"""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r"""
#define __device__
#define __forceinline__ inline
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>
static std::mt19937_64 rng(13);
static float off(float v) {  // by up to two units in the last place
    for (int k = (int)(rng() % 5) - 2; k; k += k < 0 ? 1 : -1) v = std::nextafter(v, k < 0 ? -INFINITY : INFINITY);
    return v;
}
static float __fdividef(float a, float b) { return off(a / b); }
static float rsqrtf(float x) { return off((float)(1.0 / std::sqrt((double)x))); }
#include "bound_f32.cuh"
using namespace plan;

static double u(double a, double b) { return a + (b - a) * ((double)(rng() >> 11) * 0x1p-53); }
static double lg(double a, double b) { return std::exp(u(std::log(a), std::log(b))); }
static void split(double x, float &h, float &l) { h = (float)x; l = (float)(x - (double)h); }

int main() {
    long n = 0, bad = 0, unsure = 0, said[2] = {0, 0};
    for (int i = 0; i < 4000000; ++i) {
        const double G = lg(1e-6, 1e2), shear = i % 3 ? 1.5 : 0.0, X = i % 4 ? 0.1 : 4.0;
        double S[7], p[3], v[3], dir[3], e[3], len = 0, el = 0, D2 = 0;
        S[6] = lg(1e-9, 1e-3);
        const double m = (double)(float)(S[6] * lg(1e-8, 1e2)), M = S[6] + m, D = X * lg(1e-11, 1.0);
        for (int d = 0; d < 3; ++d) {
            dir[d] = u(-1, 1);
            e[d] = u(-1, 1);
            len += dir[d] * dir[d];
            el += e[d] * e[d];
        }
        for (int d = 0; d < 3; ++d) {
            p[d] = (double)(float)u(-X, X);
            if (d == 1 && (i & 1)) p[d] = p[d] + 0.37 * X;  // a sheared ghost
            S[d] = p[d] + dir[d] / std::sqrt(len) * D;
            D2 += (S[d] - p[d]) * (S[d] - p[d]);
        }
        if (!(D2 > 0)) continue;
        // the relative velocity for which the energy is close to zero
        const double dx = S[0] - p[0];
        const double speed = std::sqrt(2.0 * M * G / std::sqrt(D2) * (1.0 + u(-1.0, 1.0) * std::pow(10.0, -(double)(rng() % 9))));
        for (int d = 0; d < 3; ++d) {
            v[d] = (double)(float)u(-1e-2, 1e-2);
            S[3 + d] = v[d] + e[d] / std::sqrt(el) * speed + (d == 1 ? shear * dx : 0.0);
        }
        const double ex = (S[3] - 0.0 * dx) - v[0], ey = (S[4] - shear * dx) - v[1], ez = (S[5] - 0.0 * dx) - v[2];
        const double E = 0.5 / M * (ex * ex + ey * ey + ez * ez) - G / std::sqrt(D2);
        float sh[6], sl[6], Mf, l;
        for (int k = 0; k < 6; ++k) split(S[k], sh[k], sl[k]);
        split(S[6], Mf, l);
        CandF f;
        for (int d = 0; d < 3; ++d) {
            split(p[d], f.ph[d], f.pl[d]);
            split(v[d], f.vh[d], f.vl[d]);
        }
        split(m, f.w, l);
        for (int way = 0; way < 3; ++way) {
            // the candidate's own limits, and those of the whole box
            const BoundLimits own = bound_limits(f, (float)shear), all = bound_limits((float)(1.4 * X), 2e-2f, (float)shear);
            const int got = way == 0 ? bound_hilo(f, Mf, sh, sl, (float)G, (float)shear, own)
                                     : bound_hilo_fast(f, Mf, sh, sl, (float)G, (float)shear, way == 1 ? own : all);
            ++n;
            if (got < 0) ++unsure;
            else if (got == (E < 0)) ++said[got];
            else if (bad++ < 8) printf("distance %g in %g, shear %g, speed %g: %d, energy %g\n", std::sqrt(D2), X, shear, speed, got, E);
        }
    }
    printf("%ld states, %ld unsure, %ld wrong, unbound %ld, bound %ld\n", n, unsure, bad, said[0], said[1]);
    return bad || !said[0] || !said[1];
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
