"""The FP32 unbinding test against FP64 over all shares of a clump's mass, on the CPU (no GPU).

ub_test (unbind_f32.cuh) may say -1 (too close to call), never another answer than the FP64 test
of src/tree.hpp:4615-4674: for members of 10^-8 to 99.9% of the mass, distances and velocities from
the clump's whole extent down to 10^-8 of the coordinates, strong and no shear, energies at every
distance from zero. The fast reciprocal and reciprocal root are off by up to two units in the last
place here, in either direction, as on the device.
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
static std::mt19937_64 rng(11);
static float off(float v) {  // by up to two units in the last place
    for (int k = (int)(rng() % 5) - 2; k; k += k < 0 ? 1 : -1) v = std::nextafter(v, k < 0 ? -INFINITY : INFINITY);
    return v;
}
static float __fdividef(float a, float b) { return off(a / b); }
static float rsqrtf(float x) { return off((float)(1.0 / std::sqrt((double)x))); }
#include "unbind_f32.cuh"
using namespace plan;

static double u(double a, double b) { return a + (b - a) * ((double)(rng() >> 11) * 0x1p-53); }
static double lg(double a, double b) { return std::exp(u(std::log(a), std::log(b))); }
static void split(double x, float &h, float &l) { h = (float)x; l = (float)(x - (double)h); }

int main() {
    long n = 0, bad = 0, unsure = 0, said[2] = {0, 0}, light = 0, light_unsure = 0;
    for (int i = 0; i < 6000000; ++i) {
        const double G = lg(1e-6, 1e2), shear = i % 3 ? 1.5 : 0.0;
        double S[7], p[3], v[3];
        S[6] = lg(1e-9, 1e-3);
        const double left = i % 2 ? lg(1e-3, 1.0) : 1.0 - lg(1e-8, 0.5);  // of the mass, when the member is gone
        const double m = (double)(float)(S[6] * (1.0 - left)), M = S[6], Mr = M - m;
        if (!(Mr > 0) || !(m > 0)) continue;
        const double D = 0.1 * lg(1e-8, 1.0);
        double dir[3], len = 0;
        for (int d = 0; d < 3; ++d) { S[d] = u(-0.1, 0.1); dir[d] = u(-1, 1); len += dir[d] * dir[d]; }
        for (int d = 0; d < 3; ++d) p[d] = (double)(float)(S[d] + dir[d] / std::sqrt(len) * D);
        // the relative velocity for which the energy is close to zero
        double dx[3], D2 = 0;
        for (int d = 0; d < 3; ++d) { dx[d] = (S[d] * M - p[d] * m) / Mr - p[d]; D2 += dx[d] * dx[d]; }
        if (!(D2 > 0)) continue;
        const double speed = std::sqrt(2.0 * M * G / std::sqrt(D2) * (1.0 + u(-1.0, 1.0) * std::pow(10.0, -(double)(rng() % 9))));
        double e[3], el = 0;
        for (int d = 0; d < 3; ++d) { e[d] = u(-1, 1); el += e[d] * e[d]; }
        for (int d = 0; d < 3; ++d) {
            const double want = e[d] / std::sqrt(el) * speed + (d == 1 ? shear * dx[0] : 0.0);  // (com' - v) here
            v[d] = (double)(float)u(-1e-2, 1e-2);
            S[3 + d] = v[d] + want * Mr / M;
        }
        // as the reference writes it
        double c[6];
        for (int d = 0; d < 3; ++d) {
            c[d] = (S[d] * M - p[d] * m) / Mr;
            c[3 + d] = (S[3 + d] * M - v[d] * m) / Mr;
        }
        const double ddx = c[0] - p[0];
        const double ex = (c[3] - 0.0 * ddx) - v[0], ey = (c[4] - shear * ddx) - v[1], ez = (c[5] - 0.0 * ddx) - v[2];
        const double E = 0.5 / M * (ex * ex + ey * ey + ez * ez) -
                         G / std::sqrt(ddx * ddx + (c[1] - p[1]) * (c[1] - p[1]) + (c[2] - p[2]) * (c[2] - p[2]));
        float sf[13], l;
        for (int k = 0; k < 6; ++k) split(S[k], sf[k], sf[6 + k]);
        split(S[6], sf[12], l);
        UbCand f;
        for (int d = 0; d < 3; ++d) { split(p[d], f.ph[d], f.pl[d]); split(v[d], f.vh[d], f.vl[d]); }
        split(m, f.w, l);
        f.lim = bound_limits(f, (float)shear);
        const int got = ub_test(f, sf, (float)G, (float)shear);
        ++n;
        light += left > 0.9;
        if (got < 0) { ++unsure; light_unsure += left > 0.9; }
        else if (got != (E > 0)) { if (bad++ < 8) printf("mass left %g of 1, D %g, shear %g: %d, energy %g of %g\n", left, D, shear, got, E, 0.5 / M * (ex * ex + ey * ey + ez * ez)); }
        else ++said[got];
    }
    printf("%ld states, %ld unsure (%ld of %ld light members), %ld wrong, bound %ld, unbound %ld\n", n, unsure, light_unsure, light, bad, said[0], said[1]);
    return bad || !said[0] || !said[1] || light_unsure * 2 > light;
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
