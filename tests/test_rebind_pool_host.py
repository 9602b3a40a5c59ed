"""Room in the member pool for the rebinding loop's clumps (rebind_pool.cuh), on the CPU (no GPU).

A clump that accepts members and sorts them needs a segment for its members and the scanned points,
then a spare segment and the sort's records. Launches that find the pool full are repeated after a
compaction. Whatever is left of the pool then, the first call or sort must find room as long as
its bare needs fit: the launches would otherwise repeat without an end. Segments must not overlap,
and must hold what was asked for.
"""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r"""
#define __device__
#define __forceinline__ inline
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>
namespace plan {
constexpr uint32_t kNone = 0xffffffffu;
struct Pool {
    uint32_t *top;
    uint32_t cap;
};
inline uint32_t pool_try_alloc(const Pool &P, uint32_t n) {
    if ((uint64_t)*P.top + n > P.cap) return kNone;
    const uint32_t o = *P.top;
    *P.top += n;
    return o;
}
#include "rebind_pool.cuh"
}
using namespace plan;


int main() {
    std::mt19937 rng(9);
    long bad = 0, stops = 0, done = 0;
    for (int t = 0; t < 100000; ++t) {
        const uint32_t cap = 1000 + rng() % 2000000;
        uint32_t others = rng() % cap, top = 0;
        const Pool P{&top, cap};
        uint32_t m = 1 + rng() % (cap - others);
        std::vector<uint32_t> scanned(12), accepted(12);
        // each step: a call (its scanned points), and the sort if it accepts
        size_t step = 0;
        bool pending = false, stuck = false;
        auto draw = [&](size_t k) {
            scanned[k] = rng() % (m / 4 + 2);
            accepted[k] = scanned[k] && rng() % 4 ? 1 + rng() % scanned[k] : 0;
        };
        draw(0);
        while (step < 12 && !stuck) {
            // a launch: the members packed, the segments forgotten
            if (others + (uint64_t)m > cap) break;
            RbSeg g{};
            uint32_t o = others;
            top = others + m;
            const uint32_t packed = top;
            bool first = true;
            for (;; first = false) {
                if (!pending) {
                    if (step == 12) break;
                    const uint32_t a = rb_spare(P, g, m + scanned[step]);
                    if (a == kNone) {
                        if (first) stuck = true, bad += (uint64_t)packed + m + scanned[step] <= cap;
                        break;
                    }
                    if (g.spare_cap < m + scanned[step] || a + (uint64_t)g.spare_cap > cap) ++bad;
                    if (a < o + (uint64_t)m && o < a + (uint64_t)g.spare_cap) ++bad;  // over the members
                    if (accepted[step]) {
                        rb_switch(g, o);
                        o = a;
                        m += accepted[step];
                        pending = true;
                    }
                    if (++step < 12) draw(step);
                } else {
                    if (!rb_sort_room(P, g, m)) {
                        if (first) stuck = true, bad += packed + 3ull * m + 1 <= cap;
                        break;
                    }
                    if (g.spare_cap < m || g.buf_cap < 2 * m + 1) ++bad;
                    const uint64_t seg[3][2] = {{o, m}, {g.spare, g.spare_cap}, {g.buf, g.buf_cap}};
                    for (int i = 0; i < 3; ++i) {
                        if (seg[i][0] + seg[i][1] > cap) ++bad;
                        for (int j = 0; j < i; ++j)
                            if (seg[i][0] < seg[j][0] + seg[j][1] && seg[j][0] < seg[i][0] + seg[i][1]) ++bad;
                    }
                    const uint32_t r = g.spare;
                    rb_switch(g, o);
                    o = r;
                    pending = false;
                }
            }
            ++stops;
        }
        done += step == 12;
    }
    printf("%ld launches, %ld clumps done, %ld failures\n", stops, done, bad);
    return bad != 0 || !done;
}
"""


def test_first_step_finds_room(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "plan_gb300" / "csrc"), str(tmp_path / "h.cpp"), "-o", str(tmp_path / "h")],
                   check=True)
    r = subprocess.run([str(tmp_path / "h")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    print(r.stdout)
