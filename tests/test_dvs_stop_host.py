"""When a warp of --Density_Vs_Scale stops counting, on the CPU (no GPU).

The largest count of a radius rises while a warp counts the points of its leaves. The 32 lanes
run here as threads whose every look at that word finds another value; they must all take part
in the same sums, and a count that is not cut short must be the plain one.
"""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r"""
#include <atomic>
#include <barrier>
#include <cstdio>
#include <memory>
#include <random>
#include <thread>
#include <vector>
#include "dvs.cuh"
using namespace plan;

struct Shared {
    std::barrier<> turn{32};
    uint32_t value[32];
    std::atomic<uint32_t> looks{0}, gone{0};
    std::atomic<int> torn{0};  // a sum or broadcast that lacked a lane
};

struct LaneWarp {
    Shared *s;
    uint32_t at, top;
    uint32_t lane() const { return at; }
    uint32_t load(const uint32_t *word) const { return s->looks++ % 3 == 0 ? *word : top; }
    template <class F> uint32_t all(uint32_t v, F f) const {
        s->value[at] = v;
        s->turn.arrive_and_wait();
        if (s->gone) s->torn = 1;
        const uint32_t r = f();
        s->turn.arrive_and_wait();
        return r;
    }
    uint32_t first(uint32_t v) const { return all(v, [&] { return s->value[0]; }); }
    uint32_t sum(uint32_t v) const {
        return all(v, [&] {
            uint32_t t = 0;
            for (uint32_t x : s->value) t += x;
            return t;
        });
    }
};

struct Leaves {
    std::vector<uint32_t> b, e;
    uint32_t begin(uint32_t n) const { return b[n]; }
    uint32_t end(uint32_t n) const { return e[n]; }
};

int main() {
    std::mt19937 rng(3);
    int bad = 0;
    for (int trial = 0; trial < 60; ++trial) {
        Leaves t;
        std::vector<uint32_t> leaves;
        uint32_t at = 0, points = 0, want = 0;
        const uint32_t nleaf = rng() % 12;
        for (uint32_t k = 0; k < nleaf; ++k) {
            const uint32_t n = rng() % 65;
            t.b.push_back(at);
            t.e.push_back(at += n);
            leaves.push_back(k);
            points += n;
        }
        auto near = [](uint32_t p) { return p % 3 != 1; };
        for (uint32_t p = 0; p < at; ++p) want += near(p);
        // the word another warp raises: 0, or enough to stop at once, or on the way
        const uint32_t base = 5, low = 0, high = base + (trial % 3 == 0 ? points : points / 2);
        for (int stop = 0; stop < 2; ++stop) {
            Shared s;
            uint32_t inside[32], partial[32];
            std::vector<std::thread> lanes;
            for (uint32_t l = 0; l < 32; ++l)
                lanes.emplace_back([&, l] {
                    inside[l] = base;
                    partial[l] = points;
                    dvs_count_leaves(LaneWarp{&s, l, high}, t, leaves.data(), nleaf, stop ? &low : nullptr, inside[l], partial[l], near);
                    s.gone++;
                    s.turn.arrive_and_drop();
                });
            for (auto &x : lanes) x.join();
            bool same = true;
            for (uint32_t l = 1; l < 32; ++l) same = same && inside[l] == inside[0] && partial[l] == partial[0];
            if (s.torn || !same) { ++bad; printf("trial %d stop %d: lanes disagree\n", trial, stop); }
            if (!stop && (inside[0] != base + want || partial[0] != 0)) { ++bad; printf("trial %d: %u points, want %u\n", trial, inside[0] - base, want); }
            if (stop && (inside[0] > base + want || inside[0] + partial[0] < base + want)) { ++bad; printf("trial %d: bounds\n", trial); }
        }
    }
    return bad != 0;
}
"""


def test_lanes_stop_together(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++20", "-pthread", "-I", str(ROOT / "plan_gb300" / "csrc"), str(tmp_path / "h.cpp"), "-o",
                    str(tmp_path / "h")], check=True)
    r = subprocess.run([str(tmp_path / "h")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
