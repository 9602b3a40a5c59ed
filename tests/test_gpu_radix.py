"""The stable 96-bit radix sort (radix_sort.cu) on its own, around each of its ways.

One block up to a tile of 4,096 keys, staged tiles above it; from 2^18 keys on, where few keys are
expected to share their upper words, the lowest word left to runs, with runs of 2, 16, 17 and 1,000
equal upper words (more than 16 send the sort through every digit). Keys that differ in one digit
only, in none, or under a mask; against a stable sort on the host, payload and all.
"""
from __future__ import annotations

import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "plan_gb300" / "csrc"

DEVICE = r"""
#include <algorithm>
#include <cstdio>
#include <numeric>
#include <random>
#include <vector>
#include "sort.h"
namespace plan { int set_cuda_error(cudaError_t, const char *, const char *, int) { return 5; } }

struct K { uint32_t w[3]; };

int main() {
    std::mt19937 rng(2);
    const uint32_t sizes[] = {0, 1, 2, 31, 257, 4095, 4096, 4097, 8192, 100003, (1u << 18) - 1, 1u << 18, (1u << 18) + 4097, 1000003};
    int bad = 0;
    for (uint32_t n : sizes)
        for (int kind = 0; kind < 9; ++kind) {
            if (n < 8192 && kind >= 5) continue;
            std::vector<K> k(n);
            for (auto &x : k) x = K{{(uint32_t)rng(), (uint32_t)rng(), (uint32_t)rng()}};
            const uint32_t mask = kind == 4 ? 0x0f0u : 0xfffu;  // the middle word's digits
            if (kind == 1) for (auto &x : k) x.w[0] = 7, x.w[1] = x.w[1] & 0xff00u, x.w[2] = 9;  // one digit
            if (kind == 2) for (auto &x : k) x = K{{1, 2, 3}};                                    // none
            if (kind == 3) for (auto &x : k) x.w[2] %= 3, x.w[1] = 0, x.w[0] %= 5;               // a few values
            const uint32_t run = kind == 5 ? 2 : kind == 6 ? 16 : kind == 7 ? 17 : 1000;
            if (kind >= 5)
                for (uint32_t at = 100; at + 2 * run < n; at += n / 7)
                    for (uint32_t j = 1; j < run; ++j) {  // equal upper words, lowest ones that repeat too
                        k[at + j].w[1] = k[at].w[1];
                        k[at + j].w[2] = k[at].w[2];
                        k[at + j].w[0] %= 5;
                    }
            if (kind >= 5) std::shuffle(k.begin(), k.end(), rng);
            std::vector<uint32_t> order(n);
            std::iota(order.begin(), order.end(), 0u);
            auto key = [&](const K &x, int w) { return mask == 0xfffu || w == 1 ? x.w[w] : 0u; };
            std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
                for (int w = 2; w >= 0; --w)
                    if (key(k[a], w) != key(k[b], w)) return key(k[a], w) < key(k[b], w);
                return false;
            });
            for (int few = 0; few < 2; ++few) {
                std::vector<uint32_t> h(4 * (size_t)n + 4);
                for (uint32_t i = 0; i < n; ++i) {
                    for (int w = 0; w < 3; ++w) h[w * (size_t)n + i] = k[i].w[w];
                    h[3 * (size_t)n + i] = i;
                }
                uint32_t *d;
                void *scr;
                const size_t sb = plan::radix_sort96_scratch_bytes(n);
                cudaMalloc(&d, h.size() * 4);
                cudaMalloc(&scr, sb);
                cudaMemcpy(d, h.data(), h.size() * 4, cudaMemcpyHostToDevice);
                const int rc = plan::radix_sort96(d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n, n, scr, sb, 0, mask, few);
                if (rc || cudaMemcpy(h.data(), d, h.size() * 4, cudaMemcpyDeviceToHost) != cudaSuccess) { printf("cuda error\n"); return 2; }
                long differ = 0;
                for (uint32_t i = 0; i < n; ++i) {
                    const uint32_t o = order[i];
                    differ += h[3 * (size_t)n + i] != o;
                    for (int w = 0; w < 3; ++w) differ += h[w * (size_t)n + i] != k[o].w[w];
                }
                if (differ) { ++bad; printf("n %u kind %d few %d: %ld\n", n, kind, few, differ); }
                cudaFree(d);
                cudaFree(scr);
            }
        }
    return bad != 0;
}
"""


@pytest.mark.gpu
def test_radix_sort(tmp_path, built):
    from plan_gb300 import build as b

    (tmp_path / "d.cu").write_text(DEVICE)
    subprocess.run([str(b._cuda_home() / "bin" / "nvcc"), *b.ARCH, "-O3", "-std=c++17", f"-I{CSRC}", f"-I{ROOT / 'include'}",
                    str(tmp_path / "d.cu"), str(CSRC / "radix_sort.cu"), "-o", str(tmp_path / "d")], check=True)
    r = subprocess.run([str(tmp_path / "d")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
