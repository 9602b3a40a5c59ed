"""The exact ordered member sums (ordered_sum.cuh): bit for bit a left-to-right FP64 loop.

ordered_sum_chunk in one block per case against a sequential host loop, over lengths around the
chunk and row edges and over terms that reach every branch: sums that keep their binade, hover
around zero, meet ties of both parities in one row and across rows, zeros of both signs,
cancellation to zero, binade edges, terms far above and below the sum, subnormals, infinities.
"""
from __future__ import annotations

import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "plan_gb300" / "csrc"

DEVICE = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "ordered_sum.cuh"
using namespace plan;
constexpr int NS = 7;

__global__ void __launch_bounds__(256) k_sums(const double *x, uint32_t stride, const uint32_t *len, double *out, uint32_t *nloop) {
    uint32_t loops = 0;
    __shared__ __align__(16) double stage[NS * kSumStage];
    __shared__ uint2 steps[NS * kSumChunk];
    const uint32_t m = len[blockIdx.x];
    const double *base = x + (size_t)blockIdx.x * NS * stride;
    const int w = threadIdx.x >> 5;
    double acc = 0.0;
    for (uint32_t b = 0; b < m; b += kSumChunk) {
        const uint32_t k = b + threadIdx.x;
        for (int c = 0; c < NS; ++c) stage[c * kSumStage + sum_slot(threadIdx.x)] = k < m ? base[(size_t)c * stride + k] : 0.0;
        __syncthreads();
        if (w < NS) ordered_sum_chunk(stage + w * kSumStage, acc, steps + w * kSumChunk, &loops);
        __syncthreads();
    }
    if (w < NS && (threadIdx.x & 31) == 0) {
        out[blockIdx.x * NS + w] = acc;
        nloop[blockIdx.x * NS + w] = loops;
    }
}

int main() {
    std::mt19937_64 rng(11);
    const uint32_t lens[] = {0, 1, 7, 8, 9, 31, 255, 256, 257, 263, 511, 512, 513, 1000, 2047, 2500};
    const uint32_t stride = 2560;
    const int cases = 16 * 60;
    std::vector<uint32_t> len(cases);
    std::vector<double> x((size_t)cases * NS * stride, 0.0);
    auto uni = [&]() { return (double)(rng() >> 11) * 0x1p-53; };
    auto nrm = [&]() { double s = 0; for (int i = 0; i < 12; ++i) s += uni(); return s - 6.0; };
    for (int t = 0; t < cases; ++t) {
        len[t] = lens[t % 16];
        for (int c = 0; c < NS; ++c) {
            double *v = &x[((size_t)t * NS + c) * stride];
            const int kind = (t / 16 + c) % 15;
            const double m = 4.0106053e-08 * (1 + (rng() % 100) * 1e-3);
            for (uint32_t k = 0; k < len[t]; ++k) {
                double y = 0;
                switch (kind) {
                case 0: y = m; break;                                             // masses
                case 1: y = m * (double)(float)(0.07 + 1e-3 * nrm()); break;      // positions
                case 2: y = m * (double)(float)(1e-3 * nrm()); break;             // velocities around zero
                case 3: y = 0.0; break;                                           // at rest
                case 4: y = rng() % 50 ? -0.0 : m * nrm(); break;                 // mostly at rest
                case 5: y = (double)((long)(rng() % 5) - 2); break;               // cancels to zero
                case 6: y = k == 0 ? 0x1p60 : (double)(rng() % 1024) * 0.5; break; // ties: half units of 2^8's grid
                case 7: y = k == 0 ? 4503599627370497.0 : 0.5 * (double)(rng() % 4); break;    // ties, odd and even
                case 8: y = k == 0 ? -4503599627370498.0 : 0.5 * (double)((long)(rng() % 5) - 2); break;
                case 9: y = k == 0 ? 9007199254740980.0 : 0.5 * (double)(rng() % 3); break;    // to the upper edge
                case 10: y = k == 0 ? 4503599627370500.0 : -0.5 * (double)(rng() % 3); break;  // to the lower edge
                case 11: y = std::ldexp(nrm(), (int)(rng() % 400) - 200); break;  // any magnitude
                case 12: y = std::ldexp(nrm(), -1060 + (int)(rng() % 30)); break; // subnormals
                case 13: y = k == len[t] / 2 ? INFINITY : m * nrm(); break;
                case 14: y = (k % 64 < 60 ? 1 : -1) * 1e6 * uni(); break;         // in its binade, then crossing
                }
                v[k] = y;
            }
        }
    }
    double *dx, *dout;
    uint32_t *dl, *dn;
    cudaMalloc(&dx, x.size() * 8);
    cudaMalloc(&dout, cases * NS * 8);
    cudaMalloc(&dl, cases * 4);
    cudaMalloc(&dn, cases * NS * 4);
    cudaMemcpy(dx, x.data(), x.size() * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dl, len.data(), cases * 4, cudaMemcpyHostToDevice);
    k_sums<<<cases, 256>>>(dx, stride, dl, dout, dn);
    std::vector<double> out(cases * NS);
    std::vector<uint32_t> loops(cases * NS);
    cudaMemcpy(loops.data(), dn, loops.size() * 4, cudaMemcpyDeviceToHost);
    if (cudaMemcpy(out.data(), dout, out.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) { printf("cuda error\n"); return 2; }
    int bad = 0;
    long chunks[15] = {0}, looped[15] = {0};
    for (int i = 0; i < cases * NS; ++i) {
        const int kind = (i / NS / 16 + i % NS) % 15;
        chunks[kind] += (len[i / NS] + kSumChunk - 1) / kSumChunk;
        looped[kind] += loops[i];
        double s = 0.0;
        for (uint32_t k = 0; k < len[i / NS]; ++k) s = s + x[(size_t)i * stride + k];
        if (std::memcmp(&s, &out[i], 8) != 0 && !(std::isnan(s) && std::isnan(out[i]))) {
            if (bad++ < 10) printf("case %d kind %d len %u: %a, want %a\n", i, kind, len[i / NS], out[i], s);
        }
    }
    for (int k = 0; k < 15; ++k) printf("kind %d: %ld of %ld chunks term by term\n", k, looped[k], chunks[k]);
    printf("%d sums, %d differ\n", cases * NS, bad);
    // the sums that the clump stage meets must not end up in the loop
    for (int k = 0; k < 4; ++k) bad += looped[k] * 20 > chunks[k];
    return bad != 0;
}
"""


@pytest.mark.gpu
def test_ordered_sums_equal_a_sequential_loop(tmp_path, built):
    from plan_gb300 import build as b

    (tmp_path / "d.cu").write_text(DEVICE)
    subprocess.run([str(b._cuda_home() / "bin" / "nvcc"), *b.ARCH, "-O3", "-std=c++17", "--fmad=false", "-Xcompiler", "-ffp-contract=off", f"-I{CSRC}",
                    str(tmp_path / "d.cu"), "-o", str(tmp_path / "d")], check=True)
    r = subprocess.run([str(tmp_path / "d")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
