"""The step lists of the exact ordered sums (ordered_sum.cuh) at either half of a 16-byte unit.

A list of 8-byte entries may start on any 8-byte boundary; its loads of two entries may not.
Lists at an offset of one entry, with no step, a few and many listed, against a sequential loop.
"""
from __future__ import annotations

import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "plan_gb300" / "csrc"

DEVICE = r"""
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "ordered_sum.cuh"
using namespace plan;

__global__ void __launch_bounds__(256) k_sum(const double *x, const uint32_t *len, uint32_t shift, double *out) {
    __shared__ __align__(16) double stage[kSumStage];
    __shared__ __align__(16) uint2 steps[kSumChunk + 1];
    const uint32_t m = len[blockIdx.x];
    x += (size_t)blockIdx.x * 1024;
    double acc = 0.0;
    for (uint32_t b = 0; b < m; b += kSumChunk) {
        stage[sum_slot(threadIdx.x)] = b + threadIdx.x < m ? x[b + threadIdx.x] : 0.0;
        __syncthreads();
        if (threadIdx.x < 32) ordered_sum_chunk(stage, acc, steps + shift);
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = acc;
}

int main() {
    std::mt19937_64 rng(5);
    const int cases = 256;
    std::vector<double> x((size_t)cases * 1024);
    std::vector<uint32_t> len(cases);
    for (int t = 0; t < cases; ++t) {
        len[t] = 1 + rng() % 1024;
        for (uint32_t k = 0; k < 1024; ++k) {
            const double u = (double)(rng() >> 11) * 0x1p-53;
            double y = 0.1 + u;                                                              // a step per binade
            if (t % 4 == 1) y = u - 0.5;                                                     // around zero: many
            if (t % 4 == 2) y = k == 0 ? 4503599627370497.0 : 0.5 * (double)(rng() % 4);     // ties: most
            if (t % 4 == 3) y = k == 0 ? 1e6 : (rng() % 40 ? 1.0 : 0.5 + 0x1p-34);           // hardly any
            x[(size_t)t * 1024 + k] = y;
        }
    }
    double *dx, *dout;
    uint32_t *dl;
    cudaMalloc(&dx, x.size() * 8);
    cudaMalloc(&dout, cases * 8);
    cudaMalloc(&dl, cases * 4);
    cudaMemcpy(dx, x.data(), x.size() * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dl, len.data(), cases * 4, cudaMemcpyHostToDevice);
    int bad = 0;
    for (uint32_t shift = 0; shift < 2; ++shift) {
        std::vector<double> out(cases);
        k_sum<<<cases, 256>>>(dx, dl, shift, dout);
        if (cudaMemcpy(out.data(), dout, cases * 8, cudaMemcpyDeviceToHost) != cudaSuccess) { printf("cuda error\n"); return 2; }
        for (int t = 0; t < cases; ++t) {
            double s = 0.0;
            for (uint32_t k = 0; k < len[t]; ++k) s = s + x[(size_t)t * 1024 + k];
            if (std::memcmp(&s, &out[t], 8) != 0 && bad++ < 10) printf("shift %u case %d: %a, want %a\n", shift, t, out[t], s);
        }
    }
    return bad != 0;
}
"""


@pytest.mark.gpu
def test_lists_on_either_half(tmp_path, built):
    from plan_gb300 import build as b

    (tmp_path / "d.cu").write_text(DEVICE)
    subprocess.run([str(b._cuda_home() / "bin" / "nvcc"), *b.ARCH, "-O3", "-std=c++17", "--fmad=false", "-Xcompiler", "-ffp-contract=off", f"-I{CSRC}",
                    str(tmp_path / "d.cu"), "-o", str(tmp_path / "d")], check=True)
    r = subprocess.run([str(tmp_path / "d")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
