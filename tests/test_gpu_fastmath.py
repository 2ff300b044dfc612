"""The short e^x, square root and division (ct_fastmath.cuh) against FP64 and against CUDA's own division, at
the bounds that their comments state.  u = 2^-24:
    exp2x   2^-22 + 1.23 u |x|, plus u^2 terms           (results that are not flushed to 0)
    sqrt2x  u (1 + 2^-19)
    div_by  the same bits as x / b
"""
import json
import subprocess

import pytest

from covertreex_gb300 import _build

pytestmark = pytest.mark.gpu

PROGRAM = """
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "ct_fastmath.cuh"

constexpr int N = 1 << 22;
__device__ unsigned long long mix(unsigned long long z) {  // splitmix64's finaliser
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}
__device__ double unit(unsigned long long i) { return (double)(mix(i * 0x9e3779b97f4a7c15ULL + 1) >> 11) * 0x1p-53; }

__global__ void run(float* x, float* ex, float* s, float* sq, int* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    x[i] = (float)(-87.0 * pow(unit(i), 3.0));                       // dense near 0
    ex[i] = ct::exp2x(make_float2(x[i], 0.f)).x;
    s[i] = (float)exp2(-99.0 + 226.0 * unit(i + (1LL << 40)));       // 2^-99 .. 2^127
    sq[i] = ct::sqrt2x(make_float2(1.f, s[i])).y;
    const double a = ldexp(1.0 + unit(i + (2LL << 40)), (int)(mix(i) % 400) - 200);
    const double b = ldexp(1.0 + unit(i + (3LL << 40)), (int)(mix(i + 7) % 120) - 60);
    if (ct::div_by(a, b, 1.0 / b) != a / b || ct::div_by(-a, 3.0, 1.0 / 3.0) != -a / 3.0) atomicAdd(bad, 1);
}

int main() {
    float *x, *ex, *s, *sq;
    int* bad;
    if (cudaMalloc(&x, 4 * N) || cudaMalloc(&ex, 4 * N) || cudaMalloc(&s, 4 * N) || cudaMalloc(&sq, 4 * N) ||
        cudaMalloc(&bad, 4) || cudaMemset(bad, 0, 4))
        return 1;
    run<<<N / 256, 256>>>(x, ex, s, sq, bad);
    std::vector<float> hx(N), hex(N), hs(N), hsq(N);
    int hbad = 0;
    if (cudaMemcpy(hx.data(), x, 4 * N, cudaMemcpyDeviceToHost) || cudaMemcpy(hex.data(), ex, 4 * N, cudaMemcpyDeviceToHost) ||
        cudaMemcpy(hs.data(), s, 4 * N, cudaMemcpyDeviceToHost) || cudaMemcpy(hsq.data(), sq, 4 * N, cudaMemcpyDeviceToHost) ||
        cudaMemcpy(&hbad, bad, 4, cudaMemcpyDeviceToHost))
        return 1;
    double we = 0, ws = 0;  // largest error in units of its bound
    const double u = ldexp(1.0, -24);
    for (int i = 0; i < N; ++i) {
        const double e = std::exp((double)hx[i]);
        we = std::fmax(we, std::fabs(hex[i] - e) / e / (4 * u + 1.23 * u * std::fabs(hx[i])));
        const double q = std::sqrt((double)hs[i]);
        ws = std::fmax(ws, std::fabs(hsq[i] - q) / q / (u * (1 + ldexp(1.0, -19))));
    }
    printf("{\\"exp\\": %.4f, \\"sqrt\\": %.6f, \\"div\\": %d}", we, ws, hbad);
}
"""


def test_short_forms_stay_within_their_bounds(cuda_available, tmp_path):
    (tmp_path / "p.cu").write_text(PROGRAM)
    subprocess.run([_build.nvcc_path(), _build.ARCH, "-O3", "-std=c++17", f"-I{_build.CSRC}", "p.cu", "-o", "p"],
                   cwd=tmp_path, check=True)
    out = json.loads(subprocess.run([str(tmp_path / "p")], capture_output=True, text=True, check=True).stdout)
    assert out["div"] == 0, out
    assert out["exp"] <= 1.0 and out["sqrt"] <= 1.0, out
