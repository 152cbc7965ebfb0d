"""The ES window's value (one Newton step on the hardware's root and reciprocal)
against 64 bits over the whole window: no further off than with sqrtf and the
division."""
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

_SRC = r"""
#include <cmath>
#include <cstdio>
#include "common.cuh"
using namespace cuvgls;
__device__ float plain_tap(float dd, const Plan &p) {
    const float z2 = dd * dd * p.es_im2, s = 1.f - z2;
    return s > 0.f ? expf(-p.es_beta * z2 / (1.f + sqrtf(s))) : 0.f;
}
struct Err { double worst[2], sum2[2]; };
// offsets (i + 1/2) m / n, and one float below m
__global__ void compare(Plan p, int n, Err *err) {
    double worst[2] = {0, 0}, sum2[2] = {0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
        const float dd = i < n ? (float)p.m * ((float)i + 0.5f) / (float)n : nextafterf((float)p.m, 0.f);
        const float z2 = dd * dd * p.es_im2, s = 1.f - z2;
        if (!(s > 0.f)) continue;
        const double ex = exp(-(double)p.es_beta * (double)z2 / (1.0 + sqrt((double)s)));
        const double e[2] = {fabs(plain_tap(dd, p) - ex), fabs(win_tap(dd, p) - ex)};
        for (int k = 0; k < 2; ++k) {
            worst[k] = fmax(worst[k], e[k] / ex);
            sum2[k] += e[k] * e[k];
        }
    }
    for (int k = 0; k < 2; ++k) {
        atomicMax((unsigned long long *)&err->worst[k], (unsigned long long)__double_as_longlong(worst[k]));
        atomicAdd(&err->sum2[k], sum2[k]);
    }
}
int main() {
    Err *d, h;
    if (cudaMalloc(&d, sizeof(Err)) != cudaSuccess) return 1;
    for (int m = 2; m <= 16; ++m) {
        Plan p{};
        p.win = kWinES;
        p.m = m;
        p.es_beta = (float)(0.97 * 3.141592653589793 * 2.0 * m * (1.0 - 1.0 / 2.56));
        p.es_im2 = (float)(1.0 / ((double)m * m));
        if (cudaMemset(d, 0, sizeof(Err)) != cudaSuccess) return 1;
        compare<<<608, 256>>>(p, 1 << 22, d);
        if (cudaMemcpy(&h, d, sizeof(Err), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
        printf("%d %.6e %.6e %.6e %.6e\n", m, h.worst[0], h.worst[1], sqrt(h.sum2[0] / (1 << 22)),
               sqrt(h.sum2[1] / (1 << 22)));
    }
    return 0;
}
"""


def test_window_value(tmp_path):
    from cuvarbase_gb300 import build
    (tmp_path / "w.cu").write_text(_SRC)
    subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", *build.ARCH, "-O3",
                    "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC,
                    str(tmp_path / "w.cu"), "-o", str(tmp_path / "w")], check=True)
    r = subprocess.run([str(tmp_path / "w")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0
    rows = [list(map(float, line.split())) for line in r.stdout.splitlines()]
    assert len(rows) == 15
    for m, worst_plain, worst, rms_plain, rms in rows:
        assert worst <= 1.01 * worst_plain and rms <= 1.01 * rms_plain, m
