"""A wait for a tile's copy that runs out (kernels compiled with a limit of no
tries at all; the copy itself arrives): the CTAs leave, the device error word
says so, and the device goes on."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cuvarbase_gb300")

# argv: grids, row length.  Prints the error word, the outputs written and their
# number: with no tries, then with the library's kernels.
_SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "kernels.cuh"
#include "pass2_tma.cuh"
using namespace cuvgls;
#define OK(x) do { cudaError_t e = (x); if (e != cudaSuccess) { \
    fprintf(stderr, "%s: %s\n", #x, cudaGetErrorString(e)); return 1; } } while (0)
int main(int, char **argv) {
    const int ng = atoi(argv[1]), G2 = atoi(argv[2]), G1 = 160, curves = 40;
    Plan p;
    memset(&p, 0, sizeof p);
    p.G1 = G1; p.G2 = G2; p.G = (long long)G1 * G2; p.m = 8;
    p.B = pass1_cols(ng, G1); p.R = pass2_rows(ng, G2); p.nb = G2 / p.B;
    p.binv = 1.f; p.dc1 = 0.f; p.dc2 = 1.f;
    const int nf = (int)(p.G / 2);
    float2 *tab, *inter, *out;
    unsigned *flag;
    ulonglong2 *aux;
    DevCurve *cv;
    const size_t in = (size_t)ng * p.G * curves * 8, on = (size_t)nf * curves;
    OK(cudaMalloc(&tab, (fft_table_len(G1) + row_table_len(ng, G2) + p.G) * 8));
    OK(cudaMalloc(&inter, in));
    OK(cudaMalloc(&out, on * 8));
    OK(cudaMalloc(&flag, 4));
    OK(cudaMalloc(&aux, 16));
    OK(cudaMalloc(&cv, curves * sizeof(DevCurve)));
    OK(cudaMemset(inter, 0, in));
    OK(cudaMemset(aux, 0, 16));
    OK(launch_plan_tables(tab, G1, G2, p.B, ng, 0));
    p.st1 = tab; p.st2 = tab + fft_table_len(G1); p.itw = p.st2 + row_table_len(ng, G2);
    std::vector<DevCurve> h(curves);
    for (int i = 0; i < curves; ++i) {
        memset(&h[i], 0, sizeof(DevCurve));
        h[i].n = 1; h[i].nf = nf; h[i].df = 1.0; h[i].out_off = (long long)i * nf;
    }
    OK(cudaMemcpy(cv, h.data(), curves * sizeof(DevCurve), cudaMemcpyHostToDevice));
    for (int k = 0; k < 2; ++k) {
        OK(cudaMemset(flag, 0, 4));
        OK(cudaMemset(out, 0xff, on * 8));
        const GlsParams g{1, 0.f, nullptr, flag};
        if (k && ng == 3)
            OK(launch_pass2_gls(cv, curves, 0, inter, (float *)out, p, g, 0));
        else if (k)
            OK(launch_pass2_nfft(cv, curves, 0, inter, out, aux, flag, p, 0));
        else if (ng == 3)
            OK(G2 == 160 ? (launch_pass2_reg_t<160, false, false, 0>(cv, curves, 0, inter, (float *)out, p, g, 0))
             : G2 == 256 ? (launch_pass2_reg_t<256, false, false, 0>(cv, curves, 0, inter, (float *)out, p, g, 0))
                         : (launch_pass2_reg_t<400, false, false, 0>(cv, curves, 0, inter, (float *)out, p, g, 0)));
        else
            OK(G2 == 160 ? (launch_nfft_reg_t<160, false, 0>(cv, curves, 0, inter, out, aux, flag, p, 0))
                         : (launch_nfft_reg_t<400, false, 0>(cv, curves, 0, inter, out, aux, flag, p, 0)));
        OK(cudaDeviceSynchronize());
        unsigned f;
        std::vector<unsigned> o(on * (ng == 3 ? 1 : 2));
        OK(cudaMemcpy(&f, flag, 4, cudaMemcpyDeviceToHost));
        OK(cudaMemcpy(o.data(), out, o.size() * 4, cudaMemcpyDeviceToHost));
        size_t w = 0;
        for (unsigned x : o) w += x != 0xffffffffu;
        printf("%u %zu %zu\n", f, w, o.size());
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    from cuvarbase_gb300 import build
    build.build()
    d = tmp_path_factory.mktemp("wait")
    (d / "wait.cu").write_text(_SRC)
    subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", *build.ARCH, "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", build.CSRC, str(d / "wait.cu"), "-o",
                    str(d / "wait"), build.LIB, "-Xlinker", "-rpath=" + PKG], check=True)
    return str(d / "wait")


@pytest.mark.parametrize("grids,G2", [(3, 160), (3, 256), (3, 400), (1, 160), (1, 400)])
def test_wait_runs_out(harness, grids, G2):
    from cuvarbase_gb300 import _lib
    r = subprocess.run([harness, str(grids), str(G2)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    first, after = [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    assert first[0] == _lib.DEVERR_TIMEOUT and first[1] == 0
    assert after[0] == 0 and after[1] == after[2]
