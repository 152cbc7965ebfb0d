// cuvgls kernels for sm_103a.
//
// This file holds the auxiliary kernels and the length dispatch; the
// per-point kernels are in prep.cu, the pass kernels in pass_kernels.cuh, the
// direct sums in direct.cu.
//
// The path per size class (G = G1 * G2 grid cells):
//   k_prep       (prep.cu) FP64 offsets t - t0, grid cell index and
//                band-centring phase per point; counting sort of the points
//                by the column block (cell mod G2) / B their window starts in;
//                compact FP32 spreading records.
//   k_pass1      one CTA per (curve, column block).  Spreads the records of
//                the neighbouring bins into a G1 x B shared-memory tile per
//                grid (shared-memory float atomics), runs the length-G1 column
//                FFTs in shared memory, applies the inter-pass twiddle and
//                writes the tile to the intermediate buffer.
//   k_pass2_*    a task or CTA per (curve, R-row block).  Runs the length-G2
//                row FFTs of every grid, the butterflies in registers and the
//                exchange between them in shared memory, and, in the same
//                kernel, deconvolves the window and either evaluates the GLS
//                power (3 grids) or applies the output phase of the adjoint
//                NFFT (1 grid).
// The grid itself never exists in HBM: spreading is fused into pass 1.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <mutex>

#include "gls_math.cuh"
#include "kernels.cuh"
#include "pass2_tma.cuh"

namespace cuvgls {

// ---------------------------------------------------------------------------
// reference-convention gridding (just_return_gridded_data)
// ---------------------------------------------------------------------------
__global__ void k_spread_ref(const RefGridCurve *__restrict__ cvs,
                             const double *__restrict__ t,
                             const float *__restrict__ y, float *__restrict__ grid,
                             int m, float binv, float norm) {
    const RefGridCurve cv = cvs[blockIdx.y];
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cv.n) return;
    const double x = (t[cv.pt_off + j] - cv.tmin) * cv.scale;
    const double gx = (double)cv.ng * x;
    const long long u = (long long)floor(gx - (double)m);
    const float yj = y[cv.pt_off + j];
    for (int k = 0; k <= 2 * m; ++k) {
        const float d = (float)(gx - (double)(u + k));
        const float wg = expf(-d * d * binv) * norm;
        long long l = (u + k) % cv.ng;
        if (l < 0) l += cv.ng;
        atomicAdd(&grid[cv.out_off + l], yj * wg);
    }
}

// ---------------------------------------------------------------------------
// finish of a caller-given reference-convention grid (use_grid)
// ---------------------------------------------------------------------------
// One thread per output bin k; the grid is staged 128 cells at a time and
// exp(2 pi i j (ks + k) / ng) advances by multiplication along j, re-seeded
// from sincospi at every tile.
__global__ void __launch_bounds__(128)
k_grid_finish(const GridFinishCurve *__restrict__ cvs, const double2 *__restrict__ grid,
              double2 *__restrict__ out) {
    __shared__ double2 sg[128];
    const GridFinishCurve cv = cvs[blockIdx.y];
    const long long k = (long long)blockIdx.x * 128 + threadIdx.x;
    const double ng = (double)cv.ng;
    const double fr = (cv.ks + (double)k) / ng;  // cycles per grid cell
    double step_s, step_c;
    {
        double st = fr - floor(fr);
        sincospi(2.0 * st, &step_s, &step_c);
    }
    double re = 0.0, im = 0.0;
    for (long long base = 0; base < cv.ng; base += 128) {
        const long long j = base + threadIdx.x;
        __syncthreads();
        if (j < cv.ng) sg[threadIdx.x] = grid[cv.grid_off + j];
        __syncthreads();
        const int cnt = (int)min((long long)128, cv.ng - base);
        if (k < cv.nf) {
            double ph = fr * (double)base;
            ph -= floor(ph);
            double s, c;
            sincospi(2.0 * ph, &s, &c);
            for (int q = 0; q < cnt; ++q) {
                const double2 g = sg[q];
                re = fma(g.x, c, fma(-g.y, s, re));
                im = fma(g.x, s, fma(g.y, c, im));
                const double c2 = c * step_c - s * step_s;
                s = fma(s, step_c, c * step_s);
                c = c2;
            }
        }
    }
    if (k < cv.nf) {
        const double kk = cv.k0 + (double)k;
        double th = cv.n0 * kk / ng;
        th -= floor(th);
        double s, c;
        sincospi(2.0 * th, &s, &c);
        const double kh = kk / ng;  // khat / pi
        const double pk = 3.141592653589793 * kh;
        const double sc = exp(cv.b * pk * pk);
        out[cv.out_off + k] = make_double2((re * c - im * s) * sc, (re * s + im * c) * sc);
    }
}

cudaError_t launch_grid_finish(const GridFinishCurve *cv, int n_curves, long long max_nf,
                               const double2 *grid, double2 *out, cudaStream_t s) {
    if (n_curves <= 0 || max_nf <= 0) return cudaSuccess;
    const long long nb = (max_nf + 127) / 128;
    if (nb > 0x7fffffffLL || n_curves > 65535) return cudaErrorInvalidValue;
    k_grid_finish<<<dim3((unsigned)nb, n_curves), 128, 0, s>>>(cv, grid, out);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// plan tables (FP64 angles, rounded once to float)
// ---------------------------------------------------------------------------
// Turns (fraction of a full turn) of entry e of the FFT table of a length-L
// transform, in the layout the pass kernels read: the stage-A twiddles i qa / L of
// a two-level length (fft_table_len), else [stage][r - 1][k] Stockham twiddles.
__device__ double fft_table_turns(int L, int e) {
    if (two_level_la(L) > 0) {
        const int LB = L / two_level_la(L);
        const bool pr = tw_pairs(L);
        const int i = pr ? e / 2 % LB : e % LB, qa = pr ? e / (2 * LB) * 2 + e % 2 : e / LB;
        return (double)(i * qa) / (double)L;
    }
    const FacList f = fft_factors(L);
    int ns = 1;
    for (int s = 0; s < f.n; ++s) {
        const int R = f.r[s];
        if (ns > 1) {
            const int seg = ns * (R - 1);
            if (e < seg) {
                const int r = e / ns + 1, k = e % ns;
                return (double)(k * r) / (double)(ns * R);
            }
            e -= seg;
        }
        ns *= R;
    }
    return 0.0;
}

// (ng: grids, which choose the row table's layout)
__global__ void k_plan_tables(float2 *dst, int G1, int G2, int B, int ng, int n1, int n2) {
    const long long G = (long long)G1 * G2;
    const long long total = n1 + n2 + G;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        double turns;
        if (e < n1) {
            turns = fft_table_turns(G1, (int)e);
        } else if (e < n1 + n2) {
            const int x = (int)(e - n1);
            if (pass2_deep(ng, G2)) {
                const int N1 = G2 / deep_fac(G2, 0), y = x - G2;
                turns = y < 0 ? (double)(x / N1 * (x % N1)) / (double)G2
                              : (double)(y / 8 * (y % 8)) / (double)N1;
            } else {
                turns = fft_table_turns(G2, x);
            }
        } else {
            // inter-pass twiddle in the intermediate's [cb][q1][c] order
            const long long i = e - n1 - n2;
            const int c = (int)(i % B);
            const long long rest = i / B;
            const int q1 = (int)(rest % G1), cb = (int)(rest / G1);
            const long long l2 = (long long)cb * B + c;
            turns = (double)(((long long)q1 * l2) % G) / (double)G;
        }
        double s, c;
        sincospi(2.0 * turns, &s, &c);
        dst[e] = make_float2((float)c, (float)s);
    }
}

// Deconvolution table of the ES window: dst[j] = 1 / phihat(j), j = 0..n-1,
// with phihat(j) = 2 int_0^m phi(s) cos(2 pi j s / G) ds the Fourier
// transform of phi(s) = exp(beta (sqrt(1 - s^2 / m^2) - 1)) at band index j,
// in FP64 by the midpoint rule over kEsNodes nodes (phi and its derivatives
// are smooth inside [0, m); at s = m phi is e^-beta, ~1e-8, so the rule's
// endpoint error is far below FP32).  The cosines come from a rotation
// recurrence re-seeded every 64 nodes.
constexpr int kEsNodes = 256;

__global__ void __launch_bounds__(256) k_es_deconv(float *dst, int n, double G, int m,
                                                   double beta) {
    __shared__ double phi[kEsNodes];
    const double h = (double)m / kEsNodes;
    for (int q = threadIdx.x; q < kEsNodes; q += blockDim.x) {
        const double z = (q + 0.5) * h / m;
        phi[q] = exp(beta * (sqrt(1.0 - z * z) - 1.0));
    }
    __syncthreads();
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const double th = 2.0 * (double)j * h / G;  // rotation per node, in half turns
    double sr, cr;
    sincospi(th, &sr, &cr);
    double acc = 0.0;
    for (int q0 = 0; q0 < kEsNodes; q0 += 64) {
        double zs, zc;
        sincospi(th * (q0 + 0.5), &zs, &zc);
        for (int q = q0; q < q0 + 64; ++q) {
            acc = fma(phi[q], zc, acc);
            const double nc = zc * cr - zs * sr;
            zs = fma(zc, sr, zs * cr);
            zc = nc;
        }
    }
    dst[j] = (float)(1.0 / (2.0 * h * acc));
}

__global__ void k_best_finish(const unsigned long long *__restrict__ keys, int n,
                              int64_t *__restrict__ best_k, float *__restrict__ best_p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long k = keys[i];
    if (k == 0) {
        best_k[i] = -1;
        best_p[i] = -1.f;
    } else {
        best_k[i] = (int64_t)(0xFFFFFFFFu - (unsigned)(k & 0xFFFFFFFFull));
        best_p[i] = __uint_as_float((unsigned)(k >> 32));
    }
}

cudaError_t launch_best_finish(const unsigned long long *keys, int n, int64_t *best_k,
                               float *best_p, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_best_finish<<<(n + 255) / 256, 256, 0, s>>>(keys, n, best_k, best_p);
    return cudaGetLastError();
}

cudaError_t launch_plan_tables(float2 *dst, int G1, int G2, int B, int ng, cudaStream_t s) {
    const int n1 = fft_table_len(G1), n2 = row_table_len(ng, G2);
    const long long total = n1 + n2 + (long long)G1 * G2;
    const int blocks = (int)std::min<long long>((total + 255) / 256, 4096);
    k_plan_tables<<<blocks, 256, 0, s>>>(dst, G1, G2, B, ng, n1, n2);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(256)
k_deconv_rows(const float *__restrict__ dtab, float *__restrict__ dst, int G1, int G2, int R) {
    const int G = G1 * G2;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < G; e += gridDim.x * blockDim.x) {
        const int r = e % R, q2 = e / R % G2, rb = e / (R * G2);
        const int q = rb * R + r + G1 * q2;
        dst[e] = dtab[min(q, G - q)];
    }
}

cudaError_t launch_deconv_rows(const float *dtab, float *dst, int G1, int G2, int R,
                               cudaStream_t s) {
    if (G1 < R || G1 % R) return cudaErrorInvalidValue;
    const int blocks = std::min((G1 * G2 + 255) / 256, 4096);
    k_deconv_rows<<<blocks, 256, 0, s>>>(dtab, dst, G1, G2, R);
    return cudaGetLastError();
}

// The driver's tensor-map encoder, looked up once (the library links no
// driver symbols).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static std::once_flag once;
    static void *fn = nullptr;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult st;
        void *f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault,
                                             &st) == cudaSuccess &&
            st == cudaDriverEntryPointSuccess)
            fn = f;
    });
    return (PFN_cuTensorMapEncodeTiled_v12000)fn;
}

cudaError_t pass2_map(CUtensorMap &map, const float2 *inter, const Plan &p, int grids, int R) {
    const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return cudaErrorNotSupported;
    const cuuint64_t dims[3] = {(cuuint64_t)p.G1 * p.B * 2, (cuuint64_t)p.nb, (cuuint64_t)grids};
    const cuuint64_t strides[2] = {(cuuint64_t)p.G1 * p.B * 8, (cuuint64_t)p.G * 8};
    const cuuint32_t box[3] = {(cuuint32_t)(R * p.B * 2), (cuuint32_t)p.nb, 1};
    const cuuint32_t es[3] = {1, 1, 1};
    const CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)inter, dims, strides,
                           box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t launch_es_deconv(float *dst, long long G, int m, double beta, cudaStream_t s) {
    if (G < 2 || m < 1) return cudaErrorInvalidValue;
    const int n = (int)(G / 2 + 1);
    k_es_deconv<<<(n + 255) / 256, 256, 0, s>>>(dst, n, (double)G, m, beta);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
#define CUVGLS_LEN_CASES(X) X(16) X(32) X(64) X(80) X(128) X(160) X(256) X(320) \
    X(400) X(512) X(640) X(800) X(1024) X(1280) X(1600) X(2048)
#define CUVGLS_ROW_LEN_CASES(X) CUVGLS_LEN_CASES(X) X(4096)

cudaError_t launch_pass1(const DevCurve *cv, int n_curves, int max_n, const RecAB *recAB,
                         const RecC *recC, const int *binsAB, const int *binsC,
                         float2 *inter, const Plan &p, int ngrids, cudaStream_t s) {
    if (n_curves <= 0) return cudaSuccess;
#define CUVGLS_P1(L) \
    case L: return ngrids == 3 ? launch_pass1_t<3, L>(cv, n_curves, max_n, recAB, recC, binsAB, binsC, inter, p, s) \
                               : launch_pass1_t<1, L>(cv, n_curves, max_n, recAB, recC, binsAB, binsC, inter, p, s);
    switch (p.G1) {
        CUVGLS_LEN_CASES(CUVGLS_P1)
        default: return cudaErrorInvalidValue;
    }
#undef CUVGLS_P1
}

cudaError_t preload_pass_kernels(int G1, int G2, int ngrids) {
    cudaError_t e = cudaErrorInvalidValue;
#define CUVGLS_PL1(L) \
    case L: e = ngrids == 3 ? preload_pass1_t<3, L>() : preload_pass1_t<1, L>(); break;
    switch (G1) {
        CUVGLS_LEN_CASES(CUVGLS_PL1)
        default: return cudaErrorInvalidValue;
    }
#undef CUVGLS_PL1
    if (e != cudaSuccess) return e;
#define CUVGLS_PL2(L) case L: return preload_pass2_t<L>(ngrids);
    switch (G2) {
        CUVGLS_ROW_LEN_CASES(CUVGLS_PL2)
        default: return cudaErrorInvalidValue;
    }
#undef CUVGLS_PL2
}

cudaError_t launch_pass2_gls(const DevCurve *cv, int n_curves, int first,
                             const float2 *inter, float *out, const Plan &p,
                             GlsParams g, cudaStream_t s) {
    if (n_curves <= 0) return cudaSuccess;
#define CUVGLS_P2(L) case L: return launch_pass2_gls_t<L>(cv, n_curves, first, inter, out, p, g, s);
    switch (p.G2) {
        CUVGLS_ROW_LEN_CASES(CUVGLS_P2)
        default: return cudaErrorInvalidValue;
    }
#undef CUVGLS_P2
}

cudaError_t launch_pass2_nfft(const DevCurve *cv, int n_curves, int first, const float2 *inter,
                              float2 *out, const ulonglong2 *aux, unsigned *errflag, const Plan &p,
                              cudaStream_t s) {
    if (n_curves <= 0) return cudaSuccess;
#define CUVGLS_P2N(L) \
    case L: return launch_pass2_nfft_t<L>(cv, n_curves, first, inter, out, aux, errflag, p, s);
    switch (p.G2) {
        CUVGLS_ROW_LEN_CASES(CUVGLS_P2N)
        default: return cudaErrorInvalidValue;
    }
#undef CUVGLS_P2N
}

cudaError_t launch_spread_ref(const RefGridCurve *cv, int n_curves,
                              long long max_n, const double *t, const float *y,
                              float *grid, int m, float binv, float norm,
                              cudaStream_t s) {
    if (n_curves <= 0 || max_n <= 0) return cudaSuccess;
    dim3 g((unsigned)((max_n + 255) / 256), n_curves);
    k_spread_ref<<<g, 256, 0, s>>>(cv, t, y, grid, m, binv, norm);
    return cudaGetLastError();
}

}  // namespace cuvgls
