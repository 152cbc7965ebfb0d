// Host-side launch wrappers of the cuvgls kernels (implemented in kernels.cu).
#pragma once

#include <cstdint>

#include "common.cuh"

namespace cuvgls {

struct RefGridCurve {  // device copy of cuvgls_grid_curve
    long long pt_off, n, ng;
    double tmin, scale;  // x = (t - tmin) * scale
    long long out_off;
};

// Arrays of a preparation launch.  Records and bin offsets of a descriptor
// start at its rec_off / bin_off.
struct PrepArrays {
    DevCurve *cv;
    const double *t, *ry, *rdy;  // raw input: t, y, dy
    const float *ya, *wv;        // prepared input: yw (or y) and w
    RecAB *recAB;
    RecC *recC;
    int *binsAB, *binsC;         // nb + 1 offsets per descriptor
    int *curAB, *curC;           // cursors (long curves)
    ulonglong2 *aux;             // output phases of the adjoint NFFT, or null
    unsigned *errflag;
    int mode;                    // GLS mode (raw input)
    int max_nb;                  // most column blocks of the launch's plans
    int trigger;                 // let the next kernel be set up early
    int beside;                  // run beside the k_prep before: wait for it at the end
};

// Descriptors of a small batch as a kernel parameter: k_prep then takes its
// curves from here and writes the descriptors to a.cv itself, so the batch
// needs no copy of its table before its first kernel.
constexpr int kParamDesc = 32;
struct DescParam {
    int n;  // 0: none, the descriptors are in a.cv
    DevCurve cv[kParamDesc];
};
static_assert(sizeof(DescParam) + sizeof(PrepArrays) <= 3584, "kernel parameters");

// Curves of one length class (prep_class), each by one CTA or cluster: raw
// weights and statistics (raw != 0), bin offsets and records.  `list`: their
// descriptors (null: 0 .. n - 1); max_n: the longest; ngrids 3 (GLS: yw@x,
// w@x, w@2x) or 1 (NFFT: y@x).  `beside`: the kernel before it in the stream
// is a launch_prep of the same batch, which it does not wait for before its
// end.
cudaError_t launch_prep(const PrepArrays &a, const DescParam &d, const int *list, int n, int cls,
                        int max_n, int raw, int ngrids, int fp32_positions, bool beside,
                        cudaStream_t s);

// Binning of long curves: counts per segment (the counts of their
// descriptors zeroed by the caller), scan per descriptor of `list`, records
// per segment.
cudaError_t launch_bin_long(const PrepArrays &a, const SegEntry *segs, int n_segs, const int *list,
                            int n, int ngrids, int fp32_positions, cudaStream_t s);

// Segment table of the descriptors 0 .. n - 1 filled on the device, each at
// its raw_seg.
cudaError_t launch_seg_fill(const DevCurve *cv, int n, SegEntry *segs, cudaStream_t s);

// Dispatch on (G1, G2) to the compiled length templates; cudaErrorInvalidValue
// if a length has no kernel.
// (`max_n`: points of the longest of the curves)
cudaError_t launch_pass1(const DevCurve *cv, int n_curves, int max_n, const RecAB *recAB,
                         const RecC *recC, const int *binsAB, const int *binsC,
                         float2 *inter, const Plan &p, int ngrids, cudaStream_t s);

// (`first`: index of the first curve within the intermediate's chunk)
cudaError_t launch_pass2_gls(const DevCurve *cv, int n_curves, int first, const float2 *inter, float *out, const Plan &p,
                             GlsParams g, cudaStream_t s);

cudaError_t launch_pass2_nfft(const DevCurve *cv, int n_curves, int first, const float2 *inter,
                              float2 *out, const ulonglong2 *aux, unsigned *errflag, const Plan &p,
                              cudaStream_t s);

// Length templates (pass_kernels.cuh, instantiated in inst_*.cu).
template <int NG, int L1>
cudaError_t launch_pass1_t(const DevCurve *, int, int, const RecAB *, const RecC *,
                           const int *, const int *, float2 *, const Plan &, cudaStream_t);
template <int L2>
cudaError_t launch_pass2_gls_t(const DevCurve *, int, int, const float2 *, float *,
                               const Plan &, GlsParams, cudaStream_t);
template <int L2>
cudaError_t launch_pass2_nfft_t(const DevCurve *, int, int, const float2 *, float2 *,
                                const ulonglong2 *, unsigned *, const Plan &, cudaStream_t);

template <int NG, int L1>
cudaError_t preload_pass1_t();
template <int L2>
cudaError_t preload_pass2_t(int ng);
// Load the pass-1 and pass-2 kernels of a (G1, G2) plan for ngrids grids.
cudaError_t preload_pass_kernels(int G1, int G2, int ngrids);
// Load every preparation kernel of ngrids grids (prep.cu).
cudaError_t preload_prep_kernels(int ngrids, int fp32_positions);

// Fill the deconvolution table of an ES-window plan: G / 2 + 1 floats
// 1 / phihat(k'), |k'| <= G / 2 (kernels.cu: k_es_deconv).
cudaError_t launch_es_deconv(float *dst, long long G, int m, double beta, cudaStream_t s);
// The same by row blocks of R rows: dst[(rb L2 + q2) R + r], G floats.
cudaError_t launch_deconv_rows(const float *dtab, float *dst, int G1, int G2, int R, cudaStream_t s);

// Fill the tables of a plan (FFT tables of G1 and G2, then the inter-pass
// twiddles), fft_table_len(G1) + row_table_len(ng, G2) + G1 G2 entries at dst.
cudaError_t launch_plan_tables(float2 *dst, int G1, int G2, int B, int ng, cudaStream_t s);

// Host preparation of LombScargleMemory.setdata on the device for long raw
// (t, y, dy) curves, over their segments (one double4 of partA and partB
// each): k_raw_sums sums dy^-2, y dy^-2 and y; k_raw_finish writes w = dy^-2 /
// sum dy^-2 and yw = w (y - ybar) as FP32 and their partial sums.
cudaError_t launch_raw_long(const SegEntry *segs, int n_segs, const DevCurve *cv, const double *y,
                            const double *dy, double *ir, float *yw, float *w, double4 *partA,
                            double4 *partB, cudaStream_t s);
// Statistics of the descriptors of `list` from their curves' partials.
cudaError_t launch_fill_desc(DevCurve *cv, const int *list, int n, const double4 *partA,
                             const double4 *partB, int mode, cudaStream_t s);

// Per-curve best keys of the GLS pass 2 to (index, power); -1 / -1 where a
// curve had no valid power.
cudaError_t launch_best_finish(const unsigned long long *keys, int n, int64_t *best_k,
                               float *best_p, cudaStream_t s);

cudaError_t launch_spread_ref(const RefGridCurve *cv, int n_curves,
                              long long max_n, const double *t, const float *y,
                              float *grid, int m, float binv, float norm,
                              cudaStream_t s);

// Adjoint NFFT by FP64 direct summation: out[k] = sum_j y_j
// exp(+2 pi i (f0 + k df) t_j) for k < nf, complex128.
struct Direct64Curve {
    long long pt_off, n, nf, out_off;
    double f0, df;
    long long part_off;  // first partial sum of the curve within a part
    int splits;          // parts its points are cut into
};
// Parts to cut the points of a direct-sum batch into, so that `bins`
// frequencies in all still make enough CTAs of bins_per_cta (1: no parts).
int direct_splits(long long bins, int bins_per_cta, long long max_n);
int nfft_direct64_bins();
int gls_direct_bins();
// `part`: max_splits x part_stride partial sums (when max_splits > 1).
cudaError_t launch_nfft_direct64(const Direct64Curve *cv, int n_curves, long long max_nf,
                                 int max_splits, const double *t, const double *y, double2 *out,
                                 double2 *part, long long part_stride, cudaStream_t s);

// Finish of a caller-given reference-convention grid g of length ng (the
// reference's use_grid): shift by exp(2 pi i j ks / ng), inverse DFT, then
// for k < nf the phase exp(2 pi i n0 (k0 + k) / ng) and the Gaussian
// deconvolution exp(b (pi (k0 + k) / ng)^2); FP64, complex128.
struct GridFinishCurve {
    long long grid_off, ng, nf, out_off;
    double k0;   // f0 spp (tmax - tmin)
    double ks;   // k0 when the reference shifts (|f0| > 1e-9), else 0
    double n0;   // tmin / (spp (tmax - tmin)) ng
    double b;
};
cudaError_t launch_grid_finish(const GridFinishCurve *cv, int n_curves, long long max_nf,
                               const double2 *grid, double2 *out, cudaStream_t s);

// Multi-harmonic floating-mean GLS of one curve by FP64 direct sums, H
// harmonics (1..kMaxHarm): sums of w and yw against cos / sin of n phi, the
// regularised 2H x 2H normal equations solved per frequency (partial
// pivoting), P = (YX - sum XX) / YY; NaN where the system is singular.
constexpr int kMaxHarm = 8;
struct MhParams {
    double ybar, yy;
    double d[kMaxHarm];    // amplitude-prior regulariser per harmonic
    double cn0[kMaxHarm];  // prior centres of the cosine amplitudes
    double sn0[kMaxHarm];  // prior centres of the sine amplitudes
};
cudaError_t launch_mhgls_direct(int nharms, const double *t, const double *yw, const double *w,
                                long long n, const double *freqs, long long nf,
                                const MhParams &mp, double *out, cudaStream_t s);

// GLS powers by FP64 direct sums; aux of a descriptor holds its number of
// parts and inter_off its first partial sum.  `part`: max_splits x part_stride
// triples (when max_splits > 1).
cudaError_t launch_gls_direct(const DevCurve *cv, int n_curves, int max_nf, int max_splits,
                              const double *t, const float *yw, const float *w, float *out,
                              double2 *part, long long part_stride, GlsParams g, cudaStream_t s);

}  // namespace cuvgls
