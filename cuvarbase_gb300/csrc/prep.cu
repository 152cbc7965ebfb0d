// Preparation of the light curves for the pass kernels: weights and
// statistics of raw (t, y, dy) input, grid cells and band-centring phases of
// the points, and their counting sort by column block into spreading records.
//
// GB300 issues about two FP64 instructions per clock and SM, so FP64 is kept
// to what needs it: t - t0 and its product with df, one reciprocal and a few
// sums per raw point.  Positions are 64-bit fixed-point fractions of a turn
// (exact, wrap for free): the cell's row, column and offset, the doubled
// position and the centring phase are integer products.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace cuvgls {

namespace {

// ---------------------------------------------------------------------------
// positions
// ---------------------------------------------------------------------------
// floor(f n) of a fraction f, which becomes frac(f n); n < 2^31.
__device__ __forceinline__ int take_cells(u64 &f, unsigned n) {
    const u64 lo = (u64)(unsigned)f * n;
    const u64 hi = (f >> 32) * n + (lo >> 32);
    f = (hi << 32) | (unsigned)lo;
    return (int)(hi >> 32);
}

struct Geom {
    unsigned G1, G2;
    int lb;  // log2 of the columns per block
    __device__ __forceinline__ explicit Geom(int g)
        : G1((unsigned)g >> 16), G2(g & 0x1fff), lb((g >> 13) & 7) {}
};

struct Cell {
    int rc;      // row << 16 | column
    float frac;  // offset in the cell
};

// Cell of the fraction f on the grid; NaN offset where the position was not
// finite.
__device__ __forceinline__ Cell cell_at(u64 f, const Geom &g, bool nan) {
    Cell c;
    const int row = take_cells(f, g.G1), col = take_cells(f, g.G2);
    c.rc = row << 16 | col;
    c.frac = nan ? __int_as_float(0x7fffffff)
                 : __uint2float_rn((unsigned)(f >> 32)) * 2.3283064365386963e-10f;
    return c;
}

// The all-FP32 variant (t cast to float first, as
// cuvarbase/lombscargle.py:259 does).
__device__ __forceinline__ Cell cell_at32(float x, const Geom &g) {
    const int Gi = (int)(g.G1 * g.G2);
    const float u = (x - floorf(x)) * (float)Gi, fl = floorf(u);
    int ci = (int)fl;
    if (ci >= Gi) ci -= Gi;
    if (ci < 0) ci = 0;
    return Cell{(int)((unsigned)ci / g.G2) << 16 | (int)((unsigned)ci % g.G2), u - fl};
}

// Band centre kc = ki + kf of a descriptor.  GLS centres are whole numbers
// (WHOLE); the adjoint NFFT's f0 / df need not be.
struct Centre {
    long long ki;
    double kf;
};
template <bool WHOLE>
__device__ __forceinline__ Centre centre_of(double kc) {
    if (WHOLE) return Centre{(long long)kc, 0.0};
    const double f = floor(kc);
    return Centre{(long long)f, kc - f};
}

// exp(2 pi i kc x) for x turns with fraction f.
template <bool WHOLE>
__device__ __forceinline__ float2 centre_phase(u64 f, double x, const Centre &k) {
    u64 th = (u64)k.ki * f;
    if (!WHOLE && k.kf != 0.0) th += turns64(k.kf * x);
    return turn_phasor(th);
}

// Cells (x and 2x) and centring phase of one point; a point whose t is not
// finite is taken at t0 and flagged.
struct Place {
    Cell a, c;
    float2 ph;
};
template <int NG, bool F32>
__device__ __forceinline__ Place place_of(double tj, double tref, double df, const Geom &g,
                                          double kc, const Centre &k) {
    Place p;
    if (!F32) {
        const double x = (tj - tref) * df;
        const u64 f = turns64(x);
        const bool nan = !isfinite(x);
        p.a = cell_at(f, g, nan);
        if (NG == 3) p.c = cell_at(f << 1, g, nan);
        p.ph = centre_phase<NG == 3>(f, x, k);
        if (nan) p.ph.x = __int_as_float(0x7fffffff);
    } else {
        const float x = ((float)tj - (float)tref) * (float)df;
        p.a = cell_at32(x, g);
        if (NG == 3) p.c = cell_at32(2.0f * x, g);
        float th = (float)kc * x;
        th -= floorf(th);
        sincospif(2.0f * th, &p.ph.y, &p.ph.x);
    }
    return p;
}
__device__ __forceinline__ int bin_of(const Cell &c, const Geom &g) { return (c.rc & 0xFFFF) >> g.lb; }

__device__ __forceinline__ RecAB rec_ab(const Place &p, float a, float w) {
    return RecAB{p.a.rc, p.a.frac, cscale(p.ph, a), cscale(p.ph, w)};
}
__device__ __forceinline__ RecC rec_c(const Place &p, float w) {
    const float2 ph2 = make_float2(p.ph.x * p.ph.x - p.ph.y * p.ph.y, 2.f * p.ph.x * p.ph.y);
    return RecC{p.c.rc, p.c.frac, cscale(ph2, w)};
}

// Output phase of the adjoint NFFT of a descriptor: out[k] needs
// exp(2 pi i (kc + k') df t0): the turns kc df t0 and df t0 as 64-bit
// fractions.
__device__ __forceinline__ void write_aux(const DevCurve &cv, double tref,
                                          ulonglong2 *__restrict__ aux) {
    aux[cv.aux] = make_ulonglong2(turns64(cv.kc * cv.df * tref), turns64(cv.df * tref));
}

// ---------------------------------------------------------------------------
// sums
// ---------------------------------------------------------------------------
// Totals of four values over a warp in 6 FP64 adds per lane (20 for four
// butterflies): the first two steps also share the values out.  Lane l
// returns the total of value l >> 3.
__device__ __forceinline__ double warp_sum4(double a, double b, double c, double d, int lane) {
    const bool h = lane & 16, q = lane & 8;
    double s0 = (h ? c : a) + __shfl_xor_sync(0xffffffffu, h ? a : c, 16);
    const double s1 = (h ? d : b) + __shfl_xor_sync(0xffffffffu, h ? b : d, 16);
    s0 = (q ? s1 : s0) + __shfl_xor_sync(0xffffffffu, q ? s0 : s1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    return s0;
}
// Totals of four values over the CTA's first `warps` warps (the others hold
// none) into part[0 .. 3], written by threads 0 .. 3; the caller synchronises
// before they are read.  wred: 4 NT / 32.
template <int NT>
__device__ __forceinline__ void block_sum4(double a, double b, double c, double d, int warps,
                                           double *wred, double *part, int tid) {
    const int lane = tid & 31, wid = tid >> 5;
    if (wid < warps) {
        const double v = warp_sum4(a, b, c, d, lane);
        if ((lane & 7) == 0) wred[wid * 4 + (lane >> 3)] = v;
    }
    __syncthreads();
    if (wid == 0) {  // lane l: value l & 3 of warps l >> 2 (and 8 more)
        double s = (lane >> 2) < warps ? wred[lane] : 0.0;
        if (NT > 256 && warps > 8) s += 8 + (lane >> 2) < warps ? wred[32 + lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 2; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane < 4) part[lane] = s;
    }
}

// Normalisation and statistics of a descriptor from its curve's totals a =
// (sum dy^-2, sum y dy^-2, sum and count of the non-NaN y), b = (YY, sum yw,
// sum w).  ybar, which only the standard mode reads, is relative to the
// unweighted nan-mean of y, as cuvarbase's normalize_light_curves leaves it.
__device__ __forceinline__ void fill_stats(DevCurve &cv, double4 a, double4 b, int mode) {
    const double yy = b.x;
    double norm = 1.0;
    if (mode == 1) norm = 1.0 / yy;
    else if (mode == 0) {
        const double ybar = a.y / a.x - a.z / a.w;
        norm = 1.0 / (yy + ybar * ybar);
        cv.ybar = (float)ybar;
    }
    cv.yy_inv = (float)norm;
    cv.yw_sum = (float)b.y;
    cv.w_sum = (float)b.z;
}

// ---------------------------------------------------------------------------
// one curve per CTA or cluster
// ---------------------------------------------------------------------------
// Shared memory: packed counts (grid C << 16 | grids A, B) per column block,
// then their offsets (nb + 1) and, in a cluster, the counts of the earlier CTAs.
__host__ __device__ constexpr int prep_smem(int nb, bool cluster) {
    return (nb + (nb + 1) + (cluster ? nb : 0)) * 4;
}

}  // namespace

// Everything the pass kernels need of a curve, in one launch: raw weights and
// statistics (RAW), cells, counts per column block, their scan, records.  The
// points stay in registers (PPT per thread).  CL: the curve's points are
// shared out over the first CTAs of a cluster, which exchange their partial
// sums and counts through distributed shared memory (at most 2^15 points, so
// a count fits 16 bits); CTAs without points leave at once.  `chunk` points go
// to each CTA, or with 0 an even share of the curve (at least one per thread).
//
// Bound by the latency of its few steps (barriers, FP64 sums, shared
// atomics) for one curve and by FP64 issue for many; one launch instead of
// the three to six that passed yw, w, counts and cursors through memory.
template <int NT, int PPT, bool CL, bool RAW, int NG, bool F32>
__global__ void __launch_bounds__(NT)
k_prep(const PrepArrays A, const __grid_constant__ DescParam D, const int *__restrict__ list,
       int csize, int chunk) {
    extern __shared__ __align__(16) unsigned cnt[];
    __shared__ double wred[4 * NT / 32], part[8], mean[2];
    __shared__ int ws[32];
    const int tid = threadIdx.x;
    if (A.trigger) pdl_trigger();  // pass 1 may be set up
    const int ci = CL ? blockIdx.x / csize : blockIdx.x, rank = CL ? blockIdx.x % csize : 0;
    const int di = list ? list[ci] : ci;
    const DevCurve &cv = D.n ? D.cv[di] : A.cv[di];
    const int n = cv.n;
    if (CL && chunk == 0) chunk = max(NT, ((n - 1) / csize + 32) & ~31);
    const int na = CL ? (n - 1) / chunk + 1 : 1;  // CTAs with points
    if (CL && rank >= na) return;
    const Geom g(cv.geom);
    const int nb = (int)(g.G2 >> g.lb);
    unsigned *off = cnt + nb, *pre = off + nb + 1;
    for (int i = tid; i < nb; i += NT) cnt[i] = 0;
    const long long po = cv.pt_off;
    const double tref = A.t[po], df = cv.df, kc = cv.kc;
    const Centre k = centre_of<NG == 3>(kc);
    const int j0 = rank * chunk + tid, j1 = CL ? min(n, (rank + 1) * chunk) : n;
    const int warps = min(NT / 32, (j1 - j0 + tid + 31) / 32);  // with points
    float a[PPT], w[PPT];
    double y[RAW ? PPT : 1], ir[RAW ? PPT : 1];
    if (RAW) {
        double sw = 0.0, swy = 0.0, sy = 0.0;
        int cy = 0;
#pragma unroll
        for (int q = 0; q < PPT; ++q) {
            const int j = j0 + q * NT;
            ir[q] = 0.0;
            y[q] = 0.0;
            if (j < j1) {
                const double dj = A.rdy[po + j];
                y[q] = A.ry[po + j];
                ir[q] = 1.0 / (dj * dj);
                sw += ir[q];
                swy = fma(ir[q], y[q], swy);
                if (!isnan(y[q])) { sy += y[q]; ++cy; }
            }
        }
        block_sum4<NT>(sw, swy, sy, (double)cy, warps, wred, part, tid);
        if (CL) cg::this_cluster().sync();
        else __syncthreads();
        if (tid == 0) {
            double tw = 0.0, ty = 0.0;
            for (int r = 0; r < na; ++r) {
                const double *pr = CL ? cg::this_cluster().map_shared_rank(part, r) : part;
                tw += pr[0];
                ty += pr[1];
            }
            mean[0] = ty / tw;
            mean[1] = 1.0 / tw;
        }
        __syncthreads();
        const double ybar_w = mean[0], inv = mean[1];
        double yy = 0.0, ys = 0.0, wsum = 0.0;
#pragma unroll
        for (int q = 0; q < PPT; ++q) {
            a[q] = 0.f;
            w[q] = 0.f;
            if (j0 + q * NT < j1) {
                const double wj = ir[q] * inv, d = y[q] - ybar_w, wd = wj * d;
                a[q] = (float)wd;
                w[q] = (float)wj;
                yy = fma(wd, d, yy);
                ys += (double)a[q];
                wsum += (double)w[q];
            }
        }
        block_sum4<NT>(yy, ys, wsum, 0.0, warps, wred, part + 4, tid);
    } else {
#pragma unroll
        for (int q = 0; q < PPT; ++q) {
            const int j = j0 + q * NT;
            a[q] = j < j1 ? A.ya[po + j] : 0.f;
            w[q] = NG == 3 && j < j1 ? A.wv[po + j] : 0.f;
        }
        __syncthreads();  // counts zeroed
    }
    Place p[PPT];
    int rank_ac[PPT];  // of the point among its CTA's in the same blocks (A, C << 16)
    bool bad = false;
#pragma unroll
    for (int q = 0; q < PPT; ++q) {
        const int j = j0 + q * NT;
        rank_ac[q] = 0;
        if (j < j1) {
            double tj = A.t[po + j];
            if (!(isfinite(tj) && isfinite(a[q]) && isfinite(w[q]))) {
                bad = true;
                tj = isfinite(tj) ? tj : tref;
                a[q] = 0.f;
                w[q] = 0.f;
            }
            p[q] = place_of<NG, F32>(tj, tref, df, g, kc, k);
            rank_ac[q] = atomicAdd(&cnt[bin_of(p[q].a, g)], 1u) & 0xFFFFu;
            if (NG == 3) rank_ac[q] |= atomicAdd(&cnt[bin_of(p[q].c, g)], 0x10000u) & 0xFFFF0000u;
        }
    }
    // offsets: scan of the curve's counts, plus the earlier CTAs' counts
    if (CL) {
        cg::this_cluster().sync();
        for (int i = tid; i < nb; i += NT) {
            unsigned tot = 0, before = 0;
            for (int r = 0; r < na; ++r) {
                const unsigned c = cg::this_cluster().map_shared_rank(cnt, r)[i];
                if (r < rank) before += c;
                tot += c;
            }
            off[i] = tot;
            pre[i] = before;
        }
    } else {
        __syncthreads();
        for (int i = tid; i < nb; i += NT) off[i] = cnt[i];
    }
    if ((RAW || D.n) && rank == 0 && tid == 0) {
        if (D.n) A.cv[di] = cv;
        if (RAW) {
            double4 ta = make_double4(0.0, 0.0, 0.0, 0.0), tb = ta;
            for (int r = 0; r < na; ++r) {
                const double *pr = CL ? cg::this_cluster().map_shared_rank(part, r) : part;
                ta.x += pr[0]; ta.y += pr[1]; ta.z += pr[2]; ta.w += pr[3];
                tb.x += pr[4]; tb.y += pr[5]; tb.z += pr[6];
            }
            fill_stats(A.cv[di], ta, tb, A.mode);
        }
    }
    // after the last read of another CTA's shared memory
    if (CL) cg::this_cluster().barrier_arrive();
    __syncthreads();
    block_scan_counts<NT>((int *)off, nb, ws, tid);
    if (rank == 0) {
        int *bA = A.binsAB + cv.bin_off, *bC = A.binsC + cv.bin_off;
        for (int i = tid; i <= nb; i += NT) {
            bA[i] = (int)(off[i] & 0xFFFFu);
            if (NG == 3) bC[i] = (int)(off[i] >> 16);
        }
    }
    RecAB *rA = A.recAB + cv.rec_off;
    RecC *rC = A.recC + cv.rec_off;
#pragma unroll
    for (int q = 0; q < PPT; ++q) {
        if (j0 + q * NT >= j1) continue;
        const int binA = bin_of(p[q].a, g), binC = NG == 3 ? bin_of(p[q].c, g) : 0;
        const unsigned oa = off[binA] + (CL ? pre[binA] : 0);
        rA[(oa & 0xFFFFu) + (rank_ac[q] & 0xFFFF)] = rec_ab(p[q], a[q], w[q]);
        if (NG == 3) {
            const unsigned oc = off[binC] + (CL ? pre[binC] : 0);
            rC[(oc >> 16) + ((unsigned)rank_ac[q] >> 16)] = rec_c(p[q], w[q]);
        }
    }
    if (bad) atomicOr(A.errflag, 1u);
    if (A.aux != nullptr && rank == 0 && tid == 0) write_aux(cv, tref, A.aux);
    // a CTA's shared memory stays until the others have read it
    if (CL) cg::this_cluster().barrier_wait();
    // this kernel's end says that the one beside it has ended too
    if (A.beside && rank == 0) pdl_wait();
}

// ---------------------------------------------------------------------------
// long curves: a chain of kernels over segments
// ---------------------------------------------------------------------------
// One CTA per descriptor: its segments at raw_seg.
__global__ void k_seg_fill(const DevCurve *__restrict__ cvs, SegEntry *__restrict__ segs) {
    const DevCurve &cv = cvs[blockIdx.x];
    const int ns = seg_count(cv.n);
    for (int i = threadIdx.x; i < ns; i += blockDim.x)
        segs[cv.raw_seg + i] = SegEntry{(int)blockIdx.x, i * kSegPoints};
}

// Count of one segment: shared-memory histogram of the column blocks
// (packed), added to the descriptor's counts (zeroed before the launch).
// Segments of 4,096 points: a dense curve has about two points per block in
// each, and every nonzero block costs a global atomic.
template <int NG, bool F32>
__global__ void __launch_bounds__(kSegThreads)
k_bin_count(const PrepArrays A, const SegEntry *__restrict__ segs) {
    __shared__ unsigned h[kMaxBins];
    const SegEntry sg = segs[blockIdx.x];
    const DevCurve &cv = A.cv[sg.desc];
    const int tid = threadIdx.x;
    const Geom g(cv.geom);
    const int nb = (int)(g.G2 >> g.lb);
    for (int i = tid; i < nb; i += kSegThreads) h[i] = 0;
    __syncthreads();
    const long long po = cv.pt_off;
    const double tref = A.t[po], df = cv.df;
    const int cntp = min(cv.n - sg.start, kSegPoints);
#pragma unroll 4
    for (int i = tid; i < cntp; i += kSegThreads) {
        double tj = A.t[po + sg.start + i];
        if (!isfinite(tj)) tj = tref;
        const Place p = place_of<NG, F32>(tj, tref, df, g, 0.0, Centre{0, 0.0});
        atomicAdd(&h[bin_of(p.a, g)], 1u);
        if (NG == 3) atomicAdd(&h[bin_of(p.c, g)], 0x10000u);
    }
    __syncthreads();
    int *bA = A.binsAB + cv.bin_off, *bC = A.binsC + cv.bin_off;
    for (int i = tid; i < nb; i += kSegThreads) {
        const unsigned v = h[i];
        if (v & 0xFFFFu) atomicAdd(&bA[i], (int)(v & 0xFFFFu));
        if (NG == 3 && (v >> 16)) atomicAdd(&bC[i], (int)(v >> 16));
    }
}

// One CTA per descriptor: bin offsets and cursors from the counts, and the
// output phase of the adjoint NFFT in aux.
__global__ void __launch_bounds__(256)
k_bin_scan(const PrepArrays A, const int *__restrict__ list, int ngrids) {
    __shared__ int h[kMaxBins + 1];
    __shared__ int ws[32];
    const DevCurve &cv = A.cv[list ? list[blockIdx.x] : blockIdx.x];
    const int tid = threadIdx.x;
    const Geom g(cv.geom);
    const int nb = (int)(g.G2 >> g.lb);
    for (int k = 0; k < (ngrids == 3 ? 2 : 1); ++k) {
        int *b = (k ? A.binsC : A.binsAB) + cv.bin_off, *c = (k ? A.curC : A.curAB) + cv.bin_off;
        for (int i = tid; i < nb; i += 256) h[i] = b[i];
        __syncthreads();
        block_scan_counts<256>(h, nb, ws, tid);
        for (int i = tid; i <= nb; i += 256) {
            b[i] = h[i];
            if (i < nb) c[i] = h[i];
        }
        __syncthreads();  // h is reused
    }
    if (A.aux != nullptr && tid == 0) write_aux(cv, A.t[cv.pt_off], A.aux);
}

// One CTA per segment: a shared-memory rank of each point within its column
// block, one global reservation per block for the segment's run, then the
// records.  Only the ranks stay in registers: the places are computed again
// for the records, which costs two FP64 instructions a point and lets two
// CTAs share an SM (102 registers and one CTA otherwise).
template <int NG, bool F32>
__global__ void __launch_bounds__(kSegThreads, 2)
k_bin_scatter(const PrepArrays A, const SegEntry *__restrict__ segs) {
    __shared__ unsigned h[kMaxBins];         // packed counts
    __shared__ int oA[kMaxBins], oC[kMaxBins];
    const SegEntry sg = segs[blockIdx.x];
    const DevCurve &cv = A.cv[sg.desc];
    const int tid = threadIdx.x, n = cv.n;
    const Geom g(cv.geom);
    const int nb = (int)(g.G2 >> g.lb);
    for (int i = tid; i < nb; i += kSegThreads) h[i] = 0;
    __syncthreads();
    const long long po = cv.pt_off + sg.start;
    const double tref = A.t[cv.pt_off], df = cv.df, kc = cv.kc;
    const Centre k = centre_of<NG == 3>(kc);
    const int cntp = min(n - sg.start, kSegPoints);
    int rank_ac[kSegPpt];
    bool bad = false, lost = false;
#pragma unroll
    for (int q = 0; q < kSegPpt; ++q) {
        const int i = tid + q * kSegThreads;
        if (i < cntp) {
            double tj = A.t[po + i];
            if (!isfinite(tj)) tj = tref;
            const Place p = place_of<NG, F32>(tj, tref, df, g, kc, k);
            rank_ac[q] = atomicAdd(&h[bin_of(p.a, g)], 1u) & 0xFFFFu;
            if (NG == 3) rank_ac[q] |= atomicAdd(&h[bin_of(p.c, g)], 0x10000u) & 0xFFFF0000u;
        }
    }
    __syncthreads();
    for (int i = tid; i < nb; i += kSegThreads) {
        const unsigned v = h[i];
        if (v & 0xFFFFu) oA[i] = atomicAdd(&A.curAB[cv.bin_off + i], (int)(v & 0xFFFFu));
        if (NG == 3 && (v >> 16)) oC[i] = atomicAdd(&A.curC[cv.bin_off + i], (int)(v >> 16));
    }
    __syncthreads();
    RecAB *rA = A.recAB + cv.rec_off;
    RecC *rC = A.recC + cv.rec_off;
#pragma unroll
    for (int q = 0; q < kSegPpt; ++q) {
        const int i = tid + q * kSegThreads;
        if (i >= cntp) continue;
        double tj = A.t[po + i];
        float a = A.ya[po + i], w = NG == 3 ? A.wv[po + i] : 0.f;
        if (!(isfinite(tj) && isfinite(a) && isfinite(w))) {
            bad = true;
            tj = isfinite(tj) ? tj : tref;
            a = 0.f;
            w = 0.f;
        }
        const Place p = place_of<NG, F32>(tj, tref, df, g, kc, k);
        // a slot outside the curve's n records would mean that the count and
        // the scatter binned a point differently: flag it, write nothing
        const int sa = oA[bin_of(p.a, g)] + (rank_ac[q] & 0xFFFF);
        if ((unsigned)sa < (unsigned)n) rA[sa] = rec_ab(p, a, w);
        else lost = true;
        if (NG == 3) {
            const int sc = oC[bin_of(p.c, g)] + (int)((unsigned)rank_ac[q] >> 16);
            if ((unsigned)sc < (unsigned)n) rC[sc] = rec_c(p, w);
            else lost = true;
        }
    }
    if (bad) atomicOr(A.errflag, 1u);
    if (lost) atomicOr(A.errflag, 4u);
}

// Sum of the partials part[first .. first + n) in a fixed order (lane
// stride, then a butterfly): every lane gets the same total, and every
// caller reducing the same range gets the same bits.
__device__ __forceinline__ double4 warp_sum_parts(const double4 *__restrict__ part, int first,
                                                  int n, int lane) {
    double4 a = make_double4(0.0, 0.0, 0.0, 0.0);
    for (int k = lane; k < n; k += 32) {
        const double4 v = part[first + k];
        a.x += v.x;
        a.y += v.y;
        a.z += v.z;
        a.w += v.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
        a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
        a.z += __shfl_xor_sync(0xffffffffu, a.z, o);
        a.w += __shfl_xor_sync(0xffffffffu, a.w, o);
    }
    return a;
}

// Raw input, step 1, one CTA per segment: sum dy^-2, sum y dy^-2 and the
// nan-mean parts (sum and count of the non-NaN y) into partA; each dy^-2 is
// kept in ir for the second step (one FP64 division per point).
__global__ void __launch_bounds__(kSegThreads)
k_raw_sums(const SegEntry *__restrict__ segs, const DevCurve *__restrict__ cvs,
           const double *__restrict__ y, const double *__restrict__ dy,
           double *__restrict__ ir, double4 *__restrict__ partA) {
    __shared__ double wred[4 * kSegThreads / 32], part[4];
    const SegEntry sg = segs[blockIdx.x];
    const DevCurve &cv = cvs[sg.desc];
    const int tid = threadIdx.x;
    const long long o = cv.pt_off + sg.start;
    const int cntp = min(cv.n - sg.start, kSegPoints);
    double sw = 0.0, swy = 0.0, sy = 0.0;
    int cy = 0;
    for (int i = tid; i < cntp; i += kSegThreads) {
        const double yj = y[o + i], dj = dy[o + i];
        const double wj = 1.0 / (dj * dj);
        ir[o + i] = wj;
        sw += wj;
        swy = fma(wj, yj, swy);
        if (!isnan(yj)) { sy += yj; ++cy; }
    }
    block_sum4<kSegThreads>(sw, swy, sy, (double)cy, kSegThreads / 32, wred, part, tid);
    __syncthreads();
    if (tid == 0)
        partA[cv.raw_seg + sg.start / kSegPoints] = make_double4(part[0], part[1], part[2], part[3]);
}

// Step 2, one CTA per segment: w = dy^-2 / sum dy^-2 and yw = w (y - ybar) as
// FP32, and the partial sums of YY and of the stored yw and w.
__global__ void __launch_bounds__(kSegThreads)
k_raw_finish(const SegEntry *__restrict__ segs, const DevCurve *__restrict__ cvs,
             const double *__restrict__ y, const double *__restrict__ ir,
             float *__restrict__ yw, float *__restrict__ w, const double4 *__restrict__ partA,
             double4 *__restrict__ partB) {
    __shared__ double wred[4 * kSegThreads / 32], part[4], mean[2];
    const SegEntry sg = segs[blockIdx.x];
    const DevCurve &cv = cvs[sg.desc];
    const int tid = threadIdx.x;
    if (tid < 32) {
        const double4 a = warp_sum_parts(partA, cv.raw_seg, seg_count(cv.n), tid);
        if (tid == 0) {
            mean[0] = a.y / a.x;
            mean[1] = 1.0 / a.x;
        }
    }
    __syncthreads();
    const double ybar_w = mean[0], inv = mean[1];
    const long long o = cv.pt_off + sg.start;
    const int cntp = min(cv.n - sg.start, kSegPoints);
    double yy = 0.0, ys = 0.0, ws = 0.0;
    for (int i = tid; i < cntp; i += kSegThreads) {
        const double wj = ir[o + i] * inv, d = y[o + i] - ybar_w, wd = wj * d;
        const float ywf = (float)wd, wf = (float)wj;
        yy = fma(wd, d, yy);
        yw[o + i] = ywf;
        w[o + i] = wf;
        ys += (double)ywf;
        ws += (double)wf;
    }
    block_sum4<kSegThreads>(yy, ys, ws, 0.0, kSegThreads / 32, wred, part, tid);
    __syncthreads();
    if (tid == 0)
        partB[cv.raw_seg + sg.start / kSegPoints] = make_double4(part[0], part[1], part[2], 0.0);
}

// Step 3, one warp per descriptor: its curve's totals from the partials, then
// its statistics.
__global__ void __launch_bounds__(128)
k_fill_desc(DevCurve *__restrict__ cvs, const int *__restrict__ list, int n,
            const double4 *__restrict__ partA, const double4 *__restrict__ partB, int mode) {
    const int i = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (i >= n) return;  // whole warps
    const int lane = threadIdx.x & 31;
    DevCurve &cv = cvs[list[i]];
    const int ns = seg_count(cv.n);
    const double4 a = warp_sum_parts(partA, cv.raw_seg, ns, lane);
    const double4 b = warp_sum_parts(partB, cv.raw_seg, ns, lane);
    if (lane == 0) fill_stats(cv, a, b, mode);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
namespace {

template <int NT, int PPT, bool CL, bool RAW, int NG, bool F32>
cudaError_t prep_t(const PrepArrays &a, const DescParam &d, const int *list, int n, int csize,
                   int chunk, bool beside, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n * csize);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = prep_smem(a.max_nb, CL);
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    cfg.attrs = at;
    if (CL) {
        cudaLaunchAttribute &x = at[cfg.numAttrs++];
        x.id = cudaLaunchAttributeClusterDimension;
        x.val.clusterDim.x = csize;
        x.val.clusterDim.y = 1;
        x.val.clusterDim.z = 1;
    }
    if (beside) {
        cudaLaunchAttribute &x = at[cfg.numAttrs++];
        x.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        x.val.programmaticStreamSerializationAllowed = 1;
    }
    PrepArrays b = a;
    b.trigger = 1;
    b.beside = beside;
    return cudaLaunchKernelEx(&cfg, k_prep<NT, PPT, CL, RAW, NG, F32>, b, d, list, csize, chunk);
}

template <int NT, int PPT, bool CL>
cudaError_t prep_kind(const PrepArrays &a, const DescParam &d, const int *list, int n, int csize, int chunk, int raw,
                      int ngrids, int f32, bool beside, cudaStream_t s) {
    if (raw)
        return f32 ? prep_t<NT, PPT, CL, true, 3, true>(a, d, list, n, csize, chunk, beside, s)
                   : prep_t<NT, PPT, CL, true, 3, false>(a, d, list, n, csize, chunk, beside, s);
    if (ngrids == 3)
        return f32 ? prep_t<NT, PPT, CL, false, 3, true>(a, d, list, n, csize, chunk, beside, s)
                   : prep_t<NT, PPT, CL, false, 3, false>(a, d, list, n, csize, chunk, beside, s);
    return f32 ? prep_t<NT, PPT, CL, false, 1, true>(a, d, list, n, csize, chunk, beside, s)
               : prep_t<NT, PPT, CL, false, 1, false>(a, d, list, n, csize, chunk, beside, s);
}

// Loads a kernel that a first launch would load.
template <typename K>
cudaError_t load(K kernel) {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, kernel);
}
template <int NG, bool F32, bool RAW>
cudaError_t load_prep() {
    cudaError_t e = load(k_prep<kPrepThreads, kPrepPpt, false, RAW, NG, F32>);
    if (e == cudaSuccess) e = load(k_prep<kPrepThreads, kPrepPpt, true, RAW, NG, F32>);
    if (e == cudaSuccess) e = load(k_prep<kShortThreads, kShortPpt, false, RAW, NG, F32>);
    if (e == cudaSuccess) e = load(k_prep<kWideThreads, kWidePpt, true, RAW, NG, F32>);
    return e;
}
template <int NG, bool F32>
cudaError_t load_all() {
    cudaError_t e = load_prep<NG, F32, false>();
    if constexpr (NG == 3) {
        if (e == cudaSuccess) e = load_prep<NG, F32, true>();
        if (e == cudaSuccess) e = load(k_raw_sums);
        if (e == cudaSuccess) e = load(k_raw_finish);
        if (e == cudaSuccess) e = load(k_fill_desc);
    }
    if (e == cudaSuccess) e = load(k_bin_count<NG, F32>);
    if (e == cudaSuccess) e = load(k_bin_scan);
    if (e == cudaSuccess) e = load(k_bin_scatter<NG, F32>);
    return e;
}

}  // namespace

cudaError_t preload_prep_kernels(int ngrids, int fp32_positions) {
    if (ngrids == 3) return fp32_positions ? load_all<3, true>() : load_all<3, false>();
    return fp32_positions ? load_all<1, true>() : load_all<1, false>();
}

cudaError_t launch_prep(const PrepArrays &a, const DescParam &d, const int *list, int n, int cls,
                        int max_n, int raw, int ngrids, int fp32_positions, bool beside,
                        cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (a.max_nb > kMaxBins || max_n > kFusePoints) return cudaErrorInvalidValue;
    if (cls == 0) {
        if (max_n > kPrepPoints) return cudaErrorInvalidValue;
        return prep_kind<kPrepThreads, kPrepPpt, false>(a, d, list, n, 1, kPrepPoints, raw, ngrids,
                                                        fp32_positions, beside, s);
    }
    if (cls == kPrepShort) {
        if (max_n > kShortPoints) return cudaErrorInvalidValue;
        return prep_kind<kShortThreads, kShortPpt, false>(a, d, list, n, 1, kShortPoints, raw,
                                                          ngrids, fp32_positions, beside, s);
    }
    if (cls == kPrepWide) {
        int csize = 1;
        while (csize * kWidePoints < max_n) csize *= 2;
        return prep_kind<kWideThreads, kWidePpt, true>(a, d, list, n, csize, kWidePoints, raw, ngrids,
                                                       fp32_positions, beside, s);
    }
    if (max_n > kMaxCluster * kPrepPoints) return cudaErrorInvalidValue;
    int csize = 1;
    const bool spread = cls == kPrepSpread;
    while (csize < kMaxCluster && csize * (spread ? kPrepThreads : kPrepPoints) < max_n) csize *= 2;
    if (csize == 1)
        return prep_kind<kPrepThreads, kPrepPpt, false>(a, d, list, n, 1, kPrepPoints, raw, ngrids,
                                                        fp32_positions, beside, s);
    return prep_kind<kPrepThreads, kPrepPpt, true>(a, d, list, n, csize, spread ? 0 : kPrepPoints, raw,
                                                   ngrids, fp32_positions, beside, s);
}

cudaError_t launch_bin_long(const PrepArrays &a, const SegEntry *segs, int n_segs, const int *list,
                            int n, int ngrids, int fp32_positions, cudaStream_t s) {
    if (n_segs <= 0 || n <= 0) return cudaSuccess;
    if (a.max_nb > kMaxBins) return cudaErrorInvalidValue;
#define CUVGLS_BIN(NG, F32)                                            \
    do {                                                               \
        k_bin_count<NG, F32><<<n_segs, kSegThreads, 0, s>>>(a, segs);   \
        k_bin_scan<<<n, 256, 0, s>>>(a, list, NG);                      \
        k_bin_scatter<NG, F32><<<n_segs, kSegThreads, 0, s>>>(a, segs); \
    } while (0)
    if (ngrids == 3) {
        if (fp32_positions) CUVGLS_BIN(3, true);
        else CUVGLS_BIN(3, false);
    } else {
        if (fp32_positions) CUVGLS_BIN(1, true);
        else CUVGLS_BIN(1, false);
    }
#undef CUVGLS_BIN
    return cudaGetLastError();
}

cudaError_t launch_seg_fill(const DevCurve *cv, int n, SegEntry *segs, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_seg_fill<<<n, 64, 0, s>>>(cv, segs);
    return cudaGetLastError();
}

cudaError_t launch_raw_long(const SegEntry *segs, int n_segs, const DevCurve *cv, const double *y,
                            const double *dy, double *ir, float *yw, float *w, double4 *partA,
                            double4 *partB, cudaStream_t s) {
    if (n_segs <= 0) return cudaSuccess;
    k_raw_sums<<<n_segs, kSegThreads, 0, s>>>(segs, cv, y, dy, ir, partA);
    k_raw_finish<<<n_segs, kSegThreads, 0, s>>>(segs, cv, y, ir, yw, w, partA, partB);
    return cudaGetLastError();
}

cudaError_t launch_fill_desc(DevCurve *cv, const int *list, int n, const double4 *partA,
                             const double4 *partB, int mode, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_fill_desc<<<(n + 3) / 4, 128, 0, s>>>(cv, list, n, partA, partB, mode);
    return cudaGetLastError();
}

}  // namespace cuvgls
