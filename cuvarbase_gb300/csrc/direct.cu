// Direct sums in 64 bits: use_fft=False (k_gls_direct), use_double
// (k_nfft_direct64) and the multi-harmonic model (k_mhgls_direct).
//
// GB300 issues about two FP64 multiply-adds per clock and SM, so in FP64 these
// kernels are bound by their instruction count and by nothing else; a
// sincospi per (point, frequency) alone is some 25 of them.  On a uniform
// frequency grid the phasors factor instead.  A lane owns the 2 M + 1
// consecutive bins K - M .. K + M; with E = v exp(i K x) and the step phasors
// cos bx, sin bx (b = 1 .. M), which are the same for every lane,
//   sum v exp(i (K + b) x) = (P1 - P2) + i (P3 + P4),
//   sum v exp(i (K - b) x) = (P1 + P2) + i (P3 - P4),
//   P1 = sum Re E cos bx, P2 = sum Im E sin bx,
//   P3 = sum Im E cos bx, P4 = sum Re E sin bx,
// which is two multiply-adds per complex bin and point.  exp(i K x) is the
// product of a coarse and a fine table entry (32 centres from 4 + 8).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "gls_math.cuh"
#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace cuvgls {

namespace {

constexpr int kDirThreads = 256;
constexpr int kDirWarps = kDirThreads / 32;
constexpr int kCoarse = 4, kFine = 8;  // 32 centres

__device__ __forceinline__ double2 zturn(double turns) {  // exp(2 pi i turns)
    double s, c;
    sincospi(2.0 * (turns - floor(turns)), &s, &c);
    return make_double2(c, s);
}

// ---- fixed point ----
// Phasors are integers in units of 2^-56, and so are values on them (E below),
// of the power of two above the largest value of a run.  The step phasors that
// multiply E for the sums are in units of 2^-54, which makes those products
// units of E too, and a run is short enough that its sums stay within 2^62.  A
// factor is split into 27 low bits (signed) and the rest, and a product takes
// three 32 x 32 -> 64 bit multiply-adds (the low x low part, below 2^-2 of a
// unit, is left out).  These run at 24 or more per clock and SM, against 2 of
// FP64: 2.4 FP64 instructions per bin become 6 of them.  2^-56 of the largest
// value is less than what a sum in FP64 that holds this value rounds to at every
// addition: one value a thousand times the others, error of the sums relative to
// it (rms over bins, worst place of the value within its power of two), in FP64
// in sequence and here: 60 points 2.7e-16 and 1.4e-16, 300 points 6.4e-16 and
// 3.2e-16, 2,000 points 1.6e-15 and 3.6e-16, 8,192 points 3.3e-15 and 5.2e-16
// (7.1e-14 with one run for all of them).
using i64 = long long;
struct Fx {
    int h, l;  // h 2^27 + l, |l| <= 2^26
};
struct Cx {
    Fx x, y;
};
__host__ __device__ constexpr Fx fx_split(i64 v) {
    const int h = (int)((v + (1 << 26)) >> 27);
    return Fx{h, (int)((unsigned)v - ((unsigned)h << 27))};
}
__device__ __forceinline__ i64 fx_join(Fx a) { return ((i64)a.h << 27) + a.l; }
__device__ __forceinline__ i64 fx_wide(int a, int b, i64 c) { return c + (i64)a * b; }
// c + a b / 2^54
__device__ __forceinline__ i64 fx_fma(Fx a, Fx b, i64 c) {
    const i64 t = fx_wide(a.l, b.h, fx_wide(a.h, b.l, 1 << 26));
    return fx_wide(a.h, b.h, c) + (t >> 27);
}
// a b, a unit phasor b: in the units of a
__device__ __forceinline__ Cx fx_cmul(Cx a, Cx b) {
    const i64 tr = fx_wide(-a.y.l, b.y.h, fx_wide(-a.y.h, b.y.l,
                   fx_wide(a.x.l, b.x.h, fx_wide(a.x.h, b.x.l, 1 << 26))));
    const i64 ti = fx_wide(a.y.l, b.x.h, fx_wide(a.y.h, b.x.l,
                   fx_wide(a.x.l, b.y.h, fx_wide(a.x.h, b.y.l, 1 << 26))));
    const i64 re = fx_wide(-a.y.h, b.y.h, fx_wide(a.x.h, b.x.h, tr >> 27));
    const i64 im = fx_wide(a.y.h, b.x.h, fx_wide(a.x.h, b.y.h, ti >> 27));
    return Cx{fx_split((re + 2) >> 2), fx_split((im + 2) >> 2)};
}
// a b of a value a and a unit phasor b
__device__ __forceinline__ Cx fx_scale(Fx a, Cx b) {
    return Cx{fx_split((fx_fma(a, b.x, 2) >> 2)), fx_split((fx_fma(a, b.y, 2) >> 2))};
}
// a unit phasor in units of 2^-54
__device__ __forceinline__ Cx fx_step(Cx v) {
    return Cx{fx_split((fx_join(v.x) + 2) >> 2), fx_split((fx_join(v.y) + 2) >> 2)};
}
__device__ __forceinline__ int4 fx_pack(Cx v) { return make_int4(v.x.h, v.x.l, v.y.h, v.y.l); }
__device__ __forceinline__ Cx fx_unpack(int4 v) { return Cx{Fx{v.x, v.y}, Fx{v.z, v.w}}; }

// Phasors of multiples of 1 / kTurn of a turn, as products of kTurnCoarse and
// kTurnFine steps (in shared memory: the coarse ones, then the fine ones).  The
// steps are rounded once, to 2^-56: from sincospi their error would be the 2^-54
// of FP64, and every product of phasors adds its factors' errors up.
constexpr int kTurn = 2048, kTurnCoarse = 64, kTurnFine = kTurn / kTurnCoarse;
constexpr int kTurnSteps = kTurnCoarse + kTurnFine;

// cos and sin of pi num / den (at most pi / 2) by their series, in units of 2^-62.
struct HostPhasor {
    i64 c, s;
};
constexpr HostPhasor host_phasor(int num, int den) {
    constexpr unsigned long long kPi = 0xC90FDAA22168C234ULL;  // pi 2^62
    const __int128 x = ((__int128)kPi * num + den / 2) / den;
    __int128 term = (__int128)1 << 62, sum[2] = {term, 0};
    for (int n = 1; n < 32; ++n) {  // x^n / n!
        const __int128 p = term * x, d = ((__int128)n) << 62;
        term = (p + d / 2) / d;
        sum[n & 1] += n & 2 ? -term : term;
    }
    return HostPhasor{(i64)sum[0], (i64)sum[1]};
}
struct TurnSteps {
    int v[kTurnSteps][4];
    constexpr TurnSteps() : v() {
        for (int i = 0; i < kTurnSteps; ++i) {
            const int k = i < kTurnCoarse ? i : i - kTurnCoarse;
            const int quarter = i < kTurnCoarse ? kTurnCoarse / 4 : kTurn / 4;
            const HostPhasor z = host_phasor(k % quarter, 2 * quarter);
            i64 c = z.c, s = z.s;
            for (int q = k / quarter; q > 0; --q) {  // a quarter turn on
                const i64 t = c;
                c = -s;
                s = t;
            }
            const Fx x = fx_split((c + 32) >> 6), y = fx_split((s + 32) >> 6);
            v[i][0] = x.h;
            v[i][1] = x.l;
            v[i][2] = y.h;
            v[i][3] = y.l;
        }
    }
};
__device__ constexpr TurnSteps kTurnStepTable;

__device__ __forceinline__ void turn_steps(int4 *step, int tid) {
    if (tid < kTurnSteps) {
        const int *v = kTurnStepTable.v[tid];
        step[tid] = make_int4(v[0], v[1], v[2], v[3]);
    }
}
static_assert(kTurnSteps <= kDirThreads, "a step per thread");
__device__ __forceinline__ Cx turn_product(const int4 *step, int k) {
    return fx_cmul(fx_unpack(step[k / kTurnFine]), fx_unpack(step[kTurnCoarse + k % kTurnFine]));
}

// exp(2 pi i th) of a 64-bit fraction of a turn: the phasor at the nearest
// multiple of 1 / kTurn turned by the remaining angle d, |d| <= pi / kTurn, all of
// it in integers: d and sin d in units of 2^-61, cos d - 1 = -d^2 / 2 + d^4 / 24
// the same, the small terms d^5 / 120 (7e-17) and d^4 / 24 (2e-13) in FP32; those
// left out are below 2e-20.
template <typename Table>
__device__ __forceinline__ Cx fx_turn(u64 th, Table table) {
    const int k = (int)((th + (1ULL << 52)) >> 53);  // 0 .. kTurn
    const Cx e = table(k & (kTurn - 1));
    const Fx r = fx_split((i64)(th - ((u64)k << 53)));  // |r| <= 2^52, in 2^-64 turns
    constexpr i64 kTwoPi = 14148475504056880LL;        // 2 pi 2^51
    constexpr int kHi = (int)((kTwoPi + (1 << 26)) >> 27), kLo = (int)(kTwoPi - ((i64)kHi << 27));
    const i64 d = fx_fma(r, Fx{kHi, kLo}, 0);
    const int dh = (int)(d >> 21), dl = (int)(d & ((1 << 21) - 1));
    const float df = (float)dh * 9.094947017729282e-13f, q = df * df;  // 2^-40
    const float kUp = 2305843009213693952.f;                           // 2^61
    const i64 d2 = fx_wide(dh, dh, fx_wide(dh, dl, 0) >> 20);          // 2^-80
    // d^3 in 2^-59 (below 2^31), times 2^31 4 / 6
    const int d3 = (int)(fx_wide(dh, (int)(d2 >> 31), 1 << 29) >> 30);
    const i64 d36 = fx_wide(d3, 1431655765, 1 << 30) >> 31;
    const Fx sn = fx_split(d - d36 + __float2int_rn(kUp * df * q * q * (1.f / 120.f)));
    const Fx cm = fx_split(__float2int_rn(kUp * q * q * (1.f / 24.f)) - (d2 >> 20));
    // e + e (cm + i sn), the product in units of 2^-63
    const i64 re = fx_fma(cm, e.x, 64) - fx_fma(sn, e.y, 0), im = fx_fma(cm, e.y, fx_fma(sn, e.x, 64));
    return Cx{fx_split(fx_join(e.x) + (re >> 7)), fx_split(fx_join(e.y) + (im >> 7))};
}

// The warps' sums added up exactly, in two halves of 32 bits: a conversion to
// FP64 costs as much as an FP64 instruction (one per warp and sum: 0.468 against
// 0.450 ms of the GLS sums).
struct FxTotal {
    i64 hi = 0, lo = 0;
    __device__ __forceinline__ void add(i64 v) {
        hi += v >> 32;
        lo += (unsigned)v;
    }
    // in units of 2^unit
    __device__ __forceinline__ double value(int unit) const {
        return scalbn(fma((double)hi, 4294967296.0, (double)lo), unit);
    }
};

// Points of a run (one CTA, sums in 64-bit integers): 64 terms per warp, of at
// most 2^56.
constexpr int kDirRun = 64 * kDirWarps;
constexpr int kFxBits = 56;
// Exponent ex with |v| < 2^ex for the largest finite |v| of the CTA's threads;
// `sh` one shared word.
__device__ __forceinline__ int fx_exponent(double mx, u64 *sh, int tid) {
    if (tid == 0) *sh = 0;
    __syncthreads();
    u64 b = (u64)__double_as_longlong(mx);  // (not negative: ordered as integers)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const u64 v = __shfl_xor_sync(0xffffffffu, b, o);
        b = v > b ? v : b;
    }
    if ((tid & 31) == 0) atomicMax(sh, b);
    __syncthreads();
    b = *sh;
    return b >> 52 || !b ? (int)(b >> 52) - 1022 : -1010 - __clzll((i64)b);
}

// Phasor tables of a warp's tile of 32 points, one entry row of 32 points
// each: NB step phasors exp(i b x), kCoarse centres exp(i (K0 + 8 W g) x),
// kFine offsets exp(i W f x), W = 2 M + 1.
template <int M, int NB>
struct DirTable {
    static constexpr int kRows = NB + kCoarse + kFine;
    int4 row[kRows][32];

    // This lane's point: x in turns per bin, th0 the phase of K0, both as
    // fractions of a turn; `steps` from turn_steps.  Four phasors (the multiples
    // of x are exact), the rest by products of at most eight of one: an error of
    // a phasor counts as often as the phasor does, and from two phasors alone the
    // last bin would hold that of x 400 times.
    __device__ __forceinline__ void build(int lane, u64 x, u64 th0, const int4 *steps) {
        auto table = [&](int k) { return turn_product(steps, k); };
        Cx z[NB + 1];
        z[1] = fx_turn(x, table);
#pragma unroll
        for (int b = 2; b <= NB; ++b) z[b] = fx_cmul(z[b / 2], z[b - b / 2]);
#pragma unroll
        for (int b = 1; b <= NB; ++b) row[b - 1][lane] = fx_pack(fx_step(z[b]));
        constexpr int W = 2 * M + 1;
        Cx f[kFine];
        f[0] = Cx{Fx{1 << 29, 0}, Fx{0, 0}};
        f[1] = fx_turn(W * x, table);
#pragma unroll
        for (int k = 2; k < kFine; ++k) f[k] = fx_cmul(f[k / 2], f[k - k / 2]);
#pragma unroll
        for (int k = 0; k < kFine; ++k) row[NB + kCoarse + k][lane] = fx_pack(f[k]);
        const Cx w8 = fx_turn(W * kFine * x, table);
        Cx c = fx_turn(th0, table);
#pragma unroll
        for (int k = 0; k < kCoarse; ++k) {
            row[NB + k][lane] = fx_pack(c);
            c = fx_cmul(c, w8);
        }
    }
    // exp(i K x) of this lane's centre K = K0 + W lane at point p
    __device__ __forceinline__ Cx centre(int lane, int p) const {
        return fx_cmul(fx_unpack(row[NB + lane / kFine][p]),
                       fx_unpack(row[NB + kCoarse + lane % kFine][p]));
    }
    __device__ __forceinline__ Cx step(int b, int p) const { return fx_unpack(row[b][p]); }
};

// The sums of one value kind over a lane's 2 M + 1 bins, over one run.
template <int M>
struct DirSums {
    i64 c0 = 0, s0 = 0, p1[M], p2[M], p3[M], p4[M];
    __device__ __forceinline__ DirSums() {
#pragma unroll
        for (int b = 0; b < M; ++b) p1[b] = p2[b] = p3[b] = p4[b] = 0;
    }
    __device__ __forceinline__ void centre(Cx e) { c0 += fx_join(e.x); s0 += fx_join(e.y); }
    __device__ __forceinline__ void pair(int b, Cx e, Cx st) {
        p1[b] = fx_fma(e.x, st.x, p1[b]);
        p2[b] = fx_fma(e.y, st.y, p2[b]);
        p3[b] = fx_fma(e.y, st.x, p3[b]);
        p4[b] = fx_fma(e.x, st.y, p4[b]);
    }
    // real and imaginary parts of the lane's bins into re[0 .. 2 M], im[...]
    __device__ __forceinline__ void bins(i64 *re, i64 *im) const {
        re[M] = c0;
        im[M] = s0;
#pragma unroll
        for (int b = 0; b < M; ++b) {
            re[M + 1 + b] = p1[b] - p2[b];
            im[M + 1 + b] = p3[b] + p4[b];
            re[M - 1 - b] = p1[b] + p2[b];
            im[M - 1 - b] = p3[b] - p4[b];
        }
    }
};

// Adds the sums of a run over the CTA's warps: bin tid + 256 q of the CTA's 32 W
// bins to out[q], in units of 2^unit.  `red` holds 2 x kDirWarps x 32 W words.
template <int M>
__device__ __forceinline__ void dir_reduce(const DirSums<M> &v, i64 *red, int tid, int unit,
                                           double2 *out) {
    constexpr int TB = 32 * (2 * M + 1);
    const int lane = tid & 31, wid = tid >> 5;
    __syncthreads();  // the tables (or the previous kind) are no longer read
    v.bins(red + wid * TB + lane * (2 * M + 1), red + (kDirWarps + wid) * TB + lane * (2 * M + 1));
    __syncthreads();
#pragma unroll
    for (int q = 0; q < (TB + kDirThreads - 1) / kDirThreads; ++q) {
        const int b = tid + q * kDirThreads;
        FxTotal re, im;
        if (b < TB)
#pragma unroll
            for (int w = 0; w < kDirWarps; ++w) {
                re.add(red[w * TB + b]);
                im.add(red[(kDirWarps + w) * TB + b]);
            }
        out[q].x += re.value(unit);
        out[q].y += im.value(unit);
    }
}

// Points [j0, j1) of split z of a curve of n points cut into `splits` equal
// parts (the last ones may hold none); false when there is no such part.
__device__ __forceinline__ bool dir_part(long long n, int splits, int z, long long &j0,
                                         long long &j1) {
    if (z >= splits) return false;
    const long long per = (n + splits - 1) / splits;
    j0 = per * z;
    j1 = min(n, j0 + per);
    return true;
}

// ---------------------------------------------------------------------------
// adjoint NFFT (use_double): M = 6, 416 bins per CTA
// ---------------------------------------------------------------------------
constexpr int kNfM = 6, kNfBins = 32 * (2 * kNfM + 1);
using NfTable = DirTable<kNfM, kNfM>;
constexpr int kNfSmem = kDirWarps * (int)sizeof(NfTable);
static_assert(kNfSmem >= 2 * kDirWarps * kNfBins * 8, "the reduction reuses the tables");

}  // namespace

// One CTA per (416 bins, curve, part of its points); its eight warps take the
// points 32 at a time in turn, each with tables of its own, and are summed in
// shared memory at the end.  A curve cut into several parts leaves partial
// sums for k_nfft_direct64_sum.  Bound by the wide multiply-adds.  4 curves of 300 to 2,000 points and 20,000
// bins, host to host: 5.67 ms with a sincospi pair per point and 8 bins, 0.45 ms
// with factored phasors in FP64 (2.4 instructions per bin, 93 % busy), 0.235 ms
// in fixed point (0.242 ms with M = 8, 0.273 with M = 4), 0.219 ms with the
// warps' sums and the phasors of the tables in integers too; errors against 64
// bits 6.8e-13 in all of them, that of the phases.
__global__ void __launch_bounds__(kDirThreads, 2)
k_nfft_direct64(const Direct64Curve *__restrict__ cvs, const double *__restrict__ t,
                const double *__restrict__ y, double2 *__restrict__ out,
                double2 *__restrict__ part, long long part_stride) {
    extern __shared__ __align__(16) double sm[];
    __shared__ u64 top;
    __shared__ int4 steps[kTurnSteps];
    const Direct64Curve cv = cvs[blockIdx.y];
    const long long k0 = (long long)blockIdx.x * kNfBins;
    long long j0, j1;
    if (k0 >= cv.nf || !dir_part(cv.n, cv.splits, blockIdx.z, j0, j1)) return;  // whole CTA
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    NfTable &tab = reinterpret_cast<NfTable *>(sm)[wid];
    turn_steps(steps, tid);  // (the barriers below come before its first use)
    constexpr int NQ = (kNfBins + kDirThreads - 1) / kDirThreads;
    double2 v[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = make_double2(0.0, 0.0);
    bool odd = false;   // a value that is not finite, added below bin by bin
    bool lost = false;  // a time that is not finite: no bin has a value
    const double kc = (double)(k0 + kNfM);
    for (long long r0 = j0; r0 < j1; r0 += kDirRun) {
        const long long r1 = min(j1, r0 + kDirRun);
        double mx = 0.0;
        for (long long j = r0 + tid; j < r1; j += kDirThreads) {
            const double yj = fabs(y[cv.pt_off + j]);
            mx = isfinite(yj) && yj > mx ? yj : mx;
        }
        const int ex = fx_exponent(mx, &top, tid);
        DirSums<kNfM> acc;
        for (long long base = r0 + wid * 32; base < r1; base += kDirThreads) {
            const int cnt = (int)min(32LL, r1 - base);
            __syncwarp();  // the previous tile is consumed
            if (lane < cnt) {
                const double tj = t[cv.pt_off + base + lane];
                double yj = y[cv.pt_off + base + lane];
                if (!isfinite(yj)) {
                    odd = true;
                    yj = 0.0;
                }
                double a = cv.f0 * tj, b = cv.df * tj;
                a -= floor(a);
                b -= floor(b);
                const double th = fma(kc, b, a);
                lost = lost || !isfinite(th);
                tab.build(lane, turns64(b), turns64(th), steps);
                const Fx yv = fx_split(__double2ll_rn(scalbn(yj, kFxBits - ex)));
#pragma unroll
                for (int g = 0; g < kCoarse; ++g) {  // y rides on the coarse centres
                    int4 &c = tab.row[kNfM + g][lane];
                    c = fx_pack(fx_scale(yv, fx_unpack(c)));
                }
            }
            __syncwarp();
#pragma unroll 1
            for (int p = 0; p < cnt; ++p) {
                const Cx e = tab.centre(lane, p);
                acc.centre(e);
#pragma unroll
                for (int b = 0; b < kNfM; ++b) acc.pair(b, e, tab.step(b, p));
            }
        }
        dir_reduce<kNfM>(acc, reinterpret_cast<i64 *>(sm), tid, ex - kFxBits, v);
        __syncthreads();  // the next run's tables
    }
    if (__syncthreads_or(odd)) {  // inf cos and inf sin keep their own signs
        for (long long j = j0; j < j1; ++j) {
            const double tj = t[cv.pt_off + j], yj = y[cv.pt_off + j];
            if (isfinite(yj)) continue;
            double a = cv.f0 * tj, b = cv.df * tj;
            a -= floor(a);
            b -= floor(b);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const double2 e = zturn(fma((double)(k0 + tid + q * kDirThreads), b, a));
                v[q].x = fma(yj, e.x, v[q].x);
                v[q].y = fma(yj, e.y, v[q].y);
            }
        }
    }
    if (__syncthreads_or(lost)) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = make_double2(nan(""), nan(""));
    }
    double2 *dst = cv.splits > 1 ? part + blockIdx.z * part_stride + cv.part_off : out + cv.out_off;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int b = tid + q * kDirThreads;
        if (b < kNfBins && k0 + b < cv.nf) dst[k0 + b] = v[q];
    }
}

// Parts of the split curves added in order.
__global__ void __launch_bounds__(256)
k_nfft_direct64_sum(const Direct64Curve *__restrict__ cvs, const double2 *__restrict__ part,
                    long long part_stride, double2 *__restrict__ out) {
    const Direct64Curve cv = cvs[blockIdx.y];
    const long long k = (long long)blockIdx.x * 256 + threadIdx.x;
    if (cv.splits <= 1 || k >= cv.nf) return;
    double re = 0.0, im = 0.0;
    for (int z = 0; z < cv.splits; ++z) {
        const double2 v = part[z * part_stride + cv.part_off + k];
        re += v.x;
        im += v.y;
    }
    out[cv.out_off + k] = make_double2(re, im);
}

int direct_splits(long long bins, int bins_per_cta, long long max_n) {
    // about eight CTAs per SM (152 SMs, one or two resident), so that curves
    // of different lengths even out, and at least 256 points (one tile per
    // warp) each; enough bins need no parts and no second kernel
    const long long tiles = std::max(1LL, (bins + bins_per_cta - 1) / bins_per_cta);
    const long long want = (8 * 152 + tiles - 1) / tiles;
    return (int)std::max(1LL, std::min(std::min(want, (max_n + 255) / 256), 64LL));
}
int nfft_direct64_bins() { return kNfBins; }

cudaError_t launch_nfft_direct64(const Direct64Curve *cv, int n_curves, long long max_nf,
                                 int max_splits, const double *t, const double *y, double2 *out,
                                 double2 *part, long long part_stride, cudaStream_t s) {
    if (n_curves <= 0 || max_nf <= 0) return cudaSuccess;
    const long long nb = (max_nf + kNfBins - 1) / kNfBins, nr = (max_nf + 255) / 256;
    if (nr > 0x7fffffffLL || n_curves > 65535) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(
        k_nfft_direct64, cudaFuncAttributeMaxDynamicSharedMemorySize, kNfSmem);
    if (e != cudaSuccess) return e;
    k_nfft_direct64<<<dim3((unsigned)nb, n_curves, max_splits), kDirThreads, kNfSmem, s>>>(
        cv, t, y, out, part, part_stride);
    e = cudaGetLastError();
    if (e == cudaSuccess && max_splits > 1) {
        k_nfft_direct64_sum<<<dim3((unsigned)nr, n_curves), 256, 0, s>>>(cv, part, part_stride, out);
        e = cudaGetLastError();
    }
    return e;
}

// ---------------------------------------------------------------------------
// GLS (use_fft=False): three sums, M = 3, 224 bins per CTA
// ---------------------------------------------------------------------------
namespace {
constexpr int kGlM = 3, kGlBins = 32 * (2 * kGlM + 1);
// step phasors up to 2 M: those of the 2x sums are the even ones
using GlTable = DirTable<kGlM, 2 * kGlM>;
struct GlTile {
    GlTable tab;
    int2 yw[32], w[32];
};
constexpr int kGlSmem = kDirWarps * (int)sizeof(GlTile);
static_assert(kGlSmem >= 2 * kDirWarps * kGlBins * 8, "the reduction reuses the tables");

__device__ __forceinline__ float gls_direct_power(const DevCurve &cv, const GlsParams &gp,
                                                  double2 a, double2 b, double2 c) {
    return (float)gls_from_sums<double>(a.x, a.y, b.x, b.y, c.x, c.y, gp.mode, (double)gp.reg,
                                        (double)cv.w_sum, (double)cv.yw_sum, (double)cv.ybar,
                                        (double)cv.yy_inv);
}
}  // namespace

// As k_nfft_direct64 with the sums of yw and w at f and of w at 2 f (its
// phasors are the squares of the others), then the power.  The times are
// taken from the curve's first point (the power does not depend on the time
// origin), so the phases stay small.  A curve cut into parts leaves its six
// partial sums for k_gls_direct_sum.  8 curves of 300 to 2,000 points and
// 10,000 frequencies: 9.62 ms with a sincospi each, 1.10 ms with factored
// phasors in FP64 (7.7 instructions per frequency, 81 % busy), 0.47 ms in fixed
// point (0.61 ms with M = 4 and one CTA per SM), 0.435 ms with the warps' sums
// and the phasors of the tables in integers too; errors against 64 bits 2.8e-8
// in all of them.
__global__ void __launch_bounds__(kDirThreads, 2)
k_gls_direct(const DevCurve *__restrict__ cvs, const double *__restrict__ t,
             const float *__restrict__ yw, const float *__restrict__ w, float *__restrict__ out,
             double2 *__restrict__ part, long long part_stride, GlsParams gp) {
    extern __shared__ __align__(16) double sm[];
    __shared__ u64 top[2];
    __shared__ int4 steps[kTurnSteps];
    const DevCurve cv = cvs[blockIdx.y];
    const long long k0 = (long long)blockIdx.x * kGlBins;
    long long j0, j1;
    if (k0 >= cv.nf || !dir_part(cv.n, cv.aux, blockIdx.z, j0, j1)) return;  // whole CTA
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    GlTile &tile = reinterpret_cast<GlTile *>(sm)[wid];
    turn_steps(steps, tid);  // (the barriers below come before its first use)
    constexpr int NQ = (kGlBins + kDirThreads - 1) / kDirThreads;
    double2 va[NQ], vb[NQ], vc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) va[q] = vb[q] = vc[q] = make_double2(0.0, 0.0);
    // something not finite: no power of the curve is valid (the window's powers
    // are of the weights alone)
    bool lost = false;
    const bool window = gp.mode == 2;
    const double kc = cv.kc - (double)(cv.nf / 2) + (double)(k0 + kGlM);
    const double t0 = t[cv.pt_off];
    for (long long r0 = j0; r0 < j1; r0 += kDirRun) {
        const long long r1 = min(j1, r0 + kDirRun);
        float my = 0.f, mw = 0.f;
        for (long long j = cv.pt_off + r0 + tid; j < cv.pt_off + r1; j += kDirThreads) {
            const float a = fabsf(yw[j]), b = fabsf(w[j]);
            if (isfinite(a)) my = fmaxf(my, a);
            else lost = lost || !window;
            if (isfinite(b)) mw = fmaxf(mw, b);
            else lost = true;
        }
        const int ey = fx_exponent(my, &top[0], tid), ew = fx_exponent(mw, &top[1], tid);
        DirSums<kGlM> sa, sb, sc;
        for (long long base = r0 + wid * 32; base < r1; base += kDirThreads) {
            const int cnt = (int)min(32LL, r1 - base);
            __syncwarp();  // the previous tile is consumed
            if (lane < cnt) {
                const long long j = cv.pt_off + base + lane;
                const double x = (t[j] - t0) * cv.df;
                lost = lost || !isfinite(kc * x);
                tile.tab.build(lane, turns64(x), turns64(kc * x), steps);
                const double yj = isfinite(yw[j]) ? (double)yw[j] : 0.0;
                const Fx fy = fx_split(__double2ll_rn(scalbn(yj, kFxBits - ey)));
                const Fx fw = fx_split(__double2ll_rn(scalbn((double)w[j], kFxBits - ew)));
                tile.yw[lane] = make_int2(fy.h, fy.l);
                tile.w[lane] = make_int2(fw.h, fw.l);
            }
            __syncwarp();
#pragma unroll 1
            for (int p = 0; p < cnt; ++p) {
                const Cx e = tile.tab.centre(lane, p);
                const int2 vy = tile.yw[p], vw = tile.w[p];
                const Cx ea = fx_scale(Fx{vy.x, vy.y}, e), eb = fx_scale(Fx{vw.x, vw.y}, e);
                const Cx ec = fx_cmul(eb, e);
                sa.centre(ea);
                sb.centre(eb);
                sc.centre(ec);
#pragma unroll
                for (int b = 0; b < kGlM; ++b) {
                    const Cx st = tile.tab.step(b, p);
                    sa.pair(b, ea, st);
                    sb.pair(b, eb, st);
                    sc.pair(b, ec, tile.tab.step(2 * b + 1, p));
                }
            }
        }
        i64 *red = reinterpret_cast<i64 *>(sm);
        dir_reduce<kGlM>(sa, red, tid, ey - kFxBits, va);
        dir_reduce<kGlM>(sb, red, tid, ew - kFxBits, vb);
        dir_reduce<kGlM>(sc, red, tid, ew - kFxBits, vc);
        __syncthreads();  // the next run's tables
    }
    if (__syncthreads_or(lost)) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) va[q] = vb[q] = vc[q] = make_double2(nan(""), nan(""));
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int b = tid + q * kDirThreads;
        if (b >= kGlBins || k0 + b >= cv.nf) continue;
        if (cv.aux > 1) {
            double2 *d = part + 3 * (blockIdx.z * part_stride + cv.inter_off + k0 + b);
            d[0] = va[q];
            d[1] = vb[q];
            d[2] = vc[q];
        } else {
            out[cv.out_off + k0 + b] = gls_direct_power(cv, gp, va[q], vb[q], vc[q]);
        }
    }
}

// Parts of the split curves added in order, then the power.
__global__ void __launch_bounds__(256)
k_gls_direct_sum(const DevCurve *__restrict__ cvs, const double2 *__restrict__ part,
                 long long part_stride, float *__restrict__ out, GlsParams gp) {
    const DevCurve cv = cvs[blockIdx.y];
    const long long k = (long long)blockIdx.x * 256 + threadIdx.x;
    if (cv.aux <= 1 || k >= cv.nf) return;
    double2 v[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
    for (int z = 0; z < cv.aux; ++z) {
        const double2 *d = part + 3 * (z * part_stride + cv.inter_off + k);
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            v[g].x += d[g].x;
            v[g].y += d[g].y;
        }
    }
    out[cv.out_off + k] = gls_direct_power(cv, gp, v[0], v[1], v[2]);
}

int gls_direct_bins() { return kGlBins; }

cudaError_t launch_gls_direct(const DevCurve *cv, int n_curves, int max_nf, int max_splits,
                              const double *t, const float *yw, const float *w, float *out,
                              double2 *part, long long part_stride, GlsParams g, cudaStream_t s) {
    if (n_curves <= 0 || max_nf <= 0) return cudaSuccess;
    cudaError_t e =
        cudaFuncSetAttribute(k_gls_direct, cudaFuncAttributeMaxDynamicSharedMemorySize, kGlSmem);
    if (e != cudaSuccess) return e;
    k_gls_direct<<<dim3((max_nf + kGlBins - 1) / kGlBins, n_curves, max_splits), kDirThreads,
                   kGlSmem, s>>>(cv, t, yw, w, out, part, part_stride, g);
    e = cudaGetLastError();
    if (e == cudaSuccess && max_splits > 1) {
        k_gls_direct_sum<<<dim3((max_nf + 255) / 256, n_curves), 256, 0, s>>>(cv, part, part_stride,
                                                                              out, g);
        e = cudaGetLastError();
    }
    return e;
}

// ---------------------------------------------------------------------------
// multi-harmonic floating-mean GLS of one curve at any frequencies
// ---------------------------------------------------------------------------
namespace {

// Points of a run and the bits of its values.  The phasors keep their 2^-56
// here (the recurrence needs them), so the products are quarter units and a
// value has fewer bits; it is rounded once, not at each of E's two products.
constexpr int kMhRun = 64 * kDirWarps, kMhBits = 54;

// rows of sums a CTA reduces: c, s (2H each), yc, ys (H each), and sum w
__host__ __device__ constexpr int mh_sums(int H) { return 6 * H + 1; }
__host__ __device__ constexpr int mh_smem(int H) {
    // turn table, the warps' point tiles, the warps' sums and their totals
    return kTurn * 16 + kDirWarps * 32 * 24 + (kDirWarps + 1) * mh_sums(H) * 32 * 8;
}

}  // namespace

// 32 frequencies per CTA, one per lane; the eight warps take the points 32 at
// a time in turn and are summed in shared memory, so that a few thousand
// frequencies already fill the chip (with a thread per frequency, 20,000 of
// them made 157 CTAs of 128 threads for 152 SMs).  Up to four CTAs of a
// cluster share the points of the same frequencies, and the first adds their
// sums and solves: 625 CTAs left a fifth of the FP64 pipes idle at the end
// (4.1 CTAs per SM are 5 rounds).  Per point the
// phasor from fx_turn, its powers n = 2 .. 2H by the recurrence
// z_n = 2 cos(phi) z_(n-1) - z_(n-2), then the sums of
// cuvarbase/lombscargle.py:337-400 (mhdirect_sums), all in fixed point; FP64
// forms t f, adds the warps' sums, and from there on: the regulariser of
// :403-447, the 2H x 2H system solved by Gaussian elimination with partial
// pivoting, and the power of :497-536.  H = 3, 1,000 points, 20,000
// frequencies, host to host: 4.93 ms with a sincospi per point; in FP64 2.24 ms
// with the table and the clusters (54 instructions per point and frequency, the
// pipes 88 % busy), 1.97 ms with the recurrence, 1.54 ms with the phasor's
// fraction in integers; 0.79 ms in fixed point (about 100 wide multiply-adds).
// Errors against 64 bits 1.8e-13 in all of them: that of the FP64 phase t f.
template <int H>
__global__ void __launch_bounds__(kDirThreads, H <= 4 ? 2 : 1)
k_mhgls_direct(const double *__restrict__ t, const double *__restrict__ yw,
               const double *__restrict__ w, long long n, const double *__restrict__ freqs,
               long long nf, MhParams mp, double *__restrict__ out, int csize) {
    constexpr int NH = 2 * H, NS = mh_sums(H);
    const int rank = blockIdx.x % csize;
    extern __shared__ __align__(16) double sm[];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    __shared__ u64 top[2];
    int4 *turn = reinterpret_cast<int4 *>(sm);
    double *tiles = sm + 2 * kTurn;
    i64 *sums = reinterpret_cast<i64 *>(tiles + kDirWarps * 96);
    double *tot = tiles + kDirWarps * 96 + kDirWarps * NS * 32;
    double *st = tiles + wid * 96;
    int2 *sy = reinterpret_cast<int2 *>(st + 32), *sw = sy + 32;
    {  // the steps (in the point tiles' memory), then all their products
        int4 *step = reinterpret_cast<int4 *>(tiles);
        turn_steps(step, tid);
        __syncthreads();
        for (int i = tid; i < kTurn; i += kDirThreads) turn[i] = fx_pack(turn_product(step, i));
        __syncthreads();
    }
    const long long k = (long long)(blockIdx.x / csize) * 32 + lane;
    const double f = (k < nf) ? freqs[k] : 0.0;
    double ws = 0.0;    // of the points this lane staged
    // a phase that is not finite (of this lane's frequency), a value that is not
    bool lost = false, odd = false;
    // the warps' sums, in shared memory as [warp][sum][lane]
    i64 *r = sums + wid * NS * 32 + lane;
    for (int i = tid; i < NS * 32; i += kDirThreads) tot[i] = 0.0;
    const long long share = (n + csize - 1) / csize;
    const long long j1 = min(n, (rank + 1) * share);
    for (long long r0 = rank * share; r0 < j1; r0 += kMhRun) {
        const long long r1 = min(j1, r0 + kMhRun);
        double my = 0.0, mw = 0.0;
        for (long long j = r0 + tid; j < r1; j += kDirThreads) {
            const double u = fabs(yw[j]), v = fabs(w[j]);
            if (isfinite(u) && isfinite(v)) {
                my = u > my ? u : my;
                mw = v > mw ? v : mw;
            } else {
                odd = true;
            }
        }
        const int ey = fx_exponent(my, &top[0], tid), ew = fx_exponent(mw, &top[1], tid);
        i64 c[NH + 1], s[NH + 1], yc[H + 1], ys[H + 1];
#pragma unroll
        for (int m = 0; m <= NH; ++m) c[m] = s[m] = 0;
#pragma unroll
        for (int m = 0; m <= H; ++m) yc[m] = ys[m] = 0;
        for (long long base = r0 + wid * 32; base < r1; base += kDirThreads) {
            const int cnt = (int)min(32LL, r1 - base);
            __syncwarp();  // the previous tile is consumed
            if (lane < cnt) {
                st[lane] = t[base + lane];
                ws += w[base + lane];
                const Fx fy = fx_split(__double2ll_rn(scalbn(yw[base + lane], kMhBits - ey)));
                const Fx fw = fx_split(__double2ll_rn(scalbn(w[base + lane], kMhBits - ew)));
                sy[lane] = make_int2(fy.h, fy.l);
                sw[lane] = make_int2(fw.h, fw.l);
            }
            __syncwarp();
#pragma unroll 1
            for (int q = 0; q < cnt; ++q) {
                const int2 vw = sw[q], vy = sy[q];
                const Fx wq{vw.x, vw.y}, yq{vy.x, vy.y};
                const double p = st[q] * f;
                lost = lost || (__double2hiint(p) & 0x7ff00000) == 0x7ff00000;
                Cx z = fx_turn(turns64(p), [&](int i) { return fx_unpack(turn[i]); }), zp{Fx{1 << 29, 0}, Fx{0, 0}};  // power m, m - 1
                const Fx cc = fx_split(2 * fx_join(z.x));                 // 2 cos
#pragma unroll
                for (int m = 1; m <= NH; ++m) {
                    if (m > 1) {
                        const Cx zn{fx_split((fx_fma(cc, z.x, 2 - 4 * fx_join(zp.x))) >> 2),
                                    fx_split((fx_fma(cc, z.y, 2 - 4 * fx_join(zp.y))) >> 2)};
                        zp = z;
                        z = zn;
                    }
                    c[m] = fx_fma(wq, z.x, c[m]);
                    s[m] = fx_fma(wq, z.y, s[m]);
                    if (m <= H) {
                        yc[m] = fx_fma(yq, z.x, yc[m]);
                        ys[m] = fx_fma(yq, z.y, ys[m]);
                    }
                }
            }
        }
#pragma unroll
        for (int m = 1; m <= NH; ++m) {
            r[(m - 1) * 32] = c[m];
            r[(NH + m - 1) * 32] = s[m];
        }
#pragma unroll
        for (int m = 1; m <= H; ++m) {
            r[(2 * NH + m - 1) * 32] = yc[m];
            r[(2 * NH + H + m - 1) * 32] = ys[m];
        }
        __syncthreads();
        for (int i = tid; i < (NS - 1) * 32; i += kDirThreads) {
            FxTotal v;
            for (int q = 0; q < kDirWarps; ++q) v.add(sums[q * NS * 32 + i]);
            tot[i] += v.value((i < 2 * NH * 32 ? ew : ey) - kMhBits - 2);
        }
        __syncthreads();  // before the next run's sums
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ws += __shfl_xor_sync(0xffffffffu, ws, o);
    // (a value that is not finite spoils every frequency, a phase its own)
    if (__syncthreads_or(odd) || lost) ws = nan("");
    r[6 * H * 32] = __double_as_longlong(ws);
    __syncthreads();
    if (tid < 32) {
        double v = 0.0;
        for (int q = 0; q < kDirWarps; ++q) v += __longlong_as_double(sums[(q * NS + 6 * H) * 32 + tid]);
        tot[6 * H * 32 + tid] = v;
    }
    if (csize > 1) {
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        if (rank == 0)
            for (int i = tid; i < NS * 32; i += kDirThreads) {
                double v = tot[i];
                for (int q = 1; q < csize; ++q) v += cl.map_shared_rank(tot, q)[i];
                tot[i] = v;
            }
        cl.sync();  // the others' sums are read before they leave
        if (rank != 0) return;
    }
    __syncthreads();
    if (wid != 0 || k >= nf) return;
    double c[NH + 1], s[NH + 1], yc[H + 1], ys[H + 1];
    s[0] = 0.0;
#pragma unroll
    for (int m = 1; m <= NH; ++m) {
        c[m] = tot[(m - 1) * 32 + lane];
        s[m] = tot[(NH + m - 1) * 32 + lane];
    }
#pragma unroll
    for (int m = 1; m <= H; ++m) {
        yc[m] = tot[(2 * NH + m - 1) * 32 + lane];
        ys[m] = tot[(2 * NH + H + m - 1) * 32 + lane];
    }
    c[0] = tot[6 * H * 32 + lane];
    // regularised blocks: M = [[CC, CS], [CS^T, SS]], rhs = [YC; YS]
    double M[NH][NH], rhs[NH];
#pragma unroll
    for (int a = 1; a <= H; ++a) {
#pragma unroll
        for (int b = 1; b <= H; ++b) {
            const int dd = a > b ? a - b : b - a;
            const double sg = (a >= b) ? 1.0 : -1.0;  // sign(a - b), 1 at a == b
            const double reg = (a == b) ? mp.d[a - 1] : 0.0;
            const double cc = 0.5 * (c[a + b] + c[dd]) - c[a] * c[b] + reg;
            const double cs = 0.5 * (s[a + b] - sg * s[dd]) - c[a] * s[b];
            const double ss = 0.5 * (c[dd] - c[a + b]) - s[a] * s[b] + reg;
            M[a - 1][b - 1] = cc;
            M[a - 1][H + b - 1] = cs;
            M[H + b - 1][a - 1] = cs;
            M[H + a - 1][H + b - 1] = ss;
        }
        rhs[a - 1] = yc[a] - mp.ybar * c[a] + mp.d[a - 1] * mp.cn0[a - 1];
        rhs[H + a - 1] = ys[a] - mp.ybar * s[a] + mp.d[a - 1] * mp.sn0[a - 1];
    }
    // Gaussian elimination with partial pivoting on a copy
    double W[NH][NH + 1];
#pragma unroll
    for (int r = 0; r < NH; ++r) {
#pragma unroll
        for (int q = 0; q < NH; ++q) W[r][q] = M[r][q];
        W[r][NH] = rhs[r];
    }
    bool singular = false;
    for (int col = 0; col < NH; ++col) {
        int piv = col;
        double best = fabs(W[col][col]);
        for (int r = col + 1; r < NH; ++r)
            if (fabs(W[r][col]) > best) { best = fabs(W[r][col]); piv = r; }
        if (!(best > 0.0)) { singular = true; break; }
        if (piv != col)
            for (int q = col; q <= NH; ++q) {
                const double tmp = W[col][q];
                W[col][q] = W[piv][q];
                W[piv][q] = tmp;
            }
        for (int r = col + 1; r < NH; ++r) {
            const double fct = W[r][col] / W[col][col];
            for (int q = col; q <= NH; ++q) W[r][q] = fma(-fct, W[col][q], W[r][q]);
        }
    }
    double th[NH];
    if (!singular) {
        for (int r = NH - 1; r >= 0; --r) {
            double v = W[r][NH];
            for (int q = r + 1; q < NH; ++q) v = fma(-W[r][q], th[q], v);
            th[r] = v / W[r][r];
        }
    }
    if (singular) {
        out[k] = nan("");
        return;
    }
    // P = (YX - sum XX) / YY with the regularised blocks
    double xx = 0.0, yx = 0.0;
#pragma unroll
    for (int a = 0; a < H; ++a) {
        yx += th[a] * rhs[a] + th[H + a] * rhs[H + a];
#pragma unroll
        for (int b = 0; b < H; ++b)
            xx += th[a] * th[b] * M[a][b] + 2.0 * th[a] * th[H + b] * M[a][H + b] +
                  th[H + a] * th[H + b] * M[H + a][H + b];
    }
    out[k] = (2.0 * yx - xx) / mp.yy;
}

cudaError_t launch_mhgls_direct(int nharms, const double *t, const double *yw, const double *w,
                                long long n, const double *freqs, long long nf,
                                const MhParams &mp, double *out, cudaStream_t s) {
    if (n <= 0 || nf <= 0) return cudaSuccess;
    const long long nb = (nf + 31) / 32;
    if (nb > 0x7fffffffLL) return cudaErrorInvalidValue;
    // enough CTAs already (16 per SM), or too few points for one tile per warp
    int csize = 1;
    while (csize < 4 && nb * csize < 16 * 152 && n >= 2LL * csize * kDirThreads) csize *= 2;
    if (nb * csize > 0x7fffffffLL) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nb * csize));
    cfg.blockDim = dim3(kDirThreads);
    cfg.dynamicSmemBytes = mh_smem(nharms);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = csize;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = csize > 1 ? 1 : 0;
    cudaError_t e = cudaErrorInvalidValue;
    switch (nharms) {
#define CUVGLS_MH(HH)                                                                             \
    case HH:                                                                                      \
        e = cudaFuncSetAttribute(k_mhgls_direct<HH>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                 mh_smem(HH));                                                    \
        if (e != cudaSuccess) return e;                                                           \
        e = cudaLaunchKernelEx(&cfg, k_mhgls_direct<HH>, t, yw, w, n, freqs, nf, mp, out, csize); \
        break;
        CUVGLS_MH(1) CUVGLS_MH(2) CUVGLS_MH(3) CUVGLS_MH(4)
        CUVGLS_MH(5) CUVGLS_MH(6) CUVGLS_MH(7) CUVGLS_MH(8)
#undef CUVGLS_MH
        default: break;
    }
    return e;
}

}  // namespace cuvgls
