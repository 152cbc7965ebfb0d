// Pass kernels of the two-pass NFFT, templated on the transform lengths, and
// the device helpers they share with kernels.cu.
//
//   k_pass1<NG, L1>  one CTA per (curve, block of B columns).  Spreads the
//                    records of the neighbouring bins into NG padded
//                    L1 x B shared-memory tiles (shared-memory float atomics),
//                    runs the length-L1 column FFTs, applies the inter-pass
//                    twiddle exp(2 pi i q1 l2 / G) and writes the tile to the
//                    intermediate buffer ([column block][q1][column]).
//   k_pass1_long<L1> the same for one grid of the long columns.
//   k_pass2_gls_deep<L2>  one CTA per (curve, block of R rows), rows of 512 to
//                    2,048.  Runs the length-L2 row FFTs of the three grids
//                    and, in the same kernel, deconvolves the window and
//                    evaluates the GLS power of every in-band frequency.
//   k_pass2_gls_cube the same for rows of 4,096.
//   k_pass2_nfft<L2> the same for one grid, writing complex adjoint-NFFT
//                    values with the absolute-time phase.
// (Rows up to 400: pass2_tma.cuh.)
#pragma once

#include <climits>
#include <type_traits>
#include <cuda_runtime.h>

#include "fft.cuh"
#include "gls_math.cuh"
#include "kernels.cuh"
#include "pass2_tma.cuh"

namespace cuvgls {

__device__ __forceinline__ void bin_ranges(const int *__restrict__ bins, int cb,
                                           int lo, int hi, int nb, int &a0,
                                           int &a1, int &b0, int &b1) {
    if (hi - lo + 1 >= nb) {
        a0 = bins[0]; a1 = bins[nb]; b0 = 0; b1 = 0;
        return;
    }
    const int s = cb + lo, e = cb + hi;
    if (s < 0) {
        a0 = bins[s + nb]; a1 = bins[nb]; b0 = bins[0]; b1 = bins[e + 1];
    } else if (e >= nb) {
        a0 = bins[s]; a1 = bins[nb]; b0 = bins[0]; b1 = bins[e - nb + 1];
    } else {
        a0 = bins[s]; a1 = bins[e + 1]; b0 = 0; b1 = 0;
    }
}

// Band index of FFT output q, or -1 when q is outside the centred band
// k' in [-h, nf - h).
__device__ __forceinline__ int band_index(long long q, int nf, int h, long long G) {
    if (q < nf - h) return (int)q;
    if (q >= G - h) return (int)(q - G);
    return INT_MIN;
}

// Position of the n-th (from 0) set bit of m; needs n < popc(m).
__device__ __forceinline__ int nth_set_bit(unsigned m, int n) {
    int pos = 0;
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
        const int c = __popc(m & ((1u << w) - 1u));
        if (n >= c) { n -= c; m >>= w; pos += w; }
    }
    return pos;
}

// Stage A of the two-level column FFTs of a pass-1 tile (NG grids of B
// columns) that skips the units whose inputs are all zero.  Unit (g, i, c)
// transforms the elements i + LB k of column c of grid g; bit i of mAB
// (grids A and B) or mC (grid C) says that some row i + LB k holds a tap.
// A skipped unit's elements stay zero, which is their transform.  The
// remaining units are packed onto the lowest threads, so whole warps idle
// and leave their issue slots to the other CTAs of the SM.  With full masks
// this is the unit order of tile_fft2_a.
template <int L, int NG, int B, int GS, int NT>
__device__ __forceinline__ void tile_fft2_a_occ(float2 *__restrict__ buf,
                                                const float2 *__restrict__ twa, int tid,
                                                unsigned mAB, unsigned mC) {
    constexpr int LA = two_level_la(L);
    constexpr int LB = L / LA;
    static_assert(LA > 0 && LB <= 32, "two-level length with at most 32 residues");
    const int nAB = __popc(mAB), nC = NG == 3 ? __popc(mC) : 0;
    const int units = (NG == 3 ? 2 * nAB + nC : nAB) * B;
#pragma unroll 1
    for (int u = tid; u < units; u += NT) {
        const int c = u % B;
        int p = u / B, g = 0;
        unsigned mk = mAB;
        if (p >= nAB) {
            p -= nAB;
            g = 1;
            if (p >= nAB) { p -= nAB; g = 2; mk = mC; }
        }
        const int i = nth_set_bit(mk, p);
        const int base = c + g * GS;
        float2 x[LA];
#pragma unroll
        for (int k = 0; k < LA; ++k) x[k] = buf[base + phys2_ik<L>(i, k) * B];
        fft2_stage_a_regs<L>(x, twa, i);
#pragma unroll
        for (int qa = 0; qa < LA; ++qa) buf[base + phys2_ik<L>(i, qa) * B] = x[qa];
    }
}

// A record staged by pass 1: row << 16 | column of its cell, offset in the
// cell, and its values (grids A and B, or grid C twice).
struct StagedRec {
    int rc;
    float frac;
    float2 v0, v1;
};
static_assert(sizeof(StagedRec) == kStageRecBytes, "staged record size");

// One pass-1 CTA: column block blockIdx.x of curve blockIdx.y (the body of
// both pass-1 kernels below).
template <int NG, int L1, bool MANY>
__device__ __forceinline__ void pass1_body(const DevCurve *cvs, const RecAB *recAB,
                                           const RecC *recC, const int *binsAB, const int *binsC,
                                           float2 *inter, const Plan &p) {
    constexpr int B = pass1_cols(NG, L1);
    constexpr int NT = pass1_threads(NG, L1);
    constexpr int GS = tile_len(L1) * B;
    constexpr int TILE = NG * GS;
    constexpr int NTW = fft_table_len(L1);
    constexpr int NSR = pass1_stage_recs(NG, L1);
    // staged records follow the tile (and the Stockham table)
    constexpr int STAGE = TILE + (two_level_la(L1) ? 0 : NTW);
    extern __shared__ __align__(16) float2 sm[];
    float2 *tile = sm;
    const int tid = threadIdx.x;
    const int cb = blockIdx.x;
    const int c0 = cb * B;
    if (p.dependent) {
        pdl_trigger();
        pdl_wait();  // descriptors and records; the intermediate read by earlier passes
    }
    recAB = written(recAB);
    recC = written(recC);
    binsAB = written(binsAB);
    binsC = written(binsC);
    const DevCurve cv = written(cvs)[blockIdx.y];  // in flight during the zero-fill
    const int G2 = p.G2, m = p.m;
    // FFT table: read through the read-only cache (two-level lengths) or
    // staged in shared memory (Stockham lengths)
    const float2 *tws = p.st1;
    if constexpr (two_level_la(L1) == 0) {
        float2 *t = tile + TILE;
        for (int i = tid; i < NTW; i += NT) t[i] = p.st1[i];
        tws = t;
    }
    {
        float4 *t4 = reinterpret_cast<float4 *>(tile);  // 16-byte aligned
        for (int i = tid; i < TILE / 2; i += NT) t4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if ((TILE & 1) && tid == 0) tile[TILE - 1] = make_float2(0.f, 0.f);
    }

    // Spreading.  The records of the neighbouring bins (grids A and B share
    // the x-position records, grid C has its own at 2x positions; each
    // carries its cell as row and column) are staged in shared memory NSR at
    // a time, one batch of coalesced loads per round.  Then one work item per
    // (staged record, column of this block), or the gather below.
    const int lo = -((m + B - 1) / B), hi = (B + m - 2) / B;
    int a0, a1, b0, b1, e0 = 0, e1 = 0, f0 = 0, f1 = 0;
    bin_ranges(binsAB + cv.bin_off, cb, lo, hi, p.nb, a0, a1, b0, b1);
    const int nab = (a1 - a0) + (b1 - b0);
    int nc = 0;
    if (NG == 3) {
        bin_ranges(binsC + cv.bin_off, cb, lo, hi, p.nb, e0, e1, f0, f1);
        nc = (e1 - e0) + (f1 - f0);
    }
    const RecAB *rab = recAB + cv.rec_off;
    const RecC *rcc = recC + cv.rec_off;
    StagedRec *st = reinterpret_cast<StagedRec *>(sm + STAGE);
    const int ntot = nab + nc;
    // Dense column blocks of the long Stockham tiles of one grid (at least one
    // record per row of the tile) are spread by gather: the staged records are sorted
    // by the row they land in (integer shared-memory atomics and a scan),
    // then each thread sums the taps of whole rows in registers and adds
    // them to the tile with plain stores; no float atomics, which serialise
    // when several records hit the same cells.
    constexpr bool GATHER = pass1_gather(NG, L1);
    static_assert(!GATHER || NG == 1, "the three-grid columns of that length: k_pass1_long");
    int *rowcnt = reinterpret_cast<int *>(st + NSR);  // L1 + 1 (gather tiles)
    int *bucket = rowcnt + L1 + 1;                      // NSR
    int *wsum = bucket + NSR;                           // 32
    const bool dense = GATHER ? ntot >= L1 : MANY && ntot >= 2 * NT;
    // Two-level column FFTs: occ[kind * 32 + i] is set when a tap of that
    // record kind (0: A and B, 1: C) lands in a row congruent to i modulo
    // LB, so stage A can skip the all-zero units; the dense path does not
    // track it and transforms every unit.
    constexpr int LA1 = two_level_la(L1);
    constexpr int LB1 = LA1 ? L1 / LA1 : 1;
    unsigned char *occ = reinterpret_cast<unsigned char *>(st + NSR) +
                         (GATHER ? pass1_gather_bytes(L1, NSR) : 0);  // kOccBytes
    if (LA1 && tid < kOccBytes) occ[tid] = 0;  // before the first round's barrier
    if (GATHER && dense) {  // uniform over the CTA
        for (int i = tid; i <= L1; i += NT) rowcnt[i] = 0;
        __syncthreads();  // counts zeroed before the first round's atomics
    }
    // staged form of record ri of this block's window (AB records first)
    auto load_rec = [&](int ri) {
        StagedRec r;
        if (ri < nab) {
            const int k = ri < (a1 - a0) ? a0 + ri : b0 + (ri - (a1 - a0));
            const RecAB q = rab[k];
            r.rc = q.rc; r.frac = q.frac; r.v0 = q.a; r.v1 = q.b;
        } else {
            const int rj = ri - nab;
            const int k = rj < (e1 - e0) ? e0 + rj : f0 + (rj - (e1 - e0));
            const RecC q = rcc[k];
            r.rc = q.rc; r.frac = q.frac; r.v0 = q.c; r.v1 = q.c;
        }
        return r;
    };
    // Blocks of many records otherwise: one thread per record, the next one in
    // flight, its columns one after the other (no rounds, no barriers; the lanes
    // start at different columns and halves of a value, so that their adds
    // spread over the banks).
    if (MANY && dense) {
        __syncthreads();  // the tile is cleared
        const int sw = (tid >> 2) & 1;
        // adds the taps of a record's grids 0 .. n - 1 (values v[g], tiles GS apart)
        auto spread = [&](float2 *t0, int rc, float frac, const float2 *v, auto n) {
            int row = rc >> 16, x = c0 - (rc & 0xFFFF);
            if (x + B - 1 < 1 - m) { x += G2; row += 1; }
            else if (x > m) { x -= G2; row -= 1; }
            if (x + B - 1 < 1 - m || x > m) return;
            if (row < 0) row += L1;
            else if (row >= L1) row -= L1;
            float *t = reinterpret_cast<float *>(t0 + phys2<L1>(row) * B);
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const int cc = (k + tid) & (B - 1), d = x + cc;
                if (d < 1 - m || d > m) continue;
                const float wg = win_tap((float)d - frac, p);
#pragma unroll
                for (int g = 0; g < n; ++g) {
                    const float va = sw ? v[g].y : v[g].x, vb = sw ? v[g].x : v[g].y;
                    atomicAdd(t + 2 * (g * GS + cc) + sw, va * wg);
                    atomicAdd(t + 2 * (g * GS + cc) + (sw ^ 1), vb * wg);
                }
            }
        };
        auto at = [](int k, int s0, int s1, int r0) { return k < s1 - s0 ? s0 + k : r0 + (k - (s1 - s0)); };
        if (tid < nab) {
            RecAB nx = rab[at(tid, a0, a1, b0)];
            for (int k = tid; k < nab; k += NT) {
                const RecAB r = nx;
                if (k + NT < nab) nx = rab[at(k + NT, a0, a1, b0)];
                const float2 v[2] = {r.a, r.b};
                spread(tile, r.rc, r.frac, v, std::integral_constant<int, NG == 3 ? 2 : 1>());
            }
        }
        if (NG == 3 && tid < nc) {
            RecC nx = rcc[at(tid, e0, e1, f0)];
            for (int k = tid; k < nc; k += NT) {
                const RecC r = nx;
                if (k + NT < nc) nx = rcc[at(k + NT, e0, e1, f0)];
                spread(tile + 2 * GS, r.rc, r.frac, &r.c, std::integral_constant<int, 1>());
            }
        }
        __syncthreads();
    }
    for (int base = 0; !MANY || !dense; base += NSR) {
        const int cnt = min(NSR, ntot - base);
        if (GATHER && dense) {
            constexpr int RPT = (NSR + NT - 1) / NT;
            // 1. stage the round's records with the row each lands in for
            //    this block (one wrap decision per record: with G2 >= 2m + B
            //    the per-column wraps agree wherever a tap is inside the
            //    window), the offset x of its tap in column c0 kept in rc,
            //    and its rank within the row; records without a tap here
            //    are dropped
            int myrow[RPT], myrank[RPT];
#pragma unroll
            for (int q = 0; q < RPT; ++q) {
                const int j = tid + q * NT;
                myrow[q] = -1;
                myrank[q] = 0;
                if (j < cnt) {
                    StagedRec r = load_rec(base + j);
                    const int ck = r.rc & 0xFFFF;
                    int row = r.rc >> 16, x = c0 - ck;
                    if (x + B - 1 < 1 - m) { x += G2; row += 1; }
                    else if (x > m) { x -= G2; row -= 1; }
                    if (x + B - 1 >= 1 - m && x <= m) {
                        if (row < 0) row += L1;
                        else if (row >= L1) row -= L1;
                        r.rc = x;
                        st[j] = r;
                        myrow[q] = row;
                        myrank[q] = atomicAdd(&rowcnt[row], 1);
                    }
                }
            }
            __syncthreads();  // counts (and, first time, the zeroed tile)
            // 2. row offsets
            block_scan_counts<NT>(rowcnt, L1, wsum, tid);
            // 3. records in row order
#pragma unroll
            for (int q = 0; q < RPT; ++q)
                if (myrow[q] >= 0) {
                    const int at = rowcnt[myrow[q]] + myrank[q];
                    if ((unsigned)at < (unsigned)cnt) bucket[at] = tid + q * NT;
                }
            __syncthreads();
            // 4. whole rows per thread: taps summed in registers
            for (int r = tid; r < L1; r += NT) {
                float2 aA[B];
#pragma unroll
                for (int cc = 0; cc < B; ++cc) aA[cc] = make_float2(0.f, 0.f);
                // (bounds: offsets within the round's records, indices of
                // staged records)
                const int g0 = max(rowcnt[r], 0), g1 = min(rowcnt[r + 1], cnt);
                for (int e = g0; e < g1; ++e) {
                    const int j = bucket[e];
                    if ((unsigned)j >= (unsigned)cnt) continue;
                    const StagedRec rec = st[j];
#pragma unroll
                    for (int cc = 0; cc < B; ++cc) {
                        const int d = rec.rc + cc;
                        if (d < 1 - m || d > m) continue;
                        const float dd = (float)d - rec.frac;
                        const float wg = win_tap(dd, p);
                        aA[cc] = make_float2(fmaf(rec.v0.x, wg, aA[cc].x),
                                             fmaf(rec.v0.y, wg, aA[cc].y));
                    }
                }
                float2 *rp = tile + phys2<L1>(r) * B;
#pragma unroll
                for (int cc = 0; cc < B; ++cc) rp[cc] = cadd(rp[cc], aA[cc]);
            }
            __syncthreads();  // rows summed before the counts are reset
            for (int i = tid; i <= L1; i += NT) rowcnt[i] = 0;
        } else {
            for (int j = tid; j < cnt; j += NT) st[j] = load_rec(base + j);
            __syncthreads();  // staged records (and, first time, the zeroed tile)
            for (int it = tid; it < cnt * B; it += NT) {
                const int j = it / B, cc = it % B;
                const StagedRec r = st[j];
                const bool ab = base + j < nab;
                float2 *t0 = ab ? tile : tile + 2 * GS;
                // tap d of this record lands in column c0 + cc (modulo the row wrap)
                const int ck = r.rc & 0xFFFF, rk = r.rc >> 16;
                int d = c0 + cc - ck, row = rk;
                if (d < 1 - m) { d += G2; row += 1; }
                else if (d > m) { d -= G2; row -= 1; }
                if (d < 1 - m || d > m) continue;
                if (row < 0) row += L1;
                else if (row >= L1) row -= L1;
                if constexpr (LA1 > 0) occ[(ab ? 0 : 32) + row % LB1] = 1;
                const float dd = (float)d - r.frac;
                const float wg = win_tap(dd, p);
                float2 *cp = t0 + phys2<L1>(row) * B + cc;
                atomicAdd(&cp->x, r.v0.x * wg);
                atomicAdd(&cp->y, r.v0.y * wg);
                if (NG == 3 && ab) {
                    atomicAdd(&cp[GS].x, r.v1.x * wg);
                    atomicAdd(&cp[GS].y, r.v1.y * wg);
                }
            }
        }
        __syncthreads();  // the round is spread before it is overwritten
        if (base + NSR >= ntot) break;
    }

    // The intermediate of grid g is stored column-block-major,
    // I_g[cb][q1][c] (c fastest), so this CTA writes one contiguous block of
    // L1 B elements per grid.  The inter-pass twiddle
    // exp(2 pi i q1 (c0 + c) / G) comes from the plan table in the same order.
    const long long blk = (long long)cb * L1 * B;
    float2 *dst = inter + cv.inter_off + blk;
    const float2 *itw = p.itw + blk;
    const long long G = p.G;
    // vectors (g, c): base g * GS + c, element stride B
    if constexpr (two_level_la(L1) > 0) {
        // stage B stores straight to the intermediate: unit (g, c, qa) owns
        // outputs q1 = qa + LA qb, and consecutive threads run consecutive
        // (c, qa), so a warp writes contiguous runs of whole q1 rows
        constexpr int LA = two_level_la(L1), LB = L1 / LA;
        constexpr unsigned kAll = LB == 32 ? 0xFFFFFFFFu : (1u << LB) - 1u;
        unsigned mAB = kAll, mC = kAll;
        if (!dense) {  // uniform over the CTA; flags final after the last round's barrier
            const int lane = tid & 31;
            mAB = __ballot_sync(0xFFFFFFFFu, lane < LB && occ[lane] != 0);
            mC = __ballot_sync(0xFFFFFFFFu, lane < LB && occ[32 + lane] != 0);
        }
        tile_fft2_a_occ<L1, NG, B, GS, NT>(tile, tws, tid, mAB, mC);
        __syncthreads();
        float2 y[LB];
        int g, c, qa;
        if (tile_fft2_b<L1, NG * B, B, 1, GS, B, NT>(tile, tid, y, g, c, qa)) {
            // per-thread base pointers, then compile-time offsets qb La B
            // (one address computation per thread, not one per element)
            const int e0 = qa * B + c;
            float2 *d = dst + g * G + e0;
            const float2 *w = itw + e0;
#pragma unroll
            for (int qb = 0; qb < LB; ++qb) d[qb * LA * B] = cmul(y[qb], __ldg(w + qb * LA * B));
        }
    } else {
        tile_fft_any<L1, NG * B, B, 1, GS, B, NT>(tile, tws, tid);
#pragma unroll 2
        for (int e = tid; e < L1 * B; e += NT) {
            const int q1 = e / B, c = e % B;
            const float2 w = __ldg(itw + e);
            const int src = phys2<L1>(q1) * B + c;
#pragma unroll
            for (int g = 0; g < NG; ++g) dst[g * G + e] = cmul(tile[g * GS + src], w);
        }
    }
}

// Pass 1 with the compiler's own register choice ...
template <int NG, int L1, bool MANY>
__global__ void __launch_bounds__(pass1_threads(NG, L1))
k_pass1(const DevCurve *cvs, const RecAB *recAB, const RecC *recC, const int *binsAB,
        const int *binsC, float2 *inter, Plan p) {
    pass1_body<NG, L1, MANY>(cvs, recAB, recC, binsAB, binsC, inter, p);
}

// ... and, for the tiles whose smaller staging fits one more CTA per SM
// (pass1_small_stage), bound to that many CTAs per SM.  A minimum of one CTA
// per SM is not the same as no bound: it lets the compiler spend up to 255
// registers (pass 1 of rows of 400: 60 -> 110 registers, half the CTAs).
template <int NG, int L1, bool MANY>
__global__ void __launch_bounds__(pass1_threads(NG, L1), pass1_min_ctas(NG, L1))
k_pass1_occ(const DevCurve *cvs, const RecAB *recAB, const RecC *recC, const int *binsAB,
            const int *binsC, float2 *inter, Plan p) {
    pass1_body<NG, L1, MANY>(cvs, recAB, recC, binsAB, binsC, inter, p);
}

// Pass 1 of the GLS for the long columns (1,280 to 2,048): one CTA per curve,
// column block and grid.  The column FFT has three levels F0 F1 F2 with every
// butterfly in registers and in place: n = i + N1 k (N1 = F1 F2), i = j + F2 k',
// output q0 + F0 q1 + F0 F1 q2, which level 3 multiplies by the inter-pass
// twiddle and stores.  A record's taps are spread by one thread, straight from
// global memory: more of them are in flight than in rounds staged through
// shared memory and sorted by row.  Three grids of two columns in one CTA per SM
// (1,024 threads, that staging, Stockham stages) had nothing beside them to fill
// their barriers; two CTAs of one grid and four columns also halve the records
// read and give pass 2 whole 32-byte sectors.  10^6 points, 3 x 2048 x 4096
// cells: 1.066 -> 0.590 ms (0.24 ms of it the transforms, whose floor is
// 0.09 ms of stores; the rest the taps: window values and compare-and-swap
// adds, 52 % issue, L1 63 %); 1,000 points 0.413 -> 0.240 ms.
template <int L1>
__global__ void __launch_bounds__(pass1_threads(3, L1), 65536 / (64 * pass1_threads(3, L1)))
k_pass1_long(const DevCurve *cvs, const RecAB *recAB, const RecC *recC, const int *binsAB,
             const int *binsC, float2 *inter, const Plan p) {
    constexpr int B = kLongCols, NT = pass1_threads(3, L1);
    constexpr int F0 = long_fac(L1, 0), F1 = long_fac(L1, 1), F2 = long_fac(L1, 2), N1 = F1 * F2;
    static_assert(F0 * N1 == L1 && B == 4, "three levels, four columns");
    extern __shared__ __align__(16) float2 sm[];
    const int tid = threadIdx.x, cb = blockIdx.x / 3, g = blockIdx.x % 3, c0 = cb * B;
    if (p.dependent) {
        pdl_trigger();
        pdl_wait();  // descriptors and records; the intermediate read by earlier passes
    }
    recAB = written(recAB);
    recC = written(recC);
    const int *bins = written(g < 2 ? binsAB : binsC);
    const DevCurve cv = written(cvs)[blockIdx.y];  // in flight during the zero-fill
    {
        float4 *t4 = reinterpret_cast<float4 *>(sm);
        for (int i = tid; i < (L1 + F0) * B / 2; i += NT) t4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int G2 = p.G2, m = p.m;
    int a0, a1, b0, b1;
    bin_ranges(bins + cv.bin_off, cb, -((m + B - 1) / B), (B + m - 2) / B, p.nb, a0, a1, b0, b1);
    const int na = a1 - a0, ntot = na + (b1 - b0);
    const RecAB *rab = recAB + cv.rec_off;
    const RecC *rcc = recC + cv.rec_off;
    struct Rec {
        int rc;
        float frac;
        float2 v;
    };
    auto load = [&](int k) {
        k = k < na ? a0 + k : b0 + (k - na);
        Rec r;
        if (g < 2) {
            const RecAB *q = rab + k;
            r.rc = q->rc; r.frac = q->frac; r.v = g == 0 ? q->a : q->b;
        } else {
            const RecC q = rcc[k];
            r.rc = q.rc; r.frac = q.frac; r.v = q.c;
        }
        return r;
    };
    // The lanes of a warp start at different columns and halves of a value, so
    // that their adds spread over the banks.
    const int sw = (tid >> 2) & 1;
    auto spread = [&](const Rec &r) {
        // one wrap decision per record: with G2 >= 2 m + B the columns agree
        // wherever a tap is inside the window
        int row = r.rc >> 16, x = c0 - (r.rc & 0xFFFF);
        if (x + B - 1 < 1 - m) { x += G2; row += 1; }
        else if (x > m) { x -= G2; row -= 1; }
        if (x + B - 1 < 1 - m || x > m) return;
        if (row < 0) row += L1;
        else if (row >= L1) row -= L1;
        float *t = reinterpret_cast<float *>(sm + (row + row / N1) * B);
        const float va = sw ? r.v.y : r.v.x, vb = sw ? r.v.x : r.v.y;
#pragma unroll
        for (int k = 0; k < B; ++k) {
            const int cc = (k + tid) & (B - 1), d = x + cc;
            if (d < 1 - m || d > m) continue;
            const float wg = win_tap((float)d - r.frac, p);
            atomicAdd(t + 2 * cc + sw, va * wg);
            atomicAdd(t + 2 * cc + (sw ^ 1), vb * wg);
        }
    };
    constexpr int U = 2;  // records in flight per thread
    Rec nx[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (tid + u * NT < ntot) nx[u] = load(tid + u * NT);
    __syncthreads();  // the tile is cleared
    for (int k0 = tid; k0 < ntot; k0 += U * NT) {
        Rec r[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            r[u] = nx[u];
            const int k = k0 + (u + U) * NT;
            if (k < ntot) nx[u] = load(k);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k0 + u * NT < ntot) spread(r[u]);
    }
    __syncthreads();
    const int c = tid & (B - 1);
    // level 1: unit (i, c), planes of N1 + 1 slots
    const float2 *w1 = p.st1 + stage_tw_offset(L1, 2), *w2 = p.st1 + stage_tw_offset(L1, 1);
#pragma unroll 1
    for (int u = tid; u < N1 * B; u += NT) {
        const int i = u / B;
        float2 *e = sm + i * B + c, x[F0];
#pragma unroll
        for (int k = 0; k < F0; ++k) x[k] = e[k * (N1 + 1) * B];
        RegDFT<F0>::run(x);
        e[0] = x[0];
#pragma unroll
        for (int q = 1; q < F0; ++q) e[q * (N1 + 1) * B] = cmul(x[q], __ldg(w1 + (q - 1) * N1 + i));
    }
    __syncthreads();
    {  // level 2: unit (q0, j, c), one per thread
        const int j = tid / B % F2, q0 = tid / (B * F2);
        float2 *e = sm + (q0 * (N1 + 1) + j) * B + c, x[F1];
#pragma unroll
        for (int k = 0; k < F1; ++k) x[k] = e[k * F2 * B];
        RegDFT<F1>::run(x);
        e[0] = x[0];
#pragma unroll
        for (int q = 1; q < F1; ++q) e[q * F2 * B] = cmul(x[q], __ldg(w2 + (q - 1) * F2 + j));
    }
    __syncthreads();
    // level 3: unit (q1, q0, c): outputs v + F0 F1 q2, v = q0 + F0 q1
    const long long blk = (long long)cb * L1 * B;
    float2 *dst = inter + cv.inter_off + g * p.G + blk;
    const float2 *itw = p.itw + blk;
#pragma unroll 1
    for (int u = tid; u < F0 * F1 * B; u += NT) {
        const int v = u / B, q0 = v % F0, q1 = v / F0;
        const float2 *e = sm + (q0 * (N1 + 1) + q1 * F2) * B + c;
        float2 x[F2];
#pragma unroll
        for (int j = 0; j < F2; ++j) x[j] = e[j * B];
        RegDFT<F2>::run(x);
#pragma unroll
        for (int q = 0; q < F2; ++q)
            dst[u + q * F0 * F1 * B] = cmul(x[q], __ldg(itw + u + q * F0 * F1 * B));
    }
}

template <int NG, int L2, int R, int NT, int LDS, int B>
__device__ __forceinline__ void load_rows_b(float2 *tile, const float2 *__restrict__ src,
                                            int G1, long long G, int rb, int tid) {
    // Consecutive threads fill consecutive element pairs of one tile row
    // (conflict-free shared stores); each pair is a 16-byte global load.
    constexpr int PR = L2 / 2;          // element pairs per row
    static_assert(B % 2 == 0, "B must be even");
#pragma unroll 4
    for (int e = tid; e < NG * R * PR; e += NT) {
        const int pr = e % PR, v = e / PR;
        const int g = v / R, r = v - g * R;
        const int l2 = 2 * pr;
        const int cb = l2 / B, c = l2 % B;
        const float4 val = __ldg(reinterpret_cast<const float4 *>(
            src + g * G + ((long long)cb * G1 + (long long)rb * R + r) * B + c));
        float2 *d = tile + v * LDS;
        d[phys2<L2>(l2)] = make_float2(val.x, val.y);
        d[phys2<L2>(l2 + 1)] = make_float2(val.z, val.w);
    }
}

// Rows rb R .. rb R + R - 1 of NG grids, transformed along the row (length
// L2) into the padded tile; ends with a barrier.  With a two-level split
// whose LB is a multiple of B, stage A reads its inputs straight from the
// intermediate: unit (g, r, i = ih B + c) takes elements i + LB k, all in
// column block ih + (LB / B) k at column c, and consecutive threads run
// consecutive (c, r), so a warp reads whole R x B blocks.  Otherwise the
// rows are loaded into the tile first.
template <int NG, int L2, int R, int NT, int LDS, int B>
__device__ __forceinline__ void rows_fft_b(float2 *tile, const float2 *__restrict__ src,
                                           const float2 *__restrict__ tab, int G1, long long G,
                                           int rb, int tid) {
    constexpr int LA = two_level_la(L2);
    if constexpr (LA > 0 && (L2 / LA) % B == 0) {
        constexpr int LB = L2 / LA, IH = LB / B;
        const int kstride = IH * G1 * B;  // elements between column blocks ih and ih + IH
#pragma unroll 1
        for (int u = tid; u < NG * R * LB; u += NT) {
            const int c = u % B;
            int t = u / B;
            const int r = t % R;
            t /= R;
            const int ih = t % IH, g = t / IH;
            const float2 *s = src + g * G + (ih * G1 + rb * R + r) * B + c;
            float2 x[LA];
#pragma unroll
            for (int k = 0; k < LA; ++k) x[k] = __ldg(s + k * kstride);
            const int i = ih * B + c;
            fft2_stage_a_regs<L2>(x, tab, i);
            float2 *d = tile + (g * R + r) * LDS;
#pragma unroll
            for (int qa = 0; qa < LA; ++qa) d[phys2_ik<L2>(i, qa)] = x[qa];
        }
        __syncthreads();
        tile_fft2_b_inplace<L2, NG * R, 1, 0, LDS, 1, NT>(tile, tid);
    } else {
        load_rows_b<NG, L2, R, NT, LDS, B>(tile, src, G1, G, rb, tid);
        const float2 *tws = tab;
        if constexpr (LA == 0) {
            float2 *t = tile + NG * R * LDS;
            for (int i = tid; i < fft_table_len(L2); i += NT) t[i] = tab[i];
            tws = t;
        }
        __syncthreads();
        tile_fft_any<L2, NG * R, 1, 0, LDS, 1, NT>(tile, tws, tid);
    }
}

// Pass 2 of the GLS for rows of 4,096: one row of one curve per CTA of 256
// threads.  Each grid's row is transformed in three levels of 16 with every
// butterfly in registers: n = i + 256 k, i = j + 16 k', output
// q2 = q0 + 16 q1 + 256 qb.
//   level 1  thread i reads its 16 elements straight from the intermediate
//            and leaves [q0][i] in the exchange tile;
//   level 2  thread (q0, j), in place;
//   level 3  thread (q1, q0) holds the outputs q0 + 16 q1 + 256 qb.
// The outputs stay in registers (grid A's parked in shared memory and read
// back by the same thread), so the powers need no further pass.  The planes'
// pitch of 257 keeps all accesses free of bank conflicts.  3 x 2048 rows of
// three grids: 0.631 -> 0.350 ms (0.406 with two columns per pass-1 block, 0.465
// with 80 registers and three CTAs per SM); 604 MB read, 0.09 ms at the
// measured copy rate: it is held by latency (two CTAs per SM) and by the L1
// pipe (56 %: a row is 1,024 pieces of 32 bytes, its powers 4-byte stores).
template <bool ES>
__global__ void __launch_bounds__(256, 2)
k_pass2_gls_cube(const DevCurve *cvs, const float2 *inter, float *__restrict__ out, const Plan p,
                 const GlsParams gp) {
    constexpr int L2 = 4096, P = kCubePitch;
    extern __shared__ __align__(16) float2 sm[];
    float2 *ex = sm, *park = sm + 16 * P;
    const int tid = threadIdx.x, q1r = blockIdx.x;
    if (p.dependent) {
        pdl_trigger();
        pdl_wait();
    }
    inter = written(inter);
    const DevCurve cv = written(cvs)[blockIdx.y];
    constexpr int B = kGlsCols;
    const int G1 = p.G1, G = (int)p.G;
    const int lo = tid & 15, hi = tid >> 4;
    // element l = tid + 256 k of the row lies at ((l / B) G1 + row) B + l % B
    const float2 *src = inter + cv.inter_off + ((long long)(tid / B) * G1 + q1r) * B + tid % B;
    const int kstride = 256 * G1;
    const float2 *w1 = p.st2 + 240 + tid, *w2 = p.st2 + lo;  // Stockham tables of 4096
    float2 y[16], yb[16], x[16];
    // (volatile: the loads stay ahead of the levels they are to overlap)
    auto fetch = [](const float2 *q) {
        float2 v;
        asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(q) : "memory");
        return v;
    };
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = fetch(src + k * kstride);
#pragma unroll
    for (int g = 0; g < 3; ++g) {
        RegDFT<16>::run(x);
        if (g) __syncthreads();  // the grid before is read
        ex[tid] = x[0];
#pragma unroll
        for (int q = 1; q < 16; ++q) ex[q * P + tid] = cmul(x[q], __ldg(w1 + (q - 1) * 256));
        if (g < 2) {  // the next grid's row, in flight during levels 2 and 3
            src += p.G;
#pragma unroll
            for (int k = 0; k < 16; ++k) x[k] = fetch(src + k * kstride);
        }
        __syncthreads();
        float2 *e = ex + hi * P + lo;  // (q0, j) = (hi, lo)
#pragma unroll
        for (int k = 0; k < 16; ++k) y[k] = e[16 * k];
        RegDFT<16>::run(y);
        e[0] = y[0];
#pragma unroll
        for (int q = 1; q < 16; ++q) e[16 * q] = cmul(y[q], __ldg(w2 + (q - 1) * 16));
        __syncthreads();
        e = ex + lo * P + 16 * hi;  // (q0, q1) = (lo, hi)
#pragma unroll
        for (int j = 0; j < 16; ++j) y[j] = e[j];
        RegDFT<16>::run(y);
        if (g == 0) {
#pragma unroll
            for (int q = 0; q < 16; ++q) park[q * 256 + tid] = y[q];
        } else if (g == 1) {
#pragma unroll
            for (int q = 0; q < 16; ++q) yb[q] = y[q];
        }
    }
    const int nf = cv.nf, h = nf / 2, lo_end = nf - h, hi_start = G - h;
    const bool write = gp.best == nullptr || out != nullptr;
    float *o = out + cv.out_off + h;
    const int q0 = q1r + G1 * tid;
    const float *drow = ES ? p.drow + (long long)q1r * L2 + tid : nullptr;
    const Fm2 fm(cv, gp.reg);
    unsigned long long key = 0;
    const unsigned ibase = (unsigned)(cv.best_off + h);
    auto emit = [&](float P, int k) {
        if (write) o[k] = P;
        if (gp.best != nullptr && P >= 0.f) {  // valid powers only
            const unsigned long long kk = ((unsigned long long)__float_as_uint(P) << 32) |
                                          (0xFFFFFFFFu - (ibase + (unsigned)k));
            key = kk > key ? kk : key;
        }
    };
    // two frequencies at a time; f(qb, ka, kb, ina, inb, A0, A1, D)
    auto pairs = [&](auto f) {
#pragma unroll
        for (int qb = 0; qb < 16; qb += 2) {
            // (no band reaches the middle fifth of the grid: sigma >= 1.25)
            if (5 * qb >= 2 * 16 && 5 * (qb + 2) <= 3 * 16) continue;
            const int qA = q0 + G1 * 256 * qb, qB = qA + G1 * 256;
            const bool ina = qA < lo_end || qA >= hi_start;
            const bool inb = qB < lo_end || qB >= hi_start;
            if (!ina && !inb) continue;
            const float2 A0 = park[qb * 256 + tid], A1 = park[(qb + 1) * 256 + tid];
            const int ka = qA < lo_end ? qA : qA - G, kb = qB < lo_end ? qB : qB - G;
            float2 D;
            if constexpr (ES) D = make_float2(__ldg(drow + 256 * qb), __ldg(drow + 256 * (qb + 1)));
            else D = make_float2(win_deconv<false>(ka, p), win_deconv<false>(kb, p));
            f(qb, ka, kb, ina, inb, A0, A1, D);
        }
    };
    if (gp.mode == 1) {
        pairs([&](int qb, int ka, int kb, bool ina, bool inb, float2 A0, float2 A1, float2 D) {
            const float2 pw = fm.power(A0, A1, yb[qb], yb[qb + 1], y[qb], y[qb + 1], D);
            if (ina) emit(pw.x, ka);
            if (inb) emit(pw.y, kb);
        });
    } else {
        auto one = [&](float2 A, float2 Bv, float2 C, float d) {
            return gls_from_sums<float>(A.x * d, A.y * d, Bv.x * d, Bv.y * d, C.x * d, C.y * d,
                                        gp.mode, gp.reg, cv.w_sum, cv.yw_sum, cv.ybar, cv.yy_inv);
        };
        pairs([&](int qb, int ka, int kb, bool ina, bool inb, float2 A0, float2 A1, float2 D) {
            if (ina) emit(one(A0, yb[qb], y[qb], D.x), ka);
            if (inb) emit(one(A1, yb[qb + 1], y[qb + 1], D.y), kb);
        });
    }
    if (gp.best != nullptr) {
#pragma unroll
        for (int of = 16; of > 0; of >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, key, of);
            key = v > key ? v : key;
        }
        if ((tid & 31) == 0 && key != 0) atomicMax(gp.best + cv.best_slot, key);
    }
}

// Pass 2 of the GLS for rows of 512 to 2,048: R rows of one curve per CTA, each
// grid transformed in three levels with every butterfly in registers, as
// k_pass2_gls_cube: n = i + N1 k (N1 = 8 F1), i = j + 8 k', output q0 + F0 q1 +
// F0 F1 qb.  Level 3 leaves the eight outputs of a thread in its registers for
// the powers, which went back to shared memory and were read again before.
// Per cell on grids of 320 columns: rows of 512 10.5 -> 7.1 ps, 640 8.5 -> 8.4,
// 800 9.7 -> 8.8, 1,024 12.2 -> 10.1, 1,280 20.2 -> 11.2 (without the next grid's
// loads ahead 7.6, 9.4, 10.5, 11.4, 11.8).  Held by latency: 13 to 24 warps per
// SM between three barriers a grid.
template <int L2, bool ES>
__global__ void __launch_bounds__(deep_threads(L2), deep_ctas(L2))
k_pass2_gls_deep(const DevCurve *cvs, const float2 *inter, float *__restrict__ out, const Plan p,
                 const GlsParams gp) {
    constexpr int R = deep_rows(L2), NT = deep_threads(L2);
    constexpr int F0 = deep_fac(L2, 0), F1 = deep_fac(L2, 1), N1 = 8 * F1;
    constexpr int P0 = deep_plane(L2), PR = deep_pitch(L2), T = L2 / 8;
    static_assert(F0 * N1 == L2 && N1 % 4 == 0, "three levels");
    extern __shared__ __align__(16) float2 sm[];
    const int tid = threadIdx.x, rb = blockIdx.x;
    if (p.dependent) {
        pdl_trigger();
        pdl_wait();
    }
    inter = written(inter);
    const DevCurve cv = written(cvs)[blockIdx.y];
    constexpr int lb = 2;
    static_assert(1 << lb == kGlsCols, "blocks of four columns");
    const int G1 = p.G1, G = (int)p.G;
    const float2 *w1 = p.st2, *w2 = p.st2 + L2;
    const float2 *src = inter + cv.inter_off + (long long)rb * R * kGlsCols;
    const int kstride = N1 * G1;  // elements between column blocks of n and n + N1
    const int r3 = tid % R, v3 = tid / R;  // level-3 unit: row, q1 = v3 % F1, q0 = v3 / F1
    const bool act = NT == R * T || v3 < T;
    float2 ya[8], yb[8], yc[8], x[F0];
    // level-1 unit (ih, r, c), i = ih B + c
    const bool one = N1 * R == NT || tid < N1 * R;
    static_assert(N1 * R <= NT && F0 * 8 * R <= NT, "a unit per thread");
    const int i1 = ((tid >> lb) / R << lb) + (tid & ((1 << lb) - 1)), r1 = (tid >> lb) % R;
    src += (((long long)((tid >> lb) / R) * G1 + r1) << lb) + (tid & ((1 << lb) - 1));
    // (volatile: the loads stay ahead of the levels they are to overlap)
    auto fetch = [](const float2 *q) {
        float2 v;
        asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(q) : "memory");
        return v;
    };
    if (one) {
#pragma unroll
        for (int k = 0; k < F0; ++k) x[k] = fetch(src + k * kstride);
    }
#pragma unroll
    for (int g = 0; g < 3; ++g) {
        if (one) RegDFT<F0>::run(x);
        if (g) __syncthreads();  // the grid before is read
        if (one) {
            float2 *d = sm + r1 * PR + i1 + (i1 >> 3);
            d[0] = x[0];
#pragma unroll
            for (int q = 1; q < F0; ++q) d[q * P0] = cmul(x[q], __ldg(w1 + q * N1 + i1));
            if (g < 2) {  // the next grid's rows, in flight during levels 2 and 3
                src += p.G;
#pragma unroll
                for (int k = 0; k < F0; ++k) x[k] = fetch(src + k * kstride);
            }
        }
        __syncthreads();
        // level 2: unit (r, q0, j), in place
        if (F0 * 8 * R == NT || tid < F0 * 8 * R) {
            const int j = tid & 7, q0 = (tid >> 3) % F0, r = (tid >> 3) / F0;
            float2 *e = sm + r * PR + q0 * P0 + j, u[F1];
#pragma unroll
            for (int k = 0; k < F1; ++k) u[k] = e[9 * k];
            RegDFT<F1>::run(u);
            e[0] = u[0];
#pragma unroll
            for (int q = 1; q < F1; ++q) e[9 * q] = cmul(u[q], __ldg(w2 + q * 8 + j));
        }
        __syncthreads();
        float2 *y = g == 0 ? ya : g == 1 ? yb : yc;
        if (act) {
            const float2 *e = sm + r3 * PR + (v3 / F1) * P0 + 9 * (v3 % F1);
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] = e[j];
            RegDFT<8>::run(y);
        }
    }
    const int nf = cv.nf, h = nf / 2, lo_end = nf - h, hi_start = G - h;
    const bool write = gp.best == nullptr || out != nullptr;
    float *o = out + cv.out_off + h;
    const int qv = v3 / F1 + F0 * (v3 % F1), q0 = rb * R + r3 + G1 * qv;
    const float *drow = ES ? p.drow + ((long long)rb * L2 + qv) * R + r3 : nullptr;
    const Fm2 fm(cv, gp.reg);
    unsigned long long key = 0;
    const unsigned ibase = (unsigned)(cv.best_off + h);
    auto emit = [&](float P, int k) {
        if (write) o[k] = P;
        if (gp.best != nullptr && P >= 0.f) {  // valid powers only
            const unsigned long long kk = ((unsigned long long)__float_as_uint(P) << 32) |
                                          (0xFFFFFFFFu - (ibase + (unsigned)k));
            key = kk > key ? kk : key;
        }
    };
    // two frequencies at a time; f(qb, ka, kb, ina, inb, D)
    auto pairs = [&](auto f) {
#pragma unroll
        for (int qb = 0; qb < 8; qb += 2) {
            const int qA = q0 + G1 * T * qb, qB = qA + G1 * T;
            const bool ina = qA < lo_end || qA >= hi_start;
            const bool inb = qB < lo_end || qB >= hi_start;
            if (!ina && !inb) continue;
            const int ka = qA < lo_end ? qA : qA - G, kb = qB < lo_end ? qB : qB - G;
            float2 D;
            if constexpr (ES)
                D = make_float2(__ldg(drow + T * R * qb), __ldg(drow + T * R * (qb + 1)));
            else
                D = make_float2(win_deconv<false>(ka, p), win_deconv<false>(kb, p));
            f(qb, ka, kb, ina, inb, D);
        }
    };
    if (act && gp.mode == 1) {
        pairs([&](int qb, int ka, int kb, bool ina, bool inb, float2 D) {
            const float2 pw = fm.power(ya[qb], ya[qb + 1], yb[qb], yb[qb + 1], yc[qb], yc[qb + 1], D);
            if (ina) emit(pw.x, ka);
            if (inb) emit(pw.y, kb);
        });
    } else if (act) {
        auto one = [&](float2 A, float2 Bv, float2 C, float d) {
            return gls_from_sums<float>(A.x * d, A.y * d, Bv.x * d, Bv.y * d, C.x * d, C.y * d,
                                        gp.mode, gp.reg, cv.w_sum, cv.yw_sum, cv.ybar, cv.yy_inv);
        };
        pairs([&](int qb, int ka, int kb, bool ina, bool inb, float2 D) {
            if (ina) emit(one(ya[qb], yb[qb], yc[qb], D.x), ka);
            if (inb) emit(one(ya[qb + 1], yb[qb + 1], yc[qb + 1], D.y), kb);
        });
    }
    if (gp.best != nullptr) {
#pragma unroll
        for (int of = 16; of > 0; of >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, key, of);
            key = v > key ? v : key;
        }
        if ((tid & 31) == 0 && key != 0) atomicMax(gp.best + cv.best_slot, key);
    }
}

// Adjoint-NFFT finish of a pass-2 tile: deconvolution and the phase of the
// absolute time origin, complex output per in-band frequency.
template <bool ES, int L2, int R, int NT, int LDS>
__device__ __forceinline__ void nfft_finish(const float2 *tile, const DevCurve &cv,
                                            float2 *__restrict__ out,
                                            const ulonglong2 *__restrict__ aux, const Plan &p,
                                            int rb, int tid) {
    const ulonglong2 ax = aux[cv.aux];
    const long long G = p.G;
    const int G1 = p.G1;
    const int nf = cv.nf, h = nf / 2;
    for (int e = tid; e < R * L2; e += NT) {
        const int r = e % R, q2 = e / R;
        const int kp = band_index((long long)(rb * R + r) + (long long)G1 * q2, nf, h, G);
        if (kp == INT_MIN) continue;
        const float D = ES ? __ldg(p.drow + (long long)rb * R * L2 + e) : win_deconv<false>(kp, p);
        const float2 ph = turn_phasor(ax.x + (unsigned long long)(long long)kp * ax.y);
        out[cv.out_off + kp + h] = cmul(cscale(tile[r * LDS + phys2<L2>(q2)], D), ph);
    }
}

template <int L2>
__global__ void __launch_bounds__(pass2_threads(1, L2))
k_pass2_nfft(const DevCurve *cvs, const float2 *inter, float2 *__restrict__ out,
             const ulonglong2 *aux, Plan p) {
    constexpr int R = pass2_rows(1, L2);
    constexpr int NT = pass2_threads(1, L2);
    constexpr int LDS = row_stride(L2);
    extern __shared__ __align__(16) float2 sm[];
    float2 *tile = sm;
    const int tid = threadIdx.x, rb = blockIdx.x;
    if (p.dependent) {
        pdl_trigger();
        pdl_wait();
    }
    inter = written(inter);
    aux = written(aux);
    const DevCurve cv = written(cvs)[blockIdx.y];
    rows_fft_b<1, L2, R, NT, LDS, kNfftCols>(tile, inter + cv.inter_off, p.st2, p.G1, p.G, rb, tid);

    if (p.win == kWinES) nfft_finish<true, L2, R, NT, LDS>(tile, cv, out, aux, p, rb, tid);
    else nfft_finish<false, L2, R, NT, LDS>(tile, cv, out, aux, p, rb, tid);
}

// ---- launch templates (explicitly instantiated in the inst_*.cu files) ----
// Raise a kernel's dynamic shared-memory limit to `bytes`.  `done` is the
// caller's per-kernel cache (one per device): every length instantiation has
// its own, because instantiations share a function type but not attributes.
template <typename K>
static cudaError_t allow_smem(K kernel, size_t bytes, size_t (&done)[64]) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (bytes <= 48 * 1024 || bytes <= done[dev]) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)bytes);
    if (e == cudaSuccess) done[dev] = bytes;
    return e;
}

// Whether a launch takes the kernel that also spreads by records: it is
// compiled apart, because the registers of that path cost the others 2 % to
// 3 % (2,000 curves of 320 x 400 cells 1746 -> 1787 us).  It pays from a few
// rounds per thread on: 16 curves of 50 to 5,000 points on 160 x 160 cells
// 57 -> 43 us, 48 curves of 100 to 20,000 points 455 -> 379 us.
template <int NG, int L1>
bool pass1_many(int max_n, const Plan &p) {
    constexpr int B = pass1_cols(NG, L1);
    const int bins = (B + p.m - 2) / B + (p.m + B - 1) / B + 1;
    const long long recs = (long long)max_n * (NG == 3 ? 2 : 1) * bins * B / p.G2;
    return recs >= 4LL * pass1_threads(NG, L1);
}

template <int NG, int L1, typename K>
cudaError_t launch_pass1_k(K kernel, size_t (&done)[64], int n_curves, const Plan &p, int per,
                           cudaStream_t s, const DevCurve *cv, const RecAB *recAB, const RecC *recC,
                           const int *binsAB, const int *binsC, float2 *inter) {
    const size_t smem = (size_t)pass1_smem(NG, L1, p.G);
    const cudaError_t e = allow_smem(kernel, smem, done);
    if (e != cudaSuccess) return e;
    const dim3 grid(p.G2 / pass1_cols(NG, L1) * per, n_curves);
    Plan q = p;
    q.dependent = small_launch((long long)grid.x * grid.y);
    return launch_pdl(kernel, q.dependent, grid, pass1_threads(NG, L1), smem, s, cv, recAB, recC,
                      binsAB, binsC, inter, q);
}

template <int NG, int L1>
cudaError_t launch_pass1_t(const DevCurve *cv, int n_curves, int max_n, const RecAB *recAB,
                           const RecC *recC, const int *binsAB, const int *binsC,
                           float2 *inter, const Plan &p, cudaStream_t s) {
    static size_t done[2][64] = {{0}};  // per instantiation
    auto go = [&](auto kernel, int k) {
        return launch_pass1_k<NG, L1>(kernel, done[k], n_curves, p, pass1_long(NG, L1) ? 3 : 1, s,
                                      cv, recAB, recC, binsAB, binsC, inter);
    };
    if constexpr (pass1_long(NG, L1)) {
        return go(k_pass1_long<L1>, 0);
    } else if constexpr (pass1_small_stage(NG, L1)) {
        return pass1_many<NG, L1>(max_n, p) ? go(k_pass1_occ<NG, L1, true>, 1)
                                            : go(k_pass1_occ<NG, L1, false>, 0);
    } else if constexpr (pass1_gather(NG, L1)) {
        return go(k_pass1<NG, L1, false>, 0);
    } else {
        return pass1_many<NG, L1>(max_n, p) ? go(k_pass1<NG, L1, true>, 1)
                                            : go(k_pass1<NG, L1, false>, 0);
    }
}

template <int L2>
cudaError_t launch_pass2_gls_t(const DevCurve *cv, int n_curves, int first, const float2 *inter,
                               float *out, const Plan &p, GlsParams g, cudaStream_t s) {
    if constexpr (pass2_reg(3, L2)) {
        if (p.win == kWinES)  // (sigma 1.28)
            return launch_pass2_reg_t<L2, true, false>(cv, n_curves, first, inter, out, p, g, s);
        return p.narrow
                   ? launch_pass2_reg_t<L2, false, true>(cv, n_curves, first, inter, out, p, g, s)
                   : launch_pass2_reg_t<L2, false, false>(cv, n_curves, first, inter, out, p, g, s);
    } else if constexpr (pass2_deep(3, L2)) {
        static size_t done[2][64] = {{0}};  // per window and device
        const bool es = p.win == kWinES;
        const size_t smem = (size_t)pass2_smem(3, L2);
        cudaError_t e = es ? allow_smem(k_pass2_gls_deep<L2, true>, smem, done[1])
                           : allow_smem(k_pass2_gls_deep<L2, false>, smem, done[0]);
        if (e != cudaSuccess) return e;
        const dim3 grid(p.G1 / deep_rows(L2), n_curves);
        Plan q = p;
        q.dependent = small_launch((long long)grid.x * grid.y);
        return es ? launch_pdl(k_pass2_gls_deep<L2, true>, q.dependent, grid, deep_threads(L2), smem, s,
                               cv, inter, out, q, g)
                  : launch_pdl(k_pass2_gls_deep<L2, false>, q.dependent, grid, deep_threads(L2), smem, s,
                               cv, inter, out, q, g);
    } else {
        static_assert(pass2_cube(3, L2), "no other rows");
        static size_t done[2][64] = {{0}};  // per window and device
        const bool es = p.win == kWinES;
        const size_t smem = (size_t)pass2_smem(3, L2);
        cudaError_t e = es ? allow_smem(k_pass2_gls_cube<true>, smem, done[1])
                           : allow_smem(k_pass2_gls_cube<false>, smem, done[0]);
        if (e != cudaSuccess) return e;
        const dim3 grid(p.G1, n_curves);
        Plan q = p;
        q.dependent = small_launch((long long)grid.x * grid.y);
        return es ? launch_pdl(k_pass2_gls_cube<true>, q.dependent, grid, 256, smem, s, cv, inter, out, q, g)
                  : launch_pdl(k_pass2_gls_cube<false>, q.dependent, grid, 256, smem, s, cv, inter, out, q, g);
    }
}

template <int L2>
cudaError_t launch_pass2_nfft_t(const DevCurve *cv, int n_curves, int first, const float2 *inter,
                                float2 *out, const ulonglong2 *aux, unsigned *errflag,
                                const Plan &p, cudaStream_t s) {
    if constexpr (pass2_reg(1, L2)) {
        return p.win == kWinES
                   ? launch_nfft_reg_t<L2, true>(cv, n_curves, first, inter, out, aux, errflag, p, s)
                   : launch_nfft_reg_t<L2, false>(cv, n_curves, first, inter, out, aux, errflag, p, s);
    } else {
        static size_t done[64] = {0};  // per instantiation
        cudaError_t e = allow_smem(k_pass2_nfft<L2>, (size_t)pass2_smem(1, L2), done);
        if (e != cudaSuccess) return e;
        const dim3 grid(p.G1 / pass2_rows(1, L2), n_curves);
        Plan q = p;
        q.dependent = small_launch((long long)grid.x * grid.y);
        return launch_pdl(k_pass2_nfft<L2>, q.dependent, grid, pass2_threads(1, L2),
                          (size_t)pass2_smem(1, L2), s, cv, inter, out, aux, q);
    }
}

// Load the pass kernels of a length now (CUDA loads kernels lazily, at
// their first launch, which would otherwise land in the first batch of a new
// plan class: a stall of milliseconds in a serving loop).
template <int NG, int L1>
cudaError_t preload_pass1_t() {
    cudaFuncAttributes a;
    if constexpr (pass1_long(NG, L1)) {
        return cudaFuncGetAttributes(&a, k_pass1_long<L1>);
    } else if constexpr (pass1_small_stage(NG, L1)) {
        const cudaError_t e = cudaFuncGetAttributes(&a, k_pass1_occ<NG, L1, false>);
        return e != cudaSuccess ? e : cudaFuncGetAttributes(&a, k_pass1_occ<NG, L1, true>);
    } else {
        const cudaError_t e = cudaFuncGetAttributes(&a, k_pass1<NG, L1, false>);
        if constexpr (pass1_gather(NG, L1)) return e;
        else return e != cudaSuccess ? e : cudaFuncGetAttributes(&a, k_pass1<NG, L1, true>);
    }
}
template <int L2>
cudaError_t preload_pass2_t(int ng) {
    cudaFuncAttributes a;
    if constexpr (pass2_reg(3, L2)) {
        if (ng != 3) {
            const cudaError_t e = cudaFuncGetAttributes(&a, k_pass2_nfft_reg<L2, true, kWaitTries>);
            return e != cudaSuccess ? e : cudaFuncGetAttributes(&a, k_pass2_nfft_reg<L2, false, kWaitTries>);
        }
        cudaError_t e = cudaFuncGetAttributes(&a, k_pass2_gls_reg<L2, true, false, kWaitTries>);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_pass2_gls_reg<L2, false, true, kWaitTries>);
        return e != cudaSuccess ? e : cudaFuncGetAttributes(&a, k_pass2_gls_reg<L2, false, false, kWaitTries>);
    } else if constexpr (pass2_deep(3, L2)) {
        if (ng != 3) return cudaFuncGetAttributes(&a, k_pass2_nfft<L2>);
        const cudaError_t e = cudaFuncGetAttributes(&a, k_pass2_gls_deep<L2, true>);
        return e != cudaSuccess ? e : cudaFuncGetAttributes(&a, k_pass2_gls_deep<L2, false>);
    } else {
        if (ng != 3) return cudaFuncGetAttributes(&a, k_pass2_nfft<L2>);
        const cudaError_t e = cudaFuncGetAttributes(&a, k_pass2_gls_cube<true>);
        return e != cudaSuccess ? e : cudaFuncGetAttributes(&a, k_pass2_gls_cube<false>);
    }
}

#define CUVGLS_INSTANTIATE_ROW_LEN(L)                                               \
    template cudaError_t launch_pass2_gls_t<L>(const DevCurve *, int, int, const float2 *, \
                                               float *, const Plan &, GlsParams,     \
                                               cudaStream_t);                        \
    template cudaError_t launch_pass2_nfft_t<L>(const DevCurve *, int, int, const float2 *, \
                                                float2 *, const ulonglong2 *, unsigned *, \
                                                const Plan &, cudaStream_t);                       \
    template cudaError_t preload_pass2_t<L>(int);

#define CUVGLS_INSTANTIATE_LEN(L)                                                   \
    template cudaError_t launch_pass1_t<3, L>(const DevCurve *, int, int, const RecAB *, \
                                              const RecC *, const int *, const int *, \
                                              float2 *, const Plan &, cudaStream_t); \
    template cudaError_t launch_pass1_t<1, L>(const DevCurve *, int, int, const RecAB *, \
                                              const RecC *, const int *, const int *, \
                                              float2 *, const Plan &, cudaStream_t); \
    template cudaError_t launch_pass2_gls_t<L>(const DevCurve *, int, int, const float2 *, \
                                               float *, const Plan &, GlsParams,     \
                                               cudaStream_t);                        \
    template cudaError_t launch_pass2_nfft_t<L>(const DevCurve *, int, int, const float2 *, \
                                                float2 *, const ulonglong2 *, unsigned *, \
                                                const Plan &, cudaStream_t);                       \
    template cudaError_t preload_pass1_t<3, L>();                                  \
    template cudaError_t preload_pass1_t<1, L>();                                  \
    template cudaError_t preload_pass2_t<L>(int);

}  // namespace cuvgls
