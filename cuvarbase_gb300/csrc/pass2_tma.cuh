// Pass 2 of the GLS for rows whose outputs fit in registers.
//
//   k_pass2_gls_reg<L2, ES>  persistent CTAs; a task is R rows of one curve.
//     The rows of its three grids arrive one after the other by TMA and each
//     goes through the two-level row FFT:
//       stage A  one unit (r, i) reads its LA inputs from the arrived tile,
//                transforms them and writes them to the exchange tile;
//       stage B  one thread per (r, qa) reads LB values and transforms them.
//     A thread's outputs q2 = qa + LA qb of the three grids stay in its
//     registers, so the power of those frequencies is evaluated and written
//     without a further pass through shared memory.
//
// What it replaces (a CTA per R rows; the three grids' outputs back to shared
// memory and read again) was held by the L1 data pipe: 75 % busy, of which a
// third was the outputs' way through shared memory and the deconvolution
// table's scattered reads.  2,000 curves of 320 x 400 cells 1.80 -> 1.61 ms,
// 1.585 with the next tile in L2 and two twiddles to a load (now at 54 % issue,
// 54 % of the L1 pipe and of DRAM), 20,000 of 160 x 160 4.11 -> 2.82 ms (the old tile also had two- to four-way bank conflicts).
//   NARROW  sigma >= kNarrowSigma: only the outputs near both ends of a row can
//     be in band; the rest are neither finished nor kept, and grid A is not
//     parked.  400 curves of 1024 x 400 cells at sigma 4 833 -> 774 us (781 with a
//     second tile in flight in the memory that frees, 981 with five CTAs per SM).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "fft.cuh"
#include "gls_math.cuh"
#include "kernels.cuh"

namespace cuvgls {

// ---- mbarrier and TMA ----
__device__ __forceinline__ unsigned smem_addr(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *b) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long *b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)),
                 "r"(bytes)
                 : "memory");
}
// Waits for the phase of the given parity, a bounded number of times; false
// when that ran out.
constexpr int kWaitTries = 1 << 18;  // each suspends for up to some microseconds
template <int TRIES = kWaitTries>
__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned parity) {
    const unsigned a = smem_addr(b);
    for (int k = 0; k < TRIES; ++k) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred p;\n"
            " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z,
                                            unsigned long long *b) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_addr(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_addr(b))
        : "memory");
}

// Orders this thread's own loads and stores of shared memory before the copies
// into the same bytes that another thread issues after the next barrier: the
// copies are the async proxy's, and a barrier alone orders one proxy only.  (2,000
// curves of 320 x 400 cells 3.537 -> 3.553 ms, 1,000 NFFTs 0.941 -> 0.948.)
__device__ __forceinline__ void before_copy() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Asks for the same box in L2, ahead of its load.
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap *map, int x, int y, int z) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(map),
                 "r"(x), "r"(y), "r"(z)
                 : "memory");
}

// Offset of row r in the exchange tile, beside r pitches: it spreads the
// stores of stage A (four columns of four rows per half-warp) and the loads
// of stage B (all rows at one or two qa) over the 16 bank pairs.
template <int R>
__device__ __forceinline__ int row_shift(int r) {
    if constexpr (R == 16) return 4 * (r & 3) + (r >> 2);
    else if constexpr (R == 8) return 4 * (r & 3) + 2 * (r >> 2);
    else return 4 * (r & 3);
}

// P of two frequencies in packed FP32x2 arithmetic (floating mean), as
// gls_from_sums: A, B, C are (re, im) per grid for the frequencies x and y.
struct Fm2 {
    float2 nyw, hw, pn;
    __device__ __forceinline__ Fm2(const DevCurve &cv, float reg)
        : nyw(make_float2(-cv.yw_sum, -cv.yw_sum)),
          hw(make_float2(0.5f * cv.w_sum + reg, 0.5f * cv.w_sum + reg)),
          pn(make_float2(cv.yy_inv, cv.yy_inv)) {}
    __device__ __forceinline__ float2 power(float2 A0, float2 A1, float2 B0, float2 B1, float2 C0,
                                            float2 C1, float2 D) const {
        const float2 half = make_float2(0.5f, 0.5f), mhalf = make_float2(-0.5f, -0.5f);
        const float2 mtwo = make_float2(-2.f, -2.f);
        const float2 YCh = __fmul2_rn(make_float2(A0.x, A1.x), D);
        const float2 YSh = __fmul2_rn(make_float2(A0.y, A1.y), D);
        const float2 C = __fmul2_rn(make_float2(B0.x, B1.x), D);
        const float2 S = __fmul2_rn(make_float2(B0.y, B1.y), D);
        const float2 C2 = __fmul2_rn(make_float2(C0.x, C1.x), D);
        const float2 S2 = __fmul2_rn(make_float2(C0.y, C1.y), D);
        const float2 mC = make_float2(-C.x, -C.y), mS = make_float2(-S.x, -S.y);
        const float2 YC = __ffma2_rn(nyw, C, YCh);
        const float2 YS = __ffma2_rn(nyw, S, YSh);
        const float2 CC = __ffma2_rn(mC, C, __ffma2_rn(half, C2, hw));
        const float2 SS = __ffma2_rn(mS, S, __ffma2_rn(mhalf, C2, hw));
        const float2 CS = __ffma2_rn(mC, S, __fmul2_rn(half, S2));
        const float2 det = __ffma2_rn(make_float2(-CS.x, -CS.y), CS, __fmul2_rn(CC, SS));
        const float2 a = __ffma2_rn(__fmul2_rn(mtwo, YS), CS, __fmul2_rn(YC, SS));
        const float2 num = __ffma2_rn(YC, a, __fmul2_rn(__fmul2_rn(YS, YS), CC));
        const float2 P = __fmul2_rn(
            make_float2(__fdividef(num.x, det.x), __fdividef(num.y, det.y)), pn);
        return make_float2((P.x >= 0.f && !isinf(P.x)) ? P.x : -1.f,
                           (P.y >= 0.f && !isinf(P.y)) ? P.y : -1.f);
    }
};

// (TRIES: the limit of the waits for a tile, which a test lets run out)
template <int L2, bool ES, bool NARROW, int TRIES>
__global__ void __launch_bounds__(pass2_reg_threads(L2), pass2_reg_ctas(L2))
k_pass2_gls_reg(const __grid_constant__ CUtensorMap map, const DevCurve *cvs,
                int n_curves, int first, float *__restrict__ out, const Plan p, const GlsParams gp) {
    constexpr int LA = two_level_la(L2), LB = L2 / LA;
    constexpr int R = pass2_rows(3, L2), NT = pass2_reg_threads(L2);
    constexpr int PITCH = pass2_reg_pitch(L2), TILE = pass2_reg_tile(L2);
    constexpr bool IP = pass2_reg_inplace(L2), PARK = IP && !NARROW;
    constexpr int NB = IP ? 1 : 2;  // tiles in flight
    constexpr int AU = R * LB, UPT = (AU + NT - 1) / NT;  // stage-A units per grid and thread
    // tiles in flight (at the 128 bytes a TMA tile needs: no static shared
    // memory lies before them), exchange tile or parked outputs, barriers
    extern __shared__ __align__(1024) unsigned char sm_tiles[];
    float2 *tiles = reinterpret_cast<float2 *>(sm_tiles), *rest = tiles + NB * TILE;
    unsigned long long *full = reinterpret_cast<unsigned long long *>(tiles + (IP && NARROW ? TILE : pass2_reg_elems(L2)));
    const int tid = threadIdx.x;
    if (p.dependent) pdl_trigger();
    if (smem_addr(tiles) & 127) {  // uniform; a copy there would fault
        if (tid == 0) atomicOr(gp.errflag, 2u);
        return;
    }
    constexpr int lb = 2;
    static_assert(1 << lb == kGlsCols, "blocks of four columns");
    const int G1 = p.G1, G = (int)p.G, nrb = G1 / R;
    const int ntask = n_curves * nrb;
    if (tid == 0) {
        for (int b = 0; b < NB; ++b) mbar_init(&full[b]);
        before_copy();
    }
    __syncthreads();
    if (p.dependent) pdl_wait();  // the intermediate and the descriptors
    cvs = written(cvs);
    // step s: grid s % 3 of this CTA's task s / 3, into tile s % NB
    auto live = [&](int s) { return blockIdx.x + (s / 3) * (int)gridDim.x < ntask; };
    // (and the tile after it brought to L2, so that its load is short: 2,000
    // curves of 320 x 400 cells 1630 -> 1607 us; two tiles ahead 1655, three 2012)
    auto issue = [&](int s) {
        if (!live(s)) return;
        const int t = blockIdx.x + (s / 3) * (int)gridDim.x, c = t / nrb, rb = t - c * nrb;
        mbar_expect(&full[s % NB], R * L2 * 8);
        tma_load_3d(tiles + (s % NB) * TILE, &map, rb * R * 2 * kGlsCols, 0, (first + c) * 3 + s % 3,
                    &full[s % NB]);
        if (!live(s + 1)) return;
        const int u = blockIdx.x + ((s + 1) / 3) * (int)gridDim.x, d = u / nrb;
        tma_prefetch_3d(&map, (u - d * nrb) * R * 2 * kGlsCols, 0, (first + d) * 3 + (s + 1) % 3);
    };
    if (tid == 0)
        for (int b = 0; b < NB; ++b) issue(b);
    const int r = tid % R, qa = tid / R;  // stage-B unit of this thread
    const bool act = NT == R * LA || tid < R * LA;
    int s = 0;
    for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
        const int ci = t / nrb, rb = t - ci * nrb;
        float2 ya[LB], yb[LB], yc[LB];
#pragma unroll
        for (int g = 0; g < 3; ++g, ++s) {
            const bool ok = mbar_wait<TRIES>(&full[s % NB], (s / NB) & 1);
            float2 *in = tiles + (s % NB) * TILE;
            float2 *ex = IP ? in : rest;
            // stage A: unit u = (ih, r, c) reads in[u + k AU], i.e. elements
            // i + LB k, i = ih B + c, of row r
            auto load = [&](float2 (&x)[LA], int u) {
#pragma unroll
                for (int k = 0; k < LA; ++k) x[k] = in[u + k * AU];
                fft2_stage_a_regs<L2>(x, p.st2, ((u >> lb) / R << lb) + (u & ((1 << lb) - 1)));
            };
            auto store = [&](const float2 (&x)[LA], int u) {
                const int i = ((u >> lb) / R << lb) + (u & ((1 << lb) - 1)), ra = (u >> lb) % R;
                float2 *d = ex + ra * PITCH + row_shift<R>(ra) + i;
#pragma unroll
                for (int q = 0; q < LA; ++q) d[(LB + 1) * q] = x[q];
            };
            float2 x[IP ? UPT : 1][LA];
            if constexpr (IP) {  // all units read before the tile is written
#pragma unroll
                for (int v = 0; v < UPT; ++v)
                    if (AU % NT == 0 || tid + v * NT < AU) load(x[v], tid + v * NT);
            } else {
#pragma unroll 1
                for (int u = tid; u < AU; u += NT) {
                    load(x[0], u);
                    store(x[0], u);
                }
            }
            // a copy never came: all threads leave, after a second bounded wait
            // for the copies in flight
            if (__syncthreads_or(!ok)) {
                if (tid == 0) {
                    atomicOr(gp.errflag, 2u);
                    for (int k = s; k < s + NB; ++k)
                        if (live(k)) mbar_wait(&full[k % NB], (k / NB) & 1);
                }
                __syncthreads();
                return;
            }
            if constexpr (IP) {
#pragma unroll
                for (int v = 0; v < UPT; ++v)
                    if (AU % NT == 0 || tid + v * NT < AU) store(x[v], tid + v * NT);
                __syncthreads();
            } else {
                if (tid == 0) issue(s + NB);  // into the tile just read
            }
            float2 *y = g == 0 ? ya : g == 1 ? yb : yc;
            if (act) {
                const float2 *e = ex + r * PITCH + row_shift<R>(r) + (LB + 1) * qa;
#pragma unroll
                for (int i = 0; i < LB; ++i) y[i] = e[i];
            }
            if constexpr (IP) {
                before_copy();
                __syncthreads();  // all read: the tile is free
                if (tid == 0) issue(s + NB);
            }
            if (act) RegDFT<LB>::run(y);
            if constexpr (PARK) {
                if (g == 0) {  // grid A parked, read back by the same thread
#pragma unroll
                    for (int qb = 0; qb < LB; ++qb) rest[qb * NT + tid] = ya[qb];
                }
            }
            if constexpr (!IP) __syncthreads();  // the exchange tile is written next
        }
        // power of the outputs q2 = qa + LA qb
        const DevCurve cv = cvs[ci];
        const int nf = cv.nf, h = nf / 2, lo_end = nf - h, hi_start = G - h;
        const bool write = gp.best == nullptr || out != nullptr;
        float *o = out + cv.out_off + h;
        const int q0 = rb * R + r + G1 * qa;
        const float *drow = ES ? p.drow + ((long long)rb * L2 + qa) * R + r : nullptr;
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
        // two frequencies at a time; f(qb, ka, kb, ina, inb, D) for each pair
        // with an output in band
        auto pairs = [&](auto f) {
#pragma unroll
            for (int qb = 0; qb < LB; qb += 2) {
                // (no band reaches the middle fifth of the grid: sigma >= 1.25)
                if (5 * qb >= 2 * LB && 5 * (qb + 2) <= 3 * LB) continue;
                if (NARROW && !narrow_pair(L2, qb)) continue;
                const int qA = q0 + G1 * LA * qb, qB = qA + G1 * LA;
                const bool ina = qA < lo_end || qA >= hi_start;
                const bool inb = qB < lo_end || qB >= hi_start;
                if (!ina && !inb) continue;
                if constexpr (PARK) {
                    ya[qb] = rest[qb * NT + tid];
                    ya[qb + 1] = rest[(qb + 1) * NT + tid];
                }
                const int ka = qA < lo_end ? qA : qA - G, kb = qB < lo_end ? qB : qB - G;
                float2 D;
                if constexpr (ES)
                    D = make_float2(__ldg(drow + LA * R * qb), __ldg(drow + LA * R * (qb + 1)));
                else
                    D = make_float2(win_deconv<false>(ka, p), win_deconv<false>(kb, p));
                f(qb, ka, kb, ina, inb, D);
            }
        };
        if (act && gp.mode == 1) {
            pairs([&](int qb, int ka, int kb, bool ina, bool inb, float2 D) {
                const float2 P = fm.power(ya[qb], ya[qb + 1], yb[qb], yb[qb + 1], yc[qb],
                                          yc[qb + 1], D);
                if (ina) emit(P.x, ka);
                if (inb) emit(P.y, kb);
            });
        } else if (act) {
            auto one = [&](float2 A, float2 B, float2 C, float D) {
                return gls_from_sums<float>(A.x * D, A.y * D, B.x * D, B.y * D, C.x * D, C.y * D,
                                            gp.mode, gp.reg, cv.w_sum, cv.yw_sum, cv.ybar,
                                            cv.yy_inv);
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
}

// Adjoint NFFT, one grid: the same row transform, in place; a thread's outputs
// are deconvolved, given the phase of the absolute time origin and written.  The phase of output k' is the product of that of
// the thread's first output and one of LB steps per curve, each from an exact
// fraction of a turn: a product instead of a sincospi per output, which held
// the kernel at 68 % issue (half of it integer and conversion instructions).
// 1,000 curves of 512 x 400 cells 0.797 -> 0.431 ms (2.4 GB moved: 0.36 ms at
// the measured copy rate).
template <int L2, bool ES, int TRIES>
__global__ void __launch_bounds__(pass2_reg_threads(L2), kNfftRegCtas)
k_pass2_nfft_reg(const __grid_constant__ CUtensorMap map, const DevCurve *cvs,
                 int n_curves, int first, float2 *__restrict__ out,
                 const ulonglong2 *aux, unsigned *__restrict__ errflag, const Plan p) {
    constexpr int LA = two_level_la(L2), LB = L2 / LA;
    constexpr int R = pass2_rows(1, L2), NT = pass2_reg_threads(L2);
    constexpr int PITCH = pass2_reg_pitch(L2), TILE = pass2_reg_exch(L2);
    constexpr int AU = R * LB, UPT = (AU + NT - 1) / NT;  // stage-A units
    extern __shared__ __align__(1024) unsigned char sm_tiles[];
    float2 *in = reinterpret_cast<float2 *>(sm_tiles), *step = in + TILE;
    unsigned long long *full = reinterpret_cast<unsigned long long *>(in + nfft_reg_elems(L2));
    const int tid = threadIdx.x;
    if (p.dependent) pdl_trigger();
    if (smem_addr(in) & 127) {  // uniform; a copy there would fault
        if (tid == 0) atomicOr(errflag, 2u);
        return;
    }
    const int G1 = p.G1, G = (int)p.G, nrb = G1 / R;
    // stage-A unit u = (ih, r, c): elements i + LB k, i = 4 ih + c, of row r
    static_assert(LB % 4 == 0, "units of four columns; two LB are whole blocks of kNfftCols");
    auto unit = [](int u, int &i, int &ra) {
        ra = (u >> 2) % R;
        i = (u >> 2) / R * 4 + (u & 3);
    };
    const int ntask = n_curves * nrb;
    if (tid == 0) {
        mbar_init(full);
        before_copy();
    }
    __syncthreads();
    if (p.dependent) pdl_wait();  // the intermediate and the descriptors
    cvs = written(cvs);
    aux = written(aux);
    auto live = [&](int s) { return blockIdx.x + s * (int)gridDim.x < ntask; };
    auto issue = [&](int s) {  // this CTA's task s
        if (!live(s)) return;
        const int t = blockIdx.x + s * (int)gridDim.x, c = t / nrb, rb = t - c * nrb;
        mbar_expect(full, R * L2 * 8);
        tma_load_3d(in, &map, rb * R * 2 * kNfftCols, 0, first + c, full);
    };
    if (tid == 0) issue(0);
    const int r = tid % R, qa = tid / R;  // stage-B unit of this thread
    const bool act = NT == R * LA || tid < R * LA;
    for (int s = 0; live(s); ++s) {
        const int t = blockIdx.x + s * (int)gridDim.x, ci = t / nrb, rb = t - ci * nrb;
        const DevCurve cv = cvs[ci];
        const ulonglong2 ax = aux[cv.aux];
        const bool ok = mbar_wait<TRIES>(full, s & 1);
        float2 x[UPT][LA];
#pragma unroll
        for (int v = 0; v < UPT; ++v) {
            const int u = tid + v * NT;
            if (AU % NT == 0 || u < AU) {
                int i, ra;
                unit(u, i, ra);
                // element l of row r lies at ((l / 8) R + r) 8 + l % 8
                const int b0 = ((i >> 3) * R + ra) * 8 + (i & 7);
                const int b1 = (((i + LB) >> 3) * R + ra) * 8 + ((i + LB) & 7);
#pragma unroll
                for (int k = 0; k < LA; ++k) x[v][k] = in[(k & 1 ? b1 : b0) + (k >> 1) * 2 * LB * R];
                fft2_stage_a_regs<L2>(x[v], p.st2, i);
            }
        }
        if (__syncthreads_or(!ok)) {  // as in k_pass2_gls_reg
            if (tid == 0) {
                atomicOr(errflag, 2u);
                mbar_wait(full, s & 1);
            }
            __syncthreads();
            return;
        }
#pragma unroll
        for (int v = 0; v < UPT; ++v) {
            const int u = tid + v * NT;
            if (AU % NT == 0 || u < AU) {
                int i, ra;
                unit(u, i, ra);
                float2 *d = in + ra * PITCH + row_shift<R>(ra) + i;
#pragma unroll
                for (int q = 0; q < LA; ++q) d[(LB + 1) * q] = x[v][q];
            }
        }
        // phases of the steps qb: those of the upper half belong to k' = q - G
        if (tid < LB)
            step[tid] = turn_phasor(
                (unsigned long long)((long long)G1 * LA * tid - (2 * tid < LB ? 0 : G)) * ax.y);
        __syncthreads();
        float2 y[LB];
        const float2 *e = in + r * PITCH + row_shift<R>(r) + (LB + 1) * qa;
        if (act) {
#pragma unroll
            for (int i = 0; i < LB; ++i) y[i] = e[i];
        }
        before_copy();
        __syncthreads();  // all read: the tile is free
        if (tid == 0) issue(s + 1);
        const int nf = cv.nf, h = nf / 2, lo_end = nf - h, hi_start = G - h;
        const int q0 = rb * R + r + G1 * qa;
        if (act) {
            RegDFT<LB>::run(y);
            float2 *o = out + cv.out_off + h;
            const float *drow = ES ? p.drow + ((long long)rb * L2 + qa) * R + r : nullptr;
            const float2 ph0 = turn_phasor(ax.x + (unsigned long long)q0 * ax.y);
#pragma unroll
            for (int qb = 0; qb < LB; ++qb) {
                // (no band reaches the middle fifth of the grid: sigma >= 1.25)
                if (5 * qb >= 2 * LB && 5 * (qb + 1) <= 3 * LB) continue;
                const int q = q0 + G1 * LA * qb;
                const int k = 2 * qb < LB ? q : q - G;
                if (2 * qb < LB ? q >= lo_end : q < hi_start) continue;
                const float D = ES ? __ldg(drow + LA * R * qb) : win_deconv<false>(k, p);
                o[k] = cmul(cscale(y[qb], D), cmul(ph0, step[qb]));
            }
        }
        // (the next task's steps are written two barriers on)
    }
}

// Tensor map of a chunk's intermediate for tiles of R rows of one grid:
// (G1 B complex values of a column block, column blocks, curve x grid).
cudaError_t pass2_map(CUtensorMap &map, const float2 *inter, const Plan &p, int grids, int R);

// CTAs of a persistent kernel that fit the device at once, kept per kernel
// and device in `slots` (0: not asked yet).
template <typename K>
cudaError_t resident_ctas(K kernel, int threads, int smem, int (&slots)[64]) {
    int dev = 0, n = 0, sms = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (slots[dev]) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem);
    if (e == cudaSuccess) slots[dev] = (n > 0 ? n : 1) * sms;
    return e;
}

template <int L2, bool ES, int TRIES = kWaitTries>
cudaError_t launch_nfft_reg_t(const DevCurve *cv, int n_curves, int first, const float2 *inter,
                              float2 *out, const ulonglong2 *aux, unsigned *errflag, const Plan &p,
                              cudaStream_t s) {
    static int slots[64] = {0};  // resident CTAs, per instantiation and device
    constexpr int NT = pass2_reg_threads(L2), R = pass2_rows(1, L2);
    const int smem = (int)pass2_smem(1, L2);
    cudaError_t e = resident_ctas(k_pass2_nfft_reg<L2, ES, TRIES>, NT, smem, slots);
    if (e != cudaSuccess) return e;
    int dev = 0;
    cudaGetDevice(&dev);
    CUtensorMap map;
    e = pass2_map(map, inter, p, first + n_curves, R);
    if (e != cudaSuccess) return e;
    const long long tasks = (long long)n_curves * (p.G1 / R);
    if (tasks > 0x3fffffffLL || p.B != kNfftCols) return cudaErrorInvalidValue;
    Plan q = p;
    q.dependent = small_launch(tasks);
    return launch_pdl(k_pass2_nfft_reg<L2, ES, TRIES>, q.dependent,
                      dim3((int)(tasks < slots[dev] ? tasks : slots[dev])), NT, smem, s, map, cv,
                      n_curves, first, out, aux, errflag, q);
}

template <int L2, bool ES, bool NARROW, int TRIES = kWaitTries>
cudaError_t launch_pass2_reg_t(const DevCurve *cv, int n_curves, int first, const float2 *inter,
                               float *out, const Plan &p, GlsParams g, cudaStream_t s) {
    static int slots[64] = {0};  // resident CTAs, per instantiation and device
    constexpr int NT = pass2_reg_threads(L2), R = pass2_rows(3, L2);
    const int smem = NARROW && pass2_reg_inplace(L2) ? (pass2_reg_tile(L2) + 2) * 8 : (int)pass2_smem(3, L2);
    cudaError_t e = resident_ctas(k_pass2_gls_reg<L2, ES, NARROW, TRIES>, NT, smem, slots);
    if (e != cudaSuccess) return e;
    int dev = 0;
    cudaGetDevice(&dev);
    CUtensorMap map;
    e = pass2_map(map, inter, p, 3 * (first + n_curves), R);
    if (e != cudaSuccess) return e;
    const long long tasks = (long long)n_curves * (p.G1 / R);
    if (tasks > 0x3fffffffLL || p.B != kGlsCols) return cudaErrorInvalidValue;
    Plan q = p;
    q.dependent = small_launch(tasks);
    return launch_pdl(k_pass2_gls_reg<L2, ES, NARROW, TRIES>, q.dependent,
                      dim3((int)(tasks < slots[dev] ? tasks : slots[dev])), NT, smem, s, map, cv,
                      n_curves, first, out, q, g);
}

}  // namespace cuvgls
