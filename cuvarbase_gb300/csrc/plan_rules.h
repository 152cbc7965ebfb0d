// Compile-time rules shared by the host planner and the kernel templates:
// the menu of transform lengths, the radix sequence of each length, the
// tile shapes (columns B per pass-1 CTA, rows R per pass-2 CTA), the thread
// counts and the shared-memory footprints.  Host and device evaluate the
// same constexpr functions, so a plan the host picks always has a kernel.
#pragma once

#ifdef __CUDACC__
#define CUVGLS_HD __host__ __device__
#else
#define CUVGLS_HD
#endif

namespace cuvgls {

// Transform lengths with a compiled kernel: 2^a 5^c, multiples of 16.
constexpr int kLens[] = {16, 32, 64, 80, 128, 160, 256, 320, 400, 512,
                         640, 800, 1024, 1280, 1600, 2048};
constexpr int kNumLens = sizeof(kLens) / sizeof(kLens[0]);
// Row lengths (pass 2): the same and 4096.  A 4096-row grid (G up to
// 2048 x 4096) halves the sub-bands of very wide bands, and with them the
// spreading, which every sub-band repeats over all points of the curve; a
// 4096-long column tile would leave one column per pass-1 CTA and double the
// CTAs each record is spread into.
constexpr int kRowLens[] = {16, 32, 64, 80, 128, 160, 256, 320, 400, 512,
                            640, 800, 1024, 1280, 1600, 2048, 4096};
constexpr int kNumRowLens = sizeof(kRowLens) / sizeof(kRowLens[0]);

// Measured cost of the pass kernels on GB300, in ps per grid cell per curve,
// by transform length: pass 1 by column length G1 (kLens order), pass 2 by
// row length G2 (kRowLens order).  From 10,000-curve batches of curves with
// N log-uniform in [50, 5000] on 128,000- to 1,310,720-cell grids (ES window,
// m = 5); lengths marked * were not measured and are interpolated.  (The
// 320-long columns have since run 6 CTAs per SM instead of 5, 6 % faster;
// their entry is kept, since per cell pass 1 also depends on the points per
// curve and 6.1 would make 320 x 80 beat 160 x 160 at nf = 2e4, measured 8 %
// slower on these curves.)  Pass 1
// also pays per point (~0.23 ns per point of the curve, whatever the shape),
// which the shape choice can leave out.  (The kernels have become faster since,
// unevenly: rows of 400 6.3 ps, 160 5.6, 512 7.0, 640 8.4, 800 8.8, 1,024 10,
// 1,280 11, 4,096 about 13, columns of 2,048 about 10.  The entries are kept, so
// that a number of frequencies keeps its grid.)
constexpr float kPass1PsPerCell[] = {18.f /*16*/, 8.f /*32*/, 7.5f /*64 **/, 8.6f /*80*/,
                                     7.f /*128 **/, 6.4f /*160*/, 7.1f /*256*/, 6.5f /*320*/,
                                     6.3f /*400*/, 6.8f /*512*/, 6.f /*640*/, 6.8f /*800*/,
                                     6.5f /*1024*/, 15.2f /*1280*/, 20.5f /*1600*/,
                                     22.f /*2048 **/};
constexpr float kPass2PsPerCell[] = {6.7f /*16*/, 6.2f /*32*/, 8.5f /*64*/, 7.9f /*80*/,
                                     8.5f /*128 **/, 7.9f /*160*/, 9.3f /*256*/, 9.3f /*320*/,
                                     7.f /*400*/, 9.9f /*512*/, 8.4f /*640*/, 9.6f /*800*/,
                                     12.f /*1024*/, 20.f /*1280*/, 25.5f /*1600*/,
                                     28.f /*2048 **/, 30.f /*4096 **/};
static_assert(sizeof(kPass1PsPerCell) / sizeof(float) == sizeof(kLens) / sizeof(int),
              "one pass-1 cost per column length");
static_assert(sizeof(kPass2PsPerCell) / sizeof(float) == sizeof(kRowLens) / sizeof(int),
              "one pass-2 cost per row length");

// Elements a thread holds in registers during one FFT stage (target).
constexpr int kEPT = 16;
constexpr int kMaxThreads = 1024;
constexpr int kMaxTile = kEPT * kMaxThreads;  // complex elements per CTA
constexpr int kSmemLimit = 227 * 1024;
constexpr int kMaxFac = 12;

struct FacList {
    int n;
    int r[kMaxFac];
};

// Radix sequence of L = 2^a 5^c: the radix-5 stages first, then 16s, then
// the remaining power of two (2, 4, 8 or 16); 1600 is 20 x 20 x 4.
CUVGLS_HD constexpr FacList fft_factors(int L) {
    FacList f{0, {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0}};
    int x = L;
    if (x == 1600) { f.r[f.n++] = 20; f.r[f.n++] = 20; x = 4; }
    while (x % 5 == 0) { f.r[f.n++] = 5; x /= 5; }
    while (x % 3 == 0) { f.r[f.n++] = 3; x /= 3; }
    while (x % 16 == 0 && x > 16) { f.r[f.n++] = 16; x /= 16; }
    if (x > 1) f.r[f.n++] = x;
    return f;
}

CUVGLS_HD constexpr bool len_ok(int L) {
    FacList f = fft_factors(L);
    int p = 1;
    for (int i = 0; i < f.n; ++i) {
        int r = f.r[i];
        if (r != 2 && r != 3 && r != 4 && r != 5 && r != 8 && r != 16 && r != 20) return false;
        p *= r;
    }
    return p == L;
}

// Product of the radices before stage s (the Stockham span Ns).
CUVGLS_HD constexpr int fft_ns(int L, int s) {
    FacList f = fft_factors(L);
    int p = 1;
    for (int i = 0; i < s; ++i) p *= f.r[i];
    return p;
}

// Stage twiddles are stored per stage as [r = 1..R-1][k = 0..Ns-1]; stage 0
// (Ns = 1) needs none.  Offset of stage s and the total table length.
CUVGLS_HD constexpr int stage_tw_offset(int L, int s) {
    FacList f = fft_factors(L);
    int off = 0, ns = 1;
    for (int i = 0; i < s; ++i) {
        if (ns > 1) off += ns * (f.r[i] - 1);
        ns *= f.r[i];
    }
    return off;
}
CUVGLS_HD constexpr int stage_tw_total(int L) {
    return stage_tw_offset(L, fft_factors(L).n);
}

// Padded position of element i along a transform: one slot after every 16
// elements, which spreads the strided Stockham writes over the banks.
CUVGLS_HD constexpr int padded(int i) { return i + (i >> 4); }
CUVGLS_HD constexpr int padded_len(int L) { return L + (L >> 4); }

// Two-level split L = La * Lb with both factors register-DFT sizes (<= 32);
// La is the factor closest to sqrt(L) from below, unless that leaves Lb not
// a multiple of 4: then the split with Lb a multiple of 4 and La closest to
// sqrt(L) (so that a pass-2 stage A can read whole 4-column blocks; this
// only changes 80 = 10 x 8).  0 when there is none.
CUVGLS_HD constexpr bool reg_dft_ok(int r) {
    return r == 4 || r == 5 || r == 8 || r == 10 || r == 16 || r == 20 || r == 25 ||
           r == 32;
}
CUVGLS_HD constexpr int two_level_la(int L) {
    int best = 0;
    for (int la = 4; la <= 32; ++la)
        if (L % la == 0 && reg_dft_ok(la) && reg_dft_ok(L / la) && la * la <= L) best = la;
    if (best == 0 || (L / best) % 4 == 0) return best;
    int alt = 0;
    long long dist = 0;
    for (int la = 4; la <= 32; ++la)
        if (L % la == 0 && reg_dft_ok(la) && reg_dft_ok(L / la) && (L / la) % 4 == 0) {
            const long long d = (long long)la * la > L ? (long long)la * la - L
                                                       : L - (long long)la * la;
            if (alt == 0 || d < dist) { alt = la; dist = d; }
        }
    return alt ? alt : best;
}

// Position of element n of a length-L tile vector: two-level lengths pad one
// slot per Lb elements, the others one per 16.
CUVGLS_HD constexpr int phys2_len(int L) {
    return two_level_la(L) ? L + L / (L / two_level_la(L)) : padded_len(L);
}

CUVGLS_HD constexpr int threads_for(int elems) {
    return elems <= kEPT * 128 ? 128
         : elems <= kEPT * 256 ? 256
         : elems <= kEPT * 512 ? 512 : 1024;
}

template <int L>
CUVGLS_HD constexpr int phys2(int n) {
    if constexpr (two_level_la(L) > 0) {
        constexpr int LB = L / two_level_la(L);
        return n + n / LB;
    } else {
        return padded(n);
    }
}

// Table an FFT of length L reads: the stage-A twiddles of a two-level length,
// [qa][i] or, with pairs, those of 2 p and 2 p + 1 side by side as [p][i][2]
// (one 16-byte load: pass 1 of 2,000 curves of 320 x 400 cells 1750 -> 1733 us,
// pass 2 1607 -> 1587; columns of 1,024, where La is 32, would lose 1 %), the
// Stockham stage twiddles otherwise; an even number of entries.
CUVGLS_HD constexpr bool tw_pairs(int L) { return two_level_la(L) <= 20; }
CUVGLS_HD constexpr int fft_table_len(int L) {
    const int la = two_level_la(L);
    if (la == 0) return (stage_tw_total(L) + 1) / 2 * 2;
    return tw_pairs(L) ? (la + 1) / 2 * 2 * (L / la) : L;
}
CUVGLS_HD constexpr int tile_len(int L) { return phys2_len(L); }
// Row stride of a pass-2 tile.
CUVGLS_HD constexpr int row_stride(int L) { return tile_len(L); }
CUVGLS_HD constexpr int round32(int x) { return (x + 31) / 32 * 32; }

// Threads for V vectors of length L: one per stage-B unit of a two-level
// length (at least 128), the Stockham rule otherwise.
CUVGLS_HD constexpr int fft_threads(int V, int L) {
    return two_level_la(L) ? (round32(V * two_level_la(L)) < 128 ? 128
                                                                   : round32(V * two_level_la(L)))
                           : threads_for(V * L);
}
CUVGLS_HD constexpr bool tile_fits(int V, int L) {
    return two_level_la(L) ? V * two_level_la(L) <= kMaxThreads : V * L <= kMaxTile;
}

// Whether the columns of this length go through k_pass1_long (the three grids
// of a column block in CTAs of their own): those without a two-level split,
// in three levels F0, F1, F2, the Stockham radices in reverse.
CUVGLS_HD constexpr bool pass1_long(int ng, int L1) { return ng == 3 && two_level_la(L1) == 0; }
CUVGLS_HD constexpr int long_fac(int L1, int level) { return fft_factors(L1).r[2 - level]; }
constexpr int kLongCols = 4;

// Columns per pass-1 CTA for ng grids of column length L1.
CUVGLS_HD constexpr int pass1_cols(int ng, int L1) {
    if (pass1_long(ng, L1)) return kLongCols;
    int b = (ng == 1) ? 8 : 4;
    while (b > 2 && !tile_fits(ng * b, L1)) b /= 2;
    return b;
}

// Whether the rows of this length keep their outputs in registers
// (k_pass2_gls_reg, k_pass2_nfft_reg): a two-level split with at most 20
// outputs of each grid per thread.
CUVGLS_HD constexpr bool pass2_reg(int ng, int L2) {
    return two_level_la(L2) > 0 && L2 / two_level_la(L2) <= 20;
}

// Whether the GLS rows of this length go through k_pass2_gls_cube: three
// levels of 16, one row of one curve per CTA.
CUVGLS_HD constexpr bool pass2_cube(int ng, int L2) { return ng == 3 && L2 == 4096; }
constexpr int kCubePitch = 257;   // of its exchange tile: 16 planes of 256 elements

// Whether the GLS rows of this length go through k_pass2_gls_deep: three levels
// F0, F1 and F2 = 8 (the outputs of each grid per thread); the exchange tile's
// slot of element j + 8 k of plane q0 is q0 P0 + 9 k + j.
CUVGLS_HD constexpr int deep_fac(int L2, int level) {
    if (level == 2) return 8;
    const int f0 = L2 == 512 ? 8 : L2 == 640 || L2 == 800 ? 10 : L2 == 1600 ? 20 : 16;
    return level == 0 ? f0 : L2 / 8 / f0;
}
CUVGLS_HD constexpr bool pass2_deep(int ng, int L2) {
    return ng == 3 && !pass2_reg(3, L2) && !pass2_cube(3, L2);
}
CUVGLS_HD constexpr int deep_rows(int L2) { return L2 <= 800 ? 4 : 2; }
CUVGLS_HD constexpr int deep_threads(int L2) { return (deep_rows(L2) * L2 / 8 + 31) / 32 * 32; }
// CTAs per SM: as many as the registers of three grids' outputs and one
// butterfly allow (measured: 512 8.6 ps per cell with two, 7.1 with three; 1,024
// 10.7 and 10.1; 640, 800 and 1,280 are slower with three).
CUVGLS_HD constexpr int deep_ctas(int L2) {
    return L2 == 512 || L2 == 1024 ? 3 : L2 == 2048 ? 1 : 2;
}
// pitches that keep every access free of bank conflicts: planes 8 (mod 16)
// apart, rows 4 (of four) or 8 (of two)
CUVGLS_HD constexpr int deep_plane(int L2) { return (9 * deep_fac(L2, 1) + 7) / 16 * 16 + 8; }
CUVGLS_HD constexpr int deep_pitch(int L2) {
    return (deep_fac(L2, 0) * deep_plane(L2) + 15) / 16 * 16 + 16 / deep_rows(L2);
}
// Entries of the row table: exp(2 pi i q0 i / L2) as [q0][i], then
// exp(2 pi i q1 j / (8 F1)) as [q1][j].
CUVGLS_HD constexpr int deep_table_len(int L2) { return L2 + L2 / deep_fac(L2, 0); }

CUVGLS_HD constexpr int row_table_len(int ng, int L2) {
    return pass2_deep(ng, L2) ? deep_table_len(L2) : fft_table_len(L2);
}

// Rows per pass-2 CTA for ng grids of row length L2: 16 for short register
// rows, so that a CTA still transforms a few thousand elements; 8 for the other
// register rows (32-byte runs of powers); 4 or 2 for the longer GLS rows, 1 for
// those of 4,096; for the one-grid rows beyond, 16 or as many as fit the tile.
CUVGLS_HD constexpr int pass2_rows(int ng, int L2) {
    if (pass2_reg(ng, L2)) return L2 <= 160 ? 16 : 8;
    if (pass2_deep(ng, L2)) return deep_rows(L2);
    if (pass2_cube(ng, L2)) return 1;
    int r = 16;
    while (r > 2 && !tile_fits(ng * r, L2)) r /= 2;
    return r;
}

CUVGLS_HD constexpr int pass1_threads(int ng, int L1) {
    // (one thread per level-2 butterfly)
    if (pass1_long(ng, L1)) return kLongCols * L1 / long_fac(L1, 1);
    return fft_threads(ng * pass1_cols(ng, L1), L1);
}
// k_pass2_gls_reg: a thread per stage-B unit; row pitch of the exchange tile
// (room for row_shift).  Rows above 160 are exchanged in place, in the one
// tile a grid arrives in, and park grid A's outputs in shared memory: 96
// registers and four CTAs per SM, which matters more there than copies ahead
// of their use (400: 1.66 ms per 2,000 curves of 320 x 400 cells; 1.77 with
// two tiles and three CTAs, 2.02 with two tiles, an exchange tile of their own
// and two CTAs).  Shorter rows have a tile to exchange in and two in flight
// (160: 2.89 ms per 20,000 curves of 160 x 160 cells; 3.16 in place).
CUVGLS_HD constexpr int pass2_reg_threads(int L2) {
    return round32(pass2_rows(3, L2) * two_level_la(L2));
}
CUVGLS_HD constexpr int pass2_reg_pitch(int L2) { return (tile_len(L2) + 11 + 15) / 16 * 16; }
CUVGLS_HD constexpr bool pass2_reg_inplace(int L2) { return L2 > 160; }
CUVGLS_HD constexpr int pass2_reg_ctas(int L2) { return pass2_reg_inplace(L2) ? 4 : 3; }
// elements of the exchange tile and of a tile in flight
CUVGLS_HD constexpr int pass2_reg_exch(int L2) {
    return pass2_rows(3, L2) * pass2_reg_pitch(L2) + 16;
}
CUVGLS_HD constexpr int pass2_reg_tile(int L2) {
    return pass2_reg_inplace(L2) ? pass2_reg_exch(L2) : pass2_rows(3, L2) * L2;
}
// Upsampling from which the band reaches only the first and the last 5/34 of the
// rows' outputs (nf <= G / 3.4): there k_pass2_gls_reg keeps the outputs qb of
// those (in pairs) and nothing else.
constexpr double kNarrowSigma = 3.4;
CUVGLS_HD constexpr bool narrow_pair(int L2, int qb) {  // of outputs qb, qb + 1
    const int la = two_level_la(L2), reach = 5 * L2 / 34 + 1;
    return qb * la <= reach || (qb + 2) * la > L2 - reach - 1;
}
// k_pass2_nfft_reg: in place in one tile, four CTAs per SM (1,000 curves of
// 512 x 400 cells 0.431 ms; 0.442 with a tile ahead, 0.452 with five CTAs).
// (columns per pass-1 block of every one-grid plan, and of every GLS plan)
constexpr int kNfftCols = 8, kGlsCols = 4;
CUVGLS_HD constexpr bool cols_ok() {
    for (int l : kLens)
        if (pass1_cols(1, l) != kNfftCols || pass1_cols(3, l) != kGlsCols) return false;
    return true;
}
static_assert(cols_ok(), "pass 2 reads blocks of eight and of four columns");
constexpr int kNfftRegCtas = 4;
CUVGLS_HD constexpr int nfft_reg_elems(int L2) {
    return pass2_reg_exch(L2) + L2 / two_level_la(L2);
}
// elements of shared memory before the barriers
CUVGLS_HD constexpr int pass2_reg_elems(int L2) {
    return pass2_reg_inplace(L2)
               ? pass2_reg_tile(L2) + L2 / two_level_la(L2) * pass2_reg_threads(L2)
               : 2 * pass2_reg_tile(L2) + pass2_reg_exch(L2);
}

CUVGLS_HD constexpr int pass2_threads(int ng, int L2) {
    return fft_threads(ng * pass2_rows(ng, L2), L2);
}

// Shared memory (bytes) of a pass-1 CTA: ng padded column tiles (and the
// Stockham twiddles for lengths without a two-level split), then the staged
// records (packed row/column, offset, two complex values; 24 bytes each).
constexpr int kStageRecBytes = 24;

CUVGLS_HD constexpr long long pass1_tile_bytes(int ng, int L1) {
    // two-level lengths read their FFT table through the read-only cache;
    // Stockham lengths stage it in shared memory
    return (long long)(ng * tile_len(L1) * pass1_cols(ng, L1) +
                       (two_level_la(L1) ? 0 : fft_table_len(L1))) * 8;
}

// Records a pass-1 CTA stages per round: 256, or, for the 1024-thread CTAs
// of the long Stockham columns of one grid (one CTA per SM), as many as fit (in steps of
// 256, up to 4096) beside the row counts and the row-sorted record list of
// the gather spreading, so that a dense curve (tens of thousands of records
// per column block) takes a few rounds rather than one barrier pair per 256
// records.
CUVGLS_HD constexpr bool pass1_gather(int ng, int L1) { return pass1_threads(ng, L1) == 1024; }

// Gather spreading's extra shared memory: L1 + 1 row counts, one record
// index per staged record, 32 warp sums of the block scan.
CUVGLS_HD constexpr long long pass1_gather_bytes(int L1, int recs) {
    return (long long)(L1 + 1 + recs + 32) * 4;
}

// Row-residue occupancy flags of the sparse spreading: one byte per (record
// kind, residue i < Lb) of the two-level column FFT, which lets stage A skip
// the all-zero units.
constexpr int kOccBytes = 64;

// CTAs per SM that `bytes` of shared memory per CTA allow (228 KB per SM,
// 1 KB of it reserved per CTA).
CUVGLS_HD constexpr int smem_ctas(long long bytes) { return (int)(233472 / (bytes + 1024)); }

// Registers a thread of the pass-1 kernels needs without spilling (56-60
// across the lengths).
constexpr int kPass1Regs = 56;

// Whether staging 192 records per round instead of 256 fits one more pass-1
// CTA per SM of the three GLS grids, within the register budget of
// kPass1Regs per thread: on the 320-long columns (192 threads) 6 CTAs per SM
// instead of 5, pass 1 of the bench workload 9.62 -> 9.08 ms.  (Only the
// three-grid tiles, where it was measured; the one-grid NFFT tiles keep 256.)
CUVGLS_HD constexpr bool pass1_small_stage(int ng, int L1) {
    return ng == 3 && !pass1_gather(ng, L1) &&
           smem_ctas(pass1_tile_bytes(ng, L1) + kOccBytes + 192LL * kStageRecBytes) >
               smem_ctas(pass1_tile_bytes(ng, L1) + kOccBytes + 256LL * kStageRecBytes) &&
           65536 / (pass1_threads(ng, L1) *
                    smem_ctas(pass1_tile_bytes(ng, L1) + kOccBytes + 192LL * kStageRecBytes)) >=
               kPass1Regs;
}

// CTAs per SM a pass-1 kernel is compiled to keep resident (its launch
// bound): the small-stage count, else 1 (no register cap).
CUVGLS_HD constexpr int pass1_min_ctas(int ng, int L1) {
    return pass1_small_stage(ng, L1)
               ? smem_ctas(pass1_tile_bytes(ng, L1) + kOccBytes + 192LL * kStageRecBytes)
               : 1;
}

CUVGLS_HD constexpr int pass1_stage_recs(int ng, int L1) {
    if (!pass1_gather(ng, L1)) return pass1_small_stage(ng, L1) ? 192 : 256;
    int r = 4096;
    while (r > 256 && pass1_tile_bytes(ng, L1) + (long long)r * kStageRecBytes +
                              pass1_gather_bytes(L1, r) + kOccBytes > kSmemLimit)
        r -= 256;
    return r;
}

CUVGLS_HD constexpr long long pass1_smem(int ng, int L1, long long G) {
    // (one slot of padding per level-1 plane)
    if (pass1_long(ng, L1)) return (long long)kLongCols * (L1 + long_fac(L1, 0)) * 8;
    return pass1_tile_bytes(ng, L1) + (long long)pass1_stage_recs(ng, L1) * kStageRecBytes +
           (pass1_gather(ng, L1) ? pass1_gather_bytes(L1, pass1_stage_recs(ng, L1)) : 0) +
           kOccBytes;
}

// Shared memory of a pass-2 CTA: ng * R padded rows and the stage twiddles.
CUVGLS_HD constexpr long long pass2_smem(int ng, int L2) {
    if (pass2_reg(ng, L2))
        return ((ng == 3 ? pass2_reg_elems(L2) : nfft_reg_elems(L2)) + 2LL) * 8;
    if (pass2_deep(ng, L2)) return 8LL * deep_rows(L2) * deep_pitch(L2);
    if (pass2_cube(ng, L2)) return (16LL * kCubePitch + L2) * 8;  // exchange tile, grid A
    return (long long)(ng * pass2_rows(ng, L2) * row_stride(L2) +
                       (two_level_la(L2) ? 0 : fft_table_len(L2))) * 8;
}

}  // namespace cuvgls
