// pf_bin.cuh -- the chosen form's fused fold+bin kernel for CE and AOV.
//
// Included by the two semantics units after pf_fold.cuh (same namespace).
//
// Per (point, trial period) the reference computes
//     q = RN(t_corr / P)                  (FP64 divide)
//     folded = (float)(q - floor(q))      (FP64 floor, f64->f32 convert)
//     bin = (size_t)(folded / bin_size)   (f32 divide)
// which on B200 puts three instructions per evaluation on the narrow XU
// pipe (floor, conversion, the divide's reciprocal), ~16 ops/clk/SM.
// Here the bin comes from three FP64 operations and integer arithmetic:
//     q' = t_corr * RN(1/P)               within 2 ulp of RN(t_corr / P)
//     r  = RD(q' + 1.5*2^52)              low word = floor(q')
//     y  = RD(q' * n*2^20 + 1.5*2^52)     mantissa = 2^51 + floor(q'*n*2^20)
//     row = (y >> 20) - n*floor(q')       = floor(frac(q') * n)  (mod 2^32)
// The 20 low bits of y are frac(q')*n's fractional bits.  The reference's
// quotient folded / bin_size differs from frac(q')*n by less than a bound
// delta(n) (f32 divide, bin-width rounding, f64->f32 rounding of the phase,
// and q' versus RN(t_corr/P); computed on the host).  When frac(q')*n lies
// within that bound of an integer the evaluation recomputes the reference's
// exact sequence (the correctly rounded quotient via fold_exact, then the
// float fold and divide), so bin occupancies are identical by construction;
// about 3e-5 of evaluations take that branch at n = 10.
//
// Valid while |q| * n < 2^30 (checked per CTA from the batch's max|t|;
// otherwise the CTA runs the generic loop).  While also |q| < 2^19 one FP64
// operation does it (fast_bin32): y = RD(t_corr * (RN(1/P) * 2^32) +
// 1.5*2^52 + D) on the exact product leaves floor(frac(q') * 2^32) + D in its
// low word f, and the 64-bit product f * n holds the row (high word) and the
// position within it (low word, the edge test: D puts the guard below it).
//
// CE counters are 16-bit halves of 32-bit words (curve length * overlaps <
// 65536), doubling the cells per SM; AOV keeps a
// 32-bit count and a 32-bit fixed-point magnitude sum per bin.  Updates are
// `red.shared.add.u32` (no return value, no dependency chain).
//
// What bounds it: the shared-memory pipe.  Every lane of a warp reads the
// same staged point, and a 128-bit broadcast load occupies the pipe about
// 2.6 times as long as a conflict-free reduction (1.62 against 0.62 in the
// same units, 32 warps per SM), so one 16-byte point record and one
// reduction per evaluation were bound by the load.  Three things shrink it:
//   - CE takes its points sorted by magnitude column (ce_sort_kernel), so a
//     point is its time alone and the counter word and increment stay in
//     registers for a column's run.  Curves with few points for each column
//     they meet spend more on their runs (each padded to four points, about
//     30 instructions) than that saves: MIXED takes the points in their own
//     order with the column in the last bits of the time, five instructions
//     more per point (10 x 40 columns, 120 points a curve: 1.05 -> 0.91 ms;
//     10 x 64, 700 points: 0.94 -> 0.73).  The tuner weighs the two;
//   - a thread holds CELLS = 2 periods, for AOV also 3, so one load serves as
//     many evaluations (AOV samples from 256 points on 0.64 -> 0.60 ms with 3;
//     CE 10% slower with 3, both slower with 4: too few warps); staging the
//     times as floats and converting each was 5-7% slower, as the conversions
//     take the XU pipe;
//   - the guard rides in the FMA's constant and the product is one wide
//     multiply, so an evaluation is DFMA, IMAD.WIDE, IMAD, RED and half a
//     three-way minimum (6.4 instructions with all overheads on 4096 points,
//     11.1 before).
// Measured, 3000 ragged curves (20-2000 points) x 20000 periods, CE 10 x 10
// then AOV 15, plan with peaks: 12.06 -> 10.40 ms and 11.63 -> 8.99 ms (9.57
// and 8.86 ms with the statistics below, CE 9.09 with their table); CE 200 x
// 4096 x 10000 x 2 derivatives 7.26 -> 5.14 ms.  CE [1024,4096):
// issue 61%, fmaheavy pipe 73%, shared-memory pipe 50%; AOV: shared-memory
// pipe 88% (its two reductions per evaluation).
#pragma once

namespace pfk {
namespace PF_KNS {

// Resident CTAs per SM the bin kernel is compiled for: 1024 cells (CE, the
// shared-memory limit of 10 x 10 counters) and 1280 (AOV; 1024 measured 2-3%
// slower), 1536 with three cells per thread, per SM.
template <int ALGO, int BLOCK, int CELLS>
constexpr int bin_min_blocks() {
    return (ALGO == ALGO_CE ? 1024 : CELLS == 3 ? 1536 : 1280) / (BLOCK * CELLS);
}

// Fire-and-forget shared reduction.  No "memory" clobber: the counters it
// updates are never read inside the point loop, so the compiler may hoist
// the next points' shared loads above it (independent point chains overlap).
// The epilogue's counter reads are ordered after the loop by an explicit
// compiler barrier plus __syncwarp().
__device__ __forceinline__ void red_shared_u32(uint32_t addr, uint32_t v) {
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v));
}

// Both halves of a 32 x 32 bit product from one wide multiply (written as a
// C++ 64-bit product the compiler took a low and a high multiply).
__device__ __forceinline__ void mul_wide_u32(uint32_t a, uint32_t b, uint32_t& lo,
                                             uint32_t& hi) {
    asm("{ .reg .u64 w; mul.wide.u32 w, %2, %3; mov.b64 {%0, %1}, w; }"
        : "=r"(lo), "=r"(hi)
        : "r"(a), "r"(b));
}

// A time that was a float has 29 zero bits at the end of its double; a CE
// point's magnitude column (below 4096) is kept in the last 12.
constexpr uint32_t kColumnBits = 0xFFFu;
__device__ __forceinline__ double with_column(double t, uint32_t col) {
    return __hiloint2double(__double2hiint(t), (int)((uint32_t)__double2loint(t) | col));
}
__device__ __forceinline__ uint32_t column_of(double t) {
    return (uint32_t)__double2loint(t) & kColumnBits;
}
__device__ __forceinline__ double without_column(double t) {
    return __hiloint2double(__double2hiint(t),
                            (int)((uint32_t)__double2loint(t) & ~kColumnBits));
}

__device__ __forceinline__ void compiler_fence() { asm volatile("" ::: "memory"); }

__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

constexpr double kMagic15 = 6755399441055744.0;  // 1.5 * 2^52

// Curves shorter than this take the CE statistic's logs from a table.
constexpr uint32_t kXlxTable = 512;
static_assert(kXlxTable * 4 <= kBinTile * 8, "the table takes the staged tile's place");

// A staged point of the shared-histogram kernel (pf_binwarp.cuh): its time,
// and its magnitude bin (CE) or fixed-point magnitude (AOV).
struct BinPoint {
    double t;
    uint32_t a, b;
};

// c log2 c of a count (zero for c = 0 and 1): one log per bin, no divide,
// ln 2 applied once at the end.  A count (< 2^16 here: the bin kernels run
// curves of fewer than 65536 points) becomes a float exactly by placing it
// in the mantissa of 2^23, which costs a bitwise OR and an add instead of an
// integer-to-float conversion.  Explicit roundings, so that every kernel
// that sums these terms in the same order gets the same bits.
__device__ __forceinline__ float ce_xlx(uint32_t c) {
    const float f = __fsub_rn(__uint_as_float(c | 0x4B000000u), 8388608.0f);
    return __fmul_rn(f, log2f(fmaxf(f, 1.0f)));
}

// CE of one cell from its running sum of row terms, over n points.
__device__ __forceinline__ float ce_finish(float acc, uint32_t n) {
    return __fmul_rn(acc, 0.69314718055994531f / (float)n);
}

// AOV of one cell from sum_b X_b^2 / c_b (fixed-point bin sums X_b); per
// curve, xx_n = X^2 / n and scale = (n - nP) / (nP - 1).
__device__ __forceinline__ double aov_xx_n(const CurveDesc& cd) {
    return cd.fix_sumx * cd.fix_sumx / (double)cd.n;
}
__device__ __forceinline__ double aov_scale(uint32_t n, uint32_t nP) {
    return ((double)n - (double)nP) / ((double)nP - 1.0);
}
__device__ __forceinline__ float aov_finish(double sbx, double xx_n, double sumx2,
                                            double scale) {
    const double s1 = fmax(sbx - xx_n, 0.0);
    const double s2 = __dadd_rn(sumx2, -sbx);
#if PF_SEM_CPU_TU
    return (s2 <= 0.0) ? 0.0f : (float)(scale * (s1 / s2));
#else
    return (float)(scale * (s1 / (s2 <= 0.0 ? 0.0 : s2)));
#endif
}

// The chosen form's CE statistic of CELLS cells at once.  Counters are read
// through 32-bit shared addresses (tbase = the thread's first column, the
// cells cell_bytes apart).  Each row term
// C_j ln C_j - sum_i c_ij ln c_ij is non-negative, so FP32 accumulation keeps
// the relative error near 1e-7 (FP64 here costs registers in the binning
// loop, measured slower).  Per row, the magnitude bins are taken in pairs
// (the two 16-bit halves of a word).  A cell's sum is one long chain of
// loads, logs and adds, so two rows of every cell run side by side, with one
// cell per thread (large histograms, few resident warps) four words of each
// (10 x 64 columns, 20 points a curve: 2.51 -> 1.95 ms) (tuning
// samples of 10 x 10 bins, one cell and row at a time -> this: [64,256) 1.31
// -> 1.15 ms, [256,1024) 0.76 -> 0.70, [1024,4096) 0.60 -> 0.57; the floor is
// the log's 110 operations per cell on the XU pipe).  8-bit counters for
// curves under 256 points, which double the resident warps, were slower
// (1.15 -> 1.18 ms).
//
// TABLE: c log2 c comes from a table in shared memory at `table` (byte c * 4;
// the same ce_xlx values) and the counters count in units of 4, so that a
// counter is the table's byte offset: two operations per count instead of
// six, and none on the XU pipe.  Small counts fall on different banks or on
// the same word, so the lookups hardly conflict.  Samples: [64,256) 1.15 -> 1.05
// ms, [256,1024) 0.70 -> 0.65; CE of 3000 ragged curves x 20000 periods 9.57 ->
// 9.09 ms.
__device__ __forceinline__ float lds_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
template <bool CNT16, int CELLS, bool TABLE, int UNROLL>
__device__ __forceinline__ void ce_stat_fast(uint32_t tbase, uint32_t cell_bytes, uint32_t nP,
                                             uint32_t W, uint32_t cols, uint32_t n,
                                             uint32_t table, float (&out)[CELLS]) {
    auto xlx = [&](uint32_t c) -> float {
        if constexpr (TABLE) return lds_f32(table + c);
        else return ce_xlx(c);
    };
    float acc[CELLS];
#pragma unroll
    for (int c = 0; c < CELLS; c++) acc[c] = 0.0f;
    auto rows = [&](auto rows_tag, uint32_t j) {
        constexpr int R = decltype(rows_tag)::value;
        uint32_t col[R][CELLS];
        float row[R][CELLS];
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int c = 0; c < CELLS; c++) {
                col[r][c] = 0u;
                row[r][c] = 0.0f;
            }
        uint32_t at = tbase + j * (cols * 4u);
#pragma unroll UNROLL
        for (uint32_t wi = 0; wi < W; wi++, at += nP * (cols * 4u)) {
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int c = 0; c < CELLS; c++) {
                    const uint32_t wv = lds_u32(at + r * (cols * 4u) + c * cell_bytes);
                    // Both 16-bit halves summed at once: each half's total
                    // is below 2^16, so no carry crosses halves.
                    col[r][c] += wv;
                    row[r][c] = __fadd_rn(
                        row[r][c], CNT16 ? __fadd_rn(xlx(wv & 0xFFFFu), xlx(wv >> 16)) : xlx(wv));
                }
        }
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int c = 0; c < CELLS; c++) {
                const uint32_t t = CNT16 ? (col[r][c] & 0xFFFFu) + (col[r][c] >> 16) : col[r][c];
                acc[c] = __fadd_rn(acc[c], __fsub_rn(xlx(t), row[r][c]));
            }
    };
    uint32_t j = 0;
#pragma unroll 1
    for (; j + 2 <= nP; j += 2) rows(std::integral_constant<int, 2>{}, j);
    if (j < nP) rows(std::integral_constant<int, 1>{}, j);
#pragma unroll
    for (int c = 0; c < CELLS; c++) out[c] = ce_finish(acc[c], n);
}

// An unsigned integer as a double: placed in the mantissa of 2^52, which is
// then taken off (exact, and no conversion instruction).
__device__ __forceinline__ double u32_to_double(uint32_t v) {
    return __dadd_rn(__hiloint2double(0x43300000, (int)v), -4503599627370496.0);
}

// 1 / c rounded to nearest for a count 1 <= c < 65536: two Newton steps
// r += r (1 - c r) from the hardware's approximation.  With a start good to
// 2^-18 the second step's error is below 2^-70 of the result, and 1 / c for
// c < 2^16 lies at least 2^-70 from every midpoint of two doubles, so the
// last rounding is the right one (checked against __drcp_rn for every c).
__device__ __forceinline__ double count_rcp(uint32_t c) {
    const double x = u32_to_double(c);
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = __fma_rn(r, __fma_rn(-x, r, 1.0), r);
    return __fma_rn(r, __fma_rn(-x, r, 1.0), r);
}

__global__ void count_rcp_kernel(uint32_t n, double* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = count_rcp(i + 1u);
}

// The chosen form's AOV sum_b X_b^2 / c_b over the fixed-point bin sums X_b
// (empty bins have X_b = 0 and contribute nothing), CELLS cells at once
// ([64,256) samples 0.87 -> 0.81 ms against library reciprocals and integer
// conversions).  Counters [bin][count, sum][cols].
template <int CELLS>
__device__ __forceinline__ void aov_sbx_fast(uint32_t tbase, uint32_t cell_bytes, uint32_t nP,
                                             uint32_t cols, double (&sbx)[CELLS]) {
#pragma unroll
    for (int c = 0; c < CELLS; c++) sbx[c] = 0.0;
#pragma unroll 2
    for (uint32_t b = 0; b < nP; b++) {
#pragma unroll
        for (int c = 0; c < CELLS; c++) {
            const uint32_t at = tbase + b * (2u * cols * 4u) + c * cell_bytes;
            const uint32_t cnt = lds_u32(at);
            const double Xd = u32_to_double(lds_u32(at + cols * 4u));
            sbx[c] = __fma_rn(__dmul_rn(Xd, Xd), count_rcp(max(cnt, 1u)), sbx[c]);
        }
    }
}

// Statistic forms.  REF_STATS: the reference's operation sequence
// (periodfind/cuda/ce.cu:160-178, aov.cu:84-121), so identical bins give
// values bit-identical to the plain form.  Otherwise the same statistic
// computed from the integer bins with one log (CE) or one reciprocal (AOV)
// per bin and no divide:
//   CE  = (sum_j C_j ln C_j - sum_ij c_ij ln c_ij) / n,  C_j = sum_i c_ij
//         (the bin counts c over n points; the reference's p_ij ln(p_j/p_ij)
//         summed, with the 1/n scale taken out of the logs);
//   AOV = (n - nP)/(nP - 1) * s1 / s2, s1 = sum_b X_b^2 / c_b - X^2 / n,
//         s2 = sum x^2 - sum_b X_b^2 / c_b (X_b the fixed-point bin sums).
// MIXED (CE): points in their own order instead of sorted by column.
template <int ALGO, bool CNT16, int BLOCK, bool REF_STATS, int ROUNDS, int CELLS, bool MIXED>
__device__ __forceinline__ void bin_item(const FoldParams& p, const WorkItem w, uint32_t item) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr uint32_t kCols = BLOCK * CELLS;  // counter columns of the CTA
    // CE: the times of the staged points (doubles), sorted by magnitude
    // column.  AOV: the times and the fixed-point magnitudes.
    double* tile_t = reinterpret_cast<double*>(smem);
    uint32_t* tile_a = reinterpret_cast<uint32_t*>(smem + kBinTile * sizeof(double));
    unsigned char* cnt_raw = smem + bin_tile_bytes(ALGO);
    const uint32_t cnt_base = (uint32_t)__cvta_generic_to_shared(cnt_raw);

    stamp_start(p, item);
    const CurveDesc cd = p.curves[w.curve];
    const uint32_t n = cd.n;
    const int tid = threadIdx.x;
    const float period_dt = p.pdts[w.pdt];
    const uint32_t nP = p.n_phase, nM = p.n_mag;

    // Counter layout: CE  [W words][nP rows][kCols] u32, W = nM or ceil(nM/2)
    //                 AOV [nP][2][kCols] u32 (count, fixed-point sum): a bin's
    //                 sum lies a constant kCols words after its count, so the
    //                 second reduction takes an immediate address offset.
    // Cell c of thread tid owns column c * BLOCK + tid.
    const uint32_t W = (ALGO == ALGO_CE) ? (CNT16 ? (nM + 1) / 2 : nM) : 1;
    const uint32_t slots = (ALGO == ALGO_CE) ? nP * W : 2 * nP;
    const uint32_t tbase = cnt_base + tid * 4;

    // The item covers ROUNDS x CELLS x BLOCK periods; in round r thread tid
    // takes periods p0 + (r * CELLS + c) * BLOCK + tid, c < CELLS, all at
    // once.  A dead cell repeats the last period.
    auto period_at = [&](uint32_t j) -> uint32_t { return w.p0 + min(j, w.np - 1u); };
    // Range guard for y = q * n * 2^20 over the `cells` periods of each thread
    // of the warp from j on: |t_corr / P| is at most y (max|t| + |pdt| max|t|^2
    // y / 2), y the largest |1/P| (infinite for a P of 0).  2: |q| < 2^19 as
    // well, so the phase's 32 fraction bits come from one FMA; 1: the
    // three-operation bin; 0: the exact sequence.  The cell constants (1 / P as a double-double, pdt / 2P) are
    // finite exactly when P is finite and non-zero and pdt is finite;
    // non-finite periods or derivatives (device-pointer callers are not
    // checked on the host) take the exact sequence, whose bins are always
    // clamped.
    auto range_of = [&](uint32_t j, int cells) -> int {
        uint32_t least = 0x7F800000u;  // the smallest |P|, 0 for what is not finite
#pragma unroll
        for (int c = 0; c < cells; c++) {
            const uint32_t per =
                __float_as_uint(p.periods[period_at(j + (uint32_t)(c * BLOCK))]) & 0x7FFFFFFFu;
            least = min(least, per < 0x7F800000u ? per : 0u);
        }
        const double y = __drcp_rn((double)__uint_as_float(__reduce_min_sync(0xffffffffu, least)));
        const double tmax = (double)__uint_as_float(*p.tmax_bits);
        const double q = y * __fma_rn(0.5 * fabs((double)period_dt) * tmax * tmax, y, tmax);
        return q * (double)nP < 1073741824.0 ? q < 524288.0 ? 2 : 1 : 0;  // 2^30
    };
    // With one cell per thread the item's rounds share it; with several each of
    // its rounds has its own, as the shortest of 512 periods would take all of them
    // out of the fast range (2000 curves of 300 points x 1000 periods x 3
    // derivatives, half the cells beyond it: AOV 1.74 -> 1.28 ms, CE 1.92 ->
    // 1.73; AOV on the ragged plan within it 8.36 -> 8.24).
    constexpr bool kItemRange = CELLS == 1 || ROUNDS == 1;
    const int item_range = kItemRange ? range_of((uint32_t)tid, ROUNDS * CELLS) : 0;
    // The two FP64 divides of the AOV statistic that depend on the curve only.
    __shared__ double s_aov[2];
    if (ALGO == ALGO_AOV && !REF_STATS && tid == 0) {
        s_aov[0] = aov_xx_n(cd);
        s_aov[1] = aov_scale(n, nP);
    }

    const double nd20 = (double)nP * 1048576.0;
    const uint32_t n_neg = 0u - nP;
    // Edge test: ((ylo + D) mod 2^20) < 2D, as one IMAD and one compare on
    // the fraction bits moved to the top of the word.
    const uint32_t edge_add = p.edge_d << 12;
    const uint32_t edge_lim = (2u * p.edge_d) << 12;
    const uint32_t edge32_lim = p.edge32_lim;

    // CE: the curve's sorted times and its runs of equal magnitude column
    // (see ce_sort_kernel), n_pad counting the runs' padding; mixed: its points
    // in their own order, each with its column.
    const float* src_t = p.t + cd.off;
    const uint32_t* runs = nullptr;
    uint32_t n_pad = n;
    if constexpr (ALGO == ALGO_CE && !MIXED) {
        src_t = p.ts + (cd.off * p.ts_mul + (int64_t)w.curve * p.ts_pad);
        runs = p.runs + (cd.off * p.run_mul + (int64_t)w.curve * p.run_pad);
        n_pad = runs[0];
    }

    auto stage = [&](uint32_t base, uint32_t cnt) {
        const float4* gt = reinterpret_cast<const float4*>(src_t + base);
        const uint32_t n4 = (cnt + 3) >> 2;
        for (uint32_t i4 = tid; i4 < n4; i4 += BLOCK) {
            float4 q = gt[i4];
            if constexpr (ALGO == ALGO_AOV) {
                uint4 a = reinterpret_cast<const uint4*>(p.aux32 + cd.off + base)[i4];
                // The packed arrays end in zeros; a repeated time with
                // magnitude 0 keeps the padding out of the edge test of t = 0.
                if (4 * i4 + 3 >= cnt) {
                    const float last = src_t[base + cnt - 1];
                    if (4 * i4 + 1 >= cnt) { q.y = last; a.y = 0u; }
                    if (4 * i4 + 2 >= cnt) { q.z = last; a.z = 0u; }
                    if (4 * i4 + 3 >= cnt) { q.w = last; a.w = 0u; }
                }
                reinterpret_cast<uint4*>(tile_a)[i4] = a;
            }
            if constexpr (MIXED) {
                if (4 * i4 + 3 >= cnt) {
                    const float last = src_t[base + cnt - 1];
                    if (4 * i4 + 1 >= cnt) q.y = last;
                    if (4 * i4 + 2 >= cnt) q.z = last;
                    if (4 * i4 + 3 >= cnt) q.w = last;
                }
                const ushort4 k = reinterpret_cast<const ushort4*>(p.cols + cd.off + base)[i4];
                reinterpret_cast<double2*>(tile_t)[2 * i4] =
                    make_double2(with_column(q.x, k.x), with_column(q.y, k.y));
                reinterpret_cast<double2*>(tile_t)[2 * i4 + 1] =
                    make_double2(with_column(q.z, k.z), with_column(q.w, k.w));
            } else {
                reinterpret_cast<double2*>(tile_t)[2 * i4] = make_double2(q.x, q.y);
                reinterpret_cast<double2*>(tile_t)[2 * i4 + 1] = make_double2(q.z, q.w);
            }
        }
    };
    // CE statistic by table (ce_stat_fast) where the table fits the staged
    // tile's place, which it takes after the round's last point.
    const bool table = ALGO == ALGO_CE && !REF_STATS && CNT16 && n < kXlxTable;
    const uint32_t unit = table ? 4u : 1u;
    // A curve that fits one tile is staged once for every round.
    const bool one_tile = n_pad <= kBinTile && !(table && ROUNDS > 1);
    if (one_tile) {
        __syncthreads();
        stage(0, n_pad);
        __syncthreads();
    }

#pragma unroll 1
    for (int r = 0; r < ROUNDS; r++) {
    const uint32_t j0 = (uint32_t)(r * CELLS * BLOCK + tid);
    const bool active = j0 < w.np;  // a thread with any live cell runs all
    auto cell_period = [&](int c) -> uint32_t { return period_at(j0 + (uint32_t)(c * BLOCK)); };
    const int range = kItemRange ? item_range : range_of(j0, CELLS);
    // RN(1/P), times 2^32 where the one-FMA bin applies (exact), and pdt / 2P.
    double ys[CELLS], pc[CELLS];
#pragma unroll
    for (int c = 0; c < CELLS; c++) {
        Cell s;
        cell_setup<FOLD_EXACT>(s, p.periods[cell_period(c)], period_dt);
        ys[c] = s.yhi * (range == 2 ? 4294967296.0 : 1.0);
        pc[c] = s.c;
    }
    for (uint32_t k = 0; k < slots; k++)
#pragma unroll
        for (int c = 0; c < CELLS; c++)
            reinterpret_cast<uint32_t*>(cnt_raw)[k * kCols + c * BLOCK + tid] = 0u;

    uint32_t run_no = 0, run_at = 0, run = 0;  // CE: run number, its first position, its word
    if constexpr (ALGO == ALGO_CE && !MIXED) run = runs[1];

    for (uint32_t base = 0; base < n_pad; base += kBinTile) {
        const uint32_t cnt = min(kBinTile, n_pad - base);
        if (!one_tile) {
            __syncthreads();
            stage(base, cnt);
            __syncthreads();
        }
        if (!active) continue;

        // t_corr = t - c t^2 for the fast bins.  AOV takes it in one FMA from
        // the point's square, which is exact (t has 24 bits) and which the
        // thread's cells share (250 x 4096 points x 10000 periods x 2
        // derivatives with peaks: 8.40 -> 8.03 ms).  It differs from the
        // reference's by its rounding of c t: |c t^2 / P| n 2^-53 <= 2^-23 of a
        // bin while |q| n < 2^30, which the guard's two units of 2^-20 cover;
        // the exact sequence keeps the reference's order.  CE keeps that order
        // here too: its groups of 16 points have no register left for the
        // squares (4 % gained with a derivative, 1 % lost to spills without).
        auto t_corr = [&](double td, double c_) -> double {
            if constexpr (ALGO == ALGO_AOV) return __fma_rn(-c_, __dmul_rn(td, td), td);
            else return td - c_ * td * td;
        };
        // Fast bin of one point: row (+2^31 bias) and the edge-test value
        // ((fraction + D) << 12); the point is near an edge iff ev < edge_lim.
        auto fast_bin = [&](double td, double y_, double c_, auto has_pdt_tag,
                            uint32_t& ev) -> uint32_t {
            constexpr bool HAS_PDT = decltype(has_pdt_tag)::value;
            double a = td;
            if constexpr (HAS_PDT) a = t_corr(td, c_);
            const double qh = __dmul_rn(a, y_);
            const double r = __dadd_rd(qh, kMagic15);
            const double y = __fma_rd(qh, nd20, kMagic15);
            const uint32_t ylo = (uint32_t)__double2loint(y);
            const uint32_t yup = (uint32_t)__double2hiint(y);
            ev = ylo * 4096u + edge_add;
            return __funnelshift_r(ylo, yup, 20) + (uint32_t)__double2loint(r) * n_neg;
        };
        // |q| < 2^19: y = RD(t_corr * (RN(1/P) * 2^32) + 1.5*2^52 + D), one
        // FMA on the exact product (closer to t_corr / P than the rounded
        // product fast_bin uses, so the same guard holds), leaves
        // f = floor(frac(q') * 2^32) + D in its low word.  The 64-bit product
        // f * n then holds the row in its high word and the position within
        // the row, D n further on, in its low word: a point within D n of an
        // edge on either side is one whose low word is below 2 D n, and the
        // rows of all others are unchanged by D.  One FP64 operation and one
        // integer multiply per point, and nothing added for the edge test.
        // The row carries no bias.
        auto fast_bin32 = [&](double td, double y32, double c_, auto has_pdt_tag,
                              uint32_t& ev) -> uint32_t {
            constexpr bool HAS_PDT = decltype(has_pdt_tag)::value;
            double a = td;
            if constexpr (HAS_PDT) a = t_corr(td, c_);
            const double y = __fma_rd(a, y32, p.magic32);
            const uint32_t f = (uint32_t)__double2loint(y);
            uint32_t row;
            mul_wide_u32(f, nP, ev, row);
            return row;
        };
        // The reference's exact sequence (correctly rounded quotient, float
        // fold, f32 divide, then % n_phase: a folded phase of 1.0f gives bin
        // n_phase, which wraps to 0): the bin (+2^31 bias).
        auto exact_row = [&](double td, const Cell& s, auto has_pdt_tag) -> uint32_t {
            constexpr bool HAS_PDT = decltype(has_pdt_tag)::value;
            const float folded = fold_exact<HAS_PDT>(td, s);
            const uint32_t pb = min(trunc_u(folded / p.phase_bin_size), nP);
            return 0x80000000u + (pb == nP ? 0u : pb);
        };
        // One update: CE adds `inc` to the row's word at `at` (the column's
        // word of this cell); AOV adds `inc` to the count and `a` to the sum.
        // The row is kept opaque to the compiler: it would otherwise take
        // row << k out of the 64-bit product with a funnel shift and a mask,
        // where a shift-and-add of the high word is one operation.
        auto add = [&](uint32_t row, uint32_t at, uint32_t inc, uint32_t a) {
            asm("" : "+r"(row));
            if constexpr (ALGO == ALGO_CE) {
                red_shared_u32(row * (kCols * 4) + at, inc);
            } else {
                const uint32_t a0 = row * (2 * kCols * 4) + at;
                red_shared_u32(a0, inc);
                red_shared_u32(a0 + kCols * 4, a);
            }
        };

        // The first word (row 0, cell 0) and the increment of a CE column.
        auto column_word = [&](uint32_t col) -> uint32_t {
            return tbase + (CNT16 ? col >> 1 : col) * (nP * kCols * 4);
        };
        auto column_unit = [&](uint32_t col) -> uint32_t {
            return (CNT16 && (col & 1u)) ? unit << 16 : unit;
        };
        auto body = [&](auto has_pdt_tag, auto fast_tag, auto f32_tag) {
            constexpr bool FAST = decltype(fast_tag)::value;
            constexpr bool F32 = decltype(f32_tag)::value;
            // Fast bin (unbiased with F32, +2^31 otherwise; the counter
            // address is the same either way) and its edge limit.
            auto bin_of = [&](double td, double y_, double c_, uint32_t& ev) -> uint32_t {
                if constexpr (F32) return fast_bin32(td, y_, c_, has_pdt_tag, ev);
                else return fast_bin(td, y_, c_, has_pdt_tag, ev);
            };
            const uint32_t lim = F32 ? edge32_lim : edge_lim;
            // G staged points from position i, the first `live` of them
            // real: no branch per point; a group whose smallest edge-test
            // value is below the limit is revisited and its near-edge
            // points are moved to the reference's bin.
            // Mixed: each point's counter word and increment come from its
            // column instead of from the run.
            auto group = [&](auto g_tag, auto mask_tag, uint32_t i, uint32_t live, uint32_t at,
                             uint32_t inc) {
                constexpr int G = decltype(g_tag)::value;
                constexpr bool MASK = decltype(mask_tag)::value;
                double td[G];
                uint32_t ta[G];
#pragma unroll
                for (int k = 0; k < G; k += 2) {
                    const double2 q = reinterpret_cast<const double2*>(tile_t + i)[k >> 1];
                    td[k] = q.x;
                    td[k + 1] = q.y;
                }
                if constexpr (ALGO == ALGO_AOV) {
#pragma unroll
                    for (int k = 0; k < G; k += 4) {
                        const uint4 q = reinterpret_cast<const uint4*>(tile_a + i)[k >> 2];
                        ta[k] = q.x;
                        ta[k + 1] = q.y;
                        ta[k + 2] = q.z;
                        ta[k + 3] = q.w;
                    }
                }
                uint32_t emin[CELLS];
#pragma unroll
                for (int c = 0; c < CELLS; c++) emin[c] = 0xFFFFFFFFu;
#pragma unroll
                for (int k = 0; k < G; k++) {
                    uint32_t ak = at, ik = inc;
                    if constexpr (MIXED) {
                        const uint32_t col = column_of(td[k]);
                        ak = column_word(col);
                        ik = column_unit(col);
                        td[k] = without_column(td[k]);
                    }
                    if (MASK && (uint32_t)k >= live) ik = 0u;
#pragma unroll
                    for (int c = 0; c < CELLS; c++) {
                        uint32_t ev;
                        const uint32_t row = bin_of(td[k], ys[c], pc[c], ev);
                        emin[c] = min(emin[c], ev);
                        add(row, ak + c * BLOCK * 4, ik, ALGO == ALGO_AOV ? ta[k] : 0u);
                    }
                }
                uint32_t em = emin[0];
#pragma unroll
                for (int c = 1; c < CELLS; c++) em = min(em, emin[c]);
                if (em < lim) {
                    // Which of the group's evaluations are near an edge,
                    // then each of those (rarely more than one).
                    uint32_t near = 0;
#pragma unroll
                    for (int c = 0; c < CELLS; c++)
#pragma unroll
                        for (int k = 0; k < G; k++) {
                            // (a square kept for here would cost registers)
                            double t = td[k];
                            if constexpr (ALGO == ALGO_AOV && decltype(has_pdt_tag)::value)
                                asm("" : "+d"(t));
                            uint32_t ev;
                            bin_of(t, ys[c], pc[c], ev);
                            if (ev < lim) near |= 1u << (c * G + k);
                        }
                    if constexpr (MASK) {
                        const uint32_t m = (1u << live) - 1u;  // 0 < live < G
#pragma unroll
                        for (int c = 0; c < CELLS; c++) near &= ~((((1u << G) - 1u) ^ m) << (c * G));
                    }
                    while (near) {
                        const uint32_t e = __ffs(near) - 1;
                        near &= near - 1;
                        const uint32_t c = e / G, k = e % G;
                        Cell s;
                        cell_setup<FOLD_EXACT>(s, p.periods[cell_period(c)], period_dt);
                        double t = tile_t[i + k];
                        uint32_t ak = at, ik = inc;
                        if constexpr (MIXED) {
                            ak = column_word(column_of(t));
                            ik = column_unit(column_of(t));
                            t = without_column(t);
                        }
                        uint32_t ev;
                        const uint32_t row =
                            bin_of(t, s.yhi * (F32 ? 4294967296.0 : 1.0), s.c, ev);
                        const uint32_t ex =
                            exact_row(t, s, has_pdt_tag) - (F32 ? 0x80000000u : 0u);
                        if (ex != row) {
                            // u32 wraparound keeps packed halves and sums exact.
                            const uint32_t a = ALGO == ALGO_AOV ? tile_a[i + k] : 0u;
                            add(row, ak + c * BLOCK * 4, 0u - ik, 0u - a);
                            add(ex, ak + c * BLOCK * 4, ik, a);
                        }
                    }
                }
            };
            // Beyond the fast range: kSide cells side by side (three would take
            // 8 registers more of the whole kernel), set up once per tile (the
            // case above one after the other, set up for every run of points:
            // CE 2.63 -> 1.92 ms).
            constexpr int kSide = FAST || CELLS == 3 ? 1 : CELLS;
            Cell slow[kSide];
            auto set_up = [&](int c0) {
#pragma unroll
                for (int c = 0; c < kSide; c++)
                    cell_setup<FOLD_EXACT>(slow[c], p.periods[cell_period(c0 + c)], period_dt);
            };
            if constexpr (!FAST && kSide == CELLS) set_up(0);
            // m points from tile position i (a multiple of 4).
            auto span = [&](uint32_t i, uint32_t m, uint32_t at, uint32_t inc) {
                if constexpr (FAST) {
                    // Groups of 16 (CE runs; 16 were slower for AOV, whose two
                    // reductions per point need the registers), then 8, 4
                    // and the rest of the last four.
                    using G16 = std::integral_constant<int, 16>;
                    using G8 = std::integral_constant<int, 8>;
                    using G4 = std::integral_constant<int, 4>;
                    using Whole = std::false_type;
                    uint32_t k = 0;
                    if constexpr (ALGO == ALGO_CE && !MIXED) {
#pragma unroll 1
                        for (; k + 16 <= m; k += 16) group(G16{}, Whole{}, i + k, 16u, at, inc);
                        if (k + 8 <= m) {
                            group(G8{}, Whole{}, i + k, 8u, at, inc);
                            k += 8;
                        }
                    } else {
#pragma unroll 1
                        for (; k + 8 <= m; k += 8) group(G8{}, Whole{}, i + k, 8u, at, inc);
                    }
                    if (k + 4 <= m) {
                        group(G4{}, Whole{}, i + k, 4u, at, inc);
                        k += 4;
                    }
                    if (k < m) group(G4{}, std::true_type{}, i + k, m - k, at, inc);
                } else {
                    constexpr int kUnroll = kSide == 1 ? 4 : 2;
#pragma unroll 1
                    for (int c0 = 0; c0 < CELLS; c0 += kSide) {
                        if constexpr (kSide < CELLS) set_up(c0);
#pragma unroll kUnroll
                        for (uint32_t k = 0; k < m; k++) {
                            double t = tile_t[i + k];
                            uint32_t ak = at + c0 * BLOCK * 4, ik = inc;
                            if constexpr (MIXED) {
                                ak = column_word(column_of(t));
                                ik = column_unit(column_of(t));
                                t = without_column(t);
                            }
                            const uint32_t a = ALGO == ALGO_AOV ? tile_a[i + k] : 0u;
#pragma unroll
                            for (int c = 0; c < kSide; c++)
                                add(exact_row(t, slow[c], has_pdt_tag), ak + c * BLOCK * 4, ik, a);
                        }
                    }
                }
            };
            if constexpr (ALGO == ALGO_AOV) {
                span(0u, cnt, tbase, 1u);
            } else if constexpr (MIXED) {
                span(0u, cnt, 0u, 0u);
            } else {
                // The runs (one magnitude column each) that meet this tile.
                const uint32_t end = base + cnt;
                while (run != 0u && run_at < end) {
                    const uint32_t len = run & 0xFFFFu, col = run >> 16;
                    const uint32_t lo = max(run_at, base), hi = min(run_at + len, end);
                    const uint32_t next = runs[run_no + 2];
                    if (hi > lo)
                        span(lo - base, hi - lo, column_word(col), column_unit(col));
                    const uint32_t next_at = run_at + ((len + 3u) & ~3u);
                    if (next_at > end) break;  // the rest lies in the next tile
                    run_at = next_at;
                    run = next;
                    run_no++;
                }
            }
        };
        using T_ = std::true_type;
        using F_ = std::false_type;
        if (period_dt != 0.0f) {
            if (range == 2) body(T_{}, T_{}, T_{});
            else if (range == 1) body(T_{}, T_{}, F_{});
            else body(T_{}, F_{}, F_{});
        } else {
            if (range == 2) body(F_{}, T_{}, T_{});
            else if (range == 1) body(F_{}, T_{}, F_{});
            else body(F_{}, F_{}, F_{});
        }
    }
    // Every lane of the warp reaches this barrier (inactive lanes skip the
    // statistic after it).
    compiler_fence();
    __syncwarp();
    if constexpr (!REF_STATS) {
        if (table) {  // uniform over the CTA
            __syncthreads();
            for (uint32_t c = tid; c <= n; c += BLOCK)
                reinterpret_cast<float*>(tile_t)[c] = ce_xlx(c);
            __syncthreads();
        }
        if (active) {
            float res[CELLS];
            if constexpr (ALGO == ALGO_CE) {
                constexpr int kUnroll = CELLS == 1 ? 4 : MIXED ? 2 : 1;
                if (table)
                    ce_stat_fast<CNT16, CELLS, true, kUnroll>(
                        tbase, BLOCK * 4, nP, W, kCols, n,
                        (uint32_t)__cvta_generic_to_shared(tile_t), res);
                else
                    ce_stat_fast<CNT16, CELLS, false, kUnroll>(tbase, BLOCK * 4, nP, W, kCols, n,
                                                               0u, res);
            } else {
                double sbx[CELLS];
                aov_sbx_fast<CELLS>(tbase, BLOCK * 4, nP, kCols, sbx);
#pragma unroll
                for (int c = 0; c < CELLS; c++)
                    res[c] = aov_finish(sbx[c], s_aov[0], cd.fix_sumx2, s_aov[1]);
            }
#pragma unroll
            for (int c = 0; c < CELLS; c++)
                if (j0 + (uint32_t)(c * BLOCK) < w.np)
                    p.out[(size_t)w.curve * ((size_t)p.n_per * p.n_pdt) +
                          (size_t)cell_period(c) * p.n_pdt + w.pdt] = res[c];
        }
        continue;
    }
    // The reference statistic (one cell per thread).
    if (active) {
    const uint32_t pi = cell_period(0);
    const size_t out_idx =
        (size_t)w.curve * ((size_t)p.n_per * p.n_pdt) + (size_t)pi * p.n_pdt + w.pdt;
    const uint32_t* cnt32 = reinterpret_cast<const uint32_t*>(cnt_raw);
    if constexpr (ALGO == ALGO_CE) {
        auto count = [&](uint32_t j, uint32_t i) -> uint32_t {
            if constexpr (CNT16) {
                const uint32_t wv = cnt32[((i >> 1) * nP + j) * kCols + tid];
                return (i & 1u) ? (wv >> 16) : (wv & 0xFFFFu);
            } else {
                return cnt32[(i * nP + j) * kCols + tid];
            }
        };
        if (p.bins) {
            uint32_t* o = p.bins + out_idx * ((size_t)nP * nM);
            for (uint32_t j = 0; j < nP; j++)
                for (uint32_t i = 0; i < nM; i++) o[j * nM + i] = count(j, i);
        }
        const float divf = (float)((unsigned long long)n * p.p_overlap * p.m_overlap);
        float ce = 0.0f;
        for (uint32_t j = 0; j < nP; j++) {
            float p_j = 0.0f;
            for (uint32_t i = 0; i < nM; i++) p_j += (float)count(j, i) / divf;
#if PF_SEM_CPU_TU
            for (uint32_t i = 0; i < nM; i++) {
                const float p_ij = (float)count(j, i) / divf;
                if (p_ij != 0.0f) ce += p_ij * logf(p_j / p_ij);
            }
#else
            float ce_contrib = 0.0f;
            for (uint32_t i = 0; i < nM; i++) {
                const float p_ij = (float)count(j, i) / divf;
                if (p_ij != 0) ce_contrib += p_ij * logf(p_j / p_ij);
            }
            ce += ce_contrib;
#endif
        }
        p.out[out_idx] = ce;
    } else {
        const uint32_t* sums = cnt32 + kCols;
        if (p.bins) {
            uint32_t* o = p.bins + out_idx * (size_t)nP;
            for (uint32_t b = 0; b < nP; b++) o[b] = cnt32[2 * b * kCols + tid];
        }
        const double xbar = cd.fix_sumx / (double)n;
        double s1 = 0.0, sbx = 0.0;
        for (uint32_t b = 0; b < nP; b++) {
            const uint32_t c = cnt32[2 * b * kCols + tid];
            const uint32_t X = sums[2 * b * kCols + tid];
            if (c != 0u) {
                const double nb = (double)c;
                const double Xd = (double)X;
                const double mu = Xd / nb;
                const double r = mu - xbar;
                s1 = __fma_rn(nb * r, r, s1);
                sbx = __fma_rn(Xd, mu, sbx);
            }
        }
        const double s2 = __dadd_rn(cd.fix_sumx2, -sbx);
        const double scale = ((double)n - (double)nP) / ((double)nP - 1.0);
#if PF_SEM_CPU_TU
        p.out[out_idx] = (s2 <= 0.0) ? 0.0f : (float)(scale * (s1 / s2));
#else
        p.out[out_idx] = (float)(scale * (s1 / (s2 <= 0.0 ? 0.0 : s2)));
#endif
    }
    }  // a live cell
    }  // rounds
    stamp_end(p, item);
}

// One CTA per item of the device work queue (see WorkQueue); an item is
// ROUNDS x CELLS x BLOCK consecutive periods.  (Persistent CTAs measured 1-8%
// slower in every class.)
template <int ALGO, bool CNT16, int BLOCK, bool REF_STATS, int ROUNDS, int CELLS, bool MIXED>
__global__ void __launch_bounds__(BLOCK, bin_min_blocks<ALGO, BLOCK, CELLS>())
    bin_kernel(const FoldParams p) {
    bin_item<ALGO, CNT16, BLOCK, REF_STATS, ROUNDS, CELLS, MIXED>(
        p, queue_item<BLOCK * ROUNDS * CELLS>(p, blockIdx.x), blockIdx.x);
}

// CE times sorted by magnitude column, for bin_kernel: equal columns lie
// together, so the kernel keeps a column's counter address and increment in
// registers for the whole run and a staged point is its time alone (8 bytes
// instead of a 16-byte record).  Counts do not depend on the order.  Per
// curve: ts = the runs one after the other, each padded to a multiple of 4
// with repeats of its first time; runs = {padded total, then one word
// (column << 16) | length per non-empty column, then 0}.  cols = the column of
// each point in the curve's own order, for the MIXED form.
__global__ void __launch_bounds__(256)
    ce_sort_kernel(const float* __restrict__ t, const float* __restrict__ m,
                   const CurveDesc* __restrict__ curves, uint32_t n_curves, uint32_t n_mag,
                   float mag_bin_size, CeSortLayout lay, float* __restrict__ ts,
                   uint32_t* __restrict__ runs, uint16_t* __restrict__ cols) {
    extern __shared__ uint32_t sort_cnt[];  // [n_mag] counts, [n_mag] write positions
    uint32_t* sort_pos = sort_cnt + n_mag;
    const uint32_t c = blockIdx.x;
    if (c >= n_curves) return;
    const CurveDesc cd = curves[c];
    float* tc = ts + (cd.off * lay.ts_mul + (int64_t)c * lay.ts_pad);
    uint32_t* rc = runs + (cd.off * lay.run_mul + (int64_t)c * lay.run_pad);
    // MagBin (periodfind/cuda/ce.cu:70-72; rust/src/ce.rs:79).
    auto column = [&](uint32_t i) -> uint32_t {
        const unsigned long long mb64 =
            static_cast<unsigned long long>(m[cd.off + i] / mag_bin_size);
        return (uint32_t)(mb64 % n_mag);
    };
    for (uint32_t k = threadIdx.x; k < n_mag; k += 256) sort_cnt[k] = 0u;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < cd.n; i += 256) {
        const uint32_t k = column(i);
        cols[cd.off + i] = (uint16_t)k;
        atomicAdd(&sort_cnt[k], 1u);
    }
    for (uint32_t i = cd.n + threadIdx.x; i < ((cd.n + 3u) & ~3u); i += 256) cols[cd.off + i] = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t at = 0, r = 0;
        for (uint32_t k = 0; k < n_mag; k++) {
            const uint32_t len = sort_cnt[k];
            sort_pos[k] = at;
            if (len) rc[1 + r++] = (k << 16) | len;
            at += (len + 3u) & ~3u;
        }
        rc[1 + r] = 0u;
        rc[0] = at;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < cd.n; i += 256)
        tc[atomicAdd(&sort_pos[cols[cd.off + i]], 1u)] = t[cd.off + i];
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < n_mag; k += 256) {
        const uint32_t len = sort_cnt[k], end = sort_pos[k];
        if (!len) continue;
        const float first = tc[end - len];
        for (uint32_t e = end; e < end - len + ((len + 3u) & ~3u); e++) tc[e] = first;
    }
}

// CE per-point bin data of the shared-histogram kernel (pf_binwarp.cuh):
// {16-bit counter word of the magnitude column, increment}.
__global__ void ce_binaux_kernel(const float* __restrict__ m, uint2* __restrict__ aux,
                                 const CurveDesc* __restrict__ curves, uint32_t n_curves,
                                 uint32_t n_mag, float mag_bin_size) {
    const uint32_t c = blockIdx.x;
    if (c >= n_curves) return;
    const CurveDesc cd = curves[c];
    const uint32_t n4 = (cd.n + 3u) & ~3u;
    for (uint32_t i = threadIdx.x; i < n4; i += blockDim.x) {
        uint2 v = make_uint2(0u, 0u);
        if (i < cd.n) {
            // MagBin (periodfind/cuda/ce.cu:70-72; rust/src/ce.rs:79).
            const unsigned long long mb64 =
                static_cast<unsigned long long>(m[cd.off + i] / mag_bin_size);
            const uint32_t mb = (uint32_t)(mb64 % n_mag);
            v.x = mb >> 1;
            v.y = (mb & 1u) ? 0x10000u : 1u;
        }
        aux[cd.off + i] = v;
    }
}

}  // namespace PF_KNS
}  // namespace pfk
