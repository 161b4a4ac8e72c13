// pf_fpw.cuh -- FPW (fast phase-folding weighted) and BLS periodograms, included by
// each arithmetic unit after pf_fold.cuh and pf_bin.cuh.
//
// Statistic (rust/src/fpw.rs:12-66; periodfind/cuda/fpw.cu:45-224): each
// point carries an inverse variance w = 1 / err^2 and w * m; the fold puts
// it in one of n_bins phase bins; per bin V = sum w, Y = sum w * m; the
// value is sum over bins with V > 0 of Y^2 / (2 V).  Maximum is best.
//
// Decomposition: a CTA per (curve, period derivative, tile of BLOCK trial
// periods); thread j owns one period (the chosen form: two) for the whole curve and keeps its own
// V and Y in shared memory ([bin][thread], so a warp's updates touch
// consecutive words), adding the
// points in curve order -- the Rust path's order, so the sums round as it
// does.  The curve streams through shared memory in 16-byte point records,
// 256 points per tile.
//
// The bin is the reference's for the unit's semantics:
//   CUDA build: (size_t)(folded / bin_size), clamped to n_bins - 1
//               (fpw.cu:28-30, 115-117);
//   Rust path:  (folded * n_bins) as usize, clamped (fpw.rs:44);
// with folded = (float)|q - floor(q)| for the correctly rounded quotient q.
//
// Plain form: that sequence for every point (FP64 divide).  Chosen form: the
// CE / AOV bin kernel's fast bin, the reference sequence within the proven
// guard of a bin edge (divide-free, the same quotient).
#pragma once

#ifndef PF_KNS
#error "include after defining PF_KNS"
#endif

namespace pfk {
namespace PF_KNS {

constexpr uint32_t kFpwTile = 256;

// The reference's bin of a folded phase, with this unit's arithmetic.
__device__ __forceinline__ uint32_t fpw_ref_bin(float folded, const FpwParams& p) {
#if PF_SEM_CPU_TU
    const uint32_t b = trunc_u(folded * (float)p.n_bins);
#else
    const uint32_t b = trunc_u(folded / p.bin_size);
#endif
    return min(b, p.n_bins - 1u);
}

// BLS (Box Least Squares, rust/src/bls.rs:19-134; periodfind/cuda/bls.cu:
// 56-308) shares the binning: the second sum is w * (m - weighted mean), the
// bins sit one row down so that row 0 holds the zero of the prefix sums, and
// the value is the best s^2 / (r (W - r)) over the windows of nb_min ..
// nb_max consecutive bins (wrapping) whose weight fraction r / W lies in
// (0, 1); 0 when W <= 0.
//
// FPW value of one cell from its bins (row k: ld(k) = (V, Y)).
template <class LD>
__device__ __forceinline__ float fpw_value(LD&& ld, uint32_t nb) {
    float acc = 0.0f;
    for (uint32_t k = 0; k < nb; k++) {
        const float2 x = ld(k);
        if (x.x > 0.0f) acc += x.y * x.y / (2.0f * x.x);
    }
    return acc;
}

// BLS values of CELLS cells at once (row k of cell c: ld(k, c), put(k, c, x)).
// Prefix sums in place, in the reference's order (bls.rs:83-89): row k + 1
// becomes row k + row k + 1.  Then every (phase, width) window, phase-major:
// the window's start row is read once per phase.  The sums are the
// reference's: end <= nb gives row[end] - row[phi] (x - y is x + (-y)
// exactly), a wrapping window (total - row[phi]) + row[end - nb]; the maximum
// does not depend on the order of the windows.
template <int CELLS, class LD, class PUT>
__device__ __forceinline__ void bls_values(LD&& ld, PUT&& put, uint32_t nb, uint32_t nb_min,
                                           uint32_t nb_max, float (&acc)[CELLS]) {
    float2 tot[CELLS];
#pragma unroll
    for (int c = 0; c < CELLS; c++) {
        tot[c] = ld(0, c);
        acc[c] = 0.0f;
    }
    for (uint32_t k = 0; k < nb; k++)
#pragma unroll
        for (int c = 0; c < CELLS; c++) {
            float2 x = ld(k + 1, c);
            x.x = tot[c].x + x.x;
            x.y = tot[c].y + x.y;
            put(k + 1, c, x);
            tot[c] = x;
        }
    for (uint32_t phi = 0; phi < nb; phi++) {
        float2 a[CELLS], rest[CELLS];
#pragma unroll
        for (int c = 0; c < CELLS; c++) {
            a[c] = ld(phi, c);
            rest[c] = make_float2(tot[c].x - a[c].x, tot[c].y - a[c].y);
        }
        // The windows that end in rows lo .. hi (consecutive), their sums
        // row + base.  No branch in the loop, so that the loads and divides of
        // several windows overlap (a cell outside the weight range scores 0,
        // and a NaN score leaves the maximum as a comparison would).
        auto windows = [&](uint32_t lo, uint32_t hi, const float2 (&base)[CELLS]) {
#pragma unroll 4
            for (uint32_t k = lo; k <= hi; k++) {
#pragma unroll
                for (int c = 0; c < CELLS; c++) {
                    const float2 e = ld(k, c);
                    const float r = e.x + base[c].x, sy = e.y + base[c].y;
                    const float r_frac = r / tot[c].x;
                    const float bls = (sy * sy) / (r * (tot[c].x - r));
                    acc[c] = fmaxf(acc[c], r_frac > 0.0f && r_frac < 1.0f ? bls : 0.0f);
                }
            }
        };
        float2 minus[CELLS];
#pragma unroll
        for (int c = 0; c < CELLS; c++) minus[c] = make_float2(-a[c].x, -a[c].y);
        windows(phi + nb_min, min(phi + nb_max, nb), minus);
        // Wrapping: widths of at least nb - phi + 1.
        if (phi + nb_max > nb)
            windows(max(phi + nb_min, nb + 1u) - nb, phi + nb_max - nb, rest);
    }
    // No weight, no window.
#pragma unroll
    for (int c = 0; c < CELLS; c++)
        if (!(tot[c].x > 0.0f)) acc[c] = 0.0f;
}

// The plain form.
template <int BLOCK, bool BLS>
__global__ void __launch_bounds__(BLOCK)
    fpw_kernel(const FpwParams p, uint32_t tiles_per_row) {
    // One 16-byte record per staged point: a single 128-bit shared load.
    struct alignas(16) Point {
        float t, iv, ivy;
    };
    constexpr uint32_t kRow0 = BLS ? 1u : 0u;  // rows before bin 0
    extern __shared__ __align__(16) unsigned char fsm[];
    Point* st = reinterpret_cast<Point*>(fsm);
    // Per-thread bins: V rows then Y rows, row k (bin k - kRow0) of thread tid.
    float* bins = reinterpret_cast<float*>(st + kFpwTile);
    const uint32_t rows = p.n_bins + kRow0;
    auto ld = [&](uint32_t k) -> float2 {
        return make_float2(bins[k * BLOCK + threadIdx.x], bins[(rows + k) * BLOCK + threadIdx.x]);
    };
    auto put = [&](uint32_t k, float2 x) {
        bins[k * BLOCK + threadIdx.x] = x.x;
        bins[(rows + k) * BLOCK + threadIdx.x] = x.y;
    };

    const uint64_t cta = blockIdx.x;
    const uint32_t tile = (uint32_t)(cta % tiles_per_row);
    const uint64_t row = cta / tiles_per_row;     // curve * n_pdt + pdt
    const uint64_t c = row / p.n_pdt;
    const uint32_t d = (uint32_t)(row % p.n_pdt);
    const int tid = threadIdx.x;
    const uint64_t pi = (uint64_t)tile * BLOCK + tid;
    const bool active = pi < p.n_per;

    const int64_t off = p.off[c];
    const uint32_t n = p.len[c];
    const uint32_t nb = p.n_bins;
    for (uint32_t k = 0; k < rows; k++) put(k, make_float2(0.0f, 0.0f));
    Cell s;
    cell_setup<FOLD_REF>(s, p.periods[active ? pi : (uint64_t)tile * BLOCK], p.pdts[d]);

    for (uint32_t base = 0; base < n; base += kFpwTile) {
        const uint32_t cnt = min(kFpwTile, n - base);
        __syncthreads();
        for (uint32_t i = tid; i < cnt; i += BLOCK)
            st[i] = Point{p.t[off + base + i], p.iv[off + base + i], p.ivy[off + base + i]};
        __syncthreads();
        if (!active) continue;
#pragma unroll 4
        for (uint32_t i = 0; i < cnt; i++) {
            const Point pt = st[i];
            const uint32_t bin = fpw_ref_bin(fold_ref(pt.t, s), p) + kRow0;
            float2 x = ld(bin);
            x.x += pt.iv;
            x.y += pt.ivy;
            put(bin, x);
        }
    }
    if (!active) return;
    float acc[1];
    if constexpr (BLS)
        bls_values<1>([&](uint32_t k, int) { return ld(k); },
                      [&](uint32_t k, int, float2 x) { put(k, x); }, nb, p.nb_min, p.nb_max, acc);
    else
        acc[0] = fpw_value(ld, nb);
    p.out[(uint64_t)c * (p.n_per * p.n_pdt) + pi * p.n_pdt + d] = acc[0];
}

// The chosen form: the bin from the one-FMA construction of the CE / AOV
// bin kernel (pf_bin.cuh, fast_bin32: the guard rides in the FMA's constant,
// so a point's edge test is its product's low word against a limit), a
// thread holding CELLS trial periods, whose updates share the staged
// point's load (2 up to 32 bins; 1 beyond, where shared memory holds so few
// cells that the warps are needed to hide latency: BLS(50) kernel 5.2 ms with
// two, 2.8 with one).  Four points are read and binned before the first of their
// read-modify-writes (the staged tile and the bins share one array, so a
// point read cannot move above an earlier bin store); a group with a point
// near an edge corrects that point's bin first, as float sums cannot be
// taken back.  Updates stay in point order (same bin, same rounding).  Beyond
// the one-FMA range the bins of a group are taken together in the same way
// (30 curves x 2000 points x 2000 periods from 0.0005 on: 138 us; a branch and
// the exact sequence at every point took 333, with one period per thread 223).
//
// Bound: the shared-memory pipe, 97% busy for FPW (per evaluation half a
// 128-bit broadcast load, an 8-byte load and an 8-byte store), 76% for BLS.
// FPW(10) with uncertainties, 100 curves x 4096 points x 10000 periods x 2:
// 4.77 ms, the call from host arrays 9.02 -> 6.62 ms; BLS(50), 150 x 1500 x
// 10000, whose 1250 windows per cell cost as much as its points: the call 5.46
// -> 3.74 ms (4.15 ms with one window loop and a select per wrap).
template <int BLOCK, bool BLS, int CELLS>
__global__ void __launch_bounds__(BLOCK)
    fpw_chosen_kernel(const FpwParams p, uint32_t tiles_per_row) {
    struct alignas(16) Point {
        double t;
        float iv, ivy;
    };
    constexpr uint32_t kCols = BLOCK * CELLS;
    constexpr uint32_t kRow0 = BLS ? 1u : 0u;  // rows before bin 0
    extern __shared__ __align__(16) unsigned char fsm[];
    Point* st = reinterpret_cast<Point*>(fsm);
    // (V, Y) of row k (bin k - kRow0) of cell c of thread tid: one 8-byte
    // access per update, a warp's on consecutive words.
    float2* bins = reinterpret_cast<float2*>(st + kFpwTile) + threadIdx.x;
    auto ld = [&](uint32_t k, int c) -> float2 { return bins[k * kCols + c * BLOCK]; };
    auto put = [&](uint32_t k, int c, float2 x) { bins[k * kCols + c * BLOCK] = x; };
    __shared__ double warp_min[BLOCK / 32];

    const uint64_t cta = blockIdx.x;
    const uint32_t tile = (uint32_t)(cta % tiles_per_row);
    const uint64_t row = cta / tiles_per_row;     // curve * n_pdt + pdt
    const uint64_t cv = row / p.n_pdt;
    const uint32_t dt = (uint32_t)(row % p.n_pdt);
    const int tid = threadIdx.x;
    const uint64_t p0 = (uint64_t)tile * kCols, pi0 = p0 + tid;
    const bool active = pi0 < p.n_per;  // a thread with any live cell runs all

    const int64_t off = p.off[cv];
    const uint32_t n = p.len[cv];
    const uint32_t nb = p.n_bins;
    for (uint32_t k = 0; k < nb + kRow0; k++)
#pragma unroll
        for (int c = 0; c < CELLS; c++) put(k, c, make_float2(0.0f, 0.0f));
    const float period_dt = p.pdts[dt];
    Cell s[CELLS];
    double mn = INFINITY;
#pragma unroll
    for (int c = 0; c < CELLS; c++) {
        const uint64_t pi = pi0 + (uint64_t)c * BLOCK;
        const float period = p.periods[pi < p.n_per ? pi : p0];
        cell_setup<FOLD_EXACT>(s[c], period, period_dt);
        mn = fmin(mn, fabs((double)period));
    }

    // The fast bin is exact away from bin edges while |q| * n_bins < 2^30 (the
    // same bound as the chosen CE / AOV kernels), checked for the CTA from
    // max|t| and its smallest |P|.
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    if ((tid & 31) == 0) warp_min[tid >> 5] = mn;
    __syncthreads();
    double pmin = warp_min[0];
#pragma unroll
    for (int k = 1; k < BLOCK / 32; k++) pmin = fmin(pmin, warp_min[k]);
    const double qb =
        p.tmax / pmin + fabs((double)period_dt) * p.tmax * p.tmax / (2.0 * pmin * pmin);
    const bool fast = qb * (double)nb < 1073741824.0;  // 2^30
    const bool fast32 = fast && qb < 524288.0;         // and |q| < 2^19: one FMA

    auto exact_bin = [&](double td, int c) -> uint32_t {
        return fpw_ref_bin(period_dt != 0.0f ? fold_exact<true>(td, s[c])
                                             : fold_exact<false>(td, s[c]),
                           p);
    };
    // RANGE: kF32 one FMA; kFast, beyond it, floor(q' n_bins) - n_bins floor(q')
    // from a round-down floor and a round-down FMA with 20 fraction bits; kAny
    // the reference's sequence for every point.
    enum : int { kAny, kFast, kF32 };
    auto run = [&](auto pdt_tag, auto range_tag) {
        constexpr bool HAS_PDT = decltype(pdt_tag)::value;
        constexpr int RANGE = decltype(range_tag)::value;
        double ys[CELLS], pc[CELLS];
#pragma unroll
        for (int c = 0; c < CELLS; c++) {
            ys[c] = RANGE == kF32 ? s[c].yhi * 4294967296.0 : s[c].yhi;  // exact
            pc[c] = s[c].c;
        }
        // A point's bin and its edge test (near an edge below the limit).
        auto fast_bin = [&](double td, int c, uint32_t& ev) -> uint32_t {
            double a = td;
            if constexpr (HAS_PDT) a = td - pc[c] * td * td;
            uint32_t b;
            if constexpr (RANGE == kF32) {
                const double y = __fma_rd(a, ys[c], p.magic32);
                mul_wide_u32((uint32_t)__double2loint(y), nb, ev, b);
            } else {
                const double qh = __dmul_rn(a, ys[c]);
                const double r = __dadd_rd(qh, kMagic15);
                const double y = __fma_rd(qh, (double)nb * 1048576.0, kMagic15);
                const uint32_t ylo = (uint32_t)__double2loint(y);
                // biased by 2^31 by the magic constant's top mantissa bit
                b = __funnelshift_r(ylo, (uint32_t)__double2hiint(y), 20) +
                    (uint32_t)__double2loint(r) * (0u - nb) - 0x80000000u;
                ev = ylo * 4096u + (p.edge_d << 12);
            }
            return b;
        };
        const uint32_t lim = RANGE == kF32 ? p.edge32_lim : (2u * p.edge_d) << 12;
        // G points from i: their bins, then their updates.
        auto group = [&](auto g_tag, uint32_t i) {
            constexpr int G = decltype(g_tag)::value;
            Point q[G];
            uint32_t b[G][CELLS];
#pragma unroll
            for (int k = 0; k < G; k++) q[k] = st[i + k];
            if constexpr (RANGE != kAny) {
                uint32_t ev[G][CELLS], least = 0xFFFFFFFFu;
#pragma unroll
                for (int k = 0; k < G; k++)
#pragma unroll
                    for (int c = 0; c < CELLS; c++) {
                        b[k][c] = fast_bin(q[k].t, c, ev[k][c]);
                        least = min(least, ev[k][c]);
                    }
                if (least < lim) {
#pragma unroll
                    for (int k = 0; k < G; k++)
#pragma unroll
                        for (int c = 0; c < CELLS; c++)
                            if (ev[k][c] < lim) b[k][c] = exact_bin(q[k].t, c);
                }
            } else {
#pragma unroll
                for (int k = 0; k < G; k++)
#pragma unroll
                    for (int c = 0; c < CELLS; c++) b[k][c] = exact_bin(q[k].t, c);
            }
#pragma unroll
            for (int k = 0; k < G; k++) {
                float2 x[CELLS];
#pragma unroll
                for (int c = 0; c < CELLS; c++) x[c] = ld(b[k][c] + kRow0, c);
#pragma unroll
                for (int c = 0; c < CELLS; c++) {
                    x[c].x += q[k].iv;
                    x[c].y += q[k].ivy;
                }
#pragma unroll
                for (int c = 0; c < CELLS; c++) put(b[k][c] + kRow0, c, x[c]);
            }
        };
        for (uint32_t base = 0; base < n; base += kFpwTile) {
            const uint32_t cnt = min(kFpwTile, n - base);
            __syncthreads();
            for (uint32_t i = tid; i < cnt; i += BLOCK)
                st[i] = Point{(double)p.t[off + base + i], p.iv[off + base + i],
                              p.ivy[off + base + i]};
            __syncthreads();
            if (!active) continue;
            constexpr int kG = 4;
            uint32_t i = 0;
#pragma unroll 1
            for (; i + kG <= cnt; i += kG) group(std::integral_constant<int, kG>{}, i);
#pragma unroll 1
            for (; i < cnt; i++) group(std::integral_constant<int, 1>{}, i);
        }
    };
    using T_ = std::true_type;
    using F_ = std::false_type;
    using Any = std::integral_constant<int, kAny>;
    using Fast = std::integral_constant<int, kFast>;
    using F32 = std::integral_constant<int, kF32>;
    if (!fast) run(F_{}, Any{});  // exact_bin tests the derivative itself
    else if (period_dt != 0.0f) fast32 ? run(T_{}, F32{}) : run(T_{}, Fast{});
    else fast32 ? run(F_{}, F32{}) : run(F_{}, Fast{});

    if (!active) return;
    float acc[CELLS];
    if constexpr (BLS) {
        bls_values<CELLS>(ld, put, nb, p.nb_min, p.nb_max, acc);
    } else {
#pragma unroll
        for (int c = 0; c < CELLS; c++)
            acc[c] = fpw_value([&](uint32_t k) { return ld(k, c); }, nb);
    }
#pragma unroll
    for (int c = 0; c < CELLS; c++) {
        const uint64_t pi = pi0 + (uint64_t)c * BLOCK;
        if (pi < p.n_per)
            p.out[cv * (p.n_per * p.n_pdt) + pi * p.n_pdt + dt] = acc[c];
    }
}

}  // namespace PF_KNS
}  // namespace pfk
