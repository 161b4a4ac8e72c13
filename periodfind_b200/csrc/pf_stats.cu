// pf_stats.cu -- the 'stats' output on the device: per periodogram row, the
// values the reference computes on the host with numpy
// (periodfind/__init__.py:338-400, Statistics.statistics_from_data):
//   mean   = np.mean(data), std = np.std(data)   (float32, numpy's pairwise
//            summation order: leaves of <= 128 elements summed with eight
//            accumulators, halves split at multiples of 8, as np.add.reduce)
//   median = np.median(data), mad = np.median(|data - median|)
//            (exact order statistics; the mean of the two middle values for
//            an even count; NaN anywhere gives NaN, as numpy)
//   the n best entries (smallest for CE, largest otherwise; NaN ranks
//            largest, as np.argpartition), best first.
//
// One CTA per curve.  The row is staged in shared memory where it fits, so
// its dozen passes do not go to L2.  Order statistics by selection over
// order-preserving keys, in slices of the row's own key range.  What bounded
// the earlier form was serial work of one thread (the list of summation
// leaves, a 256-bin scan per radix digit, the search for the best cell's
// index) and, up to 8192 cells, a bitonic sort; all of it is now done by the
// whole CTA: 400 rows of 20000 cells 2.02 -> 0.10 ms, 100 rows of 1000
// 36 -> 15 us.  Bound: latency of the passes (two barriers each).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "pf_launch.h"

namespace pfk {

namespace {

constexpr int kStatThreads = 512;
constexpr int kPrepThreads = 256;
constexpr uint32_t kBins = 2048;
constexpr size_t kStageBytes = 190 * 1024;  // a longer row is read from global memory
constexpr int kLeaf = 128;  // numpy's pairwise block size

// Order-preserving key of a float (NaN ranks above +inf, as in numpy sorts).
__device__ __forceinline__ uint32_t fkey(float v) {
    if (isnan(v)) return 0xFFFFFFFFu;
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unkey(uint32_t k) {
    if (k == 0xFFFFFFFFu) return __uint_as_float(0x7FC00000u);
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// The element transform of each pass: the row itself, its squared deviation
// from the mean (np.std), or its absolute deviation from the median (MAD).
enum : int { T_X = 0, T_SQDEV = 1, T_ABSDEV = 2 };
__device__ __forceinline__ float elem(const float* x, uint32_t i, int tr, float ref) {
    const float v = x[i];
    if (tr == T_SQDEV) {
        const float d = __fsub_rn(v, ref);
        return __fmul_rn(d, d);
    }
    if (tr == T_ABSDEV) return fabsf(__fsub_rn(v, ref));
    return v;
}


// numpy's recursion as a binary tree of depth `depth` (every node there is a
// leaf): the node reached by path `q` (its top `d` bits first) at depth d.
__device__ __forceinline__ void tree_node(uint32_t n, uint32_t q, uint32_t d, uint32_t& lo,
                                          uint32_t& m, uint32_t& leaf_at) {
    lo = 0;
    m = n;
    leaf_at = d;
    for (uint32_t b = 0; b < d; b++) {
        if (m <= (uint32_t)kLeaf) {
            leaf_at = b;
            return;
        }
        uint32_t n2 = m / 2;
        n2 -= n2 % 8;
        if ((q >> (d - 1 - b)) & 1u) {
            lo += n2;
            m -= n2;
        } else {
            m = n2;
        }
    }
}

// Depth of that tree: a node of m elements splits into parts of at most
// m / 2 + 8.
__host__ __device__ inline uint32_t tree_depth(uint32_t n) {
    uint32_t depth = 0;
    for (uint32_t m = n; m > (uint32_t)kLeaf; m = m / 2 + 8) depth++;
    return depth;
}

// np.add.reduce of the transformed row, all THREADS threads participating:
// eight lanes per leaf (numpy's eight accumulators; fewer than 8 elements are
// summed one by one from -0.0), then the tree level by level.  node: 2^depth
// floats.
template <int THREADS>
__device__ float pairwise_tree(const float* x, uint32_t n, int tr, float ref, uint32_t depth,
                               float* node) {
    const uint32_t lane8 = threadIdx.x & 7u, paths = 1u << depth;
    for (uint32_t g0 = (threadIdx.x >> 5) * 4u; g0 < paths; g0 += THREADS / 8) {
        const uint32_t g = g0 + ((threadIdx.x & 31u) >> 3);
        uint32_t lo, m, at;
        tree_node(n, g, depth, lo, m, at);
        // A leaf above the last level is summed by its all-left path only.
        const bool mine = g < paths && (g & ((1u << (depth - at)) - 1u)) == 0u;
        const uint32_t full = m < 8 ? 0u : m - (m % 8);
        float r = 0.0f;
        if (mine && full) {
            r = elem(x, lo + lane8, tr, ref);
            for (uint32_t i = 8; i < full; i += 8)
                r = __fadd_rn(r, elem(x, lo + i + lane8, tr, ref));
        }
        __syncwarp();
        r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 1));
        r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 2));
        r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 4));
        if (mine && lane8 == 0) {
            if (!full) r = -0.0f;
            for (uint32_t i = full; i < m; i++) r = __fadd_rn(r, elem(x, lo + i, tr, ref));
            node[g] = r;
        }
    }
    for (int d = (int)depth - 1; d >= 0; d--) {
        __syncthreads();
        const uint32_t step = 1u << (depth - d);
        for (uint32_t q = threadIdx.x; q < (1u << d); q += THREADS) {
            uint32_t lo, m, at;
            tree_node(n, q, (uint32_t)d, lo, m, at);
            if (m > (uint32_t)kLeaf)
                node[q * step] = __fadd_rn(node[q * step], node[q * step + step / 2]);
        }
    }
    __syncthreads();
    const float r = node[0];
    __syncthreads();
    return r;
}

// Key of the k-th smallest transformed element (0-based), whose key lies in
// [key_lo, key_hi], and how many elements have a key <= it: histograms of
// up to kBins equal slices of the key range, narrowed to the slice that
// holds the rank.  All threads participate.
__device__ uint32_t select_key(const float* x, uint32_t n, int tr, float ref, uint32_t k,
                                uint32_t key_lo, uint32_t key_hi, uint32_t* hist,
                                uint32_t* n_le) {
    __shared__ uint32_t s_warp[kStatThreads / 32], s_bin, s_before, s_count;
    constexpr uint32_t kPer = kBins / kStatThreads;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    uint32_t base = key_lo, width = key_hi - key_lo, below = 0;
    for (;;) {
        const int bits = 32 - __clz(width);
        const int shift = bits > 11 ? bits - 11 : 0;
        for (uint32_t b = threadIdx.x; b < kBins; b += kStatThreads) hist[b] = 0u;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += kStatThreads) {
            const uint32_t d = fkey(elem(x, i, tr, ref)) - base;
            if (d <= width) atomicAdd(&hist[d >> shift], 1u);
        }
        __syncthreads();
        uint32_t mine[kPer], sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < kPer; j++) sum += mine[j] = hist[threadIdx.x * kPer + j];
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (uint32_t)o) inc += v;
        }
        if (lane == 31) s_warp[wid] = inc;
        __syncthreads();
        uint32_t before = below + inc - sum;
        for (uint32_t w = 0; w < wid; w++) before += s_warp[w];
        // Exactly one thread's bins hold rank k.
        if (k >= before && k < before + sum) {
            uint32_t j = 0;
            while (k >= before + mine[j]) before += mine[j++];
            s_bin = threadIdx.x * kPer + j;
            s_before = before;
            s_count = mine[j];
        }
        __syncthreads();
        const uint32_t bin = s_bin;
        below = s_before;
        const uint32_t count = s_count;
        __syncthreads();
        if (shift == 0) {
            *n_le = below + count;
            return base + bin;
        }
        const uint32_t top = base + width;
        base += bin << shift;
        width = min((1u << shift) - 1u, top - base);
    }
}

// np.median of the transformed row without NaN.
__device__ float median_row(const float* x, uint32_t n, int tr, float ref, uint32_t key_lo,
                             uint32_t key_hi, uint32_t* hist) {
    const uint32_t k1 = (n - 1) / 2;
    uint32_t le;
    const uint32_t a = select_key(x, n, tr, ref, k1, key_lo, key_hi, hist, &le);
    if (n % 2) return unkey(a);
    uint32_t b = a;
    if (le < k1 + 2) {  // the next larger key
        __shared__ uint32_t s_next;
        if (threadIdx.x == 0) s_next = 0xFFFFFFFFu;
        __syncthreads();
        uint32_t nx = 0xFFFFFFFFu;
        for (uint32_t i = threadIdx.x; i < n; i += kStatThreads) {
            const uint32_t kk = fkey(elem(x, i, tr, ref));
            if (kk > a) nx = min(nx, kk);
        }
        nx = __reduce_min_sync(0xffffffffu, nx);
        if ((threadIdx.x & 31) == 0) atomicMin(&s_next, nx);
        __syncthreads();
        b = s_next;
        __syncthreads();
    }
    // the mean of the two middle values: np.mean of a two-element array
    return __fdiv_rn(__fadd_rn(__fadd_rn(-0.0f, unkey(a)), unkey(b)), 2.0f);
}

__global__ void __launch_bounds__(kStatThreads)
    stats_kernel(const float* __restrict__ pg, uint32_t n, int use_max, uint32_t n_top,
                      uint32_t depth, int staged, float* __restrict__ stats,
                      int64_t* __restrict__ top_idx, float* __restrict__ top_val) {
    extern __shared__ __align__(16) unsigned char ssm[];
    __shared__ uint32_t hist[kBins];
    __shared__ uint32_t s_lo, s_hi, s_cnt, s_warp[kStatThreads / 32];
    __shared__ unsigned long long s_best;
    float* node = reinterpret_cast<float*>(ssm);
    const uint64_t c = blockIdx.x;
    const float* x = pg + c * (uint64_t)n;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;

    // Stage the row; smallest and largest key; the best cell (lowest index
    // among equals).  A NaN's key is the largest of all.
    if (threadIdx.x == 0) {
        s_lo = 0xFFFFFFFFu;
        s_hi = 0u;
        s_best = ~0ull;
    }
    __syncthreads();
    {
        float* xs = reinterpret_cast<float*>(ssm + ((size_t)4 << depth));
        uint32_t lo = 0xFFFFFFFFu, hi = 0u;
        unsigned long long best = ~0ull;
        for (uint32_t i = threadIdx.x; i < n; i += kStatThreads) {
            const float v = x[i];
            if (staged) xs[i] = v;
            const uint32_t k = fkey(v);
            lo = min(lo, k);
            hi = max(hi, k);
            const unsigned long long r = ((unsigned long long)(use_max ? ~k : k) << 32) | i;
            best = r < best ? r : best;
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long r = __shfl_xor_sync(0xffffffffu, best, o);
            best = r < best ? r : best;
        }
        if (lane == 0) {
            atomicMin(&s_lo, lo);
            atomicMax(&s_hi, hi);
            atomicMin(&s_best, best);
        }
        if (staged) x = xs;
    }
    __syncthreads();
    const uint32_t key_lo = s_lo, key_hi = s_hi;
    const bool any_nan = key_hi == 0xFFFFFFFFu;

    // np.mean, then np.std as in numpy's _var: mean kept as float32, the
    // squared deviations summed pairwise, divided by n, square root.
    const float fn = (float)n;
    const float mean = __fdiv_rn(pairwise_tree<kStatThreads>(x, n, T_X, 0.0f, depth, node), fn);
    const float ssq = pairwise_tree<kStatThreads>(x, n, T_SQDEV, mean, depth, node);
    float med = __uint_as_float(0x7FC00000u), mad = med;
    if (!any_nan) {
        med = median_row(x, n, T_X, 0.0f, key_lo, key_hi, hist);
        // The largest deviation is at one end of the row's range (rounding is
        // monotone); infinities can give NaN deviations, which rank last.
        const float e1 = fabsf(__fsub_rn(unkey(key_lo), med));
        const float e2 = fabsf(__fsub_rn(unkey(key_hi), med));
        const uint32_t dev_hi =
            isinf(e1) || isinf(e2) || isnan(e1) || isnan(e2) ? 0xFFFFFFFFu : fkey(fmaxf(e1, e2));
        mad = median_row(x, n, T_ABSDEV, med, 0x80000000u, dev_hi, hist);
    }
    if (threadIdx.x == 0) {
        stats[4 * c + 0] = mean;
        stats[4 * c + 1] = __fsqrt_rn(__fdiv_rn(ssq, fn));
        stats[4 * c + 2] = med;
        stats[4 * c + 3] = mad;
    }

    // The n_top best, best first, lowest index first among equals.
    if (n_top == 0) return;
    int64_t* ti = top_idx + c * n_top;
    const uint32_t m = min(n_top, n);
    if (m == 1) {
        if (threadIdx.x == 0) {
            const uint32_t i = (uint32_t)s_best;
            ti[0] = i;
            top_val[c * n_top] = x[i];
        }
    } else {
        // The key of the m-th best as a threshold; the cells strictly better
        // (fewer than m), then the lowest-index ties.
        uint32_t le;
        const uint32_t thr =
            select_key(x, n, T_X, 0.0f, use_max ? n - m : m - 1, key_lo, key_hi, hist, &le);
        if (threadIdx.x == 0) s_cnt = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += kStatThreads) {
            const uint32_t kk = fkey(x[i]);
            if (use_max ? kk > thr : kk < thr) ti[atomicAdd(&s_cnt, 1u)] = i;
        }
        __syncthreads();
        uint32_t have = s_cnt;
        for (uint32_t i0 = 0; i0 < n && have < m; i0 += kStatThreads) {
            const uint32_t i = i0 + threadIdx.x;
            const bool tie = i < n && fkey(x[i]) == thr;
            const unsigned b = __ballot_sync(0xffffffffu, tie);
            if (lane == 0) s_warp[wid] = __popc(b);
            __syncthreads();
            uint32_t at = have, all = 0;
            for (uint32_t w = 0; w < kStatThreads / 32; w++) {
                if (w < wid) at += s_warp[w];
                all += s_warp[w];
            }
            at += __popc(b & ((1u << lane) - 1u));
            if (tie && at < m) ti[at] = i;
            have += all;
            __syncthreads();
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            // Best first (insertion sort on (key, index); m is small).
            for (uint32_t a = 1; a < m; a++) {
                const int64_t v = ti[a];
                const uint32_t kv = fkey(x[v]);
                int b = (int)a - 1;
                while (b >= 0) {
                    const uint32_t kb = fkey(x[ti[b]]);
                    const bool after = use_max ? (kb < kv || (kb == kv && ti[b] > v))
                                               : (kb > kv || (kb == kv && ti[b] > v));
                    if (!after) break;
                    ti[b + 1] = ti[b];
                    b--;
                }
                ti[b + 1] = v;
            }
            for (uint32_t a = 0; a < m; a++) top_val[c * n_top + a] = x[ti[a]];
        }
    }
    for (uint32_t a = m + threadIdx.x; a < n_top; a += kStatThreads) {
        ti[a] = -1;
        top_val[c * n_top + a] = 0.0f;
    }
}

// Magnitude preparation on the device, a CTA per curve, with the values
// the reference's prepare_magnitudes gets from numpy (periodfind/_utils.py:
// 29-45): kind 1 centres, m - np.mean(m) (numpy's pairwise float32 sum
// divided by n); kind 2 normalises, ((m - min) / (max - min)) * 0.999 +
// 5e-4 in float32 with NaN propagating through min / max.  Curve c is
// m[off[c] .. off[c+1]); its output goes to the same place in out.
__global__ void __launch_bounds__(kPrepThreads)
    prep_mags_kernel(const float* __restrict__ m, const int64_t* __restrict__ off, int kind,
                     float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char psm[];
    __shared__ float s_lo[kPrepThreads / 32], s_hi[kPrepThreads / 32];
    __shared__ int s_nan;
    const uint64_t c = blockIdx.x;
    const int64_t lo = off[c];
    const uint32_t n = (uint32_t)(off[c + 1] - lo);
    if (n == 0) return;  // uniform over the CTA
    const float* x = m + lo;
    float* y = out + lo;
    if (kind == 1) {
        const float sum = pairwise_tree<kPrepThreads>(x, n, T_X, 0.0f, tree_depth(n),
                                                      reinterpret_cast<float*>(psm));
        const float mean = __fdiv_rn(sum, (float)n);
        for (uint32_t i = threadIdx.x; i < n; i += kPrepThreads) y[i] = __fsub_rn(x[i], mean);
        return;
    }
    // np.min / np.max: exact, any order; NaN anywhere gives NaN.
    float mn = INFINITY, mx = -INFINITY;
    int nan_local = 0;
    for (uint32_t i = threadIdx.x; i < n; i += kPrepThreads) {
        const float v = x[i];
        nan_local |= isnan(v) ? 1 : 0;
        mn = fminf(mn, v);
        mx = fmaxf(mx, v);
    }
    if (threadIdx.x == 0) s_nan = 0;
    __syncthreads();
    if (nan_local) atomicOr(&s_nan, 1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        s_lo[threadIdx.x >> 5] = mn;
        s_hi[threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    float cmin = s_lo[0], cmax = s_hi[0];
    for (int w = 1; w < kPrepThreads / 32; w++) {
        cmin = fminf(cmin, s_lo[w]);
        cmax = fmaxf(cmax, s_hi[w]);
    }
    if (s_nan) cmin = cmax = __uint_as_float(0x7FC00000u);
    const float range = __fsub_rn(cmax, cmin);
    for (uint32_t i = threadIdx.x; i < n; i += kPrepThreads)
        y[i] = __fadd_rn(__fmul_rn(__fdiv_rn(__fsub_rn(x[i], cmin), range), 0.999f), 5e-4f);
}

}  // namespace

uint32_t stats_leaf_count(uint32_t n) {
    // The number of leaves of numpy's recursion over n elements (host side).
    uint32_t count = 0;
    uint32_t stack[64];
    int sp = 0;
    stack[sp++] = n;
    while (sp > 0) {
        const uint32_t m = stack[--sp];
        if (m <= (uint32_t)kLeaf) {
            count++;
            continue;
        }
        uint32_t n2 = m / 2;
        n2 -= n2 % 8;
        stack[sp++] = m - n2;
        stack[sp++] = n2;
    }
    return count;
}

cudaError_t launch_stats(const float* pg, uint64_t n_curves, uint32_t n_cells, int use_max,
                         uint32_t n_top, float* stats, int64_t* top_idx, float* top_val,
                         cudaStream_t s) {
    if (n_curves == 0) return cudaSuccess;
    const uint32_t depth = tree_depth(n_cells);
    size_t smem = (size_t)4 << depth;
    const size_t with_row = smem + (size_t)n_cells * 4;
    const int staged = with_row <= kStageBytes;
    if (staged) smem = with_row;
    if (smem > kStageBytes) return cudaErrorInvalidValue;
    cudaError_t e = allow_smem(stats_kernel, smem);
    if (e != cudaSuccess) return e;
    stats_kernel<<<(unsigned)n_curves, kStatThreads, smem, s>>>(
        pg, n_cells, use_max, n_top, depth, staged, stats, top_idx, top_val);
    return cudaGetLastError();
}

cudaError_t launch_prep_mags(const float* m, const int64_t* d_off, uint64_t n_curves,
                             uint32_t max_len, int kind, float* out, cudaStream_t s) {
    if (n_curves == 0) return cudaSuccess;
    if (kind != 1 && kind != 2) return cudaErrorInvalidValue;
    if (n_curves > 0x7FFFFFFFull) return cudaErrorInvalidValue;
    const size_t smem = kind == 1 ? (size_t)4 << tree_depth(max_len) : 0;
    if (smem > 200u * 1024u) return cudaErrorInvalidValue;
    cudaError_t e = allow_smem(prep_mags_kernel, smem);
    if (e != cudaSuccess) return e;
    prep_mags_kernel<<<(unsigned)n_curves, kPrepThreads, smem, s>>>(m, d_off, kind, out);
    return cudaGetLastError();
}

}  // namespace pfk
