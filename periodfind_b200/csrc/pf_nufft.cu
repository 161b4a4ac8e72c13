// pf_nufft.cu -- Lomb-Scargle sums on a uniform frequency grid by a
// non-uniform FFT.
//
// On the grid f_k = f0 + k df the two sums the power needs,
//     S_k = sum_i y_i e^{2 pi i t_i f_k},   Q_k = sum_i e^{4 pi i t_i f_k}
// (mag_cos + i mag_sin, and cos_cos = (n + Re Q) / 2, cos_sin = Im Q / 2),
// are Fourier sums over points at x_i = t_i df on the unit circle.  The
// direct kernels (pf_lsrec.cuh, pf_fold.cuh) cost n operations per
// frequency.  Here a CTA takes one curve and kNufftModes consecutive
// frequencies around f_c: it spreads the points' values y_i e^{2 pi i t_i f_c}
// onto a grid of twice as many cells with a kernel of width kW cells, takes
// one FFT of the grid in shared memory, and divides each mode by the kernel's
// transform (Dutt and Rokhlin 1993; the kernel exp(beta (sqrt(1 - z^2) - 1))
// and beta = 2.3 kW are those of Barnett, Magland and af Klinteberg 2019,
// whose error at width 8 is about 1e-7 of the norm of the input).  Cost per
// block: two FFTs of 8192 points and about kW grid updates per point,
// whatever the number of frequencies a point is needed at.
//
// Arithmetic: phases and grid positions are reduced in FP64 (the centre
// phase t f_c and t df are good to 1e-11 turns), values, kernel and FFT are
// FP32.  The spreading is exact in any order, so results are the same from run
// to run: a tile of at most 512 points is added to the grid with 32-bit integer
// reductions in units of 2^-31 of the sum of its magnitudes, which bounds every
// cell, and then taken into FP32 registers, a thread holding the 16 cells
// that its first FFT pass needs.  (Float sums kept in order by giving each
// cell to one warp were 2.5 times slower on long curves: 1.52 against 0.59 ms
// for 83 curves of 4096-16384 points x 50000 frequencies.)
//
// Measured, 300 curves of 64-16384 points x 50000 frequencies: 14.95 ms with
// the recurrence, 1.14 ms with this form; error of the power against FP64
// 6.8e-6 and 2.5e-7 (2-norm).  Bound: short curves by the FFTs (about 29000 SM
// cycles a block: barriers and shared memory), long ones by the spreading's
// issue slots (staging arithmetic, 16 reductions per point and sum).  The
// direct sums stay for grids below kNufftMinFreqs and where they are faster
// on the tuner's sample.
//
// Cells where the normal matrix is near singular (f = 0, or a grid frequency
// on which the sampling aliases) amplify any error of the sums, and the
// direct sums there can be exactly singular: those cells are evaluated again
// point by point, a warp per cell.
#define PF_SEM_CPU_TU 0
#define PF_KNS sem_cuda_nufft
#include "pf_fold.cuh"

namespace pfk {
namespace PF_KNS {

constexpr int kM = 8192;                 // grid cells (transform length)
constexpr int kThreads = kM / 16;        // 16 grid cells per thread and pass
constexpr int kW = 8;                    // kernel width in cells
constexpr float kBeta = 2.3f * kW;
constexpr int kTilePts = kThreads;       // points added between two flushes, one per thread
static_assert(kNufftModes == kM / 2, "two grid cells per mode");

// Grid storage: one float skipped every 16, so that the strided stores of
// the first pass fall on different banks.
__device__ __forceinline__ int pad(int i) { return i + (i >> 4); }
constexpr int kPadded = kM + kM / 16;

struct Smem {
    float re[kPadded], im[kPadded];  // while spreading: integers
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
    return make_float2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
    return make_float2(a.x - b.x, a.y - b.y);
}
// Four-point transform with positive exponent, in place.
__device__ __forceinline__ void fft4(float2& x0, float2& x1, float2& x2, float2& x3) {
    const float2 a = cadd(x0, x2), b = csub(x0, x2), c = cadd(x1, x3), e = csub(x1, x3);
    const float2 d = make_float2(-e.y, e.x);
    x0 = cadd(a, c);
    x1 = cadd(b, d);
    x2 = csub(a, c);
    x3 = csub(b, d);
}
// Sixteen-point transform with positive exponent: X[k] ends in v[k].
__device__ __forceinline__ void fft16(float2 (&v)[16]) {
    constexpr float c1 = 0.92387953251128674f, s1 = 0.38268343236508977f;
    constexpr float h = 0.70710678118654752f;
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) fft4(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
    // v[4 k1 + n2] times e^{2 pi i n2 k1 / 16}
    v[5] = cmul(v[5], make_float2(c1, s1));
    v[6] = cmul(v[6], make_float2(h, h));
    v[7] = cmul(v[7], make_float2(s1, c1));
    v[9] = cmul(v[9], make_float2(h, h));
    v[10] = make_float2(-v[10].y, v[10].x);
    v[11] = cmul(v[11], make_float2(-h, h));
    v[13] = cmul(v[13], make_float2(s1, c1));
    v[14] = cmul(v[14], make_float2(-h, h));
    v[15] = cmul(v[15], make_float2(-c1, -s1));
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) fft4(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
    // X[k1 + 4 k2] is in v[4 k1 + k2]: transpose.
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = a + 1; b < 4; b++) {
            const float2 t = v[4 * a + b];
            v[4 * a + b] = v[4 * b + a];
            v[4 * b + a] = t;
        }
}

// One radix-16 pass of the self-sorting FFT over the grid: sub-transforms of
// length NS become ones of length 16 NS.  The first (NS = 1) takes its input
// in v, the others from the grid.
// Twiddles come from a table of e^{2 pi i k / kM} rounded from FP64: six of a
// pass's fifteen are read, the others are one product of two of them (powers
// of the first by repeated products cost a fifth of the result's accuracy).
template <int NS>
__device__ __forceinline__ void pass16(Smem& sm, const float2* __restrict__ tw,
                                       float2 (&v)[16]) {
    const int tid = threadIdx.x;
    const int q = tid % NS;
    if constexpr (NS > 1) {
#pragma unroll
        for (int r = 0; r < 16; r++) {
            const int i = pad(tid + r * kThreads);
            v[r] = make_float2(sm.re[i], sm.im[i]);
        }
        constexpr int kStep = kM / (16 * NS);
        float2 w[4], w4[4];
#pragma unroll
        for (int r = 1; r < 4; r++) {
            w[r] = __ldg(tw + q * r * kStep);
            w4[r] = __ldg(tw + q * 4 * r * kStep);
        }
#pragma unroll
        for (int r = 1; r < 16; r++) {
            const float2 f = r < 4 ? w[r & 3] : (r & 3) ? cmul(w4[r >> 2], w[r & 3]) : w4[r >> 2];
            v[r] = cmul(v[r], f);
        }
    }
    fft16(v);
    __syncthreads();
    const int o = (tid / NS) * (NS * 16) + q;
#pragma unroll
    for (int r = 0; r < 16; r++) {
        const int i = pad(o + r * NS);
        sm.re[i] = v[r].x;
        sm.im[i] = v[r].y;
    }
    __syncthreads();
}

// Spread one of the two sums' points and transform the grid.  After it, the
// three radix-16 passes are done and mode(j) below finishes the last, radix-2
// one.  MULT = 1: S (values y, |y| <= y_max); MULT = 2: Q (values 1).
template <int MULT>
__device__ __forceinline__ void spread_and_transform(Smem& sm, const float2* __restrict__ tw,
                                                     const float* __restrict__ t,
                                                     const float* __restrict__ y, uint32_t n,
                                                     double fc, double df, float y_max,
                                                     unsigned (&s_sum)[2]) {
    // Grid units of a tile: its values' magnitudes sum to less than kRange
    // units, so no cell reaches 2^31 even where all of them meet in one at
    // phase 0 (2^13 are left for half a unit of rounding per point and a few
    // 2^-24 of the scale, the sine and the weight).  A fixed share of the
    // largest value would hold a curve with one value far off in fewer bits: one
    // of 85 in 511 points of a 0.3 sinusoid gave a power error of 5.6e-6
    // (2-norm) against 3.1e-7 and 1.0e-6 of the direct sums.  The magnitudes
    // are added as integers (s_sum, zero at entry: this tile's and the next
    // one's), rounded up to 2^-22 of the largest, so that the unit is the same
    // from run to run.
    constexpr float kRange = 2147475456.0f;
    const int tid = threadIdx.x;
    int* gre = reinterpret_cast<int*>(sm.re);
    int* gim = reinterpret_cast<int*>(sm.im);
    // Times come sorted, so neighbouring points land in neighbouring cells: a
    // tile takes every tiles-th point of the curve, which keeps the lanes of
    // a warp apart on the grid.
    const uint32_t tiles = (n + kTilePts - 1) / kTilePts;
    const uint64_t at0 = (uint64_t)tid * tiles;
    // (squares of sums of less than 10^8 such values are zero in the direct form)
    const float per_value = y_max > 1e-27f ? __fdiv_rn(4194304.0f, y_max) : 0.0f;
    const float per_unit = y_max * 0x1p-22f;
    float value = 1.0f, scale = 0.0f, unit = 0.0f;
    auto fetch = [&](uint32_t k) {  // tile k's value, and its part of the sum
        value = at0 + k < n ? y[at0 + k] : 0.0f;
        const unsigned sum =
            __reduce_add_sync(0xffffffffu, __float2uint_ru(fabsf(value) * per_value));
        if ((tid & 31) == 0) atomicAdd(&s_sum[k & 1u], sum);
    };
    if constexpr (MULT == 1) {
        fetch(0);
    } else {
        scale = kRange / (float)min(max(n, 1u), (uint32_t)kTilePts);
        unit = 1.0f / scale;
    }
    float2 v[16];
#pragma unroll
    for (int r = 0; r < 16; r++) {
        const int i = pad(tid + r * kThreads);
        gre[i] = 0;
        gim[i] = 0;
        v[r] = make_float2(0.0f, 0.0f);
    }
    __syncthreads();
    for (uint32_t k = 0; k < tiles; k++) {
        const uint64_t at = at0 + k;
        if constexpr (MULT == 1) {
            const float sum = (float)max(s_sum[k & 1u], 1u);
            scale = fminf(kRange / sum * per_value, 1e38f);
            unit = sum / kRange * per_unit;
        }
        if (at < n) {
            const double td = (double)t[at];
            double th = td * (fc * MULT);
            th -= rint(th);
            float s, c;
            sincospif(2.0f * (float)th, &s, &c);
            const float a = MULT == 1 ? scale * value : scale;
            s *= a;
            c *= a;
            double x = td * (df * MULT);
            x -= floor(x);
            const double u = x * (double)kM;
            const double m = floor(u);
            const float fr = (float)(u - m);
            const int first = (int)m - (kW / 2 - 1);
#pragma unroll
            for (int l = 0; l < kW; l++) {
                const float z = ((float)(l - (kW / 2 - 1)) - fr) * (2.0f / kW);
                // beta (sqrt(1 - z^2) - 1) without the cancellation near z = 0
                const float zz = z * z;
                const float r = sqrtf(fmaxf(1.0f - zz, 0.0f));
                const float w = __expf(__fdividef(-kBeta * zz, 1.0f + r));
                const int i = pad((first + l) & (kM - 1));
                atomicAdd(&gre[i], __float2int_rn(c * w));
                atomicAdd(&gim[i], __float2int_rn(s * w));
            }
        }
        const bool more = k + 1 < tiles;
        if (MULT == 1 && more) fetch(k + 1);
        __syncthreads();
        if (MULT == 1 && tid == 0) s_sum[k & 1u] = 0u;
#pragma unroll
        for (int r = 0; r < 16; r++) {
            const int i = pad(tid + r * kThreads);
            v[r].x = fmaf(unit, (float)gre[i], v[r].x);
            v[r].y = fmaf(unit, (float)gim[i], v[r].y);
            if (more) {
                gre[i] = 0;
                gim[i] = 0;
            }
        }
        __syncthreads();
    }
    pass16<1>(sm, tw, v);
    pass16<16>(sm, tw, v);
    pass16<256>(sm, tw, v);
}

// Mode of index j (0 <= j < kM / 2) after the radix-16 passes: kappa = j for
// j < kM / 4, else j - kM / 2 (the last pass gives two modes per j, of which
// exactly one lies in the kept half).
__device__ __forceinline__ float2 mode(const Smem& sm, const float2* __restrict__ tw, int j) {
    const int a = pad(j), b = pad(j + kM / 2);
    const float2 w = __ldg(tw + j);
    const float2 x = make_float2(sm.re[a], sm.im[a]);
    const float2 z = cmul(make_float2(sm.re[b], sm.im[b]), w);
    return j < kM / 4 ? cadd(x, z) : csub(x, z);
}

__global__ void __launch_bounds__(kThreads, 2)
    nufft_kernel(const NufftParams p) {
    extern __shared__ __align__(16) unsigned char nsm[];
    Smem& sm = *reinterpret_cast<Smem*>(nsm);
    const uint32_t c = p.order[blockIdx.x / p.blocks];
    const uint32_t k0 = (blockIdx.x % p.blocks) * (uint32_t)kNufftModes;
    const CurveDesc cd = p.curves[c];
    const float* t = p.t + cd.off;
    const float* y = p.m + cd.off;
    const float2* tw = reinterpret_cast<const float2*>(p.table);
    const float* deconv = p.table + 2 * kM;
    const uint32_t n = cd.n;
    if (p.stamps && threadIdx.x == 0) p.stamps[2 * (size_t)blockIdx.x] = global_ns();
    const double fc = p.f0 + (double)(k0 + kNufftModes / 2) * p.df;
    constexpr int kPer = kNufftModes / kThreads;  // modes per thread

    // Largest |y|.  A point that is not finite makes every power NaN, as in the
    // direct form (an infinite sum is so with one sign in one of the two terms
    // and the other in the other): written at once, without the transforms.
    __shared__ unsigned s_max, s_sum[2];
    if (threadIdx.x == 0) s_max = s_sum[0] = s_sum[1] = 0u;
    __syncthreads();
    unsigned my_max = 0u;
    bool bad = false;
    for (uint32_t i = threadIdx.x; i < n; i += kThreads) {
        const float yi = y[i];
        bad = bad || !(fabsf(yi) < INFINITY) || !(fabsf(t[i]) < INFINITY);
        my_max = max(my_max, __float_as_uint(fabsf(yi)));
    }
    my_max = __reduce_max_sync(0xffffffffu, my_max);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_max, my_max);
    bad = __syncthreads_or(bad ? 1 : 0) != 0;
    float* out = p.out + (size_t)c * p.n_freq;
    if (bad) {
        const uint32_t k1 = min(k0 + (uint32_t)kNufftModes, p.n_freq);
        for (uint32_t k = k0 + threadIdx.x; k < k1; k += kThreads)
            out[k] = __uint_as_float(0x7FC00000u);
        if (p.stamps && threadIdx.x == 0) p.stamps[2 * (size_t)blockIdx.x + 1] = global_ns();
        return;
    }
    const float y_max = __uint_as_float(s_max);
    float2 q[kPer];
    spread_and_transform<2>(sm, tw, t, y, n, fc, p.df, 1.0f, s_sum);
#pragma unroll
    for (int i = 0; i < kPer; i++) q[i] = mode(sm, tw, threadIdx.x + i * kThreads);
    __syncthreads();
    spread_and_transform<1>(sm, tw, t, y, n, fc, p.df, y_max, s_sum);

    unsigned again = 0;  // the thread's near-singular modes
#pragma unroll
    for (int i = 0; i < kPer; i++) {
        const int j = threadIdx.x + i * kThreads;
        const int kappa = j < kM / 4 ? j : j - kM / 2;
        const uint64_t k = (uint64_t)k0 + (uint32_t)(kappa + kNufftModes / 2);
        if (k >= p.n_freq) continue;
        const float dc = deconv[kappa < 0 ? -kappa : kappa];
        const float2 sv = mode(sm, tw, j);
        const LSAcc a{sv.x * dc, sv.y * dc, 0.5f * fmaf(q[i].x, dc, (float)n),
                      0.5f * q[i].y * dc};
        const float det = a.cos_cos * ((float)n - a.cos_cos) - a.cos_sin * a.cos_sin;
        if (!(det > kNufftSingular * (float)n * (float)n)) again |= 1u << i;
        out[k] = ls_power(a, n);
    }
    // Near-singular modes point by point, a warp each.
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int i = 0; i < kPer; i++) {
        unsigned todo = __ballot_sync(0xffffffffu, (again >> i) & 1u);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const int j = (int)(threadIdx.x & ~31u) + src + i * kThreads;
            const int kappa = j < kM / 4 ? j : j - kM / 2;
            const uint32_t k = k0 + (uint32_t)(kappa + kNufftModes / 2);
            const double f = p.f0 + (double)k * p.df;
            LSAcc a{0.0f, 0.0f, 0.0f, 0.0f};
            for (uint32_t e = lane; e < n; e += 32) {
                double th = (double)t[e] * f;
                th -= rint(th);
                float s, co;
                sincosf(kTwoPi * (float)th, &s, &co);
                const float ye = y[e];
                a.mag_cos += ye * co;
                a.mag_sin += ye * s;
                a.cos_cos += co * co;
                a.cos_sin += co * s;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                a.mag_cos += __shfl_xor_sync(0xffffffffu, a.mag_cos, o);
                a.mag_sin += __shfl_xor_sync(0xffffffffu, a.mag_sin, o);
                a.cos_cos += __shfl_xor_sync(0xffffffffu, a.cos_cos, o);
                a.cos_sin += __shfl_xor_sync(0xffffffffu, a.cos_sin, o);
            }
            if (lane == 0) out[k] = ls_power(a, n);
        }
    }
    if (p.stamps && threadIdx.x == 0) p.stamps[2 * (size_t)blockIdx.x + 1] = global_ns();
}

// The table: e^{2 pi i k / kM} for k < kM, then 1 / (the kernel's transform at
// mode k) for k <= kNufftModes / 2 (the trapezoidal rule on the even kernel,
// which has all but vanished at its ends).
__global__ void nufft_table_kernel(float* __restrict__ table) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kM) return;
    double sn, cs;
    sincospi(2.0 * (double)k / kM, &sn, &cs);
    table[2 * k] = (float)cs;
    table[2 * k + 1] = (float)sn;
    if (k > kNufftModes / 2) return;
    constexpr int kNodes = 96;
    double sum = 0.5;  // half the value at z = 0
    for (int i = 1; i < kNodes; i++) {
        const double z = (double)i / kNodes;
        sum += exp((double)kBeta * (sqrt(1.0 - z * z) - 1.0)) *
               cospi((double)k * kW * z / (double)kM);
    }
    table[2 * kM + k] = (float)(1.0 / (sum * kW / kNodes));
}

}  // namespace PF_KNS

cudaError_t launch_nufft_table(float* table, cudaStream_t s) {
    static_assert(kNufftTableFloats == 2 * PF_KNS::kM + kNufftModes / 2 + 1, "table size");
    PF_KNS::nufft_table_kernel<<<PF_KNS::kM / 64, 64, 0, s>>>(table);
    return cudaGetLastError();
}

cudaError_t launch_nufft(const NufftParams& p, uint32_t n_curves, cudaStream_t s) {
    if (n_curves == 0) return cudaSuccess;
    const int smem = (int)sizeof(PF_KNS::Smem);
    cudaError_t e = allow_smem(PF_KNS::nufft_kernel, smem);
    if (e != cudaSuccess) return e;
    PF_KNS::nufft_kernel<<<n_curves * p.blocks, PF_KNS::kThreads, smem, s>>>(p);
    return cudaGetLastError();
}

}  // namespace pfk
