// fdk_fft.cu -- the FDK / FBP ramp filter by fast Fourier transforms, for
// detector rows of up to 2048 pixels.
//
// The linear convolution of a row with the ramp kernel, q = tau h * g, is O(W^2)
// directly.  Here a group of threads transforms two rows at a time as one
// complex sequence of N >= 2 W points (a power of two; the kernel is real, so
// the rows stay apart), multiplies by the kernel's spectrum and transforms
// back.  What makes this exact enough in FP32 is the form of the convolution: a
// row's projections are large and smooth and the ramp's output small, so the
// spectrum of g itself would carry rounding errors of the large low
// frequencies into a small result (4e-6 to 2e-5 relative, against 1e-6 to 4e-6
// of direct FP32 sums).  Summed by parts, q = k * dg with the row's differences
// dg[n] = g[n] - g[n-1] (zero before the row and after it) and the running sums
// k[m] = sum_{i <= m} tau h[i], both of the output's size: 1.5e-7.
// The sums in closed form (h is symmetric and sums to zero, so k[-m-1] = -k[m]):
// Ram-Lak k[m] = (1 / (pi^2 tau)) sum of 1/i^2 over odd i > m, a trigamma value
// (Abramowitz & Stegun 6.4.6, 6.4.12); Shepp-Logan 1 / (pi^2 tau (2 m + 1)).
// Rows of a pair are scaled by powers of two to a common magnitude, so neither
// takes rounding errors of the other's size.
// A row with a difference outside the transforms' range (peak_limit: an
// infinity, a NaN, a difference that overflows, a masked pixel of the storage
// type's lowest value) is transformed as zeros and summed directly instead
// (direct_rows): a transform spreads its rounding, 1.5e-7 of the row's largest
// difference, over all outputs, while half of the Ram-Lak taps are zero and
// leave the outputs they do not join to such a pixel as they are.
//
// The transform: N = 16 * 16 * R3 (R3 = 1 for rows of up to 128 pixels), decimation
// in frequency forward (radices 16, 16, R3, results in digit-reversed order), the product, and decimation in time
// back, so no reordering pass exists.  A thread holds 16 complex values, and the
// passes exchange them through shared memory (one complex of padding per 16:
// every access of a half warp falls on 32 banks).  What bounds it: the
// exchanges and the block barriers between them.  Measured against a 3xTF32
// Toeplitz product on the tensor cores (O(W^2) operations): 276 k rows of 1024
// pixels, FP16 in, FP32 out, 4.72 -> 1.67 ms; 184 k of 512, 0.93 -> 0.58; 26 k FP32
// rows of 2000, 1.65 -> 0.37.
#include <type_traits>

#include "common.cuh"
#include "fdk_taps.cuh"
#include "internal.h"

namespace pyronn {

namespace {

constexpr int FFT_THREADS = 256;
constexpr int FFT_BLOCKS = 3;  // per SM (80 registers; 2 / 4 blocks: 2.11 / 2.88 ms on the 512^3 scan's rows)
constexpr int FFT_MAX_WIDTH = 2048;

__host__ __device__ constexpr int pad16(int p)
{
    return p + (p >> 4);
}

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
// a (wx + i wy) forward, a (wx - i wy) inverse
template <bool INV>
__device__ __forceinline__ float2 cmul(float2 a, float wx, float wy)
{
    const float s = INV ? -wy : wy;
    return make_float2(fmaf(a.x, wx, -a.y * s), fmaf(a.x, s, a.y * wx));
}

// discrete Fourier transforms of 2, 4, 8 and 16 points in registers, natural
// order in and out: X[k] = sum_n x[n] exp(-+ 2 pi i n k / R)
template <bool INV>
__device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c, float2 &d)
{
    const float2 s = cadd(a, c), t = csub(a, c), u = cadd(b, d), v = csub(b, d);
    a = cadd(s, u);
    c = csub(s, u);
    const float2 m = make_float2(t.x + v.y, t.y - v.x), p = make_float2(t.x - v.y, t.y + v.x);
    b = INV ? p : m;
    d = INV ? m : p;
}

template <bool INV, int R>
__device__ __forceinline__ void dft(float2 *x)
{
    constexpr float C1 = 0.92387953251128674f, S1 = 0.38268343236508977f, H = 0.70710678118654752f;
    if constexpr (R == 1) {
    } else if constexpr (R == 2) {
        const float2 a = x[0];
        x[0] = cadd(a, x[1]);
        x[1] = csub(a, x[1]);
    } else if constexpr (R == 4) {
        dft4<INV>(x[0], x[1], x[2], x[3]);
    } else if constexpr (R == 8) {
        // n = n2 + 2 n1, k = k1 + 4 k2
        dft4<INV>(x[0], x[2], x[4], x[6]);
        dft4<INV>(x[1], x[3], x[5], x[7]);
        x[3] = cmul<INV>(x[3], H, -H);
        x[5] = cmul<INV>(x[5], 0.0f, -1.0f);
        x[7] = cmul<INV>(x[7], -H, -H);
        float2 y[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = cadd(x[2 * k], x[2 * k + 1]), y[k + 4] = csub(x[2 * k], x[2 * k + 1]);
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = y[k];
    } else {
        static_assert(R == 16, "radix");
        // n = n2 + 4 n1, k = k1 + 4 k2
#pragma unroll
        for (int n = 0; n < 4; ++n) dft4<INV>(x[n], x[n + 4], x[n + 8], x[n + 12]);
        x[5] = cmul<INV>(x[5], C1, -S1), x[9] = cmul<INV>(x[9], H, -H), x[13] = cmul<INV>(x[13], S1, -C1);
        x[6] = cmul<INV>(x[6], H, -H), x[10] = cmul<INV>(x[10], 0.0f, -1.0f), x[14] = cmul<INV>(x[14], -H, -H);
        x[7] = cmul<INV>(x[7], S1, -C1), x[11] = cmul<INV>(x[11], -H, -H), x[15] = cmul<INV>(x[15], -C1, S1);
        float2 y[16];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            dft4<INV>(x[4 * k], x[4 * k + 1], x[4 * k + 2], x[4 * k + 3]);
#pragma unroll
            for (int j = 0; j < 4; ++j) y[k + 4 * j] = x[4 * k + j];
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = y[k];
    }
}

// k[m] tau of the running sums above, m >= 0
__device__ float running_sum(int kind, int m)
{
    const double inv_pi2 = 0.10132118364233777;  // 1 / pi^2
    if (kind != PYRONN_FILTER_RAM_LAK) return (float)(inv_pi2 / (2.0 * m + 1.0));
    // sum over odd i > m of 1 / i^2 = trigamma(n / 2) / 4, n the first such i
    double x = 0.5 * (double)((m & 1) ? m + 2 : m + 1), s = 0.0;
    for (; x < 8.0; x += 1.0) s += 1.0 / (x * x);
    const double r = 1.0 / x, r2 = r * r;
    s += r + 0.5 * r2 + r * r2 * (1.0 / 6.0 - r2 * (1.0 / 30.0 - r2 * (1.0 / 42.0 - r2 * (1.0 / 30.0))));
    return (float)(0.25 * inv_pi2 * s);
}

template <int R3>
struct Plan {
    static constexpr int N = 256 * R3, M = N / 16;      // points; threads per row pair
    static constexpr int PAIRS = FFT_THREADS / M;        // row pairs in flight per block
    static constexpr int PN = pad16(N);                  // padded points
    // the group's lanes of a warp (half a warp for M = 16), and its parts of 32
    static constexpr int LANES = M < 32 ? M : 32, PARTS = M / LANES;
    __device__ static unsigned lane_mask(int lane) { return LANES == 32 ? 0xffffffffu : 0xffffu << (lane & 16); }
    // shared memory: the pairs' points, the kernel's spectrum, the twiddles
    // w_N^(t q) [q][t] and w_M^(t2 q) [q][t2], q = 1 .. 15
    static constexpr size_t SMEM = sizeof(float2) * ((size_t)PAIRS * PN + PN + 15 * M + 15 * R3);
};

// The sixteen values of thread t through the forward passes: x[k] in is point
// t + k M, out the spectrum's point 16 t + k in digit-reversed order.
template <int R3>
__device__ __forceinline__ void forward(float2 (&x)[16], float2 *buf, const float2 *tw1, const float2 *tw2, int t)
{
    constexpr int M = Plan<R3>::M;
    dft<false, 16>(x);
    buf[pad16(t)] = x[0];
#pragma unroll
    for (int q = 1; q < 16; ++q) {
        const float2 w = tw1[(q - 1) * M + t];
        buf[pad16(q * M + t)] = cmul<false>(x[q], w.x, w.y);
    }
    __syncthreads();
    const int t2 = t % R3, base = (t / R3) * M + t2;
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = buf[pad16(base + k * R3)];
    dft<false, 16>(x);
    if (R3 == 1) return;  // (the sixteen points are the thread's)
    buf[pad16(base)] = x[0];
#pragma unroll
    for (int q = 1; q < 16; ++q) {
        const float2 w = tw2[(q - 1) * R3 + t2];
        buf[pad16(base + q * R3)] = cmul<false>(x[q], w.x, w.y);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = buf[17 * t + k];
#pragma unroll
    for (int s = 0; s < 16 / R3; ++s) dft<false, R3>(x + s * R3);
}

// The reverse: x[k] in is point 16 t + k of the spectrum, out point t + k M
// times N.
template <int R3>
__device__ __forceinline__ void inverse(float2 (&x)[16], float2 *buf, const float2 *tw1, const float2 *tw2, int t)
{
    constexpr int M = Plan<R3>::M;
    const int t2 = t % R3, base = (t / R3) * M + t2;
    if (R3 > 1) {
#pragma unroll
        for (int s = 0; s < 16 / R3; ++s) dft<true, R3>(x + s * R3);
#pragma unroll
        for (int k = 0; k < 16; ++k) buf[17 * t + k] = x[k];
        __syncthreads();
        x[0] = buf[pad16(base)];
#pragma unroll
        for (int q = 1; q < 16; ++q) {
            const float2 w = tw2[(q - 1) * R3 + t2];
            x[q] = cmul<true>(buf[pad16(base + q * R3)], w.x, w.y);
        }
    }
    dft<true, 16>(x);
#pragma unroll
    for (int k = 0; k < 16; ++k) buf[pad16(base + k * R3)] = x[k];
    __syncthreads();
    x[0] = buf[pad16(t)];
#pragma unroll
    for (int q = 1; q < 16; ++q) {
        const float2 w = tw1[(q - 1) * M + t];
        x[q] = cmul<true>(buf[pad16(q * M + t)], w.x, w.y);
    }
    dft<true, 16>(x);
}

// The bits of the least magnitude of a row's differences that takes the row out
// of the transforms' range: 2^64, 2^14 for FP16 storage (whose lowest value is
// -65504), both far above any line integral.
template <typename Tin>
__host__ __device__ constexpr unsigned peak_limit()
{
    return (127u + (std::is_same<Tin, __half>::value ? 14u : 64u)) << 23;
}

// The Feldkamp cosine weight of column j on a row at height vv.
__device__ __forceinline__ float cosine_weight(int j, float vv, float sdd, float du, float cu)
{
    const float uu = ((float)j - cu) * du;
    return sdd * rsqrtf(fmaf(sdd, sdd, fmaf(uu, uu, vv * vv)));
}

// The rows `first` (if bad_a) and `first` + 1 (if bad_b) of a pair by direct
// FP32 sums over the taps that are not zero, in the order of fdk.cu's kernel.
// nan_rows: a row that holds an infinity or a NaN is written as NaNs.  Called by
// the whole block (`scratch`: a word per warp); every group has the row and the
// taps in its own `buf`.
template <typename Tin, typename Tout, int R3>
__device__ __noinline__ void direct_rows(const Tin *in, Tout *out, long long first, bool bad_a, bool bad_b, int det_h,
                                         int W, float sdd, float dv, float du, float cv, float cu, int kind,
                                         int weight_output, int nan_rows, float2 *buf, unsigned *scratch)
{
    using P = Plan<R3>;
    constexpr int M = P::M;
    const int tid = threadIdx.x, grp = tid / M, t = tid % M;
    float *g = reinterpret_cast<float *>(buf), *taps = g + P::N;  // W <= N / 2 of each; buf is 2 N floats and more
    for (int r = 0; r < 2; ++r) {
        const bool bad = r == 0 ? bad_a : bad_b;
        const float vv = ((float)(int)((first + r) % det_h) - cv) * dv;
        const Tin *row = in + (first + r) * W;
        bool nonfinite = false;
        if (bad)
            for (int j = t; j < W; j += M) {
                float x = load_as_float(row + j);
                if (!weight_output && sdd > 0.0f) x *= cosine_weight(j, vv, sdd, du, cu);
                nonfinite |= !isfinite(x);
                g[j] = x;
                taps[j] = fdk_tap(kind, j, du);
            }
        const bool any = __any_sync(P::lane_mask(tid & 31), nonfinite);
        if (tid % P::LANES == 0) scratch[tid / P::LANES] = any;
        __syncthreads();  // the row is read completely before it is written
        if (bad) {
            bool all_nan = false;
            for (int w = 0; w < P::PARTS; ++w) all_nan |= nan_rows && scratch[grp * P::PARTS + w];
            for (int j = t; j < W; j += M) {
                float q = 0.0f;
                if (kind == PYRONN_FILTER_RAM_LAK) {  // odd offsets and the centre
                    for (int k = (j + 1) & 1; k < W; k += 2) q = fmaf(taps[abs(j - k)], g[k], q);
                    q = fmaf(taps[0], g[j], q);
                } else {
                    for (int k = 0; k < W; ++k) q = fmaf(taps[abs(j - k)], g[k], q);
                }
                if (all_nan) q = __uint_as_float(0x7fffffffu);
                if (weight_output && sdd > 0.0f) q *= cosine_weight(j, vv, sdd, du, cu);
                store_from_float(out + (first + r) * W + j, q);
            }
        }
        __syncthreads();
    }
}

// in and out may be the same buffer: a pair's rows are read completely before
// they are written, by the threads that own them.
template <typename Tin, typename Tout, int R3>
__global__ void __launch_bounds__(FFT_THREADS, FFT_BLOCKS)
    fdk_filter_fft_kernel(const Tin *in, Tout *out, long long rows, int det_h, int W, float sdd, float dv, float du,
                          float cv, float cu, int kind, int weight_output, int nan_rows)
{
    using P = Plan<R3>;
    constexpr int M = P::M, LANES = P::LANES;
    extern __shared__ __align__(16) float2 fft_smem[];
    __shared__ unsigned peak[2][FFT_THREADS / LANES];
    float2 *spectrum = fft_smem + P::PAIRS * P::PN, *tw1 = spectrum + P::PN, *tw2 = tw1 + 15 * M;
    const int tid = threadIdx.x, grp = tid / M, t = tid % M, lane = tid & 31;
    float2 *buf = fft_smem + grp * P::PN;

    for (int i = tid; i < 15 * M; i += FFT_THREADS) {
        const int q = i / M + 1;
        float s, c;
        sincospif(-2.0f * (float)((i % M) * q % P::N) / (float)P::N, &s, &c);
        tw1[i] = make_float2(c, s);
    }
    for (int i = tid; i < 15 * R3; i += FFT_THREADS) {
        const int q = i / R3 + 1;
        float s, c;
        sincospif(-2.0f * (float)((i % R3) * q % M) / (float)M, &s, &c);
        tw2[i] = make_float2(c, s);
    }
    __syncthreads();
    float2 x[16];
    // the kernel's spectrum (every group computes it, the first stores it),
    // with the inverse transform's 1 / N
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int n = t + k * M, m = n < P::N / 2 ? n : P::N - 1 - n;
        const float v = m < W ? running_sum(kind, m) / (du * (float)P::N) : 0.0f;
        x[k] = make_float2(n < P::N / 2 ? v : -v, 0.0f);
    }
    forward<R3>(x, buf, tw1, tw2, t);
    if (grp == 0) {
#pragma unroll
        for (int k = 0; k < 16; ++k) spectrum[17 * t + k] = x[k];
    }
    __syncthreads();

    const long long pairs = (rows + 1) / 2;
    for (long long p0 = (long long)blockIdx.x * P::PAIRS; p0 < pairs; p0 += (long long)gridDim.x * P::PAIRS) {
        const long long ra = 2 * (p0 + grp);
        const bool live_a = ra < rows, live_b = ra + 1 < rows;
        const float va = ((float)(int)(ra % det_h) - cv) * dv, vb = ((float)(int)((ra + 1) % det_h) - cv) * dv;
        const Tin *ia = in + ra * W, *ib = ia + W;
        auto weight = [&](int j, float vv) { return cosine_weight(j, vv, sdd, du, cu); };
        // the rows' values, then their differences
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int j = t + k * M;
            float2 g = make_float2(live_a && j < W ? load_as_float(ia + j) : 0.0f,
                                   live_b && j < W ? load_as_float(ib + j) : 0.0f);
            if (!weight_output && sdd > 0.0f) g = make_float2(g.x * weight(j, va), g.y * weight(j, vb));
            x[k] = g;
            buf[j] = g;
        }
        __syncthreads();
        unsigned pa = 0u, pb = 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int j = t + k * M;
            if (j > 0) x[k] = csub(x[k], buf[j - 1]);
            pa = max(pa, __float_as_uint(x[k].x) & 0x7fffffffu);
            pb = max(pb, __float_as_uint(x[k].y) & 0x7fffffffu);
        }
        // point N / 2 (after the last pixel of a row of N / 2)
        x[8] = make_float2(0.0f, 0.0f);
        if (t == 0) {
            x[8] = csub(x[8], buf[P::N / 2 - 1]);
            pa = max(pa, __float_as_uint(x[8].x) & 0x7fffffffu);
            pb = max(pb, __float_as_uint(x[8].y) & 0x7fffffffu);
        }
        pa = __reduce_max_sync(P::lane_mask(lane), pa);
        pb = __reduce_max_sync(P::lane_mask(lane), pb);
        if (lane % LANES == 0) peak[0][tid / LANES] = pa, peak[1][tid / LANES] = pb;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < P::PARTS; ++w) {
            pa = max(pa, peak[0][grp * P::PARTS + w]);
            pb = max(pb, peak[1][grp * P::PARTS + w]);
        }
        // powers of two that bring the largest difference into [1, 2)
        const unsigned ea = pa >> 23, eb = pb >> 23;  // 0: zero (or flushed)
        const bool bad_a = pa >= peak_limit<Tin>(), bad_b = pb >= peak_limit<Tin>();
        const float sa = ea == 0u || bad_a ? 1.0f : __uint_as_float((254u - ea) << 23);
        const float sb = eb == 0u || bad_b ? 1.0f : __uint_as_float((254u - eb) << 23);
        // the factors back: zero for a row of zeros, which stays zeros; NaN marks
        // a row that is summed directly
        const float nan = __uint_as_float(0x7fffffffu);
        const float ua = bad_a ? nan : (ea == 0u ? 0.0f : 1.0f / sa), ub = bad_b ? nan : (eb == 0u ? 0.0f : 1.0f / sb);
#pragma unroll
        for (int k = 0; k < 9; ++k) x[k] = make_float2(bad_a ? 0.0f : x[k].x * sa, bad_b ? 0.0f : x[k].y * sb);
#pragma unroll
        for (int k = 9; k < 16; ++k) x[k] = make_float2(0.0f, 0.0f);
        forward<R3>(x, buf, tw1, tw2, t);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float2 w = spectrum[17 * t + k];
            x[k] = cmul<false>(x[k], w.x, w.y);
        }
        inverse<R3>(x, buf, tw1, tw2, t);
        Tout *oa = out + ra * W, *ob = oa + W;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int j = t + k * M;
            if (j < W) {
                float qa = x[k].x * ua, qb = x[k].y * ub;
                if (weight_output && sdd > 0.0f) qa *= weight(j, va), qb *= weight(j, vb);
                if (live_a && !isnan(ua)) store_from_float(oa + j, qa);
                if (live_b && !isnan(ub)) store_from_float(ob + j, qb);
            }
        }
        // every thread is done with the exchange buffer
        if (__syncthreads_or(isnan(ua) || isnan(ub)))
            direct_rows<Tin, Tout, R3>(in, out, 2 * (p0 + grp), isnan(ua), isnan(ub), det_h, W, sdd, dv, du, cv, cu, kind,
                                       weight_output, nan_rows, buf, peak[0]);
    }
}

template <typename Tin, typename Tout, int R3>
cudaError_t launch_plan(const void *in, void *out, long long rows, int det_h, int W, float sdd, float dv, float du,
                        float cv, float cu, int kind, int weight_output, int nan_rows, cudaStream_t stream)
{
    using P = Plan<R3>;
    auto kernel = fdk_filter_fft_kernel<Tin, Tout, R3>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P::SMEM);
    if (e != cudaSuccess) return e;
    // persistent blocks: the kernel's spectrum and the twiddles once per block
    const long long groups = ((rows + 1) / 2 + P::PAIRS - 1) / P::PAIRS;
    const unsigned grid = (unsigned)(groups < 148 * FFT_BLOCKS ? groups : 148 * FFT_BLOCKS);
    kernel<<<grid, FFT_THREADS, P::SMEM, stream>>>((const Tin *)in, (Tout *)out, rows, det_h, W, sdd, dv, du, cv, cu,
                                                   kind, weight_output, nan_rows);
    return cudaGetLastError();
}

}  // namespace

bool fdk_fft_supported(int W)
{
    return W <= FFT_MAX_WIDTH;
}

cudaError_t launch_fdk_filter_fft(const void *in, void *out, int in_dtype, int out_dtype, long long rows, int det_h,
                                  int W, float sdd, float dv, float du, float cv, float cu, int kind,
                                  int weight_output, cudaStream_t stream)
{
    // rows with infinities or NaNs: NaNs throughout on distinct, aligned buffers
    // of quad rows, the direct sums' in every other call
    const char *ib = (const char *)in, *ob = (const char *)out;
    const size_t n = (size_t)rows * (size_t)W;
    const bool overlap = ib < ob + n * dtype_size(out_dtype) && ob < ib + n * dtype_size(in_dtype);
    const int nan_rows = W % 4 == 0 && (uintptr_t)in % 16 == 0 && (uintptr_t)out % 16 == 0 && !overlap;
    return dispatch_dtypes(in_dtype, out_dtype, [&](auto tin, auto tout) -> cudaError_t {
        using Tin = typename decltype(tin)::type;
        using Tout = typename decltype(tout)::type;
        auto launch = W <= 128    ? launch_plan<Tin, Tout, 1>
                      : W <= 256  ? launch_plan<Tin, Tout, 2>
                      : W <= 512  ? launch_plan<Tin, Tout, 4>
                      : W <= 1024 ? launch_plan<Tin, Tout, 8>
                                  : launch_plan<Tin, Tout, 16>;
        return launch(in, out, rows, det_h, W, sdd, dv, du, cv, cu, kind, weight_output, nan_rows, stream);
    });
}

}  // namespace pyronn
