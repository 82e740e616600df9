// proj2d.cu -- 2D parallel-beam and fan-beam projector / backprojector.
//
// Forward (ParallelProjection2D / FanProjection2D): one thread per detector
// pixel, blockIdx.y = view, blockIdx.z = batch elements; the ray march follows
// kernel_project2D (par_projector_2D_CudaKernel.cu.cc:28-102): box edges
// index_to_physical(0|N) - 0.5 in mm, first sample at the entry with weight
// 1/2, alpha advanced in a float, step 0.2 * min(spacing) mm, end correction
// only when the sum is > 0, result scaled by |ray (.) spacing| (:141).
// The reference samples a border/linear texture at index + 0.5; here the
// same bilinear interpolation is done with exact FP32 weights.  The samples of
// a ray that fall in one cell -- about four -- are summed in closed form
// (sum_cells), at the march's own alphas, and slices of a batch that share
// their geometry share the walk.  What bounds it: instruction issue, then the
// L1 lines of the cell loads.
// Given a workspace, the call first writes two copies of the batch as
// bilinear CELLS -- the cell of floors x, y in [-2, N] holds the four taps
// V(x + {0,1}, y + {0,1}), with zeros outside the slice -- one x-fastest and one
// y-fastest.  (The box starts half a millimetre below pixel 0: at index -1 for
// 0.5 mm pixels, where rounding puts some rays' first sample a hair below -1;
// the second border cell keeps every ray of such a view, and so every lane of
// its warps, on the unclamped path.)  The cells hold FP32 taps for every
// storage type, so a visit is one 16-byte load with no bounds tests and no
// widening.  A warp's 32 threads are 32 neighbouring detector pixels, so their
// cells lie along the detector direction: views whose rays run mostly along y
// read the x-fastest cells, the others the y-fastest ones, so the warp's loads
// stay on few cache lines.  Without a workspace the taps are read from the
// caller's slice with a bounds test each.  Taps are combined in the same order
// on every path, so the choice does not change a result.
//
// Backward (ParallelBackprojection2D / FanBackprojection2D): one thread per
// pixel, loop over views, linear interpolation along the detector row;
// launches of few pixels split each pixel's views over BP2_VSPLIT threads.
#include <math_constants.h>
#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace pyronn {

namespace {

constexpr float PI_REF = 3.14159265359f;  // par_backprojector_2D_CudaKernel.cu.cc:32
constexpr int FP2_BLOCK = 128;

constexpr int BP2_BLOCK_X = 32;
constexpr int BP2_BLOCK_Y = 8;
constexpr int BP2_CHUNK = BP2_BLOCK_X * BP2_BLOCK_Y;  // views per shared-memory table
constexpr int BP2_VSPLIT = 4;                          // view groups of a small slice's backprojection
constexpr long long BP2_SPLIT_MAX_PIXELS = 131072;     // pixels per launch up to which view groups are used
constexpr long long BP2_SPLIT_MAX_SHARED = 600000;     // the same, threads of several slices
constexpr long long BP2_SHARE_MIN_PIXELS = 80000;      // pixels per launch from which a thread takes several slices
constexpr long long BP2_NS8_MIN_PIXELS = 8000000;      // pixels per launch from which a thread takes eight slices
static_assert(BP2_NS8_MIN_PIXELS / 8 > BP2_SPLIT_MAX_SHARED, "eight slices are never split");

// Two values on the packed FP32 instructions: one issue slot for both (the
// kernels here are bound by issue).
__device__ __forceinline__ float2 pair(float a, float b) { return make_float2(a, b); }

// The forward walks a ray along its view's MAJOR axis m (the one its rays run
// mostly along), the other being the minor axis n.  A bilinear cell holds the
// four taps V(m0,n0), V(m1,n0), V(m0,n1), V(m1,n1), widened to FP32 whatever
// the storage type (exact, so 16-bit storage gives the FP32 result of the
// rounded input).  A source of taps is indexed by the floors (m, n) of a
// sample and the slice s of the thread's slices.

// From the caller's slices, taps outside them zero.
template <typename T>
struct BorderTaps {
    static constexpr bool ALIGN_COLUMNS = false;
    const T *img;
    size_t slice;
    int s_m, s_n, M, N;  // element strides and extents of the axes
    __device__ __forceinline__ float4 operator()(int m0, int n0, int s) const
    {
        const bool vm0 = (unsigned)m0 < (unsigned)M, vm1 = (unsigned)(m0 + 1) < (unsigned)M;
        const bool vn0 = (unsigned)n0 < (unsigned)N, vn1 = (unsigned)(n0 + 1) < (unsigned)N;
        const T *p = img + s * slice;
        const int base = m0 * s_m + n0 * s_n;
        float4 w;
        w.x = (vm0 && vn0) ? load_as_float(p + base) : 0.0f;
        w.y = (vm1 && vn0) ? load_as_float(p + base + s_m) : 0.0f;
        w.z = (vm0 && vn1) ? load_as_float(p + base + s_n) : 0.0f;
        w.w = (vm1 && vn1) ? load_as_float(p + base + s_m + s_n) : 0.0f;
        return w;
    }
};

// From a cell copy whose fast axis is n: columns of `pitch` cells, `slice`
// cells per slice.  The copy holds floors in [-2, extent]; CLAMP takes others
// to the nearest of these, whose taps are zero like theirs (for rays not
// proven inside).
template <bool CLAMP>
struct CellTaps {
    static constexpr bool ALIGN_COLUMNS = !CLAMP;
    const float4 *cells;  // floor (-2, -2)
    size_t slice;
    unsigned pitch;
    int M, N;
    __device__ __forceinline__ float4 operator()(int m0, int n0, int s) const
    {
        if (CLAMP) m0 = min(max(m0, -2), M), n0 = min(max(n0, -2), N);
        return __ldg(cells + s * slice + ((unsigned)m0 * pitch + (unsigned)n0 + 2u * (pitch + 1u)));
    }
};

__device__ __forceinline__ float bilinear(const float4 &w, float tm, float tn)
{
    return lerp_ref(lerp_ref(w.x, w.z, tn), lerp_ref(w.y, w.w, tn), tm);
}

// The alpha sequence a_0 = entry, a_{k+1} = fl(a_k + step) of kernel_project2D
// (par_projector_2D_CudaKernel.cu.cc:58-102) in closed form over runs of equal
// increments: inside the binade [2^e, 2^(e+1)) of a, a = M u with u = 2^(e-23)
// and M in [2^23, 2^24), every exact sum a_k + step lies at the same offset
// from the grid of multiples of u, so each step adds D u with D = round(step /
// u); a result equal to 2^(e+1) (M = 2^24) is also right (the sum lies within
// u/2 of it on either side's grid).  A sum halfway between two grid values
// goes to the even one, so from an even M on the increment is the even one of
// the two neighbours of step / u.
// Given a sample at a < am, returns n >= 1 samples a + j delta, j < n, all of
// them below am, n <= kmax, and their successor a_{n} in `next`.  Where the
// closed form does not hold (a not positive normal, the step past a binade),
// n = 1.  n stays below 2^22, so j is exact in FP32.
__device__ __forceinline__ int alpha_run(float a, float am, float step, int kmax, float &delta, float &next)
{
    delta = 0.0f;
    next = __fadd_rn(a, step);
    const int sb = __float_as_int(step), se = (sb >> 23) & 0xff;
    const int bits = __float_as_int(a), be = (bits >> 23) & 0xff;
    if (bits <= 0 || be <= 23 || be == 0xff || sb <= 0 || se == 0 || se == 0xff) return 1;  // (u normal too)
    const unsigned ms = (unsigned)(sb & 0x7fffff) | 0x800000u;
    const unsigned M = (unsigned)(bits & 0x7fffff) | 0x800000u;
    // D = round(step / u), step / u = ms 2^(se - be)
    const int sh = be - se;
    unsigned D;
    if (sh < 0) {
        return 1;  // step >= 2^24 u: no second sample in the binade
    } else if (sh == 0) {
        D = ms;
    } else if (sh >= 25) {
        D = 0u;  // step below u / 2: the sequence stalls at a
    } else {
        const unsigned rem = ms & ((1u << sh) - 1u), half = 1u << (sh - 1);
        D = ms >> sh;
        if (rem == half) {
            if (M & 1u) return 1;
            D += D & 1u;
        } else {
            D += rem > half ? 1u : 0u;
        }
    }
    unsigned n = min((unsigned)kmax, 1u << 22);
    if (D > 0u) {
        // results a + j D u stay on this grid while M + j D <= 2^24
        n = min(n, (0x1000000u - M) / D);
        if (n == 0u) return 1;
        // and the march stops at the first alpha not below am (am > a, so its
        // binade is e or above; two or more above, it is out of reach)
        const int amb = __float_as_int(am), ae = (amb >> 23) & 0xff;
        if (ae - be <= 1) {
            const unsigned am_u = ((unsigned)(amb & 0x7fffff) | 0x800000u) << (ae - be);  // am / u, exact
            n = min(n, (am_u - M + D - 1u) / D);
        }
    }
    delta = (float)D * __int_as_float((be - 23) << 23);               // D u, exact: D <= 2^24
    next = __int_as_float((be << 23) + (int)(M + n * D) - 0x800000);  // M + n D = 2^24 gives 2^(e+1)
    return (int)n;
}

// The iteration bound of the march.
__device__ __forceinline__ int march2d_max_iter(float a, float am, float step)
{
    const double bound = ((double)am - (double)a) / (double)step + 4.0;
    return bound > 1.0e8 ? 100000000 : (int)bound;
}

// A ray through index space: position (bm + a gm, bn + a gn) at alpha a.
struct Ray2D {
    float a, am, step, gm, bm, gn, bn;
    __device__ __forceinline__ float m(float al) const { return fmaf(al, gm, bm); }
    __device__ __forceinline__ float n(float al) const { return fmaf(al, gn, bn); }
};

// (m in .x, n in .y)
struct FloorFrac2 {
    int mi, ni;
    float2 f;
};
// floor_frac (common.cuh) of both halves
__device__ __forceinline__ FloorFrac2 floor_frac2(float2 x)
{
    const float magic = 12582912.0f;
    const float2 y = __fadd2_rd(x, pair(magic, magic));
    FloorFrac2 r;
    r.mi = __float_as_int(y.x) - FLOOR_BIAS;
    r.ni = __float_as_int(y.y) - FLOOR_BIAS;
    r.f = __ffma2_rn(__fadd2_rn(y, pair(-magic, -magic)), pair(-1.0f, -1.0f), x);
    return r;
}

// A linear run of samples: the coordinates c0 + j d at sample j, and the
// number of samples from a fraction f to the cell's far faces, r0 - f inv
// (ninv = -inv).
struct Run2D {
    float2 c0, d, ninv, r0;
    __device__ __forceinline__ static void face(float d, float &ninv, float &r0)
    {
        const bool moves = fabsf(d) > 1.0e-30f;
        const float inv = moves ? __frcp_rn(d) : 0.0f;
        ninv = -inv;
        r0 = !moves ? 1.0e30f : (d > 0.0f ? inv : 0.0f);
    }
    __device__ __forceinline__ void set(const Ray2D &ray, float a, float delta)
    {
        c0 = pair(ray.m(a), ray.n(a));
        d = pair(delta * ray.gm, delta * ray.gn);
        face(d.x, ninv.x, r0.x);
        face(d.y, ninv.y, r0.y);
    }
    __device__ __forceinline__ FloorFrac2 at(float j) const { return floor_frac2(__ffma2_rn(pair(j, j), d, c0)); }
};

// The sums of `kmax` (or all) samples of the ray from alpha `a` on, for NS
// slices: samples at the march's own alphas, one cell visit at a time.  The
// step is a fifth of a pixel, so a ray takes about four samples per cell, and
// inside a cell the interpolant along the ray is a quadratic in the sample
// number: the L samples of a visit add up to L times the interpolant at their
// middle plus the cross term's spread, C dm dn L (L^2 - 1) / 12 with C the
// cell's mixed difference.  (The interpolant is continuous across cell faces:
// a sample within rounding of a face may go to either cell.)  Returns the
// alpha after the last sample and the last sample's alpha in `a_last`.
//
// ALIGN_COLUMNS: the lanes of `mask` (neighbouring rays) walk the columns of
// the major axis together, a few (COLS) at a time -- a lane visits cells only up
// to the warp's common column, counted from the first lane's entry -- so a
// warp's loads fall on few columns, at neighbouring n.  Free-running lanes
// spread over as many columns as lines (10 L1 cycles per load, the L1 98 %
// busy); strict alignment (COLS = 1) idles lanes whose neighbours cross more
// rows.  64 fan slices of 512^2, four per thread: 21.7 ms free-running; 17.0
// and 14.4 ms for COLS = 1 and 2 in scalar arithmetic; packed, 11.63 / 11.72 /
// 11.93 / 12.37 / 12.84 ms for 4 / 6 / 8 / 12 / 16.  With one slice per thread 16 is
// best, with three 8 (0.460 ms against 0.473 for 4 on 387 x 451 slices).
template <int NS, typename Taps>
__device__ __forceinline__ float sum_cells(const Ray2D &ray, float a, int kmax, const Taps &taps, unsigned mask,
                                           float (&acc)[NS], float &a_last)
{
    constexpr int COLS = NS == 1 ? 16 : (NS == 4 ? 4 : 8);
#pragma unroll
    for (int s = 0; s < NS; ++s) acc[s] = 0.0f;
    Run2D run;
    float nf, jf, spread0, next = a;
    bool alive;
    auto next_run = [&]() {  // the next run of equal increments (one to three per ray)
        a = next;
        alive = a < ray.am && kmax > 0;
        if (!alive) return;
        float delta;
        const int n = alpha_run(a, ray.am, ray.step, kmax, delta, next);
        kmax -= n;
        nf = (float)n;
        jf = 0.0f;
        run.set(ray, a, delta);
        spread0 = run.d.x * run.d.y * (1.0f / 12.0f);
        a_last = fmaf(nf - 1.0f, delta, a);  // exact: a value of the sequence
    };
    a_last = a;
    next_run();
    FloorFrac2 p = floor_frac2(pair(ray.m(a), ray.n(a)));
    // the lane's column: the floor along m in the ray's direction, relative
    // to the first lane's entry
    int sign = 0, off = 0;
    if (Taps::ALIGN_COLUMNS) {
        sign = ray.gm < 0.0f ? -1 : 1;
        off = -__reduce_min_sync(mask, alive ? sign * p.mi : 0x7fffffff);
    }
    // AHEAD: a visit's taps are loaded while the previous visit is computed
    // (one slice: 5 % faster; two or more have no registers for it: 0.65 -> 0.90 ms
    // on three 387 x 451 fan slices)
    constexpr bool AHEAD = NS == 1;
    float4 w[NS], ahead[AHEAD ? NS : 1];
    if (AHEAD && alive) {
#pragma unroll
        for (int s = 0; s < NS; ++s) ahead[s] = taps(p.mi, p.ni, s);
    }
    for (int column = COLS - 1; alive; column += COLS) {
        while (alive && (!Taps::ALIGN_COLUMNS || sign * p.mi + off <= column)) {
#pragma unroll
            for (int s = 0; s < NS; ++s) w[s] = AHEAD ? ahead[s] : taps(p.mi, p.ni, s);
            // samples of this visit: up to the nearer face or the run's end,
            // at least one (ceiling by a sum rounded up, as floor_frac's;
            // exact below 2^22, and nf is)
            const float2 r = __ffma2_rn(p.f, run.ninv, run.r0);
            const float c = fminf(fminf(r.x, r.y), nf - jf);
            const float L = fmaxf(__fadd_rn(__fadd_ru(c, 12582912.0f), -12582912.0f), 1.0f);
            const float h = fmaf(L, 0.5f, -0.5f);
            const float2 mid = __ffma2_rn(pair(h, h), run.d, p.f);
            const float spread = fmaf(L, L, -1.0f) * spread0;
            jf += L;
            if (jf >= nf) next_run();
            p = run.at(jf);
            if (AHEAD && alive) {
#pragma unroll
                for (int s = 0; s < NS; ++s) ahead[s] = taps(p.mi, p.ni, s);
            }
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const float2 lo = pair(w[s].x, w[s].y), hi = pair(w[s].z, w[s].w);
                const float2 dn = __ffma2_rn(lo, pair(-1.0f, -1.0f), hi);
                const float2 q = __ffma2_rn(pair(mid.y, mid.y), dn, lo);
                const float v = fmaf(dn.y - dn.x, spread, fmaf(mid.x, q.y - q.x, q.x));
                acc[s] = fmaf(L, v, acc[s]);
            }
        }
    }
    return a;
}

// Ray segments.  A launch with few rays fills a fraction of the GPU's warp
// slots while each thread walks some hundred cells in sequence.  Its rays are
// marched by SEG2D threads each, one per band of columns along the major axis
// (so the lanes of a warp, neighbouring rays, stay on common columns), and the
// block adds the bands' sums in order before the end correction (a different
// order of FP32 additions than one thread's: the results differ in the last
// bits).  Used up to SEG2D_MAX_RAYS rays per launch (batch x views x pixels), or
// SEG2D_MAX_RAYS_SHARED where the slices of a batch share their geometry and a
// thread can take several: measured per call, segments / one thread per ray,
// 256^2 parallel slices, 66 k rays 0.139 / 0.191 ms, 132 k (two slices) 0.187 /
// 0.204, 198 k (three) 0.238 / 0.221; one 387 x 451 fan slice (234 k) 0.348 /
// 0.384, one 512^2 fan slice (369 k) 0.555 / 0.551.
constexpr int SEG2D = 4;
constexpr long long SEG2D_MAX_RAYS = 300000, SEG2D_MAX_RAYS_SHARED = 150000;

// The number of the ray's samples at alphas below `limit`, at most kmax, and
// the alpha that follows them.
__device__ __forceinline__ int samples_before(const Ray2D &ray, float limit, int kmax, float &a)
{
    int n = 0;
    float delta, next;
    a = ray.a;
    for (; a < limit && n < kmax; a = next) n += alpha_run(a, limit, ray.step, kmax - n, delta, next);
    return n;
}

// The sums of one ray's samples, sample 0 with weight 1/2 (SEG > 1: those of
// band `seg` of the `extent` columns), and for the thread that holds the last
// sample its value, the value at the exit and the end correction's last step
// (am - fl(a_n - step)).
template <int SEG, int NS, typename Taps>
__device__ __forceinline__ void march_ray(const Ray2D &ray, const Taps &taps, unsigned mask, int seg, int extent,
                                          float (&sum)[NS], float (&last)[NS], float (&end_val)[NS],
                                          float &last_step, bool &holds_last)
{
    int kmax = march2d_max_iter(ray.a, ray.am, ray.step), k0 = 0;
    float a = ray.a;
    if (SEG > 1) {
        // band boundaries in the ray's direction; neighbouring bands evaluate
        // the same bound, so every sample falls in one band (a bound that is
        // not a number, or behind the ray, leaves the earlier band empty)
        auto bound = [&](int i) {
            const float m = (float)extent * ((float)(ray.gm < 0.0f ? SEG - i : i) / (float)SEG);
            return fminf((m - ray.bm) / ray.gm, ray.am);
        };
        if (seg > 0) k0 = samples_before(ray, bound(seg), kmax, a);
        float b;  // the alpha after the band: not below the exit if the band holds the last sample
        const int k1 = samples_before(ray, seg < SEG - 1 ? bound(seg + 1) : ray.am, kmax, b);
        holds_last = k1 > k0 && (!(b < ray.am) || k1 == kmax);
        kmax = max(k1 - k0, 0);
    } else {
        holds_last = a < ray.am && kmax > 0;
    }
    float a_last;
    const float a_end = sum_cells<NS>(ray, a, kmax, taps, mask, sum, a_last);
    auto sample = [&](float al, int s) {
        const FloorFrac fm = floor_frac(ray.m(al)), fn = floor_frac(ray.n(al));
        return bilinear(taps(fm.i, fn.i, s), fm.f, fn.f);
    };
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        if (k0 == 0 && kmax > 0 && a < ray.am) sum[s] -= 0.5f * sample(a, s);
        if (holds_last) last[s] = sample(a_last, s), end_val[s] = sample(ray.am, s);
    }
    if (holds_last) last_step = ray.am - (a_end - ray.step);
}

// SEG = 1: one thread per detector pixel and NS slices (NS > 1: slices that
// share the geometry).  SEG > 1: FP2_BLOCK / SEG pixels per block, warp w of
// the block marching range w of their rays.
template <typename T, typename Tout, bool FAN, int SEG, int NS>
// (8 blocks per SM, 64 registers, hold the walk; four slices need 72.  More
// or fewer resident blocks measured within 1 to 5 % slower.)
__global__ void __launch_bounds__(FP2_BLOCK, NS >= 3 ? 7 : 8)
    projection2d_kernel(const T *__restrict__ vol, const float4 *__restrict__ cells_x,
                        const float4 *__restrict__ cells_y, Tout *__restrict__ sino, Geom2D geo,
                        int X, int Y, int W, int n_proj, int batch, int geom_batch)
{
    constexpr int RAYS = FP2_BLOCK / SEG;  // rays per block
    static_assert(RAYS % 32 == 0, "warps within a segment");
    static_assert(SEG == 1 || NS == 1, "ranges take one slice");
    const int lane = threadIdx.x % RAYS, seg = threadIdx.x / RAYS;
    const int u = blockIdx.x * RAYS + lane;
    const int p = blockIdx.y;
    const int b = blockIdx.z * NS;
    const bool live = u < W;
    const int g = geom_batch == 1 ? 0 : b;
    const float sx = geo.volume_spacing[2 * g + 1], sy = geo.volume_spacing[2 * g + 0];
    const float ox = geo.volume_origin[2 * g + 1], oy = geo.volume_origin[2 * g + 0];
    const float ds = geo.detector_spacing[g], dorg = geo.detector_origin[g];
    const float2 ray_in = reinterpret_cast<const float2 *>(geo.rays)[(size_t)g * n_proj + p];
    const float uu = __fmaf_rn((float)u, ds, dorg);  // index_to_physical, helper_grid.h

    double srcx, srcy, rx, ry;
    if (!FAN) {
        // par_projector_2D_CudaKernel.cu.cc:120-132.  The virtual source point
        // is formed in FP32 as the reference forms it (ray * (-sid) + u_vec *
        // u, the second product fused) before the FP64 box test: a ray that
        // grazes the box -- along an axis with a 1e-17 cross component, say
        // -- enters or misses on that rounding, as in the reference.
        const float fx = (float)X, fy = (float)Y;
        const float sid =
            __fmul_rn(sqrtf(__fadd_rn(__fmul_rn(__fmul_rn(__fmul_rn(fx, sx), fx), sx),
                                      __fmul_rn(__fmul_rn(__fmul_rn(fy, sy), fy), sy))),
                      1.2f);
        rx = ray_in.x;
        ry = ray_in.y;
        srcx = (double)__fmaf_rn(-ray_in.y, uu, __fmul_rn(ray_in.x, -sid));
        srcy = (double)__fmaf_rn(ray_in.x, uu, __fmul_rn(ray_in.y, -sid));
    } else {
        // fan_projector_2D_CudaKernel.cu.cc:122-133
        const double sid = geo.sid[g], sdd = geo.sdd[g];
        srcx = ray_in.x * -sid;
        srcy = ray_in.y * -sid;
        const double lx = ray_in.x * sdd + (double)(-ray_in.y) * uu;
        const double ly = ray_in.y * sdd + (double)ray_in.x * uu;
        const double inv = 1.0 / sqrt(lx * lx + ly * ly);
        rx = lx * inv;
        ry = ly * inv;
    }

    // box in mm (the reference's -0.5 is in mm, :38-39,50-51), FP64
    double amin = 0.0, amax = CUDART_INF;
    if (rx != 0.0) {
        const double e0 = (double)ox - 0.5, e1 = (double)X * sx + ox - 0.5;
        const double rc = 1.0 / rx;
        const double a0 = (e0 - srcx) * rc, a1 = (e1 - srcx) * rc;
        amin = fmin(a0, a1);
        amax = fmax(a0, a1);
    }
    if (ry != 0.0) {
        const double e0 = (double)oy - 0.5, e1 = (double)Y * sy + oy - 0.5;
        const double rc = 1.0 / ry;
        const double a0 = (e0 - srcy) * rc, a1 = (e1 - srcy) * rc;
        amin = fmax(amin, fmin(a0, a1));
        amax = fmin(amax, fmax(a0, a1));
    }

    Ray2D ray;
    ray.step = 0.2f * fminf(sx, sy);
    const float dx = (float)rx, dy = (float)ry;
    float sum[NS], last[NS], end_val[NS], last_step = 0.0f;
#pragma unroll
    for (int s = 0; s < NS; ++s) sum[s] = last[s] = end_val[s] = 0.0f;
    bool holds_last = false;
    const bool hit = live && ray.step > 0.0f && amin < amax;
    // sample positions in index space: idx = (src + a r - o) / s; the major
    // axis is the one the view's rays run mostly along (fan: the central ray)
    const bool along_x = fabsf(ray_in.x) > fabsf(ray_in.y);
    const float bx = (float)((srcx - ox) / sx), by = (float)((srcy - oy) / sy);
    const float gx = dx * (1.0f / sx), gy = dy * (1.0f / sy);
    ray.bm = along_x ? bx : by, ray.bn = along_x ? by : bx;
    ray.gm = along_x ? gx : gy, ray.gn = along_x ? gy : gx;
    ray.a = (float)amin;
    ray.am = (float)amax;
    const int M = along_x ? X : Y, N = along_x ? Y : X;
    // the last slices of a batch that NS does not divide: the thread's
    // slices are the batch's last NS
    const int b0 = NS == 1 ? b : min(b, batch - NS);
    if (cells_x) {
        const size_t slice = (size_t)(X + 3) * (Y + 3);
        const float4 *cells = (along_x ? cells_y : cells_x) + b0 * slice;
        const unsigned pitch = N + 3;
        // every position of the march lies between its two end points (half a
        // cell of slack for the rounding of the positions)
        const float m0 = ray.m(ray.a), n0 = ray.n(ray.a), m1 = ray.m(ray.am), n1 = ray.n(ray.am);
        const float mmax = (float)M + 0.5f, nmax = (float)N + 0.5f;
        const bool inside = hit && m0 >= -1.5f && m1 >= -1.5f && m0 <= mmax && m1 <= mmax && n0 >= -1.5f &&
                            n1 >= -1.5f && n0 <= nmax && n1 <= nmax && max(X, Y) < (1 << 20);
        const unsigned mask = __ballot_sync(0xffffffffu, inside);
        if (inside)
            march_ray<SEG, NS>(ray, CellTaps<false>{cells, slice, pitch, M, N}, mask, seg, M, sum, last, end_val,
                               last_step, holds_last);
        else if (hit)
            march_ray<SEG, NS>(ray, CellTaps<true>{cells, slice, pitch, M, N}, 0u, seg, M, sum, last, end_val, last_step,
                               holds_last);
    } else if (hit) {
        const size_t slice = (size_t)X * Y;
        march_ray<SEG, NS>(ray, BorderTaps<T>{vol + b0 * slice, slice, along_x ? 1 : X, along_x ? X : 1, M, N}, 0u, seg, M,
                           sum, last, end_val, last_step, holds_last);
    }
    if (SEG > 1) {
        __shared__ float s_sum[SEG][RAYS];
        __shared__ float s_last[RAYS], s_end[RAYS], s_step[RAYS];
        s_sum[seg][lane] = sum[0];
        if (holds_last) s_last[lane] = last[0], s_end[lane] = end_val[0], s_step[lane] = last_step;
        __syncthreads();
        if (seg != 0) return;
#pragma unroll
        for (int r = 1; r < SEG; ++r) sum[0] += s_sum[r][lane];
        if (sum[0] != 0.0f) last[0] = s_last[lane], end_val[0] = s_end[lane], last_step = s_step[lane];
    }
    if (!live) return;
    const float scale = sqrtf((dx * sx) * (dx * sx) + (dy * sy) * (dy * sy));  // :141
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        float pixel = sum[s] * ray.step;
        if (pixel > 0.0f) {  // :88-100
            pixel -= 0.5f * ray.step * last[s];
            pixel += 0.5f * last_step * last[s];
            pixel += 0.5f * last_step * end_val[s];
        }
        const int bs = NS == 1 ? b : min(b, batch - NS) + s;
        store_from_float(sino + ((size_t)bs * n_proj + p) * W + u, pixel * scale);
    }
}

// The taps p[0] and p[1] of a sinogram row, one whose flag is clear zero
// (CHECK), as their value a and difference d for the lerp a + t d: FP32 keeps
// the taps themselves (its lerp is the reference's form), 16-bit storage takes
// the difference with one mixed-precision subtraction (lerp_first's bits).
template <bool CHECK, typename T>
__device__ __forceinline__ float2 row_taps(const T *p, bool in0, bool in1)
{
    if constexpr (std::is_same<T, float>::value) {
        return pair(!CHECK || in0 ? __ldg(p) : 0.0f, !CHECK || in1 ? __ldg(p + 1) : 0.0f);
    } else {
        const unsigned short *q = reinterpret_cast<const unsigned short *>(p);
        const unsigned short r0 = !CHECK || in0 ? __ldg(q) : 0, r1 = !CHECK || in1 ? __ldg(q + 1) : 0;
        if constexpr (std::is_same<T, __half>::value) {
            const float a = __half2float(__ushort_as_half(r0));
            return pair(a, sub_f32_f16<false>(r1, a));
        } else {
            const float a = __uint_as_float((unsigned)r0 << 16);
            return pair(a, sub_f32_bf16<false>(r1, a));
        }
    }
}

// acc[s] += w * lerp(taps of slice s, t), slices in pairs on the packed FP32
// instructions (the same roundings as one at a time)
template <bool CHECK, int NS, typename T>
__device__ __forceinline__ void add_row_lerps(const char *const (&base)[NS], unsigned off, bool in0, bool in1, float t,
                                              float w, float (&acc)[NS])
{
    constexpr bool F32 = std::is_same<T, float>::value;
    float2 v[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) v[s] = row_taps<CHECK>(reinterpret_cast<const T *>(base[s] + off), in0, in1);
#pragma unroll
    for (int s = 0; s + 1 < NS; s += 2) {
        const float2 a = pair(v[s].x, v[s + 1].x), b = pair(v[s].y, v[s + 1].y);
        const float2 base = F32 ? __ffma2_rn(a, pair(-t, -t), a) : a;
        const float2 l = __ffma2_rn(b, pair(t, t), base);
        const float2 r = __ffma2_rn(l, pair(w, w), pair(acc[s], acc[s + 1]));
        acc[s] = r.x, acc[s + 1] = r.y;
    }
    if constexpr (NS % 2 != 0) {
        constexpr int s = NS - 1;
        acc[s] = fmaf(F32 ? lerp_ref(v[s].x, v[s].y, t) : fmaf(t, v[s].y, v[s].x), w, acc[s]);
    }
}

// Detector index of pixel c for one fan view by the reference's own FP32
// steps: source r * (-SID), central point source + r * SDD, intersectLines2D
// (pixel, source, centre, centre + (-r.y, r.x)) and physical_to_index
// (fan_backprojector_2D_CudaKernel.cu.cc:47-59, helper_geometry_gpu.h:28-44),
// each operation rounded once.  Used for pixels near the source's depth,
// where the lines are nearly parallel and the reference's FP32 intersection
// differs from the exact one: its denominator below 1e-6 gives NaN, which the
// texture unit samples as coordinate 0 (measured on B200: half of the view's
// first texel, i.e. index -0.5); just above it, a far-off point.
__device__ __forceinline__ float fan_index_reference_steps(float cx, float cy, float rx, float ry, float sid, float sdd,
                                                        float dorg, float ds)
{
    const float srcx = __fmul_rn(rx, -sid), srcy = __fmul_rn(ry, -sid);
    const float cpx = __fadd_rn(srcx, __fmul_rn(rx, sdd)), cpy = __fadd_rn(srcy, __fmul_rn(ry, sdd));
    const float detx = -ry, dety = rx;
    const float p4x = __fadd_rn(cpx, detx), p4y = __fadd_rn(cpy, dety);
    const float a1 = __fsub_rn(cx, srcx), b1 = __fsub_rn(cpy, p4y);
    const float a2 = __fsub_rn(cy, srcy), b2 = __fsub_rn(cpx, p4x);
    const float dn = __fsub_rn(__fmul_rn(a1, b1), __fmul_rn(a2, b2));
    if (dn < 1.0e-6f && dn > -1.0e-6f) return -0.5f;
    const float x12 = __fsub_rn(__fmul_rn(cx, srcy), __fmul_rn(cy, srcx));
    const float x34 = __fsub_rn(__fmul_rn(cpx, p4y), __fmul_rn(cpy, p4x));
    const float x = __fdiv_rn(__fsub_rn(__fmul_rn(x12, b2), __fmul_rn(a1, x34)), dn);
    const float y = __fdiv_rn(__fsub_rn(__fmul_rn(x12, b1), __fmul_rn(a2, x34)), dn);
    const float s = __fadd_rn(__fmul_rn(x, detx), __fmul_rn(y, dety));
    return __fdiv_rn(__fsub_rn(s, dorg), ds);
}

// One thread per pixel, views in chunks of BP2_CHUNK whose per-view
// constants the block first puts in shared memory (one view per thread):
// parallel beam (-r.y, r.x) / detector spacing, fan beam (r.x, r.y, SID |r|^2,
// SDD |r|^2 / detector spacing), so a view costs each pixel one broadcast load.
// Fan beam: a geometry in which some view's source depth line comes within
// 2e-2 mm of the slice (the source inside or at the field) needs the
// reference's FP32 steps near that line (fan_index_reference_steps), which
// would cost the common case registers and occupancy; two instantiations are
// launched instead, NEAR_DEPTH = false and true, and each block checks the
// geometry first and leaves the work to the instantiation that matches it.
// VSPLIT > 1 (launches of few pixels, which leave most warp slots idle): the
// block's 8 thread rows are VSPLIT groups of 8 / VSPLIT pixel rows, group v
// summing part v of every chunk's views; the groups' sums are added in
// order at the end (the results differ from one thread's in the last bits).
// NS > 1 (slices that share their geometry): the thread's pixel in NS slices;
// a view's detector position, weight and tap flags are computed once, and a
// block whose pixels all project inside the rows leaves the flags out.  One slice
// of a fan or in view groups keeps flags and row pointers: a second loop and its
// test cost it more than they save (180 views: one fan slice of 128^2, 30 -> 24 us
// without; 16 of 256^2 with a geometry each, in fan beam, 341 -> 251 us; but one
// parallel slice of 1024^2, 90 views, 72 us with, 92 without).
template <typename T, typename Tout, bool FAN, bool NEAR_DEPTH, int VSPLIT, int NS>
// (eight slices: up to 128 registers; held to 80 / 64 / 48 the 64-slice fan
// batch in FP16 takes 2.89 / 3.36 / 3.82 instead of 2.77 ms; two parallel slices:
// 32 registers, two of 256^2 in FP32 at 180 views 41 -> 29 us)
__global__ void __launch_bounds__(BP2_BLOCK_X *BP2_BLOCK_Y, NS == 8 ? 2 : (NS == 2 && !FAN ? 8 : 0))
    backprojection2d_kernel(const T *__restrict__ sino, Tout *__restrict__ vol, Geom2D geo, int X, int Y, int W,
                            int n_proj, int batch, int geom_batch)
{
    constexpr int ROWS = BP2_BLOCK_Y / VSPLIT;  // pixel rows per block
    constexpr bool ALWAYS_FLAGS = NS == 1 && (FAN || VSPLIT > 1);
    __shared__ float4 tab[BP2_CHUNK];
    const int vg = threadIdx.y / ROWS;          // view group
    const int i0 = blockIdx.x * BP2_BLOCK_X, j0 = blockIdx.y * ROWS;
    const int i = i0 + threadIdx.x, j = j0 + threadIdx.y % ROWS;
    const int tid = threadIdx.y * BP2_BLOCK_X + threadIdx.x;
    // the last slices of a batch that NS does not divide: the batch's last NS
    const int b = NS == 1 ? blockIdx.z : min((int)blockIdx.z * NS, batch - NS);
    const bool live = i < X && j < Y;
    const int g = geom_batch == 1 ? 0 : b;
    const float sx = geo.volume_spacing[2 * g + 1], sy = geo.volume_spacing[2 * g + 0];
    const float ox = geo.volume_origin[2 * g + 1], oy = geo.volume_origin[2 * g + 0];
    const float2 *rays = reinterpret_cast<const float2 *>(geo.rays) + (size_t)g * n_proj;
    float sid = 0.0f, sdd = 0.0f;
    if (FAN) {
        sid = geo.sid[g];
        sdd = geo.sdd[g];
        // a view's depth <c - src, r> is affine in the pixel centre c, so its
        // extremes over the slice are at the corners of the pixel-centre box
        const float x0 = ox, x1 = ox + (float)(X - 1) * sx, y0 = oy, y1 = oy + (float)(Y - 1) * sy;
        bool near = false;
        for (int n = tid; n < n_proj; n += BP2_BLOCK_X * BP2_BLOCK_Y) {
            const float2 r = __ldg(&rays[n]);
            const float base = sid * (r.x * r.x + r.y * r.y);
            const float d0 = fmaf(x0, r.x, fmaf(y0, r.y, base)), d1 = fmaf(x1, r.x, fmaf(y0, r.y, base));
            const float d2 = fmaf(x0, r.x, fmaf(y1, r.y, base)), d3 = fmaf(x1, r.x, fmaf(y1, r.y, base));
            near |= fminf(fminf(d0, d1), fminf(d2, d3)) < 2.0e-2f && fmaxf(fmaxf(d0, d1), fmaxf(d2, d3)) > -2.0e-2f;
        }
        if (__syncthreads_or(near) != NEAR_DEPTH) return;  // the other instantiation's block
    }
    const float ds = geo.detector_spacing[g], dorg = geo.detector_origin[g];
    const float ids = 1.0f / ds;
    const float sdo = dorg * ids;  // detector origin in pixels
    const float cx = (float)i * sx + ox, cy = (float)j * sy + oy;
    const size_t slice = (size_t)n_proj * W;
    const T *sino_b = sino + b * slice;
    float acc[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) acc[s] = 0.0f;
    // the pixel's detector position in the view of constants q and its weight
    auto position = [&](const float4 &q, float &w) {
        w = 1.0f;
        if (!FAN) return fmaf(cx, q.x, fmaf(cy, q.y, -sdo));  // (<c, d> - origin) / spacing, :51
        // intersectLines2D(pixel, source, centre, centre + det) of
        // fan_backprojector_2D_CudaKernel.cu.cc:52-57 in closed form:
        // s = SDD |r|^2 <c, d> / (<c, r> + SID |r|^2), weight 1 / |c - src|^2
        const float cd = fmaf(cy, q.x, -cx * q.y);
        const float cr = fmaf(cx, q.x, cy * q.y);
        const float den = cr + q.z;  // <c - src, r>: the pixel's depth from the source
        float sidx = fmaf(q.w * cd, fast_rcp(den), -sdo);
        // within 1e-2 mm of the source's depth, the reference's FP32 steps decide
        if (NEAR_DEPTH && fabsf(den) < 1.0e-2f)
            sidx = fan_index_reference_steps(cx, cy, q.x, q.y, sid, sdd, dorg, ds);
        const float ex = fmaf(q.x, sid, cx), ey = fmaf(q.y, sid, cy);
        w = fast_rcp(fmaf(ex, ex, ey * ey));
        return sidx;
    };
    // detector positions of pixels inside the field stay far below 2^22;
    // a pixel whose position is larger misses the row either way
    auto clamped = [&](float sidx) { return fminf(fmaxf(sidx, -4.0f), (float)W + 4.0f); };
    // (offsets within a chunk are 32-bit: shared rows of 2^22 pixels and more
    // go one view at a time, taps past element 2^30 - 16 count as outside)
    const int chunk = ALWAYS_FLAGS || W < (1 << 22) ? BP2_CHUNK : 1;
    for (int n0 = 0; n0 < n_proj; n0 += chunk) {
        const int cnt = min(chunk, n_proj - n0);
        __syncthreads();  // the previous chunk's constants are no longer read
        bool all = W < (1 << 20);
        if (tid < cnt) {
            const float2 r = __ldg(&rays[n0 + tid]);
            float4 q;
            if (FAN) {
                const float rr = r.x * r.x + r.y * r.y;
                q = make_float4(r.x, r.y, sid * rr, sdd * rr * ids);
            } else {
                // detector direction (-r.y, r.x), par_backprojector_2D_CudaKernel.cu.cc:48-49
                q = make_float4(-r.y * ids, r.x * ids, 0.0f, 0.0f);
            }
            tab[tid] = q;
            // the block's pixels project between its corners' projections
            // (the detector position is monotonic along any line of pixels at
            // positive depth): all of them between the row's first and last
            // tap, with half a pixel of slack, need no tap flags
            if (!ALWAYS_FLAGS) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float px = (float)((c & 1) ? min(i0 + BP2_BLOCK_X, X) - 1 : i0) * sx + ox;
                    const float py = (float)((c & 2) ? min(j0 + ROWS, Y) - 1 : j0) * sy + oy;
                    float s = fmaf(px, q.x, fmaf(py, q.y, -sdo));
                    if (FAN) {
                        const float den = fmaf(px, q.x, py * q.y) + q.z;
                        s = fmaf(q.w * fmaf(py, q.x, -px * q.y), fast_rcp(den), -sdo);
                        all = all && den > 0.1f;
                    }
                    all = all && s >= 0.5f && s <= (float)W - 1.5f;
                }
            }
        }
        bool inside = false;
        if (ALWAYS_FLAGS)
            __syncthreads();
        else
            inside = __syncthreads_and(all);  // for all the chunk's views
        if (!live) continue;
        const int kb = VSPLIT == 1 ? 0 : vg * cnt / VSPLIT, ke = VSPLIT == 1 ? cnt : (vg + 1) * cnt / VSPLIT;
        if constexpr (ALWAYS_FLAGS) {
            // one slice: row pointers and flags, four views' loads in flight
            const T *row = sino_b + (size_t)(n0 + kb) * W;
#pragma unroll(NEAR_DEPTH ? 1 : 4)
            for (int k = kb; k < ke; ++k, row += W) {
                float w;
                const FloorFrac ff = floor_frac(clamped(position(tab[k], w)));
                const float2 v = row_taps<true>(row + ff.i, (unsigned)ff.i < (unsigned)W, (unsigned)(ff.i + 1) < (unsigned)W);
                acc[0] = fmaf(std::is_same<T, float>::value ? lerp_ref(v.x, v.y, ff.f) : fmaf(ff.f, v.y, v.x), w, acc[0]);
            }
        } else {
            auto add_views = [&](auto check_c) {
                constexpr bool CHECK = decltype(check_c)::value;
                // offsets count from 8 elements before the chunk's first row, so
                // a row's element -1 has one too
                const char *base[NS];
#pragma unroll
                for (int s = 0; s < NS; ++s)
                    base[s] = reinterpret_cast<const char *>(sino_b + s * slice + (size_t)n0 * W) - 8 * sizeof(T);
                const unsigned Wt = min(W, (1 << 30) - 16);
                unsigned row = (unsigned)kb * (unsigned)W + 8u;
#pragma unroll(NEAR_DEPTH ? 1 : (NS == 1 ? 4 : 2))
                for (int k = kb; k < ke; ++k, row += W) {
                    float w;
                    const float sidx = position(tab[k], w);
                    const FloorFrac ff = floor_frac(CHECK ? clamped(sidx) : sidx);
                    const bool in0 = (unsigned)ff.i < Wt, in1 = (unsigned)(ff.i + 1) < Wt;
                    add_row_lerps<CHECK, NS, T>(base, (row + (unsigned)ff.i) * (unsigned)sizeof(T), in0, in1, ff.f, w, acc);
                }
            };
            inside ? add_views(std::false_type{}) : add_views(std::true_type{});
        }
    }
    if (VSPLIT > 1) {
        __shared__ float s_acc[VSPLIT][NS][ROWS][BP2_BLOCK_X];
#pragma unroll
        for (int s = 0; s < NS; ++s) s_acc[vg][s][threadIdx.y % ROWS][threadIdx.x] = acc[s];
        __syncthreads();
        if (vg != 0) return;
#pragma unroll
        for (int r = 1; r < VSPLIT; ++r)
#pragma unroll
            for (int s = 0; s < NS; ++s) acc[s] += s_acc[r][s][threadIdx.y][threadIdx.x];
    }
    if (!live) return;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        float out;
        if (!FAN)
            out = PI_REF * acc[s] / (float)n_proj;  // :58
        else
            out = sid * sdd * PI_REF * acc[s] / (float)n_proj;  // fan_backprojector_2D_CudaKernel.cu.cc:64
        store_from_float(vol + ((size_t)(b + s) * Y + j) * X + i, out);
    }
}

// Both cell copies of the batch: cell (xc, yc), xc in [0, X+2], yc in
// [0, Y+2], has its low corner at pixel (xc-2, yc-2).  A block loads a 33 x 33
// tile along x and writes 32 x 32 cells x-fastest (along x) and y-fastest
// (along y); grid (ceil((X+3)/32), ceil((Y+3)/32), batch), block 32 x 8.
template <typename T>
__global__ void __launch_bounds__(256) pad_cells2d_kernel(const T *__restrict__ in,
                                                          float4 *__restrict__ cells_x,
                                                          float4 *__restrict__ cells_y, int X, int Y)
{
    __shared__ float tile[33][34];  // [y - (yc0-2)][x - (xc0-2)], widened
    const int Xc = X + 3, Yc = Y + 3;
    const int xc0 = blockIdx.x * 32, yc0 = blockIdx.y * 32;
    const T *img = in + (size_t)blockIdx.z * X * Y;
    for (int r = threadIdx.y; r < 33; r += 8) {
        const int y = yc0 - 2 + r;
        for (int c = threadIdx.x; c < 33; c += 32) {
            const int x = xc0 - 2 + c;
            float v = 0.0f;
            if (y >= 0 && y < Y && x >= 0 && x < X) v = load_as_float(img + (size_t)y * X + x);
            tile[r][c] = v;
        }
    }
    __syncthreads();
    const size_t slice = (size_t)blockIdx.z * Xc * Yc;
    for (int r = threadIdx.y; r < 32; r += 8) {
        {  // x-fastest: thread x along xc
            const int xc = xc0 + threadIdx.x, yc = yc0 + r;
            if (xc < Xc && yc < Yc)
                cells_x[slice + (size_t)yc * Xc + xc] = make_float4(
                    tile[r][threadIdx.x], tile[r + 1][threadIdx.x], tile[r][threadIdx.x + 1], tile[r + 1][threadIdx.x + 1]);
        }
        {  // y-fastest: thread x along yc
            const int yc = yc0 + threadIdx.x, xc = xc0 + r;
            if (xc < Xc && yc < Yc)
                cells_y[slice + (size_t)xc * Yc + yc] = make_float4(
                    tile[threadIdx.x][r], tile[threadIdx.x][r + 1], tile[threadIdx.x + 1][r], tile[threadIdx.x + 1][r + 1]);
        }
    }
}

// Slices per thread (1 to 4) of a batch that shares its geometry: the fewest
// instructions, a thread costing `walk` per step and `slice` more for each
// slice, the last group repeating slices where the number does not divide the
// batch (three fan slices of 387 x 451 by threes instead of twice two: forward
// 0.655 -> 0.460 ms, back 0.202 -> 0.147; also the best for three slices of 256^2,
// 66 k rays, where it leaves the fewest threads: 0.187 -> 0.179).
int best_slices(int batch, int walk, int slice)
{
    int best = 1;
    long long best_cost = (long long)batch * (walk + slice);
    for (int ns = 2; ns <= 4 && ns <= batch; ++ns) {
        const long long cost = (long long)((batch + ns - 1) / ns) * (walk + ns * slice);
        if (cost < best_cost) best = ns, best_cost = cost;
    }
    return best;
}

template <typename Tin, typename Tout>
cudaError_t fp_typed(const void *volume, void *sinogram, bool fan, const Dims2D &d, const Geom2D &g,
                     void *workspace, cudaStream_t stream)
{
    using C = float4;
    C *cells_x = nullptr, *cells_y = nullptr;
    if (workspace) {
        const size_t n = (size_t)d.batch * (d.vol_x + 3) * (d.vol_y + 3);
        cells_x = (C *)workspace;
        cells_y = (C *)((char *)workspace + (n * sizeof(C) + 255) / 256 * 256);
        const dim3 tgrid((d.vol_x + 3 + 31) / 32, (d.vol_y + 3 + 31) / 32, d.batch);
        pad_cells2d_kernel<Tin><<<tgrid, dim3(32, 8), 0, stream>>>((const Tin *)volume, cells_x, cells_y, d.vol_x,
                                                                  d.vol_y);
    }
    // segments per ray for launches of few rays (see SEG2D), else up to four
    // slices of one geometry per thread (the walk costs a visit about 33
    // instructions, a slice 9 more: 64 fan slices of 512^2, FP16, 41.4 -> 21.7 ms
    // by cell visits and four slices per thread, 13.2 ms with aligned columns,
    // 12.0 ms on packed instructions; eight slices per thread 12.2 ms)
    const bool share = d.geom_batch == 1 && d.batch >= 2;
    const bool segs = (long long)d.batch * d.n_proj * d.det_w <= (share ? SEG2D_MAX_RAYS_SHARED : SEG2D_MAX_RAYS);
    const int ns = segs || !share ? 1 : best_slices(d.batch, 33, 9);
    const int rays = segs ? FP2_BLOCK / SEG2D : FP2_BLOCK;
    const dim3 grid((d.det_w + rays - 1) / rays, d.n_proj, (d.batch + ns - 1) / ns);
    auto launch = [&](auto kernel) {
        kernel<<<grid, FP2_BLOCK, 0, stream>>>((const Tin *)volume, cells_x, cells_y, (Tout *)sinogram, g, d.vol_x,
                                               d.vol_y, d.det_w, d.n_proj, d.batch, d.geom_batch);
    };
    auto launch_beam = [&](auto fan_c) {
        constexpr bool FAN = decltype(fan_c)::value;
        if (segs)
            launch(projection2d_kernel<Tin, Tout, FAN, SEG2D, 1>);
        else if (ns == 4)
            launch(projection2d_kernel<Tin, Tout, FAN, 1, 4>);
        else if (ns == 3)
            launch(projection2d_kernel<Tin, Tout, FAN, 1, 3>);
        else if (ns == 2)
            launch(projection2d_kernel<Tin, Tout, FAN, 1, 2>);
        else
            launch(projection2d_kernel<Tin, Tout, FAN, 1, 1>);
    };
    fan ? launch_beam(std::true_type{}) : launch_beam(std::false_type{});
    return cudaGetLastError();
}

template <typename Tin, typename Tout>
cudaError_t bp_typed(const void *sinogram, void *volume, bool fan, const Dims2D &d, const Geom2D &g,
                     cudaStream_t stream)
{
    const dim3 block(BP2_BLOCK_X, BP2_BLOCK_Y);
    // Slices of one geometry per thread.  A view costs a pixel about 24
    // instructions (fan) and a slice 5 to 6 more: per call, 64 fan slices of
    // 512^2 in FP16 7.47 ms with one, 2.9 - 3.1 with four, 2.77 with eight;
    // eight leave smaller launches short of threads (48 parallel slices of
    // 256^2, 3.1 M pixels: 0.435 ms with four, 0.497 with eight; 32 of 512^2,
    // 8.4 M: 1.74 / 1.44).
    const long long pixels = (long long)d.vol_x * d.vol_y;
    // Launches of few pixels need the threads: 180 views, per call, one slice per
    // thread / several: eight 64^2 fan slices (33 k pixels) 26 / 36 us, four of 128^2
    // (66 k) 30 / 36, two of 200^2 (80 k) 38 / 26; parallel 23 / 31, 22 / 31, 31 / 29.
    const bool share = d.geom_batch == 1 && d.batch >= 2 && d.batch * pixels >= BP2_SHARE_MIN_PIXELS;
    const int ns = !share                                                     ? 1
                   : d.batch >= 8 && d.batch * pixels >= BP2_NS8_MIN_PIXELS ? 8
                                                                              : best_slices(d.batch, 24, 6);
    const int groups = (d.batch + ns - 1) / ns;
    // view groups for launches of few threads (see VSPLIT; three fan slices of
    // 387 x 451, 349 k threads: 0.248 ms with, 0.272 without; four of 512^2, 262 k:
    // 0.298 / 0.322; 16 of 512^2, 1.05 M: 0.920 / 0.855; one slice per thread, 180
    // views: one parallel 512^2 slice, 262 k pixels, 57 us with, 52 without; 320^2,
    // 102 k, 35 / 32; fan 79 / 79 and 40 / 52)
    const bool split = groups * pixels <= (ns == 1 ? BP2_SPLIT_MAX_PIXELS : BP2_SPLIT_MAX_SHARED);
    const int rows = split ? BP2_BLOCK_Y / BP2_VSPLIT : BP2_BLOCK_Y;
    const dim3 grid((d.vol_x + BP2_BLOCK_X - 1) / BP2_BLOCK_X, (d.vol_y + rows - 1) / rows, groups);
    auto launch = [&](auto kernel) {
        kernel<<<grid, block, 0, stream>>>((const Tin *)sinogram, (Tout *)volume, g, d.vol_x, d.vol_y, d.det_w,
                                           d.n_proj, d.batch, d.geom_batch);
    };
    auto launch_slices = [&](auto ns_c) {
        constexpr int NS = decltype(ns_c)::value;
        // (eight slices leave at least BP2_NS8_MIN_PIXELS / 8 threads: no view groups)
        auto launch_split = [&](auto vsplit_c) {
            constexpr int VSPLIT = decltype(vsplit_c)::value;
            if (fan) {  // every block runs in exactly one of the two (see the kernel)
                launch(backprojection2d_kernel<Tin, Tout, true, false, VSPLIT, NS>);
                launch(backprojection2d_kernel<Tin, Tout, true, true, VSPLIT, NS>);
            } else {
                launch(backprojection2d_kernel<Tin, Tout, false, false, VSPLIT, NS>);
            }
        };
        if constexpr (NS < 8) {
            if (split) return launch_split(std::integral_constant<int, BP2_VSPLIT>{});
        }
        launch_split(std::integral_constant<int, 1>{});
    };
    if (ns == 8)
        launch_slices(std::integral_constant<int, 8>{});
    else if (ns == 4)
        launch_slices(std::integral_constant<int, 4>{});
    else if (ns == 3)
        launch_slices(std::integral_constant<int, 3>{});
    else if (ns == 2)
        launch_slices(std::integral_constant<int, 2>{});
    else
        launch_slices(std::integral_constant<int, 1>{});
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_projection2d(const void *volume, void *sinogram, int in_dtype, int out_dtype, bool fan,
                                const Dims2D &d, const Geom2D &g, void *workspace, cudaStream_t stream)
{
    return dispatch_dtypes(in_dtype, out_dtype, [&](auto tin, auto tout) {
        using Tin = typename decltype(tin)::type;
        using Tout = typename decltype(tout)::type;
        return fp_typed<Tin, Tout>(volume, sinogram, fan, d, g, workspace, stream);
    });
}

cudaError_t launch_backprojection2d(const void *sinogram, void *volume, int in_dtype, int out_dtype, bool fan,
                                    const Dims2D &d, const Geom2D &g, cudaStream_t stream)
{
    return dispatch_dtypes(in_dtype, out_dtype, [&](auto tin, auto tout) {
        using Tin = typename decltype(tin)::type;
        using Tout = typename decltype(tout)::type;
        return bp_typed<Tin, Tout>(sinogram, volume, fan, d, g, stream);
    });
}

}  // namespace pyronn
