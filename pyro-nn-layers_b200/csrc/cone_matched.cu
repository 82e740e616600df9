// cone_matched.cu -- matched cone backprojector: the exact transpose of the
// software-interpolation forward projector.
//
// The reference's backprojector (voxel-driven, bilinear on the detector,
// 1/w^2 weights, cone_backprojector_3D_CudaKernel.cu.cc:84-118) is not the
// transpose of its ray-driven projector, so <A x, y> != <x, A^T y>.  This
// kernel walks every ray with the forward projector's samples and weights
// (cone_ray.cuh, linear form) and scatters sino[ray] * weight * trilinear
// weight into the eight taps with FP32 atomics: the result is A^T y for the
// linear forward operator, which equals the reference forward projector on
// every ray whose line integral is > 0 (e.g. any non-negative volume).
//
// Given a workspace for them, the rays scatter into CELL accumulators, the
// transpose of the forward's FP32 cell copy: element (x, y, z), z fastest, sums
// what falls on the taps V(x + {0,1}, y + {0,1}) at z, so a sample is two
// adjacent 16-byte vector additions instead of eight scalar atomics to eight
// rows; a second kernel adds each voxel's four cell entries.  Views whose
// detector v axis runs along z lay warps along v, like the forward: a warp's
// additions fall on consecutive cells.  What bounds it: the L2's additions.
#include "common.cuh"
#include "cone_ray.cuh"
#include "internal.h"

namespace pyronn {

namespace {

constexpr int MB_X = 32;
constexpr int MB_Y = 8;

__device__ __forceinline__ void scatter_trilinear(float *__restrict__ vol, float x, float y, float z, float val,
                                                  int X, int Y, int Z)
{
    const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    const int x0 = (int)fx, y0 = (int)fy, z0 = (int)fz;
    const float tx = x - fx, ty = y - fy, tz = z - fz;
    // weights of lerp_ref(a, b, t) = a (1 - t) + b t
    const float wx[2] = {1.0f - tx, tx}, wy[2] = {1.0f - ty, ty}, wz[2] = {1.0f - tz, tz};
#pragma unroll
    for (int dz = 0; dz < 2; ++dz) {
        const int zz = z0 + dz;
        if ((unsigned)zz >= (unsigned)Z) continue;
#pragma unroll
        for (int dy = 0; dy < 2; ++dy) {
            const int yy = y0 + dy;
            if ((unsigned)yy >= (unsigned)Y) continue;
            const float wzy = val * wz[dz] * wy[dy];
#pragma unroll
            for (int dx = 0; dx < 2; ++dx) {
                const int xx = x0 + dx;
                if ((unsigned)xx >= (unsigned)X) continue;
                atomicAdd(vol + ((size_t)zz * Y + yy) * X + xx, wzy * wx[dx]);
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(MB_X *MB_Y)
    cone_scatter_kernel(const T *__restrict__ sino, float *__restrict__ vol, const ConeFpView *__restrict__ views,
                        const float *__restrict__ step_ptr, const float *__restrict__ spacing_ptr, int X, int Y,
                        int Z, int W, int H, int n_proj, int geom_batch)
{
    const int u = blockIdx.x * MB_X + threadIdx.x;
    const int v = blockIdx.y * MB_Y + threadIdx.y;
    const int p = blockIdx.z % n_proj;
    const int b = blockIdx.z / n_proj;
    if (u >= W || v >= H) return;
    const float y = load_as_float(sino + (((size_t)b * n_proj + p) * H + v) * (size_t)W + u);
    if (y == 0.0f) return;
    const int g = geom_batch == 1 ? 0 : b;
    const float step = step_ptr[g];
    if (!in_footprint(views[(size_t)g * n_proj + p], u, v)) return;
    const ConeRay ray = cone_ray_setup(views[(size_t)g * n_proj + p], u, v, X, Y, Z, 0.0, step,
                                       spacing_ptr[g * 3 + 2], spacing_ptr[g * 3 + 1], spacing_ptr[g * 3 + 0]);
    float *vol_b = vol + (size_t)b * Z * Y * X;
    cone_ray_weights(ray, step, [&](float px, float py, float pz, float w) {
        scatter_trilinear(vol_b, px, py, pz, y * w, X, Y, Z);
    });
}

// z entries of a column of cell accumulators beyond the volume's: floors
// [-1, Z] and the next
constexpr int ACC_PLANES = 3;

// Cell accumulators of one volume: [X+2][Y+2][Z+3], element (x + 1, y + 1, z + 1)
// for floors (x, y, z); `cells` is floor (-1, -1, -1).
struct CellAccumulators {
    float4 *cells;
    int X, Y, Z;

    // the cell of floors (x, y, z) in [-1, N]
    __device__ __forceinline__ float4 *cell(int x, int y, int z) const
    {
        return cells + ((size_t)((x + 1) * (Y + 2) + y + 1) * (Z + ACC_PLANES) + (z + 1));
    }
};

// One ray's additions: consecutive samples in one cell (half a step apart by
// default, about 1.4 per cell) are summed in registers and added once.
// CHECK: a sample whose floor lies outside [-1, N] touches no voxel.
template <bool CHECK>
struct CellScatter {
    const CellAccumulators &acc;
    float4 *cur;
    float2 lo[2], hi[2];  // at z, at z + 1: the (x0, x1) pairs of y0 and y1

    __device__ __forceinline__ explicit CellScatter(const CellAccumulators &a) : acc(a), cur(nullptr) { clear(); }
    __device__ __forceinline__ void clear()
    {
        lo[0] = lo[1] = hi[0] = hi[1] = make_float2(0.0f, 0.0f);
    }
    __device__ __forceinline__ void flush()
    {
        if (!cur) return;
        atomicAdd(cur, make_float4(lo[0].x, lo[0].y, lo[1].x, lo[1].y));
        atomicAdd(cur + 1, make_float4(hi[0].x, hi[0].y, hi[1].x, hi[1].y));
    }
    __device__ __forceinline__ void add(float x, float y, float z, float val)
    {
        // x and y, and the weights of each (x0, x1) pair, on the packed FP32
        // instructions
        constexpr float MAGIC = 12582912.0f;  // floor_frac's
        const float2 p = make_float2(x, y), fl = __fadd2_rd(p, make_float2(MAGIC, MAGIC));
        const float2 f = __ffma2_rn(__fadd2_rn(fl, make_float2(-MAGIC, -MAGIC)), make_float2(-1.0f, -1.0f), p);
        const int ix = __float_as_int(fl.x) - FLOOR_BIAS, iy = __float_as_int(fl.y) - FLOOR_BIAS;
        const FloorFrac fz = floor_frac(z);
        if (CHECK && ((unsigned)(ix + 1) > (unsigned)(acc.X + 1) || (unsigned)(iy + 1) > (unsigned)(acc.Y + 1) ||
                      (unsigned)(fz.i + 1) > (unsigned)(acc.Z + 1)))
            return;
        float4 *c = acc.cell(ix, iy, fz.i);
        if (c != cur) {
            flush();
            cur = c;
            clear();
        }
        // weights of lerp_ref(a, b, t) = a (1 - t) + b t
        const float h = val * fz.f, l = val * (1.0f - fz.f), ty0 = 1.0f - f.y;
        const float2 wx = make_float2(1.0f - f.x, f.x);
        const float2 w0 = __fmul2_rn(make_float2(ty0, ty0), wx), w1 = __fmul2_rn(make_float2(f.y, f.y), wx);
        lo[0] = __ffma2_rn(make_float2(l, l), w0, lo[0]), lo[1] = __ffma2_rn(make_float2(l, l), w1, lo[1]);
        hi[0] = __ffma2_rn(make_float2(h, h), w0, hi[0]), hi[1] = __ffma2_rn(make_float2(h, h), w1, hi[1]);
    }
};

template <bool CHECK>
__device__ __forceinline__ void scatter_ray(const ConeRay &ray, float step, float y, const CellAccumulators &acc)
{
    CellScatter<CHECK> s(acc);
    cone_ray_weights(ray, step, [&](float px, float py, float pz, float w) { s.add(px, py, pz, y * w); });
    s.flush();
}

// Grid: ray_block order (cone_ray.cuh).  z mode: a warp is 32 consecutive v at
// one u, its sinogram values staged through shared memory; else 32
// consecutive u.
template <typename T>
__global__ void __launch_bounds__(MB_X *MB_Y)
    cone_scatter_cells_kernel(const T *__restrict__ sino, CellAccumulators acc, const ConeFpView *__restrict__ views,
                              const float *__restrict__ step_ptr, const float *__restrict__ spacing_ptr, int W, int H,
                              int n_proj, int g)
{
    __shared__ float tile[MB_Y][MB_X + 1];
    const RayBlock rb = ray_block(blockIdx.x, W, H, n_proj);
    const ConeFpView &view = views[(size_t)g * n_proj + rb.p];
    const T *img = sino + (size_t)rb.p * H * (size_t)W;
    int u, v;
    float y = 0.0f;
    if (view_is_z_mode(view)) {
        const int t = threadIdx.y * MB_X + threadIdx.x;
        const int iv = rb.tile_v * 32 + t / MB_Y, iu = rb.tile_u * 32 + rb.sub * MB_Y + t % MB_Y;
        tile[t % MB_Y][t / MB_Y] = iu < W && iv < H ? load_as_float(img + (size_t)iv * W + iu) : 0.0f;
        __syncthreads();
        u = rb.tile_u * 32 + rb.sub * MB_Y + threadIdx.y;
        v = rb.tile_v * 32 + threadIdx.x;
        y = tile[threadIdx.y][threadIdx.x];
    } else {
        u = rb.tile_u * 32 + threadIdx.x;
        v = rb.tile_v * 32 + rb.sub * MB_Y + threadIdx.y;
        if (u < W && v < H) y = load_as_float(img + (size_t)v * W + u);
    }
    if (u >= W || v >= H || y == 0.0f || !in_footprint(view, u, v)) return;
    const float step = step_ptr[g];
    const ConeRay ray = cone_ray_setup(view, u, v, acc.X, acc.Y, acc.Z, 0.0, step, spacing_ptr[g * 3 + 2],
                                       spacing_ptr[g * 3 + 1], spacing_ptr[g * 3 + 0]);
    if (march_inside(ray, acc.X, acc.Y, acc.Z))
        scatter_ray<false>(ray, step, y, acc);
    else
        scatter_ray<true>(ray, step, y, acc);
}

// The volume from its cell accumulators: a 32 (x) x 32 (z) tile of one y per
// block, read along z and written along x.
__global__ void __launch_bounds__(256) gather_cells_kernel(const float4 *__restrict__ cells, float *__restrict__ vol,
                                                           int X, int Y, int Z)
{
    __shared__ float tile[32][33];
    const int x0 = blockIdx.x * 32, z0 = blockIdx.z * 32, y = blockIdx.y;
    const size_t s_y = Z + ACC_PLANES, s_x = s_y * (Y + 2);
    const int z = z0 + threadIdx.x;
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int x = x0 + k;
        if (x < X && z < Z) {
            const float4 *c = cells + (x + 1) * s_x + (y + 1) * s_y + (z + 1);
            tile[k][threadIdx.x] = (__ldg(c).x + __ldg(c - s_x).y) + (__ldg(c - s_y).z + __ldg(c - s_x - s_y).w);
        }
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int x = x0 + threadIdx.x, zz = z0 + k;
        if (x < X && zz < Z) vol[((size_t)zz * Y + y) * X + x] = tile[threadIdx.x][k];
    }
}

template <typename T>
cudaError_t scatter_cells(const void *sinogram, float *volume, const Dims3D &d, const ConeFpView *views,
                          const float *step, const float *spacing, void *cells, cudaStream_t stream)
{
    const CellAccumulators acc{(float4 *)cells, d.vol_x, d.vol_y, d.vol_z};
    const size_t voxels = (size_t)d.vol_z * d.vol_y * d.vol_x, pixels = (size_t)d.n_proj * d.det_h * d.det_w;
    const dim3 block(MB_X, MB_Y), ggrid((d.vol_x + 31) / 32, d.vol_y, (d.vol_z + 31) / 32);
    for (int b = 0; b < d.batch; ++b) {
        cudaError_t e = cudaMemsetAsync(cells, 0, cone_scatter_cells_bytes(d.vol_z, d.vol_y, d.vol_x), stream);
        if (e != cudaSuccess) return e;
        cone_scatter_cells_kernel<T><<<ray_block_count(d.det_w, d.det_h, d.n_proj), block, 0, stream>>>(
            (const T *)sinogram + b * pixels, acc, views, step, spacing, d.det_w, d.det_h, d.n_proj,
            d.geom_batch == 1 ? 0 : b);
        gather_cells_kernel<<<ggrid, dim3(32, 8), 0, stream>>>((const float4 *)cells, volume + b * voxels, d.vol_x,
                                                               d.vol_y, d.vol_z);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

bool cone_ray_grid_fits(int det_w, int det_h, int n_proj)
{
    return ray_blocks_fit(det_w, det_h, n_proj);
}

size_t cone_scatter_cells_bytes(int vol_z, int vol_y, int vol_x)
{
    // cells are indexed with 32-bit columns, y is a grid dimension
    if (vol_y > 65535 || (long long)(vol_x + 2) * (vol_y + 2) >= (1LL << 31)) return 0;
    return (size_t)(vol_x + 2) * (vol_y + 2) * (vol_z + ACC_PLANES) * sizeof(float4);
}

cudaError_t launch_cone_scatter_cells(const void *sinogram, float *volume, int in_dtype, const Dims3D &d,
                                      const ConeFpView *views, const float *step, const float *spacing, void *cells,
                                      cudaStream_t stream)
{
    return dispatch_dtypes(in_dtype, PYRONN_FLOAT32, [&](auto tin, auto) {
        return scatter_cells<typename decltype(tin)::type>(sinogram, volume, d, views, step, spacing, cells, stream);
    });
}

cudaError_t launch_cone_scatter(const void *sinogram, float *volume, int in_dtype, const Dims3D &d,
                                const ConeFpView *views, const float *step, const float *spacing,
                                cudaStream_t stream)
{
    cudaError_t e = cudaMemsetAsync(volume, 0, sizeof(float) * (size_t)d.batch * d.vol_z * d.vol_y * d.vol_x, stream);
    if (e != cudaSuccess) return e;
    const dim3 block(MB_X, MB_Y);
    const dim3 grid((d.det_w + MB_X - 1) / MB_X, (d.det_h + MB_Y - 1) / MB_Y, d.n_proj * d.batch);
    if (grid.z > 65535) return cudaErrorInvalidConfiguration;
    switch (in_dtype) {
    case PYRONN_FLOAT32:
        cone_scatter_kernel<float><<<grid, block, 0, stream>>>((const float *)sinogram, volume, views, step, spacing,
                                                               d.vol_x, d.vol_y, d.vol_z, d.det_w, d.det_h, d.n_proj,
                                                               d.geom_batch);
        break;
    case PYRONN_BFLOAT16:
        cone_scatter_kernel<__nv_bfloat16><<<grid, block, 0, stream>>>((const __nv_bfloat16 *)sinogram, volume, views,
                                                                       step, spacing, d.vol_x, d.vol_y, d.vol_z,
                                                                       d.det_w, d.det_h, d.n_proj, d.geom_batch);
        break;
    case PYRONN_FLOAT16:
        cone_scatter_kernel<__half><<<grid, block, 0, stream>>>((const __half *)sinogram, volume, views, step, spacing,
                                                                d.vol_x, d.vol_y, d.vol_z, d.det_w, d.det_h, d.n_proj,
                                                                d.geom_batch);
        break;
    default:
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace pyronn
