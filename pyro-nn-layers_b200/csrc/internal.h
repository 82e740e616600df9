// internal.h -- launcher interfaces between the C-ABI layer and the kernels.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/pyronn_b200.h"

namespace pyronn {

// Per-view cone forward geometry in voxel-index space, built in FP64 on the
// device from P = [M | p4]: inv_ar = diag(1/spacing) M^-1 (row major) and
// src = (C - origin) / spacing with C = -M^-1 p4 the camera centre.
struct ConeFpView {
    double inv_ar[9];
    double src[3];
    // detector footprint of the volume box [-0.5, N] per axis, in pixel
    // indices (u_min, u_max, v_min, v_max), widened by 2 pixels: a ray whose
    // pixel lies outside misses the box; unbounded (+-inf) when the box's
    // corners do not all lie on one side of the source
    float foot[4];
};

// Per-view cone backprojection matrix in voxel-index space:
// row r = (P[r,0] sx, P[r,1] sy, P[r,2] sz, P[r,:] . (ox, oy, oz, 1)).
struct ConeBpView {
    float4 row[3];
};

struct Dims2D {
    int batch, vol_y, vol_x, n_proj, det_w, geom_batch;
};

struct Geom2D {
    const float *volume_origin, *detector_origin, *volume_spacing, *detector_spacing;
    const float *rays, *sid, *sdd;  // sid/sdd null for parallel beam
};

struct Dims3D {
    int batch, vol_z, vol_y, vol_x, n_proj, det_h, det_w, geom_batch;
};

// geometry preparation (geometry.cu)
cudaError_t launch_cone_fp_prepare(const float *P, const float *spacing, const float *origin, int geom_batch,
                                   int n_proj, int vol_x, int vol_y, int vol_z, ConeFpView *out, cudaStream_t stream);
cudaError_t launch_cone_bp_prepare(const float *P, const float *spacing, const float *origin, int geom_batch,
                                   int n_proj, ConeBpView *out, cudaStream_t stream);

// 2D (proj2d.cu)
// workspace: room for the two cell copies (pyronn_projection2d_workspace_size), or null
cudaError_t launch_projection2d(const void *volume, void *sinogram, int in_dtype, int out_dtype, bool fan,
                                const Dims2D &d, const Geom2D &g, void *workspace, cudaStream_t stream);
cudaError_t launch_backprojection2d(const void *sinogram, void *volume, int in_dtype, int out_dtype, bool fan,
                                    const Dims2D &d, const Geom2D &g, cudaStream_t stream);

// cone (cone_fp.cu / cone_bp.cu); tex == 0 selects the software path;
// only_if: a device word, the launch does nothing where it is 0 (or null)
cudaError_t launch_cone_fp(const void *volume, void *sinogram, int in_dtype, int out_dtype, const Dims3D &d,
                           int batch_index, const ConeFpView *views, const float *step, const float *spacing,
                           cudaTextureObject_t tex, cudaStream_t stream);
cudaError_t launch_cone_bp(const void *sinogram, void *volume, int in_dtype, int out_dtype, const Dims3D &d,
                           int batch_index, const ConeBpView *views, const float *mult, cudaTextureObject_t tex,
                           cudaStream_t stream, const unsigned *only_if = nullptr);

// software forward projector over padded, view-oriented copies (cone_fp_padded.cu)
size_t cone_fp_padded_scratch_bytes(int vol_z, int vol_y, int vol_x, int in_dtype);
// the same with a second batch element's copies
size_t cone_fp_padded_pair_bytes(int vol_z, int vol_y, int vol_x, int in_dtype);
bool cone_fp_padded_supported(const Dims3D &d, int in_dtype);
// flags: zeroed header words of the workspace (the kernel records which copies it needs)
// pairs: scratch is of cone_fp_padded_pair_bytes, and elements of shared
// geometry go two at a time
cudaError_t launch_cone_fp_padded(const void *volume, void *sinogram, int in_dtype, int out_dtype, const Dims3D &d,
                                  const ConeFpView *views, const float *step, const float *spacing, void *scratch,
                                  bool pairs, unsigned *flags, cudaStream_t stream);

// matched (exact-adjoint) scatter backprojector (cone_matched.cu); FP32 output
// FDK weighting + ramp filtering of `rows` detector rows (fdk.cu)
cudaError_t launch_fdk_filter(const void *in, void *out, int in_dtype, int out_dtype, long long rows, int det_h,
                              int W, float sdd, float dv, float du, float cv, float cu, int kind, int weight_output,
                              cudaStream_t stream);
// the same by fast Fourier transforms (fdk_fft.cu): rows of at most 2048 pixels
bool fdk_fft_supported(int W);
cudaError_t launch_fdk_filter_fft(const void *in, void *out, int in_dtype, int out_dtype, long long rows, int det_h,
                                  int W, float sdd, float dv, float du, float cv, float cu, int kind,
                                  int weight_output, cudaStream_t stream);

// whether the ray block order's grid (cone_ray.cuh) fits one launch
bool cone_ray_grid_fits(int det_w, int det_h, int n_proj);
// the same over cell accumulators (`cells`: device, cone_scatter_cells_bytes,
// 16-byte aligned; 0 bytes where they do not apply)
size_t cone_scatter_cells_bytes(int vol_z, int vol_y, int vol_x);
cudaError_t launch_cone_scatter_cells(const void *sinogram, float *volume, int in_dtype, const Dims3D &d,
                                      const ConeFpView *views, const float *step, const float *spacing, void *cells,
                                      cudaStream_t stream);
cudaError_t launch_cone_scatter(const void *sinogram, float *volume, int in_dtype, const Dims3D &d,
                                const ConeFpView *views, const float *step, const float *spacing,
                                cudaStream_t stream);

// TMA-staged software backprojector (cone_bp_tma.cu); err = device error flag
// (copy: a copy of cone_bp_tma_copy_bytes will be given)
bool cone_bp_tma_supported(const void *sinogram, int in_dtype, const Dims3D &d, bool copy);
// whether the sinogram's own rows can be staged
bool cone_bp_tma_aligned(const void *sinogram, int in_dtype, const Dims3D &d);
// Bytes of the copy of the sinogram the TMA backprojector stages its boxes
// from: 32-bit tap pairs of a 16-bit sinogram where that pays (one shared-memory
// load per lerp), rows at a 16-byte pitch where the sinogram's are none; else 0.
size_t cone_bp_tma_copy_bytes(int in_dtype, const Dims3D &d);
// `copy` (device, 16-byte aligned, cone_bp_tma_copy_bytes) or null.  `direct`, with
// a copy: a device word that is set, and nothing else written, where launch_cone_bp
// should do the work (given the same word, it works only then); or null.
cudaError_t launch_cone_bp_tma(const void *sinogram, void *volume, int in_dtype, int out_dtype, const Dims3D &d,
                               const ConeBpView *views, const float *mult, unsigned *err, void *copy,
                               unsigned *direct, cudaStream_t stream);
// testing hook (pyronn_debug_starve_tma_wait): while enabled, the last pass of
// every TMA backprojector block issues no copies and expects bytes that never
// arrive, so its bounded wait runs out and the block reports the timeout
void cone_bp_tma_starve_last_pass(int enable);

// texture-array cache (texcache.cu)
struct CachedArray;
enum ArrayKind { ARRAY_VOLUME_3D = 0, ARRAY_SINOGRAM_LAYERED = 1 };
// Returns an array of the given kind/extent whose previous users are done
// (or were on the same stream).  half_texels selects an FP16 texel format.
cudaError_t array_acquire(int kind, int w, int h, int d, bool half_texels, cudaStream_t stream, CachedArray **out);
cudaTextureObject_t array_texture(CachedArray *a);
// Copies one batch element (w*h*d elements of dtype) into the array on stream.
cudaError_t array_fill(CachedArray *a, const void *src, int dtype, cudaStream_t stream);
// Marks the array as in use by work already enqueued on stream.
cudaError_t array_release(CachedArray *a, cudaStream_t stream);
int array_cache_clear();

size_t dtype_size(int dtype);

// record a failure as the calling thread's last error (capi.cu); return status
int report_error(int status, const char *fmt, ...) __attribute__((format(printf, 2, 3)));
int report_cuda_error(cudaError_t e, const char *what);

}  // namespace pyronn
