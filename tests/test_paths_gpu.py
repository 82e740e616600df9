"""GPU parity of the kernels' size- and geometry-dependent paths against the
FP64 oracle, at the sizes where each path begins, ends or wraps.

Tolerances (relative L2) are those of test_ops_gpu.py: FP32 arithmetic on the
same (storage-rounded) input, 2e-5 for ray marches, 1e-5 for backprojections.
"""
import numpy as np
import pytest
import torch

import oracle
import pyronn_layers as pl
from pyronn_layers import _capi, fbp, geometry, phantoms
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def t(a, dev, dtype=torch.float32):
    return torch.as_tensor(np.asarray(a)).to(device=dev, dtype=dtype)


def noise(seed, shape):
    return np.random.Generator(np.random.PCG64(seed)).uniform(0.2, 1.0, shape).astype(np.float32)


# ------------------------------------------------------------- 2D forward


@pytest.mark.parametrize("fan", [False, True])
@pytest.mark.parametrize("batch,views,width", [
    (1, 9, 40),      # ray segments (one band of columns per thread)
    (1, 97, 3100),   # one thread per ray, one slice (above the segments' limit)
    (2, 97, 780),    # two slices per thread
    (3, 83, 610),    # three slices per thread
    (4, 83, 460),    # four slices per thread
    (5, 61, 500),    # three per thread, the last group overlapping
    (7, 61, 400),    # four per thread, the last group overlapping
])
def test_2d_forward_walks(cuda, batch, views, width, fan):
    """Every walk of the 2D forward (segments; one to four slices per thread) against the oracle, and without the workspace the same bits."""
    shape, sp, ds = (23, 37), (0.8, 1.0), 60.0 / width
    if fan:
        geo = geometry.FanBeam2D(shape, sp, width, ds, views, 60.0, 90.0)
        fwd, ofwd, name = pl.fan_projection2d, oracle.fan_projection2d, "pyronn_fan_projection2d"
    else:
        geo = geometry.ParallelBeam2D(shape, sp, width, ds, views)
        fwd, ofwd, name = pl.parallel_projection2d, oracle.parallel_projection2d, "pyronn_parallel_projection2d"
    img = noise(batch, (batch,) + shape)
    out = fwd(t(img, cuda), geo.detector_shape, *geo.args())
    ref = ofwd(img, geo.detector_shape, *geo.args())
    assert rel_l2(out.cpu().numpy(), ref) < 2e-5
    gp = pl.ops.Geometry2D(batch, cuda, *geo.args()[:4], geo.args()[-1], views, *(geo.args()[4:6] if fan else ()))
    plain = torch.empty_like(out)
    x = t(img, cuda)
    _capi.call(name, x.data_ptr(), plain.data_ptr(), 0, 0, batch, *shape, views, width, *gp.pointers(), gp.g, 0, 0,
               torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(plain, out)


@pytest.mark.parametrize("spacing", [(1.0, 1.0), (0.8, 1.3), (0.05, 0.05), (5.0 * 2.0 ** -3 * (1 + 2.0 ** -12),) * 2])
@pytest.mark.parametrize("length", [1.0, 0.37, 40.0])
def test_2d_forward_alpha_sequences(cuda, spacing, length):
    """Ray vectors of any length (steps of a fraction of a cell up to several
    cells), steps whose float sums are ties, and rays whose alphas cross
    binades: the samples sit where the one-at-a-time float march puts them."""
    shape, views, width = (33, 29), 24, 51
    geo = geometry.ParallelBeam2D(shape, spacing, width, 40.0 * max(spacing) / width, views)
    args = geo.args()[:4] + (geo.ray_vectors * np.float32(length),)
    img = noise(5, (1,) + shape)
    out = pl.parallel_projection2d(t(img, cuda), (views, width), *args)
    ref = oracle.parallel_projection2d(img, (views, width), *args)
    assert rel_l2(out.cpu().numpy(), ref) < 2e-5


def test_2d_forward_source_inside(cuda):
    """A fan source inside the slice: the march starts at negative alphas."""
    geo = geometry.FanBeam2D((40, 40), (1.0, 1.0), 64, 1.0, 16, 9.0, 40.0)
    img = noise(6, (2, 40, 40))
    out = pl.fan_projection2d(t(img, cuda), geo.detector_shape, *geo.args())
    ref = oracle.fan_projection2d(img, geo.detector_shape, *geo.args())
    assert rel_l2(out.cpu().numpy(), ref) < 2e-5


# ---------------------------------------------------------- 2D backprojection


@pytest.mark.parametrize("fan", [False, True])
@pytest.mark.parametrize("batch,shape,views,width,dtype", [
    (1, (33, 65), 70, 90, torch.float32),       # one slice, view groups
    (2, (31, 33), 257, 60, torch.bfloat16),     # two slices per thread; two view chunks
    (3, (40, 37), 33, 91, torch.float32),       # three per thread
    (5, (40, 37), 33, 30, torch.float16),       # three per thread, overlapping; pixels off the detector
    (7, (40, 37), 33, 91, torch.bfloat16),      # four per thread, overlapping
])
def test_2d_backprojection_walks(cuda, batch, shape, views, width, dtype, fan):
    """The splits of the 2D backprojection (view groups; one to four slices per
    thread; blocks wholly inside the detector rows and blocks that
    need tap flags) against the oracle."""
    if fan:
        geo = geometry.FanBeam2D(shape, (0.8, 1.0), width, 1.1, views, 900.0, 1300.0)
        bwd, obwd = pl.fan_backprojection2d, oracle.fan_backprojection2d
    else:
        geo = geometry.ParallelBeam2D(shape, (0.8, 1.0), width, 0.9, views)
        bwd, obwd = pl.parallel_backprojection2d, oracle.parallel_backprojection2d
    p = t(noise(batch, (batch,) + geo.detector_shape), cuda, dtype)
    out = bwd(p, geo.volume_shape, *geo.args(), out_dtype=torch.float32)
    ref = obwd(p.float().cpu().numpy(), geo.volume_shape, *geo.args())
    assert rel_l2(out.cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("fan", [False, True])
@pytest.mark.parametrize("batch,shape,dtype", [(7, (900, 800), torch.float32), (9, (960, 940), torch.float16)])
def test_2d_backprojection_shared_slices(cuda, batch, shape, dtype, fan):
    """Launches without view groups: four and eight slices per thread (the last
    group overlapping) give each slice the bits of a call of its own."""
    if fan:
        geo = geometry.FanBeam2D(shape, (0.8, 1.0), 2000, 1.1, 3, 900.0, 1300.0)
        bwd = pl.fan_backprojection2d
    else:
        geo = geometry.ParallelBeam2D(shape, (0.8, 1.0), 2000, 0.9, 3)
        bwd = pl.parallel_backprojection2d
    p = t(noise(batch, (batch,) + geo.detector_shape), cuda, dtype)
    out = bwd(p, geo.volume_shape, *geo.args(), out_dtype=torch.float32)
    for b in range(batch):
        one = bwd(p[b:b + 1], geo.volume_shape, *geo.args(), out_dtype=torch.float32)
        assert torch.equal(one[0], out[b])


# -------------------------------------------------------------- cone forward


def test_cone_forward_fp32_cell_pitch(cuda):
    """A volume (60 x 8 x 60, z y x) whose FP32 cell copy (three z entries
    beyond the volume) needs a padded x pitch for its biased index not to
    wrap, with rays through its upper z face."""
    geo = geometry.ConeBeam3D((60, 8, 60), (1.0, 1.0, 1.0), (64, 40), (2.5, 2.0), 6, 90.0, 170.0, step_size=0.5)
    vol = noise(12, (2,) + geo.volume_shape)
    out = pl.cone_projection3d(t(vol, cuda), geo.detector_shape, *geo.args())
    ref = oracle.cone_projection3d(vol, geo.detector_shape, *geo.args())
    assert rel_l2(out.cpu().numpy(), ref) < 2e-5


# ------------------------------------------------- matched cone backprojection


def _tilted(geo, angle):
    """The scan's projection matrices with the object turned about the y axis."""
    c, s = np.cos(angle), np.sin(angle)
    r = np.array([[c, 0, s, 0], [0, 1, 0, 0], [-s, 0, c, 0], [0, 0, 0, 1]])
    return (geo.projection_matrices.astype(np.float64) @ r).astype(np.float32)


@pytest.mark.parametrize("vol_shape,det,batch,tilt,dtype", [
    ((1, 1, 1), (3, 3), 1, 0.0, torch.float32),
    ((5, 33, 31), (9, 40), 2, 0.0, torch.bfloat16),
    ((34, 20, 23), (40, 33), 3, 0.0, torch.float32),
    ((20, 21, 22), (33, 31), 1, 0.5 * np.pi, torch.float32),  # detector rows along z: warps along u
    ((20, 21, 22), (33, 31), 1, 0.4, torch.float16),
])
def test_matched_backprojection_cells(cuda, vol_shape, det, batch, tilt, dtype):
    """The matched backprojection over cell accumulators, and with a workspace
    of the per-view part alone (scattered into the volume), against the FP64
    oracle: FP32 sums of FP32 weights, 1e-5 (as the backprojections)."""
    geo = geometry.ConeBeam3D(vol_shape, (1.0, 0.9, 1.1), det, (1.3, 1.2), 7, 60.0, 100.0, step_size=0.5)
    args = (geo.volume_origin, geo.volume_spacing, _tilted(geo, tilt), geo.step_size)
    p = t(noise(21, (batch,) + geo.detector_shape), cuda, dtype)
    ref = oracle.cone_backprojection3d_matched(p.float().cpu().numpy(), vol_shape, *args)
    out = pl.cone_backprojection3d_matched(p, vol_shape, *args)
    assert rel_l2(out.cpu().numpy(), ref) < 1e-5
    g = pl.ops.GeometryCone(batch, cuda, *args, 1.0, geo.detector_shape[0])
    n = _capi.workspace_size("pyronn_cone_backprojection3d_matched", g.g, geo.detector_shape[0])
    ws = torch.empty(n, dtype=torch.uint8, device=cuda)
    plain = torch.full_like(out, 7.0)
    _capi.call("pyronn_cone_backprojection3d_matched", p.data_ptr(), plain.data_ptr(), pl.ops.storage_code(dtype),
               batch, *geo.detector_shape, *vol_shape, g.volume_origin.data_ptr(), g.volume_spacing.data_ptr(),
               g.projection_matrices.data_ptr(), g.step_size.data_ptr(), g.g, ws.data_ptr(), n,
               torch.cuda.current_stream().cuda_stream)
    assert rel_l2(plain.cpu().numpy(), ref) < 1e-5


# -------------------------------------------------------- cone backprojection


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("vol_shape,det,pitch,batch", [
    ((9, 10, 33), (7, 1), 3.0, 1),      # one-pixel rows
    ((17, 21, 40), (31, 37), 1.6, 2),   # rows of no multiple of 16 bytes, batch of two
    ((33, 40, 45), (29, 129), 0.7, 1),  # a row one element past a multiple of 16 bytes
    ((48, 50, 52), (23, 29), 3.1, 1),   # the same with more than 100 voxels per pixel (16-bit: paired copy)
])
def test_cone_backprojection_unaligned_rows(cuda, vol_shape, det, pitch, batch, dtype):
    """Detector rows TMA cannot address: over a pitched (or paired) copy given
    the queried workspace, by direct gathers given the views' part alone; both
    against the oracle.  The second sinogram starts off a 16-byte boundary."""
    geo = geometry.ConeBeam3D(vol_shape, (1.0, 0.9, 1.1), det, (pitch, pitch), 9, 160.0, 260.0)
    sino = t(noise(31, (batch,) + geo.detector_shape), cuda, dtype)
    shifted = torch.empty(sino.numel() + 1, device=cuda, dtype=dtype)[1:].view(sino.shape)
    shifted.copy_(sino)
    ref = oracle.cone_backprojection3d(sino.float().cpu().numpy(), vol_shape, *geo.args())
    gc = pl.ops.GeometryCone(batch, cuda, *geo.args(), geo.detector_shape[0])
    code = pl.ops.storage_code(dtype)
    query = ("pyronn_cone_backprojection3d", batch, *geo.detector_shape, *vol_shape, code, 0, gc.g)
    full, views = _capi.workspace_size(*query), _capi.workspace_size(query[0], 0, *query[2:])
    assert full > views
    for p in (sino, shifted):
        for nbytes in (full, views):
            ws = torch.empty(nbytes, dtype=torch.uint8, device=cuda)
            out = torch.full((batch,) + vol_shape, 7.0, device=cuda)
            _capi.call(query[0], p.data_ptr(), out.data_ptr(), code, 0, 0, batch, *geo.detector_shape, *vol_shape,
                       *gc.pointers(), gc.g, ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream)
            assert rel_l2(out.cpu().numpy(), ref) < 1e-5


# ------------------------------------------------------------------ ramp filter


@pytest.mark.parametrize("filt", ["ram-lak", "shepp-logan"])
@pytest.mark.parametrize("rows,width", [
    ((1, 1, 1), 1), ((1, 3, 5), 2),          # tiny rows; an odd number of rows
    ((2, 9, 1), 255), ((1, 3, 40), 256),     # transforms of 512 points, the widest exactly half
    ((1, 5, 13), 257), ((1, 2, 7), 512),     # 1024 points
    ((1, 1, 11), 513), ((1, 2, 3), 1024),    # 2048 points
    ((1, 1, 3), 1025), ((1, 1, 3), 2047), ((1, 1, 2), 2048),  # 4096 points
    ((1, 1, 3), 2049),                       # direct sums
])
def test_filter_widths(cuda, rows, width, filt):
    """The ramp filter at the edges of its transform lengths against the FP64
    oracle: 1e-5, as test_fbp_gpu.py; rows of very different magnitude are
    each held to it."""
    b, n, h = rows
    p = noise(width, rows + (width,))
    p[:, :, ::2] *= np.float32(1e-6)
    out = fbp.fdk_filter(t(p, cuda), 800.0, (1.1, 0.7), None, filt).cpu().numpy()
    kind = oracle.filters.RAM_LAK if filt == "ram-lak" else oracle.filters.SHEPP_LOGAN
    ref = oracle.fdk_filter(p, 800.0, 1.1, 0.7, (h - 1) / 2, (width - 1) / 2, kind)
    for i in np.ndindex(*rows):
        assert rel_l2(out[i], ref[i]) < 1e-5


def test_filter_keeps_rows_apart(cuda):
    """Infinities and NaNs in a row make that row NaN and leave the others as
    they are; a row of zeros stays zeros."""
    p = noise(3, (1, 1, 8, 300))
    clean = fbp.fdk_filter(t(p, cuda), 500.0, (1.0, 1.0))
    q = p.copy()
    q[0, 0, 1, 17], q[0, 0, 4, 299], q[0, 0, 6] = np.inf, np.nan, 0.0
    out = fbp.fdk_filter(t(q, cuda), 500.0, (1.0, 1.0))
    for r in (0, 2, 3, 5, 7):
        assert torch.equal(out[0, 0, r], clean[0, 0, r]) or rel_l2(out[0, 0, r].cpu().numpy(),
                                                                   clean[0, 0, r].cpu().numpy()) < 1e-6
    assert torch.isnan(out[0, 0, 1]).all() and torch.isnan(out[0, 0, 4]).all()
    assert (out[0, 0, 6] == 0).all()


# ---------------------------------------------------- cone forward, batches


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,tilt", [(2, 0.0), (3, 0.0), (2, 0.5 * np.pi), (3, 0.4)])
def test_cone_forward_pairs_are_bit_exact(cuda, batch, tilt, dtype):
    """Two elements per launch (given the batched workspace) take the same
    samples in the same order as one at a time: the same bits, in every view
    mode, for an odd element left over, and for rays on the clamped path."""
    geo = geometry.ConeBeam3D((21, 26, 30), (1.0, 0.9, 1.1), (33, 41), (1.2, 1.3), 9, 60.0, 110.0, step_size=0.5)
    args = (geo.volume_origin, geo.volume_spacing, _tilted(geo, tilt), geo.step_size, 1.0)
    x = t(noise(41, (batch,) + geo.volume_shape), cuda, dtype)
    g = pl.ops.GeometryCone(batch, cuda, *args, geo.detector_shape[0])
    code = pl.ops.storage_code(dtype)
    name, dims = "pyronn_cone_projection3d", (batch, *geo.volume_shape, *geo.detector_shape)
    outs = []
    for query in (name, name + "_batched"):
        n = _capi.workspace_size(query, *dims, code, 0, g.g)
        ws = torch.empty(n, dtype=torch.uint8, device=cuda)
        out = torch.full((batch,) + geo.detector_shape, 7.0, device=cuda)
        _capi.call(name, x.data_ptr(), out.data_ptr(), code, 0, 0, *dims, *g.pointers(), g.g, ws.data_ptr(), n,
                   torch.cuda.current_stream().cuda_stream)
        outs.append((n, out))
    assert outs[1][0] > outs[0][0]
    assert torch.equal(outs[0][1], outs[1][1]) and bool((outs[1][1] != 0).any())


def test_cone_forward_pair_of_wide_range(cuda):
    """FP16 values beyond the packed lerps' range in the second element of a
    pair: both take the FP32 lerps (test_cone_projection_wide_fp16_range's
    tolerance)."""
    geo = geometry.ConeBeam3D((21, 26, 30), (1.0, 0.9, 1.1), (33, 41), (1.2, 1.3), 5, 60.0, 110.0, step_size=0.5)
    vol = np.stack([phantoms.ellipsoid_phantom_3d(geo.volume_shape, geo.volume_spacing, seed=s, n=6)[0] for s in (1, 2)])
    vol[1] *= 60000.0 / vol[1].max()
    x = t(vol, cuda, torch.float16)
    out = pl.cone_projection3d(x, geo.detector_shape, *geo.args(), out_dtype=torch.float32)
    ref = oracle.cone_projection3d(x.float().cpu().numpy(), geo.detector_shape, *geo.args())
    for b in range(2):
        assert rel_l2(out[b].cpu().numpy(), ref[b]) < 2e-5


# ------------------------------------------------------ texture interpolation


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("width", [20, 21, 22])
def test_texture_fill_widths(cuda, width, dtype):
    """Texture arrays filled four texels per thread (widths of a multiple of
    four, aligned input) and one at a time hold the same texels: both ops of
    a batch whose second element starts off the four-texel alignment equal a
    call per element."""
    geo = geometry.ConeBeam3D((5, 7, width), (1.0, 0.9, 1.1), (9, width), (1.2, 1.3), 3, 60.0, 100.0, step_size=0.5)
    for op, shape, out_shape in ((pl.cone_projection3d, geo.volume_shape, geo.detector_shape),
                                 (pl.cone_backprojection3d, geo.detector_shape, geo.volume_shape)):
        n = int(np.prod(shape))
        store = t(noise(51, (2 * n + 1,)), cuda, dtype)
        aligned, shifted = store[:2 * n].view((2,) + shape), store[1:].view((2,) + shape)
        for x in (aligned, shifted):
            both = op(x, out_shape, *geo.args(), hardware_interp=True)
            for b in range(2):
                one = op(x[b:b + 1].clone(), out_shape, *geo.args(), hardware_interp=True)
                assert torch.equal(one[0], both[b])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("vol_shape", [(33, 40, 64), (31, 41, 65), (70, 24, 40)])
def test_cone_backprojection_tall_columns(cuda, vol_shape, dtype):
    """16-bit sinograms of many voxels per detector pixel take columns of 32
    voxels, with the paired copy and without it: the same bits, for depths on
    either side of a tile, and the oracle's values."""
    geo = geometry.ConeBeam3D(vol_shape, (1.0, 1.0, 1.0), (20, 32), (4.0, 4.0), 9, 160.0, 260.0)
    assert np.prod(vol_shape) >= 100 * 20 * 32
    sino = t(noise(61, (1,) + geo.detector_shape), cuda, dtype)
    gc = pl.ops.GeometryCone(1, cuda, *geo.args(), geo.detector_shape[0])
    code = pl.ops.storage_code(dtype)
    outs = []
    for batch in (1, 0):  # with the paired copy, and the views' part alone
        n = _capi.workspace_size("pyronn_cone_backprojection3d", batch, *geo.detector_shape, *vol_shape, code, 0, 1)
        ws = torch.empty(n, dtype=torch.uint8, device=cuda)
        out = torch.full((1,) + vol_shape, 7.0, device=cuda)
        _capi.call("pyronn_cone_backprojection3d", sino.data_ptr(), out.data_ptr(), code, 0, 0, 1,
                   *geo.detector_shape, *vol_shape, *gc.pointers(), 1, ws.data_ptr(), n,
                   torch.cuda.current_stream().cuda_stream)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    ref = oracle.cone_backprojection3d(sino.float().cpu().numpy(), vol_shape, *geo.args())
    assert rel_l2(outs[0].cpu().numpy(), ref) < 1e-5
