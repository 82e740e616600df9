"""Tests of the cone backprojector's column loop and of its choice of kernel."""
import numpy as np
import pytest
import torch

import oracle
import pyronn_layers as pl
from pyronn_layers import _capi, geometry
from conftest import rel_l2

DVS = [0.9899, 0.7003, 0.6501, 0.3301]


def _bound(v):
    """Half an ulp of the position in the box (a row above v) and of the value."""
    return 0.5 * sum(np.spacing(x.astype(np.float32)).astype(np.float64) for x in (v + 1.0, v))


def _chain(dv, base, depth):
    """Positions of every second voxel by running FP32 sums of 2 dv."""
    out, l = [], np.float32(base)
    for _ in range(0, depth, 2):
        out.append(l)
        l = np.float32(l + np.float32(2) * dv)
    return np.array(out, np.float64)


def _one_view(rows, dv, depth, cuda, dtype):
    """The backprojection of one view whose detector row is v = 0.5 + dv z, every
    detector row holding one value: FP64 [batch, depth, y, x]."""
    y, x, w = 144, 32, 38
    h = len(rows)
    batch = 128 if depth == 32 else 1  # 16-bit: enough voxels and tiles for columns of 32
    assert depth == 16 or depth * y * x >= 100 * h * w
    P = np.array([[[1.0, 0, 0, 2.0], [0, 0, dv, 0.5], [0, 0, 0, 1.0]]], np.float32)
    p = torch.as_tensor(np.broadcast_to(rows[:, None], (batch, 1, h, w)).copy()).to(device=cuda, dtype=dtype)
    out = pl.cone_backprojection3d(p, (depth, y, x), np.zeros(3), np.ones(3), P, 1.0, 1.0, out_dtype=torch.float32)
    return out.double().cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,depth", [(torch.float32, 16), (torch.float16, 32), (torch.bfloat16, 32)])
@pytest.mark.parametrize("dv", DVS)
def test_column_positions_do_not_drift(cuda, dtype, depth, dv):
    """A sinogram of the row numbers: a voxel's value is its position.  Rounded
    are the position from the column base (one FMA; the base itself is exact)
    and the v lerp, half an ulp each."""
    got = _one_view(np.arange(38, dtype=np.float32), dv, depth, cuda, dtype)
    v = 0.5 + np.arange(depth) * float(np.float32(dv))
    assert (np.abs(got - v[None, :, None, None]) <= _bound(v)[None, :, None, None]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,depth", [(torch.float32, 16), (torch.bfloat16, 32)])
def test_column_lerp_of_rows_far_apart(cuda, dtype, depth):
    """Rows whose difference overflows: the v lerp is a (1 - t) + t b, finite
    for finite taps (two roundings, after the position's)."""
    dv, a = 0.6501, float(np.float32(2.5e38) if dtype == torch.float32 else torch.tensor(2.5e38, dtype=dtype))
    got = _one_view(np.where(np.arange(38) % 2, -a, a).astype(np.float32), dv, depth, cuda, dtype)
    v = 0.5 + np.arange(depth) * float(np.float32(dv))
    t, low = v - np.floor(v), np.where(np.floor(v) % 2, -a, a)
    bound = 2 * a * _bound(v) + 1.5 * 2.0 ** 104  # (an ulp of a)
    assert (np.abs(got - (low * (1 - 2 * t))[None, :, None, None]) <= bound[None, :, None, None]).all()


@pytest.mark.parametrize("depth", [16, 32])
def test_drift_bound_tells_running_sums(depth):
    """Running sums would miss the bound above at the positions it is asked of."""
    worst = 0.0
    for dv in DVS:
        v = 0.5 + np.arange(0, depth, 2) * float(np.float32(dv))
        worst = max(worst, float((np.abs(_chain(np.float32(dv), 1.5, depth) - (v + 1.0)) / _bound(v)).max()))
    assert worst > 1.5


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("vol_shape,batch", [
    ((64, 16, 48), 256),  # 2048 tiles of 32 voxels: tall columns
    ((49, 16, 64), 256),  # the same, the last tile in part empty
    ((64, 16, 48), 255),  # 2040: columns of 16
    ((65, 16, 47), 256),  # an odd number of 16-voxel tiles along z: columns of 16
])
def test_column_heights(cuda, vol_shape, batch, dtype):
    """Either column height with the paired copy and without it: the same bits,
    and the oracle's values to FP32 rounding (1e-5, as the other paths)."""
    geo = geometry.ConeBeam3D(vol_shape, (1.0, 1.0, 1.0), (20, 24), (5.0, 4.2), 5, 160.0, 260.0)
    assert np.prod(vol_shape) >= 100 * 20 * 24
    rng = np.random.Generator(np.random.PCG64(71))
    three = rng.uniform(0.2, 1.0, (3,) + geo.detector_shape).astype(np.float32)
    which = np.arange(batch) * 3 // batch
    sino = torch.as_tensor(three[which]).to(device=cuda, dtype=dtype)
    gc = pl.ops.GeometryCone(batch, cuda, *geo.args(), geo.detector_shape[0])
    code = pl.ops.storage_code(dtype)
    outs = []
    for b in (batch, 0):  # with the paired copy, and the views' part alone
        n = _capi.workspace_size("pyronn_cone_backprojection3d", b, *geo.detector_shape, *vol_shape, code, 0, 1)
        ws = torch.empty(n, dtype=torch.uint8, device=cuda)
        out = torch.full((batch,) + vol_shape, 7.0, device=cuda)
        _capi.call("pyronn_cone_backprojection3d", sino.data_ptr(), out.data_ptr(), code, 0, 0, batch,
                   *geo.detector_shape, *vol_shape, *gc.pointers(), 1, ws.data_ptr(), n,
                   torch.cuda.current_stream().cuda_stream)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    first = [int(np.argmax(which == k)) for k in range(3)]
    ref = oracle.cone_backprojection3d(sino[first].float().cpu().numpy(), vol_shape, *geo.args())
    assert rel_l2(outs[0][first].cpu().numpy(), ref) < 1e-5
    for b in range(batch):
        assert torch.equal(outs[0][b], outs[0][first[which[b]]])


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("vol_shape,det,pitch,batch,fits", [
    ((40, 44, 48), (61, 67), 1.3, 1, True),     # about one row per voxel
    ((40, 44, 48), (301, 331), 0.26, 1, False),  # six: the boxes overflow
    ((17, 9, 33), (151, 133), 0.4, 3, False),
    ((1, 1, 1), (5, 3), 1.0, 2, False),  # the tile reaches past the detector
])
def test_rows_off_16_bytes(cuda, vol_shape, det, pitch, batch, fits, dtype):
    """Rows TMA cannot address, given the copy's workspace: staged from it where
    the boxes fit, else the direct kernel's bits; the oracle's values either
    way, nothing written past the workspace."""
    geo = geometry.ConeBeam3D(vol_shape, (1.0, 1.0, 1.0), det, (pitch, pitch), 9, 160.0, 260.0)
    rng = np.random.Generator(np.random.PCG64(72))
    sino = torch.as_tensor(rng.uniform(0.2, 1.0, (batch,) + geo.detector_shape)).to(device=cuda, dtype=dtype)
    gc = pl.ops.GeometryCone(batch, cuda, *geo.args(), geo.detector_shape[0])
    code = pl.ops.storage_code(dtype)
    outs = []
    for b in (batch, 0):
        n = _capi.workspace_size("pyronn_cone_backprojection3d", b, *geo.detector_shape, *vol_shape, code, 0, 1)
        ws = torch.full((n + 256,), 0xA5, dtype=torch.uint8, device=cuda)
        out = torch.full((batch,) + vol_shape, 7.0, device=cuda)
        _capi.call("pyronn_cone_backprojection3d", sino.data_ptr(), out.data_ptr(), code, 0, 0, batch,
                   *geo.detector_shape, *vol_shape, *gc.pointers(), 1, ws.data_ptr(), n,
                   torch.cuda.current_stream().cuda_stream)
        assert bool((ws[n:] == 0xA5).all())
        outs.append((out, ws[16:20].view(torch.int32).item()))
    assert outs[0][1] == (0 if fits else 1) and outs[1][1] == 0
    if not fits:
        assert torch.equal(outs[0][0], outs[1][0])
    ref = oracle.cone_backprojection3d(sino.float().cpu().numpy(), vol_shape, *geo.args())
    for out, _ in outs:
        assert rel_l2(out.cpu().numpy(), ref) < 1e-5
