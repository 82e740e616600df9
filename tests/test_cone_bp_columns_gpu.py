"""GPU tests of the cone backprojector's column loop."""
import numpy as np
import pytest
import torch

import pyronn_layers as pl

DVS = [0.9899, 0.7003, 0.6501, 0.3301]


def _bound(v):
    """Half an ulp of the position in the box (a row above v) and of the value."""
    return 0.5 * np.spacing((v + 1.0).astype(np.float32)) + 0.5 * np.spacing(v.astype(np.float32))


def _chain(dv, base, depth):
    """Positions of every second voxel by running FP32 sums of 2 dv."""
    out, l = [], np.float32(base)
    for _ in range(0, depth, 2):
        out.append(l)
        l = np.float32(l + np.float32(2) * dv)
    return np.array(out, np.float64)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,depth", [(torch.float32, 16), (torch.float16, 32), (torch.bfloat16, 32)])
@pytest.mark.parametrize("dv", DVS)
def test_column_positions_do_not_drift(cuda, dtype, depth, dv):
    """One view whose detector row is v = 0.5 + dv z, over a sinogram of the row
    numbers: a voxel's value is its position.  Rounded are the position from
    the column base (one FMA; the base itself is exact) and the v lerp, half
    an ulp each."""
    dv = np.float32(dv)
    y, x, h, w = 144, 32, 38, 38
    vol, batch = (depth, y, x), (64 if depth == 32 else 1)  # 16-bit: enough voxels and tiles for columns of 32
    assert depth == 16 or depth * y * x >= 100 * h * w
    P = np.array([[[1.0, 0, 0, 2.0], [0, 0, dv, 0.5], [0, 0, 0, 1.0]]], np.float32)
    rows = np.broadcast_to(np.arange(h, dtype=np.float32)[:, None], (batch, 1, h, w))
    p = torch.as_tensor(rows.copy()).to(device=cuda, dtype=dtype)
    out = pl.cone_backprojection3d(p, vol, np.zeros(3), np.ones(3), P, 1.0, 1.0, out_dtype=torch.float32)
    v = 0.5 + np.arange(depth) * float(dv)
    bound = _bound(v)
    got = out.double().cpu().numpy()
    assert (np.abs(got - v[None, :, None, None]) <= bound[None, :, None, None]).all()


@pytest.mark.parametrize("depth", [16, 32])
def test_drift_bound_tells_running_sums(depth):
    """Running sums would miss the bound above at the positions it is asked of."""
    worst = 0.0
    for dv in DVS:
        v = 0.5 + np.arange(0, depth, 2) * float(np.float32(dv))
        worst = max(worst, float((np.abs(_chain(np.float32(dv), 1.5, depth) - (v + 1.0)) / _bound(v)).max()))
    assert worst > 1.5
