"""GPU tests of the 2D backprojection's splits around the sizes where they
change: slices per thread, view groups and per-element geometry, against the
FP64 oracle (FP32 sums of FP32 weights, 1e-5) and bit against bit."""
import numpy as np
import pytest
import torch

import oracle
import pyronn_layers as pl
from pyronn_layers import geometry
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _geo(fan, shape, width, views, sid=900.0):
    if fan:
        return geometry.FanBeam2D(shape, (0.8, 1.0), width, 1.1, views, sid, 1300.0), pl.fan_backprojection2d, \
            oracle.fan_backprojection2d
    return geometry.ParallelBeam2D(shape, (0.8, 1.0), width, 0.9, views), pl.parallel_backprojection2d, \
        oracle.parallel_backprojection2d


def _noise(seed, shape, cuda, dtype):
    p = np.random.Generator(np.random.PCG64(seed)).uniform(0.2, 1.0, shape).astype(np.float32)
    return torch.as_tensor(p).to(device=cuda, dtype=dtype)


@pytest.mark.parametrize("fan", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,shape", [
    (2, (199, 201)),  # 79 998 pixels: a slice per thread
    (2, (200, 201)),  # two slices per thread, view groups
    (3, (200, 201)),  # three
    (4, (200, 201)),  # four
    (5, (200, 201)),  # three, the last group overlapping
    (7, (200, 201)),  # four, the last group overlapping
])
@pytest.mark.parametrize("width,views", [(120, 257), (419, 33)])  # pixels off the detector; all inside
def test_shared_slices_with_view_groups(cuda, batch, shape, width, views, dtype, fan):
    geo, bwd, obwd = _geo(fan, shape, width, views)
    p = _noise(batch, (batch,) + geo.detector_shape, cuda, dtype)
    out = bwd(p, shape, *geo.args(), out_dtype=torch.float32)
    for b in range(batch):
        assert torch.equal(bwd(p[b:b + 1], shape, *geo.args(), out_dtype=torch.float32)[0], out[b])
    ends = [0, batch - 1]
    ref = obwd(p[ends].float().cpu().numpy(), shape, *geo.args())
    assert rel_l2(out[ends].cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("fan", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(256, 256), (257, 256), (362, 363)])  # two slices: 131 072 pixels, above, far above
def test_geometry_per_element(cuda, shape, dtype, fan):
    """A slice per thread, with view groups up to 131 072 pixels and without."""
    geos = [_geo(fan, shape, 200, 19, sid) for sid in (700.0, 900.0)]
    args = [np.stack(a) for a in zip(geos[0][0].args(), geos[1][0].args())]
    p = _noise(9, (2,) + geos[0][0].detector_shape, cuda, dtype)
    out = geos[0][1](p, shape, *args, out_dtype=torch.float32)
    for b, (geo, bwd, obwd) in enumerate(geos):
        ref = obwd(p[b:b + 1].float().cpu().numpy(), shape, *geo.args())
        assert rel_l2(out[b].cpu().numpy(), ref[0]) < 1e-5
