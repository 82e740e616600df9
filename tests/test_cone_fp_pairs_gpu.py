"""Cone forward batches that march two elements at a time: workspace and bits."""
import numpy as np
import pytest
import torch

import pyronn_layers as pl
from pyronn_layers import _capi, geometry


def _project(x, geo, query, cuda):
    """The forward with the workspace that `query` asks for; (bytes, sinogram)."""
    batch, code = x.shape[0], pl.ops.storage_code(x.dtype)
    g = pl.ops.GeometryCone(batch, cuda, *geo.args(), geo.detector_shape[0])
    dims = (batch, *geo.volume_shape, *geo.detector_shape)
    n = _capi.workspace_size(query, *dims, code, 0, g.g)
    ws = torch.full((n + 256,), 0xA5, dtype=torch.uint8, device=cuda)
    out = torch.full((batch,) + geo.detector_shape, 7.0, device=cuda)
    _capi.call("pyronn_cone_projection3d", x.data_ptr(), out.data_ptr(), code, 0, 0, *dims, *g.pointers(), g.g,
               ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
    assert bool((ws[n:] == 0xA5).all())  # nothing is written past the workspace
    return n, out


GEO = geometry.ConeBeam3D((21, 26, 30), (1.0, 0.9, 1.1), (33, 41), (1.2, 1.3), 9, 60.0, 110.0, step_size=0.5)
NAME = "pyronn_cone_projection3d"


@pytest.mark.gpu
@pytest.mark.parametrize("wide", [(0, 1), (1, 0), (1, 1), (0, 0, 1), (0, 1, 0), (0, 0, 0, 1), (0, 0, 1, 0, 0)])
def test_pairs_of_mixed_range(cuda, wide):
    """FP16 elements beyond the packed lerps' range beside others: two at a time
    gives the bits of one at a time, and an element before the first such one
    those of a call of its own."""
    rng = np.random.Generator(np.random.PCG64(81))
    vol = rng.uniform(0.2, 1.0, (len(wide),) + GEO.volume_shape)
    vol[np.array(wide) == 1] *= 60000.0
    x = torch.as_tensor(vol).to(device=cuda, dtype=torch.float16)
    one, two = _project(x, GEO, NAME, cuda), _project(x, GEO, NAME + "_batched", cuda)
    assert two[0] > one[0] and torch.equal(one[1], two[1])
    first = wide.index(1) if 1 in wide else len(wide)
    for b in range(len(wide)):
        alone = _project(x[b:b + 1].contiguous(), GEO, NAME, cuda)[1][0]
        if b < first or wide[b]:
            assert torch.equal(alone, two[1][b])


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("vol_shape", [(1, 1, 1), (60, 8, 60), (33, 17, 21)])
@pytest.mark.parametrize("tilted", [False, True])
def test_pairs_stay_in_their_workspace(cuda, vol_shape, dtype, tilted):
    """The copies of two elements, of views in either mode, in the bytes the
    query asks for: the bits of one at a time."""
    geo = geometry.ConeBeam3D(vol_shape, (1.0, 1.0, 1.0), (40, 36), (2.5, 2.0), 5, 90.0, 170.0, step_size=0.5)
    if tilted:  # every other view turned: detector rows along z
        geo.projection_matrices = geo.projection_matrices.copy()
        geo.projection_matrices[::2] = geo.projection_matrices[::2][:, :, [0, 2, 1, 3]]
    x = torch.as_tensor(np.random.Generator(np.random.PCG64(82)).uniform(0.2, 1.0, (3,) + vol_shape)).to(cuda, dtype)
    one, two = _project(x, geo, NAME, cuda), _project(x, geo, NAME + "_batched", cuda)
    assert torch.equal(one[1], two[1]) and bool((two[1] != 0).any())


@pytest.mark.parametrize("dtype,elem", [(0, 4), (1, 2), (2, 2)])
@pytest.mark.parametrize("vol", [(512, 512, 512), (181, 203, 219), (60, 8, 60)])
def test_pair_workspace_holds_two_elements(vol, dtype, elem):
    """Two elements' copies and no more: per element two padded copies and the
    cells (16 bytes each; FP32 ones have a plane more; up to 2 % of x pitch and
    section padding), beside the per-view part."""
    z, y, x = vol
    dims = (2, z, y, x, 16, 40, 60)
    views = _capi.workspace_size(NAME, *dims, dtype, 1, 1)
    cells = 16 * (x + 2) * (y + 2) * (z + (3 if elem == 4 else 2))
    copies = 2 * (x + 3) * (y + 3) * (z + 3) * elem + cells
    pair = _capi.workspace_size(NAME + "_batched", *dims, dtype, 0, 1)
    assert 2 * copies <= pair - views <= 2.02 * copies + 4096
    assert pair >= _capi.workspace_size(NAME, *dims, dtype, 0, 1)
