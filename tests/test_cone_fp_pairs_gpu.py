"""GPU tests of cone forward batches that march two elements at a time."""
import numpy as np
import pytest
import torch

import pyronn_layers as pl
from pyronn_layers import _capi, geometry

pytestmark = pytest.mark.gpu


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
