"""Prepared packs of host geometry are found by content, never by identity."""
import numpy as np
import pytest
import torch

from pyronn_layers import geometry, ops


def _x(batch):
    return torch.zeros((batch, 4, 4))


def test_pack_is_keyed_by_content():
    geo = geometry.FanBeam2D((4, 4), (1.0, 1.0), 7, 1.0, 5, 30.0, 50.0)
    args = [np.array(a) for a in geo.args()]

    def pack(batch=1):
        vo, do, vs, ds, si, sd, rays = args
        return ops._geometry_2d(_x(batch), 5, vo, do, vs, ds, rays, si, sd)

    a = pack()
    assert pack() is a
    args[6] = args[6].copy()  # the same values in another array
    assert pack() is a
    args[4][0] = 31.0  # an array changed in place is other geometry
    b = pack()
    assert b is not a and float(b.sid) == 31.0 and float(a.sid) == 30.0
    assert pack(2) is not b  # rows are prepared per batch size
    args[6] = torch.from_numpy(args[6])  # a CPU tensor of the same values
    assert pack() is b
    args[6] = args[6].tolist()
    assert pack() is b


def test_pack_kinds_and_errors():
    par = geometry.ParallelBeam2D((4, 4), (1.0, 1.0), 7, 1.0, 5)
    p = ops._geometry_2d(_x(1), 5, *par.args())
    assert not p.fan and ops._geometry_2d(_x(1), 5, *par.args()) is p
    with pytest.raises(ValueError):
        ops._geometry_2d(_x(1), 6, *par.args())  # rays of another view count
    n = len(ops._PACKS)
    cone = geometry.ConeBeam3D((4, 4, 4), (1, 1, 1), (6, 6), (1, 1), 3, 50.0, 80.0)
    x = torch.zeros((2, 4, 4, 4))
    c = ops._geometry_cone(x, 3, *cone.args())
    assert ops._geometry_cone(x, 3, *cone.args()) is c and c.g == 1 and len(ops._PACKS) == n + 1


def test_pack_cache_is_bounded():
    par = geometry.ParallelBeam2D((4, 4), (1.0, 1.0), 7, 1.0, 5)
    vo, do, vs, ds, rays = par.args()
    for k in range(ops._HOST_GEOM_CACHE_SIZE + 8):
        ops._geometry_2d(_x(1), 5, vo, np.float32([k]), vs, ds, rays)
    assert len(ops._PACKS) <= ops._HOST_GEOM_CACHE_SIZE
