"""Cached geometry outlives the work that reads it, on whatever stream, and
dropping an entry waits for nothing."""
import threading

import numpy as np
import pytest
import torch

import pyronn_layers as pl
from pyronn_layers import geometry, ops


class _Tensor:
    def __init__(self):
        self.recorded = []

    def record_stream(self, stream):
        self.recorded.append(stream)


def test_cached_geometry_is_recorded_once_per_stream(monkeypatch):
    current, capturing = [1], [False]
    monkeypatch.setattr(ops, "_stream", lambda device: current[0])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: "stream %d" % current[0])
    pack = ops.Geometry2D(1, "cpu", *geometry.ParallelBeam2D((4, 4), (1.0, 1.0), 7, 1.0, 5).args(), 5)
    dev = torch.device("cuda", 0)
    tensors = [_Tensor(), _Tensor()]
    monkeypatch.setattr(pack, "tensors", lambda: tensors)
    assert ops._launch_stream(pack, dev) == 1 and tensors[0].recorded == []  # not of the cache: its caller's
    pack.streams = set()
    for current[0] in (1, 2, 1, 2):
        assert ops._launch_stream(pack, dev) == current[0]
    capturing[0], current[0] = True, 3
    ops._launch_stream(pack, dev)
    for t in tensors:
        assert t.recorded == ["stream 1", "stream 2"]


def test_every_tensor_of_a_pack_is_recorded():
    fan = geometry.FanBeam2D((4, 4), (1.0, 1.0), 7, 1.0, 5, 30.0, 50.0)
    vo, do, vs, ds, si, sd, rays = fan.args()
    cone = geometry.ConeBeam3D((4, 4, 4), (1, 1, 1), (6, 6), (1, 1), 3, 50.0, 80.0)
    for pack in (ops.Geometry2D(1, "cpu", *geometry.ParallelBeam2D((4, 4), (1.0, 1.0), 7, 1.0, 5).args(), 5),
                 ops.Geometry2D(1, "cpu", vo, do, vs, ds, rays, 5, si, sd),
                 ops.GeometryCone(1, "cpu", *cone.args(), 3)):
        assert sorted(t.data_ptr() for t in pack.tensors()) == sorted(pack.pointers())


def _geo(k):
    return geometry.ConeBeam3D((24, 24, 24), (1.0, 1.0, 1.0), (30, 32), (1.3, 1.3), 40, 90.0 + 0.25 * k, 150.0)


@pytest.mark.gpu
@pytest.mark.parametrize("backward", [False, True])
def test_eviction_beside_a_busy_stream(cuda, backward):
    """A projection queued behind a long wait on a side stream keeps its
    geometry while the cache turns over and its memory is asked for again, and
    the turn-over does not wait for that stream."""
    x = torch.rand((1, 24, 24, 24), device=cuda, requires_grad=backward)

    def run(geo):
        y = pl.cone_projection3d(x, geo.detector_shape, *geo.args())
        if not backward:
            return y
        return torch.autograd.grad(y, x, torch.ones_like(y))[0]

    def ask_for_memory():
        return [torch.full((n,), float("nan"), device=cuda) for n in (1, 3, 40 * 12)
                for _ in range(2 * ops._HOST_GEOM_CACHE_SIZE)]

    want = run(_geo(0))
    junk = ask_for_memory()  # (its kernel is loaded and its memory allocated once)
    del junk
    for k in range(1, ops._HOST_GEOM_CACHE_SIZE + 8):  # fills the caches; everything is loaded and allocated once
        run(_geo(k))
    run(_geo(0))
    run(_geo(1))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run(_geo(1))  # (this stream's buffers are allocated)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(1 << 30)  # about half a second
        got = run(_geo(0))  # a pack made on the other stream
    for k in range(100, 100 + ops._HOST_GEOM_CACHE_SIZE + 8):
        run(_geo(k))
    junk = ask_for_memory()
    assert not side.query(), "dropping geometry waited for another stream"
    torch.cuda.synchronize()
    assert torch.equal(got, want) and all(bool(torch.isnan(j).all()) for j in junk)


@pytest.mark.gpu
def test_threads_share_the_caches(cuda):
    """Threads with a stream each, over more geometry than the caches hold: each
    call's result is that of the call alone."""
    x = torch.rand((1, 24, 24, 24), device=cuda)
    geos = [_geo(300 + k) for k in range(ops._HOST_GEOM_CACHE_SIZE + 16)]

    def project(k):
        return pl.cone_projection3d(x, geos[k].detector_shape, *geos[k].args())

    want = [project(k) for k in range(len(geos))]
    torch.cuda.synchronize()
    errors = []

    def work(seed):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                order = np.random.Generator(np.random.PCG64(seed)).permutation(np.repeat(np.arange(len(geos)), 3))
                got = [(int(k), project(int(k))) for k in order]
                stream.synchronize()
                assert all(torch.equal(y, want[k]) for k, y in got)
                stream.synchronize()
        except BaseException as e:  # reported by the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors and not any(t.is_alive() for t in threads)
