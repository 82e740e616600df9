"""GPU tests of the ramp filter on rows outside the ordinary range: infinities,
NaNs, masked pixels of the storage type's lowest value and neighbours whose
difference overflows, against direct FP64 sums over the taps that are not zero."""
import numpy as np
import pytest
import torch

from pyronn_layers import _capi
from conftest import rel_l2

pytestmark = pytest.mark.gpu

SDD, DV, DU = 500.0, 1.1, 0.8


def _taps(kind, width):
    m = np.arange(width, dtype=np.float64)
    if kind == 1:
        return -2.0 / (np.pi ** 2 * DU * (4.0 * m * m - 1.0))
    h = np.where(m % 2 == 1, -1.0 / (np.pi ** 2 * np.maximum(m, 1.0) ** 2 * DU), 0.0)
    h[0] = 0.25 / DU
    return h


def _direct(rows, kind):
    """Each row's filter and the sum of the terms' magnitudes, FP64."""
    n, width = rows.shape
    k = np.arange(width)
    h = _taps(kind, width)[np.abs(k[:, None] - k[None, :])]
    u = (k - (width - 1) / 2) * DU
    v = (np.arange(n) - (n - 1) / 2) * DV
    g = rows.astype(np.float64) * (SDD / np.sqrt(SDD ** 2 + u[None, :] ** 2 + v[:, None] ** 2))
    with np.errstate(invalid="ignore"):
        terms = np.where(h != 0.0, h * g[:, None, :], 0.0)
        return terms.sum(-1), np.abs(terms).sum(-1)


def _rows(width, dtype):
    low = float(torch.finfo(dtype).min)
    p = np.random.Generator(np.random.PCG64(width)).uniform(0.2, 1.0, (7, width))
    p[1, width // 3] = np.inf
    p[2, width // 2] = np.nan
    p[3, ::2], p[3, 1::2] = -0.6 * low, 0.6 * low  # neighbours whose difference overflows
    p[4, width // 5] = low
    p[6] = 0.0
    return torch.as_tensor(p).to(dtype)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("width", [37, 128, 129, 256, 300, 511, 1025, 2048, 2049])
@pytest.mark.parametrize("in_place", [False, True])
def test_filter_rows_out_of_range(cuda, width, dtype, kind, in_place):
    if in_place and dtype != torch.float32:
        pytest.skip("in place: one storage type; 16-bit outputs overflow")
    rows = _rows(width, dtype)
    x = rows.to(cuda)
    out = x if in_place else torch.empty((7, width), device=cuda)
    code = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}[dtype]
    _capi.call("pyronn_fdk_filter", x.data_ptr(), out.data_ptr(), code, 0, 1, 1, 7, width, SDD, DV, DU, 3.0,
               (width - 1) / 2, kind, 0, torch.cuda.current_stream().cuda_stream)
    got = out.double().cpu().numpy()
    ref, size = _direct(rows.double().numpy(), kind)
    if width % 4 == 0 and width <= 2048 and not in_place:
        ref[1:3] = np.nan
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    np.testing.assert_array_equal(np.isposinf(got), np.isposinf(ref))
    np.testing.assert_array_equal(np.isneginf(got), np.isneginf(ref))
    # sequential FP32 sums of `width` products, the cosine weight within 4 ulp
    bound = (width + 8) * 2.0 ** -24 * size + 1e-37
    for r in (1, 2, 3, 4):
        ok = np.isfinite(ref[r])
        assert (np.abs(got[r][ok] - ref[r][ok]) <= bound[r][ok]).all()
    for r in (0, 5):
        assert rel_l2(got[r], ref[r]) < 1e-5
    assert (got[6] == 0).all()


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("rows", [1, 2, 31, 33, 700])
@pytest.mark.parametrize("width", [1, 2, 63, 127, 128, 129])
def test_filter_short_rows(cuda, width, rows, kind):
    """Rows about the width of the shortest transform, two groups of threads to
    a warp: each row to 1e-5 (as test_fbp_gpu.py), whatever its neighbours."""
    p = np.random.Generator(np.random.PCG64(width + rows)).uniform(0.2, 1.0, (rows, width)).astype(np.float32)
    p[1::3] *= np.float32(1e-7)
    x = torch.as_tensor(p, device=cuda)
    out = torch.empty_like(x)
    _capi.call("pyronn_fdk_filter", x.data_ptr(), out.data_ptr(), 0, 0, 1, 1, rows, width, SDD, DV, DU, (rows - 1) / 2,
               (width - 1) / 2, kind, 0, torch.cuda.current_stream().cuda_stream)
    ref, _ = _direct(p, kind)
    got = out.double().cpu().numpy()
    for r in range(rows):
        assert rel_l2(got[r], ref[r]) < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("width,kind", [(48, 0), (255, 1), (2048, 0), (2049, 0), (2049, 1), (3000, 1), (4096, 0)])
def test_filter_in_place_and_types(cuda, width, kind, in_place, dtype):
    """Ordinary rows of every storage type, filtered in place and not, by
    transforms and (above 2048) by direct sums: 1e-5, and half an ulp of 16-bit
    outputs."""
    p = np.random.Generator(np.random.PCG64(width)).uniform(0.2, 1.0, (5, width))
    x = torch.as_tensor(p, dtype=dtype, device=cuda)
    ref, _ = _direct(x.double().cpu().numpy(), kind)
    out = x if in_place else torch.empty_like(x)
    code = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}[dtype]
    _capi.call("pyronn_fdk_filter", x.data_ptr(), out.data_ptr(), code, code, 1, 1, 5, width, SDD, DV, DU, 2.0,
               (width - 1) / 2, kind, 0, torch.cuda.current_stream().cuda_stream)
    rounding = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -11}[dtype]
    assert rel_l2(out.double().cpu().numpy(), ref) < 1e-5 + rounding
