"""Unpadded transposed convolution of small square maps (conv_window.cu): every instance against float64, rows that do not fill a
warp, channel counts that do not fill a group, infinite weights."""
import pytest
import torch

from boundflow_b200 import _lib

pytestmark = pytest.mark.gpu


def _backward(A, W, stride, pad=0):
    """Layer-level call without slopes: A [M, Co, w, w], W [Co, Ci, k, k]."""
    M, Co, w, _ = A.shape
    Ci, k = W.shape[1], W.shape[2]
    ow = (w - 1) * stride + k - 2 * pad
    out = torch.full((M, Ci, ow, ow), float("nan"), device="cuda")
    lib = _lib.load()
    _lib.check(lib.bf_crown_relu_conv2d_bwd_fp32(A.data_ptr(), _lib.SIDE_LOWER, None, None, None, None, W.data_ptr(), None, out.data_ptr(), None, 1,
                                                 None, 0, 1, M, Ci, ow, ow, Co, w, w, k, k, stride, stride, pad, pad, None))
    return out


GEOMETRIES = [(3, 1, w) for w in (2, 3, 4, 5, 6, 7, 8, 10, 12, 14)] + [(k, 2, w) for k in (3, 4) for w in (2, 3, 4, 5, 6, 7)]


@pytest.mark.parametrize("k, stride, w", GEOMETRIES)
@pytest.mark.parametrize("rows, ci, co", [(1, 1, 4), (33, 3, 12), (70, 9, 20), (301, 32, 36)])
def test_windows_against_float64(k, stride, w, rows, ci, co):
    g = torch.Generator().manual_seed(100 * w + 10 * k + ci)
    A = torch.randn((rows, co, w, w), generator=g)
    W = torch.randn((co, ci, k, k), generator=g)
    ref = torch.nn.functional.conv_transpose2d(A.double(), W.double(), stride=stride)
    size = torch.nn.functional.conv_transpose2d(A.double().abs(), W.double().abs(), stride=stride)
    # a serial FP32 sum of n products is within n * 2^-24 of the sum of their magnitudes
    n = co * ((k + stride - 1) // stride) ** 2
    err = (_backward(A.cuda(), W.cuda(), stride).cpu().double() - ref).abs()
    assert (err <= n * 2.0**-24 * size).all()


@pytest.mark.parametrize("w", (6, 8, 10))
@pytest.mark.parametrize("rows, ci, co", [(2047, 1, 3), (2048, 1, 3), (2085, 2, 16)])
def test_padded_maps_against_float64(w, rows, ci, co):
    g = torch.Generator().manual_seed(w + ci)
    A = torch.randn((rows, co, w, w), generator=g)
    W = torch.randn((co, ci, 4, 4), generator=g)
    ref = torch.nn.functional.conv_transpose2d(A.double(), W.double(), stride=2, padding=1)
    size = torch.nn.functional.conv_transpose2d(A.double().abs(), W.double().abs(), stride=2, padding=1)
    err = (_backward(A.cuda(), W.cuda(), 2, 1).cpu().double() - ref).abs()
    assert (err <= 4 * co * 2.0**-24 * size).all()  # four products per channel


@pytest.mark.parametrize("k, stride, w", [(3, 1, 3), (4, 2, 4), (3, 1, 14)])
def test_infinite_weight_reaches_only_its_taps(k, stride, w):
    A = torch.ones((40, 4, w, w), device="cuda")
    W = torch.ones((4, 3, k, k), device="cuda")
    W[1, 2, 0, 0] = float("inf")
    out = _backward(A, W, stride)
    reach = torch.zeros_like(out[0, 2], dtype=torch.bool)
    reach[0:(w - 1) * stride + 1:stride, 0:(w - 1) * stride + 1:stride] = True
    assert torch.isinf(out[:, 2][:, reach]).all() and torch.isfinite(out[:, 2][:, ~reach]).all() and torch.isfinite(out[:, :2]).all()
