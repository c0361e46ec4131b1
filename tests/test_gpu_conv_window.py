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


def _serial(A, W, stride, pad=0):
    """Each sum over output channels, kernel rows, kernel columns ascending, one rounding a term: on inputs in steps of 2^-12 every
    product and sum is exact in float64 before it is rounded to float32 (products in steps of 2^-24, sums below 2^20)."""
    M, Co, w, _ = A.shape
    Ci, k = W.shape[1], W.shape[2]
    ow = (w - 1) * stride + k - 2 * pad
    out = torch.zeros((M, Ci, ow, ow), device="cuda")
    for co in range(Co):
        for r in range(k):
            for c in range(k):
                ys = [y for y in range(w) if 0 <= y * stride + r - pad < ow]
                xs = [x for x in range(w) if 0 <= x * stride + c - pad < ow]
                part = out[:, :, ys[0] * stride + r - pad:ys[-1] * stride + r - pad + 1:stride, xs[0] * stride + c - pad:xs[-1] * stride + c - pad + 1:stride]
                x = A[:, co, ys[0]:ys[-1] + 1, xs[0]:xs[-1] + 1].double()[:, None]
                part.copy_((x * W[co, :, r, c].double()[None, :, None, None] + part.double()).float())
    return out


def _grid(shape, g):
    return (torch.randn(shape, generator=g, device="cuda") * 4096).round() / 4096


# few rows (single channels), rows of several tiles per block with a ragged last one (groups of channels, odd counts of chunks), channel
# counts that no 16-byte window word fits
@pytest.mark.parametrize("k, stride, w", GEOMETRIES)
@pytest.mark.parametrize("rows, ci, co", [(40, 12, 8), (33, 3, 5), (40, 9, 31), (700, 32, 8), (20011, 4, 12), (5003, 24, 20)])
def test_windows_keep_the_order_of_sums(k, stride, w, rows, ci, co):
    g = torch.Generator("cuda").manual_seed(1000 * w + 10 * k + ci)
    A, W = _grid((rows, co, w, w), g), _grid((co, ci, k, k), g)
    assert torch.equal(_backward(A, W, stride), _serial(A, W, stride))


@pytest.mark.parametrize("w", (6, 8, 10))
@pytest.mark.parametrize("rows, ci, co", [(2048, 1, 5), (3001, 2, 7), (20011, 1, 12), (25601, 2, 6)])
def test_padded_maps_keep_the_order_of_sums(w, rows, ci, co):
    g = torch.Generator("cuda").manual_seed(w + rows)
    A, W = _grid((rows, co, w, w), g), _grid((co, ci, 4, 4), g)
    assert torch.equal(_backward(A, W, 2, 1), _serial(A, W, 2, 1))


@pytest.mark.parametrize("k, stride, w", [(3, 1, 3), (4, 2, 4), (3, 1, 14)])
def test_infinite_weight_reaches_only_its_taps(k, stride, w):
    A = torch.ones((40, 4, w, w), device="cuda")
    W = torch.ones((4, 3, k, k), device="cuda")
    W[1, 2, 0, 0] = float("inf")
    out = _backward(A, W, stride)
    reach = torch.zeros_like(out[0, 2], dtype=torch.bool)
    reach[0:(w - 1) * stride + 1:stride, 0:(w - 1) * stride + 1:stride] = True
    assert torch.isinf(out[:, 2][:, reach]).all() and torch.isfinite(out[:, 2][:, ~reach]).all() and torch.isfinite(out[:, :2]).all()
