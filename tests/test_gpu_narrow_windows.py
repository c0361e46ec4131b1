"""Transposed convolutions of narrow maps on the FP32 kernels (8-pixel segments, one and two image rows per thread): the bits of a sum over
output channels, then kernel rows, then kernel columns in ascending order, whatever the size."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from boundflow_b200.csrc import build

    build.build()
    return torch.device("cuda", 0)


# 4x4 / 2: two rows per thread on five to eight rows from 24 -> 32 channels on, one row on either side of each line; the other kernels: one row, among
# them maps whose tile of two rows would not fit shared memory
@pytest.mark.parametrize("Ci,Co,H,W,k,s,p", [(24, 32, 5, 7, 4, 2, 1), (33, 35, 8, 6, 4, 2, 1), (40, 32, 7, 8, 4, 2, 0), (32, 33, 6, 8, 4, 2, 0), (23, 32, 6, 6, 4, 2, 0),
                                             (24, 31, 8, 8, 4, 2, 0), (32, 32, 4, 4, 4, 2, 0), (32, 32, 9, 8, 4, 2, 0), (3, 16, 2, 3, 3, 1, 1), (4, 16, 8, 8, 3, 1, 1),
                                             (3, 8, 8, 8, 5, 1, 2), (8, 16, 16, 8, 5, 1, 2), (32, 16, 5, 5, 3, 1, 0), (16, 16, 7, 7, 3, 2, 1), (9, 10, 19, 18, 3, 2, 0)])
def test_narrow_maps_keep_the_order_of_sums(dev, monkeypatch, Ci, Co, H, W, k, s, p):
    from boundflow_b200 import _lib

    monkeypatch.setenv("BF_B200_FORCE_FFMA", "1")
    lib = _lib.load()
    Ho, Wo = (H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1
    g = torch.Generator("cuda").manual_seed(Ci + Co + H)
    M = 40
    A = torch.randn(M, Co, Ho, Wo, generator=g, device=dev)
    w = torch.randn(Co, Ci, k, k, generator=g, device=dev)
    out = torch.full((M, Ci, H, W), float("nan"), device=dev)
    _lib.check(lib.bf_crown_relu_conv2d_bwd(A.data_ptr(), 0, None, None, None, None, w.data_ptr(), None, out.data_ptr(), None, 1, None, 0, M, 1, Ci, H, W, Co, Ho, Wo,
                                            k, k, s, s, p, p, None))
    # one multiply-add per product: exact in float64 before the rounding to float32
    want = torch.zeros(M, Ci, H, W, device=dev)
    hs, ws = torch.arange(H, device=dev), torch.arange(W, device=dev)
    for co in range(Co):
        for r in range(k):
            for c in range(k):
                hn, wn = hs + p - r, ws + p - c
                rows, cols = (hn >= 0) & (hn % s == 0) & (hn // s < Ho), (wn >= 0) & (wn % s == 0) & (wn // s < Wo)
                i, j = hs[rows], ws[cols]
                x = A[:, co][:, hn[rows] // s][:, :, wn[cols] // s].double()[:, None]
                part = want[:, :, i[:, None], j]
                want[:, :, i[:, None], j] = (x * w[co, :, r, c].double()[None, :, None, None] + part.double()).float()
    assert torch.equal(out, want)
