"""Forward interval kernels at the edges of their tiles and dispatch rules, against float64.

Error of a float32 sum of n products in any order: at most n * 2^-24 * sum |c w| (+ the same for the radius), first order.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from boundflow_b200.csrc import build

    build.build()
    return torch.device("cuda", 0)


# 16-row / 16- and 32-column tiles (K <= 1024), K split over a cluster (K > 1024; ragged, unaligned, shorter than eight ranks), 64 x 64 tiles
@pytest.mark.parametrize("B,K,N", [(1, 1, 1), (16, 63, 16), (17, 64, 17), (37, 1024, 130), (100, 65, 513), (200, 512, 512), (640, 30, 1000), (16, 8192, 10), (1, 1025, 1),
                                   (33, 1568, 100), (200, 4096, 65), (31, 1031, 33), (513, 2050, 513), (640, 1100, 1000)])
def test_ibp_linear_tiles(dev, B, K, N):
    from boundflow_b200 import _lib

    lib = _lib.load()
    g = torch.Generator("cuda").manual_seed(B + K + N)
    l = torch.randn(B, K, generator=g, device=dev)
    u = l + torch.rand(B, K, generator=g, device=dev)
    W = torch.randn(N, K, generator=g, device=dev)
    b = torch.randn(N, generator=g, device=dev)
    split = torch.randint(-1, 2, (B, N), generator=g, device=dev, dtype=torch.int8)
    out = [torch.full((B, N), float("nan"), device=dev) for _ in range(2)]
    bad = torch.zeros(B, dtype=torch.int32, device=dev)
    _lib.check(lib.bf_ibp_linear(l.data_ptr(), u.data_ptr(), _lib.IN_LOWER_UPPER, 1, W.data_ptr(), b.data_ptr(), split.data_ptr(), N, None, None,
                                 out[0].data_ptr(), out[1].data_ptr(), bad.data_ptr(), B, K, N, None))
    l64, u64, W64 = l.relu().double(), u.relu().double(), W.double()
    c, r = (l64 + u64) / 2, (u64 - l64) / 2
    mid, dev_ = c @ W64.t(), r @ W64.abs().t()
    lo, up = mid - dev_ + b.double(), mid + dev_ + b.double()
    lo, up = torch.where(split > 0, lo.clamp(min=0), lo), torch.where(split < 0, up.clamp(max=0), up)
    tol = (K + 4) * 2.0 ** -24 * (c.abs() @ W64.abs().t() + dev_) + 1e-6
    assert ((out[0].double() - lo).abs() <= tol).all() and ((out[1].double() - up).abs() <= tol).all()
    sure = ((lo - up).abs() > 2 * tol).all(dim=1)
    assert torch.equal(bad[sure].bool(), (lo > up).any(dim=1)[sure])


# channel tiles of 16, 32 and 64, ragged pixels and channels, kernels larger than a slab (clusters along K: below, above 1024 taps)
@pytest.mark.parametrize("B,Ci,H,W,Co,k,s,p", [(1, 1, 5, 7, 1, 1, 1, 0), (3, 1, 28, 28, 16, 4, 2, 1), (2, 3, 9, 11, 17, 3, 1, 1), (5, 16, 14, 14, 33, 4, 2, 1),
                                               (64, 8, 16, 16, 32, 3, 2, 1), (300, 3, 16, 15, 20, 5, 1, 2), (7, 64, 8, 8, 70, 4, 2, 1), (40, 40, 13, 13, 64, 3, 1, 0)])
def test_ibp_conv_tiles(dev, B, Ci, H, W, Co, k, s, p):
    from boundflow_b200 import _lib

    lib = _lib.load()
    g = torch.Generator("cuda").manual_seed(B + Ci + Co + k)
    l = torch.randn(B, Ci, H, W, generator=g, device=dev)
    u = l + torch.rand(l.shape, generator=g, device=dev)
    w = torch.randn(Co, Ci, k, k, generator=g, device=dev)
    b = torch.randn(Co, generator=g, device=dev)
    conv = lambda x, ww: torch.nn.functional.conv2d(x, ww, None, s, p)
    l64, u64, w64 = l.relu().double(), u.relu().double(), w.double()
    c, r = (l64 + u64) / 2, (u64 - l64) / 2
    mid, dev_ = conv(c, w64) + b.double()[:, None, None], conv(r, w64.abs())
    split = torch.randint(-1, 2, mid.shape, generator=g, device=dev, dtype=torch.int8)
    out = [torch.full(mid.shape, float("nan"), device=dev) for _ in range(2)]
    bad = torch.zeros(B, dtype=torch.int32, device=dev)
    _lib.check(lib.bf_ibp_conv2d(l.data_ptr(), u.data_ptr(), _lib.IN_LOWER_UPPER, 1, w.data_ptr(), b.data_ptr(), split.data_ptr(), split[0].numel(), None,
                                 None, out[0].data_ptr(), out[1].data_ptr(), bad.data_ptr(), B, Ci, H, W, Co, k, k, s, s, p, p, None))
    lo, up = mid - dev_, mid + dev_
    lo, up = torch.where(split > 0, lo.clamp(min=0), lo), torch.where(split < 0, up.clamp(max=0), up)
    tol = (Ci * k * k + 4) * 2.0 ** -24 * (conv(c.abs(), w64.abs()) + dev_) + 1e-6
    assert ((out[0].double() - lo).abs() <= tol).all() and ((out[1].double() - up).abs() <= tol).all()
    sure = ((lo - up).abs() > 2 * tol).flatten(1).all(dim=1)
    assert torch.equal(bad[sure].bool(), (lo > up).flatten(1).any(dim=1)[sure])


# 32 x 64 tiles of the CROWN backward step: one row, ragged rows, columns and k, one slab and several, rows of a domain across tiles
@pytest.mark.parametrize("B,S,K,N", [(1, 1, 20, 30), (1, 9, 64, 64), (3, 11, 65, 61), (37, 9, 130, 257), (128, 9, 256, 256), (5, 40, 513, 100), (64, 9, 100, 784)])
@pytest.mark.parametrize("side", [0, 1])
def test_backward_small_tiles(dev, B, S, K, N, side):
    from boundflow_b200 import _lib

    lib = _lib.load()
    g = torch.Generator("cuda").manual_seed(B * K + N)
    A = torch.randn(B, S, K, generator=g, device=dev)
    au, al, bu = (torch.rand(B, K, generator=g, device=dev) for _ in range(3))
    W = torch.randn(K, N, generator=g, device=dev)
    b = torch.randn(K, generator=g, device=dev)
    out = torch.full((B, S, N), float("nan"), device=dev)
    delta = torch.full((B, S), 2.0, device=dev)
    _lib.check(lib.bf_crown_relu_linear_bwd(A.data_ptr(), side, au.data_ptr(), al.data_ptr(), bu.data_ptr(), None, None, W.data_ptr(), b.data_ptr(),
                                            out.data_ptr(), delta.data_ptr(), 1, B, S, K, N, None))
    A64, pos = A.double(), A >= 0
    lo, hi = (al, au) if side == 0 else (au, al)
    lam = A64 * torch.where(pos, lo.double()[:, None], hi.double()[:, None])
    icpt = A64 * torch.where(pos == (side == 1), bu.double()[:, None], torch.zeros_like(A64))
    ref, ref_d = lam @ W.double(), 2.0 + (icpt + lam * b.double()).sum(-1)
    tol = (K + 2) * 2.0 ** -24 * (lam.abs() @ W.double().abs()) + 1e-6
    tol_d = (2 * K + 4) * 2.0 ** -24 * (2.0 + (icpt.abs() + (lam * b.double()).abs()).sum(-1))
    assert ((out.double() - ref).abs() <= tol).all()
    assert ((delta.double() - ref_d).abs() <= tol_d).all()


# tensor-core ReLU + transposed convolution: ragged channels (Co % 16, Ci below a block, several blocks), odd maps, rows that no window reaches
# ((H + 2p - k) % s != 0), rows shorter and longer than a tile, both sides, with and without a ReLU
@pytest.mark.parametrize("B,S,Ci,H,W,Co,k,s,p", [(8, 40, 8, 9, 9, 16, 3, 1, 1), (5, 80, 13, 14, 11, 21, 4, 2, 1), (4, 64, 32, 16, 16, 64, 3, 1, 1), (4, 64, 64, 16, 16, 64, 4, 2, 1),
                                                 (30, 50, 32, 9, 7, 40, 3, 2, 0), (3, 40, 20, 33, 32, 17, 4, 2, 1), (300, 70, 9, 2, 3, 8, 2, 1, 0)])
@pytest.mark.parametrize("side,relu", [(0, True), (1, True), (0, False)])
def test_conv_backward_tensor_cores(dev, B, S, Ci, H, W, Co, k, s, p, side, relu):
    from boundflow_b200 import _lib

    lib = _lib.load()
    Ho, Wo = (H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1
    g = torch.Generator("cuda").manual_seed(B + Ci + Co)
    A = torch.randn(B, S, Co, Ho, Wo, generator=g, device=dev)
    au, al, bu = (torch.rand(B, Co, Ho, Wo, generator=g, device=dev) for _ in range(3))
    w = torch.randn(Co, Ci, k, k, generator=g, device=dev)
    b = torch.randn(Co, generator=g, device=dev)
    out = torch.full((B, S, Ci, H, W), float("nan"), device=dev)
    delta = torch.full((B, S), 2.0, device=dev)
    nbytes = lib.bf_crown_relu_conv2d_bwd_scratch_bytes(B, S, Co, Ho, Wo)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    before = _lib.tc_launch_count()
    a_u, a_l, b_u = (au.data_ptr(), al.data_ptr(), bu.data_ptr()) if relu else (None, None, None)
    _lib.check(lib.bf_crown_relu_conv2d_bwd(A.data_ptr(), side, a_u, a_l, b_u, None, w.data_ptr(), b.data_ptr(), out.data_ptr(), delta.data_ptr(), 1,
                                            scratch.data_ptr(), nbytes, B, S, Ci, H, W, Co, Ho, Wo, k, k, s, s, p, p, None))
    assert _lib.tc_launch_count() == before + 1
    lam, icpt = A.double(), torch.zeros_like(A, dtype=torch.float64)
    if relu:
        pos = A >= 0
        lo, hi = (al, au) if side == 0 else (au, al)
        icpt = lam * torch.where(pos == (side == 1), bu.double()[:, None], icpt)
        lam = lam * torch.where(pos, lo.double()[:, None], hi.double()[:, None])
    opad = (H - ((Ho - 1) * s - 2 * p + k), W - ((Wo - 1) * s - 2 * p + k))
    conv_t = lambda x, ww: torch.nn.functional.conv_transpose2d(x.flatten(0, 1), ww, None, s, p, output_padding=opad).view(out.shape)
    ref = conv_t(lam, w.double())
    ref_d = 2.0 + (icpt + lam * b.double()[:, None, None]).sum((2, 3, 4))
    # operands are exact; the sums keep the bound of an FP32 sum of Co k^2 / s^2 products
    tol = (Co * (k * k) / (s * s) + 8) * 2.0 ** -24 * conv_t(lam.abs(), w.double().abs()) + 1e-6
    tol_d = (2 * Co * Ho * Wo + 8) * 2.0 ** -24 * (2.0 + (icpt.abs() + (lam * b.double()[:, None, None]).abs()).sum((2, 3, 4)))
    assert ((out.double() - ref).abs() <= tol).all()
    assert ((delta.double() - ref_d).abs() <= tol_d).all()


# an input's interval bounds are the same bits in every batch: all kernels behind one layer sum in one order (also above 1024 terms)
@pytest.mark.parametrize("K,N", [(700, 33), (1025, 1), (1568, 100), (4096, 65)])
def test_ibp_linear_bits_do_not_depend_on_the_batch(dev, K, N):
    from boundflow_b200 import _lib

    lib = _lib.load()
    g = torch.Generator("cuda").manual_seed(K + N)
    most = 148 * 64  # a 64 x 64 tile per SM
    l = torch.randn(most, K, generator=g, device=dev)
    u = l + torch.rand(most, K, generator=g, device=dev)
    W = torch.randn(N, K, generator=g, device=dev)

    def bounds(rows):
        out = [torch.full((rows, N), float("nan"), device=dev) for _ in range(2)]
        _lib.check(lib.bf_ibp_linear(l.data_ptr(), u.data_ptr(), _lib.IN_LOWER_UPPER, 1, W.data_ptr(), None, None, 0, None, None, out[0].data_ptr(),
                                     out[1].data_ptr(), None, rows, K, N, None))
        return torch.stack(out)

    whole = bounds(most)
    for rows in (1, 17, 200):
        assert torch.equal(bounds(rows), whole[:, :rows])


# the same of convolutions, of intervals and of plain rows; all three channel-tile widths above 1024 terms, ragged pixels, several images in a tile
@pytest.mark.parametrize("Ci,H,W,Co,k,s,p", [(65, 7, 6, 16, 4, 1, 1), (130, 5, 9, 30, 3, 2, 1), (65, 9, 9, 70, 4, 2, 0), (12, 9, 8, 17, 3, 1, 1)])
def test_forward_conv_bits_do_not_depend_on_the_batch(dev, Ci, H, W, Co, k, s, p):
    from boundflow_b200 import _lib

    lib = _lib.load()
    Ho, Wo = (H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1
    g = torch.Generator("cuda").manual_seed(Ci + Co)
    most = 2000
    x = torch.randn(most, Ci, H, W, generator=g, device=dev)
    r = torch.rand(most, Ci, H, W, generator=g, device=dev)
    w = torch.randn(Co, Ci, k, k, generator=g, device=dev)
    b = torch.randn(Co, generator=g, device=dev)

    def run(B):
        lo, up, y = (torch.full((B, Co, Ho, Wo), float("nan"), device=dev) for _ in range(3))
        _lib.check(lib.bf_ibp_conv2d(x.data_ptr(), r.data_ptr(), _lib.IN_MID_RAD, 0, w.data_ptr(), b.data_ptr(), None, 0, None, None, lo.data_ptr(), up.data_ptr(),
                                     None, B, Ci, H, W, Co, k, k, s, s, p, p, None))
        _lib.check(lib.bf_rows_conv2d_fwd(x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), B, Ci, H, W, Co, Ho, Wo, k, k, s, s, p, p, None))
        return lo, up, y

    whole = run(most)
    for B in (1, 7):
        assert all(torch.equal(part, full[:B]) for part, full in zip(run(B), whole))
    # against float64: n products and sums, in any order
    conv = lambda a, ww: torch.nn.functional.conv2d(a[:7].double(), ww.double(), None, s, p)
    tol = (Ci * k * k + 4) * 2.0**-24 * (conv(x.abs(), w.abs()) + conv(r, w.abs())) + 1e-6
    bias = b.double()[:, None, None]
    for got, ref in zip(whole, (conv(x, w) - conv(r, w.abs()), conv(x, w) + conv(r, w.abs()), conv(x, w))):
        assert ((got[:7].double() - (ref + bias)).abs() <= tol).all()


# (rows, Ci, map, Co, kernel, stride, padding): plain rows whose sums are cut in four, two and not at all, on both sides of each line (74 and 76, 296 and 298
# tiles; 126 and 128, 252 and 261 taps), parts of unequal length, a part without taps, one row, and eight channels a thread with channels past the end
@pytest.mark.parametrize("M,Ci,H,Co,k,s,p", [(1, 16, 14, 32, 4, 2, 1), (37, 32, 16, 20, 3, 1, 1), (38, 32, 16, 20, 3, 1, 1), (148, 32, 16, 20, 3, 1, 1), (149, 32, 16, 20, 3, 1, 1),
                                             (5, 14, 8, 17, 3, 1, 1), (5, 8, 8, 17, 4, 2, 1), (40, 28, 16, 20, 3, 1, 1), (40, 29, 16, 20, 3, 1, 1), (149, 16, 8, 64, 4, 1, 0), (7, 33, 7, 33, 3, 1, 1), (3, 40, 9, 70, 5, 2, 2), (74, 16, 8, 64, 3, 1, 1),
                                             (75, 32, 8, 64, 3, 1, 1), (300, 16, 8, 64, 3, 1, 1), (2, 130, 6, 65, 3, 1, 1), (9, 2, 10, 16, 8, 1, 0)])
def test_plain_rows_cut_in_parts(dev, M, Ci, H, Co, k, s, p):
    from boundflow_b200 import _lib

    lib, g = _lib.load(), torch.Generator("cuda").manual_seed(M + Ci + Co)
    x, w, b = torch.randn(M, Ci, H, H, generator=g, device=dev), torch.randn(Co, Ci, k, k, generator=g, device=dev), torch.randn(Co, generator=g, device=dev)
    Ho = (H + 2 * p - k) // s + 1
    conv = lambda t, u, v: torch.nn.functional.conv2d(t.double(), u.double(), v.double(), stride=s, padding=p)

    def run():
        y = torch.full((M, Co, Ho, Ho), float("nan"), device=dev)
        _lib.check(lib.bf_rows_conv2d_fwd(x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), M, Ci, H, H, Co, Ho, Ho, k, k, s, s, p, p, None))
        return y

    # a sum of K products in any order is off by at most (K + 4) u times the sum of their magnitudes, u = 2^-24
    bound = (Ci * k * k + 4) * 2.0**-24 * conv(x.abs(), w.abs(), b.abs())
    assert ((run().double() - conv(x, w, b)).abs() <= bound).all()
    # an infinite weight counts where its tap lies inside the image, also in the middle parts of a sum
    w[Co - 1, Ci // 2, 0, 0] = float("inf")
    want, got = conv(x, torch.where(w.isinf(), 0, w), b), run()
    inside = torch.nn.functional.conv2d(x[:, Ci // 2 : Ci // 2 + 1].sign().double(), torch.nn.functional.pad(torch.ones(1, 1, 1, 1, device=dev, dtype=torch.float64), (0, k - 1, 0, k - 1)), stride=s, padding=p)
    assert torch.equal(got[:, Co - 1].isposinf(), inside[:, 0] > 0) and torch.equal(got[:, Co - 1].isneginf(), inside[:, 0] < 0)
    assert not got.isnan().any() and ((got.double() - want).abs() <= bound)[:, : Co - 1].all()
