"""Linear layers of few coefficient rows on the tensor cores (crown_small_tc.cu): edges of feature tiles, row tiles, stages, clusters and rings."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from boundflow_b200.csrc import build

    build.build()
    return torch.device("cuda", 0)


class _Chain:
    """Linear (ReLU Linear)* on device weights, with its packed images; gradients and bounds by bf_chain_alpha_grad."""

    def __init__(self, Ws, bs, dev):
        from boundflow_b200 import _lib

        self.lib, self._lib, self.R = _lib.load(), _lib, len(Ws) - 1
        self.keep = [t.to(dev).contiguous() for t in Ws + bs]
        W, b = self.keep[:len(Ws)], self.keep[len(Ws):]
        desc = (_lib.LayerDesc * (2 * self.R + 1))()
        for i, w in enumerate(W):
            d = desc[2 * i]
            d.op, d.W, d.bias, d.n_in, d.n_out = _lib.OP_LINEAR, w.data_ptr(), b[i].data_ptr(), w.shape[1], w.shape[0]
            if i < self.R:
                desc[2 * i + 1].op, desc[2 * i + 1].n_in, desc[2 * i + 1].n_out = _lib.OP_RELU, w.shape[0], w.shape[0]
        self.h = ctypes.c_void_p()
        _lib.check(self.lib.bf_chain_create(desc, 2 * self.R + 1, ctypes.byref(self.h)))
        n = int(self.lib.bf_chain_tc_bytes(self.h))
        self.pack = torch.empty(n, dtype=torch.uint8, device=dev)
        _lib.check(self.lib.bf_chain_tc_prepare(self.h, self.pack.data_ptr(), n, None))

    def grad(self, C, pre_l, pre_u, alpha, mid, rad):
        D, S, _ = C.shape
        ptrs = lambda ts: (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])
        grad = [torch.full_like(a, float("nan")) for a in alpha]
        lower = torch.full((D, S), float("nan"), device=C.device)
        n = int(self.lib.bf_chain_alpha_workspace_bytes(self.h, D, S))
        ws = torch.empty(n, dtype=torch.uint8, device=C.device)
        tc = self._lib.tc_launch_count()
        self._lib.check(self.lib.bf_chain_alpha_grad(self.h, C.data_ptr(), ptrs(pre_l), ptrs(pre_u), ptrs(alpha), mid.data_ptr(), rad.data_ptr(),
                                                     self._lib.NORM_BOX, 0.0, ptrs(grad), lower.data_ptr(), 1, ws.data_ptr(), n, D, S, None))
        st = ctypes.c_int(-1)
        self._lib.check(self.lib.bf_chain_tc_status(self.h, ctypes.byref(st)))
        assert st.value == 0
        return grad, lower, self._lib.tc_launch_count() - tc

    def close(self):
        self.lib.bf_chain_destroy(self.h)


# (D, S, widths): one row; two rows past a tile; sums of 65, 96 and 97 terms, odd widths; few rows of long sums (clusters of four, rings that turn); rows
# per domain 1, 7 (more than two domains in a block), 8, 32; one tile and 129 features; more tiles than SMs, one CTA each; the largest counts of the rule
@pytest.mark.parametrize("D, S, dims", [(1, 1, (65, 65, 3)), (34, 1, (70, 96, 66, 5)), (5, 7, (97, 129, 128, 8)), (9, 8, (128, 255, 100, 9)), (3, 32, (300, 127, 33)),
                                        (2, 9, (1000, 777, 10)), (11, 9, (1570, 100, 10)), (48, 9, (784, 256, 256, 10)), (37, 9, (512, 512, 512, 10)),
                                        (263, 9, (256, 256, 256, 10)), (785, 9, (256, 256, 255, 10)), (160, 9, (784, 512, 10)), (1, 9, (4100, 130, 10))])
def test_gradients_and_bounds_against_float64(dev, D, S, dims):
    g = torch.Generator().manual_seed(D + sum(dims))
    Ws = [torch.randn((n, k), generator=g) * (2.0 / k) ** 0.5 for k, n in zip(dims, dims[1:])]
    bs = [torch.randn((n,), generator=g) * 0.1 for n in dims[1:]]
    R = len(Ws) - 1
    # relaxations with slopes away from zero: no sign of a coefficient hangs on a rounding that a zero slope would amplify
    pre_l = [-0.5 - torch.rand((D, n), generator=g) for n in dims[1:-1]]
    pre_u = [0.5 + torch.rand((D, n), generator=g) for n in dims[1:-1]]
    alpha = [0.3 + 0.5 * torch.rand((D, n), generator=g) for n in dims[1:-1]]
    mid, rad = torch.rand((D, dims[0]), generator=g), 0.05 * torch.rand((D, dims[0]), generator=g)
    C = torch.randn((D, S, dims[-1]), generator=g)
    chain = _Chain(Ws, bs, dev)
    got, lower, launches = chain.grad(C.to(dev), [t.to(dev) for t in pre_l], [t.to(dev) for t in pre_u], [t.to(dev) for t in alpha], mid.to(dev), rad.to(dev))
    again = chain.grad(C.to(dev), [t.to(dev) for t in pre_l], [t.to(dev) for t in pre_u], [t.to(dev) for t in alpha], mid.to(dev), rad.to(dev))
    chain.close()
    assert launches > 0, "no layer took the tensor cores"
    assert torch.equal(lower, again[1]) and all(torch.equal(a, b) for a, b in zip(got, again[0]))  # run to run

    A, bound, size, Ah, up, low, icpt = C.double(), 0.0, 0.0, [], [], [], []
    for r in range(R):
        l, u = pre_l[r].double()[:, None], pre_u[r].double()[:, None]
        up.append(u / (u - l)); icpt.append(-l * u / (u - l)); low.append(alpha[r].double()[:, None])
    for r in reversed(range(R)):
        bound = bound + A @ bs[r + 1].double()
        A = A @ Ws[r + 1].double()
        Ah.insert(0, A)
        bound = bound + torch.where(A < 0, A * icpt[r], 0.0).sum(-1)
        size = size + torch.where(A < 0, A * icpt[r], 0.0).abs().sum(-1)
        A = A * torch.where(A >= 0, low[r], up[r])
    bound = bound + A @ bs[0].double()
    A = A @ Ws[0].double()
    m, q = mid.double()[:, None], rad.double()[:, None]
    want = bound + (A * m).sum(-1) - (A.abs() * q).sum(-1)
    size = size + (A.abs() * (m + q)).sum(-1) + 1
    # FP32 coefficients of R + 1 contractions of the widest sums: n rounded terms are within n * 2^-24 of the sum of their magnitudes, and random signs make that
    # sum about sqrt(n) times the result, so (R + 1) * sqrt(n) * 2^-24 of the terms that enter the bound, taken four times
    tol = 4 * (R + 1) * max(dims) ** 0.5 * 2.0**-24
    assert ((lower.cpu().double() - want).abs() <= tol * size).all(), float(((lower.cpu().double() - want).abs() / size).max() / 2.0**-24)
    # Gradients: FP32 coefficients within tol of the largest may have either sign.  Such an input coefficient moves its h by at most 2 rad, such a hidden one
    # takes the other slope: both spread through the layers above by magnitudes (dv), and everything else is compared as the bounds are.
    h, dh = m - A.sign() * q, torch.where(A.abs() <= tol * A.abs().amax(), 2 * q, 0.0)
    sharp = 0
    for r in range(R):
        v, dv = h @ Ws[r].double().t() + bs[r].double(), dh @ Ws[r].double().abs().t()
        ref = -torch.where(Ah[r] >= 0, Ah[r] * v, 0.0).sum(1)
        top = Ah[r].abs().amax()
        near = Ah[r].abs() <= tol * top
        bound = (8 * tol * Ah[r].abs() * v.abs().amax() + Ah[r].abs() * dv + torch.where(near, tol * top * (v.abs() + dv), 0.0)).sum(1)
        assert ((got[r].cpu().double() - ref).abs() <= bound).all(), r
        sharp = sharp + (bound <= 0.05 * ref.square().mean().sqrt()).double().mean() / R
        h = torch.where(Ah[r] >= 0, low[r] * v, up[r] * v + icpt[r])
        dh = torch.where(near, (low[r] * v).abs() + (up[r] * v + icpt[r]).abs(), 0.0) + torch.maximum(low[r], up[r]) * dv
    assert sharp >= 0.9  # of the entries: the bound is at most a twentieth of the gradients' size


# (D, S, widths, launches): 784 columns beyond one wave of FFMA tiles and beyond the rule of few rows (315 tiles of 128 x 32) take the 3xTF32 kernel in the
# backward sweep, whose other layers stay on FFMA tiles; the gradient sweep's layers are all of few rows.  With 5400 rows the 256-wide layers of the
# backward sweep would be on the 3xTF32 kernel, too, and are not.
@pytest.mark.parametrize("D, S, dims, launches", [(160, 9, (784, 100, 100, 10), 1 + 2), (300, 9, (784, 128, 128, 128, 10), 1 + 3), (300, 9, (784, 256, 256, 256, 10), 1 + 3),
                                                  (600, 9, (784, 256, 256, 256, 10), 3 + 3)])
def test_backward_sweeps_with_a_large_layer_keep_the_others_on_fp32_units(dev, D, S, dims, launches):
    g = torch.Generator().manual_seed(D)
    Ws, bs = [torch.randn((n, k), generator=g) for k, n in zip(dims, dims[1:])], [torch.randn((n,), generator=g) for n in dims[1:]]
    rand = lambda *s: torch.rand(s, generator=g).to(dev)
    chain = _Chain(Ws, bs, dev)
    _, _, counted = chain.grad(rand(D, S, dims[-1]), [-rand(D, n) for n in dims[1:-1]], [rand(D, n) for n in dims[1:-1]], [rand(D, n) for n in dims[1:-1]], rand(D, dims[0]), rand(D, dims[0]))
    chain.close()
    assert counted == launches


@pytest.mark.parametrize("N", (5, 128, 200))
def test_infinities_pass_as_on_the_fp32_units(dev, N):
    """One Linear layer with positive weights and a negative bias on a box below zero: a row with an infinite coefficient is bounded by minus
    infinity, the others are as they were."""
    K, B, S = 100, 3, 4
    g = torch.Generator().manual_seed(N)
    W, b = torch.rand((K, N), generator=g) + 0.5, -torch.rand((K,), generator=g) - 0.5
    C = torch.rand((B, S, K), generator=g) + 0.1
    C[:, 1, 7] = float("inf")
    chain = _Chain([W], [b], dev)
    mid, rad = torch.full((B, N), -1.0, device=dev), torch.full((B, N), 0.25, device=dev)
    lib, _lib, Cd = chain.lib, chain._lib, C.to(dev)
    n = int(lib.bf_chain_crown_workspace_bytes(chain.h, B, S, 1))
    ws, out, launches = torch.empty(n, dtype=torch.uint8, device=dev), torch.empty((B, S), device=dev), _lib.tc_launch_count()
    _lib.check(lib.bf_chain_crown(chain.h, 1, _lib.SIDE_LOWER, Cd.data_ptr(), None, None, None, None, mid.data_ptr(), rad.data_ptr(), _lib.NORM_BOX, 0.0,
                                  out.data_ptr(), ws.data_ptr(), n, B, S, None))
    assert _lib.tc_launch_count() == launches + 1
    chain.close()
    want = (C.double() @ (b.double() - 1.25 * W.double().sum(1)))[:, [0, 2, 3]]
    # two sums of K + N positive terms, each rounding at most n * 2^-24 of the result
    assert ((out[:, [0, 2, 3]].cpu().double() - want).abs() <= (K + N + 8) * 2.0**-24 * want.abs()).all()
    assert (out[:, 1] == -float("inf")).all(), out[:, 1]


# (rows of a domain, inputs, terms): one CTA a tile and clusters of two and four, first layers of 1 to 13 tiles
@pytest.mark.parametrize("B, S, n0, K", [(6, 9, 784, 512), (6, 9, 784, 1100), (40, 9, 784, 256), (1, 1, 65, 1100), (3, 2, 1600, 200), (160, 9, 129, 100)])
def test_sweeps_stay_inside_their_workspace(dev, B, S, n0, K):
    """What lies behind the bytes that the library asks for stays as it was (partial sums per row: one per part of the features)."""
    g = torch.Generator().manual_seed(n0 + K)
    chain = _Chain([torch.randn((K, n0), generator=g)], [torch.randn((K,), generator=g)], dev)
    lib, _lib = chain.lib, chain._lib
    C, mid, rad = (torch.rand(s, generator=g).to(dev) for s in ((B, S, K), (B, n0), (B, n0)))
    n, guard = int(lib.bf_chain_crown_workspace_bytes(chain.h, B, S, 1)), 1 << 20
    ws, out = torch.full((n + guard,), 0xA5, dtype=torch.uint8, device=dev), torch.empty((B, S), device=dev)
    launches = _lib.tc_launch_count()
    _lib.check(lib.bf_chain_crown(chain.h, 1, _lib.SIDE_LOWER, C.data_ptr(), None, None, None, None, mid.data_ptr(), rad.data_ptr(), _lib.NORM_BOX, 0.0,
                                  out.data_ptr(), ws.data_ptr(), n, B, S, None))
    assert _lib.tc_launch_count() == launches + 1
    assert (ws[n:] == 0xA5).all() and torch.isfinite(out).all()
    chain.close()
