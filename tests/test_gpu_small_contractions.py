"""32 x 64 tiles of the FP32 contractions (gemm_small.cuh): edges of tiles, slabs and 16-byte accesses, ragged widths."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from boundflow_b200.csrc import build

    build.build()
    return torch.device("cuda", 0)


@pytest.mark.parametrize("D, S, K, N", [(1, 1, 17, 5), (11, 3, 33, 65), (37, 9, 70, 64), (5, 9, 100, 137), (20, 9, 31, 200), (3, 2, 128, 63), (7, 5, 97, 128), (64, 9, 256, 256)])
@pytest.mark.parametrize("side", [0, 1])
def test_backward_step_against_float64(dev, D, S, K, N, side):
    from boundflow_b200 import _lib

    lib = _lib.load()
    g = torch.Generator().manual_seed(D + K + N)
    A = torch.randn((D, S, K), generator=g)
    au, al, bu = (torch.rand((D, K), generator=g) for _ in range(3))
    add, W, b = torch.randn((D, K), generator=g), torch.randn((K, N), generator=g), torch.randn((K,), generator=g)
    d = {n: t.to(dev) for n, t in dict(A=A, au=au, al=al, bu=bu, add=add, W=W, b=b).items()}
    out = torch.full((D, S, N), float("nan"), device=dev)
    delta = torch.ones((D, S), device=dev)
    _lib.check(lib.bf_crown_relu_linear_bwd(d["A"].data_ptr(), side, d["au"].data_ptr(), d["al"].data_ptr(), d["bu"].data_ptr(), None, d["add"].data_ptr(), d["W"].data_ptr(),
                                            d["b"].data_ptr(), out.data_ptr(), delta.data_ptr(), 1, D, S, K, N, None))
    a = A.double()
    pos, neg = (al, au) if side == 0 else (au, al)
    lam = a * torch.where(a >= 0, pos.double()[:, None], neg.double()[:, None]) + add.double()[:, None]
    # bu is the intercept where the upper relaxation is taken: negative coefficients of a lower bound, positive ones of an upper bound
    icpt = a * bu.double()[:, None] * ((a < 0) if side == 0 else (a >= 0))
    # n rounded terms in any order are within n * 2^-24 of the sum of their magnitudes; the scaling rounds once more
    ref, size = lam @ W.double(), (a.abs() + add.double().abs()[:, None]) @ W.double().abs()
    assert ((out.cpu().double() - ref).abs() <= (K + 2) * 2.0**-24 * size).all()
    want = 1 + (icpt + lam * b.double()).sum(-1)
    size = 1 + (icpt.abs() + (a.abs() + add.double().abs()[:, None]) * b.double().abs()).sum(-1)
    assert ((delta.cpu().double() - want).abs() <= (2 * K + 4) * 2.0**-24 * size).all()


@pytest.mark.parametrize("B, widths", [(7, (33, 70, 65)), (2, (64, 32)), (40, (31, 129)), (13, (36, 36, 100))])
@pytest.mark.parametrize("with_beta", [False, True])
def test_alpha_steps_of_ragged_layers(dev, B, widths, with_beta):
    from boundflow_b200 import workloads as W
    from boundflow_b200.crown import run_alpha_beta_crown_mlp
    from boundflow_b200.ir import InputSpec
    from oracle import crown_oracle as O

    wl = W.make_workload("c1", batch=B, eps=0.01, net=W.NetSpec((784,), [("fc", w) for w in widths] + [("fc", 10)]))
    spec = InputSpec.box(value_name="input", lower=wl.lo.to(dev), upper=wl.up.to(dev))
    inp = O.box_input(wl.lo, wl.up)
    splits = state = None
    if with_beta:  # every third unstable neuron on its midpoint's side
        splits = [torch.where(l + u > 0, 1, -1).to(torch.int8) * ((l < 0) & (u > 0) & (torch.arange(l.shape[1]) % 3 == 0)) for l, u in O.forward_ibp_trace(wl.layers, inp).pre]
        state = {n: s.to(dev) for n, s in zip(wl.relu_names, splits)}
    b, alpha, beta, _ = run_alpha_beta_crown_mlp(wl.module, spec, linear_spec_C=wl.C.to(dev), relu_split_state=state, steps=2, lr=0.1, per_batch_params=True)
    out = O.alpha_crown(wl.layers, inp, wl.C, steps=2, lr=0.1, splits=splits, optimize_beta=with_beta, return_beta=with_beta)
    # an Adam step moves a parameter by about lr in the direction of its gradient, except where that is zero up to rounding
    for r, n in enumerate(wl.relu_names):
        for got, want in ((alpha.alpha_by_relu_input, out[2]),) + (((beta.beta_by_relu_input, out[3]),) if with_beta else ()):
            same = (got[n].reshape(B, -1).cpu() - want[r].reshape(B, -1)).abs() <= 1e-3
            assert same.float().mean() >= 0.95, (r, n)


# the last three: more tiles than SMs (two adjoint CTAs per SM), the others fewer; the one before them: more only with the CTAs of the row sums
@pytest.mark.parametrize("B, S, n0, widths", [(7, 9, 33, (33, 70, 65)), (2, 9, 784, (64, 32)), (40, 9, 50, (31, 129)), (70, 1, 65, (65,)), (3, 32, 40, (100, 100)),
                                              (64, 9, 70, (512, 512)), (72, 9, 784, (512, 512)), (300, 9, 64, (128, 100)), (147, 9, 61, (197, 130))])
def test_alpha_gradient_is_exact_on_small_integers(dev, B, S, n0, widths):
    """Integer weights and inputs, slopes in quarters: every sum is exact in FP32 in any order, so the gradient of every neuron of every
    domain, and the bounds, have to be those of float64."""
    from boundflow_b200 import workloads as W
    from boundflow_b200.crown import alpha_grad_from_trace, ibp_trace
    from boundflow_b200.ir import InputSpec

    g = torch.Generator().manual_seed(B + n0)
    pick = lambda values, *shape: torch.tensor(values)[torch.randint(0, len(values), shape, generator=g)]
    wl = W.make_workload("c1", batch=1, net=W.NetSpec((n0,), [("fc", w) for w in widths] + [("fc", 10)]))
    params, dims = wl.module.bindings["params"], (n0,) + tuple(widths) + (10,)
    for k in range(1, len(dims)):
        keep = torch.rand((dims[k], dims[k - 1]), generator=g) < min(1.0, 24.0 / dims[k - 1])
        params[f"W{k}"], params[f"b{k}"] = pick((-1.0, 1.0), dims[k], dims[k - 1]) * keep, pick((-2.0, -1.0, 1.0, 2.0), dims[k])
    mid, rad = pick((-2.0, -1.0, 0.0, 1.0, 3.0), B, n0), pick((0.0, 1.0, 2.0), B, n0)
    C = pick((-1.0, 0.0, 1.0), B, S, 10)
    pre_l = [pick((-1.0, -1.0, -1.0, -2.0, 0.5), B, n) for n in widths]          # slope 1/2, inactive, active
    pre_u = [torch.where(l == -2.0, -1.0, 1.0) for l in pre_l]
    alpha = [pick((0.0, 0.25, 0.5, 1.0), B, n) for n in widths]
    trace = ibp_trace(wl.module, InputSpec.box(value_name="input", lower=(mid - rad).to(dev), upper=(mid + rad).to(dev)))
    trace.pre_l, trace.pre_u = [t.to(dev) for t in pre_l], [t.to(dev) for t in pre_u]
    grads, lower = alpha_grad_from_trace(trace, C.to(dev), [a.to(dev) for a in alpha], spec_reduce="sum")

    def contract(x, M, quarters):  # x M in float64; its terms' magnitudes stay below 2^24 of the grid of the values
        assert (x.abs() @ M.abs()).max() * 4.0**quarters < 2.0**23
        return x @ M

    Ws, bs = [params[f"W{k}"].double() for k in range(1, len(dims))], [params[f"b{k}"].double() for k in range(1, len(dims))]
    open_ = [(l < 0) & (u > 0) for l, u in zip(pre_l, pre_u)]
    up = [torch.where(o, 0.5, (l > 0).double())[:, None].double() for o, l in zip(open_, pre_l)]
    low = [torch.where(o, a.double(), (l > 0).double())[:, None] for o, l, a in zip(open_, pre_l, alpha)]
    icpt = [o.double()[:, None] * 0.5 for o in open_]
    A, R, bound, Ahat = C.double(), len(widths), 0.0, [None] * len(widths)
    for r in reversed(range(R)):
        bound = bound + A @ bs[r + 1]
        Ahat[r] = contract(A, Ws[r + 1], R - 1 - r)
        bound = bound + (torch.where(Ahat[r] < 0, Ahat[r], 0.0) * icpt[r]).sum(-1)
        A = Ahat[r] * torch.where(Ahat[r] >= 0, low[r], up[r])
    bound = bound + A @ bs[0]
    A = contract(A, Ws[0], R)
    want = bound + (A * mid.double()[:, None]).sum(-1) - (A.abs() * rad.double()[:, None]).sum(-1)
    assert torch.equal(lower.cpu().double(), want)
    h = mid.double()[:, None] - A.sign() * rad.double()[:, None]
    for r in range(R):
        v = contract(h, Ws[r].t(), r) + bs[r]
        terms = torch.where((Ahat[r] >= 0) & open_[r][:, None], Ahat[r] * v, 0.0)
        assert terms.abs().sum(1).max() * 4.0**R < 2.0**23
        assert torch.equal(grads[r].cpu().double(), -terms.sum(1)), r
        h = torch.where(Ahat[r] >= 0, low[r] * v, up[r] * v + icpt[r])


@pytest.mark.parametrize("N", (4, 60, 64, 68, 784))
def test_infinite_coefficients_keep_their_sign(dev, N):
    """One Linear layer with positive weights and a negative bias on a box below zero: a row with an infinite coefficient is
    bounded by minus infinity, whatever its width."""
    import ctypes

    from boundflow_b200 import _lib

    lib = _lib.load()
    B, S, K = 3, 2, 20
    g = torch.Generator().manual_seed(N)
    W, b = (torch.rand((K, N), generator=g) + 0.5).to(dev), (-torch.rand((K,), generator=g) - 0.5).to(dev)
    mid, rad = torch.full((B, N), -1.0, device=dev), torch.full((B, N), 0.25, device=dev)
    C = torch.rand((B, S, K), generator=g).to(dev)
    C[:, 1, 7] = float("inf")
    desc = (_lib.LayerDesc * 1)()
    desc[0].op, desc[0].W, desc[0].bias, desc[0].n_in, desc[0].n_out = _lib.OP_LINEAR, W.data_ptr(), b.data_ptr(), N, K
    chain = ctypes.c_void_p()
    _lib.check(lib.bf_chain_create(desc, 1, ctypes.byref(chain)))
    try:
        nbytes = int(lib.bf_chain_crown_workspace_bytes(chain, B, S, 1))
        ws, out = torch.empty(nbytes, dtype=torch.uint8, device=dev), torch.empty((B, S), device=dev)
        _lib.check(lib.bf_chain_crown(chain, 1, _lib.SIDE_LOWER, C.data_ptr(), None, None, None, None, mid.data_ptr(), rad.data_ptr(), _lib.NORM_BOX, 0.0,
                                      out.data_ptr(), ws.data_ptr(), nbytes, B, S, None))
    finally:
        lib.bf_chain_destroy(chain)
    assert torch.isfinite(out[:, 0]).all()
    assert (out[:, 1] == -float("inf")).all(), out[:, 1]
