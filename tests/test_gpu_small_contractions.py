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
