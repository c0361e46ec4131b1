"""An alpha / beta loop over more parameter tensors than one optimiser launch takes (16): 18 ReLUs, 18 or 36 tensors."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from boundflow_b200.csrc import build

    build.build()
    return torch.device("cuda", 0)


@pytest.mark.parametrize("with_beta", [False, True])
def test_more_tensors_than_one_launch(dev, with_beta):
    from boundflow_b200 import workloads as W
    from boundflow_b200.crown import run_alpha_beta_crown_mlp
    from boundflow_b200.ir import InputSpec
    from oracle import crown_oracle as O

    B, R = 3, 18
    wl = W.make_workload("c1", batch=B, eps=1e-5, net=W.NetSpec((784,), [("fc", 13 + r % 4) for r in range(R)] + [("fc", 10)]))
    spec = InputSpec.box(value_name="input", lower=wl.lo.to(dev), upper=wl.up.to(dev))
    inp = O.box_input(wl.lo, wl.up)
    trace = O.forward_ibp_trace(wl.layers, inp)
    unstable = [(l < 0) & (u > 0) for l, u in trace.pre]
    splits = state = None
    if with_beta:  # every unstable neuron on one side: its midpoint's
        splits = [torch.where(l + u > 0, 1, -1).to(torch.int8) * n for (l, u), n in zip(trace.pre, unstable)]
        state = {n: s.to(dev) for n, s in zip(wl.relu_names, splits)}
    b, alpha, beta, _ = run_alpha_beta_crown_mlp(wl.module, spec, linear_spec_C=wl.C.to(dev), relu_split_state=state, steps=2, lr=0.1, per_batch_params=True)
    out = O.alpha_crown(wl.layers, inp, wl.C, steps=2, lr=0.1, splits=splits, optimize_beta=with_beta, return_beta=with_beta)
    # two Adam steps move a parameter by at most 0.1 each, in the direction of its gradient: every ReLU's parameters must have moved as the oracle's
    # have, except where a gradient is zero up to rounding
    for r, n in enumerate(wl.relu_names):
        for got, want, start in ((alpha.alpha_by_relu_input, out[2], 0.5),) + (((beta.beta_by_relu_input, out[3], 0.0),) if with_beta else ()):
            got, want = got[n].reshape(B, -1).cpu(), want[r].reshape(B, -1)
            same = (got - want).abs() <= 1e-3
            assert same.float().mean() >= 0.9, (r, n)
            assert ((want - start).abs() > 0.05).any() == ((got - start).abs() > 0.05).any()


@pytest.mark.parametrize("R,B", [(0, 3), (1, 1), (16, 9), (19, 300), (19, 2000), (18, 2001), (2, 2009)])
def test_branch_scores_of_many_relus(dev, R, B):
    """Widest unstable gap: the first neuron of a tie and the earlier ReLU win, also over the edge of a launch (16 ReLUs); -inf and -1 without one."""
    from boundflow_b200 import _lib

    lib, g = _lib.load(), torch.Generator().manual_seed(R)
    widths = [1 + (37 * r) % 301 for r in range(R)]
    # bounds on a grid of quarters: many equal gaps; the last domain has no unstable neuron
    pre = [(-torch.randint(0, 5, (B, n), generator=g) / 4, torch.randint(0, 5, (B, n), generator=g) / 4) for n in widths]
    for l, _ in pre:
        l[-1] = 0
    want = (torch.full((B,), -float("inf")), torch.full((B,), -1), torch.full((B,), -1))
    for r, (l, u) in enumerate(pre):
        gap = torch.where((l < 0) & (u > 0), u - l, torch.tensor(-float("inf")))
        best = gap.max(1).values
        better = best > want[0]
        for w, v in zip(want, (best, torch.full((B,), r), (gap == best[:, None]).int().argmax(1))):
            w[better] = v[better].to(w.dtype)
    l, u = [x[0].to(dev) for x in pre], [x[1].to(dev) for x in pre]
    gap, relu, idx = torch.empty(B, device=dev), torch.empty(B, dtype=torch.int32, device=dev), torch.empty(B, dtype=torch.int32, device=dev)
    arr = lambda ts: _lib.ptr_array(ts) if ts else _lib.ptr_array([gap])
    _lib.check(lib.bf_branch_scores(arr(l), arr(u), _lib.int_array(widths or [1]), R, _lib.ptr(gap), _lib.ptr(relu), _lib.ptr(idx), B, None))
    for got, w in zip((gap, relu, idx), want):
        assert torch.equal(got.cpu(), w.to(got.dtype))
