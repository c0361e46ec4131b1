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
