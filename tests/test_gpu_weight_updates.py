"""Weights that a program changes in place between two queries: every query is about the weights as they are when it runs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from boundflow_b200.csrc import build

    build.build()
    return torch.device("cuda", 0)


def _workload(dev, B, layers):
    """A workload whose parameters live on the GPU, where the library reads them in place."""
    from boundflow_b200 import workloads as W

    wl = W.make_workload("c1", batch=B, eps=1e-3, net=W.NetSpec((784,), layers))
    params = wl.module.bindings["params"]
    for k in params:
        params[k] = params[k].to(dev)
    return wl, params


def _fresh(module):
    """The same task with parameters of its own: nothing of what was kept for `module` is for it."""
    from boundflow_b200.ir import BFTaskModule

    return BFTaskModule(tasks=module.tasks, entry_task_id=module.entry_task_id, bindings={"params": {k: v.clone() for k, v in module.bindings["params"].items()}})


def _flat(x):
    if torch.is_tensor(x):
        return [x]
    if isinstance(x, dict):
        return [t for v in x.values() for t in _flat(v)]
    return [t for v in x for t in _flat(v)]


def _queries(wl, dev):
    from boundflow_b200 import crown
    from boundflow_b200.ir import InputSpec

    lo, up, C = wl.lo.to(dev), wl.up.to(dev), wl.C.to(dev)
    wide = torch.empty(tuple(lo.shape) + (2,), device=dev)[..., 0].copy_(lo)
    box, strided, l2 = InputSpec.box(value_name="input", lower=lo, upper=up), InputSpec.box(value_name="input", lower=wide, upper=up), InputSpec.l2(value_name="input", center=lo, eps=0.01)
    both = lambda r: [r.lower, r.upper]

    def loop(m, s, **kw):
        r, alpha, _, _ = crown.run_alpha_beta_crown_mlp(m, s, linear_spec_C=C, steps=2, lr=0.1, **kw)
        return [r.lower, r.upper, alpha.alpha_by_relu_input]

    return {"query": lambda m: both(crown.run_crown_ibp_mlp(m, box, linear_spec_C=C)), "steps": lambda m: both(crown.run_crown_ibp_mlp(m, strided, linear_spec_C=C)),
            "l2": lambda m: both(crown.run_crown_ibp_mlp(m, l2, linear_spec_C=C)), "intermediate": lambda m: both(crown.run_crown_intermediate_mlp(m, box, linear_spec_C=C)[0]),
            "loop": lambda m: loop(m, box, per_batch_params=True), "shared": lambda m: loop(m, box, per_batch_params=False)}


UPDATES = {"mul_": lambda p: p.mul_(1.25), "data": lambda p: p.data.mul_(1.25), "copy_": lambda p: p.copy_(p.flip(0))}


# rows of the tensor-core kernel of few rows (9 rows a domain)
@pytest.mark.parametrize("update", list(UPDATES))
@pytest.mark.parametrize("B, name", [(B, n) for B in (1, 64) for n in ("query", "steps", "l2", "loop", "shared")] + [(1, "intermediate")])
def test_queries_of_few_rows_follow_their_weights(dev, B, name, update):
    wl, params = _workload(dev, B, [("fc", 100), ("fc", 100), ("fc", 10)])
    query = _queries(wl, dev)[name]
    before = _flat(query(wl.module))
    for p in params.values():
        UPDATES[update](p)
    got, want = _flat(query(wl.module)), _flat(query(_fresh(wl.module)))
    assert not torch.equal(got[0], before[0]) and all(torch.equal(a, b) for a, b in zip(got, want))
