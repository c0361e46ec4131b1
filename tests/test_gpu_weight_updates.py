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


# rows of the 3xTF32 kernels, whose images a chain keeps: weights of 100 and 300 columns, identity rows of the intermediate query
@pytest.mark.parametrize("update", ["mul_", "copy_"])
@pytest.mark.parametrize("name", ["query", "steps", "l2", "intermediate", "loop", "shared"])
def test_queries_of_many_rows_follow_their_weights(dev, name, update):
    wl, params = _workload(dev, 700, [("fc", 100), ("fc", 300), ("fc", 10)])
    query = _queries(wl, dev)[name]
    before = _flat(query(wl.module))
    for p in params.values():
        UPDATES[update](p)
    got, want = _flat(query(wl.module)), _flat(query(_fresh(wl.module)))
    assert not torch.equal(got[0], before[0]) and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("where", ["cpu", "double", "strided"])
def test_copied_parameters_are_copied_again(dev, where):
    """Parameters that the library cannot read in place; also by the interval pass, and in a chain with a grouped convolution."""
    from boundflow_b200 import workloads as W
    from boundflow_b200.executor import CudaTaskExecutor
    from boundflow_b200.ir import InputSpec

    as_given = {"cpu": lambda t: t.cpu(), "double": lambda t: t.to(dev).double(), "strided": lambda t: torch.stack((t, t), dim=-1).to(dev)[..., 0]}[where]
    for net in (((784,), [("fc", 100), ("fc", 10)]), ((1, 28, 28), [("conv", 8, 4, 2, 1), ("conv", 6, 4, 2, 1), ("fc", 10)])):
        wl = W.make_workload("c1" if len(net[0]) == 1 else "c2", batch=5, eps=1e-3, net=W.NetSpec(*net))
        params = wl.module.bindings["params"]
        for op in wl.module.get_entry_task().ops:
            if op.op_type == "conv2d" and params[op.inputs[1]].shape[1] % 2 == 0:
                op.attrs["groups"] = 2
                params[op.inputs[1]] = params[op.inputs[1]][:, ::2].contiguous()
        for k in params:
            params[k] = as_given(params[k])
        spec = InputSpec.box(value_name="input", lower=wl.lo.to(dev), upper=wl.up.to(dev))
        ibp = lambda m: CudaTaskExecutor().run_ibp(m, spec)
        queries = dict(_queries(wl, dev), ibp=lambda m: [ibp(m).lower, ibp(m).upper])
        for name in ("query", "loop", "ibp"):
            before = _flat(queries[name](wl.module))
            for p in params.values():
                p.mul_(1.25)
            got, want = _flat(queries[name](wl.module)), _flat(queries[name](_fresh(wl.module)))
            assert not torch.equal(got[0], before[0]) and all(torch.equal(a, b) for a, b in zip(got, want)), (net, name)


@pytest.mark.parametrize("B", [8, 700])
@pytest.mark.parametrize("given", ["cuda", "cpu"])
def test_other_streams_wait_for_images_and_copies(dev, B, given):
    """A chain compiled behind other work of one stream is used on another at once."""
    from boundflow_b200.network import compile_chain

    wl, params = _workload(dev, B, [("fc", 100), ("fc", 300), ("fc", 10)])
    if given == "cpu":
        for k in params:
            params[k] = params[k].cpu().pin_memory()
    query = _queries(wl, dev)["query"]
    want = _flat(query(_fresh(wl.module)))
    torch.cuda.synchronize()
    one, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(one):
        torch.cuda._sleep(100_000_000)
        compile_chain(wl.module, (784,), dev)
    with torch.cuda.stream(other):
        got = _flat(query(wl.module))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("B", [8, 700])
def test_weights_without_a_version_counter_are_accepted(dev, B):
    wl, params = _workload(dev, B, [("fc", 100), ("fc", 10)])
    want = _flat(_queries(wl, dev)["query"](_fresh(wl.module)))
    with torch.inference_mode():
        for k in params:
            params[k] = params[k].clone()
    assert all(torch.equal(a, b) for a, b in zip(_flat(_queries(wl, dev)["query"](wl.module)), want))


@pytest.mark.parametrize("B", [8, 700])
def test_captured_queries_follow_their_weights(dev, B):
    """A graph keeps the chain's images: a query outside packs them again in place, and the replay is about the new weights."""
    wl, params = _workload(dev, B, [("fc", 100), ("fc", 300), ("fc", 10)])
    query = _queries(wl, dev)["query"]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        query(wl.module)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _flat(query(wl.module))
    for p in params.values():
        p.mul_(1.25)
    want = _flat(query(_fresh(wl.module)))
    assert all(torch.equal(a, b) for a, b in zip(_flat(query(wl.module)), want))
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, want))
