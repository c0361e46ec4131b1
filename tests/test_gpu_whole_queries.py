"""Queries that the library answers in one call against the same queries step by step (an input set whose tensors it cannot read in place): same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from boundflow_b200.csrc import build

    build.build()
    return torch.device("cuda", 0)


def _wide(t):
    """t with a gap behind every element: not contiguous."""
    out = torch.empty(tuple(t.shape) + (2,), device=t.device)[..., 0]
    out.copy_(t)
    return out


NETS = [((784,), [("fc", 10)]), ((784,), [("fc", 33), ("fc", 10)]), ((784,), [("fc", 100), ("fc", 257), ("fc", 65), ("fc", 10)]),
        ((784,), [("fc", 9 + r) for r in range(18)] + [("fc", 10)]), ((1, 28, 28), [("conv", 8, 4, 2, 1), ("conv", 5, 4, 2, 1), ("fc", 37), ("fc", 10)])]


@pytest.mark.parametrize("ball", ["box", "linf"])
@pytest.mark.parametrize("net", range(len(NETS)))
@pytest.mark.parametrize("B", [1, 17, 150])  # both sides join in one sweep for some, not for others
def test_one_call_and_many_agree(dev, net, ball, B):
    from boundflow_b200 import crown
    from boundflow_b200 import workloads as W
    from boundflow_b200.executor import CudaTaskExecutor
    from boundflow_b200.ir import InputSpec, normalize_input_spec

    wl = W.make_workload("c1" if len(NETS[net][0]) == 1 else "c2", batch=B, eps=1e-3, net=W.NetSpec(*NETS[net]))
    lo, up, C = wl.lo.to(dev), wl.up.to(dev), wl.C.to(dev)
    make = (lambda f: InputSpec.box(value_name="input", lower=f(lo), upper=f(up))) if ball == "box" else (
        lambda f: InputSpec.linf(value_name="input", center=f(lo), eps=1e-3))
    one, many = make(lambda t: t.contiguous()), make(_wide)
    assert crown._plain_set(normalize_input_spec(one)) is not None and crown._plain_set(normalize_input_spec(many)) is None
    for f in (lambda s: CudaTaskExecutor().run_ibp(wl.module, s), lambda s: crown.run_crown_ibp_mlp(wl.module, s, linear_spec_C=C),
              lambda s: crown.run_crown_ibp_mlp(wl.module, s)):
        a, b = f(one), f(many)
        assert torch.equal(a.lower, b.lower) and torch.equal(a.upper, b.upper) and a.lower.shape == b.lower.shape
    for chunk in (7, 1024, 10**12):
        (a, pa), (b, pb) = (crown.run_crown_intermediate_mlp(wl.module, s, linear_spec_C=C, chunk_rows=chunk) for s in (one, many))
        assert torch.equal(a.lower, b.lower) and torch.equal(a.upper, b.upper) and list(pa) == list(pb)
        for n in pa:
            assert torch.equal(pa[n].lower, pb[n].lower) and torch.equal(pa[n].upper, pb[n].upper) and pa[n].lower.shape == pb[n].lower.shape


# Chains that begin with a flatten or a convolution, on both sides of where a Linear layer of 48, 50 or 64 outputs leaves the FP32 tiles (one wave of
# 64 x 64 tiles): neither sweep, the joined one only, both
@pytest.mark.parametrize("body, batches", [([("fc", 48), ("fc", 10)], (40, 78, 79, 100, 149, 157, 170)), ([("fc", 64), ("fc", 10)], (78, 80, 150, 160)),
                                           ([("conv", 16, 4, 2, 1), ("conv", 32, 4, 2, 1), ("fc", 50), ("fc", 10)], (39, 40, 60, 78, 90))])
def test_sides_join_where_no_layer_changes_its_kernel(dev, body, batches):
    from boundflow_b200 import crown
    from boundflow_b200 import workloads as W
    from boundflow_b200.ir import InputSpec

    for B in batches:
        wl = W.make_workload("c2", batch=B, eps=1e-3, net=W.NetSpec((1, 28, 28), body))
        lo, up, C = wl.lo.to(dev), wl.up.to(dev), wl.C.to(dev)
        a, b = (crown.run_crown_ibp_mlp(wl.module, InputSpec.box(value_name="input", lower=f(lo), upper=f(up)), linear_spec_C=C) for f in (torch.clone, _wide))
        assert torch.equal(a.lower, b.lower) and torch.equal(a.upper, b.upper), B


# a 100-wide MLP (few rows on the tensor cores by default) and a flatten-first one whose joined sweep would leave the FP32 tiles (by default it does not join)
@pytest.mark.parametrize("body, batches", [([("fc", 100), ("fc", 10)], (1, 17, 64, 150, 300)), ([("fc", 48), ("fc", 10)], (17, 64, 100))])
def test_switches_are_read_before_anything_is_decided(dev, monkeypatch, body, batches):
    """The first query of a chain under BF_B200_FORCE_FFMA=1 is the second one's, and its sides' one by one; a workspace sized before is large enough."""
    from boundflow_b200 import _lib, crown
    from boundflow_b200 import workloads as W
    from boundflow_b200.ir import InputSpec
    from boundflow_b200.network import compile_chain

    lib = _lib.load()
    for B in batches:
        wl = W.make_workload("c2", batch=B, eps=1e-3, net=W.NetSpec((1, 28, 28), body))
        lo, up, C = wl.lo.to(dev), wl.up.to(dev), wl.C.to(dev)
        monkeypatch.delenv("BF_B200_FORCE_FFMA", raising=False)
        chain = compile_chain(wl.module, (1, 28, 28), dev)
        S, n = int(C.shape[1]), int(lib.bf_chain_query_workspace_bytes(chain.handle, B, int(C.shape[1]), 0))
        monkeypatch.setenv("BF_B200_FORCE_FFMA", "1")
        bounds = []
        for _ in range(2):
            ws, out = torch.empty(n, dtype=torch.uint8, device=dev), torch.empty((2, B, S), device=dev)
            launches = _lib.tc_launch_count()
            _lib.check(lib.bf_chain_crown_query(chain.handle, lo.data_ptr(), up.data_ptr(), 0.0, C.data_ptr(), out[0].data_ptr(), out[1].data_ptr(), ws.data_ptr(), n, B, S, None))
            assert _lib.tc_launch_count() == launches
            bounds.append(out)
        a, b = (crown.run_crown_ibp_mlp(wl.module, InputSpec.box(value_name="input", lower=f(lo), upper=f(up)), linear_spec_C=C) for f in (torch.clone, _wide))
        torch.cuda.synchronize()
        for other in (bounds[1], torch.stack((a.lower, a.upper)), torch.stack((b.lower, b.upper))):
            assert torch.equal(bounds[0], other), B


@pytest.mark.parametrize("B", [1, 2, 8])
def test_neurons_of_linear_layers_keep_the_order_of_their_sums(dev, monkeypatch, B):
    """Bounds that decide default slopes come from the FP32 tiles at every number of rows: whole query, identity rows and given rows."""
    from boundflow_b200 import crown
    from boundflow_b200 import workloads as W
    from boundflow_b200.ir import InputSpec

    wl = W.make_workload("c1", batch=B, eps=1e-3, net=W.NetSpec((784,), [("fc", 100), ("fc", 128), ("fc", 70), ("fc", 10)]))
    lo, up, C = wl.lo.to(dev), wl.up.to(dev), wl.C.to(dev)
    rows = torch.eye(70, device=dev)[None, 20:40].expand(B, -1, -1).contiguous()

    def bounds(f):
        spec = InputSpec.box(value_name="input", lower=f(lo), upper=f(up))
        _, pre = crown.run_crown_intermediate_mlp(wl.module, spec, linear_spec_C=C, chunk_rows=50)
        trace = crown.ibp_trace(wl.module, spec)
        given = crown.crown_from_trace(trace, rows, output_value=wl.relu_names[2])
        return [t for s in pre.values() for t in (s.lower, s.upper)] + list(given)

    got = [bounds(f) for f in (torch.clone, _wide)]
    monkeypatch.setenv("BF_B200_FORCE_FFMA", "1")
    want = bounds(torch.clone)
    assert all(torch.equal(a, b) for g in got for a, b in zip(g, want))


def test_contradictions_are_reported(dev):
    """lower > upper in one input set: both routes raise, and name the same domains."""
    from boundflow_b200 import crown
    from boundflow_b200 import workloads as W
    from boundflow_b200.ir import InputSpec

    wl = W.make_workload("c1", batch=5, eps=1e-3, net=W.NetSpec(*NETS[2]))
    lo, up = wl.lo.to(dev).clone(), wl.up.to(dev).clone()
    lo[3], up[3] = up[3].clone() + 1, lo[3].clone()
    said = []
    for f in (lambda t: t.contiguous(), _wide):
        with pytest.raises(ValueError) as e:
            crown.run_crown_intermediate_mlp(wl.module, InputSpec.box(value_name="input", lower=f(lo), upper=f(up)), linear_spec_C=wl.C.to(dev))
        said.append(str(e.value))
    assert said[0] == said[1] and "[3]" in said[0]


def test_other_norms_stay_refused(dev):
    """Only "inf" balls are read as boxes of radius eps."""
    from boundflow_b200 import crown
    from boundflow_b200.ir import InputSpec, normalize_input_spec

    spec = normalize_input_spec(InputSpec.linf(value_name="input", center=torch.zeros(2, 4, device=dev), eps=0.1))

    class Odd:
        eps = 0.1

        def norm(self):
            return "3"

    class Spec:
        center, perturbation = spec.center, Odd()

    assert crown._plain_set(spec) is not None and crown._plain_set(Spec()) is None


@pytest.mark.parametrize("R,B", [(1, 1), (16, 5), (19, 33)])
def test_relaxations_in_one_launch_or_many(dev, R, B):
    """bf_relu_relax_many against bf_relu_relax: default slopes, slopes per domain and shared ones, past the edge of a launch (16 ReLUs)."""
    from boundflow_b200 import _lib
    from boundflow_b200.crown import relax_all

    lib, g = _lib.load(), torch.Generator("cuda").manual_seed(R)
    widths = [1 + (13 * r) % 70 for r in range(R)]
    l = [torch.randn(B, n, generator=g, device=dev) - 0.5 for n in widths]
    u = [x + torch.rand(x.shape, generator=g, device=dev) * 2 for x in l]
    alpha = [None if r % 3 == 0 else torch.rand(B if r % 3 == 1 else 1, n, generator=g, device=dev) for r, n in enumerate(widths)]
    strides = [n if r % 3 == 1 else 0 for r, n in enumerate(widths)]
    many = relax_all(lib, l, u, alpha, strides, widths, B, dev)
    for r, n in enumerate(widths):
        one = [torch.empty(B, n, device=dev) for _ in range(3)]
        _lib.check(lib.bf_relu_relax(l[r].data_ptr(), u[r].data_ptr(), _lib.ptr(alpha[r]), strides[r], *[t.data_ptr() for t in one], B, n, None))
        assert all(torch.equal(a[r], b) for a, b in zip(many, one))


@pytest.mark.parametrize("B", [1, 3, 40])
def test_graph_sides_in_one_sweep_or_two(dev, B):
    """The graph walker's joined sweep against one sweep a side (zero terms behind a ReLU keep the sides apart).  Twice the rows may take a convolution
    to the tensor cores: the roundings of sums of up to 1152 products, about sqrt(1152) 2^-24 = 2e-6 of the bounds, 1e-5 leaves a factor of five."""
    from boundflow_b200 import dag
    from boundflow_b200.ir import BFTaskModule, BoundTask, InputSpec, TaskKind, TaskOp

    g = torch.Generator().manual_seed(B)
    P = {"w1": torch.randn(8, 3, 3, 3, generator=g) * 0.2, "b1": torch.randn(8, generator=g) * 0.1, "w2": torch.randn(8, 8, 3, 3, generator=g) * 0.1,
         "w3": torch.randn(10, 8 * 12 * 12, generator=g) * 0.03, "b3": torch.randn(10, generator=g) * 0.1}
    conv = {"stride": 1, "padding": 1, "dilation": 1, "groups": 1}
    ops = [TaskOp("conv2d", "c1", ["x", "w1", "b1"], ["y1"], conv), TaskOp("relu", "r1", ["y1"], ["z1"]), TaskOp("conv2d", "c2", ["z1", "w2"], ["y2"], conv),
           TaskOp("add", "a", ["y2", "z1"], ["y3"]), TaskOp("relu", "r2", ["y3"], ["z3"]), TaskOp("flatten", "f", ["z3"], ["z4"], {"start_dim": 1, "end_dim": -1}),
           TaskOp("linear", "l", ["z4", "w3", "b3"], ["out"])]
    module = BFTaskModule([BoundTask("t", TaskKind.INTERVAL_IBP, ops, ["x"], ["out"])], "t", bindings={"params": {k: v.to(dev) for k, v in P.items()}})
    x = torch.rand(B, 3, 12, 12, generator=g).to(dev)
    spec = InputSpec.box(value_name="x", lower=x - 0.02, upper=x + 0.02)
    C = torch.randn(B, 9, 10, generator=g).to(dev)
    lo, up, tr = dag.crown_dag(module, spec, C)
    assert dag._sides_join(module, tr, tr.params, 9, "out")
    zero = {"y1": torch.zeros(B, 8 * 12 * 12, device=dev)}
    lo2, up2, _ = dag.crown_dag(module, spec, C, relu_pre_add_coeff_l=zero, relu_pre_add_coeff_u=zero)
    scale = torch.maximum(lo2.abs(), up2.abs()).max()
    assert (lo - lo2).abs().max() <= 1e-5 * scale and (up - up2).abs().max() <= 1e-5 * scale and lo.shape == up.shape == (B, 9)


# by their number alone, the rows of both sides would change kernels: to the tensor cores (4 to 6 inputs of 16 channels, 1 to 16 of 8) or from them
@pytest.mark.parametrize("c0, c1, H, batches", [(16, 32, 32, (1, 4, 5, 6, 8, 16)), (8, 8, 32, (2, 4, 10, 16)), (16, 32, 16, (4, 12, 14, 24)), (12, 24, 28, (2, 5, 8))])
def test_graph_sides_join_on_the_kernels_of_one_side(dev, c0, c1, H, batches):
    """Same kernels, and same bits on the FP32 ones.  The tensor-core convolution cuts its row sums at tiles that begin elsewhere in the joined block: sums of
    up to 16384 products in another order, about sqrt(16384) 2^-24 = 8e-6 of their terms' size, and the bias terms are a fraction of the bounds."""
    from boundflow_b200 import _lib, dag
    from boundflow_b200.ir import BFTaskModule, BoundTask, InputSpec, TaskKind, TaskOp

    g = torch.Generator().manual_seed(c0 + H)
    P = {}

    def conv(name, x, y, ci, co, k, s):
        P["w" + name], P["b" + name] = torch.randn(co, ci, k, k, generator=g) * (2 / (ci * k * k)) ** 0.5, torch.randn(co, generator=g) * 0.1
        return TaskOp("conv2d", name, [x, "w" + name, "b" + name], [y], {"stride": s, "padding": k // 2, "dilation": 1, "groups": 1})

    ops = [conv("1", "x", "y1", 3, c0, 3, 1), TaskOp("relu", "r1", ["y1"], ["z1"]), conv("2", "z1", "y2", c0, c0, 3, 1), TaskOp("relu", "r2", ["y2"], ["z2"]), conv("3", "z2", "y3", c0, c0, 3, 1),
           TaskOp("add", "a1", ["y3", "z1"], ["y4"]), TaskOp("relu", "r4", ["y4"], ["z4"]), conv("5", "z4", "y5", c0, c1, 3, 2), TaskOp("relu", "r5", ["y5"], ["z5"]),
           conv("6", "z5", "y6", c1, c1, 3, 1), conv("7", "z4", "y7", c0, c1, 1, 2), TaskOp("add", "a2", ["y6", "y7"], ["y8"]), TaskOp("relu", "r8", ["y8"], ["z8"]),
           TaskOp("flatten", "f", ["z8"], ["z9"], {"start_dim": 1, "end_dim": -1}), TaskOp("linear", "l", ["z9", "w9", "b9"], ["out"])]
    P["w9"], P["b9"] = torch.randn(10, c1 * (H // 2) ** 2, generator=g) * 0.03, torch.randn(10, generator=g)
    module = BFTaskModule([BoundTask("t", TaskKind.INTERVAL_IBP, ops, ["x"], ["out"])], "t", bindings={"params": {k: v.to(dev) for k, v in P.items()}})
    for B in batches:
        x = torch.rand(B, 3, H, H, generator=g).to(dev)
        spec = InputSpec.box(value_name="x", lower=x - 0.01, upper=x + 0.01)
        C = torch.randn(B, 9, 10, generator=g).to(dev)
        count = [_lib.tc_launch_count()]
        lo, up, tr = dag.crown_dag(module, spec, C)
        count.append(_lib.tc_launch_count())
        assert dag._sides_join(module, tr, tr.params, 9, "out")
        zero = {"y1": torch.zeros(B, c0 * H * H, device=dev)}
        lo2, up2, _ = dag.crown_dag(module, spec, C, relu_pre_add_coeff_l=zero, relu_pre_add_coeff_u=zero)
        count.append(_lib.tc_launch_count())
        on_tensor_cores = count[1] - count[0]
        assert count[2] - count[1] == 2 * on_tensor_cores
        scale = torch.maximum(lo2.abs(), up2.abs()).max()
        print(c0, H, B, on_tensor_cores, float((lo - lo2).abs().max() / scale))
        if on_tensor_cores == 0:
            assert torch.equal(lo, lo2) and torch.equal(up, up2), B
        assert (lo - lo2).abs().max() <= 8e-6 * scale and (up - up2).abs().max() <= 8e-6 * scale
