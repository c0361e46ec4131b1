"""Identity spec rows without an identity tensor (`bf_chain_crown_onehot`): the sweep that bounds an
intermediate value neuron by neuron must equal the dense sweep with C = rows of the identity."""
import pytest
import torch

from tests.helpers import assert_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available()
    from boundflow_b200.csrc import build

    build.build()
    return torch.device("cuda", 0)


@pytest.mark.parametrize("name,batch", [("c2", 3), ("c3", 5), ("c5", 1)])
def test_onehot_rows_equal_dense_identity(dev, name, batch):
    from boundflow_b200 import workloads as W
    from boundflow_b200.crown import crown_from_trace, ibp_trace
    from boundflow_b200.ir import InputSpec

    wl = W.make_workload(name, batch=batch)
    spec = InputSpec.box(value_name="input", lower=wl.lo.to(dev), upper=wl.up.to(dev))
    trace = ibp_trace(wl.module, spec)
    chain = trace.chain
    for r in range(1, len(chain.relu_input_names)):
        n = chain.relu_widths[r]
        # ragged window that crosses channel / row boundaries and ends at the last neuron
        for first, cnt in ((0, min(7, n)), (max(0, n - 37), min(37, n)), (n // 3, min(50, n - n // 3))):
            eye = torch.eye(n, dtype=torch.float32, device=dev)[first : first + cnt]
            lo_d, up_d = crown_from_trace(trace, eye, output_value=chain.relu_input_names[r])
            lo_o, up_o = crown_from_trace(trace, None, output_value=chain.relu_input_names[r], identity_rows=(first, cnt))
            assert_close(lo_o, lo_d, f"{name} relu {r} rows {first}+{cnt} lower")
            assert_close(up_o, up_d, f"{name} relu {r} rows {first}+{cnt} upper")


def test_onehot_rejects_bad_windows(dev):
    from boundflow_b200 import workloads as W
    from boundflow_b200.crown import crown_from_trace, ibp_trace
    from boundflow_b200.ir import InputSpec

    wl = W.make_workload("c3", batch=2)
    spec = InputSpec.box(value_name="input", lower=wl.lo.to(dev), upper=wl.up.to(dev))
    trace = ibp_trace(wl.module, spec)
    name = trace.chain.relu_input_names[1]
    n = trace.chain.relu_widths[1]
    with pytest.raises(ValueError):
        crown_from_trace(trace, None, output_value=name, identity_rows=(n - 3, 4))
    with pytest.raises(ValueError):
        crown_from_trace(trace, None, output_value=name, identity_rows=(-1, 4))


def test_intermediate_recipe_on_mlp_matches_oracle(dev):
    """The recipe with a Linear layer under every bounded value (weight-row copy as first step)."""
    from boundflow_b200 import workloads as W
    from boundflow_b200.crown import run_crown_intermediate_mlp
    from boundflow_b200.ir import InputSpec
    from oracle import crown_oracle as O

    wl = W.make_workload("c1")
    lo, up, C = wl.lo[:6], wl.up[:6], wl.C[:6]
    spec = InputSpec.box(value_name="input", lower=lo.to(dev), upper=up.to(dev))
    got, pre = run_crown_intermediate_mlp(wl.module, spec, linear_spec_C=C.to(dev), chunk_rows=64)
    ref_l, ref_u, ref_tr = O.crown_with_intermediate_crown(wl.layers, O.box_input(lo, up), C, chunk=64)
    assert_close(got.lower, ref_l, "lower")
    assert_close(got.upper, ref_u, "upper")
    for r, nm in enumerate(wl.relu_names):
        assert_close(pre[nm].lower, ref_tr.pre[r][0], f"pre {nm} lower")
        assert_close(pre[nm].upper, ref_tr.pre[r][1], f"pre {nm} upper")


@pytest.mark.parametrize("n_in", (1, 2, 3, 4, 5, 12, 31, 33, 100, 128, 255, 1020, 1024, 1030))
@pytest.mark.parametrize("B, first, S", [(1, 0, 1), (3, 2, 11), (29, 5, 35)])
def test_identity_rows_of_one_linear_layer(dev, n_in, B, first, S):
    """Rows shorter and longer than the threads that copy them, counts that do not fill a block, and the neighbours of the rows untouched."""
    import ctypes

    from boundflow_b200 import _lib

    lib = _lib.load()
    g = torch.Generator().manual_seed(n_in + S)
    W, b = torch.randn((40, n_in), generator=g), torch.randn((40,), generator=g)
    mid, rad = torch.randn((B, n_in), generator=g), torch.rand((B, n_in), generator=g)
    d = {k: t.to(dev) for k, t in dict(W=W, b=b, mid=mid, rad=rad).items()}
    desc = (_lib.LayerDesc * 1)()
    desc[0].op, desc[0].W, desc[0].bias, desc[0].n_in, desc[0].n_out = _lib.OP_LINEAR, d["W"].data_ptr(), d["b"].data_ptr(), n_in, 40
    chain = ctypes.c_void_p()
    _lib.check(lib.bf_chain_create(desc, 1, ctypes.byref(chain)))
    try:
        nbytes = int(lib.bf_chain_crown_workspace_bytes(chain, B, S, 1))
        ws, out = torch.full((nbytes + 4096,), 0x55, dtype=torch.uint8, device=dev), torch.empty((B, S), device=dev)
        _lib.check(lib.bf_chain_crown_onehot(chain, 1, _lib.SIDE_UPPER, first, None, None, None, None, d["mid"].data_ptr(), d["rad"].data_ptr(), _lib.NORM_BOX, 0.0,
                                             out.data_ptr(), ws.data_ptr(), nbytes, B, S, None))
    finally:
        lib.bf_chain_destroy(chain)
    rows, size = W[first:first + S].double(), mid.double().abs() + rad.double()
    want = mid.double() @ rows.t() + rad.double() @ rows.abs().t() + b[first:first + S].double()
    # 2 n_in products and the bias in any order
    assert ((out.cpu().double() - want).abs() <= (2 * n_in + 2) * 2.0**-24 * (size @ rows.abs().t() + b[first:first + S].double().abs())).all()
    assert (ws[nbytes:] == 0x55).all()
