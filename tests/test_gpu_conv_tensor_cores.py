"""The tensor-core ReLU + transposed convolution against float64 and against the FP32 kernels it takes the place of."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from boundflow_b200.csrc import build

    build.build()
    return torch.device("cuda", 0)


def _pair(v):
    return (v, v) if isinstance(v, int) else v


def _backward(A, w, stride, padding, H, W, *, b=None, slopes=None, side=0, delta=None, accumulate=1):
    """bf_crown_relu_conv2d_bwd on rows [B,S,Co,Ho,Wo]: (rows of the input, tensor-core launches)."""
    from boundflow_b200 import _lib

    lib = _lib.load()
    (sh, sw), (ph, pw) = _pair(stride), _pair(padding)
    B, S, Co, Ho, Wo = A.shape
    Ci, kh, kw = w.shape[1:]
    out = torch.full((B, S, Ci, H, W), float("nan"), device=A.device)
    nbytes = lib.bf_crown_relu_conv2d_bwd_scratch_bytes(B, S, Co, Ho, Wo)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device=A.device)
    au, al, bu = slopes if slopes is not None else (None, None, None)
    before = _lib.tc_launch_count()
    _lib.check(lib.bf_crown_relu_conv2d_bwd(_lib.ptr(A), side, _lib.ptr(au), _lib.ptr(al), _lib.ptr(bu), None, _lib.ptr(w), _lib.ptr(b), _lib.ptr(out),
                                            _lib.ptr(delta), accumulate, _lib.ptr(scratch), nbytes, B, S, Ci, H, W, Co, Ho, Wo, kh, kw, sh, sw, ph, pw, None))
    return out, _lib.tc_launch_count() - before


def _transposed(x, w, stride, padding, H, W):
    (sh, sw), (ph, pw) = _pair(stride), _pair(padding)
    Ho, Wo = x.shape[3:]
    opad = (H - ((Ho - 1) * sh - 2 * ph + w.shape[2]), W - ((Wo - 1) * sw - 2 * pw + w.shape[3]))
    y = torch.nn.functional.conv_transpose2d(x.flatten(0, 1), w, None, (sh, sw), (ph, pw), output_padding=opad)
    return y.view(x.shape[0], x.shape[1], w.shape[1], H, W)


def _rows(dev, kind, B, S, Co, Ho, Wo, Ci, k, g):
    kh, kw = _pair(k)
    A = torch.randn(B, S, Co, Ho, Wo, generator=g, device=dev)
    w = torch.randn(Co, Ci, kh, kw, generator=g, device=dev)
    if kind == "identity":
        A = torch.zeros(B * S, Co * Ho * Wo, device=dev)
        A[torch.arange(B * S), torch.randint(0, A.shape[1], (B * S,), generator=g, device=dev)] = 1.0
        A = A.view(B, S, Co, Ho, Wo)
    elif kind == "integers":
        A = torch.randint(-9, 10, A.shape, generator=g, device=dev).float()
        w = torch.randint(-9, 10, w.shape, generator=g, device=dev).float()
    elif kind == "sparse":
        A = A * (torch.rand(A.shape, generator=g, device=dev) < 0.03)
    return A, w


# accumulators of one and several parts, one and two tiles in tensor memory, several blocks of input channels, channels that end inside a stage
GEOMETRIES = [(8, 40, 8, 9, 9, 16, 3, 1, 1), (8, 64, 32, 32, 32, 32, 4, 2, 1), (8, 64, 32, 16, 16, 64, 3, 1, 1), (16, 100, 16, 14, 14, 32, 4, 2, 1),
              (8, 64, 16, 17, 17, 40, 3, 2, 1), (8, 60, 24, 13, 13, 20, 3, 1, 1), (4, 64, 64, 16, 16, 200, 2, 1, 0)]


# products and sums that float32 represents: any order of exact operations gives them back
@pytest.mark.parametrize("B,S,Ci,H,W,Co,k,s,p", GEOMETRIES)
@pytest.mark.parametrize("kind", ["identity", "integers"])
def test_exact_rows_stay_exact(dev, B, S, Ci, H, W, Co, k, s, p, kind):
    Ho, Wo = (H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1
    g = torch.Generator("cuda").manual_seed(B + Ci + Co)
    A, w = _rows(dev, kind, B, S, Co, Ho, Wo, Ci, k, g)
    out, launches = _backward(A, w, s, p, H, W)
    assert launches == 1
    assert torch.equal(out.double(), _transposed(A.double(), w.double(), s, p, H, W))


# no further from float64 than the FP32 kernels, and without the bias of a systematic scaling: a truncated addition loses half a unit in the
# last place (2^-24) on average, at most six of them in a row
@pytest.mark.parametrize("B,S,Ci,H,W,Co,k,s,p", GEOMETRIES)
@pytest.mark.parametrize("kind", ["dense", "sparse"])
def test_error_against_fp32_kernels(dev, monkeypatch, B, S, Ci, H, W, Co, k, s, p, kind):
    Ho, Wo = (H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1
    g = torch.Generator("cuda").manual_seed(B + Ci + Co + 1)
    A, w = _rows(dev, kind, B, S, Co, Ho, Wo, Ci, k, g)
    ref = _transposed(A.double(), w.double(), s, p, H, W)
    out, launches = _backward(A, w, s, p, H, W)
    monkeypatch.setenv("BF_B200_FORCE_FFMA", "1")
    fp32, none = _backward(A, w, s, p, H, W)
    assert (launches, none) == (1, 0)
    err, err32 = (out.double() - ref), (fp32.double() - ref)
    assert err.norm() <= err32.norm()
    assert abs((err * ref.sign()).sum() / ref.abs().sum()) <= 3 * 2.0**-24


def _network(dev, shape, convs, linears, g):
    """Chain of convs (channels, kernel, stride, padding) and Linear widths with a ReLU after every layer but the last."""
    from boundflow_b200.ir import BFTaskModule, BoundTask, TaskKind, TaskOp

    ops, params, cur = [], {}, "input"
    layers = [("c",) + c for c in convs] + [("f", n) for n in linears]
    for i, (kind, n, *geo) in enumerate(layers):
        out = "out" if i + 1 == len(layers) else f"h{i}"
        if kind == "c":
            k, s, p = geo
            params[f"W{i}"] = torch.randn(n, shape[0], k, k, generator=g, device=dev) * (2.0 / (shape[0] * k * k)) ** 0.5
            ops.append(TaskOp("conv2d", f"conv{i}", [cur, f"W{i}", f"b{i}"], [out], {"stride": (s, s), "padding": (p, p)}))
            shape = (n, (shape[1] + 2 * p - k) // s + 1, (shape[2] + 2 * p - k) // s + 1)
        else:
            if len(shape) == 3:
                ops.append(TaskOp("flatten", "flatten", [cur], ["flat"], {"start_dim": 1, "end_dim": -1}))
                cur, shape = "flat", (shape[0] * shape[1] * shape[2],)
            params[f"W{i}"] = torch.randn(n, shape[0], generator=g, device=dev) * (2.0 / shape[0]) ** 0.5
            ops.append(TaskOp("linear", f"linear{i}", [cur, f"W{i}", f"b{i}"], [out]))
            shape = (n,)
        params[f"b{i}"] = torch.randn(n, generator=g, device=dev) * 0.1
        cur = out
        if i + 1 < len(layers):
            ops.append(TaskOp("relu", f"relu{i}", [cur], [f"r{i}"]))
            cur = f"r{i}"
    task = BoundTask(task_id="t0", kind=TaskKind.INTERVAL_IBP, ops=ops, input_values=["input"], output_values=["out"])
    return BFTaskModule(tasks=[task], entry_task_id="t0", bindings={"params": params})


def _box(x, eps):
    from boundflow_b200.ir import InputSpec

    return InputSpec.box(value_name="input", lower=x - eps, upper=x + eps)


# the status word of an expired wait (set here by the host) takes the bounds of a chain whose only tensor-core kernel is the convolution's:
# 36 rows, too few for the Linear layers' kernels
def test_expired_wait_takes_the_bounds_of_conv_chains(dev):
    from boundflow_b200 import _lib
    from boundflow_b200.crown import adaptive_alpha_from_trace, alpha_crown_from_trace, crown_from_trace, ibp_trace

    g = torch.Generator("cuda").manual_seed(5)
    module = _network(dev, (3, 32, 32), [(16, 3, 1, 1), (16, 3, 1, 1)], [10], g)
    trace = ibp_trace(module, _box(torch.rand(4, 3, 32, 32, generator=g, device=dev), 0.01))
    C = torch.randn(4, 9, 10, generator=g, device=dev)
    before = _lib.tc_launch_count()
    assert torch.isfinite(torch.stack(crown_from_trace(trace, C))).all() and _lib.tc_launch_count() == before + 2
    status = trace.chain._tc_buffer[:4].view(torch.int32)
    status.fill_(1)
    try:
        assert torch.isnan(torch.stack(crown_from_trace(trace, C))).all()
        lower, upper, _alpha, _last, _metric = alpha_crown_from_trace(trace, C, adaptive_alpha_from_trace(trace), steps=2, lr=0.1, spec_reduce="mean", want_upper=True)
        assert torch.isnan(lower).all() and torch.isnan(upper).all()
    finally:
        status.zero_()


# neurons of conv layers as full rows (a ball that no window represents; windows that outgrow a small map; a graph): the bits of the FP32 kernels
@pytest.mark.parametrize("case", ["l2", "outgrown", "graph"])
def test_conv_neuron_rows_stay_on_fp32(dev, monkeypatch, case):
    from boundflow_b200 import _lib
    from boundflow_b200.crown import run_crown_ibp_mlp
    from boundflow_b200.ir import InputSpec, TaskOp

    g = torch.Generator("cuda").manual_seed(6)
    size = 6 if case == "outgrown" else 16
    module = _network(dev, (8, size, size), [(16, 3, 1, 1), (16, 3, 1, 1), (16, 3, 1, 1), (16, 3, 1, 1)], [10], g)
    x = torch.rand(2 if case == "graph" else 4, 8, size, size, generator=g, device=dev)
    if case == "graph":  # h2 + r0: not a chain any more
        ops = module.get_entry_task().ops
        at = next(i for i, o in enumerate(ops) if o.name == "relu2")
        ops[at] = TaskOp("relu", "relu2", ["s2"], ["r2"])
        ops.insert(at, TaskOp("add", "add2", ["h2", "r0"], ["s2"]))
    spec = InputSpec.l2(value_name="input", center=x, eps=0.05) if case == "l2" else _box(x, 0.01)
    before = _lib.tc_launch_count()
    got = run_crown_ibp_mlp(module, spec, output_value="h2")
    assert _lib.tc_launch_count() == before
    monkeypatch.setenv("BF_B200_FORCE_FFMA", "1")
    want = run_crown_ibp_mlp(module, spec, output_value="h2")
    assert torch.equal(got.lower, want.lower) and torch.equal(got.upper, want.upper)


# infinities pass as they do through a sum over the taps that exist: rows whose coefficients or weights are infinite, or round to infinity
@pytest.mark.parametrize("what", ["coefficient", "weight", "largest"])
@pytest.mark.parametrize("B,S,Ci,H,W,Co,k,s,p", [(8, 64, 16, 17, 17, 20, 3, 2, 1), (8, 64, 32, 16, 16, 30, 3, 1, 1)])
def test_infinities(dev, B, S, Ci, H, W, Co, k, s, p, what):
    Ho, Wo = (H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1
    g = torch.Generator("cuda").manual_seed(7)
    A, w = torch.rand(B, S, Co, Ho, Wo, generator=g, device=dev) + 0.5, torch.rand(Co, Ci, k, k, generator=g, device=dev) + 0.5
    big = 3.4028234e38 if what == "largest" else float("inf")
    if what == "weight":
        w[3, 5, 1, 1] = big
    else:
        A[1, 2, 3, 4, 5] = big
        A[1, 3, 4, 0, 0] = -big
        w *= 0.25  # the largest number stays in range behind the weight
    out, launches = _backward(A, w, s, p, H, W)
    assert launches == 1
    # every sum is of positive products (and one infinity): in float64, with the infinities in their place
    ref = _transposed(torch.where(A.isinf(), torch.zeros_like(A), A).double(), torch.where(w.isinf(), torch.zeros_like(w), w).double(), s, p, H, W)
    reach = _transposed(A.isinf().double() * A.sign(), torch.ones_like(w).double(), s, p, H, W)
    reach = reach + _transposed(torch.ones_like(A).double(), w.isinf().double(), s, p, H, W)
    ref = torch.where(reach > 0, torch.full_like(ref, float("inf")), torch.where(reach < 0, torch.full_like(ref, -float("inf")), ref))
    assert torch.equal(out.isinf(), ref.isinf()) and not out.isnan().any()
    assert torch.equal(out[ref.isinf()].double(), ref[ref.isinf()])
    # a sum of n = Co k^2 positive products (one of them minus the largest number): at most (n + 8) 2^-24 of the sum of magnitudes
    mag = _transposed(torch.where(A.isinf(), torch.zeros_like(A), A).double().abs(), torch.where(w.isinf(), torch.zeros_like(w), w).double(), s, p, H, W)
    ok = ~ref.isinf()
    assert ((out.double() - ref)[ok].abs() <= ((Co * k * k + 8) * 2.0**-24 * mag)[ok]).all()


@pytest.mark.parametrize("B,Ci,H,W,Co,k,s,p", [(3, 3, 9, 11, 17, 3, 1, 1), (2, 4, 12, 12, 40, 4, 2, 1), (5, 1, 8, 8, 5, 3, 1, 2)])
def test_infinite_weight_at_the_border_of_forward_convolutions(dev, B, Ci, H, W, Co, k, s, p):
    from boundflow_b200 import _lib

    lib = _lib.load()
    Ho, Wo = (H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1
    g = torch.Generator("cuda").manual_seed(8)
    x = torch.rand(B, Ci, H, W, generator=g, device=dev) + 0.5
    w = torch.rand(Co, Ci, k, k, generator=g, device=dev)
    w[1, 0, 0, 0] = float("inf")
    # channel 1: infinite where kernel position (0, 0) lies inside the image
    rows, cols = torch.arange(Ho, device=dev) * s - p >= 0, torch.arange(Wo, device=dev) * s - p >= 0
    hit = torch.zeros(B, Co, Ho, Wo, dtype=torch.bool, device=dev)
    hit[:, 1] = rows[:, None] & cols[None]
    out = torch.full((B, Co, Ho, Wo), float("nan"), device=dev)
    _lib.check(lib.bf_rows_conv2d_fwd(x.data_ptr(), w.data_ptr(), None, out.data_ptr(), B, Ci, H, W, Co, Ho, Wo, k, k, s, s, p, p, None))
    assert torch.equal(out == float("inf"), hit) and torch.isfinite(out[~hit]).all()
    lo, up = (torch.full((B, Co, Ho, Wo), float("nan"), device=dev) for _ in range(2))
    _lib.check(lib.bf_ibp_conv2d(x.data_ptr(), (x * 0).data_ptr(), _lib.IN_MID_RAD, 0, w.abs().data_ptr(), None, None, 0, None, None, lo.data_ptr(), up.data_ptr(),
                                 None, B, Ci, H, W, Co, k, k, s, s, p, p, None))
    assert torch.isfinite(lo[~hit]).all() and torch.isfinite(up[~hit]).all()


# a negative padding (a cropped input) reaches no output near the border: zeros there, from the FP32 kernels
def test_negative_padding(dev):
    B, S, Ci, H, W, Co, k = 8, 64, 16, 16, 17, 24, 3
    g = torch.Generator("cuda").manual_seed(11)
    A, w = _rows(dev, "integers", B, S, Co, H - 4, W - 4, Ci, k, g)
    out, _ = _backward(A, w, 1, -1, H, W)
    want = torch.nn.functional.pad(_transposed(A.double(), w.double(), 1, 0, H - 2, W - 2), (1, 1, 1, 1))
    assert torch.equal(out.double(), want)


# the dispatch's two sides: layers that were measured faster on the tensor cores, and slower
@pytest.mark.parametrize("M,Ci,H,Co,k,s,p,takes", [(512, 32, 32, 32, 4, 2, 1, 1), (512, 32, 16, 64, 3, 1, 1, 1), (512, 32, 8, 64, 2, 1, 0, 1), (40, 32, 8, 64, 3, 1, 1, 0),
                                                   (945, 8, 16, 16, 3, 1, 1, 0), (261, 16, 32, 16, 3, 1, 1, 0), (261, 128, 32, 128, 3, 1, 1, 0), (1197, 8, 16, 16, 1, 1, 0, 0),
                                                   (1062, 8, 32, 8, 4, 2, 1, 0), (512, 4, 32, 32, 4, 2, 1, 0), (300, 16, 16, 32, 5, 1, 2, 0)])
def test_dispatch(dev, M, Ci, H, Co, k, s, p, takes):
    Ho = (H + 2 * p - k) // s + 1
    g = torch.Generator("cuda").manual_seed(12)
    A, w = _rows(dev, "integers", M, 1, Co, Ho, Ho, Ci, k, g)
    out, launches = _backward(A, w, s, p, H, H)
    assert launches == takes
    # whole numbers below 2^24: both kernels are exact
    assert torch.equal(out[:16].double(), _transposed(A[:16].double(), w.double(), s, p, H, H))


# kernels of one tap and of unequal sides, strides and paddings; with and without bias, row sums, a value to add them to, slopes
@pytest.mark.parametrize("B,S,Ci,H,W,Co,k,s,p", [(8, 40, 48, 12, 13, 24, (1, 1), (1, 1), (0, 0)), (8, 40, 16, 15, 14, 32, (3, 2), (2, 1), (1, 0)),
                                                 (8, 40, 32, 14, 15, 20, (2, 3), (1, 2), (0, 1)), (6, 50, 16, 16, 16, 32, (2, 2), (2, 2), (0, 0))])
@pytest.mark.parametrize("relu,bias,sums,accumulate", [(True, True, True, 0), (False, True, True, 0), (True, False, True, 1), (True, False, True, 0),
                                                       (False, False, True, 0), (False, False, True, 1), (True, True, False, 1)])
def test_forms_of_the_call(dev, B, S, Ci, H, W, Co, k, s, p, relu, bias, sums, accumulate):
    Ho, Wo = (H + 2 * p[0] - k[0]) // s[0] + 1, (W + 2 * p[1] - k[1]) // s[1] + 1
    g = torch.Generator("cuda").manual_seed(9)
    A, w = _rows(dev, "dense", B, S, Co, Ho, Wo, Ci, k, g)
    b = torch.randn(Co, generator=g, device=dev) if bias else None
    slopes = tuple(torch.rand(B, Co, Ho, Wo, generator=g, device=dev) for _ in range(3)) if relu else None
    delta = torch.full((B, S), 2.0, device=dev) if sums else None
    out, launches = _backward(A, w, s, p, H, W, b=b, slopes=slopes, side=1, delta=delta, accumulate=accumulate)
    assert launches == 1
    lam, icpt = A.double(), torch.zeros_like(A, dtype=torch.float64)
    if relu:
        au, al, bu = (t.double()[:, None] for t in slopes)
        icpt = torch.where(A >= 0, lam * bu, icpt)
        lam = lam * torch.where(A >= 0, au, al)
    # operands are exact; the sums keep the bound of an FP32 sum of Co k^2 / s^2 products
    tol = (Co * k[0] * k[1] / (s[0] * s[1]) + 8) * 2.0**-24 * _transposed(lam.abs(), w.double().abs(), s, p, H, W) + 1e-6
    assert ((out.double() - _transposed(lam, w.double(), s, p, H, W)).abs() <= tol).all()
    if sums:
        term = lam * (b.double()[:, None, None] if bias else 0.0)
        start = 2.0 if accumulate else 0.0
        tol = (2 * Co * Ho * Wo + 8) * 2.0**-24 * (start + (icpt.abs() + term.abs()).sum((2, 3, 4)))
        assert ((delta.double() - (start + (icpt + term).sum((2, 3, 4)))).abs() <= tol).all()


# the term behind a conv ReLU (beta-CROWN's splits enter there) in the tensor-core kernel, against float64
def test_term_behind_a_conv_relu(dev):
    from boundflow_b200 import _lib
    from boundflow_b200.crown import crown_from_trace, ibp_trace

    g = torch.Generator("cuda").manual_seed(10)
    module = _network(dev, (3, 32, 32), [(16, 3, 1, 1), (32, 3, 1, 1)], [10], g)
    trace = ibp_trace(module, _box(torch.rand(4, 3, 32, 32, generator=g, device=dev), 0.01))
    C = torch.randn(4, 9, 10, generator=g, device=dev)
    add = torch.randn(4, 32 * 32 * 32, generator=g, device=dev)
    before = _lib.tc_launch_count()
    got, _ = crown_from_trace(trace, C, sides=(_lib.SIDE_LOWER,), relu_pre_add_coeff_l={"h1": add})
    assert _lib.tc_launch_count() == before + 1
    P = {n: t.double() for n, t in module.bindings["params"].items()}

    def relu_back(A, r):
        l, u = trace.pre_l[r].double()[:, None], trace.pre_u[r].double()[:, None]
        off, on = u <= 0, l >= 0
        up = torch.where(off, 0.0, torch.where(on, 1.0, u / (u - l)))
        shift = torch.where(off | on, 0.0, -u * l / (u - l))
        low = on.double()
        return torch.where(A >= 0, A * low, A * up), torch.where(A >= 0, 0.0, A * shift).sum(-1)

    def conv_back(A, name, co):
        return torch.nn.functional.conv_transpose2d(A.view(36, co, 32, 32), P["W" + name], None, 1, 1).view(4, 9, -1), A.view(4, 9, co, -1).sum(-1) @ P["b" + name]

    def bound(add, A=C.double()):
        A, c = A @ P["W2"], A @ P["b2"]
        A, d = relu_back(A, 1)
        A, e = conv_back(A + add, "1", 32)
        A, f = relu_back(A, 0)
        A, h = conv_back(A, "0", 16)
        return c + d + e + f + h + (A * trace.mid.double()[:, None]).sum(-1) - (A.abs() * trace.rad.double()[:, None]).sum(-1)

    want = bound(add.double()[:, None])
    # three layers of float32 sums: 2-norm error of a few 2^-24, against a term that is most of the bound
    assert (got.double() - want).norm() <= 64 * 2.0**-24 * want.norm() <= 1e-3 * (bound(0.0) - want).norm()
