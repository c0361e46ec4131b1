"""Whole-query entry points of the CUDA backend (IBP trace, CROWN, alpha-CROWN).

Same names, argument meaning and error behaviour as the reference's solver
stack so that callers (the BaB driver, benchmarks, tests) switch by import:

  forward_ibp_trace_mlp                 <- _forward_ibp_trace_mlp            runtime/crown_ibp.py:101-342
  run_crown_ibp_mlp                     <- run_crown_ibp_mlp                 runtime/crown_ibp.py:2054-2133
  run_crown_ibp_mlp_from_forward_trace  <- same name                         runtime/crown_ibp.py:2136-2230
  run_crown_ibp_mlp_with_relu_influence_from_forward_trace <- same name      runtime/crown_ibp.py:2201-2240
  get_crown_ibp_mlp_stats               <- same name                         runtime/crown_ibp.py:2279-2349
  run_alpha_crown_mlp                   <- same name                         runtime/alpha_crown.py:137-261
  run_alpha_beta_crown_mlp              <- same name                         runtime/alpha_beta_crown.py:643-941
  check_first_layer_infeasible_split    <- same name                         runtime/alpha_beta_crown.py:109-142
  first_layer_certificate               <- _is_infeasible_split_first_layer_convex_combo, per domain
                                                                             runtime/alpha_beta_crown.py:391-532
  run_crown_intermediate_mlp            <- the layer-by-layer refinement recipe of
                                           runtime/native_intermediate_refinement.py:923-988

All arithmetic happens in libbf_b200.so; torch only owns the device buffers and
the stream.  Tensors given on the CPU are copied to the current CUDA device and
results are returned on the device the inputs came from.
"""
from __future__ import annotations

from dataclasses import dataclass, field
from typing import Any, Dict, List, Mapping, Optional, Sequence, Tuple

import torch

from . import _lib
from .ir import IntervalState, input_mid_rad, lp_ball_of, normalize_input_spec
from .network import CudaChain, compile_chain


@dataclass
class AlphaState:
    alpha_by_relu_input: Dict[str, torch.Tensor] = field(default_factory=dict)


@dataclass
class BetaState:
    beta_by_relu_input: Dict[str, torch.Tensor] = field(default_factory=dict)


@dataclass
class AlphaCrownStats:
    steps: int
    lr: float
    objective: str
    spec_reduce: str
    relu_inputs: Tuple[str, ...]
    feasibility: str = "unknown"
    reason: str = "ok"
    infeasible_domains: Optional[torch.Tensor] = None


@dataclass
class AlphaBetaCrownStats:
    """Result of `check_first_layer_infeasible_split` (AlphaBetaCrownStats, alpha_beta_crown.py:64-76)."""

    feasibility: str
    reason: str = ""
    alpha_stats: Optional[Any] = None
    infeasible_certificate: Optional[Dict[str, Any]] = None
    branch_choices: Optional[List[Optional[Tuple[str, int]]]] = None


@dataclass
class CrownIbpStats:
    """Result of `get_crown_ibp_mlp_stats` (crown_ibp.py:63-67)."""

    supported: bool
    reason: str = ""
    ops_seen: Tuple[str, ...] = ()


def _cuda_device(t: torch.Tensor) -> torch.device:
    if t.device.type == "cuda":
        return t.device
    if not torch.cuda.is_available():
        raise RuntimeError("boundflow_b200 needs a CUDA device (no CPU fallback exists)")
    return torch.device("cuda", torch.cuda.current_device())


def _f32(t: torch.Tensor, device: torch.device) -> torch.Tensor:
    return t.detach().to(device=device, dtype=torch.float32, non_blocking=True).contiguous()


def _stream_ptr(device: torch.device) -> int:
    """Handle of the current stream (`torch.cuda.current_stream(device).cuda_stream` without the Stream object)."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if device.index is None else device.index)


class _Workspace:
    """One growing device buffer per (device, stream): sized by the library's
    *_workspace_bytes queries, reused across calls."""

    _pool: Dict[Tuple[int, int], torch.Tensor] = {}

    @classmethod
    def get(cls, device: torch.device, nbytes: int) -> torch.Tensor:
        key = (device.index or 0, _stream_ptr(device))
        buf = cls._pool.get(key)
        if buf is None or buf.numel() < nbytes:
            cls._pool.pop(key, None)
            buf = torch.empty(max(int(nbytes), 1 << 20), dtype=torch.uint8, device=device)
            cls._pool[key] = buf
        return buf


@dataclass
class ForwardTrace:
    """Device-side result of one IBP sweep."""

    chain: CudaChain
    mid: torch.Tensor           # [B, n0]
    rad: torch.Tensor           # [B, n0]
    pre_l: List[torch.Tensor]   # per ReLU [B, n_r]
    pre_u: List[torch.Tensor]
    out_l: torch.Tensor         # [B, n_out]
    out_u: torch.Tensor
    infeasible: torch.Tensor    # int32 [B]
    B: int
    norm_p: int = 0             # _lib.NORM_BOX, or NORM_L1 / NORM_L2 for an Lp-ball input (then mid = centre, rad unused)
    eps: float = 0.0
    clamped: bool = True        # a split or a constraint was applied; without one no domain can be infeasible


def _prepare_input(module: Any, input_spec: Any, batch: Optional[int] = None):
    """`batch`: number of domains when the input set is given once (leading dimension 1) for all of them, as in a
    batch of ReLU-split subdomains of one input; the row is then repeated on the device, not uploaded B times."""
    spec = normalize_input_spec(input_spec)
    center = spec.center
    device = _cuda_device(center)
    chain = compile_chain(module, tuple(int(d) for d in center.shape[1:]), device)
    B = int(center.shape[0])
    repeat = batch is not None and int(batch) > 1 and B == 1
    ball = lp_ball_of(spec)
    if ball is not None:  # L1 / L2 ball: centre + eps; the radius tensor is only used by a conv first layer (bounding box)
        mid = _f32(center, device).reshape(B, -1)
        rad = torch.full_like(mid, float(ball[1]))
    else:
        mid, rad, _lo, _up = input_mid_rad(spec)
        mid = _f32(mid, device).reshape(B, -1)
        rad = _f32(rad, device).reshape(B, -1)
    if repeat:
        B = int(batch)
        mid = mid.expand(B, -1).contiguous()
        rad = rad.expand(B, -1).contiguous()
    return spec, chain, device, B, mid, rad, center.device


def _plain_set(spec: Any):
    """(lower, upper, 0.0) of a box or (centre, None, eps) of an L-inf ball whose tensors the library can read where they are (CUDA, fp32,
    contiguous), else None: the input sets of the calls that bound a whole query in the library."""
    pert = spec.perturbation
    if hasattr(pert, "lower") and hasattr(pert, "upper"):
        a, b, eps = pert.lower, pert.upper, 0.0
    elif hasattr(pert, "eps") and (pert.norm() if hasattr(pert, "norm") else pert._normalize_p()) == "inf":
        a, b, eps = spec.center, None, float(pert.eps)
    else:
        return None
    for t in (a, b):
        if t is not None and not (t.is_cuda and t.dtype == torch.float32 and t.is_contiguous()):
            return None
    if b is not None and (b.shape != a.shape or b.device != a.device or a.shape != spec.center.shape or spec.center.device != a.device):
        return None
    return a, b, eps


def _split_tensor(raw: Any, B: int, n: int, device: torch.device, name: str):
    """int8 [B,n] or [1,n] view of a split assignment; shapes as the reference
    accepts them (runtime/relu_shape_utils.py:82-115)."""
    s = raw if torch.is_tensor(raw) else torch.as_tensor(raw)
    if s.dtype not in (torch.int8, torch.int16, torch.int32, torch.int64):
        raise TypeError(f"relu split for {name} must be integer tensor, got dtype={s.dtype}")
    s = s.to(device=device, dtype=torch.int8)
    if s.numel() == 1:
        s = s.reshape(1, 1).expand(1, n)
    elif s.numel() == n:
        s = s.reshape(1, n)
    elif s.numel() == B * n and int(s.shape[0]) == B:
        s = s.reshape(B, n)
    else:
        raise ValueError(f"relu_split_state[{name}] shape {tuple(s.shape)} cannot broadcast to [{B},{n}]")
    s = s.contiguous()
    return s, (n if int(s.shape[0]) == B else 0)


def ibp_trace(
    module: Any,
    input_spec: Any,
    *,
    relu_split_state: Optional[Mapping[str, torch.Tensor]] = None,
    relu_pre_constraints: Optional[Mapping[str, Any]] = None,
    batch: Optional[int] = None,
) -> ForwardTrace:
    """Run the IBP sweep on the device and keep everything there.  `batch`: see `_prepare_input`."""
    _spec, chain, device, B, mid, rad, _ = _prepare_input(module, input_spec, batch)
    lib = chain.lib
    R = len(chain.relu_layer_ids)
    pre_l = [torch.empty(B, n, dtype=torch.float32, device=device) for n in chain.relu_widths]
    pre_u = [torch.empty(B, n, dtype=torch.float32, device=device) for n in chain.relu_widths]
    n_out = 1
    for d in chain.output_shape:
        n_out *= int(d)
    out_l = torch.empty(B, n_out, dtype=torch.float32, device=device)
    out_u = torch.empty(B, n_out, dtype=torch.float32, device=device)
    infeasible = torch.zeros(B, dtype=torch.int32, device=device)
    splits: List[Optional[torch.Tensor]] = [None] * R
    strides = [0] * R
    if relu_split_state:
        for r, name in enumerate(chain.relu_input_names):
            if name in relu_split_state:
                splits[r], strides[r] = _split_tensor(relu_split_state[name], B, chain.relu_widths[r], device, name)
    cons_l: Optional[List[Optional[torch.Tensor]]] = None
    cons_u: Optional[List[Optional[torch.Tensor]]] = None
    if relu_pre_constraints is not None:
        if tuple(relu_pre_constraints) != tuple(chain.relu_input_names):
            raise ValueError("ReLU pre-activation constraint identities differ")
        cons_l, cons_u = [], []
        for r, name in enumerate(chain.relu_input_names):
            c = relu_pre_constraints[name]
            if tuple(c.lower.shape[1:]) != tuple(chain.relu_shapes[r]) or int(c.lower.shape[0]) != B:
                raise ValueError(f"ReLU pre-activation constraint schema differs for {name}")
            cons_l.append(_f32(c.lower, device).reshape(B, -1))
            cons_u.append(_f32(c.upper, device).reshape(B, -1))
    scratch = torch.empty(4 * (B * chain.max_width + 64), dtype=torch.float32, device=device)
    ball = lp_ball_of(_spec)
    in_b, in_mode, row_dev = rad, _lib.IN_MID_RAD, None
    first = next((l for l in chain.layers if l.op != "flatten"), None)
    if ball is not None and first is not None and first.op == "linear":
        # first Linear layer on an L1/L2 ball: deviation eps * ||W_row||_q (perturbation.py:102-134)
        W1 = first.W
        row_dev = torch.empty(int(W1.shape[0]), dtype=torch.float32, device=device)
        _lib.check(lib.bf_row_dual_norms(_lib.ptr(W1), int(W1.shape[0]), int(W1.shape[1]), ball[0], float(ball[1]), _lib.ptr(row_dev), _stream_ptr(device)))
        in_b, in_mode = row_dev, _lib.IN_CENTER_DEV
    _lib.check(
        lib.bf_chain_ibp(
            chain.interval_handle, _lib.ptr(mid), _lib.ptr(in_b), in_mode,
            _lib.ptr_array(splits), _lib.int_array(strides),
            _lib.ptr_array(cons_l), _lib.ptr_array(cons_u),
            _lib.ptr_array(pre_l), _lib.ptr_array(pre_u),
            _lib.ptr(out_l), _lib.ptr(out_u), _lib.ptr(infeasible),
            _lib.ptr(scratch), scratch.numel() * 4, B, _stream_ptr(device),
        )
    )
    # keep the temporaries alive until the stream has consumed them
    trace = ForwardTrace(chain=chain, mid=mid, rad=rad, pre_l=pre_l, pre_u=pre_u, out_l=out_l, out_u=out_u, infeasible=infeasible, B=B,
                         norm_p=(ball[0] if ball is not None else _lib.NORM_BOX), eps=(ball[1] if ball is not None else 0.0),
                         clamped=cons_l is not None or any(t is not None for t in splits))
    trace._keep = (splits, cons_l, cons_u, scratch, row_dev)  # type: ignore[attr-defined]
    return trace


def _raise_if_infeasible(trace: ForwardTrace, what: str) -> None:
    # Only splits and constraints raise the flag: without them there is nothing to wait for (a read in the middle of a query
    # leaves the GPU idle until the host has launched again, a fifth of a query on a small network: 218 -> 178 us).
    if trace.clamped and bool(trace.infeasible.any().item()):
        bad = torch.nonzero(trace.infeasible).flatten().tolist()
        raise ValueError(f"infeasible {what}: lower>upper after applying split/constraint (domains {bad[:8]}{'...' if len(bad) > 8 else ''})")


def forward_ibp_trace_mlp(
    module: Any,
    input_spec: Any,
    *,
    relu_split_state: Optional[Mapping[str, torch.Tensor]] = None,
    relu_pre_constraints: Optional[Mapping[str, Any]] = None,
) -> Tuple[Dict[str, IntervalState], Dict[str, IntervalState]]:
    """Reference-shaped result: (interval_env, relu_pre) keyed by value name.

    Raises ValueError when any domain's split or constraint is infeasible, as
    the reference does (crown_ibp.py:92-95, 205-208).  Graphs that are not chains go through `dag.forward_ibp_dag`."""
    if needs_graph_path(module):
        return _graph_trace_to_env(module, input_spec, relu_split_state, relu_pre_constraints)
    trace = ibp_trace(module, input_spec, relu_split_state=relu_split_state, relu_pre_constraints=relu_pre_constraints)
    _raise_if_infeasible(trace, "relu split")
    return _trace_to_env(trace, normalize_input_spec(input_spec).center.device)


def _graph_trace_to_env(module: Any, input_spec: Any, relu_split_state, relu_pre_constraints):
    """(interval_env, relu_pre) of a graph that is not a chain: every value of the graph, shaped like the value."""
    from .dag import forward_ibp_dag

    tr = forward_ibp_dag(module, input_spec, relu_split_state, relu_pre_constraints)
    if int(tr.infeasible.sum()) != 0:
        raise ValueError("infeasible relu split: lower > upper")
    dev = normalize_input_spec(input_spec).center.device
    params = module.bindings.get("params", {})
    env: Dict[str, IntervalState] = {}
    for name, lo in tr.lower.items():
        if name in params:
            continue
        shape = (tr.B,) + tuple(tr.shape[name])
        env[name] = IntervalState(lower=lo.reshape(shape).to(dev), upper=tr.upper[name].reshape(shape).to(dev))
    relu_pre = {x: IntervalState(lower=tr.pre_l[x].reshape((tr.B,) + tuple(tr.shape[x])).to(dev),
                                 upper=tr.pre_u[x].reshape((tr.B,) + tuple(tr.shape[x])).to(dev)) for x in dict.fromkeys(tr.relu_inputs)}
    env["__trace__"] = tr  # type: ignore[assignment]
    return env, relu_pre


def _graph_trace_from_env(module: Any, input_spec: Any, interval_env: Mapping[str, Any], relu_pre: Mapping[str, Any]):
    """The device trace of a graph for a backward-only call: the one `forward_ibp_trace_mlp` left in `interval_env` when
    its ReLU bounds are still the caller's, else a fresh interval pass whose ReLU bounds are replaced by `relu_pre`."""
    from .dag import DagTrace, forward_ibp_dag

    spec = normalize_input_spec(input_spec)
    B = int(spec.center.shape[0])
    tr = interval_env.get("__trace__") if isinstance(interval_env, Mapping) else None
    if isinstance(tr, DagTrace) and tr.B == B and set(relu_pre) == set(tr.pre_l) and all(
            relu_pre[x].lower.data_ptr() == tr.pre_l[x].data_ptr() for x in tr.pre_l):
        return tr
    tr = forward_ibp_dag(module, spec)
    device = tr.mid.device
    for x in dict.fromkeys(tr.relu_inputs):
        if x not in relu_pre:
            raise KeyError(f"missing relu pre-activation bounds for value: {x}")
        tr.pre_l[x] = _f32(relu_pre[x].lower, device).reshape(B, -1).contiguous()
        tr.pre_u[x] = _f32(relu_pre[x].upper, device).reshape(B, -1).contiguous()
    return tr


def _trace_to_env(trace: ForwardTrace, out_device: torch.device):
    chain = trace.chain
    relu_pre: Dict[str, IntervalState] = {}
    env: Dict[str, IntervalState] = {}
    for r, name in enumerate(chain.relu_input_names):
        shape = (trace.B,) + tuple(chain.relu_shapes[r])
        st = IntervalState(lower=trace.pre_l[r].reshape(shape).to(out_device), upper=trace.pre_u[r].reshape(shape).to(out_device))
        relu_pre[name] = st
        env[name] = st
    oshape = (trace.B,) + tuple(chain.output_shape)
    env[chain.output_name] = IntervalState(lower=trace.out_l.reshape(oshape).to(out_device), upper=trace.out_u.reshape(oshape).to(out_device))
    env["__trace__"] = trace  # type: ignore[assignment]
    return env, relu_pre


def _trace_from_env(module: Any, input_spec: Any, interval_env: Mapping[str, Any], relu_pre: Mapping[str, Any]) -> ForwardTrace:
    """Recover (or rebuild from tensors) the device trace for a backward-only call."""
    tr = interval_env.get("__trace__") if isinstance(interval_env, Mapping) else None
    _spec, chain, device, B, mid, rad, _ = _prepare_input(module, input_spec)
    if isinstance(tr, ForwardTrace) and tr.chain is chain and tr.B == B:
        same = all(
            relu_pre[n].lower.data_ptr() == tr.pre_l[r].data_ptr() for r, n in enumerate(chain.relu_input_names) if n in relu_pre
        )
        if same:
            return tr
    pre_l, pre_u = [], []
    for r, name in enumerate(chain.relu_input_names):
        if name not in relu_pre:
            raise KeyError(f"missing relu pre-activation bounds for value: {name}")
        pre_l.append(_f32(relu_pre[name].lower, device).reshape(B, -1))
        pre_u.append(_f32(relu_pre[name].upper, device).reshape(B, -1))
    z = torch.zeros(B, 1, dtype=torch.float32, device=device)
    ball = lp_ball_of(_spec)
    return ForwardTrace(chain=chain, mid=mid, rad=rad, pre_l=pre_l, pre_u=pre_u, out_l=z, out_u=z, infeasible=torch.zeros(B, dtype=torch.int32, device=device), B=B,
                        norm_p=(ball[0] if ball is not None else _lib.NORM_BOX), eps=(ball[1] if ball is not None else 0.0))


def _expand_spec(C: Optional[torch.Tensor], B: int, out_dim: int, device: torch.device) -> torch.Tensor:
    """[B,S,O] contiguous spec rows; None = identity, [S,O] is shared (crown_ibp.py:672-719)."""
    if C is None:
        return torch.eye(out_dim, dtype=torch.float32, device=device).unsqueeze(0).expand(B, out_dim, out_dim).contiguous()
    C = C if torch.is_tensor(C) else torch.as_tensor(C)
    C = C.detach().to(device=device, dtype=torch.float32)
    if C.dim() == 2:
        if int(C.shape[1]) != out_dim:
            raise ValueError(f"linear_spec_C shape mismatch: C={tuple(C.shape)} out=({B}, {out_dim})")
        C = C.unsqueeze(0).expand(B, C.shape[0], out_dim)
    if C.dim() != 3:
        raise ValueError(f"linear_spec_C expects rank-3 [B,S,O], got {tuple(C.shape)}")
    if int(C.shape[0]) == 1 and B > 1 and int(C.shape[2]) == out_dim:
        C = C.expand(B, C.shape[1], out_dim)  # one spec block shared by every domain: repeated on the device
    if int(C.shape[0]) != B or int(C.shape[2]) != out_dim:
        raise ValueError(f"linear_spec_C shape mismatch: C={tuple(C.shape)} out=({B}, {out_dim})")
    return C.contiguous()


def _alpha_rows(raw: Any, B: int, n: int, device: torch.device, name: str) -> Tuple[torch.Tensor, int]:
    """alpha as [B,n] (stride n) or [1,n] (stride 0), shapes as crown_ibp.py:940-1001 accepts."""
    a = raw if torch.is_tensor(raw) else torch.as_tensor(raw)
    if not torch.is_floating_point(a):
        raise TypeError(f"relu_alpha[{name}] must be floating, got dtype={a.dtype}")
    a = a.detach().to(device=device, dtype=torch.float32)
    if a.numel() == 1:
        return a.reshape(1, 1).expand(1, n).contiguous(), 0
    if a.numel() == n:
        return a.reshape(1, n).contiguous(), 0
    if a.numel() == B * n and int(a.shape[0]) == B:
        return a.reshape(B, n).contiguous(), n
    raise ValueError(f"relu_alpha[{name}] shape {tuple(a.shape)} cannot broadcast to [{B},{n}]")


def _relaxations(trace: ForwardTrace, relu_alpha: Optional[Mapping[str, torch.Tensor]], n_relu: int):
    chain, B, device = trace.chain, trace.B, trace.mid.device
    widths = chain.relu_widths[:n_relu]
    alpha: List[Optional[torch.Tensor]] = [None] * n_relu
    strides = [0] * n_relu
    if relu_alpha is not None:
        for r, (n, name) in enumerate(zip(widths, chain.relu_input_names)):
            if name in relu_alpha:
                alpha[r], strides[r] = _alpha_rows(relu_alpha[name], B, n, device, name)
    au, bu, al = relax_all(chain.lib, trace.pre_l[:n_relu], trace.pre_u[:n_relu], alpha, strides, widths, B, device)
    return au, bu, al, alpha


def relax_all(lib, pre_l, pre_u, alpha, strides, widths, B: int, device: torch.device):
    """Slopes and intercepts (upper slope, upper intercept, lower slope) of several ReLUs in one launch, [B, n_r] each."""
    pitch = [(B * n + 63) // 64 * 64 for n in widths]  # every table starts on a 256-byte boundary
    slab = torch.empty(3 * sum(pitch), dtype=torch.float32, device=device)
    tables, at = [], 0
    for _ in range(3):
        row = []
        for n, p in zip(widths, pitch):
            row.append(slab.as_strided((B, n), (n, 1), at))
            at += p
        tables.append(row)
    au, bu, al = tables
    R = len(widths)
    _lib.check(lib.bf_relu_relax_many(_lib.ptr_array(pre_l), _lib.ptr_array(pre_u), _lib.ptr_array(alpha), _lib.int_array(strides), _lib.ptr_array(au),
                                      _lib.ptr_array(bu), _lib.ptr_array(al), _lib.int_array(widths), R, B, _stream_ptr(device)))
    return au, bu, al


def crown_from_trace(
    trace: ForwardTrace,
    linear_spec_C: Optional[torch.Tensor],
    *,
    output_value: Optional[str] = None,
    relu_alpha: Optional[Mapping[str, torch.Tensor]] = None,
    relu_pre_add_coeff_l: Optional[Mapping[str, torch.Tensor]] = None,
    sides: Sequence[int] = (_lib.SIDE_LOWER, _lib.SIDE_UPPER),
    identity_rows: Optional[Tuple[int, int]] = None,
    relu_pre_add_coeff_u: Optional[Mapping[str, torch.Tensor]] = None,
    influence_out: Optional[List[torch.Tensor]] = None,
) -> Tuple[Optional[torch.Tensor], Optional[torch.Tensor]]:
    """Backward sweep(s) on the device; returns (lower, upper) [B,S] CUDA tensors.
    `identity_rows=(first, count)` stands for the spec whose rows are rows first..first+count-1 of
    the identity (neuron-wise bounds of `output_value`); no spec tensor is built for it.
    `influence_out` (an empty list) receives, per ReLU below the bounded value, the objective
    influence max over the swept sides and the spec rows of |A| [B,n_r] (crown_ibp.py:1810-1834)."""
    chain, B, device = trace.chain, trace.B, trace.mid.device
    upto = chain.layers_upto(output_value)
    out_shape = chain.layers[upto - 1].out_shape
    out_dim = 1
    for d in out_shape:
        out_dim *= int(d)
    if identity_rows is not None:
        first, S = int(identity_rows[0]), int(identity_rows[1])
        if first < 0 or S <= 0 or first + S > out_dim:
            raise ValueError(f"identity_rows {identity_rows} outside the value's {out_dim} neurons")
        C = None
    else:
        C = _expand_spec(linear_spec_C, B, out_dim, device)
        S = int(C.shape[1])
    n_relu = sum(1 for i in chain.relu_layer_ids if i < upto)
    au, bu, al, keep = _relaxations(trace, relu_alpha, n_relu)
    def add_terms(raw):
        """Per ReLU the term added to one side's coefficients behind it ([B,n] or one shared row), or None."""
        if not raw:
            return None
        terms = [None] * n_relu
        for r in range(n_relu):
            name = chain.relu_input_names[r]
            if name in raw and raw[name] is not None:
                t = raw[name].detach().to(device=device, dtype=torch.float32)
                n = chain.relu_widths[r]
                terms[r] = (t.reshape(1, n).expand(B, n) if t.numel() == n else t.reshape(B, n)).contiguous()
        return terms

    add_by_side = {_lib.SIDE_LOWER: add_terms(relu_pre_add_coeff_l), _lib.SIDE_UPPER: add_terms(relu_pre_add_coeff_u)}
    nbytes = int(chain.lib.bf_chain_crown_workspace_bytes(chain.size_handle, B, S, upto))
    ws = _Workspace.get(device, nbytes)
    outs: List[Optional[torch.Tensor]] = [None, None]
    infl = None
    if influence_out is not None:
        if C is None:
            raise NotImplementedError("objective influence needs a spec tensor")
        infl = [torch.zeros(B, chain.relu_widths[r], dtype=torch.float32, device=device) for r in range(n_relu)]
        influence_out.extend(infl)
    for side in sides:
        out = torch.empty(B, S, dtype=torch.float32, device=device)
        tail = (
            _lib.ptr_array(au), _lib.ptr_array(bu), _lib.ptr_array(al), _lib.ptr_array(add_by_side[side]),
            _lib.ptr(trace.mid), _lib.ptr(trace.rad) if trace.norm_p == _lib.NORM_BOX else None, int(trace.norm_p), float(trace.eps),
            _lib.ptr(out), _lib.ptr(ws), ws.numel(), B, S, _stream_ptr(device),
        )
        if C is None:
            _lib.check(chain.lib.bf_chain_crown_onehot(chain.handle, upto, side, first, *tail))
        elif infl is not None:
            _lib.check(chain.lib.bf_chain_crown_influence(chain.handle, upto, side, _lib.ptr(C), *tail[:9], _lib.ptr_array(infl), *tail[9:]))
        else:
            _lib.check(chain.lib.bf_chain_crown(chain.handle, upto, side, _lib.ptr(C), *tail))
        outs[side] = out
    return outs[0], outs[1]


def needs_graph_path(module: Any) -> bool:
    """True when the entry task is not a chain: an op merges values (add, concat) or does not consume
    the previous op's output (fan-out, skip connections)."""
    task = module.get_entry_task()
    cur = task.input_values[0] if task.input_values else None
    for op in task.ops:
        if op.op_type in ("add", "concat") or not op.inputs or op.inputs[0] != cur:
            return True
        cur = op.outputs[0]
    return False


def run_crown_ibp_mlp(
    module: Any,
    input_spec: Any,
    *,
    linear_spec_C: Optional[torch.Tensor] = None,
    output_value: Optional[str] = None,
    relu_alpha: Optional[Mapping[str, torch.Tensor]] = None,
    relu_pre_add_coeff_u: Optional[Mapping[str, torch.Tensor]] = None,
    relu_pre_add_coeff_l: Optional[Mapping[str, torch.Tensor]] = None,
    relu_split_state: Optional[Mapping[str, torch.Tensor]] = None,
    materialization_plan: Any = None,
    materialization_placement_plan: Any = None,
    fused_crown_executor: Any = None,
    fused_crown_steps: Sequence[Any] = (),
) -> IntervalState:
    """IBP trace + one CROWN backward sweep per side (crown_ibp.py:2054-2133).  Graphs with add / concat /
    fan-out go through the general graph path (`dag.py`), chains through the fused sweeps.  The last four arguments
    are the reference's execution-strategy arguments (when lazily kept operators are made dense, which steps a plug-in
    executor takes): accepted so that existing calls keep working, without effect here - the bounds do not depend on them."""
    if needs_graph_path(module):
        from .dag import run_crown_ibp_dag

        return run_crown_ibp_dag(module, input_spec, linear_spec_C=linear_spec_C, output_value=output_value, relu_alpha=relu_alpha,
                                 relu_pre_add_coeff_l=relu_pre_add_coeff_l, relu_pre_add_coeff_u=relu_pre_add_coeff_u,
                                 relu_split_state=relu_split_state)
    spec = normalize_input_spec(input_spec)
    if not (relu_split_state or relu_alpha or relu_pre_add_coeff_l or relu_pre_add_coeff_u):
        plain = _plain_set(spec)
        if plain is not None:
            center = spec.center
            chain = compile_chain(module, center.shape[1:], center.device)
            if output_value is None or output_value == chain.output_name:
                return _crown_query(chain, plain, linear_spec_C, center.device, int(center.shape[0]))
    trace = ibp_trace(module, input_spec, relu_split_state=relu_split_state)
    _raise_if_infeasible(trace, "relu split")
    lo, up = crown_from_trace(trace, linear_spec_C, output_value=output_value, relu_alpha=relu_alpha, relu_pre_add_coeff_l=relu_pre_add_coeff_l,
                              relu_pre_add_coeff_u=relu_pre_add_coeff_u)
    dev = spec.center.device
    return IntervalState(lower=lo.to(dev), upper=up.to(dev))


def _crown_query(chain: CudaChain, plain, linear_spec_C: Optional[torch.Tensor], device: torch.device, B: int) -> IntervalState:
    """Both CROWN bounds of the chain's output in one call of the library: what lies between stays in one workspace."""
    C = _expand_spec(linear_spec_C, B, chain.output_width, device)
    S = int(C.shape[1])
    lower, upper = torch.empty(B, S, dtype=torch.float32, device=device), torch.empty(B, S, dtype=torch.float32, device=device)
    nbytes = chain.lib.bf_chain_query_workspace_bytes(chain.size_handle, B, S, 0)
    ws = torch.empty(nbytes, dtype=torch.uint8, device=device)
    a, b, eps = plain
    _lib.check(chain.lib.bf_chain_crown_query(chain.handle, a.data_ptr(), _lib.ptr(b), eps, C.data_ptr(), lower.data_ptr(), upper.data_ptr(), ws.data_ptr(),
                                              nbytes, B, S, _stream_ptr(device)))
    return IntervalState(lower=lower, upper=upper)


def ibp_query(chain: CudaChain, plain, device: torch.device, B: int) -> IntervalState:
    """Interval bounds of the chain's output in one call of the library."""
    shape = (B,) + tuple(chain.output_shape)
    lower, upper = torch.empty(shape, dtype=torch.float32, device=device), torch.empty(shape, dtype=torch.float32, device=device)
    nbytes = chain.lib.bf_chain_query_workspace_bytes(chain.size_handle, B, 0, 0)
    ws = torch.empty(nbytes, dtype=torch.uint8, device=device)
    a, b, eps = plain
    _lib.check(chain.lib.bf_chain_ibp_query(chain.interval_handle, a.data_ptr(), _lib.ptr(b), eps, lower.data_ptr(), upper.data_ptr(), ws.data_ptr(), nbytes, B,
                                            _stream_ptr(device)))
    return IntervalState(lower=lower, upper=upper)


def run_crown_ibp_mlp_from_forward_trace(
    module: Any,
    input_spec: Any,
    *,
    interval_env: Mapping[str, Any],
    relu_pre: Mapping[str, Any],
    linear_spec_C: Optional[torch.Tensor] = None,
    output_value: Optional[str] = None,
    relu_alpha: Optional[Mapping[str, torch.Tensor]] = None,
    relu_pre_add_coeff_u: Optional[Mapping[str, torch.Tensor]] = None,
    relu_pre_add_coeff_l: Optional[Mapping[str, torch.Tensor]] = None,
    materialization_plan: Any = None,
    materialization_placement_plan: Any = None,
    fused_crown_executor: Any = None,
    fused_crown_steps: Sequence[Any] = (),
    fused_crown_context: Any = None,
) -> IntervalState:
    """Backward-only CROWN given a forward trace (crown_ibp.py:2136-2230).  The last five arguments are the
    reference's execution-strategy arguments, accepted without effect (the bounds do not depend on them)."""
    if needs_graph_path(module):
        from .dag import crown_dag

        lo, up, _tr = crown_dag(module, input_spec, linear_spec_C, output_value=output_value,
                                trace=_graph_trace_from_env(module, input_spec, interval_env, relu_pre), relu_alpha=relu_alpha,
                                relu_pre_add_coeff_l=relu_pre_add_coeff_l, relu_pre_add_coeff_u=relu_pre_add_coeff_u)
        dev = normalize_input_spec(input_spec).center.device
        return IntervalState(lower=lo.to(dev), upper=up.to(dev))
    trace = _trace_from_env(module, input_spec, interval_env, relu_pre)
    lo, up = crown_from_trace(trace, linear_spec_C, output_value=output_value, relu_alpha=relu_alpha, relu_pre_add_coeff_l=relu_pre_add_coeff_l,
                              relu_pre_add_coeff_u=relu_pre_add_coeff_u)
    dev = normalize_input_spec(input_spec).center.device
    return IntervalState(lower=lo.to(dev), upper=up.to(dev))


def run_crown_ibp_mlp_with_relu_influence_from_forward_trace(
    module: Any,
    input_spec: Any,
    *,
    interval_env: Mapping[str, Any],
    relu_pre: Mapping[str, Any],
    linear_spec_C: torch.Tensor,
    output_value: Optional[str] = None,
) -> Tuple[IntervalState, Dict[str, torch.Tensor]]:
    """Bounds plus, per ReLU input, the influence max(max_s |A_u|, max_s |A_l|) of the backward
    coefficients that reach it (crown_ibp.py:2201-2240), shaped like the pre-activation."""
    if needs_graph_path(module):
        from .dag import crown_influence_dag

        lo, up, infl_d, tr = crown_influence_dag(module, input_spec, linear_spec_C, output_value=output_value,
                                                 trace=_graph_trace_from_env(module, input_spec, interval_env, relu_pre))
        if set(infl_d) != set(relu_pre):
            raise ValueError("ReLU objective influence coverage differs")
        dev = normalize_input_spec(input_spec).center.device
        return (IntervalState(lower=lo.to(dev), upper=up.to(dev)),
                {n: infl_d[n].reshape((tr.B,) + tuple(tr.shape[n])).to(dev) for n in relu_pre})
    trace = _trace_from_env(module, input_spec, interval_env, relu_pre)
    infl: List[torch.Tensor] = []
    lo, up = crown_from_trace(trace, linear_spec_C, output_value=output_value, influence_out=infl)
    chain, B = trace.chain, trace.B
    dev = normalize_input_spec(input_spec).center.device
    if len(infl) != len(relu_pre):
        raise ValueError("ReLU objective influence coverage differs")
    out = {n: t.reshape((B,) + tuple(s)).to(dev) for n, t, s in zip(chain.relu_input_names, infl, chain.relu_shapes)}
    return IntervalState(lower=lo.to(dev), upper=up.to(dev)), out


def adaptive_alpha_from_trace(trace: ForwardTrace) -> List[torch.Tensor]:
    """alpha start = 1 where l>=0 or (l<0<u and u>-l), else 0
    (runtime/native_alpha_beta_optimizer_schedule.py:635-656)."""
    out = []
    device = trace.mid.device
    for l, u, n in zip(trace.pre_l, trace.pre_u, trace.chain.relu_widths):
        a = torch.empty(trace.B, n, dtype=torch.float32, device=device)
        _lib.check(trace.chain.lib.bf_alpha_adaptive_init(_lib.ptr(l), _lib.ptr(u), _lib.ptr(a), trace.B, n, _stream_ptr(device)))
        out.append(a)
    return out


def alpha_crown_from_trace(
    trace: ForwardTrace,
    linear_spec_C: torch.Tensor,
    alpha0: Sequence[torch.Tensor],
    *,
    steps: int,
    lr: float,
    spec_reduce: str = "mean",
    want_upper: bool = True,
    beta_splits: Optional[Sequence[Optional[torch.Tensor]]] = None,
    beta0: Optional[Sequence[torch.Tensor]] = None,
    soft_tau: float = 1.0,
    objective: str = "lower",
    lb_weight: float = 1.0,
    ub_weight: float = 1.0,
):
    """Device-resident alpha (and, with `beta_splits`, beta) loop; returns (best_lower,
    best_upper|None, best_alpha list, last alpha list, best_metric) and, with beta, a sixth
    element best_beta list.  `beta_splits[r]` is the int8 split assignment [B,n_r] or [1,n_r]
    of ReLU r (None = no split there).

    `objective` follows run_alpha_beta_crown_mlp (alpha_beta_crown.py:807-818): "lower" | "upper" | "gap" |
    "both" (with lb_weight / ub_weight).  As there, the beta term enters the lower objective only: the other
    objectives run alpha-only and hand the start beta back unchanged."""
    chain, B, device = trace.chain, trace.B, trace.mid.device
    if objective not in ("lower", "upper", "gap", "both"):
        raise ValueError(f"objective={objective!r}: expected lower | upper | gap | both")
    if objective != "lower":
        return _alpha_crown_other_objective(trace, linear_spec_C, alpha0, steps=steps, lr=lr, spec_reduce=spec_reduce, soft_tau=soft_tau,
                                            objective=objective, lb_weight=lb_weight, ub_weight=ub_weight, beta_splits=beta_splits, beta0=beta0)
    codes = {"mean": _lib.REDUCE_MEAN, "sum": _lib.REDUCE_SUM, "min": _lib.REDUCE_MIN, "softmin": _lib.REDUCE_SOFTMIN}
    if spec_reduce not in codes:
        raise ValueError(f"spec_reduce={spec_reduce!r}: expected mean | sum | min | softmin")
    if spec_reduce == "softmin" and float(soft_tau) <= 0.0:
        raise ValueError(f"soft_tau must be >0, got {soft_tau}")
    n_out = 1
    for d in chain.output_shape:
        n_out *= int(d)
    C = _expand_spec(linear_spec_C, B, n_out, device)
    S = int(C.shape[1])
    alpha = [a.detach().to(device=device, dtype=torch.float32).reshape(-1, n).expand(B, n).contiguous().clone() for a, n in zip(alpha0, chain.relu_widths)]
    best_alpha = [torch.empty_like(a) for a in alpha]
    best_lower = torch.empty(B, S, dtype=torch.float32, device=device)
    best_upper = torch.empty(B, S, dtype=torch.float32, device=device) if want_upper else None
    best_metric = torch.empty(B, dtype=torch.float32, device=device)
    reduce_code = codes[spec_reduce]
    if beta_splits is None:
        nbytes = int(chain.lib.bf_chain_alpha_workspace_bytes(chain.size_handle, B, S))
        ws = _Workspace.get(device, nbytes)
        _lib.check(
            chain.lib.bf_chain_alpha_beta_crown_reduce(
                chain.handle, _lib.ptr(C), _lib.ptr_array(trace.pre_l), _lib.ptr_array(trace.pre_u),
                _lib.ptr_array(alpha), _lib.ptr_array(best_alpha), None, None, None, None,
                _lib.ptr(trace.mid), _lib.ptr(trace.rad) if trace.norm_p == _lib.NORM_BOX else None, int(trace.norm_p), float(trace.eps),
                _lib.ptr(best_lower), _lib.ptr(best_upper), _lib.ptr(best_metric),
                int(steps), float(lr), reduce_code, float(soft_tau), _lib.ptr(ws), ws.numel(), B, S, _stream_ptr(device),
            )
        )
        return best_lower, best_upper, best_alpha, alpha, best_metric
    splits, strides = [], []
    for r, n in enumerate(chain.relu_widths):
        sp = beta_splits[r] if r < len(beta_splits) else None
        if sp is None:
            splits.append(None)
            strides.append(0)
        else:
            t, st = _split_tensor(sp, B, n, device, chain.relu_input_names[r])
            splits.append(t)
            strides.append(st)
    if beta0 is not None:
        beta = [b.detach().to(device=device, dtype=torch.float32).reshape(-1, n).expand(B, n).contiguous().clone() for b, n in zip(beta0, chain.relu_widths)]
    else:
        beta = [torch.zeros(B, n, dtype=torch.float32, device=device) for n in chain.relu_widths]
    best_beta = [b.clone() for b in beta]
    nbytes = int(chain.lib.bf_chain_alpha_beta_workspace_bytes(chain.size_handle, B, S))
    ws = _Workspace.get(device, nbytes)
    _lib.check(
        chain.lib.bf_chain_alpha_beta_crown_reduce(
            chain.handle, _lib.ptr(C), _lib.ptr_array(trace.pre_l), _lib.ptr_array(trace.pre_u),
            _lib.ptr_array(alpha), _lib.ptr_array(best_alpha), _lib.ptr_array(beta), _lib.ptr_array(best_beta),
            _lib.ptr_array(splits), _lib.int_array(strides), _lib.ptr(trace.mid), _lib.ptr(trace.rad) if trace.norm_p == _lib.NORM_BOX else None, int(trace.norm_p), float(trace.eps),
            _lib.ptr(best_lower), _lib.ptr(best_upper), _lib.ptr(best_metric),
            int(steps), float(lr), reduce_code, float(soft_tau), _lib.ptr(ws), ws.numel(), B, S, _stream_ptr(device),
        )
    )
    return best_lower, best_upper, best_alpha, alpha, best_metric, best_beta


def _shared_alpha_other(trace, linear_spec_C, alpha0, *, steps, lr, objective, spec_reduce, soft_tau, lb_weight, ub_weight):
    """Shared-alpha loop for the objectives / reductions beyond lower / mean (bf_chain_alpha_crown_shared_objective)."""
    chain, B, device = trace.chain, trace.B, trace.mid.device
    if spec_reduce == "softmin" and float(soft_tau) <= 0.0:
        raise ValueError(f"soft_tau must be >0, got {soft_tau}")
    if float(lb_weight) < 0.0 or float(ub_weight) < 0.0:
        raise NotImplementedError("the CUDA backend takes non-negative lb_weight / ub_weight")
    n_out = 1
    for d in chain.output_shape:
        n_out *= int(d)
    C = _expand_spec(linear_spec_C, B, n_out, device)
    S = int(C.shape[1])
    codes = {"mean": _lib.REDUCE_MEAN, "min": _lib.REDUCE_MIN, "softmin": _lib.REDUCE_SOFTMIN}
    alpha = [a.detach().to(device=device, dtype=torch.float32).reshape(n).contiguous().clone() for a, n in zip(alpha0, chain.relu_widths)]
    best_alpha = [torch.empty_like(a) for a in alpha]
    best_metric = torch.empty(1, dtype=torch.float32, device=device)
    paired = objective in ("gap", "both")
    rows_C = torch.cat([C, -C], dim=1).contiguous() if paired else (-C if objective == "upper" else C)
    n_rows = 2 * S if paired else S
    best_rows = torch.empty(B, n_rows, dtype=torch.float32, device=device)
    best_upper = None if paired else torch.empty(B, S, dtype=torch.float32, device=device)
    nbytes = int(chain.lib.bf_chain_alpha_shared_workspace_bytes(chain.size_handle, B, n_rows, 0))
    ws = _Workspace.get(device, nbytes)
    obj_code = {"lower": 0, "upper": 0, "gap": _lib.OBJECTIVE_GAP, "both": _lib.OBJECTIVE_BOTH}[objective]
    _lib.check(
        chain.lib.bf_chain_alpha_crown_shared_objective(
            chain.handle, _lib.ptr(rows_C), _lib.ptr_array(trace.pre_l), _lib.ptr_array(trace.pre_u), _lib.ptr_array(alpha), _lib.ptr_array(best_alpha),
            _lib.ptr(trace.mid), _lib.ptr(trace.rad) if trace.norm_p == _lib.NORM_BOX else None, int(trace.norm_p), float(trace.eps),
            _lib.ptr(best_rows), _lib.ptr(best_upper), _lib.ptr(best_metric), int(steps), float(lr), obj_code, codes[spec_reduce], float(soft_tau),
            float(lb_weight), float(ub_weight), _lib.ptr(ws), ws.numel(), B, S, _stream_ptr(device),
        )
    )
    if paired:
        return best_rows[:, :S].contiguous(), -best_rows[:, S:], best_alpha, alpha, best_metric
    if objective == "upper":
        return -best_upper, -best_rows, best_alpha, alpha, best_metric
    return best_rows, best_upper, best_alpha, alpha, best_metric


def _alpha_crown_other_objective(trace, linear_spec_C, alpha0, *, steps, lr, spec_reduce, soft_tau, objective, lb_weight, ub_weight,
                                 beta_splits, beta0):
    """objective "upper" = the lower loop on the negated spec rows (upper(C) = -lower(-C)); "gap" and "both" evaluate
    the rows and their negations side by side (2S rows per domain) through bf_chain_alpha_crown_objective."""
    chain, B, device = trace.chain, trace.B, trace.mid.device
    if spec_reduce not in ("mean", "min", "softmin"):
        raise ValueError(f"spec_reduce={spec_reduce!r}: objective {objective!r} takes mean | min | softmin")
    if spec_reduce == "softmin" and float(soft_tau) <= 0.0:
        raise ValueError(f"soft_tau must be >0, got {soft_tau}")
    n_out = 1
    for d in chain.output_shape:
        n_out *= int(d)
    C = _expand_spec(linear_spec_C, B, n_out, device)
    S = int(C.shape[1])
    tail = ()
    if beta_splits is not None:  # no beta term on these objectives: the start values come back unchanged
        beta = ([b.detach().to(device=device, dtype=torch.float32).reshape(-1, n).expand(B, n).contiguous().clone() for b, n in zip(beta0, chain.relu_widths)]
                if beta0 is not None else [torch.zeros(B, n, dtype=torch.float32, device=device) for n in chain.relu_widths])
        tail = (beta,)
    if objective == "upper":
        lo, up, best_alpha, alpha, metric = alpha_crown_from_trace(trace, -C, alpha0, steps=steps, lr=lr, spec_reduce=spec_reduce,
                                                                   want_upper=True, soft_tau=soft_tau)
        return (-up, -lo, best_alpha, alpha, metric) + tail
    if float(lb_weight) < 0.0 or float(ub_weight) < 0.0:
        raise NotImplementedError("the CUDA backend takes non-negative lb_weight / ub_weight (a row weight must not flip the sign decisions of the gradient sweep)")
    C2 = torch.cat([C, -C], dim=1).contiguous()
    alpha = [a.detach().to(device=device, dtype=torch.float32).reshape(-1, n).expand(B, n).contiguous().clone() for a, n in zip(alpha0, chain.relu_widths)]
    best_alpha = [torch.empty_like(a) for a in alpha]
    best_rows = torch.empty(B, 2 * S, dtype=torch.float32, device=device)
    best_metric = torch.empty(B, dtype=torch.float32, device=device)
    codes = {"mean": _lib.REDUCE_MEAN, "min": _lib.REDUCE_MIN, "softmin": _lib.REDUCE_SOFTMIN}
    nbytes = int(chain.lib.bf_chain_alpha_workspace_bytes(chain.size_handle, B, 2 * S))
    ws = _Workspace.get(device, nbytes)
    _lib.check(
        chain.lib.bf_chain_alpha_crown_objective(
            chain.handle, _lib.ptr(C2), _lib.ptr_array(trace.pre_l), _lib.ptr_array(trace.pre_u), _lib.ptr_array(alpha), _lib.ptr_array(best_alpha),
            _lib.ptr(trace.mid), _lib.ptr(trace.rad) if trace.norm_p == _lib.NORM_BOX else None, int(trace.norm_p), float(trace.eps),
            _lib.ptr(best_rows), _lib.ptr(best_metric), int(steps), float(lr),
            _lib.OBJECTIVE_GAP if objective == "gap" else _lib.OBJECTIVE_BOTH, codes[spec_reduce], float(soft_tau), float(lb_weight), float(ub_weight),
            _lib.ptr(ws), ws.numel(), B, S, _stream_ptr(device),
        )
    )
    return (best_rows[:, :S].contiguous(), -best_rows[:, S:], best_alpha, alpha, best_metric) + tail


def alpha_grad_from_trace(trace: ForwardTrace, linear_spec_C: torch.Tensor, alpha: Sequence[torch.Tensor], *, spec_reduce: str = "mean"):
    """Gradient of -sum_b reduce_s lower wrt alpha and the lower bounds at `alpha`."""
    chain, B, device = trace.chain, trace.B, trace.mid.device
    n_out = 1
    for d in chain.output_shape:
        n_out *= int(d)
    C = _expand_spec(linear_spec_C, B, n_out, device)
    S = int(C.shape[1])
    alpha = [a.detach().to(device=device, dtype=torch.float32).reshape(-1, n).expand(B, n).contiguous() for a, n in zip(alpha, chain.relu_widths)]
    grads = [torch.empty_like(a) for a in alpha]
    lower = torch.empty(B, S, dtype=torch.float32, device=device)
    nbytes = int(chain.lib.bf_chain_alpha_workspace_bytes(chain.size_handle, B, S))
    ws = _Workspace.get(device, nbytes)
    _lib.check(
        chain.lib.bf_chain_alpha_grad(
            chain.handle, _lib.ptr(C), _lib.ptr_array(trace.pre_l), _lib.ptr_array(trace.pre_u), _lib.ptr_array(alpha),
            _lib.ptr(trace.mid), _lib.ptr(trace.rad) if trace.norm_p == _lib.NORM_BOX else None, int(trace.norm_p), float(trace.eps), _lib.ptr_array(grads), _lib.ptr(lower),
            _lib.REDUCE_MEAN if spec_reduce == "mean" else _lib.REDUCE_SUM,
            _lib.ptr(ws), ws.numel(), B, S, _stream_ptr(device),
        )
    )
    return grads, lower


def shared_alpha_crown_from_trace(trace: ForwardTrace, linear_spec_C: Optional[torch.Tensor], alpha0: Sequence[torch.Tensor], *,
                                  steps: int, lr: float, want_upper: bool = True,
                                  beta_splits: Optional[Sequence[Optional[torch.Tensor]]] = None,
                                  beta0: Optional[Sequence[torch.Tensor]] = None, objective: str = "lower", spec_reduce: str = "mean",
                                  soft_tau: float = 1.0, lb_weight: float = 1.0, ub_weight: float = 1.0):
    """Device-resident loop with ONE alpha (and, with `beta_splits`, one beta) per neuron for the
    whole batch; returns (best_lower, best_upper|None, best_alpha list [n_r], last alpha list,
    best_metric [1]) and, with beta, a sixth element best_beta list [n_r].  `objective` lower | upper | gap | both
    and `spec_reduce` mean | min | softmin as in run_alpha_crown_mlp (alpha_crown.py:93-134); beta enters the
    lower objective only (any reduction)."""
    chain, B, device = trace.chain, trace.B, trace.mid.device
    if objective not in ("lower", "upper", "gap", "both"):
        raise ValueError(f"objective={objective!r}: expected lower | upper | gap | both")
    if spec_reduce not in ("mean", "min", "softmin"):
        raise ValueError(f"spec_reduce={spec_reduce!r}: the shared-parameter loop takes mean | min | softmin")
    if spec_reduce == "softmin" and float(soft_tau) <= 0.0:
        raise ValueError(f"soft_tau must be >0, got {soft_tau}")
    if objective != "lower" or (spec_reduce != "mean" and beta_splits is None):
        if beta_splits is not None:
            raise NotImplementedError("the beta term enters objective='lower' only (alpha_beta_crown.py:763-785)")
        return _shared_alpha_other(trace, linear_spec_C, alpha0, steps=steps, lr=lr, objective=objective, spec_reduce=spec_reduce,
                                   soft_tau=soft_tau, lb_weight=lb_weight, ub_weight=ub_weight)
    n_out = 1
    for d in chain.output_shape:
        n_out *= int(d)
    C = _expand_spec(linear_spec_C, B, n_out, device)
    S = int(C.shape[1])
    alpha = [a.detach().to(device=device, dtype=torch.float32).reshape(n).contiguous().clone() for a, n in zip(alpha0, chain.relu_widths)]
    best_alpha = [torch.empty_like(a) for a in alpha]
    best_lower = torch.empty(B, S, dtype=torch.float32, device=device)
    best_upper = torch.empty(B, S, dtype=torch.float32, device=device) if want_upper else None
    best_metric = torch.empty(1, dtype=torch.float32, device=device)
    with_beta = beta_splits is not None
    beta = best_beta = None
    splits: List[Optional[torch.Tensor]] = []
    strides: List[int] = []
    if with_beta:
        for r, n in enumerate(chain.relu_widths):
            sp = beta_splits[r] if r < len(beta_splits) else None
            if sp is None:
                splits.append(None)
                strides.append(0)
            else:
                t, st = _split_tensor(sp, B, n, device, chain.relu_input_names[r])
                splits.append(t)
                strides.append(st)
        if beta0 is not None:
            beta = [b.detach().to(device=device, dtype=torch.float32).reshape(n).contiguous().clone() for b, n in zip(beta0, chain.relu_widths)]
        else:
            beta = [torch.zeros(n, dtype=torch.float32, device=device) for n in chain.relu_widths]
        best_beta = [b.clone() for b in beta]
    nbytes = int(chain.lib.bf_chain_alpha_shared_workspace_bytes(chain.size_handle, B, S, 1 if with_beta else 0))
    ws = _Workspace.get(device, nbytes)
    codes = {"mean": _lib.REDUCE_MEAN, "min": _lib.REDUCE_MIN, "softmin": _lib.REDUCE_SOFTMIN}
    _lib.check(
        chain.lib.bf_chain_alpha_beta_crown_shared_reduce(
            chain.handle, _lib.ptr(C), _lib.ptr_array(trace.pre_l), _lib.ptr_array(trace.pre_u),
            _lib.ptr_array(alpha), _lib.ptr_array(best_alpha),
            _lib.ptr_array(beta) if with_beta else None, _lib.ptr_array(best_beta) if with_beta else None,
            _lib.ptr_array(splits) if with_beta else None, _lib.int_array(strides) if with_beta else None,
            _lib.ptr(trace.mid), _lib.ptr(trace.rad) if trace.norm_p == _lib.NORM_BOX else None, int(trace.norm_p), float(trace.eps),
            _lib.ptr(best_lower), _lib.ptr(best_upper), _lib.ptr(best_metric),
            int(steps), float(lr), codes[spec_reduce], float(soft_tau), _lib.ptr(ws), ws.numel(), B, S, _stream_ptr(device),
        )
    )
    if with_beta:
        return best_lower, best_upper, best_alpha, alpha, best_metric, best_beta
    return best_lower, best_upper, best_alpha, alpha, best_metric


def run_alpha_crown_mlp(
    module: Any,
    input_spec: Any,
    *,
    linear_spec_C: Optional[torch.Tensor] = None,
    steps: int = 20,
    lr: float = 0.2,
    alpha_init: float = 0.5,
    objective: str = "lower",
    spec_reduce: str = "mean",
    soft_tau: float = 1.0,
    lb_weight: float = 1.0,
    ub_weight: float = 1.0,
    warm_start: Optional[Any] = None,
    relu_split_state: Optional[Mapping[str, torch.Tensor]] = None,
    materialization_plan: Any = None,
    materialization_placement_plan: Any = None,
):
    """alpha-CROWN with alpha stored per ReLU neuron and shared across batch and spec rows
    (`run_alpha_crown_mlp`, runtime/alpha_crown.py:137-261): steps+1 evaluations, Adam on
    -mean(lower), clamp to [0,1], and the bounds / alpha of the evaluation with the best
    whole-batch metric.  Returns (IntervalState, AlphaState, AlphaCrownStats) like the
    reference, for objective lower | upper | gap | both and spec_reduce mean | min | softmin, on
    affine (relu affine)* chains (Linear / Conv2d / flatten) and, through the per-value graph loop, on graphs with
    add / concat / fan-out."""
    if needs_graph_path(module):
        bounds, state, _beta, stats = _run_alpha_beta_crown_graph(
            module, input_spec, linear_spec_C=linear_spec_C, relu_split_state=relu_split_state, steps=steps, lr=lr, alpha_init=alpha_init,
            beta_init=0.0, warm_start_alpha=warm_start, warm_start_beta=None, objective=objective, spec_reduce=spec_reduce, soft_tau=soft_tau,
            lb_weight=lb_weight, ub_weight=ub_weight, per_batch_params=False, optimize_beta=False)
        return bounds, state, stats
    trace = ibp_trace(module, input_spec, relu_split_state=relu_split_state)
    _raise_if_infeasible(trace, "relu split")
    chain, device = trace.chain, trace.mid.device
    ws_map = getattr(warm_start, "alpha_by_relu_input", None) if warm_start is not None else None
    alpha0 = []
    for name, n, shape in zip(chain.relu_input_names, chain.relu_widths, chain.relu_shapes):
        if ws_map is not None and name in ws_map:
            a = torch.as_tensor(ws_map[name])
            if a.dim() == 0:  # a scalar start broadcasts (relu_shape_utils.py:37-38)
                a = a.expand(n)
            if int(a.numel()) != n:
                raise ValueError(f"warm_start alpha[{name}] has {int(a.numel())} elements, the ReLU input has shape {tuple(shape)}")
            alpha0.append(a.detach().to(device=device, dtype=torch.float32).reshape(n))
        else:
            alpha0.append(torch.full((n,), float(alpha_init), dtype=torch.float32, device=device))
    best_l, best_u, best_a, _last, _metric = shared_alpha_crown_from_trace(trace, linear_spec_C, alpha0, steps=steps, lr=lr, objective=objective,
                                                                           spec_reduce=spec_reduce, soft_tau=soft_tau, lb_weight=lb_weight,
                                                                           ub_weight=ub_weight)
    dev = normalize_input_spec(input_spec).center.device
    bounds = IntervalState(lower=best_l.to(dev), upper=best_u.to(dev))
    state = AlphaState({n: a.reshape(tuple(s)).to(dev) for n, a, s in zip(chain.relu_input_names, best_a, chain.relu_shapes)})
    stats = AlphaCrownStats(steps=int(steps), lr=float(lr), objective=objective, spec_reduce=spec_reduce, relu_inputs=tuple(chain.relu_input_names))
    return bounds, state, stats


def first_layer_certificate(module: Any, input_spec: Any, relu_split_state: Mapping[str, torch.Tensor], *,
                            steps: int = 200, lr: float = 0.1, tol: float = 1e-6):
    """Per-domain first-layer infeasibility certificate (`_is_infeasible_split_first_layer_convex_combo`,
    alpha_beta_crown.py:391-532, which the reference runs for batch size 1; here for every domain).
    Returns (infeasible int32 [B]: 1 found / 0 none / -1 not evaluated, best_value float [B],
    n_halfspaces int32 [B]) as CUDA tensors.  The splits of the first ReLU over a Linear or Conv2d first
    layer are used (conv: the half-space row of a split neuron is its filter placed in the input image,
    alpha_beta_crown.py:325-387; only the rows of neurons that are split somewhere in the batch are formed);
    a chain that starts otherwise, or no split on that ReLU, gives all zeros.  Boxes, L-inf, L2 and L1 balls.  On a graph that is not a chain every
    ReLU fed by a Linear / Conv2d op on the input value contributes its half-spaces (`dag.first_layer_certificate_dag`)."""
    if needs_graph_path(module):
        from .dag import first_layer_certificate_dag

        return first_layer_certificate_dag(module, input_spec, relu_split_state, steps=steps, lr=lr, tol=tol)
    spec, chain, device, B, mid, rad, _ = _prepare_input(module, input_spec)
    ball = lp_ball_of(spec)

    def certificate(sp_t, sp_stride, W_rows, b_rows, n_rows):
        """Box / L-inf: maximum over the box; L1 / L2 ball: centre term + eps * dual norm (mid holds the centre then)."""
        if ball is not None:
            _lib.check(chain.lib.bf_first_layer_certificate_lp(
                _lib.ptr(sp_t), sp_stride, _lib.ptr(W_rows), _lib.ptr(b_rows), _lib.ptr(mid), float(ball[1]), int(ball[0]), _lib.ptr(infeasible),
                _lib.ptr(best), _lib.ptr(count), int(steps), float(lr), float(tol), B, n_rows, chain.n0, _stream_ptr(device)))
        else:
            _lib.check(chain.lib.bf_first_layer_certificate(
                _lib.ptr(sp_t), sp_stride, _lib.ptr(W_rows), _lib.ptr(b_rows), _lib.ptr(mid), _lib.ptr(rad), _lib.ptr(infeasible), _lib.ptr(best),
                _lib.ptr(count), int(steps), float(lr), float(tol), B, n_rows, chain.n0, _stream_ptr(device)))

    infeasible = torch.zeros(B, dtype=torch.int32, device=device)
    best = torch.full((B,), float("inf"), dtype=torch.float32, device=device)
    count = torch.zeros(B, dtype=torch.int32, device=device)
    first = next((l for l in chain.layers if l.op != "flatten"), None)
    if first is None or first.op not in ("linear", "conv2d") or not chain.relu_input_names or first.out_name != chain.relu_input_names[0]:
        return infeasible, best, count
    raw = relu_split_state.get(chain.relu_input_names[0]) if relu_split_state else None
    if raw is None:
        return infeasible, best, count
    n1 = chain.relu_widths[0]
    sp, stride = _split_tensor(raw, B, n1, device, chain.relu_input_names[0])
    if first.op == "conv2d":
        cols = torch.nonzero((sp != 0).any(dim=0)).flatten()   # neurons split in at least one domain, ascending
        if int(cols.numel()) == 0:
            return infeasible, best, count
        U = int(cols.numel())
        rows = cols.to(torch.int32).contiguous()
        W_rows = torch.empty(U, chain.n0, dtype=torch.float32, device=device)
        b_rows = torch.empty(U, dtype=torch.float32, device=device)
        (Ci, Hi, Wi), (Co, Ho, Wo) = first.in_shape, first.out_shape
        _lib.check(chain.lib.bf_conv2d_dense_rows(
            _lib.ptr(first.W), _lib.ptr(first.b), _lib.ptr(rows), U, _lib.ptr(W_rows), _lib.ptr(b_rows), int(Ci), int(Hi), int(Wi), int(Co), int(Ho),
            int(Wo), int(first.W.shape[2]), int(first.W.shape[3]), int(first.stride[0]), int(first.stride[1]), int(first.padding[0]),
            int(first.padding[1]), _stream_ptr(device)))
        sp_sub = sp[:, cols].contiguous()
        certificate(sp_sub, 0 if stride == 0 else U, W_rows, b_rows, U)
        return infeasible, best, count
    certificate(sp, stride, first.W, first.b, n1)
    return infeasible, best, count


def _run_alpha_beta_crown_graph(module, input_spec, *, linear_spec_C, relu_split_state, steps, lr, alpha_init, beta_init, warm_start_alpha,
                                warm_start_beta, objective, spec_reduce, soft_tau, lb_weight, ub_weight, per_batch_params, optimize_beta):
    """`run_alpha_beta_crown_mlp` on a graph that is not a chain (residual add, concat, fan-out): the loop of
    `dag.alpha_beta_crown_dag`, per-domain or shared parameters, every objective and reduction of the chain path.  The
    reference accepts these graphs because its sweep is the generic graph backward under autograd
    (crown_ibp.py:1669-2051)."""
    from .dag import alpha_beta_crown_dag

    a0 = getattr(warm_start_alpha, "alpha_by_relu_input", None) if warm_start_alpha is not None else None
    b0 = getattr(warm_start_beta, "beta_by_relu_input", None) if warm_start_beta is not None else None
    if relu_split_state and not optimize_beta and objective == "lower" and b0 is not None and any(
            float(torch.as_tensor(b).abs().max()) != 0.0 for b in b0.values()):
        raise NotImplementedError("a frozen non-zero beta is not supported; pass optimize_beta=None/True")
    best_l, best_u, best_a, best_b, tr = alpha_beta_crown_dag(module, input_spec, linear_spec_C, steps=steps, lr=lr, alpha0=a0, alpha_init=alpha_init,
                                                              relu_split_state=relu_split_state, optimize_beta=optimize_beta, beta0=b0,
                                                              beta_init=beta_init, spec_reduce=spec_reduce, soft_tau=soft_tau, objective=objective,
                                                              lb_weight=lb_weight, ub_weight=ub_weight, per_batch_params=per_batch_params)
    dev = normalize_input_spec(input_spec).center.device
    lead = (tr.B,) if per_batch_params else ()
    bounds = IntervalState(lower=best_l.to(dev), upper=best_u.to(dev))
    names = list(best_a)
    a_state = AlphaState({n: best_a[n].reshape(lead + tuple(tr.shape[n])).to(dev) for n in names})
    b_state = BetaState({n: best_b[n].reshape(lead + tuple(tr.shape[n])).to(dev) for n in names})
    stats = AlphaCrownStats(steps=int(steps), lr=float(lr), objective=objective, spec_reduce=spec_reduce, relu_inputs=tuple(names))
    stats.branch_choices = _branch_choices([tr.pre_l[n] for n in names], [tr.pre_u[n] for n in names], names,  # type: ignore[attr-defined]
                                           [int(tr.pre_l[n].shape[1]) for n in names], tr.B, tr.mid.device)
    return bounds, a_state, b_state, stats


def run_alpha_beta_crown_mlp(
    module: Any,
    input_spec: Any,
    *,
    linear_spec_C: Optional[torch.Tensor] = None,
    relu_split_state: Optional[Mapping[str, torch.Tensor]] = None,
    steps: int = 20,
    lr: float = 0.2,
    alpha_init: float = 0.5,
    beta_init: float = 0.0,
    warm_start_alpha: Optional[Any] = None,
    warm_start_beta: Optional[Any] = None,
    objective: str = "lower",
    spec_reduce: str = "mean",
    soft_tau: float = 1.0,
    per_batch_params: bool = False,
    optimize_beta: Optional[bool] = None,
    lb_weight: float = 1.0,
    ub_weight: float = 1.0,
    materialization_plan: Any = None,
    materialization_placement_plan: Any = None,
):
    """Per-domain alpha-beta optimisation (alpha_beta_crown.py:643-941).  `materialization_plan` /
    `materialization_placement_plan` (also on `run_alpha_crown_mlp`) are the reference's execution-strategy
    arguments, accepted without effect.

    Like the reference, beta (one multiplier >= 0 per split neuron and domain, start
    `beta_init` or `warm_start_beta`) is optimised together with alpha whenever a split
    assignment is given; `optimize_beta=False` freezes it at its start (the alpha-only
    loop), `None` means "as the reference".  `per_batch_params=False` (the reference's
    default) optimises one alpha / beta row shared by the whole batch with a whole-batch
    best-of.  Per-domain mode: objective lower | upper | gap | both (lb_weight / ub_weight >= 0) and
    spec_reduce mean | min | softmin (with `soft_tau`) as in the reference, plus "sum" for the lower
    objective; the upper / gap / both objectives run alpha only (the reference applies the beta term to
    objective="lower" alone, with any reduction).  Shared mode: the same objectives and mean | min | softmin.  For a single node the first-layer
    infeasibility certificate (alpha_beta_crown.py:391-532) is evaluated first, as in the
    reference (`first_layer_certificate` gives it for whole batches).  Graphs that are not chains (residual add,
    concat, fan-out) take the same arguments through the per-value loop of `dag.alpha_beta_crown_dag`.
    Infeasible splits raise ValueError like the reference.
    """
    if objective not in ("lower", "upper", "gap", "both"):
        raise ValueError(f"objective={objective!r}: expected lower | upper | gap | both")
    has_split = bool(relu_split_state)
    if optimize_beta is None:
        optimize_beta = has_split
    if optimize_beta and not has_split:
        optimize_beta = False  # nothing to constrain: beta's gradient is identically zero
    if has_split and int(normalize_input_spec(input_spec).center.shape[0]) == 1:
        # the reference's pre-check for a single node (alpha_beta_crown.py:693-714)
        cert, cert_val, _cnt = first_layer_certificate(module, input_spec, relu_split_state)
        if int(cert[0]) == 1:
            c = normalize_input_spec(input_spec).center
            zeros = torch.zeros((1, 1), device=c.device, dtype=c.dtype)
            stats = AlphaCrownStats(steps=int(steps), lr=float(lr), objective=objective, spec_reduce=spec_reduce, relu_inputs=(),
                                    feasibility="infeasible", reason=f"infeasible: first-layer certificate with max {float(cert_val[0]):.3e}")
            return IntervalState(lower=zeros, upper=zeros), AlphaState({}), BetaState({}), stats
    if needs_graph_path(module):
        return _run_alpha_beta_crown_graph(module, input_spec, linear_spec_C=linear_spec_C, relu_split_state=relu_split_state, steps=steps, lr=lr,
                                           alpha_init=alpha_init, beta_init=beta_init, warm_start_alpha=warm_start_alpha,
                                           warm_start_beta=warm_start_beta, objective=objective, spec_reduce=spec_reduce, soft_tau=soft_tau,
                                           lb_weight=lb_weight, ub_weight=ub_weight, per_batch_params=per_batch_params,
                                           optimize_beta=bool(optimize_beta))
    trace = ibp_trace(module, input_spec, relu_split_state=relu_split_state)
    _raise_if_infeasible(trace, "relu split")
    chain, B, device = trace.chain, trace.B, trace.mid.device
    rows = B if per_batch_params else 1  # shared mode: one parameter row for the whole batch (alpha_beta_crown.py:183-260)

    def _start(warm: Any, attr: str, init: float, what: str) -> List[torch.Tensor]:
        out = []
        wmap = getattr(warm, attr, None) if warm is not None else None
        for r, name in enumerate(chain.relu_input_names):
            n = chain.relu_widths[r]
            if wmap is not None and name in wmap:
                t, _ = _alpha_rows(wmap[name], rows, n, device, name)
                if not per_batch_params and int(t.shape[0]) != 1:
                    raise ValueError(f"warm start {what}[{name}] is batch-specific; expected the shared shape {tuple(chain.relu_shapes[r])}")
                out.append(t.expand(rows, n))
            else:
                out.append(torch.full((rows, n), float(init), dtype=torch.float32, device=device))
        return out

    alpha0 = _start(warm_start_alpha, "alpha_by_relu_input", alpha_init, "alpha")
    beta_start = _start(warm_start_beta, "beta_by_relu_input", beta_init, "beta")
    if linear_spec_C is None:
        n_out = 1
        for d in chain.output_shape:
            n_out *= int(d)
        linear_spec_C = torch.eye(n_out, dtype=torch.float32, device=device)
    dev = normalize_input_spec(input_spec).center.device
    loop = alpha_crown_from_trace if per_batch_params else shared_alpha_crown_from_trace
    kw = {"spec_reduce": spec_reduce, "soft_tau": soft_tau, "objective": objective, "lb_weight": lb_weight, "ub_weight": ub_weight}
    if objective != "lower":
        # the beta term enters the lower objective only (alpha_beta_crown.py:763-785): alpha-only evaluation, beta handed back
        best_l, best_u, best_a, _last, _metric = loop(trace, linear_spec_C, alpha0, steps=steps, lr=lr, **kw)
        best_b = beta_start
    elif optimize_beta:
        beta_splits = [relu_split_state.get(n) for n in chain.relu_input_names]
        best_l, best_u, best_a, _last, _metric, best_b = loop(
            trace, linear_spec_C, alpha0, steps=steps, lr=lr, beta_splits=beta_splits, beta0=beta_start, **kw)
    else:
        if has_split and any(float(b.abs().max()) != 0.0 for b in beta_start):
            raise NotImplementedError("a frozen non-zero beta is not supported; pass optimize_beta=None/True")
        best_l, best_u, best_a, _last, _metric = loop(trace, linear_spec_C, alpha0, steps=steps, lr=lr, **kw)
        best_b = beta_start
    if not per_batch_params:
        bounds = IntervalState(lower=best_l.to(dev), upper=best_u.to(dev))
        a_state = AlphaState({n: a.reshape(tuple(s)).to(dev) for n, a, s in zip(chain.relu_input_names, best_a, chain.relu_shapes)})
        b_state = BetaState({n: b.reshape(tuple(s)).to(dev) for n, b, s in zip(chain.relu_input_names, best_b, chain.relu_shapes)})
        stats = AlphaCrownStats(steps=int(steps), lr=float(lr), objective=objective, spec_reduce=spec_reduce, relu_inputs=tuple(chain.relu_input_names))
        stats.branch_choices = branch_choices_from_trace(trace)  # type: ignore[attr-defined]
        return bounds, a_state, b_state, stats
    bounds = IntervalState(lower=best_l.to(dev), upper=best_u.to(dev))
    a_state = AlphaState({n: a.reshape((B,) + tuple(s)).to(dev) for n, a, s in zip(chain.relu_input_names, best_a, chain.relu_shapes)})
    b_state = BetaState({n: b.reshape((B,) + tuple(s)).to(dev) for n, b, s in zip(chain.relu_input_names, best_b, chain.relu_shapes)})
    stats = AlphaCrownStats(steps=int(steps), lr=float(lr), objective=objective, spec_reduce=spec_reduce, relu_inputs=tuple(chain.relu_input_names))
    stats.branch_choices = branch_choices_from_trace(trace)  # type: ignore[attr-defined]
    return bounds, a_state, b_state, stats


def check_first_layer_infeasible_split(module: Any, input_spec: Any, *, relu_split_state: Mapping[str, torch.Tensor]) -> AlphaBetaCrownStats:
    """`check_first_layer_infeasible_split` (alpha_beta_crown.py:109-142): the first-layer certificate for ONE node as a
    stats object, `feasibility` "infeasible" when a certificate is found and "unknown" otherwise (no half-spaces, a batch
    of more than one input set, or no certificate)."""
    module.validate()
    spec = normalize_input_spec(input_spec)
    if int(spec.center.shape[0]) != 1:
        return AlphaBetaCrownStats(feasibility="unknown", reason="skip (batch!=1)")
    flags, values, counts = first_layer_certificate(module, spec, relu_split_state)
    flag, count = int(flags[0]), int(counts[0])
    if count == 0:
        return AlphaBetaCrownStats(feasibility="unknown", reason="ok (no first-layer split halfspaces)")
    if flag == 1:
        value = float(values[0])
        kind = "single_halfspace_max_negative" if count == 1 else "convex_combo_max_negative"
        return AlphaBetaCrownStats(feasibility="infeasible", reason=f"infeasible: {kind} with max {value:.3e}",
                                   infeasible_certificate={"type": kind, "max_value": value, "n_halfspaces": count})
    return AlphaBetaCrownStats(feasibility="unknown", reason="ok (no certificate found)" if flag == 0 else "skip (too many halfspaces)")


def get_crown_ibp_mlp_stats(module: Any) -> CrownIbpStats:
    """`get_crown_ibp_mlp_stats` (crown_ibp.py:2279-2349): whether `run_crown_ibp_mlp` of this backend takes the module,
    with the reason when it does not.  Same conditions as the reference: one INTERVAL_IBP task of linear / relu / conv2d /
    flatten(start_dim=1) / reshape / add (two inputs) / concat (two or more inputs, feature axis) ops with one output each."""
    try:
        module.validate()
        task = module.get_entry_task()
        kind = getattr(task.kind, "value", task.kind)
        if str(kind).lower().split(".")[-1] != "interval_ibp":
            return CrownIbpStats(False, f"TaskKind={task.kind}")
        if getattr(module, "task_graph", None) is not None or len(module.tasks) != 1:
            return CrownIbpStats(False, "multi-task module not supported")
        ops = tuple(op.op_type for op in task.ops)
        if not ops:
            return CrownIbpStats(False, "empty task", ops)
        unknown = [t for t in ops if t not in ("linear", "relu", "conv2d", "flatten", "reshape", "add", "concat")]
        if unknown:
            return CrownIbpStats(False, f"unsupported ops: {unknown}", ops)
        for i, op in enumerate(task.ops):
            if len(op.outputs) != 1:
                return CrownIbpStats(False, f"multi-output op not supported at op {i}: outputs={op.outputs}", ops)
            if op.op_type == "flatten" and (int(op.attrs.get("start_dim", 1)) != 1 or int(op.attrs.get("end_dim", -1)) != -1):
                return CrownIbpStats(False, f"unsupported flatten attrs at op {i}: {op.attrs}", ops)
            if op.op_type == "add" and len(op.inputs) != 2:
                return CrownIbpStats(False, f"add expects 2 inputs at op {i}, got {len(op.inputs)}", ops)
            if op.op_type == "concat":
                if len(op.inputs) < 2:
                    return CrownIbpStats(False, f"concat expects at least 2 inputs at op {i}, got {len(op.inputs)}", ops)
                if int(op.attrs.get("axis", 1)) not in (1, -1, -3):
                    return CrownIbpStats(False, f"unsupported concat axis at op {i}: {op.attrs.get('axis', 1)}", ops)
        return CrownIbpStats(True, "", ops)
    except Exception as e:  # a module that does not even validate is unsupported, with the reason
        return CrownIbpStats(False, str(e))


def branch_choices_from_trace(trace: ForwardTrace) -> List[Optional[Tuple[str, int]]]:
    """Widest-unstable-gap branching hint per domain as (ReLU input name, flat neuron index) or None
    (`_branch_choices_from_relu_pre`, alpha_beta_crown.py:145-182).  Synchronises to return Python values."""
    chain = trace.chain
    return _branch_choices(trace.pre_l, trace.pre_u, chain.relu_input_names, chain.relu_widths, trace.B, trace.mid.device)


def _branch_choices(pre_l: Sequence[torch.Tensor], pre_u: Sequence[torch.Tensor], names: Sequence[str], widths: Sequence[int], B: int,
                    device: torch.device) -> List[Optional[Tuple[str, int]]]:
    """The hint from the pre-activation bounds of the ReLUs in graph order ([B, n_r] each)."""
    if not names:
        return [None] * B
    lib = _lib.load()
    gap = torch.empty(B, dtype=torch.float32, device=device)
    relu = torch.empty(B, dtype=torch.int32, device=device)
    idx = torch.empty(B, dtype=torch.int32, device=device)
    _lib.check(lib.bf_branch_scores(_lib.ptr_array(list(pre_l)), _lib.ptr_array(list(pre_u)), _lib.int_array(list(widths)), len(widths),
                                    _lib.ptr(gap), _lib.ptr(relu), _lib.ptr(idx), B, _stream_ptr(device)))
    relu_h, idx_h = relu.cpu().tolist(), idx.cpu().tolist()
    return [None if r < 0 else (names[r], int(j)) for r, j in zip(relu_h, idx_h)]


def run_crown_intermediate_mlp(
    module: Any,
    input_spec: Any,
    *,
    linear_spec_C: Optional[torch.Tensor] = None,
    chunk_rows: int = 1024,
) -> Tuple[IntervalState, Dict[str, IntervalState]]:
    """CROWN whose ReLU-input bounds are themselves CROWN bounds.

    For every ReLU input after the first, in graph order: bound it with identity
    spec rows (in chunks of `chunk_rows` rows per domain), intersect with the
    current bounds, and re-propagate IBP under those constraints; then bound the
    spec rows.  Restates runtime/native_intermediate_refinement.py:923-988 on
    the device.  Returns (final bounds, refined pre-activation bounds)."""
    spec = normalize_input_spec(input_spec)
    plain = _plain_set(spec)
    if plain is not None and int(chunk_rows) > 0:
        return _crown_intermediate_query(module, spec, plain, linear_spec_C, int(chunk_rows))
    trace = ibp_trace(module, input_spec)
    chain, B, device = trace.chain, trace.B, trace.mid.device
    names = chain.relu_input_names

    def _state(k: int, l: torch.Tensor, u: torch.Tensor) -> IntervalState:
        shape = (B,) + tuple(chain.relu_shapes[k])
        return IntervalState(lower=l.reshape(shape), upper=u.reshape(shape))

    for r, name in enumerate(names):
        if r == 0:
            continue  # the first pre-activation's CROWN bound is its IBP bound
        n = chain.relu_widths[r]
        new_l = torch.empty(B, n, dtype=torch.float32, device=device)
        new_u = torch.empty(B, n, dtype=torch.float32, device=device)
        for s in range(0, n, int(chunk_rows)):
            cnt = min(int(chunk_rows), n - s)
            lo, up = crown_from_trace(trace, None, output_value=name, identity_rows=(s, cnt))
            new_l[:, s : s + cnt].copy_(lo)
            new_u[:, s : s + cnt].copy_(up)
        # the IBP sweep intersects every pre-activation with its constraint (max of the lower, min of the upper
        # bounds), so handing it the new bounds of this ReLU and the current bounds of the others is the
        # reference's intersect-then-re-propagate step
        cons = {nm: _state(k, new_l, new_u) if k == r else _state(k, trace.pre_l[k], trace.pre_u[k]) for k, nm in enumerate(names)}
        trace = ibp_trace(module, input_spec, relu_pre_constraints=cons)
        _raise_if_infeasible(trace, "ReLU pre-activation intersection")
    lo, up = crown_from_trace(trace, linear_spec_C)
    dev = normalize_input_spec(input_spec).center.device
    pre = {nm: IntervalState(lower=trace.pre_l[k].reshape((B,) + tuple(chain.relu_shapes[k])).to(dev), upper=trace.pre_u[k].reshape((B,) + tuple(chain.relu_shapes[k])).to(dev)) for k, nm in enumerate(names)}
    return IntervalState(lower=lo.to(dev), upper=up.to(dev)), pre


def _crown_intermediate_query(module: Any, spec: Any, plain, linear_spec_C: Optional[torch.Tensor], chunk_rows: int):
    """`run_crown_intermediate_mlp` in one call of the library."""
    center = spec.center
    device, B = center.device, int(center.shape[0])
    chain = compile_chain(module, center.shape[1:], device)
    C = _expand_spec(linear_spec_C, B, chain.output_width, device)
    S, R = int(C.shape[1]), len(chain.relu_widths)
    lower, upper = torch.empty(B, S, dtype=torch.float32, device=device), torch.empty(B, S, dtype=torch.float32, device=device)
    pre = {name: IntervalState(lower=torch.empty((B,) + tuple(s), dtype=torch.float32, device=device), upper=torch.empty((B,) + tuple(s), dtype=torch.float32, device=device))
           for name, s in zip(chain.relu_input_names, chain.relu_shapes)}
    infeasible = torch.empty(max(R, 1), B, dtype=torch.int32, device=device)
    chunk_rows = min(chunk_rows, max(chain.relu_widths[1:], default=1))  # the workspace holds a chunk
    nbytes = chain.lib.bf_chain_query_workspace_bytes(chain.size_handle, B, S, chunk_rows)
    ws = torch.empty(nbytes, dtype=torch.uint8, device=device)
    a, b, eps = plain
    states = [pre[n] for n in chain.relu_input_names]
    _lib.check(chain.lib.bf_chain_crown_intermediate(
        chain.handle, a.data_ptr(), _lib.ptr(b), eps, C.data_ptr(), lower.data_ptr(), upper.data_ptr(), _lib.ptr_array([t.lower for t in states]),
        _lib.ptr_array([t.upper for t in states]), infeasible.data_ptr(), chunk_rows, ws.data_ptr(), nbytes, B, S, _stream_ptr(device)))
    if R > 1 and bool(infeasible.any().item()):
        step = infeasible[int(torch.nonzero(infeasible.any(dim=1))[0])]  # the first step that found a contradiction
        bad = torch.nonzero(step).flatten().tolist()
        raise ValueError(f"infeasible ReLU pre-activation intersection: lower>upper after applying split/constraint (domains {bad[:8]}{'...' if len(bad) > 8 else ''})")
    return IntervalState(lower=lower, upper=upper), pre


@dataclass
class DomainBatchResult:
    """Per-domain outcome of one batch of BaB subdomains."""

    lower: torch.Tensor        # [B,S] best lower bounds
    upper: Optional[torch.Tensor]
    verdict: torch.Tensor      # int8 [B]: 1 = proven (min_s lower >= threshold - tol)
    infeasible: torch.Tensor   # int32 [B]: 1 = the split assignment is empty (bounds meaningless)
    alpha: List[torch.Tensor]  # best alpha per ReLU, [B,n_r] (warm start for the children)


def bound_split_domains(
    module: Any,
    input_spec: Any,
    *,
    linear_spec_C: torch.Tensor,
    relu_split_state: Optional[Mapping[str, torch.Tensor]],
    steps: int = 10,
    lr: float = 0.1,
    spec_reduce: str = "mean",
    warm_start_alpha: Optional[Sequence[torch.Tensor]] = None,
    threshold: float = 0.0,
    tol: float = 1e-6,
    want_upper: bool = True,
) -> DomainBatchResult:
    """Bound one batch of ReLU-split subdomains: IBP with the split clamps, alpha
    start from the adaptive rule (or the parents' alpha), `steps` Adam steps, verdicts.

    This is the node-batch evaluation of the BaB driver (runtime/bab.py:1250-1340 stacking
    split rows and calling run_alpha_beta_crown_mlp(per_batch_params=True) at 1323, then
    the proven test at 881-895) without the whole-batch ValueError: an infeasible
    domain is flagged in `infeasible` instead (the driver's per-node fallback,
    bab.py:1400-1460, exists only to recover from that exception).  No host
    synchronisation happens inside; tensors follow the input's device.

    The subdomains of one BaB problem share the input box and the spec rows: both may be given once (`lower`/`upper`
    of shape [1, ...], `linear_spec_C` [S,O] or [1,S,O]) with the batch size taken from the split tensors; they are
    then repeated on the device instead of being uploaded once per subdomain."""
    batch = None
    if relu_split_state:
        rows = [int(s.shape[0]) for s in relu_split_state.values() if torch.is_tensor(s) and s.dim() == 2]
        batch = max(rows) if rows else None
    trace = ibp_trace(module, input_spec, relu_split_state=relu_split_state, batch=batch)
    chain, B, device = trace.chain, trace.B, trace.mid.device
    a0 = list(warm_start_alpha) if warm_start_alpha is not None else adaptive_alpha_from_trace(trace)
    best_l, best_u, best_a, _last, _metric = alpha_crown_from_trace(
        trace, linear_spec_C, a0, steps=steps, lr=lr, spec_reduce=spec_reduce, want_upper=want_upper)
    verdict = torch.empty(B, dtype=torch.int8, device=device)
    # infeasible domains never count as proven; a NaN bound (e.g. the poison written when a tensor-core wait expired) neither
    _lib.check(chain.lib.bf_verdict_masked(_lib.ptr(best_l), float(threshold), float(tol), _lib.ptr(trace.infeasible), _lib.ptr(verdict), None, B, int(best_l.shape[1]), _stream_ptr(device)))
    out_dev = normalize_input_spec(input_spec).center.device
    if out_dev != device:
        return DomainBatchResult(best_l.to(out_dev), None if best_u is None else best_u.to(out_dev), verdict.to(out_dev), trace.infeasible.to(out_dev), [a.to(out_dev) for a in best_a])
    return DomainBatchResult(best_l, best_u, verdict, trace.infeasible, best_a)
