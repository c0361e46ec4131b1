"""Performance cases: the bound queries a verifier sends to this backend, through its public entry points.

Every case is one call of one entry point on a network, an input set per batch element and margin specs
(logit[y] - logit[j] for every j != y).  A case is a dict of plain values:

  kind      the entry point (see `run`)
  net       input shape and layers, e.g. "784 f100 f10" or "3x32x32 c32k3s1p1 f512 f10"; "resnet" kinds add "b" blocks
  batch     input sets (or ReLU-split subdomains of one input set) bounded by the call
  eps       radius of the input sets
  steps     optimiser steps of the alpha / beta loops
  ball      input set: "box" (L-inf ball clipped to [0,1]), "linf" or "l2"

Weights are He-normal with N(0, 0.1^2) biases, inputs uniform in [0,1]; everything is drawn on the GPU from the seed.
A program that verifies one network keeps the network's compiled form, so `prepare` compiles it.
"""
from __future__ import annotations

import math
import re

import numpy as np
import torch

from boundflow_b200.crown import (bound_split_domains, compile_chain, forward_ibp_trace_mlp, needs_graph_path, run_alpha_beta_crown_mlp,
                                  run_crown_ibp_mlp, run_crown_intermediate_mlp)
from boundflow_b200.executor import CudaTaskExecutor
from boundflow_b200.ir import BFTaskModule, BoundTask, InputSpec, TaskKind, TaskOp

MNIST_MLP = "784 f100 f100 f10"
DEEP_MLP = "784 f256 f256 f256 f256 f256 f10"
WIDE_MLP = "784 f512 f512 f512 f512 f10"
MNIST_CNN = "1x28x28 c16k4s2p1 c32k4s2p1 f100 f10"
CIFAR_CNN = "3x32x32 c32k3s1p1 c32k4s2p1 c64k3s1p1 c64k4s2p1 f512 f10"
CIFAR_RESNET = "3x32x32 c16k3s1p1 b16s1 b32s2 f10"


def listed():
    return [
        # certifying one small batch of images: latency and launches count
        {"name": "crown_mlp_64", "kind": "crown", "net": MNIST_MLP, "batch": 64, "eps": 0.02, "ball": "box"},
        # the same query over a data set's worth of inputs on a wide network: throughput
        {"name": "crown_mlp_wide_3000", "kind": "crown", "net": WIDE_MLP, "batch": 3000, "eps": 0.01, "ball": "linf"},
        # interval bounds of a CNN (the executor step of a planner-scheduled run, or certified training's forward pass)
        {"name": "ibp_cnn_200", "kind": "ibp", "net": CIFAR_CNN, "batch": 200, "eps": 2.0 / 255.0, "ball": "box"},
        # CROWN with CROWN intermediate bounds on a small CNN: many sweeps of short rows
        {"name": "crown_cnn_256", "kind": "intermediate", "net": MNIST_CNN, "batch": 256, "eps": 0.1, "ball": "box"},
        # the same on a CIFAR-sized CNN: the largest query
        {"name": "crown_cifar_64", "kind": "intermediate", "net": CIFAR_CNN, "batch": 64, "eps": 2.0 / 255.0, "ball": "box"},
        # alpha-CROWN on a batch of inputs: a serial loop of small sweeps
        {"name": "alpha_mlp_128", "kind": "alpha", "net": DEEP_MLP, "batch": 128, "eps": 0.015, "steps": 20, "ball": "box"},
        # one full frontier batch of a branch-and-bound run, alpha only
        {"name": "bab_8192", "kind": "bab", "net": WIDE_MLP, "batch": 8192, "eps": 0.02, "steps": 10, "splits": 10, "ball": "box"},
        # the node batch of a branch-and-bound run that is just starting, alpha and beta; a ragged count
        {"name": "bab_nodes_37", "kind": "alpha_beta", "net": WIDE_MLP, "batch": 37, "eps": 0.02, "steps": 10, "splits": 6, "ball": "box"},
        # alpha-CROWN on a CNN: forward and backward convolutions of coefficient rows
        {"name": "alpha_cnn_48", "kind": "alpha", "net": MNIST_CNN, "batch": 48, "eps": 0.05, "steps": 10, "ball": "box"},
        # CROWN on a residual network (graph walker)
        {"name": "crown_resnet_16", "kind": "crown", "net": CIFAR_RESNET, "batch": 16, "eps": 1.0 / 255.0, "ball": "box"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("crown", "crown", "ibp", "intermediate", "alpha", "alpha", "bab", "alpha_beta", "resnet"))
    classes = rng.choice((10, 10, rng.randint(4, 20)))
    if kind == "resnet":
        c0 = rng.choice((8, 12, 16, 24))
        net = "3x%dx%d c%dk3s1p1 b%ds1 b%ds2 f%d" % ((rng.choice((16, 28, 32)),) * 2 + (c0, c0, rng.choice((c0, 2 * c0)), classes))
        return {"kind": "crown", "net": net, "batch": _log(rng, 1, 32), "eps": rng.choice((1.0, 2.0)) / 255.0, "ball": "box"}
    cnn = kind in ("ibp", "intermediate") or (kind == "alpha" and rng.random() < 0.4)
    if cnn:
        if rng.random() < 0.6:
            h, c = rng.choice((20, 28, 28, 32)), rng.choice((8, 12, 16))
            net = "1x%dx%d c%dk4s2p1 c%dk4s2p1 f%d f%d" % (h, h, c, rng.choice((c, 2 * c)), rng.randint(40, 160), classes)
        else:
            h, c = rng.choice((16, 24, 32)), rng.choice((8, 16, 24))
            net = "3x%dx%d c%dk3s1p1 c%dk%ds2p1 f%d f%d" % (h, h, c, rng.choice((c, 32)), rng.choice((3, 4)), rng.randint(60, 300), classes)
        if kind == "ibp":
            return {"kind": kind, "net": net, "batch": _log(rng, 1, 1000), "eps": rng.uniform(0.002, 0.1), "ball": rng.choice(("box", "linf"))}
        if kind == "intermediate":
            return {"kind": kind, "net": net, "batch": _log(rng, 2, 64), "eps": rng.uniform(0.004, 0.1), "ball": "box"}
        return {"kind": kind, "net": net, "batch": _log(rng, 2, 96), "eps": rng.uniform(0.004, 0.05), "steps": rng.randint(5, 20), "ball": "box"}
    width, depth = _log(rng, 40, 512), rng.randint(1, 5)
    net = " ".join(["784"] + ["f%d" % width] * depth + ["f%d" % classes])
    eps = rng.uniform(0.005, 0.02)
    if kind == "crown":
        return {"kind": kind, "net": net, "batch": _log(rng, 1, 3000), "eps": eps, "ball": rng.choice(("box", "box", "linf", "l2"))}
    if kind == "alpha":
        return {"kind": kind, "net": net, "batch": _log(rng, 1, 600), "eps": eps, "steps": rng.randint(5, 20), "ball": rng.choice(("box", "box", "linf", "l2"))}
    net = " ".join(["784"] + ["f%d" % max(width, 64)] * max(depth, 2) + ["f%d" % classes])
    if kind == "bab":
        return {"kind": kind, "net": net, "batch": _log(rng, 200, 8000), "eps": 0.02, "steps": rng.randint(3, 10), "splits": rng.randint(1, 12), "ball": "box"}
    return {"kind": kind, "net": net, "batch": _log(rng, 2, 400), "eps": 0.02, "steps": rng.randint(5, 20), "splits": rng.randint(1, 12), "ball": "box"}


# ---------------------------------------------------------------------------
# networks
# ---------------------------------------------------------------------------
def _layers(net):
    """(input shape, [(op, out channels or width, kernel, stride, padding)])"""
    first, *rest = net.split()
    out = []
    for t in rest:
        m = re.fullmatch(r"f(\d+)|c(\d+)k(\d+)s(\d+)p(\d+)|b(\d+)s(\d+)", t)
        if m is None:
            raise ValueError("bad layer %r" % t)
        g = [int(x) if x else 0 for x in m.groups()]
        out.append(("f", g[0], 0, 0, 0) if m.group(1) else ("c",) + tuple(g[1:5]) if m.group(2) else ("b", g[5], 3, g[6], 1))
    return tuple(int(d) for d in first.split("x")), out


def _build(net, g):
    """The task module of `net` with parameters drawn from generator `g`, and the multiply-adds of its affine layers."""
    shape, layers = _layers(net)
    ops, params, macs = [], {}, []
    count = [0]

    def weight(name, dims, fan):
        params["W" + name] = torch.randn(dims, generator=g, device="cuda") * math.sqrt(2.0 / fan)
        params["b" + name] = torch.randn((dims[0],), generator=g, device="cuda") * 0.1
        return ["W" + name, "b" + name]

    def conv(cur, shp, oc, k, s, p):
        count[0] += 1
        n = str(count[0])
        ho, wo = (shp[1] + 2 * p - k) // s + 1, (shp[2] + 2 * p - k) // s + 1
        ops.append(TaskOp("conv2d", "conv" + n, [cur] + weight(n, (oc, shp[0], k, k), shp[0] * k * k), ["h" + n], {"stride": (s, s), "padding": (p, p)}))
        macs.append(oc * ho * wo * shp[0] * k * k)
        return "h" + n, (oc, ho, wo)

    def relu(cur):
        ops.append(TaskOp("relu", "relu_" + cur, [cur], ["r_" + cur]))
        return "r_" + cur

    cur = "input"
    for i, (op, n, k, s, p) in enumerate(layers):
        last = i + 1 == len(layers)
        if op == "f":
            if len(shape) == 3:
                ops.append(TaskOp("flatten", "flatten", [cur], ["flat"], {"start_dim": 1, "end_dim": -1}))
                cur, shape = "flat", (shape[0] * shape[1] * shape[2],)
            count[0] += 1
            name = str(count[0])
            out = "out" if last else "h" + name
            ops.append(TaskOp("linear", "linear" + name, [cur] + weight(name, (n, shape[0]), shape[0]), [out]))
            macs.append(n * shape[0])
            cur, shape = out, (n,)
        elif op == "c":
            cur, shape = conv(cur, shape, n, k, s, p)
        else:  # residual block: conv, relu, conv, added to the input (identity, or a 1x1 projection where the shape changes)
            a, sh = conv(cur, shape, n, 3, s, 1)
            b, sh = conv(relu(a), sh, n, 3, 1, 1)
            skip = cur if (s == 1 and shape[0] == n) else conv(cur, shape, n, 1, s, 0)[0]
            ops.append(TaskOp("add", "add_" + b, [b, skip], ["s_" + b]))
            cur, shape = "s_" + b, sh
        if not last:
            cur = relu(cur)
    task = BoundTask(task_id="t0", kind=TaskKind.INTERVAL_IBP, ops=ops, input_values=["input"], output_values=["out"])
    return BFTaskModule(tasks=[task], entry_task_id="t0", bindings={"params": params}), macs


def _clean(module, x):
    """Values of every op at the points x."""
    params, env = module.bindings["params"], {"input": x}
    for op in module.get_entry_task().ops:
        a = env[op.inputs[0]]
        if op.op_type == "linear":
            y = torch.addmm(params[op.inputs[2]], a, params[op.inputs[1]].t())
        elif op.op_type == "conv2d":
            y = torch.nn.functional.conv2d(a, params[op.inputs[1]], params[op.inputs[2]], op.attrs["stride"], op.attrs["padding"])
        elif op.op_type == "relu":
            y = torch.relu(a)
        elif op.op_type == "add":
            y = a + env[op.inputs[1]]
        else:
            y = a.flatten(1)
        env[op.outputs[0]] = y
    return env


def _margins(y, classes):
    """[B, classes - 1, classes]: e_y - e_j for every j != y in ascending order."""
    eye = torch.eye(classes, device=y.device)
    j = torch.arange(classes - 1, device=y.device).expand(y.numel(), -1)
    return eye[y].unsqueeze(1) - eye[j + (j >= y.unsqueeze(1)).long()]


def _spec(x, case):
    if case["ball"] == "linf":
        return InputSpec.linf(value_name="input", center=x, eps=case["eps"])
    if case["ball"] == "l2":
        return InputSpec.l2(value_name="input", center=x, eps=10.0 * case["eps"])
    return InputSpec.box(value_name="input", lower=(x - case["eps"]).clamp(min=0.0), upper=(x + case["eps"]).clamp(max=1.0))


def prepare(case, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    module, _ = _build(case["net"], g)
    shape = _layers(case["net"])[0]
    split = case["kind"] in ("bab", "alpha_beta")
    x = torch.rand((1 if split else case["batch"],) + shape, generator=g, device="cuda")
    env = _clean(module, x)
    C = _margins(env["out"].argmax(dim=1), int(env["out"].shape[1]))
    state = {"case": case, "module": module, "C": C, "spec": _spec(x, case)}
    if not needs_graph_path(module):
        compile_chain(module, shape, x.device)
    if case["kind"] == "ibp":
        state["executor"] = CudaTaskExecutor()
    if split:
        # every subdomain fixes some of the root's unstable neurons; a "bab" frontier has random signs (some subdomains are
        # empty, which the call reports), the nodes of "alpha_beta" have the signs of a point of the input set (never empty)
        B = case["batch"]
        _, pre = forward_ibp_trace_mlp(module, state["spec"])
        names = list(pre)
        unstable = torch.cat([((s.lower < 0) & (s.upper > 0)).reshape(-1) for s in pre.values()])
        score = torch.rand((B, unstable.numel()), generator=g, device="cuda") * unstable
        pick = torch.zeros_like(score, dtype=torch.bool).scatter_(1, score.topk(case["splits"], dim=1).indices, True) & unstable
        if case["kind"] == "bab":
            sign = torch.rand(score.shape, generator=g, device="cuda") < 0.5
        else:
            box = state["spec"].perturbation
            points = box.lower + (box.upper - box.lower) * torch.rand((B,) + shape, generator=g, device="cuda")
            at = _clean(module, points)
            sign = torch.cat([at[n] > 0 for n in names], dim=1)
        s = torch.where(sign, 1, -1).to(torch.int8) * pick
        state["splits"] = dict(zip(names, (t.contiguous() for t in s.split([p.lower.shape[1] for p in pre.values()], dim=1))))
        if case["kind"] == "alpha_beta":
            state["spec"] = InputSpec.box(value_name="input", lower=box.lower.expand(B, -1).contiguous(), upper=box.upper.expand(B, -1).contiguous())
            state["C"] = C.expand(B, -1, -1).contiguous()
            state["names"] = {n: i for i, n in enumerate(names)}
    return state


def run(state):
    case, module, spec, C = state["case"], state["module"], state["spec"], state["C"]
    if case["kind"] == "crown":
        r = run_crown_ibp_mlp(module, spec, linear_spec_C=C)
        return {"lower": r.lower, "upper": r.upper}
    if case["kind"] == "ibp":
        r = state["executor"].run_ibp(module, spec)
        return {"lower": r.lower, "upper": r.upper}
    if case["kind"] == "intermediate":
        r, pre = run_crown_intermediate_mlp(module, spec, linear_spec_C=C)
        return {"lower": r.lower, "upper": r.upper, "pre": {n: [s.lower, s.upper] for n, s in pre.items()}}
    if case["kind"] == "alpha":
        r, alpha, _, _ = run_alpha_beta_crown_mlp(module, spec, linear_spec_C=C, steps=case["steps"], lr=0.1, per_batch_params=True)
        return {"lower": r.lower, "upper": r.upper, "alpha": alpha.alpha_by_relu_input}
    if case["kind"] == "bab":
        r = bound_split_domains(module, spec, linear_spec_C=C, relu_split_state=state["splits"], steps=case["steps"], lr=0.1)
        return {"lower": r.lower, "upper": r.upper, "verdict": r.verdict, "infeasible": r.infeasible, "alpha": r.alpha}
    r, alpha, beta, stats = run_alpha_beta_crown_mlp(module, spec, linear_spec_C=C, relu_split_state=state["splits"], steps=case["steps"], lr=0.1,
                                                     per_batch_params=True)
    branch = np.array([(-1, -1) if c is None else (state["names"][c[0]], c[1]) for c in stats.branch_choices])
    return {"lower": r.lower, "upper": r.upper, "alpha": alpha.alpha_by_relu_input, "beta": beta.beta_by_relu_input, "branch": branch}


# ---------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------
def _sizes(case):
    """(input elements, [macs per affine layer], [elements of every affine layer's output], parameters, specs per input)"""
    shape, layers = _layers(case["net"])
    n0 = math.prod(shape)
    macs, widths, params = [], [], 0

    def conv(shp, oc, k, s, p):
        nonlocal params
        ho, wo = (shp[1] + 2 * p - k) // s + 1, (shp[2] + 2 * p - k) // s + 1
        params += oc * (shp[0] * k * k + 1)
        macs.append(oc * ho * wo * shp[0] * k * k)
        widths.append(oc * ho * wo)
        return oc, ho, wo

    for op, n, k, s, p in layers:
        if op == "f":
            macs.append(n * math.prod(shape))
            params += n * (math.prod(shape) + 1)
            widths.append(n)
            shape = (n,)
        elif op == "c":
            shape = conv(shape, n, k, s, p)
        else:
            if s != 1 or shape[0] != n:
                conv(shape, n, 1, s, 0)
            shape = conv(conv(shape, n, 3, s, 1), n, 3, 1, 1)
    return n0, macs, widths, params, widths[-1] - 1


def _identity_rows_macs(case):
    """Multiply-adds of one backward sweep of identity rows for every ReLU input after the first, per input set: a row that
    starts at a conv neuron only has a receptive field's worth of coefficients in the layers below it."""
    shape, layers = _layers(case["net"])
    shapes = [shape]
    for op, n, k, s, p in layers:
        shapes.append((n,) if op == "f" else (n, (shapes[-1][1] + 2 * p - k) // s + 1, (shapes[-1][2] + 2 * p - k) // s + 1))
    total = 0
    for top in range(1, len(layers) - 1):
        rows = math.prod(shapes[top + 1])
        span = 1 if layers[top][0] == "c" else None   # side of the square of coefficients that can be non-zero, None: all
        for i in range(top, -1, -1):
            op, n, k, s, _ = layers[i]
            if i != top:  # the first step copies weights
                if op == "f":
                    total += rows * n * math.prod(shapes[i])
                else:
                    pixels = shapes[i + 1][1] * shapes[i + 1][2] if span is None else min(span, shapes[i + 1][1]) * min(span, shapes[i + 1][2])
                    total += rows * pixels * n * shapes[i][0] * k * k
            if span is not None and op == "c":
                span = (span - 1) * s + k
    return total


def work(case):
    n0, macs, widths, params, S = _sizes(case)
    B, P, hidden = case["batch"], sum(macs), sum(widths[:-1])
    sets = 1 if case["kind"] == "bab" else B
    io = 4 * params + 8 * sets * n0
    ibp = 4 * B * P                      # centre and radius
    sweep = 2 * B * S * P                # one side of the spec rows through every layer
    bounds = 8 * B * S
    if case["kind"] == "ibp":
        return {"bytes": io + 8 * B * widths[-1], "flops": ibp}
    io += 4 * sets * S * (S + 1) + bounds
    if case["kind"] == "crown":
        return {"bytes": io, "flops": ibp + 2 * sweep}
    if case["kind"] == "intermediate":
        return {"bytes": io + 8 * B * hidden, "flops": ibp + 4 * B * _identity_rows_macs(case) + 2 * sweep}
    # steps + 1 lower sweeps, one upper sweep, one gradient sweep (all layers but the last) per step
    loop = (case["steps"] + 2) * sweep + case["steps"] * 2 * B * S * (P - macs[-1])
    io += 4 * B * hidden * (2 if case["kind"] == "alpha_beta" else 1) + (B * hidden if "splits" in case else 0)
    return {"bytes": io, "flops": ibp + loop}


def tolerance(case):
    # Bounds: 2e-7 to 5e-7 (2-norm) from a float64 evaluation on every network above.
    if case["kind"] in ("crown", "ibp", "intermediate"):
        return {"rel": 2e-6, "max": 1e-4}
    # An Adam step moves a parameter by about lr whatever the size of its gradient, so a parameter whose gradient vanishes
    # up to rounding may end elsewhere (max).  With the sums in another order the alphas and betas of these loops differ by up to
    # 6e-3 (2-norm), their bounds by 1e-7 to 3e-5.
    return {"rel": 2e-2, "max": 0.99, "differ": 1e-3}
