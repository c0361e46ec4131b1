"""The optimiser kernel's rounding, bit for bit: an Adam step divides by the root of its own second moment, so that the last bit
of a moment decides on the whole step of a small gradient, and with it on the trajectory of an alpha / beta loop.

The expected bits are formed in float64: a product of two float32 values is exact there, so rounding to float32 after one operation
is that operation's float32 rounding, and `fma` (product and sum, then one rounding) can differ from it only where the float64 sum
itself lies within 2^-53 of a tie.
"""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from boundflow_b200.csrc import build

    build.build()
    return torch.device("cuda", 0)


def _f32(v):
    return float(np.float32(v))


def _mul(a, b):
    return (a.double() * b).float()


def _fma(a, b, c):
    return (a.double() * (b if isinstance(b, float) else b.double()) + c.double()).float()


def _step(x, m, v, grad, sign, fused, keep_v, t, lr, S):
    """(x', m', v') of one step before the projection; `fused` and `keep_v` as in the kernel's comments."""
    bc1, bc2 = 1 - 0.9 ** (t + 1), 1 - 0.999 ** (t + 1)
    scale, o1, o2 = _f32(np.float32(-1) / np.float32(S)), _f32(1 - 0.9), _f32(1 - 0.999)
    g = _mul(_mul(grad, scale), sign)
    d = torch.where(fused, _fma(grad, scale, -m), (g.double() - m.double()).float())
    m1 = _fma(d, o1, m)
    og = _mul(g, o2)
    v1 = torch.where(keep_v, _fma(v, _f32(0.999), _mul(og, g.double())), _fma(og, g, _mul(v, _f32(0.999))))
    den = ((v1.double().sqrt().float().double() / _f32(math.sqrt(bc2))).float().double() + _f32(1e-8)).float()
    q = (m1.double() / den.double()).float()
    return _fma(q, -_f32(_f32(lr) / bc1), x), m1, v1


@pytest.mark.parametrize("B,n", [(1, 1), (3, 45), (400, 512), (70, 516), (5, 2050)])
@pytest.mark.parametrize("t", [0, 7])
def test_adam_step_bits(dev, B, n, t):
    from boundflow_b200 import _lib

    lib, lr, S = _lib.load(), 0.1, 9
    g = torch.Generator("cuda").manual_seed(B + n)
    rand = lambda: torch.rand(B, n, generator=g, device=dev)
    x, m, v, grad = rand(), rand() * 0.2 - 0.1, rand() * 0.01, rand() * 2 - 1
    lo, up = rand() * 2 - 1.5, rand() * 2 - 0.5
    improve = (torch.arange(B, device=dev) % 2).int()
    column = torch.arange(n, device=dev)
    four = torch.full((B, n), n % 4 == 0, device=dev)
    # alpha
    a1, m1, v1, g1, slope, best = x.clone(), m.clone(), v.clone(), grad.clone(), torch.empty_like(x), torch.full_like(x, -1.0)
    _lib.check(lib.bf_alpha_adam_step(a1.data_ptr(), m1.data_ptr(), v1.data_ptr(), g1.data_ptr(), improve.data_ptr(), best.data_ptr(), lo.data_ptr(),
                                      up.data_ptr(), slope.data_ptr(), t, lr, 0, S, 1, B, n, None))
    want, wm, wv = _step(x, m, v, grad, 1.0, four & (column % 4 != 0), ~four, t, lr, S)
    want = want.clamp(0, 1)
    assert torch.equal(m1, wm) and torch.equal(v1, wv) and torch.equal(a1, want)
    assert torch.equal(slope, torch.where(up <= 0, torch.zeros_like(x), torch.where(lo >= 0, torch.ones_like(x), want)))
    assert torch.equal(best, torch.where(improve[:, None] != 0, x, torch.full_like(x, -1.0))) and not g1.any()
    # beta
    split = torch.randint(-1, 2, (B, n), generator=g, device=dev, dtype=torch.int8)
    b1, m1, v1, g1, add = x.clone(), m.clone(), v.clone(), grad.clone(), torch.empty_like(x)
    _lib.check(lib.bf_beta_adam_step(b1.data_ptr(), m1.data_ptr(), v1.data_ptr(), g1.data_ptr(), split.data_ptr(), n, None, None, add.data_ptr(), t, lr, 0, S,
                                     1, B, n, None))
    none = torch.zeros_like(four)
    want, wm, wv = _step(x, m, v, grad, -split.double(), none, ~none, t, lr, S)
    want = want.clamp(min=0)
    assert torch.equal(m1, wm) and torch.equal(v1, wv) and torch.equal(b1, want)
    assert torch.equal(add, -want * split) and not g1.any()
