"""The matmul, norm, SwiGLU, rotary and routing kernels at the edges of their tiles, groups and rings, against float64.

Tolerance: every compared tensor is rounded to bf16 once, which is off by at most half a unit in the last place, 2^-8 =
3.9e-3 of an element and so of the 2-norm of any tensor (about 1.7e-3 of one with spread-out values); sums are fp32 and add
less than 1e-4 at these lengths.  The norm's output is taken of a sum that is itself rounded, which the reference repeats.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hccl_b200.ops import fused

ONE_ROUNDING = 2.0 ** -8 + 1e-4


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def _rnd(g, *shape, std=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * std).bfloat16()


@pytest.mark.parametrize("hidden", [8, 256, 512, 520, 1024, 1032, 4096, 4104, 8192])
@pytest.mark.parametrize("rows", [1, 5, 149, 1300])
@pytest.mark.parametrize("with_delta", [False, True])
def test_add_rms_norm_groups(rows, hidden, with_delta):
    g = torch.Generator(device="cuda").manual_seed(rows * 3 + hidden)
    x = _rnd(g, rows, hidden).requires_grad_()
    delta = _rnd(g, rows, hidden, std=0.5).requires_grad_() if with_delta else None
    w = (1 + 0.1 * torch.randn(hidden, device="cuda", generator=g)).bfloat16().requires_grad_()
    d_out, d_h = _rnd(g, rows, hidden), _rnd(g, rows, hidden)
    x_out, h = fused.add_rms_norm(x, delta, w, 1e-5)
    torch.autograd.backward([x_out, h] if with_delta else [h], [d_out, d_h] if with_delta else [d_h])
    s = (x.detach() + delta.detach() if with_delta else x.detach())
    assert torch.equal(x_out.detach(), s)
    s, w64 = s.double().requires_grad_(), w.detach().double().requires_grad_()
    h64 = s * torch.rsqrt(s.pow(2).mean(-1, keepdim=True) + 1e-5) * w64
    dx, dw = torch.autograd.grad(h64, [s, w64], d_h.double())
    if with_delta:
        dx = dx + d_out.double()
        assert torch.equal(delta.grad, x.grad)
    assert _rel(h.detach(), h64.detach()) <= ONE_ROUNDING
    assert _rel(w.grad, dw) <= ONE_ROUNDING
    # without the residual gradient a row of 8 elements is a difference of nearly equal terms: the fp32 terms of size |dh|
    # are what the error is relative to
    assert (x.grad.double() - dx).norm().item() <= ONE_ROUNDING * dx.norm().item() + 1e-6 * d_h.double().norm().item()
