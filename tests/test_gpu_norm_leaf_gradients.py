"""The norm's backward pass writes a gradient of its own for each of two leaves: the same values, in memory that is not shared."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hccl_b200.ops import fused


def _leaves(rows, hidden, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = [torch.randn(rows, hidden, device="cuda", generator=g).bfloat16() for _ in range(4)]
    return t[0].requires_grad_(), t[1].requires_grad_(), torch.ones(hidden, device="cuda", dtype=torch.bfloat16, requires_grad=True), t[2], t[3]


def _norm(x, delta, w):
    return fused.add_rms_norm(x, delta, w, 1e-5)


# one row and more rows than CTAs, a group of one warp and of many, two groups per CTA; with and without a residual gradient
@pytest.mark.parametrize("rows,hidden", [(1, 8), (5, 520), (300, 1024), (1300, 8192)])
@pytest.mark.parametrize("residual", [False, True])
def test_two_leaves(rows, hidden, residual):
    x, delta, w, d_out, d_h = _leaves(rows, hidden)
    outs, grads = (0, 1) if residual else (1,), (d_out, d_h) if residual else (d_h,)
    want = torch.autograd.grad([_norm(x, delta, w)[i] for i in outs], [x, delta, w], grads)
    torch.autograd.backward([_norm(x, delta, w)[i] for i in outs], grads)
    assert torch.equal(x.grad, want[0]) and torch.equal(delta.grad, want[1]) and torch.equal(w.grad, want[2])
    assert x.grad.untyped_storage().data_ptr() != delta.grad.untyped_storage().data_ptr()
    x.grad.zero_()
    assert torch.equal(delta.grad, want[1])
    torch.autograd.backward([_norm(x, delta, w)[i] for i in outs], grads)      # x holds zeros, delta a gradient: both add up
    assert torch.equal(x.grad, want[0]) and torch.equal(delta.grad, (want[1] + want[1]))


def test_leaves_that_are_not_two():
    x, delta, w, d_out, d_h = _leaves(40, 256)
    dx = torch.autograd.grad(_norm(x, delta, w), x, [d_out, d_h])[0]
    torch.autograd.backward(_norm(x, x, w), [d_out, d_h])                       # the same leaf twice
    twice = torch.autograd.grad(_norm(x, x.detach().clone().requires_grad_(), w), x, [d_out, d_h])[0]
    assert torch.equal(x.grad, twice + twice)
    x.grad = None
    torch.autograd.backward(_norm(x, delta * 1.0, w), [d_out, d_h])             # delta is no leaf
    assert torch.equal(x.grad, dx) and torch.equal(delta.grad, dx)
    x.grad = delta.grad = None
    torch.autograd.backward(_norm(x, delta.detach(), w), [d_out, d_h])
    assert torch.equal(x.grad, dx) and delta.grad is None
    x.grad = None
    torch.autograd.backward(_norm(x, delta, w), [d_out, d_h], inputs=[delta])   # only one of them is asked for
    assert x.grad is None and torch.equal(delta.grad, dx)
    seen = []
    x.grad = delta.grad = None
    x.register_hook(lambda g: seen.append(g.clone()) or g * 2)
    torch.autograd.backward(_norm(x, delta, w), [d_out, d_h])
    assert torch.equal(seen[0], dx) and torch.equal(x.grad, dx * 2) and torch.equal(delta.grad, dx)
