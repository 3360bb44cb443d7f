"""Single-pass bf16 kernels for the memory-bound pieces of a decoder layer, with autograd:

* ``add_rms_norm(x, delta, weight, eps)`` -> ``(x + delta, rms_norm(x + delta) * weight)`` (``delta=None``: norm only)
* ``swiglu(gate_up)`` -> ``silu(gate) * up`` for ``gate_up = [gate | up]`` along the last dimension
* ``rope(x, cos, sin)`` -> rotary embedding ("rotate halves") of ``x [S, heads, D]``; ``x`` may be a column slice
  of a wider projection output (row stride larger than ``heads * D``)
* ``embedding(ids, table)`` -> ``table[ids]`` with the table's gradient written in one pass over its rows
* ``rope_qkv(qkv, cos, sin, hq, hkv)`` -> ``(q, k, v)`` of a projection output ``[S, (hq + 2 hkv) * D]`` with q and k rotated

CUDA bf16 tensors run the hand-written kernels (csrc/kernels/fused_elementwise.cu); anything else (CPU tensors, other
dtypes, hidden > 8192) takes the equivalent PyTorch expression, which is also the reference the tests compare against.
"""
from __future__ import annotations

import ctypes
import sys
import types

import torch
import torch.nn.functional as F

from .. import _calls
from .._lib import lib
from ..comm import _check


_launches = 0


def _count(n=1):
    global _launches
    _launches += n


class _Module(types.ModuleType):
    """This module: its count of launches is made of two, and can be set like the variable it looks like."""

    @property
    def LAUNCHES(self):          # kernels of this module launched so far (benchmark accounting)
        return _launches + _calls.launches()

    @LAUNCHES.setter
    def LAUNCHES(self, n):
        global _launches
        _launches = n - _calls.launches()


sys.modules[__name__].__class__ = _Module


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else ctypes.c_void_p(0)


def _s():
    return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(torch.cuda.current_device()))


def _native(*tensors, hidden=None) -> bool:
    for t in tensors:
        if t is None:
            continue
        if not (t.is_cuda and t.dtype == torch.bfloat16):
            return False
    if hidden is not None and (hidden % 8 != 0 or hidden > 8192):
        return False
    if not hasattr(lib, "HcclFusedRope"):
        raise RuntimeError("libhccl_b200.so predates the fused element-wise kernels: rebuild it with `python hccl_b200/build.py`")
    return True


# ----------------------------------------------------------------------------- reference expressions
def add_rms_norm_reference(x, delta, weight, eps):
    x_out = x if delta is None else x + delta
    return x_out, F.rms_norm(x_out, (x_out.shape[-1],), weight, eps)


def swiglu_reference(gate_up):
    g, u = gate_up.chunk(2, dim=-1)
    return F.silu(g) * u


def rope_reference(x, cos, sin):
    d = x.shape[-1] // 2
    x1, x2 = x[..., :d].float(), x[..., d:].float()
    c, s = cos[:, None, :], sin[:, None, :]
    return torch.cat((x1 * c - x2 * s, x2 * c + x1 * s), dim=-1).to(x.dtype)


# ----------------------------------------------------------------------------- autograd functions
def _kept_apart(*nodes) -> bool:
    """The gradients of these inputs end in as many leaves that hold none yet: each leaf keeps the tensor it is given if nobody
    else has it, and copies it otherwise.  (Under ``autograd.grad`` the leaves keep nothing: the engine refuses to say.)"""
    try:
        return all(hasattr(n, "variable") and n.variable.grad is None and torch._C._will_engine_execute_node(n) for n in nodes) and len(set(nodes)) == len(nodes)
    except RuntimeError:
        return False


class _AddRmsNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, delta, weight, eps):
        ctx.has_delta = delta is not None
        r = _calls.add_rms_norm(x, delta, weight, eps)
        if r is not None:
            x_out, h, rstd = _calls.result(r, "HcclFusedAddRmsNormFwd")
            _count()
            ctx.save_for_backward(x_out, weight, rstd)
            return (x_out, h) if ctx.has_delta else h
        rows, hidden = x.numel() // x.shape[-1], x.shape[-1]
        x = x.contiguous()
        h = torch.empty_like(x)
        rstd = torch.empty(rows, device=x.device, dtype=torch.float32)
        if delta is not None:
            delta = delta.contiguous()
            x_out = torch.empty_like(x)
        else:
            x_out = x
        _check(lib.HcclFusedAddRmsNormFwd(_p(x), _p(delta), _p(weight), _p(x_out) if delta is not None else ctypes.c_void_p(0), _p(h), _p(rstd),
                                          rows, hidden, float(eps), _s()), "HcclFusedAddRmsNormFwd")
        _count()
        ctx.save_for_backward(x_out, weight, rstd)
        return (x_out, h) if delta is not None else h        # without delta the input itself is the residual stream

    @staticmethod
    def backward(ctx, *grads):
        dx_out, dh = grads if ctx.has_delta else (None, grads[0])
        x_out, weight, rstd = ctx.saved_tensors
        rows, hidden = x_out.numel() // x_out.shape[-1], x_out.shape[-1]
        if dh is None:
            dh = torch.zeros_like(x_out)
        dh = dh.contiguous()
        extra = dx_out.contiguous() if dx_out is not None else None
        twice = ctx.has_delta and hasattr(lib, "HcclFusedRmsNormBwdCopy") and _kept_apart(ctx.next_functions[0][0], ctx.next_functions[1][0])
        r = _calls.rms_norm_bwd(dh, x_out, weight, rstd, extra, twice)
        if r is not None:
            dx, dw, copy = _calls.result(r, "HcclFusedRmsNormBwdCopy")
            _count(2)
            return dx, (copy if ctx.has_delta else None), dw, None
        dx = torch.empty_like(x_out)
        copy = torch.empty_like(x_out) if twice else dx
        dw = torch.empty_like(weight)
        n_part = lib.HcclFusedRmsNormBwdPartials(rows)
        partial = torch.empty((n_part, hidden), device=x_out.device, dtype=torch.float32)
        if twice:
            _check(lib.HcclFusedRmsNormBwdCopy(_p(dh), _p(x_out), _p(weight), _p(rstd), _p(extra), _p(dx), _p(copy), _p(partial), _p(dw), rows, hidden,
                                               _s()), "HcclFusedRmsNormBwdCopy")
        else:                                   # also what a library without the other has
            _check(lib.HcclFusedRmsNormBwd(_p(dh), _p(x_out), _p(weight), _p(rstd), _p(extra), _p(dx), _p(partial), _p(dw), rows, hidden, _s()),
                   "HcclFusedRmsNormBwd")
        _count(2)
        return dx, (copy if ctx.has_delta else None), dw, None


class _Swiglu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gate_up):
        gate_up = gate_up.contiguous()
        out = _calls.swiglu_fwd(gate_up)
        if out is not None:
            out = _calls.result(out, "HcclFusedSwigluFwd")
            _count()
            ctx.save_for_backward(gate_up)
            return out
        f = gate_up.shape[-1] // 2
        rows = gate_up.numel() // gate_up.shape[-1]
        out = torch.empty(gate_up.shape[:-1] + (f,), device=gate_up.device, dtype=gate_up.dtype)
        _check(lib.HcclFusedSwigluFwd(_p(gate_up), _p(out), rows, f, _s()), "HcclFusedSwigluFwd")
        _count()
        ctx.save_for_backward(gate_up)
        return out

    @staticmethod
    def backward(ctx, dout):
        (gate_up,) = ctx.saved_tensors
        dgu = _calls.swiglu_bwd(gate_up, dout.contiguous())
        if dgu is not None:
            dgu = _calls.result(dgu, "HcclFusedSwigluBwd")
            _count()
            return dgu
        f = gate_up.shape[-1] // 2
        rows = gate_up.numel() // gate_up.shape[-1]
        dgu = torch.empty_like(gate_up)
        _check(lib.HcclFusedSwigluBwd(_p(gate_up), _p(dout.contiguous()), _p(dgu), rows, f, _s()), "HcclFusedSwigluBwd")
        _count()
        return dgu


class _Rope(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, cos, sin):
        s, nh, d = x.shape
        assert x.stride(2) == 1 and x.stride(1) == d, "rope: heads must be packed inside a row"
        out = _calls.rope(x, cos, sin, False)
        if out is not None:
            out = _calls.result(out, "HcclFusedRope")
            _count()
            ctx.save_for_backward(cos, sin)
            return out
        out = torch.empty((s, nh, d), device=x.device, dtype=x.dtype)
        _check(lib.HcclFusedRope(_p(x), x.stride(0), _p(out), nh * d, _p(cos), _p(sin), s, nh, d, 0, _s()), "HcclFusedRope")
        _count()
        ctx.save_for_backward(cos, sin)
        return out

    @staticmethod
    def backward(ctx, dout):
        cos, sin = ctx.saved_tensors
        s, nh, d = dout.shape
        dout = dout.contiguous()
        dx = _calls.rope(dout, cos, sin, True)
        if dx is not None:
            dx = _calls.result(dx, "HcclFusedRope")
            _count()
            return dx, None, None
        dx = torch.empty_like(dout)
        _check(lib.HcclFusedRope(_p(dout), nh * d, _p(dx), nh * d, _p(cos), _p(sin), s, nh, d, 1, _s()), "HcclFusedRope")
        _count()
        return dx, None, None


class _RopeQkv(torch.autograd.Function):
    """Query, key and value heads of one projection output.  The backward pass writes the three gradients side by side into
    one tensor; slicing the output instead makes autograd fill three zero tensors of its full size and add them up."""

    @staticmethod
    def forward(ctx, qkv, cos, sin, hq, hkv):
        s, d = qkv.shape[0], qkv.shape[1] // (hq + 2 * hkv)
        out = []
        for first, heads in ((0, hq), (hq, hkv)):
            o = torch.empty((s, heads, d), device=qkv.device, dtype=qkv.dtype)
            _check(lib.HcclFusedRope(_p(qkv[:, first * d:]), qkv.stride(0), _p(o), heads * d, _p(cos), _p(sin), s, heads, d, 0, _s()), "HcclFusedRope")
            out.append(o)
        _count(2)
        ctx.save_for_backward(cos, sin)
        ctx.set_materialize_grads(False)        # an output that nothing used has no gradient: its part is filled, not rotated
        ctx.heads = (hq, hkv, d)
        return out[0], out[1], qkv[:, (hq + hkv) * d:].view(s, hkv, d)

    @staticmethod
    def backward(ctx, dq, dk, dv):
        cos, sin = ctx.saved_tensors
        hq, hkv, d = ctx.heads
        s = cos.shape[0]
        width = (hq + 2 * hkv) * d
        like = next((g for g in (dq, dk, dv) if g is not None), None)
        if like is None:
            return None, None, None, None, None
        dqkv = torch.empty((s, width), device=like.device, dtype=like.dtype)
        for first, heads, g in ((0, hq, dq), (hq, hkv, dk)):
            part = dqkv[:, first * d:(first + heads) * d]
            if g is None:
                part.zero_()
                continue
            # rows and heads as attention left them where the kernel can read that, else a packed copy
            if not (g.stride(2) == 1 and g.stride(1) == d and g.stride(0) % 8 == 0 and g.data_ptr() % 16 == 0):
                g = g.contiguous()
            _check(lib.HcclFusedRope(_p(g), g.stride(0), _p(part), width, _p(cos), _p(sin), s, heads, d, 1, _s()), "HcclFusedRope")
            _count()
        part = dqkv[:, (hq + hkv) * d:].view(s, hkv, d)
        part.copy_(dv) if dv is not None else part.zero_()
        return dqkv, None, None, None, None


# ----------------------------------------------------------------------------- public functions
def add_rms_norm(x, delta, weight, eps: float = 1e-5, use_kernels: bool = True):
    """``x_out = x + delta`` (``delta`` may be None) and ``h = rms_norm(x_out) * weight`` in one pass; returns both."""
    global _launches
    r = _calls.add_rms_norm(x, delta, weight, eps) if use_kernels else None
    if r is not None:                                        # no gradient is recorded: no autograd function either
        if type(r) is int:
            _check(r, "HcclFusedAddRmsNormFwd")
        _launches += 1
        return r[0], r[1]
    r = _calls.add_rms_norm_grad(x, delta, weight, eps) if use_kernels else None
    if r is not None:
        x_out, h = _calls.result(r, "HcclFusedAddRmsNormFwd")
        _count()
        return x_out, h
    if use_kernels and _native(x, delta, weight, hidden=x.shape[-1]):
        if delta is None:
            return x, _AddRmsNorm.apply(x, None, weight, eps)
        return _AddRmsNorm.apply(x, delta, weight, eps)
    return add_rms_norm_reference(x, delta, weight, eps)


def swiglu(gate_up, use_kernels: bool = True):
    global _launches
    out = _calls.swiglu_fwd(gate_up) if use_kernels else None
    if out is not None or use_kernels and (out := _calls.swiglu_grad(gate_up)) is not None:
        if type(out) is int:
            _check(out, "HcclFusedSwigluFwd")
        _launches += 1
        return out
    if use_kernels and _native(gate_up) and (gate_up.shape[-1] // 2) % 8 == 0:
        return _Swiglu.apply(gate_up)
    return swiglu_reference(gate_up)


def _rope_table(t, x) -> bool:
    """A table the kernel can read for every row of x; others (a row that broadcasts, one on the host) go to PyTorch."""
    return t.is_cuda and t.dtype == torch.float32 and t.is_contiguous() and t.numel() >= x.shape[0] * (x.shape[-1] // 2)


def rope(x, cos, sin, use_kernels: bool = True):
    """x [S, heads, D] (row stride may exceed heads * D), cos / sin fp32 [S, D / 2]."""
    global _launches
    out = _calls.rope(x, cos, sin, False) if use_kernels else None
    if out is not None or use_kernels and (out := _calls.rope_grad(x, cos, sin)) is not None:
        if type(out) is int:
            _check(out, "HcclFusedRope")
        _launches += 1
        return out
    if (use_kernels and _native(x) and x.shape[-1] % 16 == 0 and x.stride(2) == 1 and x.stride(1) == x.shape[-1] and x.stride(0) % 8 == 0
            and x.data_ptr() % 16 == 0 and _rope_table(cos, x) and _rope_table(sin, x)):
        return _Rope.apply(x, cos, sin)
    return rope_reference(x, cos, sin)


def rope_qkv(qkv, cos, sin, hq: int, hkv: int, use_kernels: bool = True):
    """Splits ``qkv [S, (hq + 2 hkv) * D]`` into heads and rotates q and k: ``([S, hq, D], [S, hkv, D], [S, hkv, D])``."""
    s, d = qkv.shape[0], qkv.shape[1] // (hq + 2 * hkv)
    if (use_kernels and _native(qkv) and d % 16 == 0 and hkv > 0 and s > 0 and qkv.is_contiguous() and qkv.data_ptr() % 16 == 0
            and cos.is_cuda and sin.is_cuda and cos.dtype == torch.float32 and sin.dtype == torch.float32 and cos.shape == sin.shape == (s, d // 2)
            and cos.is_contiguous() and sin.is_contiguous()):
        return _RopeQkv.apply(qkv, cos, sin, hq, hkv)
    q = rope(qkv[:, :hq * d].view(s, hq, d), cos, sin, use_kernels=use_kernels)
    k = rope(qkv[:, hq * d:(hq + hkv) * d].view(s, hkv, d), cos, sin, use_kernels=use_kernels)
    return q, k, qkv[:, (hq + hkv) * d:].view(s, hkv, d)


def embedding(ids, table, use_kernels: bool = True):
    """Rows ``ids`` of ``table [vocab, hidden]``.  Up to 8192 tokens the table's gradient is this library's kernel."""
    out = _calls.embedding(ids, table) if use_kernels else None
    return out if out is not None else F.embedding(ids, table)
