"""Operators that record gradients: the native nodes against the Python functions that they stand in for."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hccl_b200 import _calls
from hccl_b200.comm import HcclError
from hccl_b200.ops import fused
from hccl_b200.parallel import ColumnParallelLinear, RowParallelLinear, TPContext

NAMES = ("add_rms_norm_grad", "swiglu_grad", "rope_grad", "linear")


def _rnd(*shape, seed=0):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)).bfloat16()


@pytest.fixture(params=["native", "python"])
def way(request, monkeypatch):
    if request.param == "python":
        for name in NAMES + ("embedding",):
            monkeypatch.setattr(_calls, name, _calls._nothing)
    else:
        assert _calls._module is not None
    return request.param


def _layer(seed=0, rows=40):
    """Every operator once, leaves and results that are not leaves, a strided head slice, a norm without a residual."""
    torch.manual_seed(seed)
    ctx = TPContext(None)
    up, down = ColumnParallelLinear(256, 2 * 512, ctx, "up"), RowParallelLinear(512, 256, ctx, "down")
    leaves = [_rnd(rows, 256, seed=1), _rnd(rows, 256, seed=2), _rnd(256, seed=3), _rnd(256, seed=4)]
    leaves = [t.requires_grad_() for t in leaves] + [up.weight, down.weight]
    ang = torch.rand(rows, 32, device="cuda") * 6.28
    x, h = fused.add_rms_norm(leaves[0], leaves[1], leaves[2], 1e-5)
    y = down(fused.swiglu(up(h)))
    h = fused.add_rms_norm(x + y, None, leaves[3], 1e-5)[1]
    r = fused.rope(h[:, 64:].view(rows, 3, 64), ang.cos(), ang.sin())
    return leaves, [x, h, r], ctx


def _grads(how):
    before = fused.LAUNCHES
    leaves, outs, ctx = _layer()
    ups = [_rnd(*o.shape, seed=10 + i) for i, o in enumerate(outs)]
    ups[2] = ups[2].transpose(0, 1).contiguous().transpose(0, 1)                # not packed
    if how == "grad":
        got = list(torch.autograd.grad(outs, leaves, ups))
    else:
        torch.autograd.backward(outs, ups, retain_graph=True)
        if how == "twice":
            torch.autograd.backward(outs[2:], ups[2:])
        got = [t.grad for t in leaves]
    return [o.detach() for o in outs] + got, fused.LAUNCHES - before, ctx.launches


@pytest.mark.parametrize("how", ["grad", "backward", "twice"])
def test_both_ways_give_the_same(how, monkeypatch):
    native, launched, linear = _grads(how)
    for name in NAMES:
        monkeypatch.setattr(_calls, name, _calls._nothing)
    general, launched2, linear2 = _grads(how)
    assert all(a.shape == b.shape and a.dtype == b.dtype and torch.equal(a, b) for a, b in zip(native, general, strict=True))
    assert (launched, linear) == (launched2, linear2)


def test_the_native_nodes_are_the_ones_that_run():
    _, (x, h, r), _ = _layer()
    assert [o.grad_fn.name() for o in (x, h, r)] == ["_AddRmsNormBackward", "_AddRmsNormBackward", "_RopeBackward"]
    assert not any(isinstance(o.grad_fn, torch.autograd.function.BackwardCFunction) for o in (x, h, r))


def test_only_some_outputs_and_inputs(way):
    x, d, w = _rnd(9, 64, seed=1).requires_grad_(), _rnd(9, 64, seed=2), _rnd(64, seed=3)
    x_out, h = fused.add_rms_norm(x, d, w, 1e-5)
    assert torch.equal(torch.autograd.grad(x_out, x, torch.ones_like(x_out), retain_graph=True)[0], torch.ones_like(x))
    a, b = torch.autograd.grad(h.float().sum(), x, retain_graph=True)[0], torch.autograd.grad(h.float().sum(), x)[0]
    assert torch.equal(a, b) and d.grad is None and w.grad is None
    with torch.no_grad():
        assert not fused.add_rms_norm(x, d, w, 1e-5)[1].requires_grad


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, g):
        return None


def test_outputs_whose_gradient_is_undefined(way):
    """Every leaf gets zeros, not nothing: an optimizer steps the ones and skips the others."""
    leaves, outs, _ = _layer()
    sum(_NoGradient.apply(o).float().sum() for o in outs).backward()
    assert all(t.grad is not None and not t.grad.any() for t in leaves)
    for f, x in ((fused.swiglu, _rnd(8, 64)), (lambda t: fused.rope(t.view(8, 1, 64), torch.ones(8, 32, device="cuda"), torch.zeros(8, 32, device="cuda")), _rnd(8, 64)),
                 (ColumnParallelLinear(64, 128, TPContext(None), "up"), _rnd(8, 64))):
        x.requires_grad_()
        _NoGradient.apply(f(x)).sum().backward()
        assert x.grad is not None and not x.grad.any()


def test_what_autograd_checks_is_checked(way):
    x, w = _rnd(9, 64).requires_grad_(), _rnd(64).requires_grad_()
    y = fused.swiglu(fused.add_rms_norm(x * 1, None, w, 1e-5)[1])
    y.sum().backward()
    with pytest.raises(RuntimeError, match="second time"):
        y.sum().backward()
    gate_up = x * 1
    y = fused.swiglu(gate_up)
    gate_up.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()
    seen = []
    h = fused.add_rms_norm(x, None, w, 1e-5)[1]
    h.register_hook(lambda g: seen.append(g) or 2 * g)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t) or t.cpu(), lambda t: t.cuda()):
        y = fused.swiglu(h)
    assert len(seen) == 1 and torch.equal(seen[0], h)
    y.sum().backward()
    assert len(seen) == 2


def test_compiled_backward_passes(way):
    """Compiled autograd takes the nodes into its graph, which then launches what the nodes launch."""
    from torch._dynamo import compiled_autograd
    want, launched = None, []
    for compiled in (False, True, True):                                         # the second time the graph is used again
        before = fused.LAUNCHES
        leaves, outs, ctx = _layer()                                             # no tensor has more than two uses: sums have one order
        table = _rnd(64, 256, seed=5).requires_grad_()
        loss = sum(o.float().square().sum() for o in outs) + fused.embedding(torch.arange(39, -1, -1, device="cuda"), table).float().square().sum()
        if compiled:
            with compiled_autograd._enable(torch.compile(backend="eager")):
                loss.backward()
        else:
            loss.backward()
        launched.append(fused.LAUNCHES - before + ctx.launches)
        got = [t.grad for t in leaves + [table]]
        want = want or got
        assert all(torch.equal(a, b) for a, b in zip(got, want, strict=True))
        assert len({t.data_ptr() for t in got}) == len(got)                      # every leaf has a gradient of its own
    assert launched[1:] == [launched[0] - (2 if way == "native" else 0)] * 2    # the embedding's gradient is PyTorch's there


def test_the_operators_of_compiled_passes_check_what_they_are_given():
    op = torch.ops.hccl_b200
    x, w, r = _rnd(8, 64), _rnd(64), torch.ones(8, device="cuda")
    table = torch.ones(8, 32, device="cuda")
    for f, args in ((op.norm_backward, (x[:4], x, w, r, None)), (op.norm_backward, (x, x, w[:32], r, None)), (op.norm_backward, (x, x, w, r[:4], None)),
                    (op.norm_backward, (x, x, w, r, x[:4])), (op.norm_backward, (x.float(), x, w, r, None)), (op.swiglu_backward, (x, x)), (op.swiglu_backward, (x[:, :32].half(), x)),
                    (op.rope_backward, (x, table, table)), (op.rope_backward, (x.view(8, 1, 64), table[:4], table)), (op.rope_backward, (x.view(8, 1, 64), table.half(), table)),
                    (op.linear_backward, (x, x, _rnd(32, 64))), (op.linear_backward, (x[:4], x, _rnd(64, 64))), (op.linear_backward, (x, x, w))):
        with pytest.raises(RuntimeError):
            f(*args)
    dx, dw = op.norm_backward(x, x, w, r, None)
    assert dx.shape == x.shape and dw.shape == w.shape
    assert [t.shape for t in op.linear_backward(x.to("meta"), x.to("meta"), _rnd(64, 64).to("meta"))] == [(8, 64), (64, 64)]


def test_a_refused_backward_call_raises_what_a_refused_call_raises(way):
    ctx = TPContext(None)
    layer = ColumnParallelLinear(64, 128, ctx, "odd")
    y = layer(_rnd(5, 64).requires_grad_())                                      # five rows: no inner dimension for the weight's gradient
    with pytest.raises(HcclError):
        y.sum().backward()
    x = _rnd(8, 64).requires_grad_()
    g = _rnd(8 * 32 + 1)[1:].view(8, 32)                                         # not on 16 bytes
    with pytest.raises(HcclError):
        fused.swiglu(x).backward(g)
    assert fused.swiglu(x).sum().item() == fused.swiglu(x.detach()).sum().item()


def test_streams_and_checkpoints(way):
    from torch.utils.checkpoint import checkpoint
    x, w = _rnd(512, 1024).requires_grad_(), _rnd(1024).requires_grad_()

    def f(t):
        return fused.swiglu(fused.add_rms_norm(t, None, w, 1e-5)[1])

    want = torch.autograd.grad(f(x).float().square().sum(), [x, w])
    got = torch.autograd.grad(checkpoint(f, x, use_reentrant=False).float().square().sum(), [x, w])
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(1_000_000)
        y = f(x * 1)
    torch.cuda.current_stream().wait_stream(side)
    got = torch.autograd.grad(y.float().square().sum(), [x, w])                  # the nodes run on their forward pass's stream
    assert all(torch.equal(a, b) for a, b in zip(want, got))


def test_recorded_gradients_anomaly_mode_and_batches(way):
    """Gradients that are themselves to be recorded come without a graph, batches of them are refused; anomaly mode sees the nodes."""
    x, w = _rnd(8, 64).requires_grad_(), _rnd(64).requires_grad_()
    h = fused.add_rms_norm(x, None, w, 1e-5)[1]
    up = _rnd(8, 64, seed=5).requires_grad_()
    assert not any(g.requires_grad for g in torch.autograd.grad(h, [x, w], up, create_graph=True))
    h = fused.add_rms_norm(x, None, w, 1e-5)[1]
    with pytest.raises(RuntimeError):
        torch.autograd.grad(h, x, torch.stack((up.detach(), up.detach())), is_grads_batched=True)
    with torch.autograd.set_detect_anomaly(True):
        y = fused.swiglu(fused.add_rms_norm(x, None, w, 1e-5)[1])
        want = torch.autograd.grad(y, x, torch.ones_like(y), retain_graph=True)[0]
        with pytest.raises(RuntimeError, match="nan"):
            torch.autograd.grad(y, x, torch.full_like(y, float("nan")))
    assert torch.equal(want, torch.autograd.grad(fused.swiglu(fused.add_rms_norm(x, None, w, 1e-5)[1]), x, torch.ones_like(y))[0])


# one leaf for both inputs, a leaf that holds a gradient beside one that does not (either way round), inputs that are no leaves
@pytest.mark.parametrize("case", ["same", "first", "second", "results"])
def test_leaves_and_what_they_hold(case, way):
    x, w = _rnd(16, 64, seed=1).requires_grad_(), _rnd(64, seed=3)
    d = x if case == "same" else _rnd(16, 64, seed=2).requires_grad_()
    held = {"first": x, "second": d}.get(case)
    if held is not None:
        held.grad = torch.ones_like(held)
    a, b = (x * 1, d * 1) if case == "results" else (x, d)
    x_out, h = fused.add_rms_norm(a, b, w, 1e-5)
    ups = [_rnd(16, 64, seed=6), _rnd(16, 64, seed=7)]
    one = torch.autograd.grad([x_out, h], a if case == "results" else x, ups, retain_graph=True)[0]
    torch.autograd.backward([x_out, h], ups)
    if case == "same":
        assert torch.equal(x.grad, one)                          # the sum of both inputs' parts, which `grad` gives too
        return
    assert all(torch.equal(t.grad, one + 1 if t is held else one) for t in (x, d))
    assert x.grad.data_ptr() != d.grad.data_ptr()
    x.grad.zero_()
    assert torch.equal(d.grad, one + 1 if d is held else one)
