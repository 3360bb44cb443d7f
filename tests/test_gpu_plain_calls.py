"""Calls on plain CUDA tensors go to the C API through the native module; everything that something looks at (gradients, forward
mode, transforms, tracing, subclasses, dispatch modes, hooks) goes the general way.  Both give the same."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hccl_b200 import _calls
from hccl_b200.comm import HcclError
from hccl_b200.ops import fused, mc2
from hccl_b200.ops.moe import expert_offsets


def _rnd(*shape, seed=0):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)).bfloat16()


def _tables(s, d):
    ang = torch.rand(s, d // 2, device="cuda") * 6.28
    return ang.cos(), ang.sin()


def _general(monkeypatch):
    for name in ("add_rms_norm", "rms_norm_bwd", "swiglu_fwd", "swiglu_bwd", "rope", "matmul", "expert_offsets", "collective"):
        monkeypatch.setattr(_calls, name, _calls._nothing)


def _results():
    x, d, w = _rnd(37, 520, seed=1), _rnd(37, 520, seed=2), _rnd(520, seed=3)
    torch.manual_seed(0)
    c, s = _tables(37, 64)
    heads = _rnd(37, 10 * 64, seed=4)[:, 64:9 * 64].view(37, 8, 64)
    out = [*fused.add_rms_norm(x, d, w, 1e-5), *fused.add_rms_norm(x, None, w, 1e-6), fused.swiglu(_rnd(5, 3, 64, seed=5)), fused.rope(heads, c, s),
           mc2.matmul(_rnd(72, 128, seed=6), _rnd(40, 128, seed=7)), mc2.matmul(_rnd(128, 72, seed=6), _rnd(128, 40, seed=7), trans_a=True, trans_b=False),
           expert_offsets(torch.randint(0, 9, (50, 2), device="cuda", dtype=torch.int32), 9)]
    p = [t.clone().requires_grad_() for t in (x, d, w)]
    h = fused.add_rms_norm(*p, 1e-5)
    out += torch.autograd.grad(fused.swiglu(h[1][:, :512].contiguous()).float().sum() + h[0].float().sum(), p)
    y = heads.clone().requires_grad_()
    out += torch.autograd.grad(fused.rope(y, c, s), y, _rnd(37, 8, 64, seed=8))
    return out


def test_the_native_way_gives_what_the_general_one_gives(monkeypatch):
    assert _calls._module is not None
    native = _results()
    before = fused.LAUNCHES
    _general(monkeypatch)
    general = _results()
    launched = fused.LAUNCHES - before
    monkeypatch.undo()
    _results()
    assert fused.LAUNCHES - before == 2 * launched
    assert all(a.shape == b.shape and a.dtype == b.dtype and torch.equal(a, b) for a, b in zip(native, general))


def test_input_that_is_the_residual_stream_comes_back_itself():
    x, w = _rnd(4, 64), _rnd(64)
    assert fused.add_rms_norm(x, None, w, 1e-5)[0] is x


def test_what_is_not_plain_is_left_to_the_general_way():
    x, w = _rnd(4, 64), _rnd(64)
    c, s = _tables(4, 16)
    assert _calls.add_rms_norm(x, None, w, 1e-5) is not None
    assert _calls.add_rms_norm(x.clone().requires_grad_(), None, w, 1e-5) is None
    with torch.no_grad():
        assert _calls.add_rms_norm(x.clone().requires_grad_(), None, w, 1e-5) is not None
    for bad in (x.float(), x.cpu(), x.t(), _rnd(4, 60), _rnd(4, 8200), x[:0]):
        assert _calls.add_rms_norm(bad, None, _rnd(bad.shape[-1]) if bad.shape[-1] != 64 else w, 1e-5) is None
    assert _calls.add_rms_norm(x, _rnd(1, 64), w, 1e-5) is None               # would broadcast
    assert _calls.add_rms_norm(x, None, _rnd(32), 1e-5) is None
    assert _calls.swiglu_fwd(_rnd(4, 24)) is None and _calls.swiglu_fwd(torch.nn.Parameter(x)) is None
    r = _rnd(4, 4, 16)
    assert _calls.rope(r, c, s, False) is not None
    assert _calls.rope(r, c[:1], s, False) is None and _calls.rope(r, c.cpu(), s, False) is None and _calls.rope(r.transpose(0, 1), c, s, False) is None
    assert _calls.matmul(x, _rnd(8, 32), False, True, None, None) is None     # inner dimensions differ
    assert _calls.expert_offsets(torch.zeros(4, device="cuda", dtype=torch.int64), 4, None) is None
    with pytest.raises(AssertionError):
        mc2.matmul(x, _rnd(8, 32))
    with pytest.raises(HcclError):
        mc2.matmul(_rnd(8, 12), _rnd(8, 12))                                   # the library's own refusal
    with pytest.raises(HcclError):
        fused.swiglu(_rnd(65)[1:].view(1, 64))                                 # not on 16 bytes


def test_transforms_modes_and_tracers_see_the_operators():
    x, w = _rnd(4, 64), _rnd(64)
    import torch.autograd.forward_ad as fw
    from torch._subclasses.fake_tensor import FakeTensorMode
    seen = []

    class Count(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    with Count():
        assert _calls.swiglu_fwd(x) is None
        fused.swiglu(x)
    assert seen
    with fw.dual_level():
        assert _calls.swiglu_fwd(fw.make_dual(x, torch.ones_like(x))) is None
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: fused.swiglu(x))(x)                          # refused inside a transform, batched or not
    with FakeTensorMode():
        assert _calls.swiglu_fwd(torch.empty(4, 64, device="cuda", dtype=torch.bfloat16)) is None
    traced = []
    torch.jit.trace(lambda t: (traced.append(_calls.swiglu_fwd(x)), t + 1)[1], x, check_trace=False)
    assert traced == [None]


def test_torch_function_sees_the_operators():
    """Subclasses and modes that know __torch_function__ only: what they get is what the general way gives them."""
    from torch.overrides import TorchFunctionMode

    class Named(torch.Tensor):
        pass

    x, d, w = _rnd(4, 64), _rnd(4, 64, seed=1), _rnd(64)
    c, s = _tables(4, 16)
    n = x.as_subclass(Named)
    assert _calls.add_rms_norm(n, None, w, 1e-5) is None and _calls.add_rms_norm(x, d.as_subclass(Named), w, 1e-5) is None
    assert _calls.swiglu_fwd(n) is None and _calls.rope(n.view(4, 4, 16), c, s, False) is None
    assert _calls.matmul(n, x, False, True, None, None) is None and _calls.expert_offsets(torch.zeros(4, device="cuda", dtype=torch.int32).as_subclass(Named), 4, None) is None
    x_out, h = fused.add_rms_norm(n, d, w, 1e-5)
    assert type(x_out) is Named and type(h) is Named
    want = fused.add_rms_norm(x, d, w, 1e-5)
    assert torch.equal(torch.Tensor(x_out), torch.Tensor(want[0])) and torch.equal(torch.Tensor(h), torch.Tensor(want[1]))
    assert _calls.swiglu_fwd(torch.nn.Parameter(x, requires_grad=False)) is not None
    seen = []

    class Count(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    with Count():
        assert _calls.swiglu_fwd(x) is None
        fused.swiglu(x)
    assert seen
    with torch.device("cpu"):                                                   # a default device is no such mode
        assert _calls.swiglu_fwd(x) is not None
        with Count():
            assert _calls.swiglu_fwd(x) is None
    assert _calls.swiglu_fwd(x) is not None


def test_arguments_of_other_types_are_left_to_the_general_way():
    a, b = _rnd(8, 16), _rnd(8, 16, seed=1)
    assert _calls.matmul(a, b, torch.zeros(2), True, None, None) is None        # no truth value
    assert _calls.matmul(a, b, False, True, None, "a stream") is None
    assert _calls.expert_offsets(torch.zeros(4, device="cuda", dtype=torch.int32), 4, 1.5) is None
    assert _calls.collective(0, 1, a.float(), b.float(), 0.0, 2, None) is None
    with pytest.raises(RuntimeError):
        mc2.matmul(a, b, trans_a=torch.zeros(2))


def test_saved_tensor_hooks_are_called():
    x, w = _rnd(4, 64).requires_grad_(), _rnd(64).requires_grad_()
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.cuda()):
        h = fused.swiglu(fused.add_rms_norm(x, None, w, 1e-5)[1])
    got = torch.autograd.grad(h.float().sum(), [x, w])
    assert len(packed) >= 4
    want = torch.autograd.grad(fused.swiglu(fused.add_rms_norm(x, None, w, 1e-5)[1]).float().sum(), [x, w])
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_streams():
    """The current stream, and a stream that is given."""
    side = torch.cuda.Stream()
    a, b = _rnd(64, 256), _rnd(64, 256, seed=1)
    want, off = mc2.matmul(a, b), expert_offsets(torch.arange(64, device="cuda", dtype=torch.int32), 64)
    torch.cuda.synchronize()
    for give in (False, True):
        with torch.cuda.stream(torch.cuda.current_stream() if give else side):
            torch.cuda._sleep(1_000_000)
            ids = torch.arange(64, device="cuda", dtype=torch.int32)
            out = torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
            if give:
                side.wait_stream(torch.cuda.current_stream())
            kw = {"stream": side} if give else {}
            mc2.matmul(a, b, out=out, **kw)
            got = expert_offsets(ids, 64, **kw)
        side.synchronize()
        assert torch.equal(out, want) and torch.equal(got, off)
