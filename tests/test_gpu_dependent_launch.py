"""Kernels whose start overlaps the end of the one before them: what a kernel reads must be complete, whatever comes before it
in the stream (this library's kernels, PyTorch's, a copy, an event of another stream), eager and in a graph with a fork.

Passes that follow one another have different inputs: the allocator gives them the same blocks, so that a kernel which reads too
early finds what the pass before left there, which is wrong then.  Each is compared with a run of its own inputs that waits for
every kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hccl_b200.ops import FusedAdamW, fused, mc2
from hccl_b200.ops.moe import expert_offsets
from test_matmul_plan import plan

SEEN = set()          # (m, n, k, trans_a, trans_b) of the products


def _matmul(a, b, trans_a=False, trans_b=True):
    k, m = a.shape if trans_a else reversed(a.shape)
    SEEN.add((m, b.shape[0] if trans_b else b.shape[1], k, trans_a, trans_b))
    return mc2.matmul(a, b, trans_a=trans_a, trans_b=trans_b)


def _inputs(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s, std=1.0: (torch.randn(*s, device="cuda", generator=g) * std).bfloat16()  # noqa: E731
    ang = torch.rand(96, 32, device="cuda", generator=g) * 6.28
    # rows of 1024; the products take every route of the plain matmul (test_the_chain_takes_every_route)
    return {"x": rnd(96, 1024), "w": rnd(1024), "up": rnd(2048, 1024, std=0.03), "down": rnd(1024, 1024, std=0.03), "big": rnd(2304, 1024), "cos": ang.cos(),
            "sin": ang.sin(), "p": rnd(1024, 1024, std=0.03), "wide": rnd(2504, 3080), "wide_w": rnd(7800, 3080, std=0.03), "broad": rnd(7168, 1024, std=0.03)}


def _chain(t, each=lambda: None, other=None):
    """Every result feeds the next kernel; buffers are written again by later ones.  `each` runs after every step."""
    opt = FusedAdamW([torch.nn.Parameter(t["p"].clone())], lr=1e-2)
    x, stream = t["x"], None
    for i in range(3):
        x, h = fused.add_rms_norm(x, stream, t["w"], 1e-5)
        each()
        y = _matmul(h, t["up"])
        each()
        y = fused.swiglu(y)
        each()
        y = fused.rope(y.view(96, 16, 64), t["cos"], t["sin"]).view(96, 1024)
        each()
        stream = _matmul(y, t["down"])
        each()
        if other is not None:
            side, main = other, torch.cuda.current_stream()
            side.wait_stream(main)
            with torch.cuda.stream(side):
                tall = _matmul(t["big"], stream, trans_b=True)
            z = _matmul(h, t["p"])                       # beside it
            main.wait_stream(side)
        else:
            tall = _matmul(t["big"], stream, trans_b=True)
            each()
            z = _matmul(h, t["p"])
        each()
        opt.param_groups[0]["params"][0].grad = _matmul(tall, t["big"], trans_a=True, trans_b=False).repeat(11, 1)[:1024].contiguous()
        each()
        opt.step()
        each()
        stream = _matmul(z + stream, opt.param_groups[0]["params"][0].detach(), trans_b=False)
        each()
        broad = _matmul(stream.repeat(22, 1)[:2048].contiguous(), t["broad"])
        each()
        ids = (stream.float().abs() * 100).int().clamp_(0, 63)
        off = expert_offsets(ids, 64)
        each()
    wide = _matmul(t["wide"], t["wide_w"])
    each()
    last = _matmul(wide[:512].contiguous(), wide[512:1024].contiguous())
    return [x, stream, tall, broad, off, opt.param_groups[0]["params"][0].detach(), last]


def _leaves_gradients(t, each=lambda: None):
    x, w = t["x"].clone().requires_grad_(), t["w"].clone().requires_grad_()
    h = fused.add_rms_norm(x, t["x"], w, 1e-5)[1]
    each()
    y = fused.swiglu(h)
    each()
    z = fused.rope(y.view(96, 8, 64), t["cos"], t["sin"])
    each()
    for v in (h, y, z):
        v.register_hook(lambda _: each())                   # between the kernels of the backward pass
    return torch.autograd.grad(z.sum(), [x, w])


def _one_by_one(t):
    return [r.clone() for r in _chain(t, torch.cuda.synchronize)]


def test_the_chain_takes_every_route():
    _one_by_one(_inputs(0))
    assert {plan(m, n, k, int(ta), int(tb))["route"] for m, n, k, ta, tb in SEEN} == {"split", "one_sm", "two_sm", "wide", "two_sm_split"}


@pytest.mark.parametrize("forked", [False, True])
def test_a_chain_of_kernels_gives_what_it_gives_one_by_one(forked):
    inputs = [_inputs(seed) for seed in (1, 5)]
    want = [_one_by_one(t) for t in inputs]
    side, alone = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for stream in (torch.cuda.current_stream(), alone):
        with torch.cuda.stream(stream):
            for i in range(4):
                got = _chain(inputs[i % 2], other=side if forked else None)
                stream.synchronize()
                assert all(torch.equal(a, b) for a, b in zip(got, want[i % 2]))
                del got


def test_gradients_of_a_chain():
    inputs = [_inputs(seed) for seed in (2, 6, 7)]
    want = []
    for t in inputs:
        want.append(_leaves_gradients(t, torch.cuda.synchronize))
    torch.cuda.synchronize()
    same = []
    for i in range(21):                                     # back to back; a run's results are compared and given back in its place
        got = _leaves_gradients(inputs[i % 3])
        same += [(a == b).all() for a, b in zip(got, want[i % 3])]
        del got
    assert all(bool(v) for v in same)


@pytest.mark.parametrize("forked", [False, True])
def test_a_chain_in_a_graph(forked):
    """Replayed on other inputs than the ones it was captured with; a branch on a second stream joins in the middle."""
    static, others = _inputs(3), [_inputs(seed) for seed in (4, 8)]
    want = [_one_by_one(t) for t in others]
    stream, side = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        _chain(static, other=side if forked else None)
    torch.cuda.synchronize()
    # the optimizer's own state is made during capture: its moments start from zero in every replay as they do eagerly
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = _chain(static, other=side if forked else None)
    for i in range(4):
        for k, v in others[i % 2].items():
            static[k].copy_(v)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, want[i % 2]))
