"""Kernels whose start overlaps the end of the one before them: what a kernel reads must be complete, whatever comes before it
in the stream (this library's kernels, PyTorch's, a copy, an event of another stream), eager and in a graph with a fork."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hccl_b200.ops import FusedAdamW, fused, mc2
from hccl_b200.ops.moe import expert_offsets


def _inputs(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s, std=1.0: (torch.randn(*s, device="cuda", generator=g) * std).bfloat16()  # noqa: E731
    ang = torch.rand(96, 32, device="cuda", generator=g) * 6.28
    # rows of 1024; the weights take every route of the plain matmul: split, one SM, two SMs, and a wide one where it is asked for
    return {"x": rnd(96, 1024), "w": rnd(1024), "up": rnd(2048, 1024, std=0.03), "down": rnd(1024, 1024, std=0.03), "big": rnd(2304, 1024), "cos": ang.cos(),
            "sin": ang.sin(), "p": rnd(1024, 1024, std=0.03), "wide": rnd(2504, 3080), "wide_w": rnd(7800, 3080, std=0.03)}


def _chain(t, each=lambda: None, other=None):
    """Every result feeds the next kernel; buffers are written again by later ones.  `each` runs after every step."""
    opt = FusedAdamW([torch.nn.Parameter(t["p"].clone())], lr=1e-2)
    x, stream = t["x"], None
    for i in range(3):
        x, h = fused.add_rms_norm(x, stream, t["w"], 1e-5)
        each()
        y = mc2.matmul(h, t["up"])
        each()
        y = fused.swiglu(y)
        each()
        y = fused.rope(y.view(96, 16, 64), t["cos"], t["sin"]).view(96, 1024)
        each()
        stream = mc2.matmul(y, t["down"])
        each()
        if other is not None:
            side, main = other, torch.cuda.current_stream()
            side.wait_stream(main)
            with torch.cuda.stream(side):
                two_sm = mc2.matmul(t["big"], stream, trans_b=True)
            z = mc2.matmul(h, t["p"])                       # beside it
            main.wait_stream(side)
        else:
            two_sm = mc2.matmul(t["big"], stream, trans_b=True)
            each()
            z = mc2.matmul(h, t["p"])
        each()
        opt.param_groups[0]["params"][0].grad = mc2.matmul(two_sm, t["big"], trans_a=True, trans_b=False).repeat(11, 1)[:1024].contiguous()
        each()
        opt.step()
        each()
        stream = mc2.matmul(z + stream, opt.param_groups[0]["params"][0].detach(), trans_b=False)
        each()
        ids = (stream.float().abs() * 100).int().clamp_(0, 63)
        off = expert_offsets(ids, 64)
        each()
    wide = mc2.matmul(t["wide"], t["wide_w"])
    each()
    last = mc2.matmul(wide[:512].contiguous(), wide[512:1024].contiguous())
    return [x, stream, two_sm, off, opt.param_groups[0]["params"][0].detach(), last]


def _leaves_gradients(t):
    x, w = t["x"].clone().requires_grad_(), t["w"].clone().requires_grad_()
    y = fused.swiglu(fused.add_rms_norm(x, t["x"], w, 1e-5)[1])
    return torch.autograd.grad(fused.rope(y.view(96, 8, 64), t["cos"], t["sin"]).sum(), [x, w])


@pytest.mark.parametrize("forked", [False, True])
def test_a_chain_of_kernels_gives_what_it_gives_one_by_one(forked):
    t = _inputs(1)
    want = _chain(t, torch.cuda.synchronize)
    side, alone = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for stream in (torch.cuda.current_stream(), alone):
        with torch.cuda.stream(stream):
            for _ in range(3):
                got = _chain(t, other=side if forked else None)
                stream.synchronize()
                assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_gradients_of_a_chain():
    t = _inputs(2)
    want = _leaves_gradients(t)
    torch.cuda.synchronize()
    runs = [_leaves_gradients(t) for _ in range(20)]
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for got in runs for a, b in zip(got, want))


@pytest.mark.parametrize("forked", [False, True])
def test_a_chain_in_a_graph(forked):
    """Replayed on other inputs than the ones it was captured with; a branch on a second stream joins in the middle."""
    static, fresh = _inputs(3), _inputs(4)
    want = _chain(fresh, torch.cuda.synchronize)
    stream, side = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        _chain(static, other=side if forked else None)
    torch.cuda.synchronize()
    # the optimizer's own state is made during capture: its moments start from zero in every replay as they do eagerly
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = _chain(static, other=side if forked else None)
    for k, v in fresh.items():
        static[k].copy_(v)
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, want))
