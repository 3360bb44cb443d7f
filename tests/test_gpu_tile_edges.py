"""The matmul, norm, SwiGLU, rotary and routing kernels at the edges of their tiles, groups and rings, against float64.

Tolerance: every compared tensor is rounded to bf16 once, which is off by at most half a unit in the last place, 2^-8 =
3.9e-3 of an element and so of the 2-norm of any tensor (about 1.7e-3 of one with spread-out values); sums are fp32 and add
less than 1e-4 at these lengths.  The norm's output is taken of a sum that is itself rounded, which the reference repeats.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hccl_b200.ops import fused, mc2
from hccl_b200.ops.moe import expert_offsets

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


@pytest.mark.parametrize("captured", [False, True])
def test_norm_backward_on_a_side_stream(captured):
    """The two launches of the norm's backward pass on a stream of their own, eager and replayed from a graph on other inputs."""
    g = torch.Generator(device="cuda").manual_seed(5)
    inputs = [[_rnd(g, 700, 2056), _rnd(g, 700, 2056), _rnd(g, 2056), _rnd(g, 700, 2056), _rnd(g, 700, 2056)] for _ in range(2)]

    def grads(x, delta, w, d_out, d_h):
        x, delta, w = (t.detach().requires_grad_() for t in (x, delta, w))
        return torch.autograd.grad(fused.add_rms_norm(x, delta, w, 1e-5), [x, delta, w], [d_out, d_h])

    want = [grads(*i) for i in inputs]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    if captured:
        static = [t.clone() for t in inputs[0]]
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            grads(*static)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = grads(*static)
    for i, ref in zip(inputs, want):
        with torch.cuda.stream(side):
            if captured:
                for t, v in zip(static, i):
                    t.copy_(v)
                graph.replay()
                got = [o.clone() for o in out]
            else:
                got = grads(*i)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, ref))


def test_rms_norm_of_as_many_rows_as_there_are_row_numbers():
    rows, hidden = 2 ** 31 - 8, 8
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 77 GB")
    x = torch.empty(rows, hidden, device="cuda", dtype=torch.bfloat16).fill_(3.0)
    w = torch.arange(1, 9, device="cuda").bfloat16()
    h = fused.add_rms_norm(x, None, w, 0.0)[1]
    for part in (h[:10000], h[-10000:]):
        assert torch.equal(part, w.expand(10000, hidden))
    del x, h
    torch.cuda.empty_cache()


# vectors per thread: one (small) and several, rows shorter than a block's stretch, ragged ends
@pytest.mark.parametrize("rows,f", [(1, 8), (3, 264), (700, 56), (1031, 3592), (4097, 1024)])
def test_swiglu_blocks(rows, f):
    g = torch.Generator(device="cuda").manual_seed(rows + f)
    x, dy = _rnd(g, rows, 2 * f, std=2.0).requires_grad_(), _rnd(g, rows, f)
    y = fused.swiglu(x)
    y.backward(dy)
    x64 = x.detach().double().requires_grad_()
    a, b = x64.chunk(2, dim=-1)
    y64 = a * torch.sigmoid(a) * b
    assert _rel(y.detach(), y64.detach()) <= ONE_ROUNDING
    assert _rel(x.grad, torch.autograd.grad(y64, x64, dy.double())[0]) <= ONE_ROUNDING


def test_swiglu_extremes():
    """Gates whose sigmoid saturates, infinities and NaN give what the expression gives."""
    gate = torch.tensor([-1e30, -200.0, -88.5, -20.0, 0.0, 20.0, 90.0, 1e30], device="cuda")
    x = torch.cat((gate, torch.full((8,), 2.0, device="cuda"))).bfloat16().view(1, 16)
    want = fused.swiglu_reference(x.double())
    got = fused.swiglu(x).double()
    assert torch.isfinite(got).all()
    torch.testing.assert_close(got, want, rtol=8e-3, atol=2.0 ** -126)      # the smallest normal number
    x = torch.tensor([[float("nan")] + [float("inf")] * 7 + [1.0] * 8], device="cuda").bfloat16()
    got = fused.swiglu(x)
    assert torch.isnan(got[0, 0]) and torch.isinf(got[0, 1:]).all()


@pytest.mark.parametrize("rows", [1, 40])                     # one vector per thread, several
def test_swiglu_of_every_gate(rows):
    """All bf16 gates.  Around -88 the exponential is near the largest fp32 number and the result a normal bf16 one; below
    -88.5 the exponential overflows and the result is 0."""
    gate = torch.arange(-32768, 32768, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    x = torch.cat((gate, torch.full_like(gate, 3.0))).repeat(rows, 1).requires_grad_()
    dy = torch.full((rows, gate.numel()), 2.0, device="cuda", dtype=torch.bfloat16)
    y = fused.swiglu(x)
    y.backward(dy)
    x64 = x.detach().double().requires_grad_()
    y64 = fused.swiglu_reference(x64)
    dx = torch.autograd.grad(y64, x64, dy.double())[0]
    g = gate.float()
    # 2^-126: the smallest normal number; gradients of gates near the zero of silu's slope cancel, to fp32's last place
    seen, zero = (g >= -88.5) & (g <= 1e38), (g < -88.75) & torch.isfinite(g)
    for got, want, extra in ((y.detach(), y64.detach(), 0.0), (x.grad[:, :gate.numel()], dx[:, :gate.numel()], 2e-6), (x.grad[:, gate.numel():], dx[:, gate.numel():], 0.0)):
        err = (got.double() - want).abs()
        assert (err[:, seen] <= ONE_ROUNDING * want[:, seen].abs() + 2.0 ** -126 + extra * (g[seen] > -4)).all()
        assert (got[:, zero] == 0).all()
    assert torch.isnan(y[:, torch.isnan(g) | (g == float("-inf"))]).all() and torch.isinf(y[:, g == float("inf")]).all()
    assert torch.equal(torch.signbit(y[0, g == 0]), torch.signbit(g[g == 0]))


# heads per thread: four, two, one, a last group that is not full; rows per block: many, one, one in several passes
@pytest.mark.parametrize("s,heads,d,extra", [(1, 1, 16, 0), (9, 2, 64, 128), (33, 3, 128, 0), (130, 5, 64, 16), (7, 64, 128, 2048), (3, 130, 256, 0)])
def test_rope_head_groups(s, heads, d, extra):
    g = torch.Generator(device="cuda").manual_seed(s + heads)
    x = _rnd(g, s, heads * d + extra)[:, :heads * d].view(s, heads, d).requires_grad_()
    ang = torch.rand(s, d // 2, device="cuda", generator=g) * 6.28
    cos, sin, dy = ang.cos().contiguous(), ang.sin().contiguous(), _rnd(g, s, heads, d)
    y = fused.rope(x, cos, sin)
    dx = torch.autograd.grad(y, x, dy)[0]
    c, n, h = cos.double()[:, None], sin.double()[:, None], d // 2

    def turn(t, sign):
        a, b = t.double()[..., :h], t.double()[..., h:]
        return torch.cat((a * c - sign * b * n, b * c + sign * a * n), dim=-1)

    assert _rel(y.detach(), turn(x.detach(), 1)) <= ONE_ROUNDING
    assert _rel(dx, turn(dy, -1)) <= ONE_ROUNDING


# shared counters and global ones, one round of the scan and many, one block and several passes over the ids
@pytest.mark.parametrize("pairs,experts", [(1, 1), (2047, 256), (2049, 257), (300000, 4096), (5000, 4097), (40000, 65536)])
def test_expert_offsets_ranges(pairs, experts):
    g = torch.Generator(device="cuda").manual_seed(pairs)
    idx = torch.randint(-1, experts + 1, (pairs,), device="cuda", generator=g, dtype=torch.int32)
    ok = idx[(idx >= 0) & (idx < experts)].long()
    ref = torch.zeros(experts + 1, dtype=torch.int64, device="cuda")
    ref[1:] = torch.bincount(ok, minlength=experts).cumsum(0)
    for _ in range(2):
        assert torch.equal(expert_offsets(idx, experts).long(), ref)


def _offsets_of(idx, experts):
    ok = idx[(idx >= 0) & (idx < experts)].long()
    return torch.cat((ok.new_zeros(1), torch.bincount(ok, minlength=experts).cumsum(0)))


@pytest.mark.parametrize("start", [0, 1, 3])
@pytest.mark.parametrize("pairs,experts", [(3, 5), (130, 8192), (70001, 8193), (131073, 100)])
def test_expert_offsets_of_a_table_that_starts_anywhere(pairs, experts, start):
    g = torch.Generator(device="cuda").manual_seed(pairs)
    idx = torch.randint(-1, experts + 1, (pairs + start,), device="cuda", generator=g, dtype=torch.int32)[start:]
    assert torch.equal(expert_offsets(idx, experts).long(), _offsets_of(idx, experts))


def test_expert_offsets_on_two_streams_and_in_a_graph():
    """Calls that run at the same time, with different numbers of experts, on two streams and from a replayed graph."""
    g = torch.Generator(device="cuda").manual_seed(3)
    tables = [(torch.randint(0, e, (n,), device="cuda", generator=g, dtype=torch.int32), e) for n, e in ((60000, 256), (50000, 57), (40000, 9000))]
    want = [_offsets_of(i, e) for i, e in tables]
    streams = [torch.cuda.Stream() for _ in tables]
    graph, keep = torch.cuda.CUDAGraph(), []
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=streams[2]):
        for _ in range(20):
            keep.append(expert_offsets(*tables[2]))
    got = [[], []]
    for s in streams:
        with torch.cuda.stream(s):
            torch.cuda._sleep(20_000_000)                      # all three start together
    with torch.cuda.stream(streams[2]):
        graph.replay()
    for _ in range(40):
        for i in range(2):
            with torch.cuda.stream(streams[i]):
                got[i].append(expert_offsets(*tables[i]))
    torch.cuda.synchronize()
    for outs, ref in ((got[0], want[0]), (got[1], want[1]), (keep, want[2])):
        assert all(torch.equal(o.long(), ref) for o in outs)


# rows of one 128-element block and of a part of a warp's stretch, one token and more tokens than warps, dropped pairs,
# the counting kernel of one block and of many; rows shared by several warps where tokens are few, every group of topk
@pytest.mark.parametrize("p,tokens,hidden,experts,topk", [(2, 3, 128, 2, 1), (2, 70, 1152, 16, 3), (4, 40, 8192, 64, 8), (2, 5000, 256, 8, 4),
                                                           (2, 1, 7168, 8, 8), (8, 8, 2048, 16, 2), (2, 9, 7168, 16, 5), (4, 2, 1408, 8, 1)])
def test_moe_dispatch_and_combine_edges(p, tokens, hidden, experts, topk):
    import hccl_b200 as hb
    from hccl_b200 import Communicator
    from hccl_b200.ops.moe import MoeDispatcher

    comms = Communicator.emulated(p, hb.make_config(buffer_mib=8))
    cap = 2 * tokens * topk * p
    disp = [MoeDispatcher(c, tokens, hidden, topk, experts, capacity=cap) for c in comms]
    g = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    xs = [_rnd(g, tokens, hidden) for _ in comms]
    idx = [torch.topk(torch.randn(tokens, experts, device="cuda", generator=g), min(topk, experts), dim=-1)[1].int().contiguous() for _ in comms]
    idx[0][tokens // 2, -1] = -1                                     # a dropped pair
    ws = [torch.rand(tokens, topk, device="cuda", generator=g) + 0.1 for _ in comms]
    res = [d.dispatch(x, i) for d, x, i in zip(disp, xs, idx)]
    torch.cuda.synchronize()
    per = experts // p
    for r in range(p):
        want = torch.stack([(torch.stack([(i == r * per + e).sum() for i in idx])).sum() for e in range(per)]).cumsum(0)
        assert res[r].offsets[0] == 0 and torch.equal(res[r].offsets[1:].long(), want)
        n = int(want[-1])
        src = res[r].src_info[:n]
        rank, pair = src >> 32, src & 0xFFFFFFFF
        rows = torch.stack(xs)[rank, pair // topk].float().view(n, hidden // 128, 128)
        # the scale and the bytes, bit for bit: fp32 maximum / 448 (a tensor: torch multiplies by the reciprocal of a number)
        amax = rows.abs().amax(-1).clamp_min(1e-10)
        scale = amax / torch.full_like(amax, 448.0)
        assert torch.equal(res[r].scales[:n], scale)
        want8 = (rows * (1.0 / scale).unsqueeze(-1)).to(torch.float8_e4m3fn).view(n, hidden)
        assert torch.equal(res[r].x_fp8[:n].view(torch.uint8), want8.view(torch.uint8))
        assert torch.equal(torch.stack(idx)[rank, pair // topk, pair % topk].long(),
                           torch.repeat_interleave(torch.arange(per, device="cuda"), res[r].offsets.long().diff()) + r * per)
        disp[r].y.copy_(torch.randn(cap, hidden, device="cuda", generator=g))
    out = [d.combine(w) for d, w in zip(disp, ws)]
    torch.cuda.synchronize()
    y = torch.stack([d.y for d in disp]).double()
    for r in range(p):
        slot = res[r].slot_map.view(tokens, topk)
        keep = slot != -1
        rows = y[(slot >> 32).clamp_min(0), (slot & 0xFFFFFFFF) * keep]
        ref = (rows * (ws[r].double() * keep).unsqueeze(-1)).sum(1)
        assert _rel(out[r], ref) <= ONE_ROUNDING
    assert comms[0].async_error() == hb.Result.SUCCESS
    for c in comms:
        c.destroy()


def _check_matmul(m, n, k, ta, tb):
    g = torch.Generator(device="cuda").manual_seed(m * 31 + n * 7 + k)
    a, b = _rnd(g, *((k, m) if ta else (m, k))), _rnd(g, *((n, k) if tb else (k, n)))
    out = torch.full((m + 1, n), 7.0, device="cuda", dtype=torch.bfloat16)       # the last row must stay
    mc2.matmul(a, b, trans_a=ta, trans_b=tb, out=out[:m])
    ref = (a.double().t() if ta else a.double()) @ (b.double() if not tb else b.double().t())
    assert _rel(out[:m], ref) <= ONE_ROUNDING
    assert (out[m] == 7.0).all()


LAYOUTS = [(False, True), (False, False), (True, True), (True, False)]


# column tiles whose half is no multiple of 64 (224, 192 and 160 wide), a ragged last one, full and partial row tiles
@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("m,n,k", [(4096, 3584, 128), (1024, 8192, 192), (2304, 7104, 64), (1000, 10232, 136)])
def test_wide_matmul_with_kn_weight(m, n, k, ta):
    _check_matmul(m, n, k, ta, False)


# two full rounds of wide tiles, then left-over positions and an odd last column tile as single ones; ragged in every direction
@pytest.mark.parametrize("ta,tb", LAYOUTS)
def test_wide_tile_rounds(ta, tb):
    _check_matmul(2504, 7800, 3080, ta, tb)


# (m, n, k), single items per pair after the wide ones: a second in the other accumulator, a third back in the first
WIDE_SINGLES = [((1592, 13400, 3080), 2), ((3080, 8800, 3080), 3)]


@pytest.mark.parametrize("ta,tb", LAYOUTS)
@pytest.mark.parametrize("shape", [s for s, _ in WIDE_SINGLES])
def test_wide_tiles_followed_by_several_singles(shape, ta, tb):
    _check_matmul(*shape, ta, tb)


# k-blocks: one (the halves run together), four (skew two), 17 (skew eight), 24 (the first with the full skew)
WIDE_SHORT_K = [(2504, 7800, k) for k in (64, 200, 1032, 1536)]


def test_wide_tiles_with_a_short_inner_dimension():
    """Shapes that take wide tiles only where HCCL_MC2_WIDE=1 asks for them; the switch is read once per process."""
    import os
    import subprocess
    import sys
    code = ("import sys; sys.path.insert(0, 'tests'); import test_gpu_tile_edges as t\n"
            "for shape in t.WIDE_SHORT_K:\n"
            "    for layout in t.LAYOUTS:\n"
            "        t._check_matmul(*shape, *layout)\n"
            "print('checked')")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=root, env={**os.environ, "HCCL_MC2_WIDE": "1"}, timeout=600)
    assert r.returncode == 0 and "checked" in r.stdout, r.stderr[-3000:]


# clusters of three: k-blocks and tokens that three CTAs cannot share evenly
SPLIT_OF_THREE = [(17, 10000, 840), (40, 12000, 1032), (8, 9608, 960)]


@pytest.mark.parametrize("ta,tb", LAYOUTS)
@pytest.mark.parametrize("shape", SPLIT_OF_THREE)
def test_split_matmul_over_three_ctas(shape, ta, tb):
    if ta and shape[0] % 8:
        pytest.skip("transposed A needs M % 8 == 0")
    _check_matmul(*shape, ta, tb)


# token tiles of 16 .. 128 and several of them, k-blocks fewer and more than the CTAs of a cluster, ragged N and K
@pytest.mark.parametrize("ta,tb", LAYOUTS)
@pytest.mark.parametrize("m,n,k", [(8, 8, 8), (16, 128, 64), (24, 136, 256), (64, 1024, 520), (128, 248, 2048), (136, 1000, 1032), (304, 640, 4096),
                                   (1, 264, 1024), (17, 8192, 1024)])
def test_small_output_matmul(m, n, k, ta, tb):
    if ta and m % 8:
        pytest.skip("transposed A needs M % 8 == 0")
    _check_matmul(m, n, k, ta, tb)


@pytest.mark.parametrize("m,n", [(16, 128), (512, 512)])
def test_matmul_as_the_first_work_of_a_thread(m, n):
    """A thread that has made no CUDA call yet has no current context; autograd's is one when a matmul is its first work."""
    import threading
    g = torch.Generator(device="cuda").manual_seed(m)
    a, b = _rnd(g, m, 256), _rnd(g, n, 256)
    out, want, failed = torch.empty(m, n, device="cuda", dtype=torch.bfloat16), mc2.matmul(a, b), []

    def work():
        try:
            mc2.matmul(a, b, out=out)
        except Exception as e:
            failed.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    assert torch.equal(out, want)


# the stalled CTA alone on its tile, and the first and another one of clusters of two to eight: their peers hold good partials and must
# not store sums either
@pytest.mark.parametrize("cta,k,split", [(0, 128, 1), (1, 456, 2), (2, 712, 3), (0, 1024, 4), (2, 1024, 4), (0, 2048, 8), (2, 2048, 8), (7, 2048, 8)])
def test_matmul_that_gives_up_a_wait(cta, k, split):
    """A CTA whose operands never arrive gives up after a short limit: nothing of its tile is stored, the next matmul on the
    device reports it, the one after that runs."""
    import ctypes
    from hccl_b200 import Result
    from hccl_b200._lib import lib
    from hccl_b200.comm import HcclError
    from test_matmul_plan import plan
    p = plan(16, 128, k)
    assert p["route"] == "split" and p["split"] == str(split)
    g = torch.Generator(device="cuda").manual_seed(k)
    a, b = _rnd(g, 16, k), _rnd(g, 128, k)
    out = torch.full((16, 128), 7.0, device="cuda", dtype=torch.bfloat16)
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (a, b, out)]
    lib.HcclDebugMatmulStalled.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_uint64] * 3 + [ctypes.c_int] * 3 + [ctypes.c_uint64, ctypes.c_void_p]
    assert lib.HcclDebugMatmulStalled(*ptr, 16, 128, k, 0, 1, cta, 1_000_000, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert (out == 7.0).all()
    with pytest.raises(HcclError) as e:
        mc2.matmul(a, b)
    assert e.value.code == Result.E_TIMEOUT
    _check_matmul(16, 128, k, False, True)


# all three gradients, strided ones as attention returns them, and only some of them
@pytest.mark.parametrize("s,hq,hkv,d", [(1, 1, 1, 16), (65, 8, 2, 64), (130, 16, 16, 128)])
def test_rope_qkv_matches_the_sliced_form(s, hq, hkv, d):
    g = torch.Generator(device="cuda").manual_seed(s + hq)
    base = _rnd(g, s, (hq + 2 * hkv) * d)
    ang = torch.rand(s, d // 2, device="cuda", generator=g) * 6.28
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    ups = [_rnd(g, n, s, d).transpose(0, 1) for n in (hq, hkv, hkv)]
    for used in ((0, 1, 2), (0, 2), (1,)):
        a, b = base.clone().requires_grad_(), base.clone().requires_grad_()
        got = fused.rope_qkv(a, cos, sin, hq, hkv)
        want = (fused.rope(b[:, :hq * d].view(s, hq, d), cos, sin), fused.rope(b[:, hq * d:(hq + hkv) * d].view(s, hkv, d), cos, sin),
                b[:, (hq + hkv) * d:].view(s, hkv, d))
        for x, y in zip(got, want):
            assert torch.equal(x, y)
        before = fused.LAUNCHES
        torch.autograd.backward([got[i] for i in used], [ups[i] for i in used])
        assert fused.LAUNCHES - before == len({0, 1} & set(used))           # a rotation for q and k only where one has a gradient
        torch.autograd.backward([want[i] for i in used], [ups[i] for i in used])
        assert torch.equal(a.grad, b.grad)
