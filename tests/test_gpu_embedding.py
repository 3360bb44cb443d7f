"""The embedding's gradient kernel: every row of the table, the rows in use summed in token order."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

from hccl_b200 import Result, _calls
from hccl_b200._lib import lib
from hccl_b200.ops import fused


def _case(tokens, vocab, hidden, skew=False, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    ids = torch.randint(0, vocab, (tokens,), device="cuda", generator=g)
    if skew:                                             # every other token is the same one
        ids[::2] = vocab - 1
    return ids, torch.randn(vocab, hidden, device="cuda", generator=g).bfloat16(), torch.randn(tokens, hidden, device="cuda", generator=g).bfloat16()


def _want(ids, dy, vocab):
    return torch.zeros(vocab, dy.shape[1], device="cuda", dtype=torch.float64).index_add_(0, ids, dy.double())


# one token, ids at the edges of the 256 that are looked at together, rows of one vector and of several blocks, a table that is no
# multiple of 16 rows, many tokens of one id
@pytest.mark.parametrize("tokens,vocab,hidden,skew", [(1, 1, 8, False), (255, 17, 64, False), (256, 1000, 2048, False), (257, 33, 2056, True), (1024, 4096, 8192, False),
                                                      (2000, 5, 520, True), (8192, 50000, 128, True)])
def test_against_64_bits(tokens, vocab, hidden, skew):
    ids, table, dy = _case(tokens, vocab, hidden, skew)
    t = table.clone().requires_grad_()
    out = fused.embedding(ids, t)
    assert out.grad_fn.name() == "_EmbeddingBackward" and torch.equal(out, table[ids])
    out.backward(dy)
    want = _want(ids, dy, vocab)
    # sums in fp32, one rounding to bf16 (half a unit in the last of 8 places)
    bound = want.abs() * 2 ** -8 + torch.zeros_like(want).index_add_(0, ids, dy.double().abs()) * tokens * 2 ** -24 + 1e-30
    assert ((t.grad.double() - want).abs() <= bound).all()
    assert (t.grad[torch.bincount(ids, minlength=vocab) == 0] == 0).all()
    again = torch.autograd.grad(fused.embedding(ids, t), t, dy)[0]
    assert torch.equal(again, t.grad)


# ids that are more frequent than one thread adds up alone (128), at the edges of that, of rows, of the vectors and places a block takes
@pytest.mark.parametrize("tokens,vocab,hidden,often", [(129, 1, 8, 129), (300, 40, 120, 128), (300, 40, 128, 129), (515, 9, 136, 257), (1000, 4, 2056, 640),
                                                       (8192, 300, 1032, 8192), (8192, 5000, 8, 4000)])
def test_frequent_ids(tokens, vocab, hidden, often):
    ids, _, dy = _case(tokens, vocab, hidden)
    if vocab > 1:
        ids %= vocab - 1
        ids[torch.randperm(tokens, device="cuda")[:often]] = vocab - 1
    t = torch.zeros(vocab, hidden, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    got = torch.autograd.grad(fused.embedding(ids, t), t, dy)[0]
    want = _want(ids, dy, vocab)
    bound = want.abs() * 2 ** -8 + torch.zeros_like(want).index_add_(0, ids, dy.double().abs()) * tokens * 2 ** -24 + 1e-30
    assert ((got.double() - want).abs() <= bound).all()
    assert torch.equal(got, torch.autograd.grad(fused.embedding(ids, t), t, dy)[0])


@pytest.mark.parametrize("scratch", [True, False])
def test_the_c_functions(scratch):
    """With scratch and without; ids outside the table, and no tokens at all."""
    ids, _, dy = _case(200, 50, 72)
    ids[::3] = 50
    ids[1::5] = -1
    out, s = torch.full((50, 72), 7.0, device="cuda", dtype=torch.bfloat16), torch.cuda.current_stream().cuda_stream
    call = lib.HcclFusedEmbeddingGrad if scratch else lib.HcclFusedEmbeddingBwd
    call.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_uint64] * 2 + [ctypes.c_uint32, ctypes.c_void_p]
    extra = torch.empty(8 * 200 if scratch else 50, device="cuda", dtype=torch.uint8)
    assert call(ids.data_ptr(), dy.data_ptr(), out.data_ptr(), extra.data_ptr(), 200, 50, 72, s) == 0
    keep = (ids >= 0) & (ids < 50)
    want = _want(ids[keep], dy[keep], 50)
    assert ((out.double() - want).norm() / want.norm()).item() < 4e-3
    assert call(ids.data_ptr(), dy.data_ptr(), out.data_ptr(), extra.data_ptr(), 0, 50, 72, s) == 0 and not out.any()
    assert call(ids.data_ptr(), dy.data_ptr(), out.data_ptr(), extra.data_ptr(), 8193, 50, 72, s) == Result.E_NOT_SUPPORT
    assert call(ids.data_ptr(), dy.data_ptr(), out.data_ptr(), extra.data_ptr(), 8, 1 << 63, 4096, s) == Result.E_NOT_SUPPORT


def test_what_is_left_to_pytorch():
    ids, table, _ = _case(40, 64, 64)
    assert _calls.embedding(ids, table) is None                                            # nothing is recorded
    t = table.clone().requires_grad_()
    for i, w in ((ids.int(), t), (ids.view(8, 5), t), (ids, t.detach().float().requires_grad_()), (ids.repeat(300), t), (ids[:0], t), (ids.cpu(), t)):
        assert _calls.embedding(i, w) is None
    assert fused.embedding(ids.view(8, 5), t).shape == (8, 5, 64) and fused.embedding(ids, table).grad_fn is None


def test_gradients_that_are_looked_at():
    """Recorded, batched and dual gradients: what PyTorch's embedding makes of them."""
    import torch.autograd.forward_ad as fwd
    import torch.nn.functional as F
    ids, table, dy = _case(40, 64, 64)
    t, up, tangent = table.clone().requires_grad_(), dy.clone().requires_grad_(), _case(40, 64, 64, seed=1)[2]
    got, want = ([torch.autograd.grad(f(ids, t), t, up, create_graph=True)[0]] for f in (fused.embedding, F.embedding))
    for g in (got, want):                                                                  # the penalty's gradient goes through the table's
        g.append(torch.autograd.grad(g[0].float().square().sum(), up)[0])
        f = fused.embedding if g is got else F.embedding
        g.append(torch.autograd.grad(f(ids, t), t, torch.stack((dy, 2 * dy, -dy)), is_grads_batched=True)[0])
        with fwd.dual_level():
            g += fwd.unpack_dual(torch.autograd.grad(f(ids, t), t, fwd.make_dual(dy, tangent))[0])
    assert got[1].abs().sum() > 0 and got[4] is not None
    assert all(torch.equal(a, b) for a, b in zip(got, want, strict=True))


def test_ids_that_a_hook_gives_back_as_it_likes():
    ids, table, dy = _case(40, 64, 64)
    t = table.clone().requires_grad_()
    want = torch.autograd.grad(fused.embedding(ids, t), t, dy)[0]
    for unpack in (lambda i: i.int(), lambda i: torch.stack((i, i), 1)[:, 0]):
        with torch.autograd.graph.saved_tensors_hooks(lambda i: i, unpack):
            out = fused.embedding(ids, t)
        assert torch.equal(torch.autograd.grad(out, t, dy)[0], want)


def test_gradients_that_begin_anywhere():
    """A packed view into a larger buffer at an odd element, and one that is not packed."""
    ids, table, dy = _case(40, 64, 64)
    t = table.clone().requires_grad_()
    want = torch.autograd.grad(fused.embedding(ids, t), t, dy)[0]
    odd = torch.cat((dy.new_zeros(1), dy.flatten()))[1:].view(40, 64)
    assert odd.data_ptr() % 16 != 0
    for g in (odd, dy.t().contiguous().t()):
        assert torch.equal(torch.autograd.grad(fused.embedding(ids, t), t, g)[0], want)


def test_calls_that_are_refused():
    p, s = ctypes.c_void_p(1 << 20), torch.cuda.current_stream().cuda_stream
    bwd = lib.HcclFusedEmbeddingBwd
    bwd.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_uint64] * 2 + [ctypes.c_uint32, ctypes.c_void_p]
    assert bwd(p, p, p, p, 8193, 10, 64, s) == Result.E_NOT_SUPPORT
    assert bwd(p, p, p, p, 8, 10, 60, s) == Result.E_PARA and bwd(p, ctypes.c_void_p((1 << 20) + 8), p, p, 8, 10, 64, s) == Result.E_PARA
    assert bwd(p, p, p, p, 8, 0, 64, s) == 0


def test_captured_and_side_stream():
    ids, table, dy = _case(300, 128, 256)
    t = table.clone().requires_grad_()
    want = torch.autograd.grad(fused.embedding(ids, t), t, dy)[0]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.autograd.grad(fused.embedding(ids, t), t, dy)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            got = torch.autograd.grad(fused.embedding(ids, t), t, dy)[0]
        g.replay()
    side.synchronize()
    assert torch.equal(got, want)
