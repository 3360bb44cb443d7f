"""Dispatch counts up to 4096 (token, expert) pairs inside its own blocks: positions at the edges of the warps' runs, repeated and
dropped experts, and the first number of pairs that a launch of its own counts."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import hccl_b200 as hb
from hccl_b200 import Communicator
from hccl_b200.ops.moe import MoeDispatcher


@pytest.mark.parametrize("tokens,topk,experts", [(1, 1, 2), (31, 1, 4), (33, 2, 6), (512, 1, 512), (513, 1, 8), (512, 8, 16), (4095, 1, 32), (1025, 4, 32), (2049, 2, 16)])
@pytest.mark.parametrize("same", [False, True])
def test_every_pair_has_a_slot_of_its_own(tokens, topk, experts, same):
    p, hidden = 2, 128
    comms = Communicator.emulated(p, hb.make_config(buffer_mib=8))
    cap = p * tokens * topk
    disp = [MoeDispatcher(c, tokens, hidden, topk, experts, capacity=cap) for c in comms]
    g = torch.Generator(device="cuda").manual_seed(tokens)
    xs = [torch.randn(tokens, hidden, device="cuda", generator=g).bfloat16() for _ in comms]
    idx = [torch.randint(-1, experts + 1, (tokens, topk), device="cuda", generator=g, dtype=torch.int32) for _ in comms]
    if same:
        idx = [torch.full_like(i, experts - 1) for i in idx]
    for _ in range(2):
        res = [d.dispatch(x, i) for d, x, i in zip(disp, xs, idx)]
        torch.cuda.synchronize()
        per = experts // p
        for r in range(p):
            counts = torch.stack([sum((i == r * per + e).sum() for i in idx) for e in range(per)])
            assert torch.equal(res[r].offsets.long(), torch.cat((counts.new_zeros(1), counts.cumsum(0))))
            n = int(counts.sum())
            src = res[r].src_info[:n]
            rank, pair = src >> 32, src & 0xFFFFFFFF
            assert torch.unique(src).numel() == n                      # no slot was written twice, none left out
            expert = torch.stack(idx)[rank, pair // topk, pair % topk].long()
            assert torch.equal(expert, torch.repeat_interleave(torch.arange(per, device="cuda"), counts) + r * per)
            assert (rank.diff()[expert.diff() == 0] >= 0).all()        # inside an expert the sources are in rank order
    assert comms[0].async_error() == hb.Result.SUCCESS
    for c in comms:
        c.destroy()


# one CTA adds up and scans up to 1024 experts, eight share them beyond; every CTA counts up to 8192
@pytest.mark.parametrize("experts", [1, 31, 256, 1023, 1024, 1025, 8192, 8193])
@pytest.mark.parametrize("pairs", [1, 4097, 65536])
def test_expert_offsets_at_the_edges(experts, pairs):
    from hccl_b200.ops.moe import expert_offsets
    g = torch.Generator(device="cuda").manual_seed(experts)
    ids = [torch.randint(-1, experts, (pairs,), device="cuda", generator=g, dtype=torch.int32) for _ in range(4)]
    got = [expert_offsets(i, experts) for i in ids]                     # back to back: one starts under the other's end
    for i, off in zip(ids, got):
        n = torch.bincount(i[i >= 0].long(), minlength=experts)
        assert torch.equal(off, torch.cat((n.new_zeros(1), n.cumsum(0))).int())
