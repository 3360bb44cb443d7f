"""Two-SM matmul tiles with the inner dimension split over a cluster of CTA pairs, and two-SM products that end in a round of few
tiles, against float64.  Tolerance: one rounding to bf16 and fp32 sums, as in test_gpu_tile_edges."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

from hccl_b200.ops import mc2
from test_gpu_tile_edges import LAYOUTS, _check_matmul
from test_matmul_plan import plan

# (m, n, k), pairs per tile: k-blocks that the pairs share evenly and not, ragged rows (an idle second half of a tile among them),
# columns that end inside a 32-column chunk and inside a tile, row tiles in more than one band of the raster
SPLIT_PAIRS = [((136, 520, 2056), 4), ((304, 640, 4096), 4), ((256, 1024, 2048), 4), ((264, 1272, 2120), 3), ((200, 2584, 2048), 3), ((520, 1280, 2176), 2),
               ((2312, 392, 2048), 1), ((600, 1928, 2248), 1), ((200, 9472, 2048), 1)]


@pytest.mark.parametrize("ta,tb", LAYOUTS)
@pytest.mark.parametrize("shape,pairs", SPLIT_PAIRS)
def test_split_over_pairs(shape, pairs, ta, tb):
    p = plan(*shape, int(ta), int(tb))
    assert (p["route"], p["split"]) == ("two_sm_split", str(pairs))
    _check_matmul(*shape, ta, tb)


# (m, n, k) of two-SM products that end in a round of few tiles
LAST_ROUND = [(1024, 10240, 4096), (1000, 10240, 8192), (2560, 4096, 4104), (4096, 3584, 8192)]


@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("shape", LAST_ROUND)
def test_last_round_of_few_tiles(shape, ta):
    assert plan(*shape, int(ta), 0)["route"] == "two_sm"
    _check_matmul(*shape, ta, False)


@pytest.mark.parametrize("shape", LAST_ROUND)
def test_all_tiles_of_a_product_add_in_one_order(shape):
    """Columns moved by half the matrix land in other tiles, of other rounds: the same bits."""
    m, n, k = shape
    assert plan(*shape, 0, 0)["route"] == "two_sm"
    g = torch.Generator(device="cuda").manual_seed(n)
    a, w = torch.randn(m, k, device="cuda", generator=g).bfloat16(), (torch.randn(k, n, device="cuda", generator=g) * 0.02).bfloat16()
    moved = mc2.matmul(a, w.roll(n // 2, 1), trans_b=False)
    assert torch.equal(mc2.matmul(a, w, trans_b=False).roll(n // 2, 1), moved)


def test_products_in_a_chain():
    """Back to back, on streams and in a graph: a product's start overlaps the end of the one before it."""
    g = torch.Generator(device="cuda").manual_seed(9)
    rnd = lambda *s: (torch.randn(*s, device="cuda", generator=g) * 0.05).bfloat16()  # noqa: E731
    a, w, back = rnd(1000, 4096), rnd(4096, 10240), rnd(10240, 4096)

    def chain(each=lambda: None):
        x = a
        for _ in range(4):
            each()
            y = mc2.matmul(x, w, trans_b=False)
            each()
            x = mc2.matmul(y, back, trans_b=False)
            each()
            x = x * 0.5
        return x

    want = chain(torch.cuda.synchronize)
    for _ in range(5):
        assert torch.equal(chain(), want)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        chain()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = chain()
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


# the stalled CTA in the first pair and in another one, leader and second half: the others hold good partials and store nothing
@pytest.mark.parametrize("cta", [0, 1, 2, 5])
def test_split_pairs_that_give_up_a_wait(cta):
    from hccl_b200 import Result
    from hccl_b200._lib import lib
    from hccl_b200.comm import HcclError
    m, n, k = 256, 128, 2048
    assert plan(m, n, k)["split"] == "4"
    g = torch.Generator(device="cuda").manual_seed(k)
    a, b = (torch.randn(m, k, device="cuda", generator=g)).bfloat16(), torch.randn(n, k, device="cuda", generator=g).bfloat16()
    out = torch.full((m, n), 7.0, device="cuda", dtype=torch.bfloat16)
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (a, b, out)]
    lib.HcclDebugMatmulStalled.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_uint64] * 3 + [ctypes.c_int] * 3 + [ctypes.c_uint64, ctypes.c_void_p]
    assert lib.HcclDebugMatmulStalled(*ptr, m, n, k, 0, 1, cta, 1_000_000, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert (out == 7.0).all()
    with pytest.raises(HcclError) as e:
        mc2.matmul(a, b)
    assert e.value.code == Result.E_TIMEOUT
    _check_matmul(m, n, k, False, True)
