"""Products of few tiles: every kernel and cut that the estimates choose among, at the edges of its tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_gpu_tile_edges import LAYOUTS, _check_matmul
from test_matmul_plan import plan

# (m, n, k) with [N, K] weights: one token to 128, single CTAs and clusters of two to eight, k-blocks shared evenly and not, whole
# and ragged inner dimensions, columns that end inside a tile, several token tiles
CUTS = [((1, 64, 16000), {"split": "8", "bn": "128"}), ((16, 1000, 8200), {"split": "8", "bn": "128"}), ((17, 136, 4104), {"split": "8", "bt": "32"}),
        ((33, 8, 1000), {"split": "8", "bt": "32"}), ((65, 264, 2056), {"split": "8", "bt": "32"}), ((32, 4096, 8192), {"split": "4", "bn": "128"}),
        ((100, 520, 136), {"split": "1", "bt": "32"}), ((72, 1000, 72), {"split": "1", "bt": "32"}), ((128, 8192, 1032), {"split": "1", "bt": "64"}),
        ((256, 128, 1000), {"split": "8", "bn": "64"}), ((136, 200, 1000), {"split": "8", "bt": "48"}),
        ((250, 136, 8200), {"split": "8", "bt": "64"}), ((1000, 72, 2504), {"split": "4", "bt": "64"})]


def _rows(shape, ta):
    m, n, k = shape
    return m + (-m % 8 if ta else 0), n, k                        # MN-major rows come in eights


def _token_split(shape, cut, ta, tb):
    p = plan(*_rows(shape, ta), int(ta), int(tb))
    if ta:                                                        # MN-major tokens: whole boxes of 64, weight tiles of 128 rows
        cut = {"split": cut["split"], "bn": "128", "bt": p["bt"] if p["bt"] == "128" else "64"}
    assert p["route"] == "split" and {k: p[k] for k in cut} == cut, p
    _check_matmul(*_rows(shape, ta), ta, tb)


@pytest.mark.parametrize("ta,tb", LAYOUTS)
@pytest.mark.parametrize("shape,cut", CUTS)
def test_token_split(shape, cut, ta, tb):
    _token_split(shape, cut, ta, tb)


# the cluster sizes and heights of a weight tile that the shapes above leave out: a kernel each
KERNELS = [((1, 8, 456), {"split": "2", "bn": "128"}), ((24, 8, 712), {"split": "3", "bn": "128"}), ((1, 8, 536), {"split": "1", "bn": "64"}),
           ((136, 1480, 1992), {"split": "2", "bn": "64"}), ((64, 8, 904), {"split": "4", "bn": "64"})]
KERNELS_MN = [((8, 8, 864), "3"), ((136, 5656, 4272), "3"), ((72, 2472, 1208), "4"), ((1000, 8, 4648), "8")]


@pytest.mark.parametrize("tb", [True, False])
@pytest.mark.parametrize("shape,cut", KERNELS)
def test_every_cluster_size(shape, cut, tb):
    _token_split(shape, cut, False, tb)


@pytest.mark.parametrize("tb", [True, False])
@pytest.mark.parametrize("shape,split", KERNELS_MN)
def test_every_cluster_size_with_mn_major_tokens(shape, split, tb):
    _token_split(shape, {"split": split}, True, tb)


def test_clusters_of_two_over_many_tokens():
    _token_split((128, 5872, 2440), {"split": "2", "bt": "128"}, False, True)
    _token_split((64, 464, 600), {"split": "2"}, True, True)


# short inner dimensions on one-SM tiles, long ones with few rows on 256 x 256 tiles that pairs share
OTHERS = [((1000, 4104, 72), "one_sm", {"bn": "256"}), ((520, 7304, 200), "one_sm", {"bn": "256"}), ((200, 10248, 200), "one_sm", {"bn": "128"}),
          ((120, 7000, 256), "one_sm", {"bn": "128"}), ((255, 5192, 9888), "two_sm_split", {"bn": "256", "split": "3"}),
          ((300, 2056, 12008), "two_sm_split", {"bn": "256", "split": "3"}), ((759, 3824, 1552), "two_sm", {"bn": "160"})]


@pytest.mark.parametrize("ta,tb", LAYOUTS)
@pytest.mark.parametrize("shape,route,cut", OTHERS)
def test_other_kernels(shape, route, cut, ta, tb):
    p = plan(*_rows(shape, ta), int(ta), int(tb))
    if shape == (120, 7000, 256) and (ta or not tb):              # rows on 16 bytes only: the token split's estimate is as good
        route, cut = "split", {"split": "1", "bt": "64"}
    assert p["route"] == route and {k: p[k] for k in cut} == cut, p
    _check_matmul(*_rows(shape, ta), ta, tb)


def test_a_row_that_does_not_depend_on_the_buffer_next_to_it():
    """The last columns of a 64-row tile lie beyond the matrix: nothing is written there."""
    from hccl_b200.ops import mc2
    m, n, k = 3, 72, 8200
    whole = torch.full((m * n + 64,), 7.0, device="cuda", dtype=torch.bfloat16)
    a, b = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    mc2.matmul(a, b, out=whole[:m * n].view(m, n))
    want = (a.double() @ b.double().t()).float()
    assert ((whole[:m * n].view(m, n).float() - want).norm() / want.norm()).item() < 3e-3
    assert (whole[m * n:] == 7).all()


def test_a_lone_tile_is_stored_whole_or_not_at_all():
    """Waits that run out anywhere in the middle of the work, in warps of one tile that look at different times."""
    import ctypes
    from hccl_b200._lib import lib
    from hccl_b200.comm import HcclError
    from hccl_b200.ops import mc2
    m, n, k = 128, 8192, 1024
    p = plan(m, n, k)
    assert (p["route"], p["split"], p["bt"], p["bn"]) == ("split", "1", "64", "128")
    g = torch.Generator(device="cuda").manual_seed(1)
    a, b = torch.randn(m, k, device="cuda", generator=g).bfloat16(), torch.randn(n, k, device="cuda", generator=g).bfloat16()
    want = mc2.matmul(a, b)
    f = lib.HcclDebugMatmulStalled
    f.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_uint64] * 3 + [ctypes.c_int] * 3 + [ctypes.c_uint64, ctypes.c_void_p]
    stored = 0
    for limit in [0, 200, 500, 1000] + list(range(1500, 4500, 100)) + [6000, 1_000_000]:
        out = torch.full((m, n), 7.0, device="cuda", dtype=torch.bfloat16)
        assert f(a.data_ptr(), b.data_ptr(), out.data_ptr(), m, n, k, 0, 1, -1, limit, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        tiles, wanted = (t.view(2, 64, 64, 128).transpose(1, 2).reshape(128, -1) for t in (out, want))
        whole, untouched = (tiles == wanted).all(1), (tiles == 7.0).all(1)
        assert (whole | untouched).all(), limit
        stored += int(whole.sum())
        try:                                                                     # a launch that gave up is reported to the next call
            mc2.matmul(a, b)
        except HcclError:
            pass
    assert stored >= 128 and torch.equal(mc2.matmul(a, b), want)
