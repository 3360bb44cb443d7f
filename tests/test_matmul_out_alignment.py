"""Outputs of the plain matmul that do not lie on 16 bytes: the token split stores 8 bytes at a time and takes them where it always
did, every other route stores 16 and such a call is refused before it reaches a kernel."""
import ctypes

import pytest
import torch

from hccl_b200 import Result
from hccl_b200._lib import lib
from hccl_b200.comm import HcclError


def plan(m, n, k, out_align, trans_a=0, trans_b=1):
    text = ctypes.create_string_buffer(256)
    lib.HcclDebugMatmulPlanOut.argtypes = [ctypes.c_uint64] * 3 + [ctypes.c_int] * 2 + [ctypes.c_uint32] * 2 + [ctypes.c_char_p, ctypes.c_uint32]
    assert lib.HcclDebugMatmulPlanOut(m, n, k, trans_a, trans_b, 148, out_align, text, 256) == 0
    return dict(kv.split("=") for kv in text.value.decode().split())["route"]


# (m, n, k), route on 16 bytes, on 8: the second, third and fourth were on the token split before the CTA pairs existed
SHAPES = [((16, 8192, 8192), "split", "split"), ((300, 2048, 4096), "two_sm_split", "split"), ((193, 1024, 8192), "two_sm_split", "split"),
          ((600, 1000, 4096), "two_sm_split", "split"), ((300, 2048, 2048), "two_sm_split", "refused"), ((256, 8192, 8192), "two_sm_split", "refused"),
          ((400, 1024, 1024), "one_sm", "refused"), ((4096, 57344, 8192), "wide", "refused"), ((2048, 7168, 1024), "two_sm", "refused")]


@pytest.mark.parametrize("shape,on16,on8", SHAPES)
def test_routes(shape, on16, on8):
    assert (plan(*shape, 16), plan(*shape, 8)) == (on16, on8)
    assert plan(*shape, 4) == plan(*shape, 2) == "refused"


def test_no_route_for_less_than_eight_bytes():
    assert lib.HcclMc2Matmul(ctypes.c_void_p(1 << 20), ctypes.c_void_p(1 << 21), ctypes.c_void_p((1 << 22) + 4), 16, 64, 64, 0, 1, None) == Result.E_PARA


def _out(m, n, shift):
    whole = torch.full((m * n + 16,), 7.0, device="cuda", dtype=torch.bfloat16)
    return whole, whole[shift:shift + m * n].view(m, n)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [s for s, _, on8 in SHAPES if on8 == "split"])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False)])
def test_output_on_eight_bytes(shape, ta, tb):
    from hccl_b200.ops import mc2
    from test_gpu_tile_edges import ONE_ROUNDING, _rel
    m, n, k = shape
    assert plan(m, n, k, 8, int(ta), int(tb)) == "split"
    g = torch.Generator(device="cuda").manual_seed(m)
    a, b = torch.randn(m, k, device="cuda", generator=g).bfloat16(), torch.randn(*((n, k) if tb else (k, n)), device="cuda", generator=g).bfloat16()
    whole, out = _out(m, n, 4)
    assert out.data_ptr() % 16 == 8
    mc2.matmul(a, b, trans_b=tb, out=out)
    want = a.double() @ (b.double().t() if tb else b.double())
    assert _rel(out, want) <= ONE_ROUNDING
    assert (whole[:4] == 7).all() and (whole[m * n + 4:] == 7).all()


@pytest.mark.gpu
@pytest.mark.parametrize("shape,shift", [((400, 1024, 1024), 4), ((256, 8192, 2048), 4), ((16, 256, 256), 2), ((16, 256, 256), 1)])
def test_refused(shape, shift):
    from hccl_b200.ops import mc2
    m, n, k = shape
    a, b = torch.ones(m, k, device="cuda", dtype=torch.bfloat16), torch.ones(n, k, device="cuda", dtype=torch.bfloat16)
    whole, out = _out(m, n, shift)
    with pytest.raises(HcclError) as e:
        mc2.matmul(a, b, out=out)
    assert e.value.code == Result.E_PARA
    torch.cuda.synchronize()
    assert (whole == 7).all()
