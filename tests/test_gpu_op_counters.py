"""The counts of started and finished operators live in device memory; the host reads them without waiting for the stream."""
import ctypes
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

import hccl_b200 as hb
from hccl_b200 import Communicator
from hccl_b200._lib import lib


def _counters(c):
    lib.HcclDebugOpCounters.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint64), ctypes.POINTER(ctypes.c_uint64)]
    s, f = ctypes.c_uint64(), ctypes.c_uint64()
    assert lib.HcclDebugOpCounters(c.handle, ctypes.byref(s), ctypes.byref(f)) == 0
    return s.value, f.value


def test_counters_of_operators():
    comms = Communicator.emulated(4, hb.make_config(buffer_mib=8))
    small = [torch.ones(64, device="cuda") for _ in comms]
    large = [torch.ones(1 << 18, device="cuda") for _ in comms]
    for c, s in zip(comms, small):
        c.all_reduce(s)
    torch.cuda.synchronize()
    first = [_counters(c) for c in comms]
    assert all(s == f and s >= 1 for s, f in first)
    for _ in range(3):
        for c, s in zip(comms, large):
            c.all_reduce(s)
    torch.cuda.synchronize()
    assert [_counters(c) for c in comms] == [(s + 3, f + 3) for s, f in first]
    torch.cuda._sleep(1_500_000_000)                               # most of a second
    t = time.perf_counter()
    for c, s in zip(comms, small):
        c.all_reduce(s)
    assert [_counters(c) for c in comms] == [(s + 3, f + 3) for s, f in first]
    assert time.perf_counter() - t < 0.3
    torch.cuda.synchronize()
    assert [_counters(c) for c in comms] == [(s + 4, f + 4) for s, f in first]
    for c in comms:
        c.destroy()
    handle = ctypes.c_void_p()
    s = ctypes.c_uint64()
    assert lib.HcclDebugOpCounters(handle, ctypes.byref(s), ctypes.byref(s)) != 0


def test_counters_during_a_capture():
    comms = Communicator.emulated(2, hb.make_config(buffer_mib=8))
    xs = [torch.ones(4096, device="cuda") for _ in comms]
    for c, x in zip(comms, xs):
        c.all_reduce(x)
    torch.cuda.synchronize()
    before = [_counters(c) for c in comms]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for c, x in zip(comms, xs):
            c.all_reduce(x)
        assert [_counters(c) for c in comms] == before
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert [_counters(c) for c in comms] == [(s + 2, f + 2) for s, f in before]
    for c in comms:
        c.destroy()
