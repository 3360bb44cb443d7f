"""The counts of started and finished operators live in device memory; the host reads them without waiting for the stream."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

import hccl_b200 as hb
from hccl_b200 import Communicator, Result
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
    torch.cuda._sleep(3_000_000_000)                               # more than a second
    for c, s in zip(comms, small):
        c.all_reduce(s)
    behind = torch.cuda.Event()
    behind.record()
    assert [_counters(c) for c in comms] == [(s + 3, f + 3) for s, f in first]
    assert not behind.query()                                      # read while the operators still wait for their turn
    torch.cuda.synchronize()
    assert [_counters(c) for c in comms] == [(s + 4, f + 4) for s, f in first]
    for c in comms:
        c.destroy()
    handle = ctypes.c_void_p()
    s = ctypes.c_uint64()
    assert lib.HcclDebugOpCounters(handle, ctypes.byref(s), ctypes.byref(s)) != 0


def test_a_reading_does_not_wait_for_a_stuck_operator():
    """The copy of the counters behind an operator that takes seconds, as where streams share a hardware queue: the reading gives up
    after its limit, for every communicator of the device, and the next one finds the device's answer."""
    lib.HcclDebugOpCounters.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint64), ctypes.POINTER(ctypes.c_uint64)]
    lib.HcclDebugOpCountersBehind.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    comms = Communicator.emulated(2, hb.make_config(buffer_mib=8))
    xs = [torch.ones(64, device="cuda") for _ in comms]

    def reduce():
        for c, x in zip(comms, xs):
            c.all_reduce(x)

    def read(c):
        s, f = ctypes.c_uint64(), ctypes.c_uint64()
        return lib.HcclDebugOpCounters(c.handle, ctypes.byref(s), ctypes.byref(f)), s.value, f.value

    reduce()
    torch.cuda.synchronize()
    r, started, finished = read(comms[0])
    assert r == Result.SUCCESS and started == finished >= 1
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(12_000_000_000)                          # six seconds and more
        reduce()
        done = torch.cuda.Event()
        done.record()
        assert lib.HcclDebugOpCountersBehind(comms[0].handle, side.cuda_stream) == 0
    got = [read(c)[0] for c in comms]
    assert not done.query()                                        # else it waited for the operator
    assert got == [Result.E_AGAIN] * 2
    torch.cuda.synchronize()
    assert [read(c) for c in comms] == [(Result.SUCCESS, started + 1, finished + 1)] * 2
    for c in comms:
        c.destroy()


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
