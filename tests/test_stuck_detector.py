"""What the watchdog concludes from its readings of the operator counters (no GPU needed)."""
import ctypes

import pytest

from hccl_b200._lib import lib

NONE = (0, 0, 0)


def reports(readings, budget=10.0, step=1.0):
    """Positions of the readings, one per `step` seconds, that are reported."""
    n = len(readings)
    answered = (ctypes.c_int * n)(*[r[0] for r in readings])
    started, finished = ((ctypes.c_uint64 * n)(*[r[i] for r in readings]) for i in (1, 2))
    at, out = (ctypes.c_double * n)(*[1000.0 + i * step for i in range(n)]), (ctypes.c_int * n)()
    lib.HcclDebugStuckDetector.argtypes = [ctypes.c_double, ctypes.c_uint32] + [ctypes.c_void_p] * 5
    assert lib.HcclDebugStuckDetector(budget, n, answered, started, finished, at, out) == 0
    return [i for i in range(n) if out[i]]


@pytest.mark.parametrize("name,readings,want", [
    ("idle", [(1, 5, 5)] * 40, []),
    ("busy", [(1, 5 + i, 4 + i) for i in range(40)], []),
    ("stuck after a while, reported once per budget", [(1, 5, 5)] * 20 + [(1, 6, 5)] * 25, [31, 42]),
    ("the device answers no more", [(1, 5, 5)] * 20 + [NONE] * 25, [30, 41]),
    ("no answer from the first reading on", [NONE] * 12, [11]),
    ("stuck, then no answer", [(1, 6, 5)] * 6 + [NONE] * 6, [11]),
    ("no answer for less than a budget", ([(1, 5, 5)] + [NONE] * 9) * 4, []),
    ("the answer after a silence shows an operator that moves", [(1, 6, 5)] + [NONE] * 9 + [(1, 7, 6)] * 10, []),
    ("the answer after a silence shows the same operator", [(1, 6, 5)] + [NONE] * 9 + [(1, 6, 5)] * 3, [11]),
    ("stuck, then on", [(1, 6, 5)] * 12 + [(1, 6, 6)] * 20, [11]),
])
def test_readings(name, readings, want):
    assert reports(readings) == want
