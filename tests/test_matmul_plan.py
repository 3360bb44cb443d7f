"""Which kernel a plain matmul takes, from its sizes and the switches of the environment (no GPU needed)."""
import ctypes
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def plan(m, n, k, trans_a=0, trans_b=1, sms=148):
    from hccl_b200._lib import lib
    text = ctypes.create_string_buffer(256)
    lib.HcclDebugMatmulPlan.argtypes = [ctypes.c_uint64] * 3 + [ctypes.c_int] * 2 + [ctypes.c_uint32, ctypes.c_char_p, ctypes.c_uint32]
    assert lib.HcclDebugMatmulPlan(m, n, k, trans_a, trans_b, sms, text, 256) == 0
    return dict(kv.split("=") for kv in text.value.decode().split())


def plan_with(env, *shape):
    code = f"import sys; sys.path.insert(0, 'tests'); import test_matmul_plan as t; print(t.plan(*{shape!r}))"
    base = {k: v for k, v in os.environ.items() if not k.startswith("HCCL_MC2_")}
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=ROOT, env={**base, **env})
    assert r.returncode == 0, r.stderr[-2000:]
    return eval(r.stdout.strip().splitlines()[-1])


WIDE_SHAPE = (4096, 57344, 8192)


@pytest.mark.parametrize("env,route,hints", [
    ({}, "wide", "00"),
    ({"HCCL_MC2_WIDE": "0"}, "two_sm", "00"),
    ({"HCCL_MC2_L2_HINTS": "1"}, "two_sm", "12"),                             # asking for hints keeps the kernel that takes them
    ({"HCCL_MC2_L2_HINTS": "1", "HCCL_MC2_WIDE": "1"}, "wide", "00"),
    ({"HCCL_MC2_L2_HINTS": "1", "HCCL_MC2_WIDE": "auto"}, "wide", "00"),
    ({"HCCL_MC2_2SM": "0"}, "one_sm", "00"),
])
def test_switches(env, route, hints):
    p = plan_with(env, *WIDE_SHAPE)
    assert (p["route"], p["hints"]) == (route, hints)


def test_the_gpu_tests_reach_the_forms_they_are_named_after():
    import test_gpu_tile_edges as edges
    for ta, tb in edges.LAYOUTS:
        for shape, singles in edges.WIDE_SINGLES:
            p = plan(*shape, int(ta), int(tb))
            assert p["route"] == "wide" and -(-int(p["singles"]) // 74) == singles, (shape, p)
        for shape in edges.SPLIT_OF_THREE:
            p = plan(*shape, int(ta), int(tb))
            assert p["route"] == "split" and p["split"] == "3", (shape, p)
    for shape in edges.WIDE_SHORT_K:
        assert plan(*shape)["route"] == "two_sm" and plan_with({"HCCL_MC2_WIDE": "1"}, *shape)["route"] == "wide"
