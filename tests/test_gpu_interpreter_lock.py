"""The native calls give the interpreter's lock away while the C API works: a call that waits there does not keep the other Python
threads from what it waits for."""
import ctypes
import subprocess
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

from hccl_b200 import _calls
from hccl_b200._lib import lib

# stands in for a function of the C API: returns 0 once another thread has let it go, 9 (and nobody waits any longer) after two seconds
STUB = """
#include <time.h>
static volatile int entered, released;
void reset(void) { entered = released = 0; }
int has_entered(void) { return entered; }
void let_go(void) { released = 1; }
int wait_for_it(void)
{
    struct timespec ms = {0, 1000000};
    entered = 1;
    for (int i = 0; i < 2000 && !released; ++i) nanosleep(&ms, 0);
    return released ? 0 : 9;
}
"""


@pytest.fixture(scope="module")
def stub(tmp_path_factory):
    d = tmp_path_factory.mktemp("stub")
    (d / "stub.c").write_text(STUB)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(d / "stub.so"), str(d / "stub.c")], check=True)
    return ctypes.CDLL(str(d / "stub.so"))


def _bf16(*shape):
    return torch.zeros(*shape, device="cuda", dtype=torch.bfloat16)


def _f32(*shape):
    return torch.zeros(*shape, device="cuda")


CALLS = {
    "HcclFusedAddRmsNormFwd": lambda: _calls.add_rms_norm(_bf16(4, 64), _bf16(4, 64), _bf16(64), 1e-5),
    "HcclFusedRmsNormBwdCopy": lambda: _calls.rms_norm_bwd(_bf16(4, 64), _bf16(4, 64), _bf16(64), _f32(4), None, True),
    "HcclFusedSwigluFwd": lambda: _calls.swiglu_fwd(_bf16(4, 64)),
    "HcclFusedSwigluBwd": lambda: _calls.swiglu_bwd(_bf16(4, 64), _bf16(4, 32)),
    "HcclFusedRope": lambda: _calls.rope(_bf16(4, 2, 16), _f32(4, 8), _f32(4, 8), False),
    "HcclMc2Matmul": lambda: _calls.matmul(_bf16(8, 16), _bf16(8, 16), False, True, None, None),
    "HcclMoeExpertOffsets": lambda: _calls.expert_offsets(torch.zeros(4, device="cuda", dtype=torch.int32), 4, None),
    "HcclAllReduce": lambda: _calls.collective(0, 1, _f32(4), _f32(4), 0, 2, None),
    "HcclReduceScatter": lambda: _calls.collective(1, 1, _f32(4), _f32(2), 0, 2, None),
    "HcclAllGather": lambda: _calls.collective(2, 1, _f32(4), _f32(8), 0, 2, None),
    "HcclAlltoAll": lambda: _calls.collective(3, 1, _f32(4), _f32(4), 0, 2, None),
}


def test_every_function_of_the_module_is_tried():
    assert set(CALLS) == set(_calls._module.names()) - {"HcclFusedRmsNormBwdPartials"}


@pytest.mark.parametrize("name", CALLS)
def test_another_thread_runs_while_a_call_waits(stub, name):
    real = {n: ctypes.cast(getattr(lib, n), ctypes.c_void_p).value for n in _calls._module.names()}
    stub.reset()

    def let_go():
        while not stub.has_entered():
            time.sleep(0.001)
        stub.let_go()

    helper = threading.Thread(target=let_go)
    helper.start()
    try:
        _calls._module.bind({**real, name: ctypes.cast(stub.wait_for_it, ctypes.c_void_p).value})
        answer = CALLS[name]()
    finally:
        _calls._module.bind(real)
        helper.join(10)
    assert answer is not None and not (type(answer) is int and answer != 0), answer
