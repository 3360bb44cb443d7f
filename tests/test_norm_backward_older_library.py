"""The norm's backward pass with a library that has no entry point for a second copy of the gradient (no GPU needed)."""
import ctypes
from types import SimpleNamespace

import torch

from hccl_b200 import _calls
from hccl_b200.ops import fused


class Older:
    """The entry points as they were; the gradient that they would write is left as it is."""

    def __init__(self):
        self.calls = 0

    def HcclFusedRmsNormBwdPartials(self, rows):
        return 1

    def HcclFusedRmsNormBwd(self, *args):
        assert len(args) == 11
        self.calls += 1
        return 0


def test_two_leaves(monkeypatch):
    older = Older()
    monkeypatch.setattr(fused, "lib", older)
    monkeypatch.setattr(fused, "_s", lambda *_: ctypes.c_void_p(0))
    monkeypatch.setattr(_calls, "rms_norm_bwd", _calls._nothing)
    monkeypatch.setattr(fused, "_kept_apart", lambda *_: True)
    x, w = torch.zeros(4, 64, dtype=torch.bfloat16), torch.zeros(64, dtype=torch.bfloat16)
    ctx = SimpleNamespace(has_delta=True, saved_tensors=(x, w, torch.zeros(4)), next_functions=((None, 0), (None, 0)))
    dx, d_delta, dw, _ = fused._AddRmsNorm.backward(ctx, x, x)
    assert older.calls == 1 and d_delta is dx and dw.shape == w.shape
