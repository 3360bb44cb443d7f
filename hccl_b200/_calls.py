"""Calls of the C API with torch tensors through the native module of csrc/torch/torch_calls.cc.

Each function takes what is plain and returns ``None`` for everything else; the caller then goes the general way through
``torch.autograd.Function`` and ctypes.  Where the module is not there (a library without it; a Python or a torch other than
the ones it was built for, which its file name holds) that is every call.
``result`` turns the answer into the outputs, or raises for the ``HcclResult`` of a call that failed.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import warnings

import torch          # its libraries have to be loaded before the module's

from ._lib import lib
from .build import torch_lib
from .comm import HcclError, _check


def _nothing(*_):
    return None


def _load():
    path = torch_lib()
    try:
        loader = importlib.machinery.ExtensionFileLoader("hccl_b200_torch", str(path))
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("hccl_b200_torch", loader))
        loader.exec_module(module)
        module.raises(HcclError)
        module.bind({name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in module.names()})
        if all(hasattr(lib, name) for name in module.backward_names()):
            module.bind_backward({name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in module.backward_names()})
        return module
    except (ImportError, AttributeError) as e:
        if torch.cuda.is_available():
            warnings.warn(f"{path.name} cannot be loaded ({e}): calls take the slower way through ctypes; `python hccl_b200/build.py` builds it")
        return None


_module = _load()
add_rms_norm, rms_norm_bwd, swiglu_fwd, swiglu_bwd, rope, matmul, expert_offsets, collective = (
    getattr(_module, name, _nothing)
    for name in ("add_rms_norm", "rms_norm_bwd", "swiglu_fwd", "swiglu_bwd", "rope", "matmul", "expert_offsets", "collective"))
# the same where gradients are recorded (``linear``: recorded or not)
add_rms_norm_grad, swiglu_grad, rope_grad, linear, embedding = (
    getattr(_module, name, _nothing) for name in ("add_rms_norm_grad", "swiglu_grad", "rope_grad", "linear", "embedding"))


def launches() -> int:
    """Kernels that the backward passes of these have launched (``linear`` counts in the tensor it is given)."""
    return _module.launches() if _module is not None else 0


def result(r, what: str):
    if type(r) is int:
        _check(r, what)
    return r
