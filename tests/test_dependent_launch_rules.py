"""The rules of kernels that start under the end of the kernel in front of them, read from the sources: breaking one can hang a GPU,
so no test tries it out."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "csrc" / "kernels"
CALL = re.compile(r"\b(TmemAlloc2?|AllowDependents|DependencyWait)\(")


def _kernels():
    """(name, calls in their order) of every kernel that calls AllowDependents."""
    out = []
    for path in sorted([*KERNELS.glob("*.cuh"), *KERNELS.glob("*.cu")]):
        if path.name == "dependent_launch.cuh":
            continue
        text = re.sub(r"//[^\n]*", "", path.read_text())
        text = re.sub(r"__(?:launch_bounds|cluster_dims)__\([^)]*\)", "", text)
        for part in re.split(r"__global__", text)[1:]:
            name = re.search(r"void\s+(\w+)\s*\(", part)
            calls = [m.group(1) for m in CALL.finditer(part)]
            if "AllowDependents" in calls:
                out.append((f"{path.name}:{name.group(1)}", calls))
    return out


KNOWN = _kernels()


def test_the_kernels_are_found():
    assert len(KNOWN) >= 12 and sum(any(c.startswith("TmemAlloc") for c in calls) for _, calls in KNOWN) >= 5, KNOWN


@pytest.mark.parametrize("name,calls", KNOWN, ids=[n for n, _ in KNOWN])
def test_a_follower_is_let_in_behind_the_allocation_of_tensor_memory(name, calls):
    allow = calls.index("AllowDependents")
    assert all(i < allow for i, c in enumerate(calls) if c.startswith("TmemAlloc")), (name, calls)


@pytest.mark.parametrize("name,calls", KNOWN, ids=[n for n, _ in KNOWN])
def test_every_kernel_waits(name, calls):
    assert calls.count("DependencyWait") == 1, (name, calls)
