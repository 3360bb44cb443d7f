"""What the launchers set or ask once per GPU, in a process that drives several (csrc/core/per_device.h), against a fake of
the runtime's device calls."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include "core/per_device.h"
#include <cstdio>
static int g_dev = 0, g_asked = 0;
static bool g_known = true;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = g_dev; return g_known ? cudaSuccess : cudaErrorNoDevice; }
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) { ++g_asked; *v = 100 + d; return cudaSuccess; }
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main()
{
    using namespace hccl;
    static OncePerDevice once, other;
    int n = 0, fails = 1;
    auto set = [&]() -> HcclResult { ++n; return HCCL_SUCCESS; };
    CHECK(once(set) == HCCL_SUCCESS && once(set) == HCCL_SUCCESS && n == 1);
    g_dev = 3;                                                     // the second GPU gets its own attribute
    CHECK(once(set) == HCCL_SUCCESS && n == 2 && once(set) == HCCL_SUCCESS && n == 2);
    CHECK(other([&]() -> HcclResult { return fails-- > 0 ? HCCL_E_RUNTIME : HCCL_SUCCESS; }) == HCCL_E_RUNTIME);
    CHECK(other(set) == HCCL_SUCCESS && n == 3 && other(set) == HCCL_SUCCESS && n == 3);      // a failure is tried again
    g_dev = kMaxDevices;                                           // no place to remember it: every time
    CHECK(once(set) == HCCL_SUCCESS && once(set) == HCCL_SUCCESS && n == 5);
    CHECK(SmCount() == 100 + kMaxDevices && SmCount() == 100 + kMaxDevices && g_asked == 2);
    g_dev = 0;
    CHECK(SmCount() == 100 && SmCount() == 100 && g_asked == 3);
    g_dev = 7;
    CHECK(SmCount() == 107 && g_asked == 4);
    g_known = false;
    CHECK(SmCount() == 148);
    printf("ok\n");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not Path(CUDA_HOME, "include", "cuda_runtime.h").exists(), reason="needs g++ and the CUDA headers")
def test_every_device_is_set_up_on_its_own(tmp_path):
    src, exe = tmp_path / "per_device.cc", tmp_path / "per_device"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", f"-I{ROOT / 'csrc'}", f"-I{ROOT / 'csrc' / 'include'}", f"-I{CUDA_HOME}/include", str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


def test_launchers_keep_no_process_wide_device_facts():
    """Launch attributes and SM counts go through the per-device helpers in every launcher."""
    for src in sorted((ROOT / "csrc" / "kernels").glob("*.cu")):
        for line in src.read_text().splitlines():
            assert "static bool" not in line and "static int n = 0" not in line, f"{src.name}: {line.strip()}"
