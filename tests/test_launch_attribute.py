"""launch_cooperative's programmatic-launch attribute, with the two runtime calls it makes replaced on the host (no GPU)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SOURCE = r"""
#include <cstdio>
#include <cuda_runtime.h>
__global__ void refused() {}
__global__ void taken() {}
static int with_attribute[2], without[2];
static cudaError_t launch_ex(const cudaLaunchConfig_t*, const void* k, void**) {
    ++with_attribute[k == (const void*) taken];
    return k == (const void*) taken ? cudaSuccess : cudaErrorInvalidValue;
}
static cudaError_t launch_coop(const void* k, dim3, dim3, void**, size_t, cudaStream_t) {
    ++without[k == (const void*) taken];
    return cudaSuccess;
}
#define cudaLaunchKernelExC launch_ex
#define cudaLaunchCooperativeKernel launch_coop
#include "maya_token_phase.cuh"
namespace maya { int note_launch(const char*) { return 0; } }
int main() {
    for (int i = 0; i < 3; ++i) maya::launch_cooperative<refused>(dim3(1), dim3(32), nullptr, 0, nullptr, "refused");
    for (int i = 0; i < 3; ++i) maya::launch_cooperative<taken>(dim3(1), dim3(32), nullptr, 0, nullptr, "taken");
    std::printf("%d %d %d %d\n", with_attribute[0], without[0], with_attribute[1], without[1]);
}
"""


def test_an_attribute_refused_for_one_kernel_stays_in_use_for_the_others(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc on this machine")
    src, exe = tmp_path / "launch.cu", tmp_path / "launch"
    src.write_text(SOURCE)
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", str(ROOT / "include"), "-I", str(ROOT / "project_maya_b200/csrc")]
    subprocess.run([nvcc, *flags, "-o", str(exe), str(src)], check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.split()
    # refused once, then launched without the attribute; the other kernel keeps it
    assert [int(v) for v in out] == [1, 3, 3, 0]
