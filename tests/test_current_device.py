"""The native front ends' device guard in the states torch's per-thread note of a device can leave a thread in; no GPU: a C++ program
that is linked against torch's c10_cuda and has the CUDA runtime's device functions of its own."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest
import torch

from flaggems_vllm import build

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "current_device.h"

namespace c10::cuda::_internal {
void setHasPrimaryContext(bool (*has)(c10::DeviceIndex));  // exported by c10_cuda, in no header; libtorch_cuda sets it
}

static int runtime_device = 1;  // the fake runtime's device of this thread
extern "C" cudaError_t cudaGetDevice(int* device) { *device = runtime_device; return cudaSuccess; }
extern "C" cudaError_t cudaSetDevice(int device) { runtime_device = device; return cudaSuccess; }
extern "C" cudaError_t cudaGetDeviceCount(int* count) { *count = 4; return cudaSuccess; }
static bool only_device_1(c10::DeviceIndex device) { return device == 1; }

int main(int count, char** arguments) {
    const int runtime = std::atoi(arguments[1]), noted = std::atoi(arguments[2]), wanted = std::atoi(arguments[3]);
    c10::cuda::_internal::setHasPrimaryContext(only_device_1);
    runtime_device = runtime;
    if (noted >= 0) c10::cuda::MaybeSetDevice(static_cast<c10::DeviceIndex>(noted));  // what the end of a torch guard does
    if (count > 4) {  // a call that only launches
        const dsv4::OnDevice here(static_cast<c10::DeviceIndex>(wanted), dsv4::OnDevice::kLaunchesOnly);
        std::printf("%d\n", runtime_device);
        return 0;
    }
    const bool current = dsv4::is_current(static_cast<c10::DeviceIndex>(wanted));
    const int launched_on = dsv4::with_device(static_cast<c10::DeviceIndex>(wanted), [] { return runtime_device; });
    std::printf("%d %d %d %d\n", static_cast<int>(current), launched_on, static_cast<int>(c10::cuda::current_device()), runtime_device);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    at = tmp_path_factory.mktemp("current_device")
    (at / "main.cpp").write_text(PROGRAM)
    root = Path(torch.__file__).resolve().parent
    cuda = Path(build.nvcc_path()).resolve().parent.parent
    subprocess.run([shutil.which("g++") or "g++", "-O1", "-std=c++17", "-rdynamic", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
                    f"-I{build.CSRC}", f"-I{root / 'include'}", f"-I{cuda / 'include'}", str(at / "main.cpp"), "-o", str(at / "main"), f"-L{root / 'lib'}",
                    "-lc10_cuda", "-lc10", f"-Wl,-rpath,{root / 'lib'}", "-Wl,--unresolved-symbols=ignore-all"], check=True)
    return at / "main"


@pytest.mark.parametrize("runtime,noted,wanted,current", [
    (1, -1, 1, True),   # the ordinary call
    (1, 1, 1, True),    # noted and already the runtime's
    (1, 3, 3, False),   # noted, and the runtime is still elsewhere
    (1, 3, 1, False),   # the runtime's, but torch would allocate on the noted one
    (1, 0, 0, False),
    (1, -1, 0, False),  # another device altogether
    (0, 2, 3, False),
])
def test_the_wanted_device_is_the_runtimes(program, runtime, noted, wanted, current):
    said, launched_on, torch_after, _ = map(int, subprocess.run([str(program), str(runtime), str(noted), str(wanted)], check=True, capture_output=True, text=True).stdout.split())
    assert bool(said) == current and launched_on == wanted
    assert torch_after == (noted if noted >= 0 else runtime)  # torch's device afterwards is what it was


@pytest.mark.parametrize("runtime,noted,wanted", [(1, -1, 1), (1, 1, 1), (1, 3, 3), (1, 3, 1), (1, 0, 0), (1, -1, 0), (0, 2, 3)])
def test_a_call_without_outputs_launches_on_the_wanted_device(program, runtime, noted, wanted):
    said = subprocess.run([str(program), str(runtime), str(noted), str(wanted), "launch"], check=True, capture_output=True, text=True).stdout
    assert int(said) == wanted
