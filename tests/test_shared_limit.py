"""The shared-memory limit of a kernel is only ever raised, whichever threads look at it and raise it (host code, no GPU)."""
import shutil
import subprocess

import pytest

from tilecadence_b200 import cuda_runtime

# The runtime calls that tc_host.cuh makes, on a limit of the test's own. The first look at the attributes lets another
# thread raise the limit for its launch before the first thread goes on.
SOURCE = r"""
#include <atomic>
#include <chrono>
#include <thread>
#include "tc_host.cuh"

static std::atomic<int> limit{48 * 1024};
static std::atomic<bool> first{true};
static std::thread other;
static const char code = 0;
static const void* const kernel = &code;

extern "C" {
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    a->maxDynamicSharedSizeBytes = limit;
    if (first.exchange(false)) {
        other = std::thread([] { tc::raise_shared_limit(kernel, 120 * 1024); });
        std::this_thread::sleep_for(std::chrono::milliseconds(200));
    }
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int value) { limit = value; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 1; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 1; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
}

int main() {
    int64_t values[8];
    int status = tc::kernel_resources(kernel, 160, 100 * 1024, values);
    other.join();
    if (status == 0) status = tc::raise_shared_limit(kernel, 90 * 1024);
    return status == 0 && limit == 120 * 1024 ? 0 : 1;
}
"""


def test_a_look_at_the_resources_never_lowers_the_limit_of_a_launch(tmp_path):
    nvcc = cuda_runtime.find_nvcc()
    if shutil.which("g++") is None or nvcc is None:
        pytest.skip("g++ and the CUDA headers are needed")
    source, program = tmp_path / "limit.cpp", tmp_path / "limit"
    source.write_text(SOURCE)
    includes = [cuda_runtime.CSRC / "common", cuda_runtime.INCLUDE, nvcc.parent.parent / "include"]
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", *(f"-I{path}" for path in includes), "-x", "c++", str(source),
                    "-Wl,--unresolved-symbols=ignore-all", "-o", str(program)], check=True)
    subprocess.run([str(program)], check=True, timeout=60)


def test_the_limit_is_set_in_one_place():
    setters = [path.name for path in sorted(cuda_runtime.CSRC.rglob("*.cu*"))
               if "cudaFuncAttributeMaxDynamicSharedMemorySize" in path.read_text()]
    assert setters == ["tc_host.cuh", "plan.cu"]  # the generated plan.cu always asks for the same amount
