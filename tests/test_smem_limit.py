"""allow_smem (mat3d_b200/csrc/smem_limit.cuh) called by several threads at
once: none may return, and so launch the kernel, before the kernel's limit is
set.  A host program against a stand-in for the four runtime calls."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
#include "smem_limit.cuh"
static std::atomic<int> limit{48 * 1024}, sets{0};
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void*) {
    std::this_thread::sleep_for(std::chrono::milliseconds(50));  // the first such call loads the kernel
    a->sharedSizeBytes = 1024;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, enum cudaFuncAttribute, int v) { limit = v; ++sets; return cudaSuccess; }
}
static void kernel(int) {}
int main() {
    std::atomic<int> early{0};
    std::vector<std::thread> t;
    for (int i = 0; i < 8; ++i)
        t.emplace_back([&] {
            m3d::allow_smem(kernel);
            if (limit != 226 * 1024) ++early;
        });
    for (auto& x : t) x.join();
    printf("early %d sets %d\n", early.load(), sets.load());
    return early || sets != 1;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")),
                    reason="needs g++ and the CUDA headers")
def test_no_caller_returns_before_the_limit_is_set(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "mat3d_b200", "csrc"), "-I", CUDA_INCLUDE,
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
