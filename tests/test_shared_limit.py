"""csrc/shared_limit.h against a stand-in for the runtime: launches of different sizes that start at the same time leave the
kernel with what the largest of them needs."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")), "..")

SOURCE = r"""
#include "shared_limit.h"
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>

static std::mutex mu;
static std::condition_variable cv;
static int waiting = 0, value = -1, sets = 0;
static bool fail_first = false;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 232448; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { *a = cudaFuncAttributes{}; a->sharedSizeBytes = 448; return cudaSuccess; }
// both threads have found nothing set by the time either sets it; the smaller launch's comes last
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) {
    std::unique_lock<std::mutex> lock(mu);
    if (fail_first) { fail_first = false; return cudaErrorInvalidValue; }
    ++waiting;
    cv.notify_all();
    cv.wait_for(lock, std::chrono::seconds(10), [] { return waiting >= 2; });
    value = value < 0 || v < value ? v : value;
    ++sets;
    return cudaSuccess;
}
}
static void kernel() {}
int main() {
    static hqm::SharedLimits limits, other;
    bool small = false, large = false;
    std::thread a([&] { small = hqm::allow_shared(kernel, limits, 177920); }), b([&] { large = hqm::allow_shared(kernel, limits, 206848); });
    a.join();
    b.join();
    if (!small || !large || value < 206848 || value + 448 > 232448) return printf("allowed %d, %d: %d bytes\n", small, large, value), 1;
    if (!hqm::allow_shared(kernel, limits, 206848) || sets != 2) return printf("set again\n"), 1;
    if (hqm::allow_shared(kernel, limits, 232448)) return printf("more than there is\n"), 1;
    fail_first = true;
    if (hqm::allow_shared(kernel, other, 177920) || !hqm::allow_shared(kernel, other, 206848)) return printf("a refusal that stays\n"), 1;
    return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")), reason="no CUDA headers")
def test_launches_of_different_sizes(tmp_path):
    src, exe = tmp_path / "limits.cpp", tmp_path / "limits"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-pthread", f"-I{CUDA}/include", f"-I{ROOT}/mixtral_offloading_b200/csrc", "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
