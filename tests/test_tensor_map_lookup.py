"""The tensor-map encoder's one-time look-up under threads (host code, no GPU)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "rlmusclev2_b200" / "csrc"

SOURCE = r"""
#include <chrono>
#include <thread>
#include <vector>
#include <atomic>
#include <cstdio>
#include <cuda_runtime.h>
static std::atomic<int> lookups{0};
// stands in for the runtime's look-up: slow, so that every thread arrives during the first one
static cudaError_t slow_lookup(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    ++lookups;
    std::this_thread::sleep_for(std::chrono::milliseconds(200));
    *p = reinterpret_cast<void*>(&slow_lookup);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
#define cudaGetDriverEntryPoint slow_lookup
#define cudaGetLastError() ((void)0)
#include "xpbd_mma.cuh"
int main() {
    std::atomic<int> missing{0};
    std::vector<std::thread> ts;
    for (int i = 0; i < 8; ++i) ts.emplace_back([&] { missing += xpbd::encode_tiled() == nullptr; });
    for (auto& t : ts) t.join();
    std::printf("%d %d\n", missing.load(), lookups.load());
    return 0;
}
"""


def test_no_thread_sees_a_look_up_in_progress(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    src, exe = tmp_path / "lookup.cu", tmp_path / "lookup"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC), "-o", str(exe),
                    str(src)], check=True, capture_output=True, text=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout
    missing, lookups = map(int, out.split())
    assert missing == 0 and lookups == 1
