"""The once-per-kernel launch set-up with two threads, against a CUDA runtime made for the test: the limit that a thread has
been granted stays granted."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include <chrono>
#include <thread>
#include "kernels/api.hpp"

static std::atomic<int> limit{0}, small_inside{0};
extern "C" cudaError_t cudaGetDevice(int* device) { *device = 0; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute attr, int value) {
    if (attr != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
    if (value == 1000) {        // the thread with the smaller launch is held up inside the call
        small_inside = 1;
        std::this_thread::sleep_for(std::chrono::milliseconds(200));
    }
    limit = value;
    return cudaSuccess;
}
int main() {
    const void* kernel = nullptr;       // (any handle: only the stand-ins see it)
    ep::PreparedKernel prepared;
    std::thread small([&] { prepared.prepare(kernel, 1000); });
    while (small_inside == 0) std::this_thread::yield();
    prepared.prepare(kernel, 5000);
    const bool granted = limit >= 5000;
    small.join();
    if (!granted || limit < 5000) return 1;             // what was granted has been taken back
    prepared.prepare(kernel, 2000);
    return limit >= 5000 ? 0 : 2;
}
"""


def test_a_granted_limit_is_not_taken_back(tmp_path):
    cuda = os.environ.get('CUDA_HOME', '/usr/local/cuda')
    if shutil.which('g++') is None or not os.path.exists(f'{cuda}/include/cuda_runtime.h'):
        pytest.skip('no toolkit')
    src, exe = tmp_path / 'prepared.cpp', tmp_path / 'prepared'
    src.write_text(SOURCE)
    subprocess.run(['g++', '-std=c++17', '-pthread', f'-I{ROOT}/deepep_b200/csrc', f'-I{cuda}/include', str(src), '-o', str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
