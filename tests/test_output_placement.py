"""Which caller buffers a slice loop may run in (loop_runs_in, msl_internal.h): compiled
with the host compiler, on pointer attributes as the CUDA runtime gives them."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <stdio.h>
#include <string.h>
#include "msl_internal.h"
static int in(cudaMemoryType t, int dev, size_t a, size_t n, size_t r, size_t m) {
    cudaPointerAttributes at;
    memset(&at, 0, sizeof(at));
    at.type = t;
    at.device = dev;
    return msl::loop_runs_in(at, 1, (void *)a, n, (void *)r, m);
}
int main() {
    const size_t A = 1 << 20, N = 4096, F = 1 << 24;
    printf("%d %d %d %d %d ", in(cudaMemoryTypeDevice, 1, A, N, F, N), in(cudaMemoryTypeDevice, 0, A, N, F, N),
           in(cudaMemoryTypeManaged, 1, A, N, F, N), in(cudaMemoryTypeHost, 1, A, N, F, N),
           in(cudaMemoryTypeUnregistered, -2, A, N, F, N));
    printf("%d %d ", in(cudaMemoryTypeDevice, 1, A + 8, N, F, N), in(cudaMemoryTypeDevice, 1, A + 16, N, F, N));
    printf("%d %d %d %d %d\n", in(cudaMemoryTypeDevice, 1, A, N, A + N, N), in(cudaMemoryTypeDevice, 1, A, N, A - N, N),
           in(cudaMemoryTypeDevice, 1, A, N, A + N - 8, N), in(cudaMemoryTypeDevice, 1, A, N, A - N + 8, N),
           in(cudaMemoryTypeDevice, 1, A, N, A + 16, 16));
    return 0;
}
"""


def test_only_this_gpus_aligned_memory_apart_from_what_is_read(tmp_path):
    nvcc, cxx = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", shutil.which("g++")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not cxx or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run([cxx, "-std=c++17", "-I", cuda, "-I", os.path.join(ROOT, "multislice_gb300", "csrc"),
                    str(tmp_path / "t.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    # this GPU; another GPU, managed, pinned host, ordinary host; 8 and 16 bytes off
    assert out[:7] == ["1", "0", "0", "0", "0", "0", "1"]
    # what is read right after, right before; overlapping its end, its start, inside
    assert out[7:] == ["1", "1", "0", "0", "0"]
