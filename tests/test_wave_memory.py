"""The memory of the wavefront's path state (csrc/grow_buffer.h): where the merged size does not fit, the single size is
taken, and the merged one is not asked for again. The allocator is a stand-in with a limit; nothing needs a GPU."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "caelix-renderer_b200", "csrc")

RUNTIME = r"""
#pragma once
#include <cstddef>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
cudaError_t cudaMalloc(void** p, size_t n);
cudaError_t cudaFree(void* p);
cudaError_t cudaGetLastError();
"""

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include <cuda_runtime.h>
#include "grow_buffer.h"

static std::map<void*, size_t> live;
static size_t used = 0, limit = 0;
static int mallocs = 0, frees = 0, failed = 0, errors = 0;
cudaError_t cudaMalloc(void** p, size_t n)
{
    ++mallocs;
    *p = nullptr;
    if (used + n > limit) return ++failed, cudaErrorMemoryAllocation;
    *p = malloc(1);
    live[*p] = n;
    used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    ++frees;
    used -= live.at(p);
    live.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
namespace cx
{
CaelixResult cuda_result(cudaError_t e, const char*)
{
    ++errors;
    return e == cudaErrorMemoryAllocation ? CAELIX_ERROR_OUT_OF_MEMORY : CAELIX_ERROR_CUDA;
}
}

#define CHECK(c) if (!(c)) { printf("line %d: %s (mallocs %d frees %d failed %d errors %d)\n", __LINE__, #c, mallocs, frees, failed, errors); return 1; }

int main()
{
    // Frames of 100 (one sample index per wave) or 800 bytes (eight) where 500 fit.
    cx::WaveMemory m;
    limit = 500;
    bool fits = true;
    const auto frame = [&](uint64_t merged, uint64_t single) { return m.reserve(merged, [&] { return single; }, "test", &fits); };
    CHECK(frame(100, 100) == CAELIX_OK && fits && mallocs == 1);
    void* held = m.buffer.ptr;
    for (int k = 0; k < 10; ++k) {
        CHECK(frame(800, 100) == CAELIX_OK && !fits);
        CHECK(m.buffer.ptr == held);
    }
    CHECK(mallocs == 2 && failed == 1 && frees == 0 && errors == 0);  // asked once, the working buffer kept
    // A larger frame is not asked for either; a smaller merged size is, and is kept.
    CHECK(frame(900, 200) == CAELIX_OK && !fits && failed == 1 && m.buffer.bytes == 200);
    CHECK(frame(300, 150) == CAELIX_OK && fits && m.buffer.bytes == 300 && used == 300);
    const int before = mallocs;
    for (int k = 0; k < 10; ++k) CHECK(frame(300, 150) == CAELIX_OK && fits);
    for (int k = 0; k < 10; ++k) CHECK(frame(800, 100) == CAELIX_OK && !fits);
    CHECK(mallocs == before && errors == 0);
    // A change of the setting asks again; with room it fits.
    m.forget();
    limit = 2000;
    CHECK(frame(800, 100) == CAELIX_OK && fits && used == 800);
    // A buffer too small for either size goes first; a size that does not fit at all is an error, once logged.
    m.buffer.release();
    limit = 1000;
    CHECK(frame(600, 600) == CAELIX_OK && fits);
    CHECK(frame(900, 700) == CAELIX_OK && fits && used == 900);
    CHECK(frame(1200, 1100) == CAELIX_ERROR_OUT_OF_MEMORY && !fits && errors == 1);
    CHECK(frame(800, 700) == CAELIX_OK && fits);
    m.buffer.release();
    CHECK(used == 0 && live.empty());
    return 0;
}
"""


def test_merged_size_is_asked_for_once(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Wextra", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "main.cpp"),
                    os.path.join(CSRC, "grow_buffer.cpp"), "-o", str(tmp_path / "main")], check=True)
    out = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
