"""The host's cache of tensor maps (csrc/tma.cuh), with a stand-in for the driver's encoder that writes its arguments down."""

import shutil
import subprocess
from pathlib import Path

import pytest

from llmserve_triton_kernels_b200.ops import build

PROGRAM = r"""
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>
#include <thread>
#include <vector>

static CUresult encode(CUtensorMap* map, CUtensorMapDataType, cuuint32_t, void* base, const cuuint64_t* dims, const cuuint64_t*, const cuuint32_t*,
                       const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    memset(map, 0, sizeof(*map));
    memcpy(map, &base, sizeof(base));
    memcpy((char*)map + 8, &dims[1], 8);
    return CUDA_SUCCESS;
}
static cudaError_t entry(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* r) {
    *fn = (void*)encode;
    *r = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
#define cudaGetDriverEntryPoint entry
#include "tma.cuh"

// the maps of two matrices, as a launcher asks for them: one after the other, and both are used afterwards
static int pair(uint64_t n, char* base) {
    CUtensorMap a, b;
    if (!tma::cached_map_2d_bf16(&a, base, n, 64, 64, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return 1;
    if (!tma::cached_map_2d_bf16(&b, base + 4096, n, 64, 64, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return 1;
    void* p[2];
    uint64_t rows[2];
    memcpy(&p[0], &a, 8); memcpy(&rows[0], (char*)&a + 8, 8);
    memcpy(&p[1], &b, 8); memcpy(&rows[1], (char*)&b + 8, 8);
    return p[0] != base || p[1] != base + 4096 || rows[0] != n || rows[1] != n;
}

int main() {
    char* base = (char*)0x10000;
    int wrong = pair(1, base + 64);  // an odd start: somewhere the first map of a pair is the last one that the cache has room for
    CUtensorMap one;
    wrong += !tma::cached_map_2d_bf16(&one, base, 7, 64, 64, 8, 64, CU_TENSOR_MAP_SWIZZLE_128B);
    for (uint64_t n = 1; n <= 10000; ++n) wrong += pair(n, base);
    std::vector<std::thread> threads;
    std::vector<int> counts(4, 0);
    for (int t = 0; t < 4; ++t)
        threads.emplace_back([t, &counts, base] {
            for (uint64_t n = 1; n <= 6000; ++n) counts[t] += pair(n, base + 65536 * (t + 1));
        });
    for (auto& t : threads) t.join();
    for (int c : counts) wrong += c;
    printf("%d maps are not what was asked for\n", wrong);
    return wrong != 0;
}
"""


def test_a_map_outlives_the_cache_that_it_came_from(tmp_path):
    """More shapes than the cache holds, in pairs and from several threads: every map is still what was asked for, and no freed memory is read."""
    if shutil.which("nvcc") is None and not Path("/usr/local/cuda/bin/nvcc").exists():
        pytest.skip("no nvcc")
    source, program = tmp_path / "maps.cu", tmp_path / "maps"
    source.write_text(PROGRAM)
    made = subprocess.run([build.find_nvcc(), *build.ARCH_FLAGS, "-std=c++17", "-O1", "-g", "-Xcompiler", "-fsanitize=address", "-I", str(build.CSRC), "-o", str(program), str(source)],
                          capture_output=True, text=True)
    assert made.returncode == 0, made.stdout + made.stderr
    ran = subprocess.run([str(program)], capture_output=True, text=True, timeout=120)
    assert ran.returncode == 0, ran.stdout + ran.stderr[-2000:]
