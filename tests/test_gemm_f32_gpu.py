"""The 32-bit product's kernels for few rows and for aligned rows, at the edges of their tiles: a row has the same bits whichever
kernel and tile ran, and is a 32-bit sum of the double product."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("k", [4, 20, 256, 260, 2052])
@pytest.mark.parametrize("n", [1, 15, 17, 129, 2100])
def test_rows_have_the_same_bits_in_every_kernel(n, k):
    from llmserve_triton_kernels_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(n * 7 + k)
    x = torch.randn(300, k, generator=g, device=DEV)
    w = torch.randn(n, k, generator=g, device=DEV)
    # the same operands in rows that do not start on 16 bytes: the kernel that takes every layout
    loose = torch.empty(300, k + 1, device=DEV)
    loose[:, :k] = x
    want = ops.linear(loose[:, :k], w)
    # sums of k / 16 parts of 16 unit-variance products each: about 8 standard deviations of their rounding
    torch.testing.assert_close(want, (x.double() @ w.double().t()).float(), atol=4e-6 * k**0.5, rtol=1e-5)
    for m in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 63, 64, 65, 128, 129, 300):
        assert torch.equal(ops.linear(x[:m], w), want[:m]), f"{m} rows"
    # rows with a pitch
    pitched = torch.zeros(40, k + 8, device=DEV)
    pitched[:, :k] = x[:40]
    assert torch.equal(ops.linear(pitched[:7, :k], w), want[:7]) and torch.equal(ops.linear(pitched[:, :k], w), want[:40])


SECOND_CONTEXT = """
import ctypes, sys

lib, cu = ctypes.CDLL(sys.argv[1]), ctypes.CDLL("libcuda.so.1")
ok = lambda code: code and sys.exit(f"driver error {code}")
ok(cu.cuInit(0))
for turn in range(2):  # a context stands for a device: the library's kernels are set up in each
    context, pointers = ctypes.c_void_p(), []
    ok(cu.cuCtxCreate_v2(ctypes.byref(context), 0, 0))
    M, N, K = 300, 96, 256
    for elements in (M * K, N * K, M * N):
        p = ctypes.c_uint64()
        ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(4 * elements)))
        ok(cu.cuMemsetD32_v2(p, 0x3f800000, ctypes.c_size_t(elements)))  # ones
        pointers.append(p)
    x, w, out = (ctypes.c_void_p(p.value) for p in pointers)
    for m in (1, 2, 4, 8, 16, 33, M):
        code = lib.llm_gemm_simt(x, 0, w, 0, out, 0, m, N, K, K, K, N, None)
        if code:
            sys.exit(f"context {turn}, {m} rows: the launch was refused with {code}")
        ok(cu.cuCtxSynchronize())
        row = (ctypes.c_float * N)()
        ok(cu.cuMemcpyDtoH_v2(row, ctypes.c_uint64(out.value + 4 * (m - 1) * N), ctypes.c_size_t(4 * N)))
        assert list(row) == [float(K)] * N, (turn, m)
print("same in both")
"""


def test_a_second_device_of_the_process():
    """What a kernel needs before its launch is set up wherever it runs, not once a process: a second CUDA context has, as a second GPU has,
    none of what was set in the first."""
    import subprocess
    import sys

    from llmserve_triton_kernels_b200 import ops

    ops.linear(torch.ones(1, 4, device=DEV), torch.ones(1, 4, device=DEV))
    assert ops._F32 == 0
    done = subprocess.run([sys.executable, "-c", SECOND_CONTEXT, str(ops.loaded_library_path())], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0 and "same in both" in done.stdout, done.stdout + done.stderr


@pytest.mark.parametrize("m", [1, 2, 4, 7, 16, 40])
def test_operands_that_the_kernel_in_front_writes(m):
    """Both operands are the work of a kernel that lets the product start before it has ended, and the buffers hold others until then."""
    from llmserve_triton_kernels_b200 import ops

    n, k, turns = 4000, 1028, 20
    g = torch.Generator(device=DEV).manual_seed(m)
    rows = torch.randn(turns, n + 16, k, generator=g, device=DEV)
    ones = torch.ones(k, device=DEV)
    left = torch.randn(m, k, generator=g, device=DEV)
    ops.linear(left, ops.rmsnorm(rows[0].clone(), ones, 1e-5)[:n])  # what a capture may not do has been done
    wants = []
    for t in range(turns):
        normed = ops.rmsnorm(rows[t].clone(), ones, 1e-5)
        torch.cuda.synchronize()
        wants.append((ops.linear(left, normed[:n]), ops.linear(normed[:m].clone(), normed[:n])))
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    stream, normed_rows = rows[0].clone(), torch.empty(n + 16, dtype=torch.int32, device=DEV)
    torch.arange(n + 16, out=normed_rows)
    with torch.cuda.graph(graph):
        normed = ops.rmsnorm(stream, ones, 1e-5, rows=normed_rows)
        a = ops.linear(left, normed[:n])
        normed = ops.rmsnorm(stream, ones, 1e-5, rows=normed_rows)
        b = ops.linear(normed[:m], normed[:n])
    for t in range(turns):
        stream.copy_(rows[t])
        graph.replay()
        assert torch.equal(a, wants[t][0]) and torch.equal(b, wants[t][1]), f"turn {t}"
