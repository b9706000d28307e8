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
