"""The residual stream's passes with four lanes a thread, at the edges of what they take (128 to 4,096 lanes, multiples of four, aligned),
and heads prepared by several CTAs a token, each beside its plain statement."""

import pytest
import torch

import plain_ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, dtype=torch.float32, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return torch.randn(*shape, generator=g).to(dtype).to(DEV)


@pytest.mark.parametrize("W", [124, 128, 132, 1020, 2048, 4096, 4100])
@pytest.mark.parametrize("S", [1, 3, 4, 5, 8])
@pytest.mark.parametrize("results", [0, 1, 4])
def test_hyper_mix_norm(W, S, results):
    from llmserve_triton_kernels_b200 import ops

    n = 3
    start, weight, read_in = rnd(S, n, W, seed=1), rnd(W, seed=2), rnd(S, seed=3)
    update = None
    if results:
        update = ops.StreamUpdate(ops.WeightedSum([rnd(n, W, seed=4 + b) for b in range(results)], [0.5 + b for b in range(results)]), rnd(S, S, seed=9), rnd(S, seed=10))
    for rows in (None, torch.tensor([2, 0], dtype=torch.int32, device=DEV)):
        for dtype, tol in ((torch.float32, 2e-5), (torch.bfloat16, 2.0**-8)):
            a, b = start.clone(), start.clone()
            got = ops.hyper_mix_norm(a, update, read_in, weight, 1e-5, rows=rows, out_dtype=dtype)
            want = plain_ops.hyper_mix_norm(b, update, read_in, weight, 1e-5, rows=rows, out_dtype=dtype)
            torch.testing.assert_close(got.float(), want.float(), rtol=tol, atol=tol)
            torch.testing.assert_close(a, b, rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("C", [124, 128, 132, 2048, 4096, 4100])
@pytest.mark.parametrize("count", [1, 2, 3, 4])
@pytest.mark.parametrize("shift", [0, 1])
def test_branch_sum_rmsnorm(C, count, shift):
    from llmserve_triton_kernels_b200 import ops

    n = 5
    branches = [rnd(n * C + shift, seed=b)[shift:].view(n, C) for b in range(count)]  # shift: rows that do not start on 16 bytes
    pending = ops.BranchSum(branches, [rnd(C, seed=10 + b) for b in range(count)], 1e-5, 0.5)
    for dtype, tol in ((torch.float32, 2e-5), (torch.bfloat16, 2.0**-8)):
        a, b = rnd(n, C, seed=20), rnd(n, C, seed=20)
        got, want = (f(pending, r, rnd(C, seed=21), 1e-5, dtype) for f, r in ((ops.branch_sum_rmsnorm, a), (plain_ops.branch_sum_rmsnorm, b)))
        torch.testing.assert_close(got.float(), want.float(), rtol=tol, atol=tol)
        torch.testing.assert_close(a, b, rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("n", [1, 37, 148, 149])
def test_heads_prepared_by_several_ctas(n):
    from llmserve_triton_kernels_b200 import ops

    H, G, D, V = 32, 8, 64, 64
    proj, positions = rnd(n, (H + G) * D + G * V, seed=1), torch.arange(n, dtype=torch.int32, device=DEV)
    slots, freq = torch.randperm(160, generator=torch.Generator().manual_seed(1))[:n].int().to(DEV), torch.rand(D // 2, device=DEV)
    common = dict(heads=H, kv_heads=G, dim=D, value_dim=V, freq=freq, eps=1e-5, slot_map=slots, out_dtype=torch.bfloat16)
    for name, sizes in (("head_prepare", (D, D)), ("qk_prepare", (H * D, G * D))):
        pools = [torch.zeros(10, 2, G, 16, D, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
        more = dict(q_weight=rnd(sizes[0], seed=2), k_weight=rnd(sizes[1], seed=3))
        a, b = (getattr(m, name)(proj, positions, pool=p, **common, **more) for m, p in ((ops, pools[0]), (plain_ops, pools[1])))
        a, b = (x[0] if isinstance(x, (tuple, list)) else x for x in (a, b))
        torch.testing.assert_close(a.float(), b.float(), rtol=2.0**-7, atol=1e-3)
        torch.testing.assert_close(pools[0].float(), pools[1].float(), rtol=2.0**-7, atol=1e-3)
