"""The router of few tokens (its matrix in registers and shared memory, the choice in registers up to 32 experts) gives the bits of the one
for many: rows that a warp has beside its own, widths at the edges of its steps, matrices too large for it."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("K", [4, 1020, 1024, 1028, 2048, 4096])
@pytest.mark.parametrize("experts, top, groups", [(1, 1, None), (5, 2, None), (32, 4, (4, 2)), (32, 32, None), (33, 3, None), (64, 5, (8, 3)), (30, 6, (30, 8)), (200, 7, None)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_few_tokens_have_the_bits_of_many(K, experts, top, groups, dtype):
    from llmserve_triton_kernels_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(K + experts)
    x = torch.randn(70, K + 8, generator=g, device=DEV).to(dtype)[:, :K]
    x[3] = 0.0  # all logits equal but for the bias: the lowest indices
    bias, correction = torch.randn(experts, generator=g, device=DEV), torch.randn(experts, generator=g, device=DEV)
    for scores in ("softmax", "sigmoid"):
        for gate in (False, True):
            w = torch.randn(experts + int(gate), K, generator=g, device=DEV) * K**-0.5
            for b, c in ((None, None), (bias, None), (None, correction)):
                args = (w, c, experts, top, 2.5, scores == "sigmoid", gate)
                more = dict(bias=b, shared_one=not gate, scores=scores, groups=groups)
                many = ops.route(x, *args, **more)
                for first, n in ((0, 1), (3, 1), (5, 8), (20, 32)):
                    assert torch.equal(ops.route(x[first : first + n], *args, **more), many[first : first + n])
