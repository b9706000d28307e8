"""Kernels of steps in which a request brings one token or few: sigmoid attention over whole contexts in a cluster, the recurrences' walk
without shared memory, beside the plain statement and the kernels for any step; contexts at the edges of a chunk of 32 keys and of the
shares, windows, tokens whose sums have the bits of a longer step."""

import pytest
import torch

import plain_ops
from test_kafepel_kernels_gpu import DEV, _ops, close, paged_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[1], [32, 33, 31, 600], [2041, 5, 512, 513, 100, 64, 65, 1], [700] * 20, [100] * 80])
@pytest.mark.parametrize("H,KV,page_size,window", [(32, 8, 16, None), (16, 4, 16, 40), (4, 4, 8, None), (64, 8, 16, None), (12, 2, 32, 33)])
def test_sigmoid_attention_of_one_token_a_request(lens, H, KV, page_size, window):
    ops = _ops()
    torch.manual_seed(H + len(lens))
    ctx, table, _, pages = paged_batch(lens, [1] * len(lens), page_size)
    pool = (torch.randn(pages, 2, KV, page_size, 64, device=DEV) * 0.7).bfloat16()
    for r, n in enumerate(lens):  # what an earlier request left behind this one's last token
        if n % page_size:
            pool[int(table[r, n // page_size]), :, :, n % page_size :] = torch.nan
    q = torch.randn(len(lens), H * 64 + 8, device=DEV).bfloat16()[:, : H * 64].contiguous()
    bias, mix = torch.randn(H, device=DEV), torch.randn(H, H, device=DEV) / H**0.5
    common = dict(num_heads=H, num_kv_heads=KV, key_dim=64, value_dim=64, scale=0.125, window=window)
    for more in (dict(softcap=30.0, head_bias=bias, head_mix=mix), dict(head_bias=bias), dict(softcap=2.0, head_mix=mix), {}):
        before = ops.launch_count()
        got = ops.sigmoid_attention(q, pool, table, ctx, **common, **more)
        assert ops.launch_count() == before + 1
        close(got, plain_ops.sigmoid_attention(q, pool, table, ctx, **common, **more), 1e-2, f"{sorted(more)}")
        assert torch.equal(got, ops.sigmoid_attention(q, pool, table, ctx, **common, **more))


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("v_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,D,V", [(3, 32, 16), (2, 64, 128), (2, 64, 48), (1, 128, 64)])
def test_a_token_has_the_same_bits_in_steps_of_any_length(H, D, V, v_dtype, gated):
    ops = _ops()
    torch.manual_seed(D + V)
    lens, starts = [40, 17, 1], [0, 40, 57]
    N = sum(lens)
    q, k, z = (torch.randn(N, H * D, device=DEV) * 0.5 for _ in range(3))
    v = torch.randn(N, H * V, device=DEV).to(v_dtype)
    states = torch.randn(5, H, D, V, device=DEV)
    slots = torch.tensor([4, 0, 2], dtype=torch.int32, device=DEV)
    bias, decay = torch.randn(H * D, device=DEV), torch.rand(H, device=DEV) * 0.2 + 0.8

    def scan(rows, news, s):
        cu = torch.tensor([0, news[0], news[0] + news[1], sum(news)], dtype=torch.int32, device=DEV)
        kw = dict(num_requests=3, heads=H, dim=D, value_dim=V, max_query_len=max(news))
        a, b, c, d = (t[torch.tensor(rows, device=DEV)] for t in (q, k, v, z))
        return ops.gated_scan(a, b, c, d, bias, 0.125, 0.7, s, slots, cu, **kw) if gated else ops.retention_scan(a, b, c, decay, s, slots, cu, **kw)

    whole = states.clone()
    want = scan(list(range(N)), lens, whole)  # 40 tokens: the kernel for prompts, one walk a request
    for cut in (1, 3, 16):
        mine, got, at = states.clone(), torch.empty_like(want), [0, 0, 0]
        while any(a < n for a, n in zip(at, lens)):
            news = [min(cut, n - a) for a, n in zip(at, lens)]
            rows = [starts[r] + at[r] + i for r in range(3) for i in range(news[r])]
            got[torch.tensor(rows, device=DEV)] = scan(rows, news, mine)
            at = [a + n for a, n in zip(at, news)]
        assert torch.equal(got, want) and torch.equal(mine, whole), f"portions of {cut}"
