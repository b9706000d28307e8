"""Attention of prompt portions on tcgen05 with everything that designs put around the softmax, and over a step's own tokens, beside the
plain statement: edges of the 128-token and 64-key tiles, windows, kept keys and blocks that leave tiles out, small requests that go along,
rows behind a request's end that hold NaN."""

import pytest
import torch

import plain_ops
from test_kafepel_kernels_gpu import DEV, _ops, close, paged_batch

pytestmark = pytest.mark.gpu

OPTIONS = {
    "sinks": dict(sinks=True), "sinks far above and below": dict(sinks="far"), "gate": dict(gate=True), "sinks, gate, window": dict(sinks=True, gate=True, window=70),
    "bias and window": dict(slopes=True, window=100), "cap": dict(softcap=5.0), "kept, window, cap, bias": dict(window=33, keep_first=16, softcap=20.0, slopes=True),
    "many kept": dict(window=130, keep_first=200), "kept over a tile's edge": dict(window=40, keep_first=65), "blocks": dict(chunk=100),
    "blocks and window": dict(chunk=64, window=33), "one gate a head": dict(gate="head", sinks=True),
}


@pytest.mark.parametrize("what", OPTIONS)
@pytest.mark.parametrize("H,KV,D,V,page_size", [(4, 2, 64, 64, 16), (3, 1, 64, 128, 8), (2, 2, 128, 128, 64)])
def test_options_against_plain(H, KV, D, V, page_size, what, monkeypatch):
    ops = _ops()
    torch.manual_seed(H * 100 + D)
    more = dict(OPTIONS[what])
    ctx, table, _, pages = paged_batch([700, 129, 300, 65, 40, 9], [300, 129, 128, 32, 31, 1], page_size)
    N, bf = ctx.num_tokens, torch.bfloat16
    pool = (torch.randn(pages, 2, KV, page_size, max(D, V), device=DEV) * 0.7).to(bf)
    for r, n in enumerate([700, 129, 300, 65]):  # what an earlier request left behind this one's last token
        if n % page_size:
            pool[int(table[r, n // page_size]), :, :, n % page_size :] = torch.nan
    q = torch.randn(N, H * D + 8, device=DEV).to(bf)[:, : H * D]
    if more.get("sinks"):
        more["sinks"] = torch.randn(H, device=DEV) * 2.0 if more["sinks"] is True else torch.tensor([200.0, -200.0, float("-inf"), 3.0], device=DEV)[:H].contiguous()
    if more.get("gate"):
        more["gate_per_head"] = more["gate"] == "head"
        more["gate"] = torch.randn(N, 4 + H * V + 8, device=DEV)[:, 4 : 4 + H * V]
    if more.get("slopes"):
        more["slopes"] = torch.rand(H, device=DEV) * 0.2
    common = dict(num_heads=H, num_kv_heads=KV, key_dim=D, value_dim=V, scale=0.3)
    want = plain_ops.paged_softmax_attention(q, pool, table, ctx, **common, **more)
    taken, kernel = [], ops._tcgen05_softmax_attention
    monkeypatch.setattr(ops, "_tcgen05_softmax_attention", lambda *a, **k: taken.append(kernel(*a, **k)) or taken[-1])
    got = ops.paged_softmax_attention(q, pool, table, ctx, **common, **more)
    assert taken == [(32, True)]  # requests of 32 tokens and more here, the others there
    close(got, want, 2e-2, what)
    if "slopes" in more and not more.get("softcap"):
        got = ops.biased_paged_attention(q, pool, table, ctx, **common, slopes=more["slopes"], window=more["window"])
        close(got, want, 2e-2, what + " (a projection's rows)")


@pytest.mark.parametrize("more", [dict(window=1), dict(window=4), dict(window=7, keep_first=3), dict(window=3, keep_first=70), dict(chunk=50, window=5),
                                  dict(chunk=50), dict(chunk=50, window=5, keep_first=20), dict(sinks=True, window=4)], ids=str)
@pytest.mark.parametrize("D,V,page_size", [(64, 64, 8), (64, 128, 16), (128, 128, 32), (64, 64, 64)])
def test_a_tail_whose_window_lies_in_the_last_page(D, V, page_size, more, monkeypatch):
    """Tail tiles of 1 to 8 rows that need the request's last, partly filled page alone: what stands behind its end is nobody's, wherever in
    a tile of keys the pages that are not needed would have been."""
    ops = _ops()
    torch.manual_seed(D + page_size)
    news = [129, 130, 132, 136, 33]
    ctx, table, _, pages = paged_batch([n + old for n, old in zip(news, (21, 0, 300, 1, 40))], news, page_size)
    pool = torch.randn(pages, 2, 2, page_size, max(D, V), device=DEV).bfloat16()
    for r, n in enumerate(ctx.context_lens.tolist()):
        if n % page_size:
            pool[int(table[r, n // page_size]), :, :, n % page_size :] = torch.nan
    q = torch.randn(ctx.num_tokens, 2 * D, device=DEV).bfloat16()
    more = dict(more, sinks=torch.randn(2, device=DEV)) if more.get("sinks") else more
    common = dict(num_heads=2, num_kv_heads=2, key_dim=D, value_dim=V, scale=0.3)
    got = ops.paged_softmax_attention(q, pool, table, ctx, **common, **more)
    if "chunk" in more and "keep_first" in more:  # kept keys stay visible from every block: the kernels' reading, which the plain statement does not share
        monkeypatch.setattr(ops, "_TC_ATTENTION_ENABLED", False)
        want = ops.paged_softmax_attention(q, pool, table, ctx, **common, **more)
    else:
        want = plain_ops.paged_softmax_attention(q, pool, table, ctx, **common, **more)
    close(got, want, 2e-2, str(more))


def test_every_key_scores_minus_infinity():
    """A row without a finite score is zeros; one NaN score leaves its row NaN; the rows beside them are as without them."""
    ops = _ops()
    ctx, table, _, pages = paged_batch([200], [200], 16)
    pool = torch.randn(pages, 2, 1, 16, 64, device=DEV).bfloat16()
    pool[:, 0, :, :, 0] = 1.0
    q = torch.randn(200, 64, device=DEV).bfloat16()
    common = dict(num_heads=1, num_kv_heads=1, key_dim=64, value_dim=64, scale=0.3)
    same = ops.paged_softmax_attention(q, pool, table, ctx, **common)
    q[3, 0], q[150, 0], q[160, 5] = -torch.inf, -torch.inf, torch.nan
    got = ops.paged_softmax_attention(q, pool, table, ctx, **common)
    assert bool((got[3] == 0).all()) and bool((got[150] == 0).all()) and bool(got[160].isnan().all())
    rest = torch.ones(200, dtype=torch.bool)
    rest[[3, 150, 160]] = False
    assert same.isfinite().all() and torch.equal(got[rest], same[rest])


@pytest.mark.parametrize("window", [None, 1, 64, 100])
@pytest.mark.parametrize("news", [[300, 129, 40, 5], [128], [1025, 33]])
def test_a_steps_own_tokens(news, window):
    ops = _ops()
    H, rank, bf = 3, 72, torch.bfloat16
    ctx, table, _, _ = paged_batch([n + 17 * i for i, n in enumerate(news)], news, 16)
    N = sum(news)
    torch.manual_seed(N)
    proj = torch.randn(N, H * 96 + 8, device=DEV).to(bf)
    q = proj.as_strided((N, H, 64), (proj.stride(0), 96, 1))
    q_rot, kv, fresh = torch.randn(N, H, 32, device=DEV).to(bf), torch.randn(N, H * 128, device=DEV).to(bf), torch.randn(N, rank + 32, device=DEV).to(bf)
    args = dict(dim=64, value_dim=64, rank=rank, scale=0.2, window=window)
    out, stats = ops.fresh_latent_attention(q, q_rot, kv, fresh, table, ctx, **args)
    alone = ops.fresh_latent_attention(q, q_rot, kv, fresh, table, ctx, **args, want_stats=False)
    assert torch.equal(out, alone)
    cu = ctx.cu_tokens.tolist()
    for a, b in zip(cu, cu[1:]):
        qs = torch.cat((q[a:b], q_rot[a:b]), -1).double()
        ks = torch.cat((kv[a:b, : H * 64].view(-1, H, 64), fresh[a:b, None, rank:].expand(-1, H, -1)), -1).double()
        s = torch.einsum("ihd,jhd->hij", qs, ks) * 0.2
        i, j = torch.arange(b - a, device=DEV)[:, None], torch.arange(b - a, device=DEV)[None]
        s = s.masked_fill((j > i) | ((i - j >= window) if window else torch.zeros_like(i - j, dtype=torch.bool)), -torch.inf)
        want = torch.einsum("hij,jhd->ihd", s.softmax(-1), kv[a:b, H * 64 :].view(-1, H, 64).double())
        close(out[a:b], want, 1e-2, f"tokens {a} to {b}")
        log_sum = stats[a:b, :, 0].double() * 0.6931471805599453 + stats[a:b, :, 1].double().log()
        torch.testing.assert_close(log_sum, s.logsumexp(-1).T, rtol=1e-5, atol=1e-4)
    # the next request's rows are nobody else's
    if len(news) > 1:
        kv[cu[1] : cu[2]] = torch.nan
        fresh[cu[1] : cu[2]] = torch.nan
        assert torch.equal(ops.fresh_latent_attention(q, q_rot, kv, fresh, table, ctx, **args, want_stats=False)[: cu[1]], out[: cu[1]])


@pytest.mark.parametrize("scale", [0.0, -0.3])
def test_scales_that_are_not_positive_go_the_old_way(scale):
    ops = _ops()
    torch.manual_seed(7)
    ctx, table, _, pages = paged_batch([300, 40], [200, 40], 16)
    pool, q = torch.randn(pages, 2, 2, 16, 64, device=DEV).bfloat16(), torch.randn(240, 128, device=DEV).bfloat16()
    for more in (dict(sinks=torch.randn(2, device=DEV)), dict(softcap=5.0), dict(slopes=torch.rand(2, device=DEV) * 0.2), dict(chunk=64)):
        common = dict(num_heads=2, num_kv_heads=2, key_dim=64, value_dim=64, scale=scale, **more)
        close(ops.paged_softmax_attention(q, pool, table, ctx, **common), plain_ops.paged_softmax_attention(q, pool, table, ctx, **common), 2e-2, str(more))
    kv, q_rot, fresh = torch.randn(240, 256, device=DEV).bfloat16(), torch.randn(240, 2, 32, device=DEV).bfloat16(), torch.randn(240, 72 + 32, device=DEV).bfloat16()
    got = ops.fresh_latent_attention(q.view(240, 2, 64), q_rot, kv, fresh, table, ctx, dim=64, value_dim=64, rank=72, scale=scale, window=None, want_stats=False)
    for a, b in ((0, 200), (200, 240)):
        k = torch.cat((kv[a:b, :128].view(-1, 2, 64), fresh[a:b, None, 72:].expand(-1, 2, -1)), -1).float()
        s = torch.einsum("ihd,jhd->hij", torch.cat((q[a:b].view(-1, 2, 64), q_rot[a:b]), -1).float(), k) * scale
        s = s.masked_fill(torch.ones_like(s[0], dtype=torch.bool).triu(1), -torch.inf)
        close(got[a:b], torch.einsum("hij,jhd->ihd", s.softmax(-1), kv[a:b, 128:].view(-1, 2, 64).float()), 1e-2, f"tokens {a} to {b}")


@pytest.mark.parametrize("H,KV,D,general,plain", [(4, 2, 64, 32, 32), (16, 4, 64, 48, 64), (16, 4, 128, 32, 32)])
def test_a_crowd_of_small_requests_beside_a_long_one(H, KV, D, general, plain, monkeypatch):
    """Forty requests on both sides of every threshold: which of them go along, and everybody's rows."""
    ops = _ops()
    torch.manual_seed(H + D)
    news = [200, *(31 + i % 40 for i in range(39))]
    ctx, table, _, pages = paged_batch([n + 13 * (i % 7) for i, n in enumerate(news)], news, 16)
    pool = torch.randn(pages, 2, KV, 16, D, device=DEV).bfloat16()
    qkv = torch.randn(ctx.num_tokens, (H + 2 * KV) * D, device=DEV).bfloat16()
    q = qkv[:, : H * D]
    common = dict(num_heads=H, num_kv_heads=KV, key_dim=D, value_dim=D, scale=0.2)
    taken, kernel = [], ops._tcgen05_softmax_attention
    monkeypatch.setattr(ops, "_tcgen05_softmax_attention", lambda *a, **k: taken.append(kernel(*a, **k)) or taken[-1])
    for more in ({}, dict(sinks=torch.randn(H, device=DEV)), dict(slopes=torch.rand(H, device=DEV) * 0.1)):
        close(ops.paged_softmax_attention(q, pool, table, ctx, **common, **more), plain_ops.paged_softmax_attention(q, pool, table, ctx, **common, **more), 2e-2, str(more))
    assert taken == [(general, True)] * 3
    assert ops._tc_join_tokens(ctx, H, D, D, ops._TC_ATTENTION_JOIN_CROWDED) == plain
    got = ops.paged_attention(qkv, pool, table, ctx, num_heads=H, num_kv_heads=KV, head_dim=D, scale=0.2)
    close(got, plain_ops.paged_softmax_attention(q, pool, table, ctx, **common), 2e-2, "the plain form")
