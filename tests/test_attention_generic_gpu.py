"""The general attention kernel: a row's bits are the same whether its item has eight warps (few items) or one (many), over the forms whose
keys start and end in the middle of chunks."""

import pytest
import torch

import test_attention_rows_few_gpu as rows
from test_attention_rows_few_gpu import DEV, ops, rnd  # noqa: F401

pytestmark = pytest.mark.gpu

FORMS = {
    "plain": dict(d0=64, dv=64),
    "odd": dict(d0=7, d1=6, dv=33),
    "window": dict(d0=16, dv=130, window=70, slopes=True),
    "kept": dict(d0=64, dv=64, window=40, keep_first=37, sinks=True),
    "blocks": dict(d0=64, dv=64, chunk=96, softcap=5.0),
    "two maps": dict(d0=32, dv=64, maps=2),
    "wide": dict(d0=64, dv=300),
}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("form", FORMS)
def test_bits_do_not_depend_on_the_number_of_items(ops, form, dtype, monkeypatch):  # noqa: F811
    monkeypatch.setattr(ops, "_FORCE_GENERIC_ATTENTION", True)
    f = FORMS[form]
    d0, d1, dv, maps, H, KV, page, n, context = f["d0"], f.get("d1", 0), f["dv"], f.get("maps", 1), 32, 8, 4, 65, 601
    dk, pages = maps * d0 + d1, 160
    keys, values = rnd(pages, KV, page, dk, seed=1, dtype=dtype), rnd(pages, KV, page, dv, seed=2, dtype=dtype)
    q0, q1 = rnd(n, H, maps * d0, seed=3, dtype=dtype), rnd(n, H, d1, seed=4, dtype=dtype) if d1 else None
    kw = dict(num_heads=H, num_kv_heads=KV, scale=dk**-0.5, window=f.get("window"), keep_first=f.get("keep_first"), chunk=f.get("chunk"), softcap=f.get("softcap"))
    if f.get("slopes"):
        kw["slopes"] = rnd(H, dtype=torch.float32, seed=5).abs() * 0.1
    if f.get("sinks"):
        kw["sinks"] = rnd(H, dtype=torch.float32, seed=6)
    if maps == 2:
        kw["differential"] = ops.DifferentialMaps(0.4, 1e-6, 0.5)

    def run(first, count):  # the tokens [first, first + count) as a step of their own
        table, ctx = rows.step((n,), (context,), page, pages, False)
        ctx.context_lens = torch.tensor([context - n + first + count], dtype=torch.int32, device=DEV)
        ctx.num_tokens = ctx.max_query_len = count
        ctx.cu_tokens, ctx.token_request = torch.tensor([0, count], dtype=torch.int32, device=DEV), torch.zeros(count, dtype=torch.int32, device=DEV)
        part = lambda x: None if x is None else x[first : first + count].contiguous()  # noqa: E731
        return ops.attention_rows(part(q0), part(q1), keys.data_ptr(), (KV * page * dk, page * dk, dk), values.data_ptr(), (KV * page * dv, page * dv, dv), dv,
                                  table, page, ctx, **kw)

    whole = run(0, n)  # 2,080 items
    for first, count in ((0, 1), (33, 1), (n - 2, 2), (0, 64)):
        assert torch.equal(run(first, count), whole[first : first + count])


@pytest.mark.parametrize("n", [1, 300])  # eight warps an item, one
@pytest.mark.parametrize("bad", ["query", "first key", "a chunk", "the newest key"])
def test_nan_comes_out_where_it_is_seen(ops, bad, n):  # noqa: F811
    """NaN in the only keys of a class of chunks does not leave with the class."""
    H, page, d, context = 8, 4, 16, 301
    pages = 80
    q, keys, values = rnd(n, H, d, seed=1, dtype=torch.float32), rnd(pages, 1, page, d, seed=2, dtype=torch.float32), rnd(pages, 1, page, d, seed=3, dtype=torch.float32)
    table, ctx = rows.step((n,), (context,), page, pages, False)
    run = lambda: ops.attention_rows(q, None, keys.data_ptr(), (page * d, page * d, d), values.data_ptr(), (page * d, page * d, d), d, table, page, ctx,  # noqa: E731
                                     num_heads=H, num_kv_heads=1, scale=0.25)
    clean = run()
    seen = torch.zeros(n, H, dtype=torch.bool, device=DEV)
    if bad == "query":
        q[-1, 2] = torch.nan
        seen[-1, 2] = True
    else:
        first, last = {"first key": (0, 1), "a chunk": (64, 96), "the newest key": (context - 1, context)}[bad]
        for j in range(first, last):
            keys[int(table[0, j // page]), 0, j % page] = torch.nan
        seen[torch.arange(context - n, context, device=DEV) >= first] = True
    got = run()
    assert bool(got[seen].isnan().all()) and torch.equal(got[~seen], clean[~seen])


def test_keys_that_score_minus_infinity_weigh_nothing(ops):  # noqa: F811
    """A whole chunk of them, in the first class and in others, and more of the class behind it: as in 64 bits."""
    H, page, d, context = 4, 4, 16, 600
    pages = 160
    q, keys, values = rnd(1, H, d, seed=1, dtype=torch.float32), rnd(pages, 1, page, d, seed=2, dtype=torch.float32), rnd(pages, 1, page, d, seed=3, dtype=torch.float32)
    q[..., 0] = 1.0
    table, ctx = rows.step((1,), (context,), page, pages, False)
    for first in (0, 64, 320):
        for j in range(first, first + 32):
            keys[int(table[0, j // page]), 0, j % page, 0] = -torch.inf
    got = ops.attention_rows(q, None, keys.data_ptr(), (page * d, page * d, d), values.data_ptr(), (page * d, page * d, d), d, table, page, ctx,
                             num_heads=H, num_kv_heads=1, scale=0.25)
    order = table[0].long()
    k, v = keys[order, 0].reshape(-1, d)[:context].double(), values[order, 0].reshape(-1, d)[:context].double()
    want = torch.softmax(q[0].double() @ k.T * 0.25, -1) @ v
    torch.testing.assert_close(got[0].double(), want, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("n", [1, 70])  # 32 heads: eight warps an item, one
@pytest.mark.parametrize("context", [70, 96, 255, 256, 257, 288, 700])
@pytest.mark.parametrize("window", [None, 33, 256])
def test_beside_the_same_in_64_bits(ops, context, window, n):  # noqa: F811
    H, KV, page, d, dv = 32, 8, 8, 24, 40
    pages = -(-context // page) + 2
    q, keys, values = rnd(n, H, d, seed=1, dtype=torch.float32), rnd(pages, KV, page, d, seed=2, dtype=torch.float32), rnd(pages, KV, page, dv, seed=3, dtype=torch.float32)
    table, ctx = rows.step((n,), (context,), page, pages, False)
    got = ops.attention_rows(q, None, keys.data_ptr(), (KV * page * d, page * d, d), values.data_ptr(), (KV * page * dv, page * dv, dv), dv, table, page, ctx,
                             num_heads=H, num_kv_heads=KV, scale=0.3, window=window)
    pick = lambda x: x[table[0].long()].transpose(1, 2).reshape(-1, KV, x.shape[-1])[:context].double().repeat_interleave(H // KV, 1)  # noqa: E731
    scores = torch.einsum("nhd,jhd->hnj", q.double(), pick(keys)) * 0.3
    pos, j = torch.arange(context - n, context, device=DEV)[:, None], torch.arange(context, device=DEV)[None]
    scores = scores.masked_fill(~((j <= pos) & (j > pos - (window or context + 1))), -torch.inf)
    want = torch.einsum("hnj,jhd->nhd", scores.softmax(-1), pick(values))
    # 32-bit sums of up to 700 weights near 1e-2 and of 24 products a score: some ten roundings of 6e-8 behind one another
    assert float((got.double() - want).norm()) <= 2e-6 * float(want.norm())
