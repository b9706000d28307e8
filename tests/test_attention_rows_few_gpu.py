"""Attention of steps with few rows (the keys cut over warps, the parts merged in the cluster) beside the kernel for many rows and the
32-bit one, over the forms that it takes: run lengths, groups, windows, kept keys, blocks, caps, biases, sinks, gates, two maps, turned
values; and the pieces around it for latent attention."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from llmserve_triton_kernels_b200 import ops

    return ops


def rnd(*shape, dtype=torch.bfloat16, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


def step(query_lens, contexts, page_size, pages, apart):
    g = torch.Generator().manual_seed(sum(contexts))
    cu = [0]
    for n in query_lens:
        cu.append(cu[-1] + n)
    order = torch.randperm(pages, generator=g).tolist()
    table = torch.zeros((len(contexts), max(-(-c // page_size) for c in contexts)), dtype=torch.int32)
    for r, c in enumerate(contexts):
        for p in range(-(-c // page_size)):
            table[r, p] = order.pop()
    owner = [r for r, n in enumerate(query_lens) for _ in range(n)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    return table.to(DEV), SimpleNamespace(
        num_tokens=cu[-1], num_requests=len(contexts), token_request=i32(owner), cu_tokens=i32(cu), context_lens=i32(contexts),
        max_query_len=max(query_lens), max_context_len=max(contexts), host_cu_tokens=cu, steps_apart=apart,
    )


FORMS = {
    "plain": dict(d0=64, dv=64, H=32, KV=8),
    "group of one, a short key": dict(d0=32, dv=64, H=3, KV=3),
    "a short key in two runs": dict(d0=16, d1=16, dv=128, H=6, KV=2),
    "whole group": dict(d0=64, d1=64, dv=128, H=16, KV=1),
    "window": dict(d0=64, dv=64, H=8, KV=2, window=100, slopes=True),
    "kept keys": dict(d0=64, dv=64, H=8, KV=2, window=96, keep_first=20),
    "blocks": dict(d0=64, dv=64, H=8, KV=4, chunk=128, softcap=30.0, slopes=True),
    "sink and gate": dict(d0=64, dv=64, H=8, KV=2, sinks=True, gate=1),
    "gate a head, turned": dict(d0=64, dv=64, H=8, KV=2, gate=2, turn=True),
    "turned neighbours": dict(d0=64, dv=64, H=4, KV=2, turn=True, turn_neighbours=True),
    "two maps": dict(d0=64, dv=128, H=16, KV=4, maps=2, window=200),
    "two short maps": dict(d0=32, dv=64, H=8, KV=2, maps=2, gate=1),
    "latent": dict(d0=256, d1=32, dv=256, H=32, KV=1, alias=True, window=512),
    "short latent": dict(d0=128, d1=32, dv=128, H=16, KV=1, alias=True),
    "longest": dict(d0=288, d1=32, dv=192, H=4, KV=2),
}


@pytest.mark.parametrize("queries, contexts", [((1,), (1,)), ((1,) * 8, (17, 400, 129, 2040, 1, 16, 31, 33)), ((1, 2, 1), (1500, 700, 5)), ((2, 1), (65, 64))])
@pytest.mark.parametrize("form", FORMS)
def test_few_rows_beside_the_general_kernels(ops, form, queries, contexts, monkeypatch):
    f = dict(FORMS[form])
    d0, d1, dv, H, KV, maps = f["d0"], f.get("d1", 0), f["dv"], f["H"], f["KV"], f.get("maps", 1)
    page, pages = 16, sum(-(-c // 16) for c in contexts) + 3
    n, dk = sum(queries), maps * d0 + d1
    if f.get("alias"):
        keys = rnd(pages, page, dk, seed=1)
        values, strides = keys, (page * dk, 0, dk)
        v_strides = strides
    else:
        keys, values = rnd(pages, KV, page, dk, seed=1), rnd(pages, KV, page, dv, seed=2)
        strides, v_strides = (KV * page * dk, page * dk, dk), (KV * page * dv, page * dv, dv)
    q0, q1 = rnd(n, H, maps * d0, seed=3), rnd(n, H, d1, seed=4) if d1 else None
    kw = dict(num_heads=H, num_kv_heads=KV, scale=dk**-0.5, window=f.get("window"), keep_first=f.get("keep_first"), chunk=f.get("chunk"),
              softcap=f.get("softcap"))
    if f.get("slopes"):
        kw["slopes"] = rnd(H, dtype=torch.float32, seed=5).abs() * 0.1
    if f.get("sinks"):
        kw["sinks"] = rnd(H, dtype=torch.float32, seed=6)
    if f.get("gate"):
        kw.update(gate=rnd(n, H * (dv if f["gate"] == 1 else 1) + 4, dtype=torch.float32, seed=7), gate_per_head=f["gate"] == 2)
    if maps == 2:
        kw["differential"] = ops.DifferentialMaps(0.4, 1e-6, 0.5)
    if f.get("turn"):
        angle = rnd(n, dv // 2, dtype=torch.float32, seed=8)
        kw.update(turn=torch.stack((angle.cos(), angle.sin()), -1).contiguous(), turn_neighbours=f.get("turn_neighbours", False))
    assert dk % 32 == 0 and dv % 64 == 0 and max(queries) <= 16 and max(queries) * H // KV * maps <= ops._ROWS_FEW

    def run(dtype, apart):
        table, ctx = step(queries, contexts, page, pages, apart)
        k = keys.to(dtype)
        v = k if f.get("alias") else values.to(dtype)
        return ops.attention_rows(q0.to(dtype), None if q1 is None else q1.to(dtype), k.data_ptr(), strides, v.data_ptr(), v_strides, dv, table, page, ctx, **kw).float()

    want = run(torch.float32, False)
    got, early = run(torch.bfloat16, False), run(torch.bfloat16, True)
    monkeypatch.setattr(ops, "_ROWS_FEW", 0)
    other = run(torch.bfloat16, False)
    # the same operands: what differs is the rounding of weights and results to bfloat16 (2^-9 of the largest weight each, and of two
    # maps' difference), as in the kernel for many rows
    scale = float(want.abs().max())
    assert torch.equal(got, early)
    assert float((got - want).abs().max()) <= 0.02 * scale
    assert float((got - want).norm()) <= 1.1 * float((other - want).norm()) + 1e-4 * float(want.norm())


@pytest.mark.parametrize("n, heads, dim, rot, rank", [(1, 32, 64, 32, 256), (8, 16, 64, 32, 128), (16, 3, 16, 16, 72), (5, 2, 128, 64, 33)])
@pytest.mark.parametrize("own", [False, True])
def test_latent_prepare_with_the_up_product(ops, n, heads, dim, rot, rank, own):
    width = heads * (dim + rot)
    proj = rnd(n, (16 if own else width) + rank + rot + 7, seed=1)
    queries = rnd(n, width + 8, seed=2)[:, :width] if own else None
    w_up, weight = rnd(heads, rank, dim, seed=3), rnd(rank, dtype=torch.float32, seed=4)
    freq = torch.rand(rot // 2, device=DEV)
    positions, slots = torch.arange(n, dtype=torch.int32, device=DEV) * 3, torch.arange(n, dtype=torch.int32, device=DEV)
    planes = [torch.zeros(2, 16, rank + rot, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    args = lambda plane: (proj, positions, slots, plane, weight, freq, 1e-6, heads, dim, rot, rank)  # noqa: E731
    more = dict(queries=queries, kv_col=16) if own else {}
    q_rot, q_up = ops.latent_prepare(*args(planes[0]), **more, w_up=w_up)
    assert torch.equal(q_rot, ops.latent_prepare(*args(planes[1]), **more)) and torch.equal(*planes)
    plain = (queries if own else proj[:, :width]).reshape(n, heads, dim + rot)[:, :, :dim]
    want = torch.einsum("nhd,hmd->nhm", plain.double(), w_up.double())
    # one rounding to bfloat16 behind 32-bit sums
    torch.testing.assert_close(q_up.double(), want, rtol=2.0**-8, atol=1e-4 * dim)


@pytest.mark.parametrize("splits", [1, 7, 8, 9, 32])
@pytest.mark.parametrize("dv, n_out, shift", [(256, 64, 0), (128, 33, 0), (208, 17, 0), (66, 5, 0), (256, 64, 2), (320, 16, 0)])
def test_merge_and_product_of_shares_some_without_keys(ops, splits, dv, n_out, shift):
    n, heads = 3, 5
    o, ml = rnd(n, heads, splits, dv, dtype=torch.float32, seed=1), rnd(n, heads, splits, 2, dtype=torch.float32, seed=2)
    ml[..., 1] = ml[..., 1].abs() + 0.5
    if splits > 1:  # shares without keys were never written
        ml[:, 1::2, 1:, 0] = -torch.inf
        ml[:, 1::2, 1:, 1] = 0.0
        o[:, 1::2, 1:] = torch.nan
    w = rnd(heads * n_out * dv + shift, seed=3)[shift:].view(heads, n_out, dv)
    gate = rnd(n, heads * n_out, seed=4)
    got = ops.merge_project_gate(ops.AttentionParts(o.flatten(), ml.flatten(), splits, n, heads, dv), w, gate)
    share = torch.exp2(ml[..., 0].double() - ml[..., 0].double().amax(-1, keepdim=True))
    merged = (share[..., None] * o.double().nan_to_num()).sum(2) / (share * ml[..., 1].double()).sum(2)[..., None]
    want = torch.einsum("nhd,hmd->nhm", merged, w.double()).flatten(1) * torch.sigmoid(gate.double())
    torch.testing.assert_close(got.double(), want, rtol=2.0**-8, atol=1e-5 * dv)


@pytest.mark.parametrize("leave", [False, True])
@pytest.mark.parametrize("contexts", [(40, 9), (700, 2000), (130, 1)])
@pytest.mark.parametrize("where", ["query", "first key", "newest key", "a key in the middle", "a tile of keys"])
def test_nan_comes_out_where_it_is_seen(ops, where, contexts, leave, monkeypatch):
    """A row that sees a NaN score is NaN, also where a warp's keys, or a whole share's, score nothing else; every other row is as it was."""
    H, KV, page, dk, dv = 8, 1, 16, 288 if leave else 64, 256 if leave else 64
    pages, n = sum(-(-c // page) for c in contexts) + 1, len(contexts)
    q, keys = rnd(n, H, dk, seed=1), rnd(pages, KV, page, dk, seed=2)
    values, w = rnd(pages, KV, page, dv, seed=3), rnd(H, 24, dv, seed=4)
    table, ctx = step((1,) * n, contexts, page, pages, False)

    def run():
        out = ops.attention_rows(q, None, keys.data_ptr(), (KV * page * dk, page * dk, dk), values.data_ptr(), (KV * page * dv, page * dv, dv), dv, table, page, ctx,
                                 num_heads=H, num_kv_heads=KV, scale=dk**-0.5, leave_parts=leave)
        if isinstance(out, ops.AttentionParts):
            return ops.merge_project_gate(out, w, None).view(n, H, -1)
        return ops.head_linear(out, w) if leave else out

    clean = run()
    context = contexts[0]
    at = {"first key": (0,), "newest key": (context - 1,), "a key in the middle": (context // 2,), "a tile of keys": range(16, 32)}.get(where)
    if at is None:
        q[0, 3] = torch.nan
    else:
        for j in at:
            keys[int(table[0, j // page]), :, j % page] = torch.nan
    bad = torch.zeros(n, H, dtype=torch.bool, device=DEV)
    bad[0, 3 if at is None else slice(None)] = True
    for rows_few in (ops._ROWS_FEW, 0):  # the kernel for many rows is no other way
        monkeypatch.setattr(ops, "_ROWS_FEW", rows_few)
        got = run()
        assert bool(got[bad].isnan().all()), f"{where}: NaN was lost ({'many' if rows_few == 0 else 'few'} rows)"
        if rows_few:
            assert torch.equal(got[~bad], clean[~bad])
        else:
            assert bool(got[~bad].isfinite().all())


@pytest.mark.parametrize("maps, sinks", [(1, True), (2, False)])
def test_nan_beside_sinks_and_in_one_of_two_maps(ops, maps, sinks):
    H, KV, page, d, dv, contexts = 8, 2, 16, 64, 64, (300, 20)
    dk, pages = maps * d, 25
    q, keys, values = rnd(2, H, dk, seed=1), rnd(pages, KV, page, dk, seed=2), rnd(pages, KV, page, dv, seed=3)
    table, ctx = step((1, 1), contexts, page, pages, False)
    kw = dict(num_heads=H, num_kv_heads=KV, scale=0.1)
    if sinks:
        kw["sinks"] = torch.where(torch.arange(H, device=DEV) % 2 == 0, -torch.inf, 0.5)  # (-inf: as if there were none)
    if maps == 2:
        kw["differential"] = ops.DifferentialMaps(0.4, 1e-6, 0.5)
    run = lambda: ops.attention_rows(q, None, keys.data_ptr(), (KV * page * dk, page * dk, dk), values.data_ptr(), (KV * page * dv, page * dv, dv), dv, table, page, ctx, **kw)  # noqa: E731
    clean = run()
    assert bool(clean.isfinite().all())
    keys[int(table[0, 0]), 1, 2, d * (maps - 1) :] = torch.nan  # key 2 of the first request, its last map's lanes alone
    got = run()
    seen = torch.zeros(2, H, dtype=torch.bool, device=DEV)
    seen[0, H // KV :] = True
    assert bool(got[seen].isnan().all()) and torch.equal(got[~seen], clean[~seen])


@pytest.mark.parametrize("form", ["plain", "a short key in two runs", "whole group", "sink and gate", "two maps", "latent", "short latent"])
def test_every_number_of_shares(ops, form, monkeypatch):
    """However many CTAs share a tile's keys, more than there are keys for among them: the same result up to the order of its sums."""
    f = dict(FORMS[form])
    d0, d1, dv, H, KV, maps, page, contexts = f["d0"], f.get("d1", 0), f["dv"], f["H"], f["KV"], f.get("maps", 1), 16, (3, 200, 1100)
    pages, n, dk = sum(-(-c // page) for c in contexts) + 1, len(contexts), maps * d0 + d1
    keys, values = rnd(pages, KV, page, dk, seed=1), rnd(pages, KV, page, dv, seed=2)
    q0, q1 = rnd(n, H, maps * d0, seed=3), rnd(n, H, d1, seed=4) if d1 else None
    kw = dict(num_heads=H, num_kv_heads=KV, scale=dk**-0.5)
    if f.get("sinks"):
        kw.update(sinks=rnd(H, dtype=torch.float32, seed=6), gate=rnd(n, H * dv, dtype=torch.float32, seed=7))
    if maps == 2:
        kw["differential"] = ops.DifferentialMaps(0.4, 1e-6, 0.5)
    table, ctx = step((1,) * n, contexts, page, pages, False)
    run = lambda **more: ops.attention_rows(q0, q1, keys.data_ptr(), (KV * page * dk, page * dk, dk), values.data_ptr(), (KV * page * dv, page * dv, dv), dv, table, page, ctx, **kw, **more)  # noqa: E731
    monkeypatch.setattr(ops, "_few_plan", lambda *a: 0)
    want = run().float()
    for shares in (1, 2, 4, 8):
        monkeypatch.setattr(ops, "_few_plan", lambda *a: shares)
        got = run().float()
        # weights rounded to bfloat16 on either side (2^-9 of the largest), results too
        assert float((got - want).abs().max()) <= 0.02 * float(want.abs().max()), f"{shares} shares"
    if form in ("latent", "short latent"):
        w = rnd(H, 16, dv, seed=5)
        want = ops.head_linear(want.bfloat16(), w).flatten(1).float()
        for shares in (2, 3, 9, 32):
            monkeypatch.setattr(ops, "_few_plan", lambda *a: shares)
            got = ops.merge_project_gate(run(leave_parts=True), w, None).float()
            assert float((got - want).abs().max()) <= 0.03 * float(want.abs().max()), f"{shares} shares left"


@pytest.mark.parametrize("latent", [False, True])
@pytest.mark.parametrize("news", [1, 3])
@pytest.mark.parametrize("contexts", [(15, 16, 17), (31, 32, 33), (160, 144, 47), (2000, 1999, 1)])
def test_the_newest_rows_are_the_work_of_the_kernel_in_front(ops, contexts, news, latent):
    """Keys cached before the step are read while the kernel that writes the step's own rows still runs (``steps_apart``), and those are not:
    the two kernels directly behind one another in a graph, other rows in their slots before every replay."""
    contexts = tuple(max(c, news) for c in contexts)
    H, KV, D, V, page, rank, rot, dim = 16, 4, 64, 64, 16, 128, 32, 64
    pages = sum(-(-c // page) for c in contexts) + 2
    n = news * len(contexts)
    table, ctx = step((news,) * len(contexts), contexts, page, pages, True)
    positions = [c - news + i for c in contexts for i in range(news)]
    owner = ctx.token_request.tolist()
    slots = torch.tensor([int(table[r, p // page]) * page + p % page for r, p in zip(owner, positions)], dtype=torch.int32, device=DEV)
    pos = torch.tensor(positions, dtype=torch.int32, device=DEV)
    if latent:
        pool = rnd(pages, page, rank + rot, seed=1)
        proj = rnd(n, H * (dim + rot) + rank + rot, seed=2)
        weight, freq = torch.ones(rank, device=DEV), torch.rand(rot // 2, device=DEV)
        q_lat = rnd(n, H, rank, seed=3)

        def run():
            q_rot = ops.latent_prepare(proj, pos, slots, pool, weight, freq, 1e-6, H, dim, rot, rank)
            return ops.latent_paged_attention(q_lat, q_rot, pool, table, ctx, rank=rank, scale=0.08)
    else:
        pool = rnd(pages, 2, KV, page, D, seed=1)
        proj = rnd(n, (H + KV) * D + KV * V, dtype=torch.float32, seed=2)

        def run():
            q = ops.head_prepare(proj, pos, heads=H, kv_heads=KV, dim=D, value_dim=V, q_weight=torch.ones(D, device=DEV), k_weight=torch.ones(D, device=DEV), eps=1e-6,
                                 pool=pool, slot_map=slots)
            return ops.paged_softmax_attention(q, pool, table, ctx, num_heads=H, num_kv_heads=KV, key_dim=D, value_dim=V, scale=0.125)

    run()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run()
    fresh, stale = proj.clone(), pool.clone()
    for turn in range(12):
        proj.copy_(fresh * (1.0 + turn) + turn)
        pool.copy_(stale.roll(turn, 0) * 3.0)  # what the slots held before
        graph.replay()
        torch.cuda.synchronize()
        early = got.clone()
        ctx.steps_apart = False
        pool.copy_(stale.roll(turn, 0) * 3.0)
        want = run()
        ctx.steps_apart = True
        assert torch.equal(early, want), f"turn {turn}"
