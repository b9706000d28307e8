"""A mixture of experts for many tokens, each through its own experts alone, beside the double statement of the same: token counts at the
edges of its tiles (16, 256 columns), widths that leave a tile's rows without work, every form of weights and of ends; experts that nobody uses
hold NaN, one expert is used by every token."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, dtype=torch.bfloat16, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


def stated(x, w_up, w_down, E, ff, fs, wts, act, limits, slope, shift):
    out, per = 0, 1 if act else 2
    for e in range(E + (fs > 0)):
        f = fs if e == E else ff
        use = wts[:, e] != 0
        up = x.double() @ w_up[e * per * ff : e * per * ff + per * f].double().T
        if act is None:
            g, u = up[:, :f].clamp(max=limits[e == E]), up[:, f:].clamp(-limits[e == E], limits[e == E])
            y = g * torch.sigmoid(slope * g) * (u + shift)
        else:
            y = {"relu2": lambda v: torch.relu(v) ** 2, "silu": torch.nn.functional.silu,
                 "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[act](up)
        y = y * wts[:, e : e + 1].double()
        part = y @ w_down[:, e * ff : e * ff + f].double().T
        out = out + torch.where(use[:, None], part, torch.zeros_like(part))
    return out


@pytest.mark.parametrize("m", [1, 9, 40, 257, 530])
@pytest.mark.parametrize("K, N, E, ff, fs", [(2048, 2048, 32, 704, 1408), (72, 36, 5, 40, 0), (1024, 1000, 37, 64, 136), (128, 128, 2, 8, 264), (64, 256, 256, 128, 0)])
@pytest.mark.parametrize("form, width", [("gated", 64), ("gated", 128), ("gated", 256), ("table", 128), ("relu2", 256), ("silu", 64), ("gelu_tanh", 128)])
def test_used_experts_alone(m, K, N, E, ff, fs, form, width, monkeypatch):
    from llmserve_triton_kernels_b200 import ops

    monkeypatch.setattr(ops, "_EXPERTS_MANY_WIDTH", width)  # most tokens of a tile

    act = form if form in ("relu2", "silu", "gelu_tanh") else None
    per, top = 1 if act else 2, min(4, E - 1)
    x = rnd(m, K + 8, seed=1)[:, :K]
    w_up, w_down = rnd(per * (E * ff + fs), K, seed=2, scale=K**-0.5), rnd(N, E * ff + fs, seed=3, scale=ff**-0.5)
    g = torch.Generator().manual_seed(m)
    order = torch.rand(m, E, generator=g)
    order[:, min(3, E - 1)] = -1.0  # everybody's
    chosen = order.argsort(1)[:, :top].to(DEV)
    kw = dict(activation=act) if act else dict(limit=1.5, shared_limit=1.0, slope=1.702, up_shift=1.0)
    if form == "table":
        table = torch.zeros(2 * m + 1, top, dtype=torch.int32, device=DEV)
        ids = torch.arange(m, dtype=torch.int32, device=DEV) * 2 + 1
        table[ids.long()] = chosen.int()
        kw.update(ids=ids, table=table)
        wts = torch.zeros(m, E + 1, device=DEV).scatter(1, chosen, 1.0 / top)
        wts[:, E] = 1.0
    else:
        wts = torch.zeros(m, E + 1, device=DEV).scatter(1, chosen, rnd(m, top, dtype=torch.float32, seed=5).abs() + 0.1)
        wts[::3, :E] *= torch.arange(E, device=DEV) != int(chosen[0, -1])  # tokens of fewer experts
        wts[:, E] = rnd(m, dtype=torch.float32, seed=6).abs() + 0.1
        kw.update(weights=wts[:, : E + (fs > 0)].contiguous())
    for e in range(E):
        if not bool((wts[:, e] != 0).any()):
            w_up[e * per * ff : (e + 1) * per * ff] = torch.nan
            w_down[:, e * ff : (e + 1) * ff] = torch.nan
    want = stated(x, w_up, w_down, E, ff, fs, wts, act, (1.5, 1.0), 1.702, 1.0)
    got = ops.experts_many(x, w_up, w_down, E, ff, fs, **kw, top=top)
    # the activations are rounded to bfloat16 (2^-9 each, signs at random), the sums are 32-bit
    assert float((got.double() - want).norm()) <= 3e-3 * float(want.norm())
    assert torch.equal(got, ops.experts_many(x, w_up, w_down, E, ff, fs, **kw, top=top))
    resid = rnd(m, N, dtype=torch.float32, seed=7)
    stream = resid.clone()
    assert ops.experts_many(x, w_up, w_down, E, ff, fs, **kw, top=top, sink=ops.ResidualSink(stream, None, 1e-5, alpha=0.5)) is ops.ADDED
    torch.testing.assert_close(stream.double(), resid.double() + 0.5 * got.double(), rtol=1e-6, atol=1e-5)


def test_what_it_does_not_take_goes_the_other_way():
    from llmserve_triton_kernels_b200 import ops

    x, w_up, w_down = rnd(20, 60), rnd(2 * 4 * 12, 60), rnd(32, 4 * 12)
    kw = dict(limit=1.0, shared_limit=1.0, weights=torch.ones(20, 4, device=DEV), top=4)
    before = ops.launch_count()
    assert ops.experts_many(x, w_up, w_down, 4, 12, 0, **kw) is None  # rows that do not start on 16 bytes
    assert ops.launch_count() == before
    assert ops.experts_many(x.float(), w_up.float(), w_down.float(), 4, 12, 0, **kw) is None


def test_many_tokens_wide_rows_and_a_table_with_repeats():
    """More tokens than the sort's CTA has threads, rows of more pieces than the gather asks for in advance, a table row that names an expert
    twice and token ids outside the table (which read its first row, as in the products over all experts)."""
    from llmserve_triton_kernels_b200 import ops

    m, K, N, E, ff, fs = 1100, 2304, 1152, 4, 24, 8
    x, w_up, w_down = rnd(m, K), rnd(2 * (E * ff + fs), K, seed=1, scale=K**-0.5), rnd(N, E * ff + fs, seed=2, scale=ff**-0.5)
    table = torch.tensor([[1, 3], [2, 2], [0, 1], [3, 0]], dtype=torch.int32, device=DEV)
    ids = torch.arange(m, dtype=torch.int32, device=DEV) % 6 - 1  # -1 and 4 are outside
    rows = table[torch.where((ids < 0) | (ids > 3), 0, ids).long()].long()
    wts = torch.zeros(m, E + 1, device=DEV).scatter(1, rows, 0.5)
    wts[:, E] = 1.0
    kw = dict(limit=1.5, shared_limit=1.0, slope=1.0, up_shift=1.0, ids=ids, table=table)
    got = ops.experts_many(x, w_up, w_down, E, ff, fs, **kw, top=2)
    want = stated(x, w_up, w_down, E, ff, fs, wts, None, (1.5, 1.0), 1.0, 1.0)
    assert float((got.double() - want).norm()) <= 3e-3 * float(want.norm())
    act = ops.expert_gated_act(ops.linear(x, w_up), E, ff, fs, 1.5, 1.0, 1.0, ids=ids, table=table)
    assert float((got.double() - ops.linear(act, w_down).double()).norm()) <= 1e-2 * float(want.norm())
