"""A mixture of experts for few tokens, of which only the used experts are read, beside the double statement of the same: token counts at
the edges of its tiles, widths that leave warps without work, every form of weights and of ends; experts that nobody uses hold NaN."""

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


@pytest.mark.parametrize("m", [1, 3, 8])
@pytest.mark.parametrize("K, N, E, ff, fs", [(2048, 2048, 32, 704, 1408), (1024, 1024, 16, 512, 1024), (32, 16, 1, 32, 0), (992, 48, 37, 64, 32),
                                             (2048, 160, 256, 32, 0), (96, 32, 9, 1568, 800)])
@pytest.mark.parametrize("form", ["gated", "table", "relu2", "silu", "gelu_tanh"])
def test_used_experts_alone(m, K, N, E, ff, fs, form):
    from llmserve_triton_kernels_b200 import ops

    act = form if form in ("relu2", "silu", "gelu_tanh") else None
    per, top = 1 if act else 2, min(4, E)
    x = rnd(m, K + 8, seed=1)[:, :K]
    w_up, w_down = rnd(per * (E * ff + fs), K, seed=2, scale=K**-0.5), rnd(N, E * ff + fs, seed=3, scale=ff**-0.5)
    g = torch.Generator().manual_seed(m)
    chosen = torch.rand(m, E, generator=g).argsort(1)[:, :top].to(DEV)
    kw = dict(activation=act) if act else dict(limit=1.5, shared_limit=1.0, slope=1.702, up_shift=1.0)
    if form == "table":
        table = torch.zeros(50, top, dtype=torch.int32, device=DEV)
        ids = torch.arange(m, dtype=torch.int32, device=DEV) * 2 + 1
        table[ids.long()] = chosen.int()
        kw.update(ids=ids, table=table)
        wts = torch.zeros(m, E + 1, device=DEV).scatter(1, chosen, 1.0 / top)
        wts[:, E] = 1.0
    else:
        wts = torch.zeros(m, E + 1, device=DEV).scatter(1, chosen, rnd(m, top, dtype=torch.float32, seed=5).abs() + 0.1)
        wts[:, E] = rnd(m, dtype=torch.float32, seed=6).abs() + 0.1
        kw.update(weights=wts[:, : E + (fs > 0)].contiguous())
    for e in range(E):
        if not bool((wts[:, e] != 0).any()):
            w_up[e * per * ff : (e + 1) * per * ff] = torch.nan
            w_down[:, e * ff : (e + 1) * ff] = torch.nan
    want = stated(x, w_up, w_down, E, ff, fs, wts, act, (1.5, 1.0), 1.702, 1.0)
    got = ops.experts_few(x, w_up, w_down, E, ff, fs, **kw)
    # the activations are rounded to bfloat16 (2^-9 each, signs at random), the sums are 32-bit
    assert float((got.double() - want).norm()) <= 3e-3 * float(want.norm())
    resid, weight = rnd(m, N, dtype=torch.float32, seed=7), rnd(N, dtype=torch.float32, seed=8)
    stream = resid.clone()
    handed = ops.experts_few(x, w_up, w_down, E, ff, fs, **kw, sink=ops.ResidualSink(stream, weight, 1e-5))
    new = resid.double() + got.double()
    torch.testing.assert_close(stream.double(), new, rtol=1e-6, atol=1e-5)
    torch.testing.assert_close(handed.xw.double(), new * weight.double(), rtol=2.0**-8, atol=1e-5)
    torch.testing.assert_close(handed.ss.sum(0).double(), (new * new).sum(1), rtol=1e-5, atol=1e-5)
    stream = resid.clone()
    assert ops.experts_few(x, w_up, w_down, E, ff, fs, **kw, sink=ops.ResidualSink(stream, None, 1e-5, alpha=0.5)) is ops.ADDED
    torch.testing.assert_close(stream.double(), resid.double() + 0.5 * got.double(), rtol=1e-6, atol=1e-5)


def test_what_it_does_not_take_goes_the_other_way():
    from llmserve_triton_kernels_b200 import ops

    def call(m, K, N, ff, dtype=torch.bfloat16):
        return ops.experts_few(rnd(m, K, dtype=dtype), rnd(4 * ff, K, dtype=dtype), rnd(N, 4 * ff, dtype=dtype), 4, ff, 0, activation="silu",
                               weights=torch.ones(m, 4, device=DEV))

    assert call(2, 64, 32, 32) is not None
    for args in ((9, 64, 32, 32), (2, 48, 32, 32), (2, 2080, 32, 32), (2, 64, 24, 32), (2, 64, 32, 48), (2, 64, 32, 32, torch.float32)):
        assert call(*args) is None, args


@pytest.mark.parametrize("K, N, E, ff, fs", [(2048, 256, 32, 704, 1408), (256, 64, 37, 96, 0), (512, 32, 8, 1568, 800)])
@pytest.mark.parametrize("form", ["gated", "silu"])
def test_a_row_has_its_bits_whatever_the_other_tokens_use(K, N, E, ff, fs, form):
    """The order of a token's sums depends on its own experts: beside others that use all experts, or its own, or none of them."""
    from llmserve_triton_kernels_b200 import ops

    per = 2 if form == "gated" else 1
    x = rnd(8, K, seed=1)
    w_up, w_down = rnd(per * (E * ff + fs), K, seed=2, scale=K**-0.5), rnd(N, E * ff + fs, seed=3, scale=ff**-0.5)
    kw = dict(activation="silu") if form == "silu" else dict(limit=1.5, shared_limit=1.0, slope=1.702, up_shift=1.0)
    g = torch.Generator().manual_seed(E)
    wts = torch.zeros(8, E + 1, device=DEV)
    for t in range(8):
        wts[t, torch.randperm(E, generator=g)[: min(4, E)].to(DEV)] = 0.1 + 0.2 * t
    wts[:, E] = 1.0
    wts = wts[:, : E + (fs > 0)].contiguous()
    run = lambda rows, w: ops.experts_few(x[rows].contiguous(), w_up, w_down, E, ff, fs, weights=w[rows].contiguous(), **kw)  # noqa: E731
    alone = torch.cat([run([t], wts) for t in range(8)])
    for count in (2, 3, 5, 8):
        assert torch.equal(run(list(range(count)), wts), alone[:count]), f"{count} tokens"
    crowded = wts.clone()
    crowded[1:, :E] = 0.3  # the others use every expert
    assert torch.equal(run(list(range(8)), crowded)[0], alone[0])


@pytest.mark.parametrize("tokens", [1, 2, 5, 8])
@pytest.mark.parametrize("kind", ["routed", "gated", "table"])
@pytest.mark.parametrize("sunk", [False, True])
def test_parts_give_the_same_either_way(kind, tokens, sunk, monkeypatch):
    """A part whose used experts are read alone beside itself with the products over all experts."""
    from types import SimpleNamespace

    from llmserve_triton_kernels_b200 import ops
    from llmserve_triton_kernels_b200.parts.feed_forward import RoutedGatedMLP, RoutedMLP, TableRoutedMLP

    K, E, top, ff, fs = 1024, 32, 2, 512, 256
    part = {"routed": lambda: RoutedMLP(K, E, top, ff, shared_size=fs, correction=False), "gated": lambda: RoutedGatedMLP(K, E, top, ff, fs),
            "table": lambda: TableRoutedMLP(K, 64, E, top, ff, 7.0, fs)}[kind]()
    tensors = {name: rnd(*spec.shape, seed=i, scale=0.05) for i, (name, spec) in enumerate(part.tensors().items())}
    if kind == "table":
        tensors["table"] = torch.rand(64, E, generator=torch.Generator().manual_seed(1)).argsort(1)[:, :top].to(DEV)
    part.bind(tensors, torch.bfloat16, DEV)
    x, ctx = rnd(tokens, K, seed=99), SimpleNamespace(token_ids=torch.arange(tokens, dtype=torch.int32, device=DEV) * 5)
    launches, launch = [], ops._launch
    monkeypatch.setattr(ops, "_launch", lambda name, *args: launches.append(name) or launch(name, *args))

    def run():
        launches.clear()
        stream = rnd(tokens, K, dtype=torch.float32, seed=5)
        out = part.forward(x, ctx, ops.ResidualSink(stream, None, 1e-5) if sunk else None)
        return stream if sunk else out

    monkeypatch.setattr(ops, "_EXPERTS_FEW_SHARE", 10.0)
    got = run()
    assert "llm_experts_few" in launches
    monkeypatch.setattr(ops, "_EXPERTS_FEW_SHARE", 0.0)
    want = run()
    assert "llm_experts_few" not in launches
    # inner activations rounded to bfloat16 on the one side before, on the other behind the product's rounding: 2^-8 of each
    scale = float((want - (rnd(tokens, K, dtype=torch.float32, seed=5) if sunk else 0)).norm())
    assert float((got - want).norm()) <= 8e-3 * scale
