"""The recurrences' walk without shared memory, for steps in which a request brings few tokens: a token's sums and the state have the bits of a
longer step's."""

import pytest
import torch

from test_kafepel_kernels_gpu import DEV, _ops

pytestmark = pytest.mark.gpu


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


@pytest.mark.parametrize("gated", [False, True])
def test_long_requests_walk_in_the_expected_number_of_stretches(gated, monkeypatch):
    """Every number of stretches that the rule may choose gives the same outputs and states to the sums' rounding: 24 (the most), one that fills
    the SMs once, and 1, for requests of which one has fewer tokens than there are stretches."""
    ops = _ops()
    heads, dim, value_dim, lens = 4, 64, 48, [1600, 7, 300]
    gen = torch.Generator(device=DEV).manual_seed(3)
    q, k, z = (0.3 * torch.randn(sum(lens), heads * dim, device=DEV, generator=gen) for _ in range(3))
    v = torch.randn(sum(lens), heads * value_dim, device=DEV, generator=gen)
    start = torch.randn(4, heads, dim, value_dim, device=DEV, generator=gen)
    cu = torch.tensor([0, 1600, 1607, 1907], dtype=torch.int32, device=DEV)
    slots = torch.tensor([2, 0, 3], dtype=torch.int32, device=DEV)

    def run():
        states = start.clone()
        args = (states, slots, cu, 3, heads, dim, value_dim, max(lens))
        out = ops.gated_scan(q, k, v, z, None, 0.1, 1.0, *args) if gated else ops.retention_scan(q, k, v, torch.linspace(0.9, 0.99, heads, device=DEV), *args)
        return out, states

    assert ops._scan_stretches(False, dim, value_dim, heads, 1, 1600, 1600, gated) > 8
    monkeypatch.setattr(ops, "_scan_stretches", lambda *a: 1)
    want = run()
    for n in (13, 24):
        monkeypatch.setattr(ops, "_scan_stretches", lambda *a, n=n: n)
        for got, ref in zip(run(), want):  # 32-bit sums of some hundred decaying terms in another order: 2^-24 * sqrt(1600) * their size
            assert (got - ref).abs().max() <= 4e-6 * ref.abs().max()
