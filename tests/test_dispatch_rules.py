"""Which of two kernels a step takes, at sizes where both were timed on a B200: the faster one."""

import pytest

from llmserve_triton_kernels_b200 import ops


@pytest.fixture
def b200(monkeypatch):
    monkeypatch.setattr(ops, "_sm_count", lambda: 148)
    # what the device answers: clusters of eight large CTAs leave 28 SMs without work
    at_once = {True: {1: 296, 2: 296, 4: 284, 8: 264}, False: {1: 148, 2: 148, 4: 132, 8: 120}}
    monkeypatch.setattr(ops, "_few_resident", lambda device, dk, dv, maps, leave, splits: at_once[dk <= 64 and dv <= 64][1 if leave else splits])


# (query heads, key heads, key lanes, value lanes, maps, partial results left), requests, keys, tokens a request
MANY = [((128, 1, 288, 256, 1, False), 128, 2000, 1), ((128, 1, 288, 256, 1, False), 128, 100, 1), ((128, 1, 288, 256, 1, True), 8, 2000, 1),
        ((32, 1, 288, 256, 1, False), 8, 2000, 4), ((32, 1, 288, 256, 1, False), 32, 2000, 4), ((16, 1, 128, 128, 1, False), 32, 2000, 4),
        ((32, 8, 128, 128, 2, False), 32, 100, 4), ((32, 8, 128, 128, 2, False), 32, 2000, 4), ((64, 8, 128, 128, 1, False), 32, 100, 4),
        ((64, 8, 128, 128, 1, False), 32, 2000, 4), ((32, 1, 288, 256, 1, False), 8, 2000, 1),
        ((32, 1, 288, 256, 1, False), 32, 2000, 1)]
FEW = [((32, 8, 64, 64, 1, False), 1, 100, 1), ((32, 8, 64, 64, 1, False), 128, 2000, 1), ((32, 8, 64, 64, 1, False), 32, 100, 4), ((32, 1, 288, 256, 1, True), 8, 2000, 1),
       ((32, 1, 288, 256, 1, False), 32, 100, 1), ((128, 1, 288, 256, 1, True), 1, 2000, 1), ((128, 1, 288, 256, 1, False), 8, 100, 1), ((16, 1, 128, 128, 1, False), 128, 2000, 1),
       ((32, 8, 128, 128, 2, False), 128, 2000, 1), ((32, 8, 128, 128, 2, False), 8, 100, 4), ((64, 8, 128, 128, 1, False), 8, 100, 4)]


def few_plan(shape, requests, keys, tokens):
    heads, kv, dk, dv, maps, leave = shape
    rows, n = tokens * heads // kv * maps, requests * tokens
    ctas = -(-rows // 64) * kv * requests
    many_splits = max(1, min(-(-keys // 128), (2 if dv <= 128 else 1) * 148 // ctas, 16, ops._SPLIT_SCRATCH_BYTES // (n * heads * maps * dv * 4)))
    return ops._few_plan.__wrapped__(0, keys, -(-rows // 16) * kv * requests, dk, dv, maps, leave, ops._SPLIT_SCRATCH_BYTES // (n * heads * dv * 4), ctas, many_splits)


@pytest.mark.parametrize("call", MANY)
def test_attention_of_many_tiles_stays_with_the_kernel_for_many_rows(b200, call):
    assert few_plan(*call) == 0


@pytest.mark.parametrize("call", FEW)
def test_attention_of_few_rows_takes_the_kernel_for_them(b200, call):
    assert few_plan(*call) > 0


def test_clusters_that_do_not_fit_at_once_are_not_asked_for(b200):
    # sixteen tiles: sixteen clusters of eight take two waves, sixteen of four one
    assert few_plan((64, 8, 128, 128, 1, False), 1, 2000, 4) == 4
    assert few_plan((64, 8, 128, 128, 1, False), 1, 2000, 1) == 8


@pytest.mark.parametrize("tokens, dim, one_launch", [(1, 64, True), (1, 128, True), (4, 64, True), (2, 128, True), (8, 32, True), (7, 64, True), (15, 32, True),
                                                     (8, 64, False), (4, 128, False), (8, 128, False), (16, 32, False), (16, 64, False), (16, 128, False), (1, 8, False), (1, 256, False)])
def test_latent_queries_are_multiplied_beside_the_preparation_while_that_is_shorter(tokens, dim, one_launch):
    class Rows:
        is_cuda, dtype, shape = True, ops.torch.bfloat16, (tokens, 7)

    assert ops.latent_prepare_takes_up(Rows, dim) == one_launch


# hidden, experts, top, inner size, shared inner size, matrices an expert, tokens
@pytest.mark.parametrize("used_alone, sizes", [
    (True, (2048, 32, 4, 704, 1408, 3, 1)), (True, (2048, 32, 4, 704, 1408, 3, 4)), (True, (1024, 16, 2, 512, 1024, 2, 1)), (True, (1024, 16, 2, 512, 1024, 3, 3)),
    (True, (2048, 256, 8, 256, 512, 3, 8)), (True, (2048, 8, 2, 5632, 0, 3, 2)), (True, (2048, 64, 8, 352, 704, 3, 5)),
    (False, (1024, 16, 8, 512, 0, 3, 2)), (False, (1024, 16, 8, 512, 0, 3, 8)), (False, (512, 8, 2, 128, 0, 3, 1)), (False, (1024, 64, 4, 64, 256, 3, 4)),
    (False, (2048, 16, 4, 704, 0, 3, 6)), (False, (2048, 8, 2, 1408, 0, 3, 8)), (False, (2048, 8, 2, 5632, 0, 3, 5)), (False, (64, 4, 2, 32, 0, 2, 1)),
])
def test_the_used_experts_are_read_alone_where_that_is_faster(used_alone, sizes):
    hidden, experts, top, ff, shared, matrices, tokens = sizes
    assert ops.experts_few_pay(tokens, experts, top, ff, shared, 2 * matrices * hidden) == used_alone


def test_experts_of_many_tokens_run_alone_where_that_was_measured_faster(monkeypatch):
    """Steps on both sides of the line, with both ways' times on a B200 (microseconds)."""
    from llmserve_triton_kernels_b200 import ops

    monkeypatch.setattr(ops, "_sm_count", lambda: 148)
    # (microseconds of the sweep that the rule was fitted to, each layer behind a write of 256 MB; the kernels of 1,800 tokens have gained 10 % since)
    for tokens, experts, top, ff, shared, gated, hidden, everybody, used in (
        (512, 32, 4, 704, 1408, True, 2048, 137, 106), (1800, 32, 4, 704, 1408, True, 2048, 404, 212), (120, 32, 4, 704, 1408, True, 2048, 90, 90),
        (1024, 32, 4, 704, 1408, False, 2048, 165, 137), (256, 32, 4, 704, 1408, False, 2048, 79, 84), (512, 16, 2, 512, 1024, True, 1024, 51, 57),
        (1800, 16, 2, 512, 1024, True, 1024, 106, 93), (4096, 16, 2, 512, 1024, False, 1024, 143, 148), (1800, 16, 8, 704, 1408, True, 2048, 232, 284),
        (4096, 8, 6, 512, 0, True, 512, 85, 171), (1800, 8, 2, 1408, 0, True, 2048, 194, 140), (4096, 4, 2, 2816, 0, True, 1024, 253, 277),
    ):
        assert ops.experts_many_pay(tokens, experts, top, ff, shared, gated, hidden) == (used < 0.98 * everybody), (tokens, experts, hidden)
    assert not ops.experts_many_pay(4096, 8, 8, 704, 0, True, 2048)  # every token uses every expert


# heads (times maps), key lanes, value lanes, long request, riders, their tokens, whether they were faster along with it
@pytest.mark.parametrize("heads,dk,dv,long,riders,tokens,along", [
    (32, 64, 64, 512, 4, 32, True), (32, 64, 64, 512, 16, 32, False), (32, 64, 64, 512, 63, 32, False), (32, 64, 64, 128, 8, 32, True), (32, 64, 64, 2000, 16, 32, False),
    (32, 64, 64, 512, 16, 100, True), (32, 64, 64, 2000, 63, 64, True), (8, 64, 64, 512, 16, 32, True), (32, 128, 128, 512, 63, 48, True), (64, 128, 128, 512, 16, 32, True),
    (32, 64, 128, 1800, 32, 32, True), (32, 96, 64, 512, 32, 32, True), (32, 64, 64, 512, 4, 24, False), (32, 128, 128, 512, 31, 24, False)])
def test_small_requests_go_along_with_a_long_one_where_that_is_faster(b200, heads, dk, dv, long, riders, tokens, along):
    class Step:
        host_cu_tokens = [0, long, *(long + tokens * (i + 1) for i in range(riders))]

    assert (tokens >= ops._tc_join_tokens(Step, heads, dk, dv, ops._TC_ATTENTION_JOIN_CROWDED)) == along


def test_small_requests_beside_the_general_form_in_a_crowd(b200):
    class Step:
        host_cu_tokens = [0, 512, *(512 + 48 * (i + 1) for i in range(32))]

    assert ops._tc_join_tokens(Step, 32, 64, 64, ops._TC_ATTENTION_JOIN_CROWDED_GENERAL) == 48
