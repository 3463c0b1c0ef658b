"""Rows that do not begin or end on a 16-byte boundary, and batches whose rows go through different
launches because some rows' penalties can raise a logit: by the automatic choice, which is mostly the team
kernel, and by the ring and the streaming kernel, which take over where that one does not."""
import numpy as np
import pytest
import torch

from flash_gordon_b200 import FG_OK, SamplerConfig, synth
from helpers import as_u32, assert_rows_equal, random_workload, run_gpu, run_oracle

pytestmark = pytest.mark.gpu

CONFIGS = {
    "top_k": SamplerConfig.make(temperature=0.8, top_p=0.95, top_k=20),
    "penalised": SamplerConfig.make(temperature=0.8, top_p=0.9, top_k=64, presence=0.4, frequency=0.3, repetition=1.1),
    "greedy": SamplerConfig.make(temperature=0.0, top_p=1.0, top_k=1, repetition=1.2),
}


@pytest.fixture(params=[0, 255], ids=["automatic choice", "without the team kernel"], autouse=True)
def kernels(context, request):
    context.team_controls(request.param)
    yield request.param
    context.team_controls()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind", CONFIGS)
@pytest.mark.parametrize("vocab,stride,start", [
    (1, 3, 1), (5, 9, 3), (7, 8, 1), (9, 11, 2), (2041, 2049, 0), (2047, 2047, 5), (2048, 2055, 7), (2049, 2050, 1),
    (16383, 16391, 3), (16385, 16385, 0), (100_277, 100_277, 0), (100_280, 100_283, 6),
])
def test_every_offset(context, dtype, kind, vocab, stride, start):
    """`start` elements before the first row, `stride` between rows: nine rows meet every offset
    of a row's first logit from a boundary.  What lies between the rows would win if it were
    looked at; the rows' own ends hold large values, NaN and infinities."""
    rows = 9
    w = random_workload(rows, vocab, 40 if kind != "top_k" else 0, [CONFIGS[kind]], 31 * vocab + start,
                        specials=2 if vocab > 16 else 0, dtype=dtype)
    w.logits[1::3, 0] = 30.0
    w.logits[2::3, -1] = 31.0
    w.logits[0, -1] = float("nan")
    if vocab > 1:
        w.logits[3, 0] = float("inf")
    expected = run_oracle(w)
    block = torch.full((start + rows * stride + 16,), 99.0, dtype=dtype, device="cuda")
    placed = torch.as_strided(block, (rows, vocab), (stride, 1), start)
    placed.copy_(w.logits)
    d = w.to("cuda")
    result = context.sample_batch(placed, d.configs, d.uniforms, d.history_tokens, d.history_offsets, d.history_max)
    torch.cuda.synchronize()
    assert_rows_equal(result, expected, f"{kind} V={vocab}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vocab", [12_346, 12_352])
@pytest.mark.parametrize("raising", [1, 7, 30])
def test_some_rows_of_a_small_batch_raise(context, dtype, vocab, raising):
    """`raising` of 30 rows have penalties that can raise a logit (a batch so small is one launch)."""
    rows = 30
    w = random_workload(rows, vocab, 400, some_raising(rows, raising), 5 + raising, dtype=dtype)
    assert_rows_equal(run_gpu(context, w), run_oracle(w), f"{raising} raising rows")


def some_raising(rows, raising, nucleus_every=0):
    configs = []
    for r in range(rows):
        lift = (r * 7) % rows < raising
        nucleus = nucleus_every and r % nucleus_every == 2
        greedy = r % 5 == 0 and not nucleus
        configs.append(SamplerConfig.make(temperature=0.0 if greedy else 0.9, top_p=0.9,
                                          top_k=0 if nucleus else 1 if greedy else 30,
                                          presence=-0.7 if lift else 0.5, frequency=0.2 * (r % 2),
                                          repetition=1.0 + 0.1 * (r % 3)))
    return configs


@pytest.mark.parametrize("rows,vocab,dtype,raising,nucleus_every", [
    (160, 100_277, torch.bfloat16, 20, 0), (180, 100_277, torch.bfloat16, 1, 8), (128, 131_072, torch.float32, 31, 0),
    (175, 98_049, torch.float32, 31, 11), (128, 131_072, torch.float32, 70, 0),
])
def test_rows_of_a_large_batch_in_two_kernels(context, rows, vocab, dtype, raising, nucleus_every):
    """Above 15 million logits up to a quarter of the rows, the raising ones, are a launch of their own: of the
    team kernel like the others', or of the streaming kernel beside the ring kernel's.  One launch more
    than with a single kernel."""
    w = random_workload(rows, vocab, 300, some_raising(rows, raising, nucleus_every), raising, dtype=dtype, specials=1)
    w.allow_no_topk = bool(nucleus_every)
    expected = run_oracle(w)
    before = context.launches
    assert_rows_equal(run_gpu(context, w), expected, f"{raising} raising rows")
    mixed = context.launches - before
    context.set_path(1)
    try:
        before = context.launches
        assert_rows_equal(run_gpu(context, w), expected, "streaming kernel")
        assert mixed == context.launches - before + (1 if raising < rows // 4 else 0)
    finally:
        context.set_path(0)


def test_rows_of_a_large_shard_in_two_kernels(context):
    """The same for the columns of a shard: the lists of both launches' rows are the whole rows' parts."""
    rows, vocab, width, k = 300, 104_000, 52_000, 24
    configs = [SamplerConfig.make(temperature=0.9, top_p=0.9, top_k=k, presence=-0.6 if r % 9 == 4 else 0.4, frequency=0.1)
               for r in range(rows)]
    w = random_workload(rows, vocab, 200, configs, 78)
    expected = run_oracle(w)
    d = w.to("cuda")
    scores = torch.empty(2, rows, k, device="cuda")
    ids = torch.empty(2, rows, k, dtype=torch.int32, device="cuda")
    for s in range(2):
        before = context.launches
        _, _, _, status = context.shard_topk(d.logits[:, s * width:(s + 1) * width], d.configs, s * width, vocab, k,
                                             d.history_tokens, d.history_offsets, d.history_max, out=(scores[s], ids[s]))
        assert status == FG_OK and context.launches - before == 2
    result = context.merge_select(scores, ids, rows, 2, k, [0, width], [width, width], d.configs, d.uniforms)
    assert np.array_equal(as_u32(result.tokens), expected[1])


@pytest.mark.parametrize("vocab,history,wild", [
    (100_280, 300, dict(frequency=-0.5)), (100_277, 300, dict(frequency=-0.02, presence=0.4)),
    (100_280, 300, dict(repetition=2.0 ** 50)), (100_280, 300, dict(repetition=2.0 ** -60)),
    (30_000, 16_000, dict(presence=-0.5)), (30_001, 16_000, dict(presence=-0.5)),
])
def test_rows_that_only_the_streaming_kernel_takes(context, vocab, history, wild):
    """A charge that shrinks with the count, an extreme repetition factor, a raising row with a history of half
    the vocabulary: those rows go through the streaming kernel, the others of a large batch through the
    ring kernel, a small batch whole."""
    for rows in (12, 15_500_000 // vocab):
        configs = some_raising(rows, rows // 9)
        configs[rows // 2] = SamplerConfig.make(temperature=0.9, top_p=0.9, top_k=30, **wild)
        configs[3] = SamplerConfig.make(0.0, 1.0, 1, **wild)
        w = random_workload(rows, vocab, history, configs, vocab + rows, uniform_history=False)
        assert_rows_equal(run_gpu(context, w), run_oracle(w), f"{rows} rows, {wild}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vocab", [3_001, 3_008, 32_001])
@pytest.mark.parametrize("history", [700, 8_192, 70_000])
@pytest.mark.parametrize("k,top_p", [(20, 0.9), (64, 1.0)])
def test_most_of_the_best_have_been_seen(context, dtype, vocab, history, k, top_p):
    """Uniform histories, up to many times the vocabulary, with a frequency penalty: much to count, by
    the kernel that is faster at it."""
    configs = [SamplerConfig.make(temperature=0.0 if r == 2 else 0.8, top_p=top_p, top_k=1 if r == 2 else k, presence=0.1 * r,
                                  frequency=0.02 + 0.1 * (r % 2), repetition=1.0 + 0.05 * (r % 3)) for r in range(5)]
    w = random_workload(5, vocab, history, configs, vocab + history + k, dtype=dtype)
    expected = run_oracle(w)
    for path in (0, 3):  # (3: the ring kernel wherever it can)
        context.set_path(path)
        try:
            assert_rows_equal(run_gpu(context, w), expected, f"V={vocab} H={history} path {path}")
        finally:
            context.set_path(0)


def test_unaligned_shards(context):
    """Two column ranges of unaligned rows, then the merge, against the whole rows."""
    rows, vocab, k = 11, 9_001, 24
    cfg = SamplerConfig.make(temperature=0.9, top_p=0.9, top_k=k, presence=0.3)
    w = random_workload(rows, vocab, 200, [cfg], 77)
    expected = run_oracle(w)
    d = w.to("cuda")
    scores = torch.empty(2, rows, k, device="cuda")
    ids = torch.empty(2, rows, k, dtype=torch.int32, device="cuda")
    first = [0, 4_503]
    width = [4_503, vocab - 4_503]
    for s in range(2):
        part = d.logits[:, first[s]:first[s] + width[s]]
        _, _, _, status = context.shard_topk(part, d.configs, first[s], vocab, k, d.history_tokens, d.history_offsets,
                                             d.history_max, out=(scores[s], ids[s]))
        assert status == FG_OK
    result = context.merge_select(scores, ids, rows, 2, k, first, width, d.configs, d.uniforms)
    assert np.array_equal(as_u32(result.tokens), expected[1])
