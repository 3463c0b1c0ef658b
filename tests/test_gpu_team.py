"""The team kernel (rows shared by clusters of CTAs) against the oracle, at the sizes where it can
go wrong: tiles and chunks that end anywhere, lists that overflow, seen ids to be counted, penalties
that raise a logit, session tables, broken histories, shards, a wait that runs out."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from flash_gordon_b200 import FG_ERR_FORMAT, FG_ERR_LIMIT, FG_OK, SamplerConfig, synth
from flash_gordon_b200.api import OutputExecutor
from helpers import (as_u32, assert_candidates_close, assert_rows_equal, random_workload, run_gpu,
                     run_oracle)

pytestmark = pytest.mark.gpu

PROBABILITY_RTOL = 1e-5  # probabilities: fp64 on both sides, exp() from different libraries


@pytest.fixture(params=[(1, 0), (2, 0), (4, 0), (8, 0), (8, 2), (4, 1)], ids=str)
def team(context, request):
    context.team_controls(*request.param)
    yield request.param[0]
    context.team_controls()


def check(context, w, label):
    expected = run_oracle(w, want_candidates=True)
    assert_rows_equal(run_gpu(context, w), expected, label)
    result = run_gpu(context, w, debug=True)
    assert_rows_equal(result, expected, label)
    assert_candidates_close(result, expected, PROBABILITY_RTOL, label)


CONFIGS = {
    "lowering": dict(temperature=0.9, top_p=0.9, presence=0.7, frequency=0.3, repetition=1.3),
    "raising": dict(temperature=0.8, top_p=0.95, presence=-0.9, frequency=0.1, repetition=0.8),
    "raised by presence alone": dict(temperature=0.8, top_p=0.95, presence=-0.4),
}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vocab", [1, 9, 257, 4_095, 4_097, 16_384, 16_390, 33_001, 151_936, 200_003])
def test_sizes(context, team, vocab, dtype):
    for i, (k, history, rows) in enumerate([(1, 0, 1), (20, 64, 3), (64, 4097, 2)]):
        for name, penalties in CONFIGS.items():
            cfg = SamplerConfig.make(top_k=k, **penalties)
            w = random_workload(rows, vocab, history, [cfg], 31 * vocab + i, quantize=0.0 if i == 1 else 0.5,
                                specials=min(3, vocab), dtype=dtype, stride=vocab + i)
            check(context, w, f"V={vocab} k={k} H={history} team={team} {name}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_greedy_rows(context, team, dtype):
    """NaN, infinities, values a penalty turns into one, and ordinary rows."""
    rows, vocab = 10, 30_007
    for penalties in (dict(), dict(repetition=1.2, frequency=0.4), dict(presence=-1.0, repetition=2.0 ** -30),
                      dict(repetition=2.0 ** 39)):
        w = random_workload(rows, vocab, 300, [SamplerConfig.make(0.0, 1.0, 1, **penalties)], 5, dtype=dtype)
        for r in range(3):
            w.logits[r, 17 * r + 5] = (float("nan"), float("-inf"), float("inf"))[r]
        for r in range(3, 7):  # seen huge values: the penalty may make an infinity of them
            w.logits[r, int(w.history_tokens[int(w.history_offsets[r])]) if w.history_offsets[r + 1] > w.history_offsets[r]
                     else 0] = (-3e38, 3e38, -1e30, 1e30)[r - 3]
        check(context, w, f"greedy {penalties}")


def test_worst_cases(context, team):
    """Every value ties, every later one is larger, every earlier one, and most of the best seen."""
    vocab = 120_000
    flat = torch.full((1, vocab), 1.0)
    rising = torch.arange(vocab, dtype=torch.float32).reshape(1, vocab) * 0.001
    logits = torch.cat([flat, rising, rising.flip(1)], 0)
    best = torch.arange(vocab - 1500, vocab, dtype=torch.int32)
    tokens = torch.cat([best, best[::2], torch.arange(700, dtype=torch.int32), best])
    offsets = torch.tensor([0, 1500, 2950, tokens.numel()])
    for penalties in (dict(), dict(presence=0.2, frequency=0.3), dict(presence=-0.3, frequency=0.01)):
        w = synth.Workload("edges", logits, [SamplerConfig.make(1.0, 1.0, 64, **penalties)],
                           torch.tensor([0.0, 0.5, 0.999]), tokens, offsets, 2000 + 1500)
        check(context, w, f"edges {penalties}")
        check(context, synth.Workload("edges", logits.bfloat16(), w.configs, w.uniforms, tokens, offsets, 3500), "bf16")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vocab", [1_984, 4_099, 33_000])
def test_most_of_the_vocabulary_has_been_seen(context, team, vocab, dtype):
    for k, penalties in ((50, CONFIGS["lowering"]), (64, CONFIGS["raising"]), (30, dict(temperature=0.8, top_p=0.9, repetition=0.9))):
        w = random_workload(6, vocab, 3 * vocab, [SamplerConfig.make(top_k=k, **penalties)], vocab + k, dtype=dtype)
        check(context, w, f"V={vocab} k={k} team={team}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vocab", [4_099, 33_000, 151_936])
@pytest.mark.parametrize("fill", ["-inf", "lowest", "one"])
def test_most_of_a_row_is_one_value(context, team, vocab, dtype, fill):
    """Rows under a mask, and rows of equal logits: next to nothing, fewer than k, or more than k logits stand out, and
    with a mask of finite values or none the ties are won by the smallest ids."""
    value = {"-inf": float("-inf"), "lowest": torch.finfo(dtype).min, "one": 1.0}[fill]
    for i, penalties in enumerate((dict(temperature=0.9, top_p=0.9), CONFIGS["lowering"], CONFIGS["raising"],
                                   dict(temperature=0.0, top_p=1.0, frequency=0.3, presence=-0.5),
                                   dict(temperature=0.0, top_p=1.0, repetition=1.2))):
        k = 1 if penalties["temperature"] == 0.0 else 50
        w = random_workload(4, vocab, 200, [SamplerConfig.make(top_k=k, **penalties)], vocab + i, dtype=dtype)
        allowed = torch.zeros(w.logits.shape, dtype=torch.bool)
        for r, few in enumerate((1, 30, 2000, 300)):
            where = torch.randint(0, vocab, (few,), generator=torch.Generator().manual_seed(r))
            allowed[r, where if r < 3 else torch.arange(vocab // 3, vocab // 3 + few)] = True
        w.logits = torch.where(allowed, w.logits, torch.full_like(w.logits, value))
        check(context, w, f"{fill} V={vocab} team={team} {penalties}")


def test_mixed_settings_in_one_batch(context, team):
    """Every row its own settings; rows without a top-k cut are left to their kernel."""
    rows, vocab = 40, 20_011
    configs = []
    for r in range(rows):
        penalties = list(CONFIGS.values())[r % 3] if r % 2 else dict(temperature=0.7, top_p=0.8)
        penalties = dict(penalties, temperature=0.0 if r % 5 == 0 else penalties["temperature"])
        configs.append(SamplerConfig.make(top_k=0 if r % 7 == 3 else 1 if r % 5 == 0 else 5 + r, **penalties))
    w = random_workload(rows, vocab, 500, configs, 99, dtype=torch.bfloat16)
    w.allow_no_topk = True
    assert_rows_equal(run_gpu(context, w), run_oracle(w), f"mixed, team={team}")


def test_broken_histories(context, team):
    rows, vocab = 4, 40_000
    cfg = SamplerConfig.make(0.9, 0.9, 20, presence=0.4, frequency=0.1)
    w = random_workload(rows, vocab, 100, [cfg], 7)
    d = w.to("cuda")
    tokens = d.history_tokens.clone()
    tokens[0] = vocab
    result = context.sample_batch(d.logits, d.configs, d.uniforms, tokens, d.history_offsets, 100)
    assert as_u32(result.row_status).tolist() == [FG_ERR_FORMAT, FG_OK, FG_OK, FG_OK]
    result = context.sample_batch(d.logits, d.configs, d.uniforms, d.history_tokens, d.history_offsets, 99)
    assert as_u32(result.row_status)[0] == FG_ERR_LIMIT and result.status == FG_ERR_LIMIT
    assert_rows_equal(run_gpu(context, w), run_oracle(w), "afterwards")


def test_shards(context, team):
    """Two column ranges, one of them unaligned, then the merge, against the whole rows."""
    rows, vocab, k = 11, 60_001, 24
    for cfg in (SamplerConfig.make(temperature=0.9, top_p=0.9, top_k=k, presence=0.3, frequency=0.2),
                SamplerConfig.make(0.0, 1.0, 1, presence=-0.5)):
        w = random_workload(rows, vocab, 2000, [cfg], 77)
        expected = run_oracle(w)
        d = w.to("cuda")
        scores = torch.empty(2, rows, k, device="cuda")
        ids = torch.empty(2, rows, k, dtype=torch.int32, device="cuda")
        first, width = [0, 30_503], [30_503, vocab - 30_503]
        for s in range(2):
            part = d.logits[:, first[s]:first[s] + width[s]]
            _, _, _, status = context.shard_topk(part, d.configs, first[s], vocab, k, d.history_tokens, d.history_offsets,
                                                 d.history_max, out=(scores[s], ids[s]))
            assert status == FG_OK
        result = context.merge_select(scores, ids, rows, 2, k, first, width, d.configs, d.uniforms)
        assert np.array_equal(as_u32(result.tokens), expected[1])


def test_session_tables(context, team):
    rows, vocab = 6, 50_016
    cfg = SamplerConfig.make(0.8, 0.9, 40, presence=0.3, frequency=0.4, repetition=1.1)
    w = random_workload(rows, vocab, 900, [cfg], 13)
    executor = OutputExecutor(context, vocab, rows, 2000)
    for r in range(rows):
        executor.set_session(r)
        assert executor.history_reset(w.history_tokens[w.history_offsets[r]:w.history_offsets[r + 1]].tolist()) == FG_OK
    d = w.to("cuda")
    result = executor.sample_sessions(d.logits, cfg, d.uniforms, list(range(rows)))
    assert_rows_equal(result, run_oracle(w), f"tables, team={team}")


@pytest.mark.parametrize("issue", [0, 3])
def test_a_wait_that_runs_out(context, team, issue):
    """A request that is never made: the row fails with FG_ERR_LIMIT, the others do not, and the next
    call works."""
    rows, vocab = 3, 8 * 16_000
    w = random_workload(rows, vocab, 200, [SamplerConfig.make(0.9, 0.9, 20, presence=0.4, frequency=0.1)], 17)
    context.ring_controls(wait_polls=3000, withhold=(team, issue if team < 4 else 0))  # the second row's first CTA
    try:
        result = run_gpu(context, w)
        assert result.status == FG_ERR_LIMIT and "wait ran out" in result.message
        assert as_u32(result.row_status).tolist() == [FG_OK, FG_ERR_LIMIT, FG_OK]
    finally:
        context.ring_controls()
    assert_rows_equal(run_gpu(context, w), run_oracle(w), "afterwards")


@pytest.mark.parametrize("count", [2, 3, 31, 32, 33, 64])
def test_edges_that_are_met_exactly(context, team, count):
    """Equal weights: cumulative sums that meet top_p and the draw exactly, or to a rounding."""
    vocab, draws = 5_000, [i / 32 for i in range(32)] + [0.1, 1 / 3, 0.7, 0.999999]
    logits = torch.full((len(draws), vocab), -5.0)
    logits[:, 7:7 + count] = 2.0
    for top_p in (0.25, 0.5, 1.0, float(np.float32(1 / 3)), 0.7):
        cfg = SamplerConfig.make(0.5, top_p, count)
        w = synth.Workload("exact", logits, [cfg], torch.tensor(draws), None, None, 0)
        assert_rows_equal(run_gpu(context, w), run_oracle(w), f"{count} equal weights, top_p {top_p}")


@pytest.mark.parametrize("gap", [20.0, 29.0, 29.93, 31.0, 36.0, 40.0, 800.0])
def test_sums_that_stand_still(context, gap):
    """All candidates are asked for, and the last ones weigh so little that the sum reaches top_p before them, or
    not at all."""
    vocab, draws = 3_000, [0.0, 0.3, 0.999999]
    logits = torch.full((len(draws), vocab), -900.0)
    logits[:, 5:10] = torch.tensor([0.0, -0.5, -gap, -gap - 0.25, -gap - 7.0])
    for k in (3, 4, 5, 40):
        for top_p in (1.0, float(np.nextafter(np.float32(1.0), np.float32(0.0)))):
            w = synth.Workload("tails", logits, [SamplerConfig.make(1.0, top_p, k)], torch.tensor(draws), None, None, 0)
            assert_rows_equal(run_gpu(context, w), run_oracle(w), f"gap {gap}, top_p {top_p}, k {k}")
