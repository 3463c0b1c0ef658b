"""Rows without a top-k cut whose maximum, or whose bucket edges, are not where a sample of the
row's raw logits would put them."""
import numpy as np
import pytest
import torch

from flash_gordon_b200 import SamplerConfig, synth
from helpers import as_u32, assert_rows_equal, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


def with_history(logits, cfg, counts, uniforms):
    """One row's worth of workload: `counts` maps ids to how often they have been seen."""
    tokens = torch.tensor([i for i, n in counts.items() for _ in range(n)], dtype=torch.int32)
    rows = logits.shape[0]
    offsets = torch.arange(rows + 1, dtype=torch.int64) * len(tokens)
    return synth.Workload("window", logits, [cfg], torch.tensor(uniforms), tokens.repeat(rows), offsets, len(tokens),
                          allow_no_topk=True)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vocab", [4_096, 151_936])
def test_every_value_is_a_seen_one_pushed_far_down(context, vocab, dtype):
    """All logits are masked but two seen ids at -2, whose frequency charges take them to -44.9 and
    -46.85: the second one weighs 12 % and is drawn by u = 0.95."""
    logits = torch.full((3, vocab), float("-inf"), dtype=dtype)
    logits[:, [7, 1_001]] = -2.0
    cfg = SamplerConfig.make(temperature=1.0, top_p=1.0, top_k=0, frequency=1.95)
    w = with_history(logits, cfg, {7: 22, 1_001: 23}, [0.95, 0.5, 0.875])
    expected = run_oracle(w)
    assert list(expected[1]) == [1_001, 7, 7]
    assert_rows_equal(run_gpu(context, w), expected, f"V={vocab}")


@pytest.mark.parametrize("rows", [1, 40, 160])
def test_a_seen_raw_maximum_among_columns_without_another_value(context, rows):
    """The only values of the first columns are seen ids that the penalty takes out of the window;
    the row's own maximum is 25 below their raw logits and lies in other columns."""
    vocab = 151_936
    g = torch.Generator().manual_seed(11)
    logits = torch.full((rows, vocab), float("-inf"))
    sampled = torch.arange(2_048) * vocab // 2_048
    at = torch.randperm(vocab - 80_000, generator=g)[:400] + 80_000
    at = at[~torch.isin(at, sampled)]
    logits[:, at] = -25.0 - 3.0 * torch.rand(rows, len(at), generator=g)
    logits[:, 5] = -0.5
    cfg = SamplerConfig.make(temperature=1.0, top_p=0.999, top_k=0, frequency=1.9)
    w = with_history(logits, cfg, {5: 32}, torch.rand(rows, generator=g).tolist())
    assert_rows_equal(run_gpu(context, w), run_oracle(w), f"{rows} rows")


def test_three_ties_around_a_change_of_width(context):
    """1000 logits each of 5943/1024, 5942/1024 and 5941.75/1024, interleaved, under one of 9.3 that
    places the window so that the narrow buckets end at 5942/1024, in the middle of the last one."""
    vocab = 3_001
    logits = torch.empty(4, vocab)
    logits[:, 0] = 9.3
    for i, v in enumerate((5943.0, 5942.0, 5941.75)):
        logits[:, 1 + i::3] = v / 1024.0
    cfg = SamplerConfig.make(temperature=1.0, top_p=0.5, top_k=0)
    w = synth.Workload("ties", logits, [cfg], torch.tensor([0.9, 0.95, 0.97, 0.999]), None, None, 0, allow_no_topk=True)
    expected = run_oracle(w, want_candidates=True)
    assert min(c.edge_margin for c in expected[4]) > 1e-9
    for _ in range(5):
        assert_rows_equal(run_gpu(context, w), expected, "ties")


def rows_like(kind, rows, vocab, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(rows, vocab, generator=g)
    if kind == "peak":           # one token far above the body: a sample of the row finds it or not
        x[0::2, 0] = 13.3
        x[1::2, 5] = 13.3
    elif kind == "two peaks":    # ... and its neighbour in the sample
        x[:, 0] = 14.0
        x[:, vocab // 2] = 13.0
    elif kind == "far peak":
        x[:, 0] = 20.5
    elif kind == "hill":         # thousands of values above the body
        x[:, 7:2_007] = 12.0 + x[:, 7:2_007]
    elif kind == "offset":       # a head whose logits are not centred
        x = x * 1.5 - 4.0
        x[:, ::501] += 9.0
    return x


def sizes_and_tokens_agree(context, w, least_margin=1e-10):
    """Tokens, and the sizes of the nuclei, of the rows whose top_p and draw lie `least_margin` off
    every edge of the cumulative distribution."""
    expected = run_oracle(w, want_candidates=True)
    clear = np.array([c.edge_margin for c in expected[4]]) > least_margin
    assert clear.mean() > 0.5
    result = run_gpu(context, w, debug=True)
    sizes = np.array([c.nucleus for c in expected[4]])
    assert np.array_equal(as_u32(result.row_status), expected[3])
    assert np.array_equal(as_u32(result.tokens)[clear], expected[1][clear])
    assert np.array_equal(as_u32(result.debug["count"])[clear], sizes[clear])


@pytest.mark.parametrize("form", ["f32", "widened", "bf16"])
@pytest.mark.parametrize("kind", ["peak", "two peaks", "far peak", "hill", "offset"])
@pytest.mark.parametrize("rows,vocab,temperature,top_p", [
    (2, 151_936, 1.0, 0.9), (34, 100_277, 2.0, 0.9), (150, 20_001, 0.5, 0.8), (3, 151_936, 0.3, 0.999_9), (2, 60_000, 0.2, 0.99),
    (2, 151_936, 0.1, 0.95), (2, 60_000, 0.05, 0.9), (2, 60_000, 0.04, 0.9), (3, 100_277, 5.0, 0.9),
])
def test_windows_that_are_placed_anew(context, kind, form, rows, vocab, temperature, top_p):
    x = rows_like(kind, rows, vocab, rows + vocab)
    x = x.bfloat16() if form == "bf16" else x.bfloat16().float() if form == "widened" else x
    cfg = SamplerConfig.make(temperature=temperature, top_p=top_p, top_k=0)
    uniforms = torch.rand(rows, generator=torch.Generator().manual_seed(1))
    w = synth.Workload(kind, x, [cfg], uniforms, None, None, 0, allow_no_topk=True)
    sizes_and_tokens_agree(context, w)


@pytest.mark.parametrize("form", ["f32", "bf16"])
def test_what_lies_under_a_cold_row_s_window_is_not_forgotten(context, form):
    """The lower part of a body 20 below the top weighs 7e-6 of a row of 151,936, each of its values
    about 1e-9: that decides how many values top_p takes in.  (Masses on a grid of 2^-44, 8,192 of
    them: about 1.5e-12.)"""
    vocab = 151_936
    x = rows_like("far peak", 4, vocab, 3)
    x = x.bfloat16() if form == "bf16" else x
    configs = [SamplerConfig.make(temperature=0.2, top_p=1.0 - k * 2.0 ** -24, top_k=0) for k in (100, 1_000, 3_000, 5_000)]
    w = synth.Workload("under", x, configs, torch.tensor([0.1, 0.5, 0.9, 0.3]), None, None, 0, allow_no_topk=True)
    sizes_and_tokens_agree(context, w, 2e-11)


@pytest.mark.parametrize("rows", [1, 20, 60, 150])
@pytest.mark.parametrize("kind", ["narrow", "ties", "equal", "cold", "ties with history"])
def test_rows_of_the_long_way_shared_by_teams(context, kind, rows):
    """Buckets with more members than their words or the lists take, and temperatures below the range:
    every CTA of a team does its part of every step."""
    vocab = 140_001 if rows < 60 else 40_001
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, vocab, generator=g)
    temperature, top_p = 0.9, 0.7501
    if kind == "narrow":
        x *= 0.002
    elif kind == "equal":
        x[:, :] = 0.5
        x[:, ::3] = -0.25
    elif kind == "cold":
        temperature, top_p = 0.02, 0.9
    else:
        x = torch.round(x * 2.0) * 0.5 - 20.0
    x[:, 3] = float("nan")
    x[:, 77] = float("-inf")
    cfg = SamplerConfig.make(temperature=temperature, top_p=top_p, top_k=0,
                             presence=0.3 if "history" in kind else 0.0, frequency=0.1 if "history" in kind else 0.0)
    uniforms = torch.rand(rows, generator=g).tolist()
    if "history" in kind:
        w = with_history(x, cfg, {int(i): 1 + int(i) % 3 for i in torch.randperm(vocab, generator=g)[:900]}, uniforms)
    else:
        w = synth.Workload(kind, x, [cfg], torch.tensor(uniforms), None, None, 0, allow_no_topk=True)
    sizes_and_tokens_agree(context, w)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("temperature", [1.0, 0.2])
@pytest.mark.parametrize("offset", [0.0, -30.0])
def test_a_mask_s_value_in_every_sample(context, dtype, temperature, offset):
    """Sixty values left by a mask of the type's lowest value: the samples see nothing else."""
    vocab = 151_936
    g = torch.Generator().manual_seed(9)
    x = torch.full((4, vocab), torch.finfo(dtype).min, dtype=dtype)
    sampled = torch.arange(2_048) * vocab // 2_048
    at = torch.randperm(vocab, generator=g)[:60]
    at = at[~torch.isin(at, sampled)]
    x[:, at] = (torch.randn(4, len(at), generator=g) * 3.0 + offset).to(dtype)
    cfg = SamplerConfig.make(temperature=temperature, top_p=0.95, top_k=0)
    w = synth.Workload("masked", x, [cfg], torch.rand(4, generator=g), None, None, 0, allow_no_topk=True)
    sizes_and_tokens_agree(context, w)
