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
