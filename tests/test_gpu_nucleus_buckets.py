"""Rows without a top-k cut where the value buckets, their window and the teams of CTAs can go
wrong: few and many rows (teams of eight down to one), ragged columns, logits far above or below
the sampled maximum, crowded buckets, temperatures on both sides of the short way's range, and
histories short and long, lowering and raising."""
import numpy as np
import pytest
import torch

from flash_gordon_b200 import SamplerConfig, synth
from helpers import as_u32, assert_rows_equal, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


def workload(rows, vocab, dtype, kind, temperature, top_p, history, penalties, seed):
    g = torch.Generator().manual_seed(seed)
    logits = torch.randn(rows, vocab, generator=g) * 2.0
    if kind == "spikes":       # a few values far above whatever a sample sees
        logits[:, ::997] += 9.0
    elif kind == "hill":       # thousands of them: the window is placed a second time
        logits[:, vocab // 3:vocab // 3 + min(1500, vocab // 8)] += 25.0
        logits[:, ::max(1, vocab // 2048)] = -3.0
    elif kind == "masked":     # a grammar's mask, finite and infinite
        keep = torch.rand(rows, vocab, generator=g) < 0.01
        logits[0::2][~keep[0::2]] = float("-inf")
        logits[1::2][~keep[1::2]] = torch.finfo(torch.float32).min
    elif kind == "crowded":    # values on a coarse grid: thousands of members in a bucket
        logits = torch.round(logits * 2.0) * 0.5 + 10.0
    elif kind == "wide":       # tails beyond the fine buckets and beyond the window
        logits *= 12.0
    elif kind == "shifted":
        logits += 3000.0
    elif kind == "beyond":     # magnitudes the buckets do not take
        logits *= 1e6
    if dtype == torch.bfloat16:
        logits = logits.to(torch.bfloat16)
    presence, frequency, repetition = penalties
    cfg = SamplerConfig.make(temperature=temperature, top_p=top_p, top_k=0, presence=presence, frequency=frequency,
                             repetition=repetition)
    tokens = offsets = None
    longest = 0
    if history:
        lengths = torch.randint(0, history + 1, (rows,), generator=g)
        lengths[0] = history
        offsets = torch.zeros(rows + 1, dtype=torch.int64)
        offsets[1:] = torch.cumsum(lengths, 0)
        tokens = torch.randint(0, vocab, (int(offsets[-1]),), generator=g, dtype=torch.int32)
        # the largest logits have been seen too
        best = logits.float().argmax(1).to(torch.int32)
        for r in range(rows):
            if lengths[r] > 0:
                tokens[offsets[r]:offsets[r] + min(3, int(lengths[r]))] = best[r]
        longest = history
    uniforms = torch.rand(rows, generator=g)
    return synth.Workload(kind, logits, [cfg], uniforms, tokens, offsets, longest, allow_no_topk=True)


PLAIN = (0.0, 0.0, 1.0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind,rows,vocab,temperature,top_p,history,penalties", [
    ("plain", 1, 151_936, 1.0, 0.95, 0, PLAIN),
    ("plain", 3, 100_277, 0.5, 0.9, 700, (0.5, 0.3, 1.1)),      # unaligned rows
    ("plain", 40, 32_001, 1.4, 0.999, 64, (-0.6, 0.0, 1.0)),    # raising
    ("plain", 150, 9_000, 0.8, 1.0, 3000, (0.0, -0.2, 0.8)),
    ("plain", 2, 20_000, 1.0, 0.9, 70_000, (0.2, 0.1, 1.0)),    # 32-bit counts
    ("plain", 2, 70, 1.0, 0.7, 10, (0.2, 0.1, 1.0)),            # CTAs without a column
    ("plain", 2, 300_001, 1.0, 0.95, 800, (0.2, 0.1, 1.0)),     # the coarser grid of masses
    ("plain", 2, 50_000, 0.36, 0.9, 0, PLAIN), ("plain", 2, 50_000, 0.35, 0.9, 0, PLAIN),
    ("plain", 2, 50_000, 0.18, 0.99, 90, (0.5, 0.1, 1.0)), ("plain", 2, 50_000, 0.17, 0.9, 0, PLAIN),
    ("plain", 2, 50_000, 2.6, 0.9, 0, PLAIN), ("plain", 2, 50_000, 2.7, 0.9, 40, (0.5, 0.1, 1.0)),
    ("spikes", 5, 60_000, 1.0, 0.9, 300, (1.9, 0.0, 1.0)),
    ("hill", 4, 50_000, 1.0, 0.99, 0, PLAIN), ("hill", 4, 50_000, 0.9, 0.99, 200, (1.9, 1.9, 1.0)),
    ("masked", 4, 50_000, 1.0, 0.95, 100, (0.5, 0.5, 1.0)), ("masked", 4, 50_000, 1.0, 0.95, 0, PLAIN),
    ("crowded", 3, 60_000, 1.0, 0.8, 0, PLAIN), ("crowded", 3, 60_000, 0.7, 0.8, 500, (0.3, 0.1, 1.0)),
    ("wide", 4, 60_000, 1.2, 0.9999, 0, PLAIN), ("wide", 4, 60_000, 1.2, 1.0, 900, (0.3, 0.7, 1.3)),
    ("shifted", 3, 30_000, 1.0, 0.9, 50, (0.3, 0.1, 1.0)), ("beyond", 3, 30_000, 1.0, 0.9, 50, (0.3, 0.1, 1.0)),
])
def test_buckets(context, dtype, kind, rows, vocab, temperature, top_p, history, penalties):
    w = workload(rows, vocab, dtype, kind, temperature, top_p, history, penalties, 7 * rows + vocab)
    expected = run_oracle(w, want_candidates=True)
    # (a value on the coarse grid ties with thousands: an edge may coincide with top_p.  The masses are
    # off by up to 6e-11 of their total.)
    margins = np.array([c.edge_margin for c in expected[4]])
    clear = margins > 1e-10
    result = run_gpu(context, w, debug=True)
    got = as_u32(result.tokens)
    assert np.array_equal(as_u32(result.row_status), expected[3])
    assert np.array_equal(got[clear], expected[1][clear]), (kind, got, expected[1], margins)
    if clear.all():
        assert_rows_equal(result, expected, kind)


def test_rows_of_a_mixed_batch_are_shared_out_evenly(context):
    """Every third row is one without a top-k cut; the teams take those in turn."""
    rows, vocab = 101, 12_345
    g = torch.Generator().manual_seed(3)
    configs = [SamplerConfig.make(temperature=0.9, top_p=0.9, top_k=0 if r % 3 == 1 else 20, presence=0.4 * (r % 2))
               for r in range(rows)]
    offsets = torch.arange(rows + 1, dtype=torch.int64) * 50
    tokens = torch.randint(0, vocab, (rows * 50,), generator=g, dtype=torch.int32)
    w = synth.Workload("mixed", torch.randn(rows, vocab, generator=g) * 2.0, configs, torch.rand(rows, generator=g),
                       tokens, offsets, 50, allow_no_topk=True)
    assert_rows_equal(run_gpu(context, w), run_oracle(w), "mixed")
