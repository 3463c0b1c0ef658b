"""The error words calls use in turn: whatever came before -- a failed call that nobody waited
for, a failed launch, a captured call and its replays -- a call that waits reports its own
rows' failure and nothing else."""
import pytest
import torch

from flash_gordon_b200 import FG_ERR_FORMAT, FG_OK, SamplerConfig

pytestmark = pytest.mark.gpu

ROWS, VOCAB = 4, 5000
CFG = [SamplerConfig.make(temperature=0.8, top_p=0.9, top_k=20)]


def logits(*bad_rows):
    x = torch.randn(ROWS, VOCAB, device="cuda")
    for r in bad_rows:
        x[r] = float("nan")
    return x


def sample(context, x, **kwargs):
    return context.sample_batch(x, CFG, torch.full((ROWS,), 0.5, device="cuda"), None, None, 0, **kwargs)


def test_a_waiting_call_reports_its_own_rows_only(context):
    good = logits()
    for bad_row in (3, 1, 2, 0):
        failed = sample(context, logits(bad_row))
        assert failed.status == FG_ERR_FORMAT and failed.message.startswith(f"row {bad_row}:")
        assert sample(context, good).status == FG_OK
        sample(context, logits(0), asynchronous=True)       # nobody asks about this one
        failed = sample(context, logits(bad_row))
        assert failed.status == FG_ERR_FORMAT and failed.message.startswith(f"row {bad_row}:")
        sample(context, logits(0), asynchronous=True)
        assert sample(context, good).status == FG_OK
    for _ in range(2):  # a call that is refused before any launch
        assert context.sample_batch(good, [SamplerConfig.make(top_k=65)], torch.rand(ROWS, device="cuda"), None, None,
                                    0).status != FG_OK
        assert sample(context, good).status == FG_OK


def test_captured_calls_keep_out_of_the_way(context):
    x, good = logits(), logits()
    out = (torch.empty(ROWS, dtype=torch.int32, device="cuda"), torch.empty(ROWS, device="cuda"),
           torch.empty(ROWS, dtype=torch.int32, device="cuda"))
    uniforms = torch.full((ROWS,), 0.5, device="cuda")
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        context.bind_torch_stream()
        context.prepared_sample(x, CFG, uniforms, None, None, 0, out)()
        step = context.prepared_sample(x, CFG, uniforms, None, None, 0, out)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            step()
        x[2] = float("nan")
        for _ in range(3):
            graph.replay()
            side.synchronize()
            assert out[2].tolist() == [0, 0, FG_ERR_FORMAT, 0]
            assert sample(context, good).status == FG_OK
            failed = sample(context, logits(3))
            assert failed.status == FG_ERR_FORMAT and failed.message.startswith("row 3:")
        x[2] = 0.0
        graph.replay()
        side.synchronize()
        assert out[2].tolist() == [0, 0, 0, 0]
    context.bind_torch_stream()
    assert sample(context, good).status == FG_OK


def test_router_reports_a_broken_token_once(context):
    tokens, experts, k = 9, 64, 4
    selected = torch.zeros(tokens, k, dtype=torch.int32, device="cuda")
    gates = torch.zeros(tokens, k, device="cuda")
    for broken in (None, 7, None, 2, None):
        x = torch.randn(tokens, experts, device="cuda")
        if broken is not None:
            x[broken, 5] = float("nan")
        status, message = context.router_topk(context.wrap(selected), context.wrap(gates), context.wrap(x), experts,
                                              tokens, k)
        assert status == (FG_OK if broken is None else FG_ERR_FORMAT)
        assert broken is None or f"token {broken}" in message
