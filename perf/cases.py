"""The sampling calls whose speed matters, through the package's public entry points.

A case is one call (or the pair of calls of the sharded mode) as a serving program issues it
once per decode step: rows of vocabulary logits in, token ids out.  Shapes and distributions are
those of `flash_gordon_b200.synth`, of the tests and of the operators beside the sampler, plus
generic ones: small batches, ragged histories, vocabularies that are no multiple of a vector.
`listed()` are fixed points of those ranges, `draw()` gives others.

Kinds of cases:
  topk      Context.prepared_sample / sample_batch: greedy or top-k + top-p rows, one config
  nucleus   the same without a top-k cut (top-p over the whole vocabulary)
  mixed     one batch whose rows carry their own configs: greedy, top-k with and without
            penalties (also ones that raise a logit), and rows without a top-k cut
  sessions  OutputExecutor.sample_sessions: histories kept on the GPU from step to step
  shard     Context.shard_topk on this GPU's columns, then Context.merge_select over the
            gathered candidates of all shards
  host      Context.sample_batch_host: every buffer in pinned host memory
  router    Context.router_topk: expert choice per token
  select    flash_gordon_b200.api.select: the C sampler's last step on host lists
"""
from __future__ import annotations

import math

import numpy as np
import torch

from flash_gordon_b200 import Context, SamplerConfig
from flash_gordon_b200 import api, synth

VOCAB = synth.VOCAB
DEVICE = "cuda"
MOST_LOGITS = 1024 * VOCAB          # the largest top-k batch
MOST_NUCLEUS_LOGITS = 512 * VOCAB   # the largest batch without a top-k cut


def listed():
    return [
        # the C sampler's own last step: one request at a time, candidates on the host
        dict(name="select_64", kind="select", count=64, temperature=0.7, top_k=20, top_p=0.8),
        # one user, greedy, token needed at once (the waiting form of the call)
        dict(name="greedy_1_f32", kind="topk", rows=1, vocab=VOCAB, dtype="f32", spread=3.0, gumbel=False,
             history=64, ragged=False, zipf=0.0, temperature=0.0, top_k=1, top_p=1.0, presence=0.0,
             frequency=0.0, repetition=1.1, wait=True),
        # a handful of chats on one GPU, bf16 head, short ragged histories
        dict(name="chat_8_bf16", kind="topk", rows=8, vocab=VOCAB, dtype="bf16", spread=3.0, gumbel=False,
             history=1000, ragged=True, zipf=1.1, temperature=0.7, top_k=20, top_p=0.8, presence=1.5,
             frequency=0.0, repetition=1.0, wait=False),
        # the usual decode batch
        dict(name="decode_64_f32", kind="topk", rows=64, vocab=VOCAB, dtype="f32", spread=3.0, gumbel=False,
             history=512, ragged=False, zipf=1.1, temperature=0.7, top_k=20, top_p=0.8, presence=1.5,
             frequency=0.0, repetition=1.0, wait=False),
        # the throughput batch: long histories, two penalties, a wide top-k
        dict(name="decode_1024_f32", kind="topk", rows=1024, vocab=VOCAB, dtype="f32", spread=2.0, gumbel=True,
             history=4096, ragged=False, zipf=1.0, temperature=1.0, top_k=50, top_p=0.95, presence=0.0,
             frequency=0.5, repetition=1.05, wait=False),
        # continuous batching: every request brings its own settings, the vocabulary is odd
        dict(name="mixed_200_bf16_odd", kind="mixed", rows=200, vocab=100_277, dtype="bf16", spread=2.5,
             gumbel=False, history=1500, ragged=True, zipf=1.1),
        # requests that ask for top-p alone, peaked distributions
        dict(name="top_p_32_bf16", kind="nucleus", rows=32, vocab=VOCAB, dtype="bf16", spread=2.0, gumbel=True,
             history=0, ragged=False, zipf=0.0, temperature=1.0, top_k=0, top_p=0.95, presence=0.0,
             frequency=0.0, repetition=1.0, wait=False),
        # the worst case of top-p alone: nearly flat, nuclei of tens of thousands of tokens
        dict(name="top_p_512_f32_flat", kind="nucleus", rows=512, vocab=VOCAB, dtype="f32", spread=0.5,
             gumbel=False, history=32768, ragged=False, zipf=0.0, temperature=1.2, top_k=0, top_p=0.99,
             presence=0.5, frequency=0.5, repetition=1.0, wait=False),
        # one rank's work of the vocabulary-sharded mode on eight GPUs
        dict(name="shard_256_bf16", kind="shard", rows=256, width=VOCAB // 8, shards=8, dtype="bf16", spread=4.0,
             temperature=0.8, top_k=64, top_p=0.9),
        # a decode step of the stateful executor
        dict(name="sessions_96_f32", kind="sessions", rows=96, vocab=VOCAB, dtype="f32", spread=3.0, history=700,
             temperature=0.8, top_k=40, top_p=0.9, presence=0.3, frequency=0.4, repetition=1.0),
        # logits that were computed elsewhere: host buffers in, host buffers out
        dict(name="host_16_f32", kind="host", rows=16, vocab=VOCAB, dtype="f32", spread=3.0, gumbel=False,
             history=512, ragged=False, zipf=1.1, temperature=0.7, top_k=20, top_p=0.8, presence=1.5,
             frequency=0.0, repetition=1.0),
        # expert choice of a prefill chunk
        dict(name="router_4096", kind="router", tokens=4096, experts=512, k=10, spread=1.5),
    ]


# ------------------------------------------------------------------------ drawn cases

def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _vocab(rng):
    """32 K to 200 K logits; two in three a multiple of 64 (padded heads), the others odd sizes."""
    v = _log_int(rng, 32_000, 200_000)
    return v | 1 if rng.random() < 1 / 3 else v // 64 * 64


def _rows(rng, vocab, most_logits):
    return _log_int(rng, 1, max(1, min(1024, most_logits // vocab)))


def draw(rng):
    kind = rng.choice(["topk"] * 4 + ["nucleus"] * 2 + ["mixed", "shard", "sessions", "host", "router", "select"])
    dtype = rng.choice(["f32", "bf16"])
    spread = round(rng.uniform(1.0, 4.0), 3)
    temperature, top_p = round(rng.uniform(0.5, 1.4), 3), round(rng.uniform(0.7, 1.0), 4)
    if kind == "select":
        return dict(kind=kind, count=rng.randint(1, 64), temperature=temperature, top_k=rng.randint(1, 64), top_p=top_p)
    if kind == "router":
        experts = rng.choice([64, 128, 256, 384, 512])
        return dict(kind=kind, tokens=_log_int(rng, 1, 4096), experts=experts, k=rng.randint(1, 10), spread=spread)
    if kind == "shard":
        shards, k = rng.choice([2, 4, 8]), rng.randint(8, 64)
        width = _log_int(rng, 8_000, 76_000) // 8 * 8 + rng.choice([0, 0, 1])
        return dict(kind=kind, rows=_log_int(rng, 1, 512), width=width, shards=shards, dtype=dtype, spread=spread,
                    temperature=temperature, top_k=k, top_p=top_p)
    vocab = _vocab(rng)
    if kind == "sessions":
        return dict(kind=kind, rows=_log_int(rng, 1, 256), vocab=vocab, dtype=dtype, spread=spread,
                    history=_log_int(rng, 16, 4096), temperature=temperature, top_k=rng.randint(1, 64), top_p=top_p,
                    presence=round(rng.uniform(0.0, 1.5), 2), frequency=round(rng.uniform(0.05, 1.0), 2),
                    repetition=1.0)
    history, ragged, zipf = rng.choice([0, _log_int(rng, 16, 8192), _log_int(rng, 16, 8192)]), rng.random() < 0.5, \
        rng.choice([0.0, 1.0, 1.1])
    case = dict(kind=kind, rows=1, vocab=vocab, dtype=dtype, spread=spread, gumbel=rng.random() < 0.4, history=history,
                ragged=ragged, zipf=zipf)
    if kind == "mixed":
        case["rows"] = max(8, _rows(rng, vocab, MOST_LOGITS // 4))
        case["history"] = max(16, history // 4)
        return case
    penalties = rng.choice(["presence", "frequency", "repetition", "all"]) if history else ""
    case.update(temperature=temperature, top_k=rng.randint(1, 64), top_p=top_p,
                presence=round(rng.uniform(0.1, 1.5), 2) if penalties in ("presence", "all") else 0.0,
                frequency=round(rng.uniform(0.1, 1.0), 2) if penalties in ("frequency", "all") else 0.0,
                repetition=round(rng.uniform(1.02, 1.3), 3) if penalties in ("repetition", "all") else 1.0)
    if kind == "host":
        case["rows"] = _log_int(rng, 1, 32)
        return case
    case["wait"] = rng.random() < 0.3
    if kind == "nucleus":
        case.update(rows=_rows(rng, vocab, MOST_NUCLEUS_LOGITS), top_k=0, spread=round(rng.uniform(0.5, 4.0), 3))
        return case
    case["rows"] = _rows(rng, vocab, MOST_LOGITS)
    if rng.random() < 0.25:
        case.update(temperature=0.0, top_k=1, top_p=1.0)
    return case


# ------------------------------------------------------------------------ inputs

_contexts = {}


def _context():
    """One context per process, as a serving program keeps one per GPU."""
    if DEVICE not in _contexts:
        _contexts[DEVICE] = Context()
    return _contexts[DEVICE]


def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.float32


def _logits(case, rows, columns, g):
    x = torch.randn(rows, columns, generator=g, device=DEVICE) * case["spread"]
    if case.get("gumbel"):
        u = torch.rand(rows, columns, generator=g, device=DEVICE).clamp_(1e-20, 1.0)
        x -= torch.log(-torch.log(u))
    return x.to(_dtype(case))


def _token_ids(count, vocab, zipf, g):
    """`count` ids, uniform (zipf 0) or Zipf-distributed with the popular ids spread out."""
    if zipf == 0.0:
        return torch.randint(0, vocab, (count,), generator=g, device=DEVICE, dtype=torch.int32)
    weights = np.arange(1, vocab + 1, dtype=np.float64) ** -zipf
    edges = torch.from_numpy(np.cumsum(weights) / weights.sum()).to(DEVICE)
    u = torch.rand(count, generator=g, device=DEVICE, dtype=torch.float64)
    ranks = torch.searchsorted(edges, u).clamp_(max=vocab - 1)
    return torch.randperm(vocab, generator=g, device=DEVICE)[ranks].to(torch.int32)


def _history(case, rows, g):
    """(tokens, offsets, longest) in the call's CSR form, or Nones."""
    most = case["history"]
    if most == 0:
        return None, None, 0
    if case["ragged"]:
        lengths = torch.randint(most // 4, most + 1, (rows,), generator=g, device=DEVICE)
    else:
        lengths = torch.full((rows,), most, device=DEVICE)
    offsets = torch.zeros(rows + 1, dtype=torch.int64, device=DEVICE)
    offsets[1:] = torch.cumsum(lengths, 0)
    return _token_ids(int(offsets[-1]), case["vocab"], case["zipf"], g), offsets, int(lengths.max())


def _config(case):
    return SamplerConfig.make(temperature=case["temperature"], top_p=case["top_p"], top_k=case["top_k"],
                              presence=case.get("presence", 0.0), frequency=case.get("frequency", 0.0),
                              repetition=case.get("repetition", 1.0))


def _mixed_configs(rows, seed):
    """What requests ask for: mostly top-k + top-p, some greedy, some top-p alone; penalties on
    half of them, now and then a negative presence penalty."""
    rng = np.random.RandomState(seed & 0x7fffffff)
    configs = []
    for r in range(rows):
        form = r % 8
        presence, frequency, repetition = 0.0, 0.0, 1.0
        if form in (1, 3, 4, 6):
            presence, frequency = float(rng.choice([0.2, 0.6, 1.0, -0.4])), float(rng.choice([0.0, 0.3]))
            repetition = float(rng.choice([1.0, 1.05, 1.1]))
        if form in (0, 1):
            cfg = SamplerConfig.make(temperature=0.0, top_p=1.0, top_k=1, presence=presence, frequency=frequency,
                                     repetition=repetition)
        else:
            cfg = SamplerConfig.make(temperature=float(rng.choice([0.6, 0.8, 1.0])),
                                     top_p=float(rng.choice([0.8, 0.9, 0.95])),
                                     top_k=0 if form == 2 else int(rng.choice([20, 40, 50, 64])), presence=presence,
                                     frequency=frequency, repetition=repetition)
        configs.append(cfg)
    return configs


def _outputs(rows, device):
    return (torch.empty(rows, dtype=torch.int32, device=device), torch.empty(rows, dtype=torch.float32, device=device),
            torch.empty(rows, dtype=torch.int32, device=device))


def prepare(case, seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    kind = case["kind"]
    state = {"case": case}
    if kind == "select":
        rng = np.random.RandomState(seed & 0x7fffffff)
        state.update(config=_config(case), scores=(rng.randn(case["count"]) * 3.0).astype(np.float32).tolist(),
                     ids=rng.permutation(VOCAB)[:case["count"]].tolist(), uniform=float(rng.rand()))
        return state
    context = _context()
    state["context"] = context
    if kind == "router":
        tokens, experts, k = case["tokens"], case["experts"], case["k"]
        logits = torch.randn(tokens, experts, generator=g, device=DEVICE) * case["spread"]
        selected = torch.zeros(tokens, k, dtype=torch.int32, device=DEVICE)
        gates = torch.zeros(tokens, k, device=DEVICE)
        state.update(selected=selected, gates=gates,
                     handles=(context.wrap(selected), context.wrap(gates), context.wrap(logits)))
        return state
    rows = case["rows"]
    uniforms = torch.rand(rows, generator=g, device=DEVICE)
    if kind == "shard":
        width, shards, k = case["width"], case["shards"], case["top_k"]
        scores = torch.empty(shards, rows, k, device=DEVICE)
        ids = torch.empty(shards, rows, k, dtype=torch.int32, device=DEVICE)
        for s in range(1, shards):  # what the other ranks send
            best, where = torch.topk(_logits(case, rows, width, g).float(), k, dim=1)
            scores[s], ids[s] = best, (where + s * width).to(torch.int32)
        state.update(logits=_logits(case, rows, width, g), config=_config(case), uniforms=uniforms, scores=scores,
                     ids=ids, firsts=[s * width for s in range(shards)], widths=[width] * shards)
        return state
    vocab = case["vocab"]
    logits = _logits(case, rows, vocab, g)
    if kind == "sessions":
        executor = api.OutputExecutor(context, vocab, rows, case["history"] + 1024)
        tokens = _token_ids(rows * case["history"], vocab, 1.0, g).cpu().numpy().reshape(rows, -1)
        for slot in range(rows):
            executor.set_session(slot)
            if executor.history_reset(tokens[slot].tolist()) != 0:
                raise RuntimeError("the session's history was refused")
        slots = torch.randperm(rows, generator=g, device=DEVICE).tolist()
        state.update(executor=executor, logits=logits, uniforms=uniforms, config=_config(case), slots=slots)
        return state
    tokens, offsets, longest = _history(case, rows, g)
    if kind == "host":
        pinned = lambda t: None if t is None else t.cpu().pin_memory()  # noqa: E731
        out = tuple(t.pin_memory() for t in _outputs(rows, "cpu"))
        state.update(logits=pinned(logits), config=_config(case), uniforms=pinned(uniforms), tokens=pinned(tokens),
                     offsets=pinned(offsets), longest=longest, out=out)
        return state
    configs = _mixed_configs(rows, seed) if kind == "mixed" else [_config(case)]
    out = _outputs(rows, DEVICE)
    state.update(logits=logits, configs=configs, uniforms=uniforms, tokens=tokens, offsets=offsets, longest=longest,
                 out=out)
    if not case.get("wait"):
        state["step"] = context.prepared_sample(logits, configs, uniforms, tokens, offsets, longest, out,
                                                allow_no_topk=kind != "topk")
    return state


# ------------------------------------------------------------------------ one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "select":
        status, token, logit, _ = api.select(state["config"], state["scores"], state["ids"], state["uniform"])
        return status, token, logit
    context = state["context"]
    if kind == "router":
        selected, gates, logits = state["handles"]
        status, _ = context.router_topk(selected, gates, logits, case["experts"], case["tokens"], case["k"])
        return status, state["selected"], state["gates"]
    if kind == "shard":
        _, _, shard_status, _ = context.shard_topk(
            state["logits"], state["config"], 0, case["width"] * case["shards"], case["top_k"],
            out=(state["scores"][0], state["ids"][0]), asynchronous=True)
        result = context.merge_select(state["scores"], state["ids"], case["rows"], case["shards"], case["top_k"],
                                      state["firsts"], state["widths"], state["config"], state["uniforms"],
                                      asynchronous=True)
        return state["scores"][0], state["ids"][0], shard_status, result.tokens, result.token_logits, result.row_status
    if kind == "sessions":
        result = state["executor"].sample_sessions(state["logits"], state["config"], state["uniforms"], state["slots"])
        return result.status, result.tokens, result.token_logits, result.row_status
    if kind == "host":
        result = context.sample_batch_host(state["logits"], state["config"], state["uniforms"], state["tokens"],
                                           state["offsets"], state["longest"], out=state["out"])
        return result.status, result.tokens, result.token_logits, result.row_status
    if case.get("wait"):
        result = context.sample_batch(state["logits"], state["configs"], state["uniforms"], state["tokens"],
                                      state["offsets"], state["longest"], allow_no_topk=kind == "nucleus")
        return result.status, result.tokens, result.token_logits, result.row_status
    state["step"]()
    return state["out"]


def work(case):
    """Logits once, every history token once, a draw and a result per row; selection is comparisons."""
    kind = case["kind"]
    if kind == "select":
        return {"bytes": case["count"] * 8 + 12, "flops": 0}
    if kind == "router":
        return {"bytes": case["tokens"] * (case["experts"] * 4 + case["k"] * 8), "flops": 0}
    rows, element = case["rows"], 2 if case["dtype"] == "bf16" else 4
    if kind == "shard":
        candidates = rows * case["top_k"] * 8
        return {"bytes": rows * (case["width"] * element + 20) + candidates * (case["shards"] + 1), "flops": 0}
    history = 0 if kind == "sessions" else case["history"] * 4  # a session's tables stay on the GPU
    if case.get("ragged"):
        history = history * 5 // 8
    return {"bytes": rows * (case["vocab"] * element + history + 16), "flops": 0}


def tolerance(case):
    """Token ids, statuses and the picked logits are exact: the same fp32 operations in the same
    order, sums of weights in fp64 (or finer than its steps).  Gate weights are fp64 quotients
    rounded to fp32 twice: against a 64-bit softmax they differ by 6e-8 at most."""
    if case["kind"] == "router":
        return {"rel": 2.5e-7, "max": 5e-7}
    return "exact"
