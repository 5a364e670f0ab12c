"""Workloads that time this engine through its public entry points.

Every case is a whole call as a program makes it: a request of ``Decoder.generate_ids`` (prompt in, tokens out),
the same with tokens pulled one at a time through ``Decoder.step``, a prompt through ``Decoder.prefill_ids``, a batch of
``BatchDecoder.generate_ids``, a job of ``ContinuousBatcher``.  The model has the full Qwen3-0.6B shape with seeded random
weights; it is built once per weight format and the engines on it are kept, as in a server, so a pass pays for prompts
and tokens only.

The next-token head is the embedding rolled by an odd number of rows, and the embedding is wide against what the layers
add: every pick is clear by several logits, as most picks of a trained model are, and the greedy tokens of two correct
implementations are the same whole numbers.  The cache rows that come back with them hold every layer's work.
"""

import functools
import os
import random
import sys

import numpy as np
import torch

PACKAGE = os.path.join(os.getcwd(), "qwen3-0.6b-megakernel-rtx-5090_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

import quantize  # noqa: E402
import synthetic as S  # noqa: E402
from Model.Qwen06B_architecture import BatchDecoder, Decoder  # noqa: E402
from scheduler import ContinuousBatcher  # noqa: E402

DECODER_ROWS = 8320      # cache rows of a single-sequence engine
BATCH_ROWS = 2304        # cache rows of each slot of a batched one (prompts of up to 2048 tokens)
EMBED_STD = 0.5
HEAD_ROLL = 7919
OUTPUTS_PER_PASS = 31    # sequences of a batch whose cache rows are returned beside the tokens


# ---------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # interactive use, token by token: a short prompt, then one `step` per token with its token read back
        dict(name="stream_16_8", path="stream", fmt="fp16", mode="serial", prompt=16, new=8),
        # a chat turn on an engine built with the default options
        dict(name="request_32_32", path="request", fmt="fp16", mode="serial", prompt=32, new=32),
        # a document question on the same engine; an odd prompt length
        dict(name="request_777_64", path="request", fmt="fp16", mode="serial", prompt=777, new=64),
        # the headline configuration of bench.py with its prefill: 4096-token context, batch-1 decode
        dict(name="request_4096_128", path="request", fmt="fp16", mode="tensor", prompt=4096, new=128),
        # FP8 rows at batch 1
        dict(name="request_fp8_1024_64", path="request", fmt="fp8", mode="tensor", prompt=1024, new=64),
        # a short prompt alone (time to first token), ragged against every tile
        dict(name="prefill_109", path="prefill", fmt="fp16", mode="tensor", prompt=109),
        # the longest prompt, more than one chunk, ragged
        dict(name="prefill_8191", path="prefill", fmt="fp16", mode="tensor", prompt=8191),
        # two sequences together on the persistent kernel
        dict(name="batch2_512_48", path="batch", fmt="fp16", batch=2, shortest=512, longest=512, new=48),
        # four sequences with FP8 rows, 1024-token contexts
        dict(name="batch4_fp8_1024_64", path="batch", fmt="fp8", batch=4, shortest=1024, longest=1024, new=64),
        # sixteen fp16 sequences of different lengths
        dict(name="batch16_64_1024_64", path="batch", fmt="fp16", batch=16, shortest=64, longest=1024, new=64),
        # sixty-four NVFP4 sequences, prompts of 128 to 2048 tokens
        dict(name="batch64_nvfp4_2048_64", path="batch", fmt="nvfp4", batch=64, shortest=128, longest=2048, new=64),
        # the serving job: requests queue up, at most 32 decode together, prefills overlap the decode rounds
        dict(name="serve_64x32", path="serve", fmt="fp16", requests=64, live=32, shortest=64, longest=2048, new=128),
    ]


def _between(rng, low, high):
    """A whole number of [low, high], spread over the logarithm."""
    return int(round(low * (high / low) ** rng.random()))


def draw(rng: random.Random):
    path = rng.choice(("stream", "request", "request", "request", "prefill", "prefill", "batch", "batch", "batch", "serve"))
    if path == "stream":
        mode = rng.choice(("serial", "tensor"))
        return dict(path=path, fmt=rng.choice(("fp16", "fp16", "fp8")), mode=mode,
                    prompt=_between(rng, 4, 256 if mode == "serial" else 4096), new=_between(rng, 4, 32))
    if path == "request":
        mode = rng.choice(("serial", "tensor"))
        return dict(path=path, fmt=rng.choice(("fp16", "fp16", "fp8")), mode=mode,
                    prompt=_between(rng, 8, 1024 if mode == "serial" else 8000), new=_between(rng, 8, 160))
    if path == "prefill":
        return dict(path=path, fmt=rng.choice(("fp16", "fp16", "fp8", "nvfp4")), mode="tensor", prompt=_between(rng, 24, 8191))
    longest = _between(rng, 64, 2048)
    shortest = _between(rng, max(8, longest // 16), longest)
    if path == "batch":
        return dict(path=path, fmt=rng.choice(("fp16", "fp8", "nvfp4")), batch=_between(rng, 2, 64), shortest=shortest,
                    longest=longest, new=_between(rng, 8, 64))
    return dict(path=path, fmt="fp16", requests=_between(rng, 12, 64), live=_between(rng, 8, 32), shortest=shortest,
                longest=longest, new=_between(rng, 16, 128))


# ------------------------------------------------------------------------------------- model and engines, kept as a server does
@functools.lru_cache(maxsize=None)
def _model(fmt):
    gen = torch.Generator("cuda").manual_seed(2027)

    def matrix(shape, std):
        return (torch.randn(shape, generator=gen, device="cuda") * std).to(torch.float16)

    def norm(shape):
        return (1.0 + 0.1 * torch.randn(shape, generator=gen, device="cuda")).to(torch.float16)

    def packed(w):
        if fmt == "fp8":
            return quantize.pack_rows_fp8(*quantize.quantize_rows_fp8(w))
        if fmt == "nvfp4":
            return quantize.pack_rows_nvfp4(*quantize.quantize_blocks_nvfp4(w))
        return w

    embed = matrix((S.VOCAB_SIZE, S.HIDDEN_SIZE), EMBED_STD)
    head = (embed.float() * (0.02 / EMBED_STD)).to(torch.float16).roll(HEAD_ROLL, 0).contiguous()
    layers = []
    for _ in range(S.NUM_LAYERS):
        for _, shape in S.LAYER_FIELDS:
            layers.append(norm(shape) if len(shape) == 1 else packed(matrix(shape, 0.02)))
    weights = dict(embed_weight=packed(embed), layer_weights=layers, final_norm_weight=norm((S.HIDDEN_SIZE,)),
                   lm_head_weight=packed(head))
    torch.cuda.empty_cache()
    return weights


@functools.lru_cache(maxsize=None)
def _decoder(fmt, mode):
    return Decoder(weights=_model(fmt), tokenizer=S.StubTokenizer(-1), verbose=False, max_seq_len=DECODER_ROWS,
                   weight_format=fmt, prefill_mode=mode)


@functools.lru_cache(maxsize=1)
def _batch(fmt, slots):
    return BatchDecoder(weights=_model(fmt), tokenizer=S.StubTokenizer(-1), num_sequences=slots, max_seq_len=BATCH_ROWS,
                        weight_format=fmt, prefill_mode="tensor")


@functools.lru_cache(maxsize=1)
def _batcher(fmt, live):
    # half as many slots again hold requests that are prefilled ahead
    return ContinuousBatcher(_batch(fmt, live + live // 2), eos_token_id=None, quantum=32, overlap_prefill=True,
                             live_limit=live)


def _lengths(case, count):
    """Evenly spaced from the shortest to the longest, in an order that is the case's own (any arrival order)."""
    low, high = case["shortest"], case["longest"]
    lengths = [low + (high - low) * i // max(count - 1, 1) for i in range(count)]
    random.Random(count).shuffle(lengths)
    return lengths


# --------------------------------------------------------------------------------------------------------- passes
def prepare(case, seed):
    rng = np.random.default_rng(seed)

    def ids(n):
        return rng.integers(0, S.VOCAB_SIZE, n).tolist()

    state = dict(case=case)
    if case["path"] in ("stream", "request", "prefill"):
        state["engine"] = _decoder(case["fmt"], case["mode"])
        state["prompt"] = ids(case["prompt"])
        return state
    count = case["batch"] if case["path"] == "batch" else case["requests"]
    state["prompts"] = [ids(n) for n in _lengths(case, count)]
    state["engine"] = _batch(case["fmt"], count) if case["path"] == "batch" else _batcher(case["fmt"], case["live"])
    return state


def run(state):
    case, engine = state["case"], state["engine"]
    if case["path"] == "prefill":
        engine.reset()
        engine.prefill_ids(state["prompt"])
        return _rows(engine)
    if case["path"] == "request":
        tokens = engine.generate_ids(state["prompt"], case["new"])
        return (np.array(tokens), *_rows(engine))
    if case["path"] == "stream":
        engine.reset()
        engine.prefill_ids(state["prompt"][:-1])
        tokens = [engine.step(state["prompt"][-1])]
        while len(tokens) < case["new"]:
            tokens.append(engine.step(tokens[-1]))
        return (np.array(tokens), *_rows(engine))
    if case["path"] == "batch":
        tokens = engine.generate_ids(state["prompts"], case["new"])
        rows = [(k[:, :, :n], v[:, :, :n]) for k, v, n in zip(engine._k_caches, engine._v_caches, engine.positions)]
        return np.array(tokens), rows[:OUTPUTS_PER_PASS]
    futures = [engine.submit(prompt, case["new"]) for prompt in state["prompts"]]
    engine.run_until_idle()
    return np.array([f.result().tokens for f in futures])


def _rows(engine):
    return engine._k_cache[:, :, :engine.position], engine._v_cache[:, :, :engine.position]


# ------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Weights once per prefill and once per decode step of all live sequences, cache rows written once and read once per
    step, two operations per weight and token, the causal attention's products."""
    weights = {"fp16": S.weight_bytes_fp16, "fp8": quantize.weight_bytes_fp8, "nvfp4": quantize.weight_bytes_nvfp4}[case["fmt"]]()
    row = S.NUM_LAYERS * S.KV_BYTES_PER_POSITION
    layer_ops = 2 * S.NUM_LAYERS * sum(S.math.prod(s) for _, s in S.LAYER_FIELDS if len(s) == 2)
    head_ops = 2 * S.VOCAB_SIZE * S.HIDDEN_SIZE
    pair_ops = 4 * S.NUM_LAYERS * S.Q_SIZE       # one query against one cache row, all heads and layers

    new = case.get("new", 0)
    if case["path"] in ("batch", "serve"):
        lengths = _lengths(case, case.get("batch") or case["requests"])
        together = case.get("batch") or case["live"]
    else:
        lengths, together = [case["prompt"]], 1
    filled = [n if case["path"] == "prefill" else n - 1 for n in lengths]
    steps = -(-len(lengths) // together) * new
    head = S.VOCAB_SIZE * S.HIDDEN_SIZE * {"fp16": 2, "fp8": 1, "nvfp4": 0.5625}[case["fmt"]]
    read = sum(new * n + new * (new - 1) / 2 for n in filled)
    pairs = read + sum(n * (n + 1) / 2 for n in filled)
    rows = sum(filled) + new * len(lengths)
    return {"bytes": (weights - head) + steps * weights + row * (rows + read),
            "flops": rows * layer_ops + new * len(lengths) * head_ops + pairs * pair_ops}


def tolerance(case):
    """Cache rows are fp16.  With token-serial prefill activations are fp32 and a row differs by single roundings of the
    cache and what they do downstream; the tensor-core paths round the operands of every product to fp16.  No pick is
    close, so tokens do not differ at all."""
    if case["path"] != "serve" and case.get("mode") == "serial":
        return {"rel": 1e-3, "max": 2e-2}
    return {"rel": 1e-2, "max": 2e-1}
