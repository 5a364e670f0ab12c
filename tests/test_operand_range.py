"""Activations beyond the range of fp16 (65504) through the kernels that split fp32 activations into fp16 halves.

Three models, each with one kind of operand above that range while everything around it stays ordinary (another matrix or
norm makes up for it): SwiGLU outputs near 1e5 to 1e6, RMS-normalised activations near 1e5 (norm weights of 30000), rotated
queries near 1e5 (query norm weights of 30000).  Tokens have to be the oracle's; cache rows and logits within the bounds that
ordinary models are held to (2e-2; logits relative to their size)."""

import pytest
import torch

import quantize as Q
import synthetic as S
from oracle.decoder_ref import Decoder as OracleDecoder

pytestmark = pytest.mark.gpu
VOCAB, LAYERS = 4096, 3
FP16_MAX = 65504.0


@pytest.fixture(scope="module")
def C(built_library):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_megakernel_C
    yield qwen_megakernel_C
    qwen_megakernel_C.set_weight_format("fp16")


def _model(kind, fmt):
    w = S.make_weights(seed=41, num_layers=LAYERS, vocab_size=VOCAB, norm_std=0.1, max_seq_len=16)
    lw = w["layer_weights"]

    def scale(i, f):
        lw[i] = (lw[i].float() * f).half()
    for l in range(LAYERS):
        at = 11 * l
        if kind == "swiglu":
            scale(at + 8, 400)
            scale(at + 9, 400)
            scale(at + 10, 1 / 2000)
        elif kind == "norm":
            for i in (0, 7):
                scale(at + i, 30000)
            for i in (1, 2, 3, 8, 9):
                scale(at + i, 1 / 8000)
        else:
            scale(at + 4, 30000)
            scale(at + 5, 1 / 30000)
    if kind == "norm":
        w["final_norm_weight"] = (w["final_norm_weight"].float() * 30000).half()
    engine_w, oracle_w = Q.quantize_weights_fp8(w) if fmt == "fp8" else (w, w)
    return S.weights_to(engine_w, "cuda"), oracle_w


def _check_reach(kind, oracle_w, token):
    """The model does what its name says."""
    o = OracleDecoder(oracle_w, max_seq_len=16)
    o.step(token, trace=True)
    t = o.trace[1]
    x = t["x1"]
    normed = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * oracle_w["layer_weights"][11 + 7].float()
    assert {"swiglu": t["inter"], "norm": normed, "query": t["q_rot"]}[kind].abs().max() > 1.1 * FP16_MAX


def _compare(tag, caches, want_caches, dump, logits, got, want, n):
    err = max(float((a[:, :, :n].float().cpu() - b[:, :, :n].float()).abs().max() / max(1.0, float(b[:, :, :n].float().abs().max())))
              for a, b in zip(caches, want_caches))
    lerr = float((dump.cpu() - logits).abs().max() / logits.abs().max())
    print(f"{tag}: cache {err:.2e} logits {lerr:.2e}")
    assert torch.isfinite(dump).all()
    assert got == want
    assert err < 2e-2 and lerr < 1e-2


@pytest.mark.parametrize("kind", ["swiglu", "norm", "query"])
@pytest.mark.parametrize("fmt,sequences", [("fp16", 1), ("fp8", 1), ("fp16", 2), ("fp8", 4)])
def test_decode(C, kind, fmt, sequences):
    from Model.Qwen06B_architecture import BatchDecoder, Decoder
    engine_w, oracle_w = _model(kind, fmt)
    steps, first = 20, [7, 1300, 11, 2902][:sequences]
    _check_reach(kind, oracle_w, first[0])
    tok = S.StubTokenizer(-1, VOCAB)
    dump = torch.zeros(sequences, steps, VOCAB, device="cuda")
    C.set_logits_dump(dump)
    try:
        if sequences == 1:
            eng = Decoder(weights=engine_w, tokenizer=tok, verbose=False, max_seq_len=64, weight_format=fmt)
            got, caches = [eng.generate_ids(first, steps)], [(eng._k_cache, eng._v_cache)]
        else:
            eng = BatchDecoder(weights=engine_w, tokenizer=tok, num_sequences=sequences, max_seq_len=64, weight_format=fmt,
                               engine="persistent")
            got, caches = eng.generate_ids([[t] for t in first], steps), list(zip(eng._k_caches, eng._v_caches))
    finally:
        C.set_logits_dump(None)
    for b in range(sequences):
        o = OracleDecoder(oracle_w, max_seq_len=64)
        want, logits = o.generate_ids([first[b]], steps, keep_logits=True)
        _compare(f"{kind} {fmt} x {sequences}, sequence {b}", caches[b], (o.k_cache, o.v_cache), dump[b], logits, got[b], want, steps)


@pytest.mark.parametrize("kind", ["swiglu", "norm", "query"])
@pytest.mark.parametrize("fmt,tokens", [("fp16", 40), ("fp8", 40), ("fp16", 300)])
def test_prefill(C, kind, fmt, tokens):
    """The ``prefill`` op: queries are scaled by its attention kernel; the other two kinds send the prompt through the
    persistent steps, which rewrite every row."""
    from Model.Qwen06B_architecture import Decoder
    engine_w, oracle_w = _model(kind, fmt)
    ids, steps = S.make_prompt(tokens + 1, seed=tokens, vocab_size=VOCAB), 6
    _check_reach(kind, oracle_w, ids[0])
    eng = Decoder(weights=engine_w, tokenizer=S.StubTokenizer(-1, VOCAB), verbose=False, max_seq_len=320, weight_format=fmt)
    dump = torch.zeros(steps, VOCAB, device="cuda")
    C.set_logits_dump(dump)
    try:
        got = eng.generate_ids(ids, steps)
    finally:
        C.set_logits_dump(None)
    o = OracleDecoder(oracle_w, max_seq_len=320)
    want, logits = o.generate_ids(ids, steps, keep_logits=True)
    _compare(f"{kind} {fmt}, prompt of {tokens}", (eng._k_cache, eng._v_cache), (o.k_cache, o.v_cache), dump, logits, got, want,
             tokens + steps)
