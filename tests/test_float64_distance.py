"""How far cache rows are from float64 arithmetic, for the kernels that split fp32 activations into fp16 halves.

Reference: the model in float64 on the device, with the engine's OWN cache rows as the keys and values of every layer.  A row
of layer l then differs from the reference only by what the kernels lost on the way to it, not by what earlier flips of the
fp16 cache did, and the share of values that round to another fp16 than the reference's is twice the relative error over the
fp16 spacing: errors of 1e-7 show as flips of 0.1 %.  The bar is a kernel with fp32 activations: rounded fp32 FMAs on the
CUDA cores (``set_fused(1)``), run on the same prompts."""

import math

import pytest
import torch

import quantize as Q
import synthetic as S

pytestmark = pytest.mark.gpu
VOCAB, LAYERS = 4096, 4


@pytest.fixture(scope="module")
def C(built_library):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_megakernel_C
    yield qwen_megakernel_C
    qwen_megakernel_C.set_fused(fused=2)
    qwen_megakernel_C.set_weight_format("fp16")


def _model(fmt, kind="plain"):
    w = S.make_weights(seed=5, num_layers=LAYERS, vocab_size=VOCAB, norm_std=0.1, max_seq_len=16)
    w["embed_weight"] = w["lm_head_weight"] = (w["embed_weight"].float() * 25).half()
    for l in range(LAYERS):
        at = 11 * l
        if kind == "small":      # SwiGLU outputs near 1e-3, the down matrix makes up for it
            w["layer_weights"][at + 9] = (w["layer_weights"][at + 9].float() / 200).half()
            w["layer_weights"][at + 10] = (w["layer_weights"][at + 10].float() * 100).half()
        if kind == "peaky":      # attention on few keys
            w["layer_weights"][at + 4] = (w["layer_weights"][at + 4].float() * 4).half()
    engine_w, oracle_w = Q.quantize_weights_fp8(w) if fmt == "fp8" else (w, w)
    return S.weights_to(engine_w, "cuda"), oracle_w


def flips(weights, ids, k_rows, v_rows, first):
    """Values of rows [first, len(ids)) in layers 1 and up that differ from the reference's fp16, and how many there are."""
    T = len(ids)

    def f64(t):
        return t.cuda().double()

    def rms(x, g):
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * g
    inv = (1.0 / (1e6 ** (torch.arange(0, 128, 2, dtype=torch.float32) / 128))).cuda()
    ang = (torch.arange(T, device="cuda", dtype=torch.float32)[:, None] * inv).double()[:, None]
    cos, sin = ang.cos(), ang.sin()

    def rope(x):
        return torch.cat((x[..., :64] * cos - x[..., 64:] * sin, x[..., :64] * sin + x[..., 64:] * cos), -1)
    x = f64(weights["embed_weight"])[torch.tensor(ids, device="cuda")]
    wrong = total = 0
    for l in range(LAYERS):
        w = [f64(t) for t in weights["layer_weights"][11 * l:11 * l + 11]]
        h = rms(x, w[0])
        if l > 0:
            for got, want in ((k_rows[l], rope(rms((h @ w[2].T).view(T, 8, 128), w[5]))), (v_rows[l], (h @ w[3].T).view(T, 8, 128))):
                wrong += int((got[:, first:T] != want.transpose(0, 1)[:, first:].half()).sum())
                total += got[:, first:T].numel()
        if l == LAYERS - 1:
            return wrong, total
        q = rope(rms((h @ w[1].T).view(T, 16, 128), w[4]))
        out = torch.empty(T, 16, 128, device="cuda", dtype=torch.double)
        for head in range(16):
            keys, values = k_rows[l, head // 2, :T].double(), v_rows[l, head // 2, :T].double()
            for a in range(0, T, 2048):
                b = min(T, a + 2048)
                s = q[a:b, head] @ keys[:b].T / math.sqrt(128)
                s.masked_fill_(torch.arange(b, device="cuda")[None] > torch.arange(a, b, device="cuda")[:, None], -math.inf)
                out[a:b, head] = torch.softmax(s, -1) @ values[:b]
        x = x + out.reshape(T, 2048) @ w[6].T
        h = rms(x, w[7])
        g = h @ w[8].T
        x = x + (g * torch.sigmoid(g) * (h @ w[9].T)) @ w[10].T


@pytest.mark.parametrize("fmt,sequences,bound", [("fp8", 1, 1.1), ("fp8", 2, 1.1), ("fp16", 1, 1.2), ("fp16", 2, 1.2), ("fp16", 4, 1.2)])
def test_decoded_rows(C, fmt, sequences, bound):
    """Tensor-core decode against the CUDA-core launches.  About 2400 flips of 1.5 million values a sequence on either side,
    2 % of counting noise each: 1.1 is above four sigma of it.  fp16 weights: the products of 11-bit operands lose a little
    inside the MMA itself (16 of them aligned and truncated to its internal width), measured 1.00 to 1.08.  With accumulators
    handed from MMA to MMA over whole rows these ratios were 1.13 to 1.26 (FP8 rows) and 1.6 to 1.7 (fp16 rows)."""
    from Model.Qwen06B_architecture import BatchDecoder, Decoder
    engine_w, oracle_w = _model(fmt)
    prompts = [S.make_prompt(1024 - 7 * b, seed=b, vocab_size=VOCAB) for b in range(sequences)]
    steps, share = 256, {}
    tok = S.StubTokenizer(-1, VOCAB)
    if sequences == 1:
        eng = Decoder(weights=engine_w, tokenizer=tok, verbose=False, max_seq_len=1312, weight_format=fmt, prefill_mode="tensor")
    else:
        eng = BatchDecoder(weights=engine_w, tokenizer=tok, num_sequences=sequences, max_seq_len=1312, weight_format=fmt,
                           prefill_mode="tensor", engine="persistent")
    for fused in (2, 1):
        C.set_fused(fused=fused)
        tokens = [eng.generate_ids(prompts[0], steps)] if sequences == 1 else eng.generate_ids(prompts, steps)
        ks, vs = ([eng._k_cache], [eng._v_cache]) if sequences == 1 else (eng._k_caches, eng._v_caches)
        wrong = total = 0
        for b in range(sequences):
            n, of = flips(oracle_w, prompts[b] + tokens[b][:-1], ks[b], vs[b], len(prompts[b]) - 1)
            wrong, total = wrong + n, total + of
        share[fused] = wrong / total
    print(f"{fmt} x {sequences}: tensor cores {100 * share[2]:.4f} %, CUDA cores {100 * share[1]:.4f} %")
    assert 0 < share[2] < bound * share[1]


@pytest.mark.parametrize("fmt,kind,tokens,bound", [("fp16", "small", 1024, 1.3), ("fp8", "small", 1024, 1.3), ("fp16", "plain", 100, 1.4),
                                                   ("fp16", "plain", 4096, 1.3), ("fp16", "peaky", 4096, 1.3), ("fp8", "plain", 4096, 1.3),
                                                   ("fp8", "peaky", 4096, 1.3)])
def test_prefilled_rows(C, fmt, kind, tokens, bound):
    """The ``prefill`` op in one pass against the same op as persistent steps on the CUDA cores (``set_fused(0)``).  SwiGLU
    outputs near 1e-3 are where lo halves stored as they are meet the fp16 subnormals (ratio above 10 then); attention on few
    of many keys is where truncated sums of scores and outputs show (ratios of 2 and 3 at 4096 tokens)."""
    from Model.Qwen06B_architecture import Decoder
    engine_w, oracle_w = _model(fmt, kind)
    ids = S.make_prompt(tokens, seed=tokens, vocab_size=VOCAB)
    share = {}
    for fused in (2, 0):
        C.set_fused(fused=fused)
        eng = Decoder(weights=engine_w, verbose=False, max_seq_len=(tokens + 63) // 64 * 64, weight_format=fmt)
        eng.prefill_ids(ids)
        wrong, total = flips(oracle_w, ids, eng._k_cache, eng._v_cache, 0)
        share[fused] = wrong / total
    C.set_fused(fused=2)
    print(f"{fmt} {kind} {tokens}: one pass {100 * share[2]:.4f} %, steps {100 * share[0]:.4f} %")
    assert 0 < share[2] < bound * share[0]
