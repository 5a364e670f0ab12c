"""Batched decode on the tensor-core path (``decode_batched`` / ``BatchDecoder(engine="gemm")``) against the CPU
oracle, sequence by sequence.  GEMM operands are rounded to fp16 on this path (the oracle and the persistent
kernel keep fp32 activations), so the bar is the stated tolerance: logits within 3e-2 max-abs of the oracle's,
and - on these seeds - identical greedy tokens."""

import json
import os

import pytest
import torch

import synthetic as S
from oracle.decoder_ref import Decoder as OracleDecoder

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
LOGIT_TOL = 3e-2


@pytest.fixture(scope="module")
def C(built_library):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_megakernel_C
    return qwen_megakernel_C


def _engine(w, n, max_seq_len, **kw):
    from Model.Qwen06B_architecture import BatchDecoder
    return BatchDecoder(weights=S.weights_to(w, "cuda"), tokenizer=S.StubTokenizer(-1, w["embed_weight"].shape[0]),
                        num_sequences=n, max_seq_len=max_seq_len, **kw)


@pytest.mark.parametrize("n", [1, 5, 19, 40])
def test_tiny_model_against_oracle(C, n):
    """Sequence counts that are no multiple of anything; contexts from 1 token to several rounds of the attention
    kernels, all different.  40 sequences take the bulk-copy-fed attention kernel (its 6-slot ring wraps from 193
    cache rows on)."""
    vocab, steps, L = 2048, 5, 768
    w = S.make_weights(seed=21, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    lens = [(1 + 37 * i * i) % 700 + 1 for i in range(n)]
    prompts = [S.make_prompt(Ln, seed=300 + i, vocab_size=vocab) for i, Ln in enumerate(lens)]
    eng = _engine(w, n, L, engine="gemm")
    dump = torch.zeros(n, steps, vocab, device="cuda")
    C.set_logits_dump(dump)
    try:
        got = eng.generate_ids(prompts, steps)
    finally:
        C.set_logits_dump(None)
    worst = 0.0
    for b in range(n):
        want, logits = OracleDecoder(w, max_seq_len=L).generate_ids(prompts[b], steps, keep_logits=True)
        err = float((dump[b].cpu() - logits).abs().max())
        worst = max(worst, err)
        assert got[b] == want, f"sequence {b} (prompt {lens[b]} tokens)"
        assert err < LOGIT_TOL
    print(f"decode_batched, {n} sequences: worst max |logit - oracle| = {worst:.3e}")
    assert eng.positions[:n] == [Ln - 1 + steps for Ln in lens]


@pytest.mark.parametrize("n", [17, 64, 65, 128])
def test_row_tile_edges(C, n):
    """Up to 64 live rows the GEMMs multiply 64-row tiles (a quarter of the rows in each warp's lanes), above that 128-row ones:
    sequences either side of the quarters' and the tile's edges against the oracle, one step each (same bar as above)."""
    vocab, steps, L = 2048, 1, 64
    w = S.make_weights(seed=29, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    prompts = [S.make_prompt(1 + i % 5, seed=1200 + i, vocab_size=vocab) for i in range(n)]
    eng = _engine(w, n, L, engine="gemm", prefill_mode="tensor")
    dump = torch.zeros(n, steps, vocab, device="cuda")
    C.set_logits_dump(dump)
    try:
        got = eng.generate_ids(prompts, steps)
    finally:
        C.set_logits_dump(None)
    for b in sorted({0, 7, 15, 16, 17, 31, 32, 47, 48, 63, 64, 65, 95, 96, n - 1}):
        if b < n:
            want, logits = OracleDecoder(w, max_seq_len=L).generate_ids(prompts[b], steps, keep_logits=True)
            assert got[b] == want and float((dump[b].cpu() - logits).abs().max()) < LOGIT_TOL, f"sequence {b} of {n}"


def test_long_contexts_split_over_several_ctas(C):
    """Two sequences: the attention kernel divides each sequence's cache rows among eight CTAs (nine ring chunks
    per CTA at 2300 tokens, more than the ring has slots) and the last CTA to arrive adds the partial states."""
    vocab, steps, L = 2048, 4, 2432
    w = S.make_weights(seed=23, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    lens = [2300, 901]
    prompts = [S.make_prompt(Ln, seed=450 + i, vocab_size=vocab) for i, Ln in enumerate(lens)]
    eng = _engine(w, 2, L, engine="gemm", prefill_mode="serial")
    dump = torch.zeros(2, steps, vocab, device="cuda")
    C.set_logits_dump(dump)
    try:
        got = eng.generate_ids(prompts, steps)
    finally:
        C.set_logits_dump(None)
    for b in range(2):
        want, logits = OracleDecoder(w, max_seq_len=L).generate_ids(prompts[b], steps, keep_logits=True)
        err = float((dump[b].cpu() - logits).abs().max())
        print(f"split attention, {lens[b]}-token context: max |logit - oracle| = {err:.3e}")
        assert got[b] == want and err < LOGIT_TOL
    # a second call reuses the arrival counters the first one left at zero
    assert eng.generate_ids(prompts, steps) == got


def test_both_engines_and_tensor_prefill_agree(C):
    """Four sequences through the persistent launch and through the GEMM path (with tensor-core prefill):
    same tokens."""
    vocab, steps, L = 2048, 6, 512
    w = S.make_weights(seed=22, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    prompts = [S.make_prompt(Ln, seed=400 + i, vocab_size=vocab) for i, Ln in enumerate([300, 2, 77, 190])]
    a = _engine(w, 4, L, engine="persistent").generate_ids(prompts, steps)
    b = _engine(w, 4, L, engine="gemm", prefill_mode="tensor").generate_ids(prompts, steps)
    assert a == b


def test_full_model_sixteen_sequences(C, full_cfg):
    """Qwen3-0.6B shape, 16 sequences (the B = 16 configuration's shape).  Sequence 0 is the golden prompt;
    the others are compared with the single-sequence engine where its greedy margin allows a verdict."""
    from Model.Qwen06B_architecture import Decoder
    g = json.load(open(os.path.join(GOLDEN, "full_seed0_prompt32.json")))
    w = S.make_weights(seed=full_cfg["seed"], num_layers=28, vocab_size=S.VOCAB_SIZE, max_seq_len=16)
    prompts = [g["prompt"]] + [S.make_prompt(5 + 11 * i, seed=500 + i) for i in range(15)]
    steps = 12
    eng = _engine(w, 16, 256, engine="gemm")
    dump = torch.zeros(16, steps, S.VOCAB_SIZE, device="cuda")
    C.set_logits_dump(dump)
    try:
        got = eng.generate_ids(prompts, steps)
    finally:
        C.set_logits_dump(None)
    assert got[0] == g["tokens"][:steps]
    single = Decoder(weights=eng._base._weights, tokenizer=S.StubTokenizer(-1), verbose=False, max_seq_len=256)
    ref_dump = torch.zeros(steps, S.VOCAB_SIZE, device="cuda")
    worst, checked = 0.0, 0
    for b in range(16):
        C.set_logits_dump(ref_dump)
        try:
            want = single.generate_ids(prompts[b], steps)
        finally:
            C.set_logits_dump(None)
        # compare step by step while the two runs still see the same history
        for s in range(steps):
            err = float((dump[b, s] - ref_dump[s]).abs().max())
            worst = max(worst, err)
            assert err < LOGIT_TOL
            top2 = ref_dump[s].topk(2).values
            margin = float(top2[0] - top2[1])
            if got[b][s] != want[s]:
                assert margin < 2 * err + 1e-6, f"sequence {b} step {s}: tokens differ with margin {margin:.2e}, err {err:.2e}"
                break
            checked += 1
    print(f"full model, 16 sequences: worst max |logit gemm - logit persistent| = {worst:.3e}; {checked} steps token-equal")
    assert checked >= 16 * steps - 8


def test_step_overlap_changes_nothing_but_time(C):
    """The kernels of a decode step are launched as programmatic dependents of one another (each sets itself up and
    streams its weights behind its predecessor's tail, then waits for it to complete).  Switched off, the same kernels
    run strictly one after the other: tokens and every logit must be bit-identical, through the captured graph and
    through the plain launches of the logits-dump path."""
    vocab, steps, L, n = 2048, 6, 256, 9
    w = S.make_weights(seed=23, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    prompts = [S.make_prompt(5 + 23 * i, seed=900 + i, vocab_size=vocab) for i in range(n)]
    eng = _engine(w, n, L, engine="gemm")
    results = {}
    try:
        for overlap in (True, False, True):
            C.set_step_overlap(overlap)
            graph_tokens = eng.generate_ids(prompts, steps)
            dump = torch.zeros(n, steps, vocab, device="cuda")
            C.set_logits_dump(dump)
            try:
                plain_tokens = eng.generate_ids(prompts, steps)
            finally:
                C.set_logits_dump(None)
            assert graph_tokens == plain_tokens
            results.setdefault(overlap, []).append((graph_tokens, dump.cpu()))
    finally:
        C.set_step_overlap(True)
    (tok_on, logit_on), (tok_on2, logit_on2) = results[True]
    (tok_off, logit_off), = results[False]
    assert tok_on == tok_off == tok_on2
    assert torch.equal(logit_on, logit_off) and torch.equal(logit_on, logit_on2)
    want = [OracleDecoder(w, max_seq_len=L).generate_ids(p, steps)[0] for p in prompts]
    assert tok_on == want


@pytest.mark.parametrize("mma", [1, 0])
def test_both_decode_attention_kernels(C, mma):
    """The per-sequence attention of a decode step on mma.sync tiles (default) and on the CUDA-core kernel it replaced:
    contexts of 1 .. 600 rows (chunks of 16 with ragged ends, sequences split over several CTAs), against the oracle."""
    vocab, steps, L, n = 2048, 4, 640, 7
    w = S.make_weights(seed=27, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    lens = [1, 2, 16, 17, 33, 250, 600]
    prompts = [S.make_prompt(Ln, seed=700 + i, vocab_size=vocab) for i, Ln in enumerate(lens)]
    eng = _engine(w, n, L, engine="gemm")
    dump = torch.zeros(n, steps, vocab, device="cuda")
    C.set_decode_attention(mma)
    C.set_logits_dump(dump)
    try:
        got = eng.generate_ids(prompts, steps)
    finally:
        C.set_logits_dump(None)
        C.set_decode_attention(1)
    worst = 0.0
    for b in range(n):
        want, logits = OracleDecoder(w, max_seq_len=L).generate_ids(prompts[b], steps, keep_logits=True)
        worst = max(worst, float((dump[b].cpu() - logits).abs().max()))
        assert got[b] == want, f"sequence {b} (prompt {lens[b]} tokens)"
    print(f"decode attention mma={mma}: worst max |logit - oracle| = {worst:.3e}")
    assert worst < LOGIT_TOL


def _pieces(rows, ctas):
    """The rule by which a step's attention is cut, restated: ranges per item, pieces of each sequence's ranges, number of pieces."""
    n, kv_heads = len(rows), 8
    splits = min(max(ctas // (n * kv_heads), 1), 8)
    chunks = [-(-r // 16) for r in rows]
    longest = max(16, kv_heads * sum(chunks) // 4 * (7 if splits == 1 else 12) // ctas)
    parts = [1 if -(-c // splits) <= longest else 2 if -(-c // splits) <= 2 * longest else 4 for c in chunks]
    return splits, parts, kv_heads * splits * sum(parts)


@pytest.mark.parametrize("lens,splits,cut,several_each", [
    ([1], 8, 1, False), ([700, 20, 1], 8, 1, False), ([13 * 16 + 1, 13 * 16, 12 * 16 + 1, 12 * 16, 1, 2], 6, 1, False),
    ([700] + [16 * i for i in range(1, 23)], 1, 4, False), ([1 + (53 * i) % 300 for i in range(37)], 1, 2, True),
    ([1 + (101 * i) % 400 for i in range(64)], 1, 1, True), ([40] * 128, 1, 1, True), ([1100] + [20] * 17, 2, 4, True),
    ([64] * 5 + [2048], 6, 2, True), ([50] * 6 + [2000] + [50] * 5, 3, 4, True), ([200, 2300], 8, 2, False)],
    ids=["one", "split", "edges", "cut", "37", "64", "128", "split-cut4", "split-cut2", "split3-cut4", "two"])
def test_attention_pieces(C, lens, splits, cut, several_each):
    """The attention's list of pieces: items of one range and of several, ranges whole and cut in two or four, fewer pieces than
    CTAs and more (CTAs take further pieces), every other batch with table RoPE, against the CUDA-core kernel with a CTA per item and range.
    Both round the same fp32 result to fp16, so they differ by roundings of one output and what they do downstream: 1.5e-3 of a logit
    and one fp16 step (2^-9) of layer 1's new K row at most, a quarter of the bars; in the oracle a chunk of 16 rows left out of one head of
    2048, or taken twice, moves them by 6e-2 and 8e-2.  Who takes which piece does not show: a second run is the same bit for bit."""
    vocab, steps, n = 2048, 2, len(lens)
    table = len(lens) % 2 == 0
    L = (max(lens) + 64) // 64 * 64
    ctas = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    if ctas == 296:
        got_splits, parts, total = _pieces([Ln - 1 for Ln in lens], ctas)
        assert (got_splits, max(parts), total > ctas) == (splits, cut, several_each), (got_splits, parts, total)
    w = S.make_weights(seed=31, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=L if table else 16)
    prompts = [S.make_prompt(Ln, seed=1500 + i, vocab_size=vocab) for i, Ln in enumerate(lens)]
    eng = _engine(w, n, L, engine="gemm", prefill_mode="tensor", rope_from_table=table)
    runs = []
    for mma in (1, 1, 0):
        dump = torch.zeros(n, steps, vocab, device="cuda")
        C.set_decode_attention(mma)
        C.set_logits_dump(dump)
        try:
            eng.generate_ids(prompts, steps)
        finally:
            C.set_logits_dump(None)
            C.set_decode_attention(1)
            C.configure(rope_from_table=0)
        runs.append((dump.cpu(), [k[:, :, :Ln + steps - 1].cpu() for k, Ln in zip(eng._k_caches, lens)]))
    assert torch.equal(runs[0][0], runs[1][0]) and all(torch.equal(a, b) for a, b in zip(runs[0][1], runs[1][1]))
    logit = float((runs[0][0][:, 0] - runs[2][0][:, 0]).abs().max())
    # the first step's row of layer 1: what layer 0's attention gave, through one layer
    row = max(float((a[1, :, Ln - 1].float() - b[1, :, Ln - 1].float()).abs().max()) for a, b, Ln in zip(runs[0][1], runs[2][1], lens))
    print(f"pieces, {n} sequences: logits {logit:.2e}, layer-1 row {row:.2e}")
    assert logit < 6e-3 and row < 8e-3


@pytest.mark.parametrize("n,fmt", [(17, "fp16"), (64, "fp16"), (65, "fp16"), (128, "fp16"), (64, "fp8"), (64, "nvfp4"), (65, "nvfp4")])
def test_graph_steps_match_dumped_steps(C, n, fmt):
    """What a caller without a logits dump runs - a captured step, replayed, whose LM head picks from its accumulator rows - against plain
    launches that store the logits: the same tokens and cache rows bit for bit, in every quarter of the 64- and 128-row tiles, over
    steps that each make the attention's list anew and take it from the start."""
    import quantize as Q
    vocab, steps, L = 2048, 4, 512
    w = S.make_weights(seed=33, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    pack = {"fp16": lambda x: x, "fp8": lambda x: Q.quantize_weights_fp8(x)[0], "nvfp4": lambda x: Q.quantize_weights_nvfp4(x)[0]}[fmt]
    prompts = [S.make_prompt(1 + (101 * i) % 400, seed=1600 + i, vocab_size=vocab) for i in range(n)]
    eng = _engine(pack(w), n, L, engine="gemm", prefill_mode="tensor", weight_format=fmt)
    dump = torch.zeros(n, steps, vocab, device="cuda")
    runs = []
    try:
        for target in (None, dump, None):
            C.set_logits_dump(target)
            runs.append((eng.generate_ids(prompts, steps), [(k.clone(), v.clone()) for k, v in zip(eng._k_caches, eng._v_caches)]))
    finally:
        C.set_logits_dump(None)
        C.set_weight_format("fp16")
    assert [dump[b].argmax(1).tolist() for b in range(n)] == runs[1][0]
    for tokens, rows in (runs[0], runs[2]):
        assert tokens == runs[1][0]
        assert all(torch.equal(a, b) and torch.equal(c, d) for (a, c), (b, d) in zip(rows, runs[1][1]))


@pytest.mark.parametrize("fmt", ["fp16", "fp8", "nvfp4"])
@pytest.mark.parametrize("dumped", [False, True], ids=["graph", "dump"])
def test_logits_without_a_largest_value_are_an_error(C, fmt, dumped):
    """A sequence whose logits are all NaN has no pick; what stands in its place (2^31 - 1) is an error of the step that would read its
    embedding row, as in the persistent kernels, through the LM head's own pick (graph) and the pick from stored logits (dump).
    The call before and the call behind it are sound."""
    import quantize as Q
    vocab, n = 2048, 20
    w = S.make_weights(seed=41, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    pack = {"fp16": lambda x: x, "fp8": lambda x: Q.quantize_weights_fp8(x)[0], "nvfp4": lambda x: Q.quantize_weights_nvfp4(x)[0]}[fmt]
    prompts = [S.make_prompt(1 + i % 4, seed=1700 + i, vocab_size=vocab) for i in range(n)]
    eng = _engine(pack(w), n, 64, engine="gemm", prefill_mode="tensor", weight_format=fmt)
    dump = torch.zeros(n, 3, vocab, device="cuda")
    norm = eng._base._final_norm_weight
    kept = norm.clone()
    try:
        want = eng.generate_ids(prompts, 3)
        C.set_logits_dump(dump if dumped else None)
        norm.fill_(float("nan"))
        with pytest.raises(RuntimeError, match=r"outside \[0, vocab\).*status 5"):
            eng.generate_ids(prompts, 3)
        norm.copy_(kept)
        assert eng.generate_ids(prompts, 3) == want
    finally:
        C.set_logits_dump(None)
        C.set_weight_format("fp16")


@pytest.mark.parametrize("more", [29, 49, 56, 64])
def test_rows_of_the_mma_keep_the_bits(C, more):
    """Steps of 28 fp16 sequences take 64-row products, of more 128-row ones: the sequences of both end in the same tokens and
    cache rows bit for bit."""
    vocab, steps = 2048, 6
    w = S.make_weights(seed=33, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    prompts = [S.make_prompt(3 + 5 * i, seed=600 + i, vocab_size=vocab) for i in range(more)]
    ends = []
    for n in (28, more):
        eng = _engine(w, n, 400, engine="gemm")
        tokens = eng.generate_ids(prompts[:n], steps)
        ends.append((tokens[:28], [(eng._k_caches[b][:, :, :eng.positions[b]].clone(), eng._v_caches[b][:, :, :eng.positions[b]].clone()) for b in range(28)]))
        del eng
    (t0, c0), (t1, c1) = ends
    assert t0 == t1
    assert all(torch.equal(k, x) and torch.equal(v, y) for (k, v), (x, y) in zip(c0, c1))


def test_a_refused_layer_table_changes_no_later_call(C):
    """Layer tables are read back and their matrices' tensor maps kept until another table comes.  A table that is refused half-way
    (its second layer has a null pointer) has replaced the maps of its first: a call on the table before it makes them anew."""
    vocab, n = 2048, 6
    engines = [_engine(S.make_weights(seed=seed, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16), n, 64, engine="gemm",
                       prefill_mode="tensor") for seed in (51, 52)]
    prompts = [S.make_prompt(2 + i, seed=1800 + i, vocab_size=vocab) for i in range(n)]
    want = engines[0].generate_ids(prompts, 3)
    rows = [k.clone() for k in engines[0]._k_caches[:n]]
    base = engines[1]._base
    table = base._layer_weights_packed.clone()
    table.view(torch.int64)[12 + 6] = 0
    common = (base._cos_table, base._sin_table)
    with pytest.raises(RuntimeError, match="null weight pointer"):
        C.decode_batched([1], [0], 1, base._embed_weight, table, base._final_norm_weight, base._lm_head_weight, *common,
                         engines[1]._k_caches[:1], engines[1]._v_caches[:1], [torch.zeros(1, dtype=torch.int32, device="cuda")],
                         base.num_layers, 64, base._attn_scale)
    with pytest.raises(RuntimeError, match="null weight pointer"):
        C.prefill_chunked(torch.tensor([1, 2], dtype=torch.int32), base._embed_weight, table, *common, engines[1]._k_caches[0],
                          engines[1]._v_caches[0], base.num_layers, 0, 64, base._attn_scale)
    assert engines[0].generate_ids(prompts, 3) == want
    assert all(torch.equal(a, b) for a, b in zip(rows, engines[0]._k_caches))


@pytest.mark.parametrize("what", [1, 2])
def test_attention_waits_run_out_and_leave_the_device_usable(C, what):
    """Cache rows that never come: all of them (every wait of consumers and producer runs out), or one chunk among others in flight.
    Status 4 after the budget, and steps behind it are as before: nothing lands in their shared memory."""
    vocab, n, L = 2048, 37, 768
    w = S.make_weights(seed=43, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    prompts = [S.make_prompt(1 + (131 * i) % 700, seed=1900 + i, vocab_size=vocab) for i in range(n)]
    eng = _engine(w, n, L, engine="gemm", prefill_mode="tensor")
    want = eng.generate_ids(prompts, 3)
    rows = [k.clone() for k in eng._k_caches]
    for _ in range(3):
        assert C.selftest_decode_attention_wait_timeout(300, what) == 4
        assert eng.generate_ids(prompts, 3) == want
        assert all(torch.equal(a, b) for a, b in zip(rows, eng._k_caches))


def test_refusals(C):
    vocab = 2048
    w = S.make_weights(seed=1, num_layers=2, vocab_size=vocab, max_seq_len=16)
    eng = _engine(w, 6, 64, engine="gemm")
    with pytest.raises(ValueError):
        eng.generate_ids([[1]] * 7, 2)
    base = eng._base
    log = torch.zeros(4, dtype=torch.int32, device="cuda")
    common = (base._embed_weight, base._layer_weights_packed, base._final_norm_weight, base._lm_head_weight,
              base._cos_table, base._sin_table)
    with pytest.raises(RuntimeError, match="max_seq_len"):
        C.decode_batched([1, 2], [0, 63], 2, *common, eng._k_caches[:2], eng._v_caches[:2], [log, log.clone()],
                         base.num_layers, 64, base._attn_scale)
    with pytest.raises(RuntimeError, match="share"):
        C.decode_batched([1, 2], [0, 0], 2, *common, [eng._k_caches[0]] * 2, eng._v_caches[:2], [log, log.clone()],
                         base.num_layers, 64, base._attn_scale)
    assert len(eng.generate_ids([[1, 2, 3]] * 6, 3)[5]) == 3
