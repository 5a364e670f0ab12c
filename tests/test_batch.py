"""GPU parity of the multi-sequence launch (``generate_batch`` / ``BatchDecoder``) against the CPU oracle.

Every sequence of a launch is checked on its own against the oracle run on the same prompt: identical
greedy token IDs, logits within 3e-2 max-abs (the bound stated for the fp16 engine).  Sequences differ
in length on purpose, so that each one has its own position, RoPE angles and attention split."""

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


def _batch_engine(w, n, max_seq_len, **kw):
    from Model.Qwen06B_architecture import BatchDecoder
    kw.setdefault("engine", "persistent")   # this file covers the multi-sequence persistent kernel
    return BatchDecoder(weights=S.weights_to(w, "cuda"), tokenizer=S.StubTokenizer(-1, w["embed_weight"].shape[0]),
                        num_sequences=n, max_seq_len=max_seq_len, **kw)


def _oracle(w, max_seq_len, prompts, steps):
    want, logits = [], []
    for ids in prompts:
        t, lg = OracleDecoder(w, max_seq_len=max_seq_len).generate_ids(ids, steps, keep_logits=True)
        want.append(t)
        logits.append(lg)
    return want, logits


def _run_with_dump(C, eng, prompts, steps, vocab):
    dump = torch.zeros(len(prompts), steps, vocab, device="cuda")
    C.set_logits_dump(dump)
    try:
        got = eng.generate_ids(prompts, steps)
    finally:
        C.set_logits_dump(None)
    return got, dump.cpu()


@pytest.mark.parametrize("n", [1, 2, 3, 4])
def test_tiny_model_every_group_width(C, tiny_cfg, n):
    """1, 2, 3 and 4 sequences per launch (12, 6, 4 and 3 math warps per sequence)."""
    w = S.make_weights(seed=tiny_cfg["seed"], num_layers=tiny_cfg["num_layers"], vocab_size=tiny_cfg["vocab_size"],
                       norm_std=tiny_cfg["norm_std"], max_seq_len=tiny_cfg["max_seq_len"])
    lens = [12, 5, 23, 1][:n]
    prompts = [S.make_prompt(L, seed=20 + i, vocab_size=tiny_cfg["vocab_size"]) for i, L in enumerate(lens)]
    steps = 7
    want, logits = _oracle(w, tiny_cfg["max_seq_len"], prompts, steps)
    eng = _batch_engine(w, n, tiny_cfg["max_seq_len"])
    got, dump = _run_with_dump(C, eng, prompts, steps, tiny_cfg["vocab_size"])
    for b in range(n):
        err = float((dump[b] - logits[b]).abs().max())
        print(f"batch {n}, sequence {b}: max |logit - oracle| = {err:.3e}")
        assert got[b] == want[b]
        assert err < LOGIT_TOL
    assert eng.positions[:n] == [L - 1 + steps for L in lens]
    # second call on the same engine: caches are reused from position 0, same answer
    assert eng.generate_ids(prompts, steps) == want


def test_mixed_context_lengths_split_and_unsplit(C):
    """One launch with a 1400-token context (attention split over several CTAs + merge), a 700-token
    one and two short ones: the per-sequence split counts and ring chunk counts all differ."""
    w = S.make_weights(seed=4, num_layers=2, vocab_size=2048, norm_std=0.1, max_seq_len=16)
    lens = [1400, 3, 700, 130]
    prompts = [S.make_prompt(L, seed=40 + i, vocab_size=2048) for i, L in enumerate(lens)]
    steps = 5
    want, logits = _oracle(w, 1536, prompts, steps)
    eng = _batch_engine(w, 4, 1536)
    got, dump = _run_with_dump(C, eng, prompts, steps, 2048)
    for b in range(4):
        err = float((dump[b] - logits[b]).abs().max())
        print(f"mixed contexts, sequence {b} (len {lens[b]}): max |logit - oracle| = {err:.3e}")
        assert got[b] == want[b]
        assert err < LOGIT_TOL
    # cache rows of the long sequence against the oracle's (fp16 storage)
    o = OracleDecoder(w, max_seq_len=1536)
    o.generate_ids(prompts[0], steps)
    n = lens[0] - 1 + steps
    assert (eng._k_caches[0][:, :, :n].float().cpu() - o.k_cache[:, :, :n].float()).abs().max() < 8e-3
    assert (eng._v_caches[0][:, :, :n].float().cpu() - o.v_cache[:, :, :n].float()).abs().max() < 8e-3


def test_long_contexts_jump_several_ring_laps(C):
    """Four contexts above 2000 tokens: every sequence's attention item brings about nine cache chunks
    into the 13-slot ring, so the later groups jump more than two ring laps ahead when they skip the
    other sequences' chunks (the case the issued-chunk check in front of the parity wait exists for)."""
    w = S.make_weights(seed=8, num_layers=2, vocab_size=2048, norm_std=0.1, max_seq_len=16)
    lens = [2300, 2200, 2100, 2050]
    prompts = [S.make_prompt(L, seed=80 + i, vocab_size=2048) for i, L in enumerate(lens)]
    steps = 4
    want, logits = _oracle(w, 2560, prompts, steps)
    eng = _batch_engine(w, 4, 2560)
    got, dump = _run_with_dump(C, eng, prompts, steps, 2048)
    for b in range(4):
        err = float((dump[b] - logits[b]).abs().max())
        print(f"long contexts, sequence {b} (len {lens[b]}): max |logit - oracle| = {err:.3e}")
        assert got[b] == want[b]
        assert err < LOGIT_TOL
    eng2 = _batch_engine(w, 2, 2560)
    assert eng2.generate_ids(prompts[:2], steps) == want[:2]


def test_full_model_four_sequences_match_single_sequence_and_golden(C, full_cfg):
    """Qwen3-0.6B shape.  Sequence 0 is the golden prompt (token IDs from the committed oracle run);
    all four must equal what the single-sequence engine produces for the same prompts."""
    from Model.Qwen06B_architecture import Decoder
    g = json.load(open(os.path.join(GOLDEN, "full_seed0_prompt32.json")))
    w = S.make_weights(seed=full_cfg["seed"], num_layers=28, vocab_size=S.VOCAB_SIZE, max_seq_len=128)
    prompts = [g["prompt"]] + [S.make_prompt(L, seed=60 + i) for i, L in enumerate([7, 50, 19])]
    steps = 32
    eng = _batch_engine(w, 4, 128)
    got = eng.generate_ids(prompts, steps)
    assert got[0] == g["tokens"]
    single = Decoder(weights=eng._base._weights, tokenizer=S.StubTokenizer(-1), verbose=False, max_seq_len=128)
    for b in range(4):
        assert got[b] == single.generate_ids(prompts[b], steps), f"sequence {b}"
    # deterministic: the same launch twice gives the same tokens
    assert eng.generate_ids(prompts, steps) == got


def test_eos_is_cut_on_the_host(C, tiny_cfg):
    w = S.make_weights(seed=tiny_cfg["seed"], num_layers=tiny_cfg["num_layers"], vocab_size=tiny_cfg["vocab_size"],
                       norm_std=tiny_cfg["norm_std"], max_seq_len=tiny_cfg["max_seq_len"])
    prompts = [S.make_prompt(L, seed=20 + i, vocab_size=tiny_cfg["vocab_size"]) for i, L in enumerate([12, 5])]
    eng = _batch_engine(w, 2, tiny_cfg["max_seq_len"])
    full = eng.generate_ids(prompts, 8)
    stop = full[0][3]
    eng.tokenizer = eng._base.tokenizer = S.StubTokenizer(stop, tiny_cfg["vocab_size"])
    cut = eng.generate_ids(prompts, 8)
    for b in range(2):
        want = full[b][:full[b].index(stop)] if stop in full[b] else full[b]
        assert cut[b] == want


def test_bad_arguments_are_refused(C, tiny_cfg):
    w = S.make_weights(seed=1, num_layers=2, vocab_size=tiny_cfg["vocab_size"], max_seq_len=64)
    eng = _batch_engine(w, 2, 64)
    base = eng._base
    log = torch.zeros(4, dtype=torch.int32, device="cuda")
    common = (base._embed_weight, base._layer_weights_packed, base._final_norm_weight, base._lm_head_weight,
              base._cos_table, base._sin_table)
    with pytest.raises(RuntimeError, match="share"):   # same cache twice
        C.generate_batch([1, 2], [0, 0], 2, *common, [eng._k_caches[0]] * 2, eng._v_caches[:2], [log, log.clone()],
                         base.num_layers, 64, base._attn_scale)
    with pytest.raises(RuntimeError, match="max_seq_len"):   # one sequence would run past its cache
        C.generate_batch([1, 2], [0, 63], 2, *common, eng._k_caches[:2], eng._v_caches[:2], [log, log.clone()],
                         base.num_layers, 64, base._attn_scale)
    with pytest.raises(RuntimeError, match="1 to 4"):
        C.generate_batch([1] * 5, [0] * 5, 2, *common, eng._k_caches[:1] * 5, eng._v_caches[:1] * 5, [log] * 5,
                         base.num_layers, 64, base._attn_scale)
    # still healthy
    assert len(eng.generate_ids([[1, 2, 3], [4, 5]], 3)[0]) == 3


@pytest.mark.parametrize("fmt,ctas,lens", [("fp16", 0, [1]), ("fp16", 0, [513, 2]), ("fp16", 96, [40, 1500]), ("fp16", 112, [17, 1500, 16, 2]),
                                           ("fp16", 0, [130, 1, 900]), ("fp8", 0, [1500, 15]), ("fp8", 112, [18, 1, 700, 256]),
                                           ("fp16", 100, [6, 300, 9])])
def test_tensor_core_launch_matches_group_launch(C, fmt, ctas, lens):
    """All sequences as columns of one MMA against the launch with a group of warps per sequence (``set_fused(1)``) and the
    oracle: one to four sequences (three leave columns idle), the smallest grids of either build and one below (both runs
    then take the group launch, behind prompts whose prefill the switch does not touch), contexts without old rows, around
    a 16-row cache chunk, and with every split.  Same precision, other summation order: the bound of the single-sequence
    kernels' comparison (1e-3)."""
    import quantize as Q
    vocab, steps, rows = 4104, 18, 1536
    w = S.make_weights(seed=29, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    eng_w, ora_w = Q.quantize_weights_fp8(w) if fmt == "fp8" else (w, w)
    prompts = [S.make_prompt(L, seed=200 + i, vocab_size=vocab) for i, L in enumerate(lens)]
    want, logits = _oracle(ora_w, rows, prompts, steps)
    dumps = []
    try:
        C.configure(max_ctas=ctas)
        eng = _batch_engine(eng_w, len(lens), rows, weight_format=fmt)
        for fused in (2, 1, 2):
            C.set_fused(fused=fused)
            got, dump = _run_with_dump(C, eng, prompts, steps, vocab)
            assert got == want, fused
            dumps.append(dump)
    finally:
        C.set_fused(fused=2)
        C.configure(max_ctas=0)
        C.set_weight_format("fp16")
    diff = float((dumps[0] - dumps[1]).abs().max())
    err = [max(float((d[b] - logits[b]).abs().max()) for b in range(len(lens))) for d in dumps]
    print(f"{fmt} ctas {ctas} {lens}: columns vs groups {diff:.2e}; against the oracle {err[0]:.2e}, {err[1]:.2e}")
    assert torch.equal(dumps[0], dumps[2]), "not reproducible run to run"
    assert torch.equal(dumps[0], dumps[1]) == (ctas == 100)
    assert diff < 1e-3 and max(err) < LOGIT_TOL


@pytest.mark.parametrize("fmt", ["fp16", "fp8"])
def test_every_in_place_edit_of_the_weights_is_noticed(C, fmt):
    """A launch of several sequences multiplies K-major copies of W_o and W_down and checks all bytes of the caller's
    matrices first: an edit that none of the sampled hashes of the single-sequence calls covers, the edit taken back behind a
    single-sequence call, and one in the last row of W_down."""
    import quantize as Q
    vocab, steps = 2048, 6
    w = S.make_weights(seed=51, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    eng_w, ora_w = Q.quantize_weights_fp8(w) if fmt == "fp8" else (w, w)
    dev = S.weights_to(eng_w, "cuda")
    prompts = [[5], [900]]
    try:
        eng = _batch_engine(dict(dev), 2, 64, weight_format=fmt)
        live = eng._base._weights["layer_weights"]

        def rows():
            eng.generate_ids(prompts, steps)
            return [k[:, :, :steps].clone() for k in eng._k_caches]

        def fresh():
            other = _batch_engine({k: ([t.clone() for t in v] if isinstance(v, list) else v.clone()) for k, v in eng._base._weights.items()},
                                  2, 64, weight_format=fmt)
            other.generate_ids(prompts, steps)
            return [k[:, :, :steps].clone() for k in other._k_caches]

        def same(a, b):
            return all(torch.equal(x, y) for x, y in zip(a, b))
        first = rows()
        wo, wd = live[6].view(torch.uint8), live[10].view(torch.uint8)
        keep = wo[0, 80:96].clone()
        wo[0, 80:96] = wo[1, 160:176]           # sixteen bytes between the first two samples of the first layer's W_o
        edited = rows()
        assert not same(first, edited) and same(edited, fresh())
        eng._base.generate_ids([7], 3)
        wo[0, 80:96] = keep
        assert same(rows(), first)
        wd[1023, 3040:3056] = wd[5, 64:80]
        last = rows()
        assert not same(last, first) and same(last, fresh())
    finally:
        C.set_weight_format("fp16")


@pytest.mark.parametrize("fmt", ["fp16", "fp8"])
@pytest.mark.parametrize("n,ctas", [(1, 96), (1, 97), (1, 125), (1, 128), (1, 147), (2, 99), (2, 125), (4, 113), (4, 126), (3, 148)])
def test_attention_slices_of_every_grid(C, fmt, n, ctas):
    """Groups of four CTAs share a slice of the attention outputs: 88 rows a group on 96 CTAs, 64 on 128, 68 on 125; CTAs past the
    last whole group have none.  The slices of a grid that were not read, or read twice, would show in every logit: an output
    is a sum over all of them, and contributions are about 1/24 of it against a bar of 3e-2 of logits of order one."""
    import quantize as Q
    w = S.make_weights(seed=17, num_layers=2, vocab_size=2048, norm_std=0.1, max_seq_len=16)
    engine_w, oracle_w = Q.quantize_weights_fp8(w) if fmt == "fp8" else (w, w)
    prompts = [S.make_prompt(L, seed=70 + i, vocab_size=2048) for i, L in enumerate([300, 9, 150, 40][:n])]
    want, logits = _oracle(oracle_w, 320, prompts, 5)
    eng = _batch_engine(engine_w, n, 320, weight_format=fmt)
    C.configure(max_ctas=ctas)
    try:
        got, dump = _run_with_dump(C, eng, prompts, 5, 2048)
    finally:
        C.configure(max_ctas=0)
        C.set_weight_format("fp16")
    for b in range(n):
        assert got[b] == want[b]
        assert float((dump[b] - logits[b]).abs().max()) < LOGIT_TOL


@pytest.mark.parametrize("fmt", ["fp16", "fp8"])
@pytest.mark.parametrize("n,ctas", [(1, 147), (2, 147), (1, 146), (2, 115), (4, 147), (1, 144)])
def test_norm_vectors_of_every_layer_on_grids_that_are_no_multiple_of_four(C, fmt, n, ctas):
    """Six layers whose norm vectors differ from one another as much as from one (the two buffers of a CTA alternate by layer, so that
    two layers with the vectors of each other's predecessors would show nothing), on grids that leave CTAs without an O slice or are
    rounded down because of them.  One CTA's gate / up rows normalised with another layer's vector are 16 to 24 of 3072 in every layer: with
    logits of order one about sqrt(24 / 3072) = 0.09 of what the down products add, several times the bar of 3e-2."""
    import quantize as Q
    w = S.make_weights(seed=19, num_layers=6, vocab_size=2048, norm_std=0.7, max_seq_len=16)
    engine_w, oracle_w = Q.quantize_weights_fp8(w) if fmt == "fp8" else (w, w)
    prompts = [S.make_prompt(L, seed=90 + i, vocab_size=2048) for i, L in enumerate([150, 9, 70, 40][:n])]
    want, logits = _oracle(oracle_w, 320, prompts, 6)
    eng = _batch_engine(engine_w, n, 320, weight_format=fmt)
    C.configure(max_ctas=ctas)
    try:
        got, dump = _run_with_dump(C, eng, prompts, 6, 2048)
    finally:
        C.configure(max_ctas=0)
        C.set_weight_format("fp16")
    for b in range(n):
        assert got[b] == want[b]
        assert float((dump[b] - logits[b]).abs().max()) < LOGIT_TOL


@pytest.mark.parametrize("length", [2030, 2045])
def test_two_sequences_either_side_of_the_smaller_grid(C, length):
    """Two fp16 sequences take 128 CTAs up to 2048 positions and the whole device beyond (18 steps from 2030 end at 2047, from 2045 at
    2062): the oracle's tokens, logits within the bound of every launch."""
    w = S.make_weights(seed=31, num_layers=2, vocab_size=2048, norm_std=0.1, max_seq_len=16)
    prompts = [S.make_prompt(n, seed=80 + n, vocab_size=2048) for n in (length, 700)]
    want, logits = _oracle(w, 2080, prompts, 18)
    eng = _batch_engine(w, 2, 2080)
    got, dump = _run_with_dump(C, eng, prompts, 18, 2048)
    for b in range(2):
        assert got[b] == want[b]
        assert float((dump[b] - logits[b]).abs().max()) < LOGIT_TOL
