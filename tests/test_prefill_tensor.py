"""Tensor-core chunked prefill against the CPU oracle and against the ``prefill`` op.

The chunked path rounds GEMM operands to fp16 (the decode kernel and the oracle keep fp32 activations), so
the bar is a tolerance, stated here: KV cache rows within 2e-2 max-abs of the oracle's (values are O(1),
fp16-stored), first-step logits after the prefill within 3e-2 of the oracle's, and - on these seeds - the
same greedy tokens."""

import pytest
import torch

import synthetic as S
from oracle.decoder_ref import Decoder as OracleDecoder

pytestmark = pytest.mark.gpu
CACHE_TOL = 2e-2
LOGIT_TOL = 3e-2


@pytest.fixture(scope="module")
def C(built_library):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_megakernel_C
    return qwen_megakernel_C


def _engine(w, max_seq_len, mode, **kw):
    from Model.Qwen06B_architecture import Decoder
    return Decoder(weights=S.weights_to(w, "cuda"), tokenizer=S.StubTokenizer(-1, w["embed_weight"].shape[0]),
                   verbose=False, max_seq_len=max_seq_len, prefill_mode=mode, **kw)


@pytest.mark.parametrize("n_prompt", [1, 37, 128, 513, 700, 800, 2300])
def test_cache_and_next_tokens_match_oracle(C, n_prompt):
    """Prompt lengths below a tile, one tile exactly, several tiles with a ragged tail (an odd and an even number of row tiles with K
    of the O and down products in four parts on pairs of CTAs), and many."""
    vocab, steps, L = 2048, 4, 2560
    w = S.make_weights(seed=12, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    ids = S.make_prompt(n_prompt + 1, seed=n_prompt, vocab_size=vocab)
    o = OracleDecoder(w, max_seq_len=L)
    want, logits = o.generate_ids(ids, steps, keep_logits=True)
    eng = _engine(w, L, "tensor")
    dump = torch.zeros(steps, vocab, device="cuda")
    C.set_logits_dump(dump)
    try:
        got = eng.generate_ids(ids, steps)
    finally:
        C.set_logits_dump(None)
    n = n_prompt
    kerr = float((eng._k_cache[:, :, :n].float().cpu() - o.k_cache[:, :, :n].float()).abs().max())
    verr = float((eng._v_cache[:, :, :n].float().cpu() - o.v_cache[:, :, :n].float()).abs().max())
    lerr = float((dump.cpu() - logits).abs().max())
    print(f"prompt {n_prompt}: cache max err K {kerr:.2e} V {verr:.2e}; logits max err {lerr:.2e}")
    assert kerr < CACHE_TOL and verr < CACHE_TOL
    assert lerr < LOGIT_TOL
    assert got == want


def test_packed_fp8_weights_prefill_on_the_tensor_cores(C):
    """FP8-E4M3 rows stay packed in device memory; the prefill GEMMs expand them tile by tile.  Cache rows against the
    oracle on the dequantised weights, then greedy tokens through the persistent kernel (which reads the same rows)."""
    import quantize as Q
    vocab, steps, L, n = 2048, 4, 640, 333
    w = S.make_weights(seed=14, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    eng_w, ora_w = Q.quantize_weights_fp8(w)
    ids = S.make_prompt(n + 1, seed=77, vocab_size=vocab)
    o = OracleDecoder(ora_w, max_seq_len=L)
    want, _ = o.generate_ids(ids, steps)
    try:
        eng = _engine(eng_w, L, "tensor", weight_format="fp8")
        got = eng.generate_ids(ids, steps)
        kerr = float((eng._k_cache[:, :, :n].float().cpu() - o.k_cache[:, :, :n].float()).abs().max())
        verr = float((eng._v_cache[:, :, :n].float().cpu() - o.v_cache[:, :, :n].float()).abs().max())
    finally:
        C.set_weight_format("fp16")
    print(f"packed fp8 tensor prefill, prompt {n}: cache max err K {kerr:.2e} V {verr:.2e}")
    assert kerr < CACHE_TOL and verr < CACHE_TOL
    assert got == want


def test_appends_at_a_start_position_and_agrees_with_serial_prefill(C):
    """Prefill in two calls (the second starts at position 300) and compare with the ``prefill`` op in one call, and with the
    same op as persistent steps (``set_fused(0)``), which share no kernel with either."""
    vocab, L = 2048, 1024
    w = S.make_weights(seed=13, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    ids = S.make_prompt(900, seed=3, vocab_size=vocab)
    a = _engine(w, L, "tensor")
    a.prefill_ids(ids[:300])
    a.prefill_ids(ids[300:])
    b = _engine(w, L, "serial")
    b.prefill_ids(ids)
    assert a.position == b.position == 900
    kerr = float((a._k_cache[:, :, :900].float() - b._k_cache[:, :, :900].float()).abs().max())
    verr = float((a._v_cache[:, :, :900].float() - b._v_cache[:, :, :900].float()).abs().max())
    print(f"two-call tensor prefill vs serial prefill: K {kerr:.2e} V {verr:.2e}")
    assert kerr < CACHE_TOL and verr < CACHE_TOL
    b.reset()
    C.set_fused(fused=0)
    try:
        b.prefill_ids(ids)
    finally:
        C.set_fused(fused=2)
    for mine, steps in ((a._k_cache, b._k_cache), (a._v_cache, b._v_cache)):
        assert float((mine[:, :, :900].float() - steps[:, :, :900].float()).abs().max()) < CACHE_TOL


@pytest.mark.parametrize("n_prompt", [150, 900])
def test_table_rope_mode(C, n_prompt):
    """fp16 cos / sin tables instead of the fp32 in-library table, for a short chunk (block-per-row norm kernel, four K
    splits) and a longer one (warp-per-row norm kernel)."""
    vocab, L = 2048, 1024
    w = S.make_weights(seed=14, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=L)
    ids = S.make_prompt(n_prompt, seed=4, vocab_size=vocab)
    o = OracleDecoder(w, max_seq_len=L, rope_from_tables=True)
    want, _ = o.generate_ids(ids, 3)
    eng = _engine(w, L, "tensor", rope_from_table=True)
    try:
        got = eng.generate_ids(ids, 3)
        n = n_prompt - 1
        kerr = float((eng._k_cache[:, :, :n].float().cpu() - o.k_cache[:, :, :n].float()).abs().max())
    finally:
        C.configure(rope_from_table=0)
    assert kerr < CACHE_TOL and got == want


@pytest.mark.parametrize("impl", [0, 1])
def test_both_attention_kernels(C, impl):
    """The tcgen05 attention kernel (default) and the mma.sync one, each against the oracle on a two-chunk prompt
    whose second chunk starts inside a key tile (positions 2048 .. 2249)."""
    vocab, steps, L, n = 2048, 3, 2304, 2250
    w = S.make_weights(seed=15, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    ids = S.make_prompt(n + 1, seed=8, vocab_size=vocab)
    o = OracleDecoder(w, max_seq_len=L)
    want, logits = o.generate_ids(ids, steps, keep_logits=True)
    eng = _engine(w, L, "tensor")
    dump = torch.zeros(steps, vocab, device="cuda")
    C.set_prefill_attention(impl)
    C.set_logits_dump(dump)
    try:
        got = eng.generate_ids(ids, steps)
    finally:
        C.set_logits_dump(None)
        C.set_prefill_attention(1)
    kerr = float((eng._k_cache[:, :, :n].float().cpu() - o.k_cache[:, :, :n].float()).abs().max())
    verr = float((eng._v_cache[:, :, :n].float().cpu() - o.v_cache[:, :, :n].float()).abs().max())
    lerr = float((dump.cpu() - logits).abs().max())
    print(f"attention impl {impl}: cache max err K {kerr:.2e} V {verr:.2e}; logits max err {lerr:.2e}; tokens {got} / {want}; "
          f"per step {[float((dump[i].cpu() - logits[i]).abs().max()) for i in range(steps)]}")
    assert kerr < CACHE_TOL and verr < CACHE_TOL and lerr < LOGIT_TOL
    assert got == want


def test_decode_after_tensor_prefill_is_reproducible(C):
    """Prefill on the tensor cores, then greedy decode on the persistent kernel, eight times over: tokens and every
    logit must come out bit-identical (a prefill chain launched as programmatic dependents once left the decode that
    followed it different from run to run, with identical cache rows)."""
    vocab, steps, L, n = 2048, 3, 2560, 2300
    w = S.make_weights(seed=15, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    ids = S.make_prompt(n + 1, seed=8, vocab_size=vocab)
    eng = _engine(w, L, "tensor")
    runs = []
    for _ in range(8):
        dump = torch.zeros(steps, vocab, device="cuda")
        C.set_logits_dump(dump)
        try:
            got = eng.generate_ids(ids, steps)
        finally:
            C.set_logits_dump(None)
        runs.append((got, dump.cpu()))
    assert all(r[0] == runs[0][0] for r in runs)
    assert all(torch.equal(r[1], runs[0][1]) for r in runs)
    assert runs[0][0] == OracleDecoder(w, max_seq_len=L).generate_ids(ids, steps)[0]


def test_refusals(C):
    import quantize as Q
    w = S.make_weights(seed=1, num_layers=2, vocab_size=512, max_seq_len=16)
    with pytest.raises(ValueError):        # NVFP4 rows are read by the tensor-core ops only
        _engine(Q.quantize_weights_nvfp4(w)[0], 64, "serial", weight_format="nvfp4")
    eng = _engine(w, 64, "tensor")
    with pytest.raises(RuntimeError, match="max_seq_len"):
        eng.prefill_ids(list(range(65)))
    with pytest.raises(RuntimeError, match="vocab"):
        eng.prefill_ids([1, 600])
    eng.reset()
    assert len(eng.generate_ids([1, 2, 3], 2)) == 2


@pytest.mark.parametrize("fmt,n", [("fp8", 257), ("fp8", 385), ("nvfp4", 300), ("nvfp4", 385), ("nvfp4", 1100), ("fp8", 4200)])
def test_packed_weights_expanded_once_per_layer(C, fmt, n):
    """Chunks of 512 and more (padded) rows expand a packed layer's matrices once instead of inside the GEMMs: the shortest
    such chunk (385 tokens), ones below it, ragged ones, a length with the wide tiles and split K, two chunks of which the second is
    short.  The products are the same (exact values, row scale behind the sum), so the first layer's rows equal bit for bit
    those of calls that stay below the switch; from 1024 rows on the RMSNorm kernel adds its squares in another order, which
    moves single operands to the neighbouring fp16 (2^-11 of one of 1024 products): one unit in the last place of a row's
    value, 2^-8 below 8.  Later layers to the rounding of other tiles and splits, like every two passes of this path (1e-2)."""
    import quantize as Q
    vocab, L = 2048, 4224
    w = S.make_weights(seed=33, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    eng_w, _ = (Q.quantize_weights_fp8 if fmt == "fp8" else Q.quantize_weights_nvfp4)(w)
    ids = S.make_prompt(n, seed=n, vocab_size=vocab)
    try:
        a = _engine(eng_w, L, "tensor", weight_format=fmt)
        b = _engine(eng_w, L, "tensor", weight_format=fmt)
        a.prefill_ids(ids)
        for i in range(0, n, 250):
            b.prefill_ids(ids[i:i + 250])
    finally:
        C.set_weight_format("fp16")
    for x, y in ((a._k_cache[:, :, :n], b._k_cache[:, :, :n]), (a._v_cache[:, :, :n], b._v_cache[:, :, :n])):
        first, diff = float((x[0].float() - y[0].float()).abs().max()), float((x.float() - y.float()).abs().max())
        print(f"{fmt} {n}: max difference {diff:.2e}, first layer {first:.2e}")
        assert first <= (2.0 ** -8 if n >= 1024 else 0.0) and float(x[0].abs().max()) < 8.0
        assert diff < 1e-2


@pytest.mark.parametrize("fmt,lens", [("fp16", [31]), ("fp16", [129]), ("fp16", [513]), ("fp16", [1409]), ("fp16", [4225]), ("fp8", [129]), ("fp8", [257]),
                                      ("nvfp4", [128]), ("nvfp4", [1025]), ("fp16", [1, 37, 300, 1000]), ("nvfp4", [128, 700, 64]), ("fp8", [200, 3])])
def test_launch_overlap_changes_nothing_but_time(C, fmt, lens):
    """The kernels of a pass start under the tails of their predecessors (``set_step_overlap``); launched one after the other
    they leave the same cache rows, bit for bit.  One chunk of each of the launch rules - one tile, K split four ways with each
    tile width, two chunks - packed matrices inside the GEMMs and expanded per layer, several prompts in a pass."""
    import quantize as Q
    from Model.Qwen06B_architecture import BatchDecoder
    vocab, L = 2048, 4352 if max(lens) > 2048 else 1536
    w = S.make_weights(seed=41, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    if fmt != "fp16":
        w, _ = (Q.quantize_weights_fp8 if fmt == "fp8" else Q.quantize_weights_nvfp4)(w)
    prompts = [S.make_prompt(n, seed=n, vocab_size=vocab) for n in lens]
    try:
        if len(lens) == 1:
            one = _engine(w, L, "tensor", weight_format=fmt)
            caches = [one._k_cache, one._v_cache]
        else:
            many = BatchDecoder(weights=S.weights_to(w, "cuda"), tokenizer=S.StubTokenizer(-1, vocab), num_sequences=len(lens),
                                max_seq_len=L, engine="gemm", prefill_mode="tensor", weight_format=fmt)
            caches = list(many._k_caches) + list(many._v_caches)
        rows = {}
        for overlap in (True, False, True, True):
            C.set_step_overlap(overlap)
            for c in caches:
                c.zero_()
            if len(lens) == 1:
                one.reset()
                one.prefill_ids(prompts[0])
            else:
                many.prefill_slots(list(range(len(lens))), prompts)
            got = [c.clone() for c in caches]
            assert all(torch.equal(a, b) for a, b in zip(got, rows.setdefault(0, got)))
        assert all(bool(torch.isfinite(c.float()).all()) and float(c.float().abs().max()) > 0.1 for c in rows[0])
    finally:
        C.set_step_overlap(True)
        C.set_weight_format("fp16")


@pytest.mark.parametrize("before,n", [(0, 64), (0, 65), (0, 129), (0, 320), (77, 51), (63, 1), (1000, 200), (130, 1500), (0, 4225)])
def test_attention_kernels_agree(C, before, n):
    """The tcgen05 attention against the mma.sync kernel on the same chunk: less than a key tile, one key over, an odd and an even
    number of key tiles, prompts that continue at a position inside a tile (so that the diagonal crosses it), two
    chunks.  Both round queries, keys and softmax weights to fp16 and
    add in fp32; what differs is the order of sums: 1e-2 on cache values, as between any two passes of this path."""
    vocab, L = 2048, 4352 if n > 2048 else 2048
    w = S.make_weights(seed=51, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    ids = S.make_prompt(before + n, seed=n, vocab_size=vocab)
    eng = _engine(w, L, "tensor")
    rows = []
    try:
        for kernel in (1, 0, 1):
            C.set_prefill_attention(kernel)
            eng.reset()
            for cache in (eng._k_cache, eng._v_cache):
                cache.fill_(float("nan") if kernel else 0.0)      # (rows behind the prompt do not reach the tcgen05 kernel)
            if before:
                eng.prefill_ids(ids[:before])
            eng.prefill_ids(ids[before:])
            rows.append((eng._k_cache[:, :, :before + n].float().clone(), eng._v_cache[:, :, :before + n].float().clone()))
    finally:
        C.set_prefill_attention(1)
    for a, b, again in zip(*rows):
        assert bool(torch.isfinite(a).all()) and torch.equal(a, again)
        assert float((a - b).abs().max()) < 1e-2


@pytest.mark.parametrize("fmt,cuts", [("fp16", (1100, 4000)), ("fp16", (1500, 3000, 4096)), ("fp16", (2900, 4000)), ("fp16", (4096, 7500)),
                                      ("nvfp4", (1100, 2300)), ("fp16", (400, 800)), ("fp16", (400, 513)), ("fp16", (130, 640)), ("fp8", (400, 800)),
                                      ("nvfp4", (385, 770))])
def test_rows_do_not_depend_on_how_a_prompt_is_cut(C, fmt, cuts):
    """A prompt in one call and in calls of 1024 tokens and more: every product then adds in the same order (K of the O and
    down products in two parts, the keys of a query in the same tiles and chains), so the cache rows are equal bit for bit.  So
    are those of a prompt below 1024 tokens on pairs of CTAs and its pieces of at most 512 on single ones (K in four parts,
    one RMSNorm kernel): every epilogue of either kernel, with row scales too."""
    import quantize as Q
    vocab, L = 2048, 7680 if cuts[-1] > 4300 else 4352
    w = S.make_weights(seed=61, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    if fmt != "fp16":
        w, _ = (Q.quantize_weights_fp8 if fmt == "fp8" else Q.quantize_weights_nvfp4)(w)
    ids = S.make_prompt(cuts[-1], seed=len(cuts), vocab_size=vocab)
    try:
        one, parts = (_engine(w, L, "tensor", weight_format=fmt) for _ in range(2))
        one.prefill_ids(ids)
        for a, b in zip((0,) + cuts, cuts):
            parts.prefill_ids(ids[a:b])
    finally:
        C.set_weight_format("fp16")
    for x, y in ((one._k_cache, parts._k_cache), (one._v_cache, parts._v_cache)):
        assert float(x[:, :, :cuts[-1]].float().abs().max()) > 0.1
        assert torch.equal(x[:, :, :cuts[-1]], y[:, :, :cuts[-1]])


@pytest.mark.parametrize("fmt,cuts", [("fp16", (1200, 2304)), ("fp16", (1200, 2305)), ("fp16", (1153, 2560)), ("nvfp4", (1300, 3585)),
                                      ("fp8", (2200, 4095))])
def test_residual_adds_in_the_epilogue_keep_the_bits(C, fmt, cuts):
    """From 2305 tokens on (ten row tiles) the O and down products add both parts to the residual rows themselves; the pieces of
    the prompt stay below and leave the partial matrices to the RMSNorm kernel.  Either side of the line, rows that end with a
    tile and one behind it, row scales."""
    test_rows_do_not_depend_on_how_a_prompt_is_cut(C, fmt, cuts)


@pytest.mark.parametrize("fmt,table_rope,lens", [("fp16", False, (513,)), ("fp16", True, (777,)), ("nvfp4", False, (1025,)), ("fp8", False, (640, 2400)),
                                                 ("fp16", False, (544, 4095, 1000))])
def test_heads_stored_by_the_product_keep_the_bits(C, fmt, table_rope, lens):
    """Chunks on pairs of CTAs normalise, rotate and store q, k and v in the product's epilogue; with the other attention kernel
    selected a kernel of its own does it.  The first layer's rows do not depend on the attention: equal bit for bit, for rows
    that end inside a warp's 32, behind a start position, with row scales, and nothing is written behind them."""
    import quantize as Q
    vocab, n = 2048, sum(lens)
    w = S.make_weights(seed=71, num_layers=1, vocab_size=vocab, norm_std=0.1, max_seq_len=n + 40 if table_rope else 16)
    if fmt != "fp16":
        w, _ = (Q.quantize_weights_fp8 if fmt == "fp8" else Q.quantize_weights_nvfp4)(w)
    ids = S.make_prompt(n, seed=8, vocab_size=vocab)
    rows = []
    try:
        eng = _engine(w, n + 40, "tensor", weight_format=fmt, rope_from_table=table_rope)
        for impl in (1, 0):
            C.set_prefill_attention(impl)
            eng.reset()
            eng._k_cache.zero_(), eng._v_cache.zero_()
            at = 0
            for length in lens:
                eng.prefill_ids(ids[at:at + length])
                at += length
            rows.append((eng._k_cache.clone(), eng._v_cache.clone()))
    finally:
        C.set_prefill_attention(1)
        C.configure(rope_from_table=0)
        C.set_weight_format("fp16")
    for x, y in zip(*rows):
        assert float(x[:, :, :n].float().abs().max()) > 0.1 and float(x[:, :, n:].float().abs().max()) == 0
        assert torch.equal(x, y)


def test_heads_of_packed_prompts_keep_the_bits(C):
    """Packed prompts of 896 rows (the pairs' product stores the heads) and the same prompts on their own (a kernel does)."""
    from Model.Qwen06B_architecture import BatchDecoder
    vocab, lens = 2048, [1, 37, 300, 129]
    w = S.weights_to(S.make_weights(seed=72, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16), "cuda")
    eng = BatchDecoder(weights=w, tokenizer=S.StubTokenizer(-1, vocab), num_sequences=4, max_seq_len=400, engine="gemm", prefill_mode="tensor")
    prompts = [S.make_prompt(n, seed=80 + n, vocab_size=vocab) for n in lens]
    for b, ids in enumerate(prompts):
        eng.prefill_slot(b, ids)
    want = [(k.clone(), v.clone()) for k, v in zip(eng._k_caches, eng._v_caches)]
    for k, v in zip(eng._k_caches, eng._v_caches):
        k.zero_(), v.zero_()
    eng.prefill_slots(list(range(4)), prompts)
    for b, (k, v) in enumerate(want):
        assert torch.equal(eng._k_caches[b], k) and torch.equal(eng._v_caches[b], v), b


def test_attention_waits_run_out_and_leave_the_device_usable(C):
    """Score products that stop behind the first, with keys and values in flight: status 4 after the budget, copies landed and TMEM
    freed (the prefill behind it allocates all of it on every SM), rows as before."""
    w = S.make_weights(seed=71, num_layers=2, vocab_size=2048, norm_std=0.1, max_seq_len=16)
    ids = S.make_prompt(1300, seed=1, vocab_size=2048)
    eng = _engine(w, 1536, "tensor")
    eng.prefill_ids(ids)
    before = eng._k_cache.clone(), eng._v_cache.clone()
    for _ in range(3):
        assert C.selftest_attention_wait_timeout(300) == 4
        eng.reset()
        eng.prefill_ids(ids)
        assert torch.equal(eng._k_cache, before[0]) and torch.equal(eng._v_cache, before[1])
