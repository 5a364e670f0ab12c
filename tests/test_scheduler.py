"""Continuous batching scheduler: host logic against a fake engine (CPU), and end to end on the GPU
against the single-sequence engine."""

import pytest
import torch

import synthetic as S
from scheduler import ContinuousBatcher


class FakeEngine:
    """Deterministic stand-in: the token after ``t`` at cache position ``p`` is ``(7 t + 3 p + 1) % 97``.
    Records what the scheduler asked for."""

    def __init__(self, num_sequences=4, max_seq_len=64):
        self.num_sequences, self.max_seq_len = num_sequences, max_seq_len
        self.positions = [0] * num_sequences
        self.launch_log = []

    @staticmethod
    def nxt(t, p):
        return (7 * t + 3 * p + 1) % 97

    def prefill_slot(self, b, ids):
        if any(t < 0 for t in ids):
            raise RuntimeError("bad token")
        self.positions[b] = len(ids)

    def decode_slots(self, slots, firsts, steps):
        self.launch_log.append((tuple(slots), steps))
        out = []
        for b, t in zip(slots, firsts):
            toks = []
            for _ in range(steps):
                t = self.nxt(t, self.positions[b])
                self.positions[b] += 1
                toks.append(t)
            out.append(toks)
        return out

    @classmethod
    def reference(cls, ids, n, eos=-1):
        t, p, out = ids[-1], len(ids) - 1, []
        for _ in range(n):
            t = cls.nxt(t, p)
            p += 1
            if t == eos:
                return out, "stop"
            out.append(t)
        return out, "length"


def test_every_request_matches_its_own_sequential_run():
    eng = FakeEngine(num_sequences=3)
    sch = ContinuousBatcher(eng, eos_token_id=None, quantum=5)
    reqs = [(S.make_prompt(1 + (i * 5) % 11, seed=i, vocab_size=97), 1 + (i * 7) % 23) for i in range(17)]
    futs = [sch.submit(ids, n) for ids, n in reqs]
    sch.run_until_idle()
    for (ids, n), f in zip(reqs, futs):
        r = f.result(timeout=0)
        want, why = FakeEngine.reference(ids, n)
        assert r.tokens == want and r.finish_reason == why == "length" and r.prompt_tokens == len(ids)
    assert sch.max_live == 3                                   # the slots were actually shared
    assert all(len(s) <= 3 and 1 <= q <= 5 for s, q in eng.launch_log)
    assert sch.launches == len(eng.launch_log) < sum(n for _, n in reqs)   # fewer launches than tokens
    # arrival order is admission order: request ids are handed out in submit order
    assert [f.result().rid for f in futs] == list(range(17))


def test_eos_frees_the_slot_and_is_not_returned():
    ids, n = [5, 9, 2], 30
    full, _ = FakeEngine.reference(ids, n)
    eos = full[4]
    eng = FakeEngine(num_sequences=2)
    sch = ContinuousBatcher(eng, eos_token_id=eos, quantum=3)
    f1 = sch.submit(ids, n)
    f2 = sch.submit([1, 2, 3, 4], 9)
    f3 = sch.submit([8], 4)                                    # waits for a slot
    sch.run_until_idle()
    want, why = FakeEngine.reference(ids, n, eos)
    assert why == "stop" and f1.result().tokens == want == full[:full.index(eos)]
    assert f1.result().finish_reason == "stop"
    for f, (i, k) in ((f2, ([1, 2, 3, 4], 9)), (f3, ([8], 4))):
        w, y = FakeEngine.reference(i, k, eos)
        assert f.result().tokens == w and f.result().finish_reason == y


def test_quantum_never_overruns_a_budget_and_bad_requests_fail_alone():
    eng = FakeEngine(num_sequences=2, max_seq_len=16)
    sch = ContinuousBatcher(eng, quantum=8)
    ok = sch.submit([3, 4], 3)
    too_long = sch.submit(list(range(10)), 10)                 # 9 + 10 > 16
    empty = sch.submit([], 4)
    zero = sch.submit([1, 2], 0)
    bad = sch.submit([5, -1, 7], 2)                            # the engine refuses the prompt
    later = sch.submit([6], 11)
    sch.run_until_idle()
    assert ok.result().tokens == FakeEngine.reference([3, 4], 3)[0]
    assert later.result().tokens == FakeEngine.reference([6], 11)[0]
    assert zero.result().tokens == []
    with pytest.raises(ValueError):
        too_long.result()
    with pytest.raises(ValueError):
        empty.result()
    with pytest.raises(RuntimeError):
        bad.result()
    # the first launch carried both live requests and stopped at the shorter budget
    assert eng.launch_log[0] == ((0, 1), 3)
    for b in range(2):
        assert eng.positions[b] <= 16


def test_background_thread_serves_submissions():
    eng = FakeEngine(num_sequences=4)
    sch = ContinuousBatcher(eng, quantum=4)
    sch.start()
    try:
        futs = [(ids, n, sch.submit(ids, n)) for ids, n in (([2, 3], 6), ([9], 13), ([4, 4, 4], 2))]
        for ids, n, f in futs:
            assert f.result(timeout=10).tokens == FakeEngine.reference(ids, n)[0]
    finally:
        sch.stop()


@pytest.mark.gpu
def test_gpu_continuous_batching_equals_single_sequence_engine(built_library, tiny_cfg):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from Model.Qwen06B_architecture import BatchDecoder, Decoder
    vocab = tiny_cfg["vocab_size"]
    w = S.weights_to(S.make_weights(seed=tiny_cfg["seed"], num_layers=tiny_cfg["num_layers"], vocab_size=vocab,
                                    norm_std=tiny_cfg["norm_std"], max_seq_len=16), "cuda")
    tok = S.StubTokenizer(-1, vocab)
    eng = BatchDecoder(weights=w, tokenizer=tok, num_sequences=4, max_seq_len=256, engine="persistent")
    reqs = [(S.make_prompt(3 + (i * 13) % 60, seed=100 + i, vocab_size=vocab), 4 + (i * 5) % 29) for i in range(11)]
    single = Decoder(weights=w, tokenizer=tok, verbose=False, max_seq_len=256)
    want = [single.generate_ids(ids, n) for ids, n in reqs]
    eos = want[2][3]                                           # a token that really occurs
    sch = ContinuousBatcher(eng, eos_token_id=eos, quantum=8)
    futs = [sch.submit(ids, n) for ids, n in reqs]
    sch.run_until_idle()
    for w_, f, (ids, n) in zip(want, futs, reqs):
        r = f.result(timeout=0)
        cut = w_[:w_.index(eos)] if eos in w_ else w_
        assert r.tokens == cut
        assert r.finish_reason == ("stop" if eos in w_ else "length")
    assert sch.max_live == 4 and sch.launches < sum(n for _, n in reqs)


def test_random_workloads_property():
    """Property test over random request mixes, slot counts, quanta and EOS ids: every request's answer equals
    its own sequential run, the slot limit holds, nobody overruns a budget, all futures resolve."""
    hypothesis = pytest.importorskip("hypothesis")
    from hypothesis import given, settings, strategies as st

    req = st.tuples(st.lists(st.integers(0, 96), min_size=1, max_size=12), st.integers(0, 40))

    @settings(max_examples=60, deadline=None)
    @given(reqs=st.lists(req, min_size=1, max_size=25), slots=st.integers(1, 9), quantum=st.integers(1, 17),
           eos=st.one_of(st.none(), st.integers(0, 96)))
    def run(reqs, slots, quantum, eos):
        eng = FakeEngine(num_sequences=slots, max_seq_len=64)
        sch = ContinuousBatcher(eng, eos_token_id=eos, quantum=quantum)
        futs = [sch.submit(ids, n) for ids, n in reqs]
        sch.run_until_idle()
        for (ids, n), f in zip(reqs, futs):
            r = f.result(timeout=0)
            want, why = FakeEngine.reference(ids, n, -1 if eos is None else eos) if n > 0 else ([], "length")
            assert r.tokens == want and r.finish_reason == why
        assert sch.max_live <= slots
        assert all(len(s) <= slots and len(set(s)) == len(s) and 1 <= q <= quantum for s, q in eng.launch_log)
        assert all(p <= 64 for p in eng.positions)

    run()


def test_overlapped_admission_gives_the_same_answers():
    """Prefill on its own thread: same tokens per request, slot limit respected, everything resolves; the fake
    engine's prefill sleeps so that decode rounds really run while a prefill is in flight."""
    import time

    class SlowPrefill(FakeEngine):
        def __init__(self, *a, **k):
            super().__init__(*a, **k)
            self.concurrent = 0

        def prefill_slot(self, b, ids):
            time.sleep(0.004)
            super().prefill_slot(b, ids)

        def decode_slots(self, slots, firsts, steps):
            time.sleep(0.001)
            return super().decode_slots(slots, firsts, steps)

    eng = SlowPrefill(num_sequences=3)
    sch = ContinuousBatcher(eng, eos_token_id=None, quantum=4, overlap_prefill=True)
    reqs = [(S.make_prompt(1 + (i * 5) % 11, seed=i, vocab_size=97), 2 + (i * 7) % 19) for i in range(14)]
    futs = [sch.submit(ids, n) for ids, n in reqs]
    sch.run_until_idle()
    sch.stop()
    for (ids, n), f in zip(reqs, futs):
        assert f.result(timeout=0).tokens == FakeEngine.reference(ids, n)[0]
    assert sch.max_live <= 3 and all(len(s) <= 3 for s, _ in eng.launch_log)
    # decode rounds with fewer than all slots live happened while later prefills were still running
    assert any(len(s) < 3 for s, _ in eng.launch_log[:5])


def test_live_limit_keeps_spare_slots_for_prefilled_requests():
    """With ``live_limit`` below the engine's slot count no launch carries more sequences than the limit; the other
    slots hold prefilled requests that take a seat as soon as one frees up, and every answer is still its own."""
    eng = FakeEngine(num_sequences=6)
    sch = ContinuousBatcher(eng, eos_token_id=None, quantum=4, live_limit=3)
    reqs = [(S.make_prompt(2 + (i * 3) % 7, seed=i, vocab_size=97), 3 + (i * 5) % 17) for i in range(14)]
    futs = [sch.submit(ids, n) for ids, n in reqs]
    sch.run_until_idle()
    sch.stop()
    for (ids, n), f in zip(reqs, futs):
        assert f.result(timeout=0).tokens == FakeEngine.reference(ids, n)[0]
    assert sch.max_live == 3 and all(len(s) <= 3 for s, _ in eng.launch_log)
    full = sum(1 for s, _ in eng.launch_log if len(s) == 3)
    assert full >= len(eng.launch_log) - 4        # seats are refilled at once: only the last rounds run short
    with pytest.raises(ValueError):
        ContinuousBatcher(eng, live_limit=0)


def test_waiting_requests_are_prefilled_together_when_the_engine_can():
    """An engine with ``prefill_slots`` gets every waiting request that fits its row budget in one call (prompts
    padded to multiples of 128 rows); a failing group falls back to one pass per request."""
    class Packing(FakeEngine):
        packed_prefill_rows = 512

        def __init__(self, **kw):
            super().__init__(**kw)
            self.groups = []

        def prefill_slots(self, slots, prompts):
            self.groups.append([len(p) for p in prompts])
            if any(t < 0 for p in prompts for t in p):
                raise RuntimeError("bad token")
            for b, p in zip(slots, prompts):
                self.positions[b] = len(p)

    eng = Packing(num_sequences=6, max_seq_len=400)
    sch = ContinuousBatcher(eng, eos_token_id=None, quantum=4)
    lens = [5, 130, 100, 300, 2, 7]            # rows 128 + 256 + 128 | 384 + 128 | 128
    reqs = [(S.make_prompt(n, seed=i, vocab_size=97), 6) for i, n in enumerate(lens)]
    reqs[4] = ([-3, 5], 6)                      # prompt_ids[:-1] holds a bad token: its group fails as a whole
    futs = [sch.submit(ids, n) for ids, n in reqs]
    sch.run_until_idle()
    sch.stop()
    assert eng.groups[0] == [4, 129, 99] and eng.groups[1] == [299, 1]
    for i, ((ids, n), f) in enumerate(zip(reqs, futs)):
        if i == 4:
            with pytest.raises(RuntimeError):
                f.result(timeout=0)
        else:
            assert f.result(timeout=0).tokens == FakeEngine.reference(ids, n)[0]


@pytest.mark.gpu
@pytest.mark.parametrize("table_rope", [False, True])
def test_gpu_packed_prefill_matches_one_prompt_per_pass(built_library, table_rope):
    """Several prompts through one tensor-core pass (``prefill_slots``): every slot's cache rows agree with a pass of
    its own to the rounding of a different GEMM tiling, and the tokens decoded from them are the same.  Also with
    the rotary angles read from the fp16 cos / sin tables."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_megakernel_C as C
    from Model.Qwen06B_architecture import BatchDecoder
    vocab = 2048
    w = S.weights_to(S.make_weights(seed=9, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=16), "cuda")
    tok = S.StubTokenizer(-1, vocab)
    lens = [1, 37, 128, 129, 300, 700, 64, 1000]
    prompts = [S.make_prompt(n + 1, seed=300 + i, vocab_size=vocab) for i, n in enumerate(lens)]
    if table_rope:
        w = S.weights_to(S.make_weights(seed=9, num_layers=3, vocab_size=vocab, norm_std=0.1, max_seq_len=1100), "cuda")
    eng = BatchDecoder(weights=w, tokenizer=tok, num_sequences=len(lens), max_seq_len=1100, engine="gemm", prefill_mode="tensor",
                       rope_from_table=table_rope)
    try:
        _packed_against_single(eng, lens, prompts)
    finally:
        C.configure(rope_from_table=0)


def _packed_against_single(eng, lens, prompts):
    for b, ids in enumerate(prompts):
        eng.prefill_slot(b, ids[:-1])
    want_k = [eng._k_caches[b].clone() for b in range(len(lens))]
    want_v = [eng._v_caches[b].clone() for b in range(len(lens))]
    want = eng.decode_slots(list(range(len(lens))), [ids[-1] for ids in prompts], 12)
    for b in range(len(lens)):
        eng._k_caches[b].zero_()
        eng._v_caches[b].zero_()
    eng.prefill_slots(list(range(len(lens))), [ids[:-1] for ids in prompts])   # 128 + 128 + 128 + 256 + 384 + 768 + 128 + 1024 rows
    assert eng.positions == lens
    for b, n in enumerate(lens):
        got_k = eng._k_caches[b].view(3, 8, -1, 128)[:, :, :n].float()
        ref_k = want_k[b].view(3, 8, -1, 128)[:, :, :n].float()
        got_v = eng._v_caches[b].view(3, 8, -1, 128)[:, :, :n].float()
        ref_v = want_v[b].view(3, 8, -1, 128)[:, :, :n].float()
        assert (got_k - ref_k).abs().max().item() < 1e-2 and (got_v - ref_v).abs().max().item() < 1e-2   # fp16 operands, other tile shapes
        # rows past the prompt stay untouched
        assert eng._k_caches[b].view(3, 8, -1, 128)[:, :, n:].abs().max().item() == 0
    got = eng.decode_slots(list(range(len(lens))), [ids[-1] for ids in prompts], 12)
    assert got == want


@pytest.mark.gpu
def test_gpu_overlapped_prefill_matches_serial_scheduling(built_library, tiny_cfg):
    """Tensor-core engines, 8 slots: prefill of the next request on its own stream and thread while the live
    ones decode.  A sequence's tokens do not depend on who shares its launches, so both schedules must agree."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from Model.Qwen06B_architecture import BatchDecoder
    vocab = 2048
    w = S.weights_to(S.make_weights(seed=5, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16), "cuda")
    tok = S.StubTokenizer(-1, vocab)
    reqs = [(S.make_prompt(3 + (i * 37) % 300, seed=200 + i, vocab_size=vocab), 4 + (i * 5) % 23) for i in range(20)]
    outs = []
    for overlap in (False, True):
        eng = BatchDecoder(weights=w, tokenizer=tok, num_sequences=8, max_seq_len=384, engine="gemm", prefill_mode="tensor")
        assert eng.supports_overlap
        # (one prefill pass per request: with packed passes a cache's last bits depend on the group's GEMM tiling, and
        # the two schedules form different groups)
        sch = ContinuousBatcher(eng, eos_token_id=None, quantum=8, overlap_prefill=overlap, packed_prefill=False)
        futs = [sch.submit(ids, n) for ids, n in reqs]
        sch.run_until_idle()
        sch.stop()
        outs.append([f.result(timeout=0).tokens for f in futs])
        assert all(len(t) == n for t, (_, n) in zip(outs[-1], reqs))
    assert outs[0] == outs[1]


@pytest.mark.gpu
@pytest.mark.parametrize("overlap", [False, True])
def test_gpu_four_slots_with_tensor_prefill(built_library, overlap):
    """What a four-slot server runs: the persistent engine with prefills on the tensor cores between its rounds.  It offers no
    overlap; a caller that asks for it all the same gets the same answers.  Each request's tokens equal those of the
    single-sequence engine behind the same prefill."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from Model.Qwen06B_architecture import BatchDecoder, Decoder
    vocab = 2048
    w = S.weights_to(S.make_weights(seed=5, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16), "cuda")
    tok = S.StubTokenizer(-1, vocab)
    reqs = [(S.make_prompt(3 + (i * 37) % 300, seed=200 + i, vocab_size=vocab), 4 + (i * 5) % 23) for i in range(12)]
    single = Decoder(weights=w, tokenizer=tok, verbose=False, max_seq_len=384, prefill_mode="tensor")
    want = [single.generate_ids(ids, n) for ids, n in reqs]
    eng = BatchDecoder(weights=w, tokenizer=tok, num_sequences=4, max_seq_len=384, prefill_mode="tensor")
    assert eng.engine == "persistent" and not eng.supports_overlap
    sch = ContinuousBatcher(eng, eos_token_id=None, quantum=8, overlap_prefill=overlap, packed_prefill=False)
    futs = [sch.submit(ids, n) for ids, n in reqs]
    sch.run_until_idle()
    sch.stop()
    assert [f.result(timeout=0).tokens for f in futs] == want


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["fp16", "fp8"])
def test_gpu_packed_passes_of_one_call(built_library, fmt):
    """Four packed passes (4096, 4096, 3968 and 768 rows) sent to the device in one call, each prepared while the one before
    runs, leave the cache rows of four calls bit for bit: the same kernels on the same rows.  A prompt on its own between
    two groups still takes the chunked pass.  A pass that is refused is reported, and the next call works."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_megakernel_C as C
    import quantize as Q
    from Model.Qwen06B_architecture import BatchDecoder
    vocab = 2048
    w = S.make_weights(seed=9, num_layers=2, vocab_size=vocab, norm_std=0.1, max_seq_len=16)
    if fmt == "fp8":
        w, _ = Q.quantize_weights_fp8(w)
    lens = [1900, 2100, 4000, 2000, 1, 1900, 60, 1500, 1280, 1000, 0, 700, 60]
    prompts = [S.make_prompt(n, seed=500 + i, vocab_size=vocab) if n else [] for i, n in enumerate(lens)]
    eng = BatchDecoder(weights=S.weights_to(w, "cuda"), tokenizer=S.StubTokenizer(-1, vocab), num_sequences=len(lens), max_seq_len=4096,
                       engine="gemm", prefill_mode="tensor", weight_format=fmt)
    try:
        groups = [[0, 1], [2], [3, 4, 5], [6, 7, 8, 9, 10], [11, 12]]
        for g in groups:
            if len(g) == 1:
                eng.prefill_slot(g[0], prompts[g[0]])
            else:
                eng.prefill_slots(g, [prompts[b] for b in g])
        want = [(k.clone(), v.clone()) for k, v in zip(eng._k_caches, eng._v_caches)]
        for k, v in zip(eng._k_caches, eng._v_caches):
            k.zero_()
            v.zero_()
        for _ in range(2):
            eng.prefill_many(list(range(len(lens))), prompts)
            assert eng.positions == lens
            for b, (k, v) in enumerate(want):
                assert torch.equal(eng._k_caches[b], k) and torch.equal(eng._v_caches[b], v), b
        with pytest.raises(RuntimeError, match="vocab"):
            eng.prefill_many([0, 1, 3, 5, 7], [prompts[0], prompts[1][:-1], prompts[3], prompts[5][:-1] + [vocab], prompts[7]])
        assert eng.positions[:2] == [lens[0], lens[1] - 1] and eng.positions[3] == lens[3] and eng.positions[5] == lens[5]
        eng.prefill_many([0, 1, 3, 5, 7], [prompts[b] for b in (0, 1, 3, 5, 7)])
        for b in (0, 1, 3, 5, 7):
            assert torch.equal(eng._k_caches[b][:, :, :lens[b]], want[b][0][:, :, :lens[b]])
    finally:
        C.set_weight_format("fp16")


def _host_only_engine(monkeypatch, op):
    """A batched engine of six slots whose packed passes are calls of ``op``; its caches are their slots' numbers."""
    from types import SimpleNamespace
    from Model import Qwen06B_architecture as A
    monkeypatch.setattr(A, "_require_megakernel_op", lambda name: op)
    eng = object.__new__(A.BatchDecoder)
    eng.num_sequences, eng.max_seq_len, eng.positions, eng._prefill_stream = 6, 4096, [7] * 6, None
    eng._k_caches = eng._v_caches = list(range(6))
    eng._base = SimpleNamespace(prefill_mode="tensor", apply_options=lambda: None, _embed_weight=None, _layer_weights_packed=None, _cos_table=None,
                                _sin_table=None, num_layers=1, _attn_scale=1.0)
    return eng


def test_slots_of_packed_passes_are_whole_numbers(built_library, monkeypatch):
    """Whatever int() takes names a slot, and a slot named twice in a pass is refused whatever type its names have."""
    seen = []
    eng = _host_only_engine(monkeypatch, lambda counts, lists, *args: seen.extend(args[4]))
    eng.prefill_many(torch.tensor([1.0, 4.0, 0.0]), [[1, 2], [3], [4, 5, 6]])
    assert seen == [1, 4, 0] and eng.positions == [3, 2, 7, 7, 1, 7]
    with pytest.raises(ValueError, match="distinct"):
        eng.prefill_many(torch.tensor([1, 1]), [[1, 2], [3]])
    assert seen == [1, 4, 0]


@pytest.mark.parametrize("failure", ["refused", "device"])
def test_positions_after_packed_passes_that_failed(built_library, monkeypatch, failure):
    """Three packed passes in one call.  One that is refused (the passes in front of it have run then, those behind have not), or a device
    failure of the call: the position of a slot is that of the prompt whose rows it holds."""
    rows = {b: 7 for b in range(6)}
    calls = []

    def op(counts, token_lists, *args):
        calls.append(counts)
        at = 0
        for p, n in enumerate(counts):
            if any(t >= 100 for ids in token_lists[at:at + n] for t in ids):
                raise RuntimeError("prompt token outside [0, vocab)")
            for cache, ids in zip(args[4][at:at + n], token_lists[at:at + n]):
                rows[cache] = len(ids)
            at += n
        if failure == "device" and len(calls) == 1:
            raise RuntimeError("a bounded device wait ran out")
    eng = _host_only_engine(monkeypatch, op)
    prompts = [[1] * 2000, [2] * 1900, [3] * 2048, [100 if failure == "refused" else 4] * 2048, [5] * 3000, [6] * 900]
    if failure == "refused":
        with pytest.raises(RuntimeError, match="vocab"):
            eng.prefill_many(range(6), prompts)
        assert eng.positions[:2] == [2000, 1900] and eng.positions[3] == 7
    else:
        eng.prefill_many(range(6), prompts)
        assert eng.positions == [len(ids) for ids in prompts]
    assert calls[0] == [2, 2, 2]
    assert all(eng.positions[b] == rows[b] for b in range(6))
    with pytest.raises(RuntimeError, match="vocab"):
        eng.prefill_slots([0, 1], [[1], [100]])          # one pass: as it was
    assert eng.positions[:2] == ([2000, 1900])


def _passes(C, w, vocab, lens, seed, fmt="fp16"):
    """A batched engine and the arguments that send one packed pass of its own for every prompt in one call."""
    from Model.Qwen06B_architecture import BatchDecoder
    eng = BatchDecoder(weights=w, tokenizer=S.StubTokenizer(-1, vocab), num_sequences=len(lens), max_seq_len=max(lens), engine="gemm",
                       prefill_mode="tensor", weight_format=fmt)
    base = eng._base
    prompts = [S.make_prompt(n, seed=seed + i, vocab_size=vocab) for i, n in enumerate(lens)]
    return eng, ([1] * len(lens), prompts, base._embed_weight, base._layer_weights_packed, base._cos_table, base._sin_table, eng._k_caches,
                 eng._v_caches, base.num_layers, eng.max_seq_len, base._attn_scale)


def _when_rows_appear(cache, do):
    """A thread that calls `do` as soon as the first pass has written rows of its last layer (its options have been read then).  Returns
    when the thread looks."""
    import threading
    stream, looking = torch.cuda.Stream(), threading.Event()

    def body():
        with torch.cuda.stream(stream):
            while float(cache[-1, :, 0].float().abs().max()) == 0:
                looking.set()          # (the first look loads its kernels)
        do()
    t = threading.Thread(target=body)
    t.start()
    assert looking.wait(60)
    return t


@pytest.mark.gpu
def test_gpu_options_set_by_another_thread_between_the_passes_of_a_call(built_library):
    """Options are the device's.  A call of several packed passes runs all of them with those that its first one found: an engine of
    another format (vocabulary, frequencies) that another thread makes current meanwhile changes no row."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_megakernel_C as C
    vocab, lens = 2048, [1500] * 24
    w = S.weights_to(S.make_weights(seed=12, num_layers=8, vocab_size=vocab, norm_std=0.1, max_seq_len=16), "cuda")
    eng, args = _passes(C, w, vocab, lens, 700)
    running, changes = True, 0

    def others():
        nonlocal changes
        other = torch.full((64,), 0.25)
        while running:
            C.set_weight_format("fp8")
            C.configure(vocab_size=1024)
            if changes % 4 == 0:
                C.set_inv_freq(other)
            changes += 1
    try:
        eng._base.apply_options()
        C.prefill_packed_passes(*args)
        want = [(k.clone(), v.clone()) for k, v in zip(eng._k_caches, eng._v_caches)]
        for k, v in zip(eng._k_caches, eng._v_caches):
            k.zero_(), v.zero_()
        torch.cuda.synchronize()
        eng._base.apply_options()
        thread = _when_rows_appear(eng._k_caches[0], others)
        C.prefill_packed_passes(*args)
        running = False
        thread.join()
        assert changes > 0
        for b, (k, v) in enumerate(want):
            assert torch.equal(eng._k_caches[b], k) and torch.equal(eng._v_caches[b], v), b
    finally:
        running = False
        eng._base.apply_options()
        C.set_weight_format("fp16")


@pytest.mark.gpu
def test_gpu_another_prefill_gets_in_between_the_passes_of_a_call(built_library):
    """A short prompt that another thread prefills while a call of 24 packed passes runs waits for the pass on its way, not for the call,
    and neither changes the other's rows."""
    import time
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_megakernel_C as C
    from Model.Qwen06B_architecture import Decoder
    vocab, lens = 2048, [1500] * 24
    w = S.weights_to(S.make_weights(seed=13, num_layers=8, vocab_size=vocab, norm_std=0.1, max_seq_len=16), "cuda")
    eng, args = _passes(C, w, vocab, lens, 800)
    short = Decoder(weights=w, tokenizer=S.StubTokenizer(-1, vocab), verbose=False, max_seq_len=64, prefill_mode="tensor")
    ids, done = S.make_prompt(60, seed=3, vocab_size=vocab), []
    C.prefill_packed_passes(*args)
    short.prefill_ids(ids)
    want = [x.clone() for x in (*eng._k_caches, *eng._v_caches, short._k_cache, short._v_cache)]
    for x in (*eng._k_caches, *eng._v_caches, short._k_cache, short._v_cache):
        x.zero_()
    short.reset()
    torch.cuda.synchronize()

    def other():
        short.prefill_ids(ids)
        done.append(time.perf_counter())
    thread = _when_rows_appear(eng._k_caches[0], other)
    C.prefill_packed_passes(*args)
    end = time.perf_counter()
    thread.join()
    assert done and done[0] < end
    for x, y in zip((*eng._k_caches, *eng._v_caches, short._k_cache, short._v_cache), want):
        assert torch.equal(x, y)
