"""The ``prefill`` op on the tensor cores with split activations (hi + lo fp16 halves of every fp32 operand) against the
CPU oracle, which keeps fp32 activations.

Bounds: hi + lo drops at most 2^-22 of an operand, so a first-layer row differs from the oracle's only where an fp32
result sits within rounding error (near 1e-6) of an fp16 tie of the cache (spacing near 1e-3): one fp16 ulp, in about one
value of a thousand, root mean square 1e-3 * sqrt(1e-3) = 3e-5.  Each such flip of a V row then moves the attention output
of every later layer by about that rms, which flips some per cent of the rows there: 1e-3 * sqrt(3e-2) = 1.7e-4 (the
token-serial kernel shows 0.6e-4 on three tokens), and a flip can land on a moved value: two ulps.  Operands rounded to
fp16 once show 4e-3 to 6e-3 at the largest and fail both."""

import pytest
import torch

import synthetic as S
from oracle.decoder_ref import Decoder as OracleDecoder

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,calls", [("fp16", (3,)), ("fp16", (4,)), ("fp16", (127,)), ("fp16", (2, 129, 70)), ("fp16", (1100,)),
                                       ("fp8", (5,)), ("fp8", (260,))])
def test_rows_match_fp32_oracle(built_library, fmt, calls):
    """Lengths below the op's switch to the tensor cores and at it, tile edges, a second call behind a first one, a chunk
    long enough for the wide tiles."""
    import qwen_megakernel_C as C
    import quantize as Q
    from Model.Qwen06B_architecture import Decoder
    w = S.make_weights(seed=21, num_layers=3, vocab_size=2048, norm_std=0.1, max_seq_len=16)
    engine_w, oracle_w = Q.quantize_weights_fp8(w) if fmt == "fp8" else (w, w)
    n = sum(calls)
    ids = S.make_prompt(n, seed=n, vocab_size=2048)
    o = OracleDecoder(oracle_w, max_seq_len=1280)
    o.prefill(ids)
    try:
        eng = Decoder(weights=S.weights_to(engine_w, "cuda"), verbose=False, max_seq_len=1280, weight_format=fmt)
        at = 0
        for c in calls:
            eng.prefill_ids(ids[at:at + c])
            at += c
    finally:
        C.set_weight_format("fp16")
    for got, want in ((eng._k_cache, o.k_cache), (eng._v_cache, o.v_cache)):
        want = want[:, :, :n].float()
        diff = (got[:, :, :n].float().cpu() - want).abs()
        print(f"{fmt} {calls}: max {float(diff.max()):.2e} rms {float(diff.square().mean().sqrt()):.2e} "
              f"first layer {float(diff[0].max()):.2e} {float(diff[0].square().mean().sqrt()):.2e}")
        ulp = want.abs().clamp(min=2.0) * 2.0 ** -10
        assert bool((diff[0] <= ulp[0]).all()) and bool((diff <= 2 * ulp).all())
        assert float(diff[0].square().mean().sqrt()) < 6e-5 and float(diff.square().mean().sqrt()) < 3.4e-4
    assert torch.count_nonzero(eng._k_cache[:, :, n:]) == 0


@pytest.mark.parametrize("n", [2, 12])
def test_misaligned_pointers_are_refused(built_library, n):
    """The op's pointer rules hold on both of its routes (few tokens: persistent steps; more: the chunked pass, whose
    row kernels read the embedding 16 bytes at a time)."""
    from Model.Qwen06B_architecture import Decoder
    w = S.make_weights(seed=1, num_layers=2, vocab_size=512, max_seq_len=16)
    eng = Decoder(weights=S.weights_to(w, "cuda"), verbose=False, max_seq_len=32)
    good = list(eng._common())

    def shifted(t):
        return torch.zeros(t.numel() + 8, dtype=t.dtype, device="cuda")[1:1 + t.numel()].view(t.shape)
    ids = torch.arange(n, dtype=torch.int32)
    for at in (0, 6, 7):      # embedding, K cache, V cache
        args = list(good)
        args[at] = shifted(good[at])
        with pytest.raises(RuntimeError, match="16-byte aligned"):
            eng._prefill_op(ids, *args, eng.num_layers, 0, eng.max_seq_len, eng._attn_scale)
    eng.prefill_ids(ids.tolist())
    assert torch.count_nonzero(eng._k_cache[:, :, :n]) > 0


FULL_DEVICE = r"""
import json, sys
sys.path[:0] = [{root!r}, {pkg!r}]
import torch
import synthetic as S
from Model.Qwen06B_architecture import Decoder
w = S.make_weights(seed=3, num_layers=2, vocab_size=4096, norm_std=0.1, max_seq_len=16)
eng = Decoder(weights=S.weights_to(w, "cuda"), verbose=False, max_seq_len=64)
steps = [eng.step(t) for t in {ids!r}[:-1]]              # token by token: exchange words and K-major copies exist now
rows = eng._k_cache[:, :, :eng.position].clone()
eng._k_cache.zero_(); eng._v_cache.zero_(); eng.reset()
torch.cuda.synchronize()
ballast = torch.empty(torch.cuda.mem_get_info()[0] - (160 << 20), dtype=torch.uint8, device="cuda")
free = []
for _ in range(3):
    tokens = eng.generate_ids({ids!r}, 6)
    torch.cuda.synchronize()
    free.append(torch.cuda.mem_get_info()[0])
same = bool(torch.equal(rows, eng._k_cache[:, :, :rows.shape[2]]))
del ballast
torch.cuda.empty_cache()
print(json.dumps(dict(tokens=tokens, free=free, same=same, again=eng.generate_ids({ids!r}, 6))))
"""


def test_prompt_is_prefilled_step_by_step_where_the_workspace_does_not_fit(built_library):
    """A process whose device memory is given away (160 MB left; the chunked pass wants 285 MB): prompts go through the
    persistent steps, bit for bit as decoded token by token, no call keeps memory, and once there is room again the
    chunked pass gives the same tokens."""
    import json
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    pkg = os.path.join(root, "qwen3-0.6b-megakernel-rtx-5090_b200")
    ids = S.make_prompt(12, seed=5, vocab_size=4096)
    want = OracleDecoder(S.make_weights(seed=3, num_layers=2, vocab_size=4096, norm_std=0.1, max_seq_len=16),
                         max_seq_len=64).generate_ids(ids, 6)[0]
    proc = subprocess.run([sys.executable, "-c", FULL_DEVICE.format(root=root, pkg=pkg, ids=ids)], capture_output=True, text=True,
                          timeout=600)
    assert proc.returncode == 0, proc.stdout[-2000:] + proc.stderr[-4000:]
    res = json.loads(proc.stdout.strip().splitlines()[-1])
    assert res["tokens"] == want and res["again"] == want and res["same"]
    assert res["free"][0] == res["free"][-1] and res["free"][0] > 100 << 20


def test_unfused_switch_covers_the_prefill_op(built_library):
    """``set_fused(0)`` is the unfused kernel for every op: a prompt prefilled under it leaves the rows that decoding it
    token by token leaves, bit for bit."""
    import qwen_megakernel_C as C
    from Model.Qwen06B_architecture import Decoder
    w = S.make_weights(seed=9, num_layers=2, vocab_size=512, norm_std=0.1, max_seq_len=16)
    ids = S.make_prompt(40, seed=2, vocab_size=512)
    eng = Decoder(weights=S.weights_to(w, "cuda"), verbose=False, max_seq_len=64)
    rows = []
    try:
        for fused in (0, 2):
            C.set_fused(fused=fused)
            eng.reset()
            eng.prefill_ids(ids)
            rows.append((eng._k_cache.clone(), eng._v_cache.clone()))
            eng.reset()
            for t in ids:
                eng.step(t)
            if fused == 0:
                assert torch.equal(rows[-1][0], eng._k_cache) and torch.equal(rows[-1][1], eng._v_cache)
    finally:
        C.set_fused(fused=2)
    assert float((rows[0][0].float() - rows[1][0].float()).abs().max()) < 8e-3


def test_error_text_survives_another_threads_call(built_library):
    """The text of a failed call is the failing thread's until its next call: a pass that another thread runs in between (and
    that clears the device's error) does not take it away; the thread's own next call does."""
    import threading
    import qwen_megakernel_C as C
    from Model.Qwen06B_architecture import Decoder
    w = S.weights_to(S.make_weights(seed=9, num_layers=2, vocab_size=512, max_seq_len=16), "cuda")
    eng = Decoder(weights=w, verbose=False, max_seq_len=64)
    eng.prefill_ids([1, 2, 3, 4, 5])
    assert C._lib.qmk_selftest_gemm_wait_timeout(0) != 0
    thread = threading.Thread(target=lambda: (eng.reset(), eng.generate_ids([1, 2, 3, 4, 5, 6], 2)))
    thread.start()
    thread.join()
    assert b"budget_us" in C._lib.qmk_last_error()
    eng.reset()
    eng.generate_ids([1, 2, 3, 4, 5, 6], 2)
    assert b"budget_us" not in C._lib.qmk_last_error()


def test_error_text_is_of_the_threads_own_last_call(built_library):
    """The other direction: a call that succeeded has no text, whatever another thread failed at since (the void ops tell by the
    text).  A later call that returns a status clears the text, also where it does no work; a thread without a call of its own
    sees the device's last error."""
    import threading
    import qwen_megakernel_C as C
    from Model.Qwen06B_architecture import Decoder
    w = S.weights_to(S.make_weights(seed=9, num_layers=2, vocab_size=512, max_seq_len=16), "cuda")
    eng = Decoder(weights=w, verbose=False, max_seq_len=64)
    seen = []

    def elsewhere(*calls):
        thread = threading.Thread(target=lambda: seen.extend(call() for call in calls))
        thread.start()
        thread.join()

    def text():
        return C._lib.qmk_last_error().decode()

    eng.prefill_ids([1, 2, 3, 4, 5])
    elsewhere(lambda: C._lib.qmk_selftest_gemm_wait_timeout(0), text)
    assert seen[0] == 2 and "budget_us" in seen[1] and text() == ""
    elsewhere(text)
    assert "budget_us" in seen[2]                      # (no call of its own: the device's last error)
    assert C._lib.qmk_sync_status() == 2 and "budget_us" in text()      # asked for: the device's status and its text
    elsewhere(lambda: eng.prefill_ids([6]))
    assert C._lib.qmk_sync_status() == 0 and text() == ""
    for quiet in (lambda: C._lib.qmk_set_step_overlap(-1), lambda: C._lib.qmk_configure(-1, -1, -1, -1, -1), C._lib.qmk_num_ctas,
                  lambda: C._lib.qmk_selftest_wait_timeout(300), lambda: C._lib.qmk_decode_batched(1, *[None] * 2, 0, *[None] * 9, 1, 1, 1.0, None)):
        assert C._lib.qmk_selftest_gemm_wait_timeout(0) == 2 and "budget_us" in text()
        quiet()
        assert text() == ""
    assert C._lib.qmk_gemm_f16_tn(None, None, None, 100, 64, 64, None) != 0 and text() not in ("", "budget_us must be in [1, 1e6]")
    assert C._lib.qmk_engine_apply(None) != 0 and "handle" in text()


def test_short_prompts_do_not_wait_for_a_chunked_pass(built_library):
    """The workspace of the chunked pass is held for a whole pass (some 20 ms here).  A call of the op that does not use it -
    measured on one that is refused before any GPU work - returns meanwhile."""
    import threading
    import time
    from Model.Qwen06B_architecture import Decoder
    w = S.weights_to(S.make_weights(seed=9, num_layers=28, vocab_size=512, max_seq_len=16), "cuda")
    long = Decoder(weights=w, verbose=False, max_seq_len=8192, prefill_mode="tensor")
    short = Decoder(weights=w, verbose=False, max_seq_len=64)
    ids = S.make_prompt(8191, seed=1, vocab_size=512)
    passes, stop = [], threading.Event()

    def prefill():
        with torch.cuda.stream(torch.cuda.Stream()):
            while not stop.is_set():
                t0 = time.perf_counter()
                long.reset()
                long.prefill_ids(ids)
                passes.append(time.perf_counter() - t0)
    short.prefill_ids([1, 2])
    thread = threading.Thread(target=prefill)
    thread.start()
    try:
        while len(passes) < 2:
            time.sleep(0.005)
        waits = []
        for _ in range(40):
            t0 = time.perf_counter()
            with pytest.raises(RuntimeError, match="vocab"):
                short.prefill_ids([600])
            waits.append(time.perf_counter() - t0)
            time.sleep(0.003)
    finally:
        stop.set()
        thread.join()
    waits.sort()
    print(f"pass {sorted(passes)[len(passes) // 2] * 1e3:.1f} ms, refused short call {waits[20] * 1e3:.3f} / {waits[-1] * 1e3:.3f} ms")
    assert waits[20] < 0.1 * sorted(passes)[len(passes) // 2]


@pytest.mark.parametrize("before,n", [(900, 5), (2300, 33), (700, 140), (64, 64)])
def test_short_prompt_behind_a_long_context(built_library, before, n):
    """Few query tiles share out their keys among CTAs and the partial outputs are added up: against the oracle, with the
    bounds of the other rows here."""
    from Model.Qwen06B_architecture import Decoder
    w = S.make_weights(seed=22, num_layers=3, vocab_size=2048, norm_std=0.1, max_seq_len=16)
    ids = S.make_prompt(before + n, seed=n, vocab_size=2048)
    o = OracleDecoder(w, max_seq_len=2560)
    o.prefill(ids)
    eng = Decoder(weights=S.weights_to(w, "cuda"), verbose=False, max_seq_len=2560)
    eng.prefill_ids(ids[:before])
    eng.prefill_ids(ids[before:])
    for got, want in ((eng._k_cache, o.k_cache), (eng._v_cache, o.v_cache)):
        want = want[:, :, before:before + n].float()
        diff = (got[:, :, before:before + n].float().cpu() - want).abs()
        print(f"{before} + {n}: max {float(diff.max()):.2e} rms {float(diff.square().mean().sqrt()):.2e}")
        ulp = want.abs().clamp(min=2.0) * 2.0 ** -10
        assert bool((diff <= 2 * ulp).all()) and float(diff.square().mean().sqrt()) < 3.4e-4
