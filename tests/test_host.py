"""CPU tests of the boundary: the C-ABI library builds, loads and exports every symbol the header
declares; the op module validates arguments like the reference binding; nothing computes here."""

import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol(built_library):
    header = open(os.path.join(ROOT, "include", "qwen_megakernel.h")).read()
    declared = set(re.findall(r"\b((?:launch_ldg|qmk)_\w+)\s*\(", header))
    assert {"launch_ldg_decode_direct", "launch_ldg_decode_persistent", "launch_ldg_generate_nosync",
            "launch_ldg_prefill"} <= declared
    lib = ctypes.CDLL(built_library)
    for name in sorted(declared):
        assert hasattr(lib, name), f"{name} declared in the header but not exported"
    import qwen_megakernel_C as C
    assert declared == set(C.EXPORTED_SYMBOLS)


def test_engine_handle_argument_checks(built_library):
    """qmk_engine_create refuses null pointers and unknown weight formats before touching a GPU; destroying a null
    handle is a no-op."""
    import qwen_megakernel_C as C
    lib = C._lib
    handle = ctypes.c_void_p()
    assert lib.qmk_engine_create(None, ctypes.byref(handle)) != 0
    cfg = C._EngineConfig(0, 151936, 5, 0, -1, -1, -1, -1, None)
    assert lib.qmk_engine_create(ctypes.byref(cfg), ctypes.byref(handle)) != 0 and not handle
    assert lib.qmk_engine_destroy(None) == 0
    assert lib.qmk_engine_apply(None) != 0


def test_refusals_without_an_engine_have_a_text(built_library):
    """Calls that fail before there is an engine to keep the error: the text is theirs, not an older one."""
    import qwen_megakernel_C as C
    lib = C._lib
    handle = ctypes.c_void_p()
    cfg = C._EngineConfig(0, 151936, 5, 0, -1, -1, -1, -1, None)
    assert lib.qmk_engine_create(ctypes.byref(cfg), ctypes.byref(handle)) != 0 and b"weight format" in lib.qmk_last_error()
    assert lib.qmk_engine_apply(None) != 0 and b"handle" in lib.qmk_last_error()
    if not torch.cuda.is_available():
        assert lib.qmk_set_fused(1, 1) != 0 and lib.qmk_last_error() == b"no CUDA device"
        assert lib.qmk_decode_batched(1, None, None, 1, *[None] * 9, 1, 1, 1.0, None) != 0 and lib.qmk_last_error() == b"no CUDA device"
    assert lib.qmk_engine_destroy(None) == 0


@pytest.mark.parametrize("fmt", ["fp16", "fp8"])
@pytest.mark.parametrize("n", [1, 2, 3, 4])
def test_norm_vectors_are_not_overwritten_in_use_on_any_grid(built_library, fmt, n):
    """The persistent tensor-core kernels copy layer L's norm vectors over layer L - 2's when the slot of layer L - 1's last chunk is
    free, i.e. the chunk `slots` before it was handed back.  With the real chunk counts of every CTA of every grid that
    a limit on the CTAs leads to, that chunk is a gate / up chunk of L - 2 or a later one (post_ln is read in front of them).  An
    attention item adds chunks between q|k|v and O."""
    import qwen_megakernel_C as C
    launched = {}
    for ctas in range(1, 270):
        grid = C.selftest_decode_ring(fmt, n, ctas)[0]
        assert (grid > 0) == ((112 if n > 2 else 96) <= ctas <= (160 if fmt == "fp8" else 256))
        assert grid == 0 or ctas - 3 <= grid <= ctas and (ctas % 4 or grid == ctas) or (fmt, n) == ("fp16", 1) and grid == 171 < ctas
        launched[grid] = ctas
    for grid in sorted(launched)[1:]:
        for cta in range(grid):
            _, slots, qkv, o, gate_up, down = C.selftest_decode_ring(fmt, n, grid, cta)
            for attention in (0, 1, 8):
                layer = [0] * (qkv + attention + o) + [1] * (gate_up + down)       # 1: behind the last use of post_ln
                handed_back = 2 * len(layer) - 1 - slots                            # counted from layer L - 2's first chunk
                assert handed_back >= len(layer) or handed_back >= 0 and layer[handed_back], (grid, cta)


@pytest.mark.parametrize("fmt", ["fp16", "fp8"])
def test_the_warps_that_make_the_split_weights_have_a_quad_of_every_slice(built_library, fmt):
    """One sequence: the last two of twelve warps take part in the merge of a group's attention outputs where its slice (512 quads over
    the groups of four CTAs) has one for them, and make the weights of all.  So no slice of a grid that is launched is shorter than
    twelve quads."""
    import qwen_megakernel_C as C
    for grid in {C.selftest_decode_ring(fmt, 1, ctas)[0] for ctas in range(1, 270)} - {0}:
        groups = grid // 4
        assert min(512 * (g + 1) // groups - 512 * g // groups for g in range(groups)) >= 12, grid


def test_abi_version_handshake(built_library):
    import qwen_megakernel_C as C
    from Model import Qwen06B_architecture as A
    assert C.abi_version() == 2 == A.EXTENSION_ABI_VERSION
    assert C.scratch_bytes() < 8 << 20   # 4 copies x 4 sequences of the exchange area


def test_reference_constants_and_surface(built_library):
    from Model import Qwen06B_architecture as A
    assert (A.NUM_LAYERS, A.NUM_KV_HEADS, A.HEAD_DIM, A.HIDDEN_SIZE, A.INTERMEDIATE_SIZE) == (28, 8, 128, 1024, 3072)
    assert (A.Q_SIZE, A.KV_SIZE, A.MAX_SEQ_LEN, A.VOCAB_SIZE, A.ROPE_THETA) == (2048, 1024, 2048, 151936, 1e6)
    for name in ("load_weights", "_pack_layer_weights", "Decoder", "generate", "_require_megakernel_op"):
        assert hasattr(A, name)
    for name in ("step", "reset", "position", "generate"):
        assert hasattr(A.Decoder, name)
    with pytest.raises(RuntimeError, match="unavailable"):
        A._require_megakernel_op("no_such_op")


def test_pack_layer_weights_layout(built_library):
    from Model.Qwen06B_architecture import _pack_layer_weights
    import synthetic as S
    w = S.make_weights(seed=1, num_layers=2, vocab_size=64)
    t = _pack_layer_weights(w["layer_weights"])
    assert t.dtype == torch.int64 and t.numel() == 2 * 12 and t.data_ptr() % 16 == 0
    tab = t.view(2, 12)
    for li in range(2):
        for j in range(11):
            assert tab[li, j].item() == w["layer_weights"][li * 11 + j].data_ptr()
        assert tab[li, 11].item() == 0


def test_argument_validation_matches_reference_binding(built_library):
    """dtype / device / contiguity / size checks raise RuntimeError before any launch
    (reference: qwen_ops.cpp:142-150, 219-221)."""
    import qwen_megakernel_C as C
    dummy = [torch.zeros(4)] * 19
    with pytest.raises(RuntimeError, match="int32"):
        C.prefill(torch.zeros(3, dtype=torch.int64), *dummy, 1, 0, 16, 0.1)
    with pytest.raises(RuntimeError, match="contiguous"):
        C.prefill(torch.zeros(6, dtype=torch.int32)[::2], *dummy, 1, 0, 16, 0.1)
    assert C.prefill(torch.zeros(0, dtype=torch.int32), *dummy, 1, 0, 16, 0.1) is None
    if not torch.cuda.is_available():
        with pytest.raises(RuntimeError, match="no CUDA device"):
            C.generate_nosync(1, 2, *dummy, torch.zeros(4, dtype=torch.int32), 1, 0, 16, 0.1)
        with pytest.raises(RuntimeError, match="no CUDA device"):
            C.decode(1, *dummy, 1, 0, 16, 0.1)
        with pytest.raises(RuntimeError, match="CUDA device"):
            from Model.Qwen06B_architecture import Decoder
            Decoder(weights={})


def test_stub_tokenizer_roundtrip():
    import synthetic as S
    tok = S.StubTokenizer(eos_token_id=7, vocab_size=100)
    assert tok.encode("5 17 230") == [5, 17, 30]
    assert tok.decode([5, 17]) == "5 17"
    assert tok.apply_chat_template([{"role": "user", "content": "1 2"}]) == "1 2"


def test_build_rejects_a_stack_frame_in_a_decode_megakernel():
    """build.py reads ptxas' report: a decode megakernel with a per-thread stack frame must fail the build."""
    import build
    ok = ("ptxas info    : Function properties for _ZN3qmk23qwen3_decode_megakernelEN4qmkp6ParamsE\n"
          "    8 bytes stack frame, 4 bytes spill stores, 4 bytes spill loads\n"
          "ptxas info    : Function properties for _ZN3qmk17rope_table_kernelEPfi\n"
          "    400 bytes stack frame, 0 bytes spill stores, 0 bytes spill loads\n")
    build.check_stack_frames(ok)          # small frame; other kernels are not held to the limit
    bad = ok.replace("    8 bytes stack frame", "    408 bytes stack frame")
    with pytest.raises(RuntimeError, match="stack frame"):
        build.check_stack_frames(bad)


def test_engine_choice_for_four_sequences():
    """``BatchDecoder(engine="auto")`` with four sequences takes the persistent engine only where its launch runs on the
    tensor cores and contexts stay below the crossover; three and five do not depend on any of it."""
    from Model.Qwen06B_architecture import BatchDecoder
    auto, room = BatchDecoder.auto_engine, 1 << 34
    for fmt in ("fp16", "fp8"):
        assert auto(4, fmt, 151936, 2048, 148, room) == "persistent"
        assert auto(4, fmt, 151936, 2048, 111, room) == "gemm"           # smaller grid than the launch is built for
        assert auto(4, fmt, 151936, 2048, 148, 100 << 20) == "gemm"      # no room for the K-major copies
        assert auto(4, fmt, 151936, 16384, 148, room) == "gemm"
        assert auto(4, fmt, 4104, 16384, 100, 0) == "persistent"         # the GEMM step does not read this vocabulary
        assert auto(3, fmt, 151936, 32768, 0, 0) == "persistent" and auto(5, fmt, 151936, 64, 148, room) == "gemm"
    assert auto(4, "fp16", 151936, 8320, 148, room) == "gemm" and auto(4, "fp8", 151936, 8320, 148, room) == "persistent"
    assert auto(4, "fp8", 151936, 2048, 200, room) == "gemm" and auto(4, "fp16", 151936, 2048, 200, room) == "persistent"
    assert [auto(n, "nvfp4", 151936, 2048, 148, room) for n in (1, 4, 9)] == ["gemm"] * 3


BUFFER_GROUP = r"""
#include "buffer_group.h"
#include <cstdio>
#include <cstdlib>
#include <set>
int main() {
  // five buffers; call 0 .. 4 of the allocator is the one that is refused (5: none)
  for (int refused = 0; refused <= 5; ++refused) {
    void *p[5] = {};
    const qmk_tc::Buffer group[] = {{&p[0], 8}, {&p[1], 16}, {&p[2], 24}, {&p[3], 32}, {&p[4], 40}};
    std::set<void *> live;
    int calls = 0;
    auto make = [&](void **at, std::size_t bytes) {
      if (calls++ == refused) { *at = &calls; return 2; }        // (an allocator may leave anything behind)
      if (bytes != 8u * static_cast<unsigned>(calls)) std::exit(10);
      live.insert(*at = std::malloc(bytes));
      return 0;
    };
    auto drop = [&](void *q) { if (live.erase(q) != 1) std::exit(11); std::free(q); };
    const int first = qmk_tc::make_all(group, 0, make, drop);
    if (first != (refused < 5 ? 2 : 0)) return 12;
    for (void *q : p)
      if ((q != nullptr) != (refused == 5)) return 13;           // all or none
    if (live.size() != (refused == 5 ? 5u : 0u)) return 14;
    if (refused == 5) continue;
    calls = 0;
    refused = refused + 100;                                     // there is room again
    if (qmk_tc::make_all(group, 0, make, drop) != 0 || live.size() != 5) return 15;
    refused -= 100;
    qmk_tc::drop_all(group, drop);
    if (!live.empty()) return 16;
  }
  return 0;
}
"""


def test_workspace_buffers_come_all_or_none(tmp_path):
    """The workspaces of the tensor-core paths are groups of buffers.  Whichever of them is refused, none is left: a later call
    finds no part of a group that it would take for the whole, and makes it once there is room."""
    import subprocess
    src = tmp_path / "group.cpp"
    src.write_text(BUFFER_GROUP)
    csrc = os.path.join(ROOT, "qwen3-0.6b-megakernel-rtx-5090_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", csrc, "-o", str(tmp_path / "group"), str(src)], check=True)
    assert subprocess.run([str(tmp_path / "group")]).returncode == 0
    # and no buffer of the batched decode is made beside the group
    code = open(os.path.join(csrc, "prefill_sm100.cu")).read()
    body = code[code.index("int ensure_decode_workspace("):code.index("if (w.logits_vocab < vocab)")]
    assert "make_all" in body and "cudaMalloc" not in body
