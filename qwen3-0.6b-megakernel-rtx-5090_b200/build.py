"""Builds the C-ABI shared library for sm_100a with plain nvcc, in-tree.

    python build.py [--force]

Output: ``libqwen_megakernel.so`` next to this file.  It takes the place of the
reference's torch extension build (``setup.py:20-37``, ``-arch=sm_120``): same
exported launcher symbols, different architecture, no libtorch dependency.
"""

from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCES = [os.path.join(HERE, "csrc", "megakernel_sm100.cu"), os.path.join(HERE, "csrc", "megakernel_batch_sm100.cu"),
           os.path.join(HERE, "csrc", "megakernel_tc_sm100.cu"), os.path.join(HERE, "csrc", "megakernel_tc_fp8_sm100.cu"),
           *(os.path.join(HERE, "csrc", f"megakernel_tc_{fmt}seqs{n}_sm100.cu") for fmt in ("", "fp8_") for n in (2, 4)),
           os.path.join(HERE, "csrc", "prefill_sm100.cu")]
HEADERS = [os.path.join(os.path.dirname(HERE), "include", "qwen_megakernel.h"),
           os.path.join(HERE, "csrc", "megakernel_device.cuh"), os.path.join(HERE, "csrc", "megakernel_params.h"),
           os.path.join(HERE, "csrc", "megakernel_batch.cuh"), os.path.join(HERE, "csrc", "megakernel_fused.cuh"),
           os.path.join(HERE, "csrc", "megakernel_tc.cuh"), os.path.join(HERE, "csrc", "megakernel_tc_multi.cuh"), os.path.join(HERE, "csrc", "megakernel_tc.h"), os.path.join(HERE, "csrc", "megakernel_batch.h"),
           os.path.join(HERE, "csrc", "gemm_tcgen05.cuh"), os.path.join(HERE, "csrc", "gemm_pair_tcgen05.cuh"), os.path.join(HERE, "csrc", "prefill_sm100.h"),
           os.path.join(HERE, "csrc", "prefill_kernels.cuh"), os.path.join(HERE, "csrc", "engine_internal.h"), os.path.join(HERE, "csrc", "buffer_group.h"),
           os.path.join(HERE, "csrc", "attention_tcgen05.cuh"), os.path.join(HERE, "csrc", "decode_attention_mma.cuh")]
LIB_PATH = os.path.join(HERE, "libqwen_megakernel.so")

NVCC_FLAGS = [
    "-std=c++17", "-O3", "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "--expt-extended-lambda", "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC", "-shared",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def is_stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    built = os.path.getmtime(LIB_PATH)
    return any(os.path.getmtime(p) > built for p in SOURCES + HEADERS + [os.path.abspath(__file__)])


MAX_STACK_BYTES = 16   # per-thread stack the persistent decode kernels may use (see check_stack_frames)


def check_stack_frames(ptxas_log: str) -> None:
    """The persistent decode kernels carve 220+ KB of shared memory out of each SM, which leaves ~30 KB of L1
    for 416 threads: a per-thread stack of a few hundred bytes (spills, locally indexed arrays) turns every
    touch into an L2 round trip on the critical path (measured: 975 -> 1237 us/token with a 400-byte frame).
    ptxas reports the frame of every entry point; the build fails when a decode megakernel exceeds the limit."""
    lines = ptxas_log.splitlines()
    bad = []
    for i, line in enumerate(lines):
        if "Function properties for" in line and "qwen3_decode" in line and "$" not in line.split("for", 1)[1]:
            name = line.split("for", 1)[1].strip()
            props = lines[i + 1] if i + 1 < len(lines) else ""
            try:
                frame = int(props.strip().split(" bytes stack frame")[0])
            except ValueError:
                continue
            if frame > MAX_STACK_BYTES:
                bad.append(f"{name}: {props.strip()}")
    if bad:
        raise RuntimeError("decode megakernel with a per-thread stack frame over %d bytes:\n  %s" %
                           (MAX_STACK_BYTES, "\n  ".join(bad)))


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile if the library is missing or older than its sources; return its path."""
    if not force and not is_stale():
        return LIB_PATH
    tmp = LIB_PATH + ".tmp"
    cmd = [_nvcc(), *NVCC_FLAGS, "-Xptxas", "-v", "-o", tmp, *SOURCES]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + proc.stdout + proc.stderr)
    check_stack_frames(proc.stderr)
    os.replace(tmp, LIB_PATH)
    if verbose:
        print(proc.stderr)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
