// Host-visible handles of the tensor-core builds of the fused decode megakernel (megakernel_tc_sm100.cu: fp16 rows;
// megakernel_tc_fp8_sm100.cu: FP8-E4M3 rows; megakernel_tc_*seqs*_sm100.cu: two and four sequences per launch).
#ifndef QMK_MEGAKERNEL_TC_H_
#define QMK_MEGAKERNEL_TC_H_

#include <stddef.h>

namespace qmk_fused_tc {
struct Build {
  const void *kernel;          // __global__ entry, launched cooperatively with one Params argument
  size_t smem_bytes;           // dynamic shared memory of one CTA
  int (*grid)(int ctas);       // the largest grid of at most `ctas` CTAs that its shared-memory slices and its ring are sized for, or 0
  int rows_per_chunk;          // rows are owned in units of this many: the vocabulary is a multiple of it
  void (*ring)(int ncta, int cta, int (&out)[5]);   // slots of the ring; a layer's q|k|v, O, gate / up and down chunks of a CTA
};
const Build &build_f16();
const Build &build_fp8();
const Build &build_f16_seqs2();   // up to two sequences (megakernel_tc_multi.cuh)
const Build &build_f16_seqs4();   // up to four
const Build &build_fp8_seqs2();
const Build &build_fp8_seqs4();
// The build that reads weight format `wfmt` (0 fp16 rows, 1 FP8-E4M3 rows).
inline const Build &build(int wfmt) { return wfmt ? build_fp8() : build_f16(); }
// The build for a launch of `nseq` sequences with their own caches.  Three sequences take the four-sequence build, which
// leaves columns of its MMAs idle.
inline const Build &build_seqs(int wfmt, int nseq) {
  return nseq <= 2 ? (wfmt ? build_fp8_seqs2() : build_f16_seqs2()) : (wfmt ? build_fp8_seqs4() : build_f16_seqs4());
}
}  // namespace qmk_fused_tc

#endif  // QMK_MEGAKERNEL_TC_H_
