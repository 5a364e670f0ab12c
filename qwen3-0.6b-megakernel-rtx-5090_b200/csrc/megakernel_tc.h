// Host-visible handles of the tensor-core builds of the fused single-sequence decode megakernel
// (megakernel_tc_sm100.cu: fp16 rows; megakernel_tc_fp8_sm100.cu: FP8-E4M3 rows).
#ifndef QMK_MEGAKERNEL_TC_H_
#define QMK_MEGAKERNEL_TC_H_

#include <stddef.h>

namespace qmk_fused_tc {
struct Build {
  const void *kernel;          // __global__ entry, launched cooperatively with one Params argument
  size_t smem_bytes;           // dynamic shared memory of one CTA
  int min_ctas, max_ctas;      // grids the kernel's shared-memory slices and its ring are sized for
  int rows_per_chunk;          // rows are owned in units of this many: the vocabulary is a multiple of it
};
const Build &build_f16();
const Build &build_fp8();
// The build that reads weight format `wfmt` (0 fp16 rows, 1 FP8-E4M3 rows).
inline const Build &build(int wfmt) { return wfmt ? build_fp8() : build_f16(); }
}  // namespace qmk_fused_tc

#endif  // QMK_MEGAKERNEL_TC_H_
