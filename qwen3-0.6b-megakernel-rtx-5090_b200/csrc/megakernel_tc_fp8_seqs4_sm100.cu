// Tensor-core decode megakernel for up to four sequences per launch, FP8-E4M3 rows (see megakernel_tc_multi.cuh): their operands and residual sums
// leave room for a ring of 14 slots.
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>

#include "../../include/qwen_megakernel.h"

#include "megakernel_params.h"

#define QMK_NS qmkt8s4
#define QMK_MAX_SEQ 1
#define QMK_TC_BUILD 1
#define QMK_TC_FP8 1
#define QMK_TC_SEQS 4
#define QMK_NSLOTS 14
#define QMK_SLOT_BYTES 8832
#define QMK_EMPTY_UNITS 12
#include "megakernel_device.cuh"
#include "megakernel_fused.cuh"
#include "megakernel_tc.cuh"
#include "megakernel_tc_multi.cuh"
#include "megakernel_tc.h"

namespace qmk_fused_tc {
const Build &build_fp8_seqs4() {
  static const Build b = {reinterpret_cast<const void *>(qmkt8s4::qwen3_decode_megakernel_tc_seqs), qmkt8s4::TC_SMEM_BYTES, qmkt8s4::tc_grid,
                          qmkt8s4::CH_ROWS, qmkt8s4::tc_ring};
  return b;
}
}  // namespace qmk_fused_tc
