// Tensor-core decode megakernel for up to four sequences per launch, fp16 rows (see megakernel_tc_multi.cuh): their operands and residual sums
// leave room for a ring of 14 slots.
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>

#include "../../include/qwen_megakernel.h"

#include "megakernel_params.h"

#define QMK_NS qmkts4
#define QMK_MAX_SEQ 1
#define QMK_TC_BUILD 1
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
const Build &build_f16_seqs4() {
  static const Build b = {reinterpret_cast<const void *>(qmkts4::qwen3_decode_megakernel_tc_seqs), qmkts4::TC_SMEM_BYTES, qmkts4::tc_grid,
                          qmkts4::CH_ROWS, qmkts4::tc_ring};
  return b;
}
}  // namespace qmk_fused_tc
