// FP8-E4M3 build of the tensor-core decode megakernel (see megakernel_tc.cuh): the same ring of 18 slots, a chunk = eight
// packed rows of 1040 bytes.
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>

#include "../../include/qwen_megakernel.h"

#include "megakernel_params.h"

#define QMK_NS qmkt8
#define QMK_MAX_SEQ 1
#define QMK_TC_BUILD 1
#define QMK_TC_FP8 1
#define QMK_NSLOTS 18
#define QMK_SLOT_BYTES 8832
#define QMK_EMPTY_UNITS 12
#include "megakernel_device.cuh"
#include "megakernel_fused.cuh"
#include "megakernel_tc.cuh"
#include "megakernel_tc.h"

namespace qmk_fused_tc {
const Build &build_fp8() {
  static const Build b = {reinterpret_cast<const void *>(qmkt8::qwen3_decode_megakernel_tc), qmkt8::TC_SMEM_BYTES, qmkt8::tc_grid,
                          qmkt8::CH_ROWS, qmkt8::tc_ring};
  return b;
}
}  // namespace qmk_fused_tc
