// Tensor-core side of the library: the tcgen05 GEMM and (built on it) the chunked prompt prefill.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <mutex>
#include <atomic>
#include <chrono>
#include <thread>
#include <algorithm>
#include <string>

#include "../../include/qwen_megakernel.h"
#include "gemm_tcgen05.cuh"
#include "gemm_pair_tcgen05.cuh"
#include "prefill_sm100.h"
#include "prefill_kernels.cuh"
#include "attention_tcgen05.cuh"
#include "decode_attention_mma.cuh"
#include "buffer_group.h"
#include "engine_internal.h"
#include <vector>

namespace qmk_tc {

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

std::mutex g_mu;
EncodeTiledFn g_encode = nullptr;
bool g_attr_set[16] = {};
int g_sms[16] = {};

// The driver's tensor-map encoder, looked up through the runtime (no link against libcuda).
EncodeTiledFn encoder() {
  if (g_encode) return g_encode;
  void *fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess)
    return nullptr;
  g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  return g_encode;
}

}  // namespace

// Tensor map of a row-major fp16 matrix [rows x cols]: boxes of box_rows x 64 elements, 128-byte swizzle.
int make_map_f16(CUtensorMap *map, const void *ptr, uint64_t rows, uint64_t cols, uint32_t box_rows, std::string *err) {
  EncodeTiledFn enc = encoder();
  if (!enc) { *err = "cuTensorMapEncodeTiled is not available from this driver"; return QMK_ERR_CUDA; }
  if ((reinterpret_cast<uintptr_t>(ptr) & 15u) || (cols * 2) % 16) { *err = "matrix not 16-byte aligned"; return QMK_ERR_BAD_ARGUMENT; }
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * 2};
  const cuuint32_t box[2] = {64, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { *err = "cuTensorMapEncodeTiled failed with code " + std::to_string(static_cast<int>(r)); return QMK_ERR_CUDA; }
  return QMK_OK;
}

// Packed weight rows (weight formats 1 and 2): bytes of values, where the NVFP4 block scales and the 16-byte trailer
// with the fp32 scale sit inside a row, and the bytes between rows.
PackedRow packed_row(int wq, int K) {
  PackedRow r;
  r.data_bytes = wq == 1 ? static_cast<uint32_t>(K) : static_cast<uint32_t>(K) / 2;
  r.bs_off = r.data_bytes;
  r.scale_off = wq == 1 ? r.data_bytes : r.data_bytes + static_cast<uint32_t>(K) / 16;
  r.pitch = r.scale_off + 16;
  return r;
}

// Tensor map of the VALUES of a packed matrix (bytes; scales and trailers stay outside the mapped extent): boxes of
// box_rows rows x one 64-value K block, no swizzle - the expanding warps read it linearly.
int make_map_packed(CUtensorMap *map, const void *ptr, uint64_t rows, int K, uint32_t box_rows, int wq, std::string *err) {
  EncodeTiledFn enc = encoder();
  if (!enc) { *err = "cuTensorMapEncodeTiled is not available from this driver"; return QMK_ERR_CUDA; }
  const PackedRow pr = packed_row(wq, K);
  if ((reinterpret_cast<uintptr_t>(ptr) & 15u) || K % 64 || K > qmk_gemm::MAX_K_PACKED || pr.pitch % 16) {
    *err = "packed matrix: base not 16-byte aligned, or K not a multiple of 64 (NVFP4: of 256, rows must stay 16-byte aligned) up to 3072";
    return QMK_ERR_BAD_ARGUMENT;
  }
  const cuuint64_t dims[2] = {pr.data_bytes, rows};
  const cuuint64_t strides[1] = {pr.pitch};
  const cuuint32_t box[2] = {qmk_gemm::raw_row_bytes(wq), box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { *err = "cuTensorMapEncodeTiled failed with code " + std::to_string(static_cast<int>(r)); return QMK_ERR_CUDA; }
  return QMK_OK;
}
// Output matrix of the pair kernel [rows x cols], fp32 or fp16: blocks of 32 rows x 128 bytes, 128-byte swizzle.
int make_map_c(CUtensorMap *map, const void *ptr, uint64_t rows, uint64_t cols, bool f16, std::string *err) {
  EncodeTiledFn enc = encoder();
  if (!enc) { *err = "cuTensorMapEncodeTiled is not available from this driver"; return QMK_ERR_CUDA; }
  const cuuint64_t size = f16 ? 2 : 4;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15u) || (cols * size) % 16) { *err = "matrix not 16-byte aligned"; return QMK_ERR_BAD_ARGUMENT; }
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * size};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / size), 32};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(ptr), dims, strides,
                         box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { *err = "cuTensorMapEncodeTiled (output) failed with code " + std::to_string(static_cast<int>(r)); return QMK_ERR_CUDA; }
  return QMK_OK;
}
int make_map_b(CUtensorMap *map, const void *ptr, uint64_t rows, int K, uint32_t box_rows, int wq, std::string *err) {
  return wq ? make_map_packed(map, ptr, rows, K, box_rows, wq, err) : make_map_f16(map, ptr, rows, static_cast<uint64_t>(K), box_rows, err);
}

// 3-D tensor map of an fp16 KV cache [heads][max_seq_len][128] of which the first `rows` positions of every head are
// valid: boxes of 64 dims x 64 positions of one head, 128-byte swizzle; positions >= rows read as zeros.
int make_map_kv(CUtensorMap *map, const void *cache, uint64_t rows, uint64_t max_seq_len, uint64_t heads, std::string *err) {
  EncodeTiledFn enc = encoder();
  if (!enc) { *err = "cuTensorMapEncodeTiled is not available from this driver"; return QMK_ERR_CUDA; }
  if (reinterpret_cast<uintptr_t>(cache) & 15u) { *err = "cache not 16-byte aligned"; return QMK_ERR_BAD_ARGUMENT; }
  const cuuint64_t dims[3] = {128, rows, heads};
  const cuuint64_t strides[2] = {256, max_seq_len * 256};
  const cuuint32_t box[3] = {64, 64, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(cache), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { *err = "cuTensorMapEncodeTiled (cache) failed with code " + std::to_string(static_cast<int>(r)); return QMK_ERR_CUDA; }
  return QMK_OK;
}

// Width of the N tiles for C[M x N] = A[M x K] * B[N x K]^T (M, N multiples of 128).  `map_b` must have been made
// with that many rows per box.  Skinny problems are bound by how many SMs pull operands at once and by the fixed
// cost of a CTA (launch, barrier and TMEM set-up, pipeline fill, epilogue - worth about 320 columns of streaming in
// the launch lists of decode steps), so: as few waves as possible, then the narrower tile.  `b_tiles` = B tiles a
// CTA multiplies per K block (2 for the fused gate/up kernel, whose widest tile is 64).
static int sm_count() {
  int dev = 0;
  cudaGetDevice(&dev);
  int sms = (dev >= 0 && dev < 16) ? g_sms[dev] : 0;
  if (sms == 0) {
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (dev >= 0 && dev < 16) g_sms[dev] = sms;
  }
  return sms > 0 ? sms : 148;
}
thread_local int t_ah = 1;                     // fp16 halves per activation (SplitActScope)
thread_local const float *t_row_scale[3] = {nullptr, nullptr, nullptr};   // row scales of the next GEMMs' fp16 B matrices
thread_local unsigned int t_ring_budget = 0;   // shared-memory budget of the ring (0 = the compile-time depth, one CTA per SM)
static int pick_box_n(int M, int N, int b_tiles) {
  const int sms = sm_count() * (t_ring_budget ? 2 : 1);   // CTA slots of one wave: rings sized to a budget share an SM in pairs
  int best = 0;
  long best_cost = 0;
  for (int bn = b_tiles == 2 ? 64 : 128; bn >= 32; bn /= 2) {
    const long ctas = static_cast<long>(M / qmk_gemm::BM) * (N / bn);
    const long cost = ((ctas + sms - 1) / sms) * (b_tiles * bn + 320);
    if (best == 0 || cost < best_cost) { best = bn; best_cost = cost; }
  }
  return best;
}
int gemm_sm_count() { return sm_count(); }
int gemm_box_n(int M, int N) { return pick_box_n(M, N, 1); }
int gemm_box_n_fused(int M, int N) { return pick_box_n(M, N, 2); }

// Launches of a decode step, and of a prefill chunk behind its first kernel, carry the programmatic-stream-serialisation
// attribute (see pdl_wait in prefill_kernels.cuh): who builds the chain switches it on for the calling thread.
thread_local bool t_pdl = false;
PdlScope::PdlScope(bool on) : prev_(t_pdl) { t_pdl = on; }
PdlScope::~PdlScope() { t_pdl = prev_; }
bool pdl_active() { return t_pdl; }

// The kernel for an N tile, epilogue and weight format, and its dynamic shared memory.
using GemmKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const qmk_gemm::Groups,
                            int, int, unsigned int *, unsigned long long, int);
// One row tile of at most 64 rows (short A boxes): the tiles decode steps take.
template <int WQ>
static GemmKernel gemm_kernel_64(int bn, bool fuse) {
  if (fuse) return bn == 32 ? qmk_gemm::gemm_f16_tn_kernel<32, true, WQ, 1, false, 64> : nullptr;
  return bn == 32 ? qmk_gemm::gemm_f16_tn_kernel<32, false, WQ, 1, false, 64> : bn == 128 ? qmk_gemm::gemm_f16_tn_kernel<128, false, WQ, 1, false, 64> : nullptr;
}
static GemmKernel gemm_kernel_64(int bn, bool fuse, int wq) {
  return wq == 0 ? gemm_kernel_64<0>(bn, fuse) : wq == 1 ? gemm_kernel_64<1>(bn, fuse) : gemm_kernel_64<2>(bn, fuse);
}
template <int WQ, bool RS = false>
static GemmKernel gemm_kernel_wq(int bn, bool fuse) {
  if (fuse) return bn == 32 ? qmk_gemm::gemm_f16_tn_kernel<32, true, WQ, 1, RS> : qmk_gemm::gemm_f16_tn_kernel<64, true, WQ, 1, RS>;
  return bn == 32 ? qmk_gemm::gemm_f16_tn_kernel<32, false, WQ, 1, RS>
                  : bn == 64 ? qmk_gemm::gemm_f16_tn_kernel<64, false, WQ, 1, RS> : qmk_gemm::gemm_f16_tn_kernel<128, false, WQ, 1, RS>;
}
// Split activations: at most 128 B rows per stage, packed 64.
static GemmKernel gemm_kernel_split(int bn, bool fuse, int wq) {
  if (wq == 0 && bn == (fuse ? 64 : 128)) return fuse ? qmk_gemm::gemm_f16_tn_kernel<64, true, 0, 2> : qmk_gemm::gemm_f16_tn_kernel<128, false, 0, 2>;
  if (fuse) return wq == 0 ? qmk_gemm::gemm_f16_tn_kernel<32, true, 0, 2> : qmk_gemm::gemm_f16_tn_kernel<32, true, 1, 2>;
  if (bn == 32) return wq == 0 ? qmk_gemm::gemm_f16_tn_kernel<32, false, 0, 2> : qmk_gemm::gemm_f16_tn_kernel<32, false, 1, 2>;
  return wq == 0 ? qmk_gemm::gemm_f16_tn_kernel<64, false, 0, 2> : qmk_gemm::gemm_f16_tn_kernel<64, false, 1, 2>;
}
static int split_max_rows(int wq) { return wq == 0 ? 128 : 64; }
static bool box_n_ok(int box_n, bool fuse, int wq) {
  const int rows = fuse ? 2 * box_n : box_n;
  if (t_ah == 2) return wq < 2 && (box_n == 32 || box_n == 64 || box_n == 128) && rows <= split_max_rows(wq);
  return box_n == 32 || box_n == 64 || (box_n == 128 && rows == 128);
}
// (split activations exist for fp16 and FP8 weights; `scaled`: fp16 matrices with row scales)
static GemmKernel gemm_kernel(int bn, bool fuse, int wq, int ah, bool scaled, int am = 128) {
  if (am == 64) return gemm_kernel_64(bn, fuse, wq);
  if (ah == 2) return gemm_kernel_split(bn, fuse, wq);
  if (wq == 0) return scaled ? gemm_kernel_wq<0, true>(bn, fuse) : gemm_kernel_wq<0, false>(bn, fuse);
  return wq == 1 ? gemm_kernel_wq<1>(bn, fuse) : gemm_kernel_wq<2>(bn, fuse);
}
static size_t gemm_smem(int bn, bool fuse, int wq, int ah) { return qmk_gemm::smem_bytes_for(fuse ? 2 * bn : bn, wq, ah); }

// Pairs of CTAs (gemm_pair_tcgen05.cuh): C matrices fp32 or fp16, or the SwiGLU of a gate and an up matrix.
using PairKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap,
                            const CUtensorMap, const qmk_pair::Args,
                            unsigned int *, unsigned long long);
static PairKernel pair_kernel(int mode, bool scaled) {
  if (mode == 0) return scaled ? qmk_pair::gemm_pair_kernel<0, true> : qmk_pair::gemm_pair_kernel<0, false>;
  if (mode == 1) return scaled ? qmk_pair::gemm_pair_kernel<1, true> : qmk_pair::gemm_pair_kernel<1, false>;
  if (mode == 2) return scaled ? qmk_pair::gemm_pair_kernel<2, true> : qmk_pair::gemm_pair_kernel<2, false>;
  if (mode == 3) return scaled ? qmk_pair::gemm_pair_kernel<3, true> : qmk_pair::gemm_pair_kernel<3, false>;
  return scaled ? qmk_pair::gemm_pair_kernel<4, true> : qmk_pair::gemm_pair_kernel<4, false>;
}

// Opt-in shared-memory size of every tile variant, once per device (outside any stream capture).
int ensure_gemm_attrs(std::string *err) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(g_mu);
  if (dev >= 0 && dev < 16 && !g_attr_set[dev]) {
    cudaError_t e = cudaSuccess;
    for (int ah = 1; ah < 3 && e == cudaSuccess; ++ah)
      for (int wq = 0; wq < 4 - ah && e == cudaSuccess; ++wq)
        for (int fuse = 0; fuse < 2 && e == cudaSuccess; ++fuse)
          for (int bn = 32; bn <= (ah == 2 ? split_max_rows(wq) / (fuse ? 2 : 1) : fuse ? 64 : 128) && e == cudaSuccess; bn *= 2)
            for (int scaled = 0; scaled < (wq == 0 && ah == 1 ? 2 : 1) && e == cudaSuccess; ++scaled)
              e = cudaFuncSetAttribute(reinterpret_cast<const void *>(gemm_kernel(bn, fuse != 0, wq, ah, scaled != 0)),
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(gemm_smem(bn, fuse != 0, wq, ah)));
    for (int wq = 0; wq < 3 && e == cudaSuccess; ++wq)
      for (int fuse = 0; fuse < 2 && e == cudaSuccess; ++fuse)
        for (int bn = 32; bn <= 128 && e == cudaSuccess; bn *= 2)
          if (gemm_kernel_64(bn, fuse != 0, wq))
            e = cudaFuncSetAttribute(reinterpret_cast<const void *>(gemm_kernel_64(bn, fuse != 0, wq)), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(qmk_gemm::smem_bytes_for(fuse ? 2 * bn : bn, wq, 1, 64)));
    for (int mode = 0; mode < 5 && e == cudaSuccess; ++mode)
      for (int scaled = 0; scaled < 2 && e == cudaSuccess; ++scaled)
        e = cudaFuncSetAttribute(reinterpret_cast<const void *>(pair_kernel(mode, scaled != 0)), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(qmk_pair::SMEM_BYTES));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(qmk_pf::causal_attention_mma, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               qmk_pf::ATM_SMEM_BYTES);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(qmk_pf::causal_attention_split, cudaFuncAttributeMaxDynamicSharedMemorySize, qmk_pf::ATM_SMEM_BYTES);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(qmk_attn::causal_attention_tc<>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(qmk_attn::SMEM_BYTES));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(qmk_pf::decode_attention_ring, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               qmk_pf::DAR_SMEM_BYTES);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(qmk_pf::decode_attention_mma<>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               qmk_pf::DAM_SMEM_BYTES);
    if (e != cudaSuccess) { *err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e); return QMK_ERR_CUDA; }
    g_attr_set[dev] = true;
  }
  return QMK_OK;
}

// Packed-weight fields of a launch: row geometry for K and the groups' base pointers.
static bool set_packed(qmk_gemm::Groups *gr, int wq, int K, int ngroups, const void *const *raws, std::string *err) {
  for (int g = 0; g < qmk_gemm::MAX_GROUPS; ++g) gr->braw[g] = nullptr;
  gr->raw_pitch = gr->raw_bs_off = gr->raw_scale_off = 0;
  for (int g = 0; g < ngroups; ++g) gr->row_scale[g] = wq == 0 ? t_row_scale[g] : nullptr;
  if (wq == 0) return true;
  if (wq < 0 || wq > 2 || !raws || K > qmk_gemm::MAX_K_PACKED) { *err = "gemm: bad packed-weight arguments"; return false; }
  const PackedRow pr = packed_row(wq, K);
  gr->raw_pitch = pr.pitch;
  gr->raw_bs_off = pr.bs_off;
  gr->raw_scale_off = pr.scale_off;
  for (int g = 0; g < ngroups; ++g) {
    if (!raws[g]) { *err = "gemm: null packed matrix"; return false; }
    gr->braw[g] = static_cast<const unsigned char *>(raws[g]);
  }
  return true;
}

// Ring depth of a launch (see qmk_gemm::ring_geometry): `sb` = B rows per stage; returns the dynamic shared memory.
thread_local float *t_amax_val = nullptr;   // the next single-matrix GEMM of this thread leaves (value, column) pairs here
thread_local int *t_amax_idx = nullptr;
// A launch of at most one CTA per SM takes the full depth whatever the budget: nothing of its own shares the SM, and with the
// three stages of a 128-wide tile that fit 96 KB its K loop waits for L2.  Prompts of 31 / 109 / 500 / 1000 tokens with every
// kernel of the chain a programmatic dependent 1.07 / 1.24 / 1.79 / 2.42 -> 0.91 / 1.06 / 1.56 / 2.10 ms (2000: no such launch).
// `kblocks`: no more stages than that.
static size_t set_ring(qmk_gemm::Groups *gr, int sb, int wq, long ctas, int am, int kblocks) {
  const qmk_gemm::RingGeometry g = qmk_gemm::ring_geometry(sb, wq, ctas > sm_count() ? t_ring_budget : 0, t_ah, am, kblocks);
  gr->stages = g.stages;
  gr->ring_bytes = g.ring_bytes;
  return g.smem_bytes;
}

RingBudgetScope::RingBudgetScope(unsigned int bytes) : prev_(t_ring_budget) { t_ring_budget = bytes; }
RingBudgetScope::~RingBudgetScope() { t_ring_budget = prev_; }
SplitActScope::SplitActScope(bool on) : prev_(t_ah) { t_ah = on ? 2 : 1; }
SplitActScope::~SplitActScope() { t_ah = prev_; }
void set_argmax_target(float *val, int *idx) { t_amax_val = val; t_amax_idx = idx; }
thread_local bool t_out_f16 = false;        // the next grouped GEMM of this thread stores fp16
void set_out_f16(bool on) { t_out_f16 = on; }
size_t selftest_ring(qmk_gemm::Groups *gr) { return set_ring(gr, 128, 0, 1, 128, 1); }

// Weights for the next launches of this thread to bring into L2 (see PrefetchScope).
thread_local PrefetchList t_prefetch;
PrefetchScope::PrefetchScope(const PrefetchList &list) : prev_(t_prefetch) { t_prefetch = list; }
PrefetchScope::~PrefetchScope() { t_prefetch = prev_; }
static void set_prefetch(qmk_gemm::Groups *gr, long ctas) {
  gr->prefetch_behind = t_prefetch.behind;
  for (int i = 0; i < qmk_gemm::MAX_PREFETCH; ++i) {
    gr->prefetch[i] = static_cast<const unsigned char *>(t_prefetch.ptr[i]);
    gr->prefetch_bytes[i] = t_prefetch.ptr[i] ? static_cast<uint32_t>(t_prefetch.bytes[i]) : 0u;
    gr->prefetch_piece[i] = static_cast<uint32_t>(((t_prefetch.bytes[i] + ctas - 1) / ctas + 15) / 16 * 16);
  }
}

// A maps with short boxes (`a_box_rows` < 128 rows per box, a multiple of 8; decode steps with few live rows): one
// row tile only, and the epilogue must stay inside the box.
static bool a_box_ok(int a_box_rows, int M, int *rows, uint32_t *a_box_bytes, std::string *err) {
  *a_box_bytes = 0;
  if (a_box_rows <= 0 || a_box_rows == qmk_gemm::BM) return true;
  if (a_box_rows % 8 || a_box_rows > qmk_gemm::BM || M != qmk_gemm::BM) { *err = "gemm: bad A box"; return false; }
  if (*rows > a_box_rows) *rows = a_box_rows;
  *a_box_bytes = static_cast<uint32_t>(a_box_rows) * qmk_gemm::BK * 2;
  return true;
}

// Rows of the MMA for a launch with `live` rows: 64 where its only row tile has a short A box and the tile has such a kernel, with
// packed weights up to 64, with fp16 weights up to 28 rows.  us per step of fp16 sequences, 64-row -> 128-row products, 48 steps from 64
// tokens, 16 / 20 / 24 / 28 / 30 / 32 / 36 / 40 / 48 / 64 sequences 778 / 730 / 738 / 749 / 756 / 763 / 779 / 838 / 883 / 917 -> 785 / 737 / 742 / 751 /
// 752 / 755 / 771 / 836 / 866 / 902; from 128 to 1024 tokens, 16 / 24 / 28 / 30 / 32 / 40 / 48 / 64 sequences 922 / 1011 / 1055 / 1084 / 1108 / 1224 / 1290 /
// 1475 -> 928 / 1015 / 1059 / 1084 / 1103 / 1206 / 1281 / 1461: the two meet at 29 or 30 (every number from 23 to 42 was timed, three runs
// of a side within 0.1 %).  Packed weights gain at every size.  A row's sums are the same bit for bit.
static int mma_rows(const qmk_gemm::Groups &gr, int live, int box_n, bool fuse, int wq) {
  const bool fits = gr.a_box_bytes > 0 && gr.a_box_bytes <= 64u * qmk_gemm::BK * 2 && t_ah == 1 && gr.row_scale[0] == nullptr && gemm_kernel_64(box_n, fuse, wq);
  return fits && live <= (wq == 0 ? 28 : 64) ? 64 : qmk_gemm::BM;
}

// C_g[M x N_g] fp32 = A[M x K] * B_g[N_g x K]^T for up to three matrices B_g in one launch.  M, N_g multiples of
// 128; K a multiple of 64; every B map made with `box_n` rows per box (gemm_box_n(M, sum of N_g)).
int launch_gemm_grouped(const CUtensorMap &map_a, int ngroups, const CUtensorMap *const *maps_b, float *const *Cs,
                        const int *Ns, int M, int K, int box_n, unsigned int *status, int timeout_ms, cudaStream_t stream,
                        std::string *err, int live_rows, int a_box_rows, int wq, const void *const *raws) {
  bool bad = M <= 0 || K <= 0 || M % qmk_gemm::BM || K % qmk_gemm::BK ||
             !box_n_ok(box_n, false, wq) || ngroups < 1 || ngroups > qmk_gemm::MAX_GROUPS;
  for (int g = 0; !bad && g < ngroups; ++g) bad = Ns[g] <= 0 || Ns[g] % 128;
  if (bad) {
    *err = "gemm: M and N must be multiples of 128 and K a multiple of 64";
    return QMK_ERR_BAD_ARGUMENT;
  }
  const int arc = ensure_gemm_attrs(err);
  if (arc != QMK_OK) return arc;
  qmk_gemm::Groups gr;
  gr.kblocks_per_split = 0;
  gr.split_stride = 0;
  if (!set_packed(&gr, wq, K, ngroups, raws, err)) return QMK_ERR_BAD_ARGUMENT;
  gr.out_f16 = t_out_f16 ? 1 : 0;
  gr.amax_val = ngroups == 1 ? t_amax_val : nullptr;   // (set around the LM-head launch of a decode step only)
  gr.amax_idx = ngroups == 1 ? t_amax_idx : nullptr;
  int tiles = 0;
  for (int g = 0; g < qmk_gemm::MAX_GROUPS; ++g) {
    gr.C[g] = g < ngroups ? Cs[g] : nullptr;
    gr.N[g] = g < ngroups ? Ns[g] : 0;
    tiles += gr.N[g] / box_n;
  }
  const CUtensorMap &b0 = *maps_b[0], &b1 = *maps_b[ngroups > 1 ? 1 : 0], &b2 = *maps_b[ngroups > 2 ? 2 : 0];
  dim3 grid(tiles, M / qmk_gemm::BM);
  const unsigned long long budget = static_cast<unsigned long long>(timeout_ms) * 1000000ull;
  int rows = live_rows > 0 ? live_rows : M;   // rows the epilogue stores (the rest of the tile is padding)
  if (!a_box_ok(a_box_rows, M, &rows, &gr.a_box_bytes, err)) return QMK_ERR_BAD_ARGUMENT;
  const int am = mma_rows(gr, rows, box_n, false, wq);
  set_prefetch(&gr, static_cast<long>(grid.x) * grid.y);
  const size_t smem = set_ring(&gr, box_n, wq, static_cast<long>(grid.x) * grid.y, am, K / qmk_gemm::BK);
  cudaError_t e = launch_kernel(gemm_kernel(box_n, false, wq, t_ah, gr.row_scale[0] != nullptr, am), grid, dim3(qmk_gemm::threads_for(wq, t_ah)), smem, stream,
                                map_a, b0, b1, b2, gr, rows, K, status, budget, 0);
  if (e != cudaSuccess) { *err = std::string("gemm launch: ") + cudaGetErrorString(e); return QMK_ERR_CUDA; }
  return QMK_OK;
}

// act[M x N] fp16 = silu(A * Gate^T) * (A * Up^T): the gate/up pair of the MLP with the SwiGLU in the epilogue.
// Both maps made with `box_n` (64 or 32) rows per box.
int launch_gemm_swiglu(const CUtensorMap &map_a, const CUtensorMap &map_gate, const CUtensorMap &map_up, __half *act, int M,
                       int N, int K, unsigned int *status, int timeout_ms, cudaStream_t stream, std::string *err,
                       int box_n, int live_rows, int a_box_rows, int wq, const void *raw_gate, const void *raw_up) {
  if (M <= 0 || N <= 0 || K <= 0 || M % qmk_gemm::BM || N % 128 || K % qmk_gemm::BK ||
      !box_n_ok(box_n, true, wq)) {
    *err = "gemm: M and N must be multiples of 128 and K a multiple of 64";
    return QMK_ERR_BAD_ARGUMENT;
  }
  const int arc = ensure_gemm_attrs(err);
  if (arc != QMK_OK) return arc;
  qmk_gemm::Groups gr;
  gr.C[0] = reinterpret_cast<float *>(act); gr.C[1] = nullptr; gr.C[2] = nullptr;
  gr.N[0] = N; gr.N[1] = 0; gr.N[2] = 0;
  gr.kblocks_per_split = 0;
  gr.split_stride = 0;
  const void *raws[2] = {raw_gate, raw_up};
  if (!set_packed(&gr, wq, K, 2, raws, err)) return QMK_ERR_BAD_ARGUMENT;
  gr.amax_val = nullptr;
  gr.out_f16 = 0;
  gr.amax_idx = nullptr;
  int rows = live_rows > 0 ? live_rows : M;
  if (!a_box_ok(a_box_rows, M, &rows, &gr.a_box_bytes, err)) return QMK_ERR_BAD_ARGUMENT;
  const unsigned long long budget = static_cast<unsigned long long>(timeout_ms) * 1000000ull;
  const int am = mma_rows(gr, rows, box_n, true, wq);
  set_prefetch(&gr, static_cast<long>(N / box_n) * (M / qmk_gemm::BM));
  const size_t smem = set_ring(&gr, 2 * box_n, wq, static_cast<long>(N / box_n) * (M / qmk_gemm::BM), am, K / qmk_gemm::BK);
  cudaError_t e = launch_kernel(gemm_kernel(box_n, true, wq, t_ah, gr.row_scale[0] != nullptr, am), dim3(N / box_n, M / qmk_gemm::BM), dim3(qmk_gemm::threads_for(wq, t_ah)),
                                smem, stream, map_a, map_gate, map_up, map_up, gr, rows, K, status, budget, 0);
  if (e != cudaSuccess) { *err = std::string("gemm launch: ") + cudaGetErrorString(e); return QMK_ERR_CUDA; }
  return QMK_OK;
}

// Split-K form for problems with few output tiles and a long K (decode steps, O and down of a prefill): `splits` CTAs per
// tile, partial matrices C + z * M * N.  K / 64 must be a multiple of `splits`.  `map_b` made with `box_n` rows per box.
int launch_gemm_splitk(const CUtensorMap &map_a, const CUtensorMap &map_b, float *C, int M, int N, int K, int splits,
                       unsigned int *status, int timeout_ms, cudaStream_t stream, std::string *err, int box_n,
                       int live_rows, int a_box_rows, int wq, const void *raw) {
  if (M <= 0 || N <= 0 || K <= 0 || M % qmk_gemm::BM || N % 128 || K % qmk_gemm::BK || splits < 1 ||
      (K / qmk_gemm::BK) % splits || !box_n_ok(box_n, false, wq) || N % box_n) {
    *err = "gemm: bad split-K shape";
    return QMK_ERR_BAD_ARGUMENT;
  }
  const int arc = ensure_gemm_attrs(err);
  if (arc != QMK_OK) return arc;
  qmk_gemm::Groups gr;
  gr.C[0] = C; gr.C[1] = nullptr; gr.C[2] = nullptr;
  gr.N[0] = N; gr.N[1] = 0; gr.N[2] = 0;
  gr.kblocks_per_split = K / qmk_gemm::BK / splits;
  gr.split_stride = static_cast<size_t>(M) * N;
  if (!set_packed(&gr, wq, K, 1, &raw, err)) return QMK_ERR_BAD_ARGUMENT;
  gr.amax_val = nullptr;
  gr.out_f16 = 0;
  gr.amax_idx = nullptr;
  int rows = live_rows > 0 ? live_rows : M;
  if (!a_box_ok(a_box_rows, M, &rows, &gr.a_box_bytes, err)) return QMK_ERR_BAD_ARGUMENT;
  const unsigned long long budget = static_cast<unsigned long long>(timeout_ms) * 1000000ull;
  const int am = mma_rows(gr, rows, box_n, false, wq);
  set_prefetch(&gr, static_cast<long>(N / box_n) * (M / qmk_gemm::BM) * splits);
  const size_t smem = set_ring(&gr, box_n, wq, static_cast<long>(N / box_n) * (M / qmk_gemm::BM) * splits, am, gr.kblocks_per_split);
  cudaError_t e = launch_kernel(gemm_kernel(box_n, false, wq, t_ah, gr.row_scale[0] != nullptr, am), dim3(N / box_n, M / qmk_gemm::BM, splits), dim3(qmk_gemm::threads_for(wq, t_ah)),
                                smem, stream, map_a, map_b, map_b, map_b, gr, rows, K, status, budget, 0);
  if (e != cudaSuccess) { *err = std::string("gemm launch: ") + cudaGetErrorString(e); return QMK_ERR_CUDA; }
  return QMK_OK;
}

// The pair kernel: up to three matrices B_g (maps with 128 rows per box) against A, mode 0 fp32 (K split in `splits` parts, the
// partial matrices M rounded up to 256 rows apart), 1 fp16, 2 SwiGLU of maps_b[0] (gate) and maps_b[1] (up) with N = Ns[0] outputs,
// 3 fp32 added to C (K in two parts, added in order), 4 q / k / v heads to where `heads` says (no C maps are read).
// maps_c: make_map_c.  M a multiple of 128; the last tile may reach 128 rows past it, as far as the C maps go.
int launch_gemm_pair(int mode, const CUtensorMap &map_a, int ngroups, const CUtensorMap *const *maps_b, const CUtensorMap *const *maps_c,
                     const int *Ns, int M, int K, int splits, unsigned int *status, int timeout_ms, cudaStream_t stream, std::string *err,
                     const qmk_pair::Heads *heads = nullptr) {
  const int columns = mode == 2 ? qmk_pair::TN / 2 : qmk_pair::TN, matrices = mode == 2 ? 1 : ngroups;
  bool bad = mode < 0 || mode > 4 || (mode == 4) != (heads != nullptr) || M <= 0 || M % 128 || K <= 0 || splits < 1 || K % (qmk_pair::BK * splits) || ngroups < 1 || ngroups > 3 ||
             (mode == 2 && ngroups != 2) || (splits > 1 && ((mode != 0 && mode != 3) || ngroups != 1)) || (mode == 3 && splits != 2);
  for (int g = 0; !bad && g < matrices; ++g) bad = Ns[g] <= 0 || Ns[g] % columns;
  for (int g = 0; !bad && g < ngroups; ++g) bad = (t_row_scale[g] == nullptr) != (t_row_scale[0] == nullptr);   // scales for all or for none
  if (bad) { *err = "gemm: bad shape for pairs of CTAs"; return QMK_ERR_BAD_ARGUMENT; }
  const int arc = ensure_gemm_attrs(err);
  if (arc != QMK_OK) return arc;
  qmk_pair::Args a;
  a.heads = heads ? *heads : qmk_pair::Heads{};
  a.n_tiles = 0;
  for (int g = 0; g < 3; ++g) {
    a.N[g] = g < matrices ? Ns[g] : 0;
    a.row_scale[g] = g < ngroups ? t_row_scale[g] : nullptr;
    a.n_tiles += a.N[g] / columns;
  }
  a.m_tiles = (M + qmk_pair::TM - 1) / qmk_pair::TM;
  a.splits = splits;
  a.kblocks = K / qmk_pair::BK / splits;
  const int tiles = a.m_tiles * a.n_tiles * (mode == 3 ? 1 : splits), pairs = std::min(tiles, sm_count() / 2);
  const unsigned long long budget = static_cast<unsigned long long>(timeout_ms) * 1000000ull;
  const cudaError_t e = launch_kernel(pair_kernel(mode, a.row_scale[0] != nullptr), dim3(2 * pairs), dim3(qmk_pair::THREADS), qmk_pair::SMEM_BYTES, stream,
                                      map_a, *maps_b[0], *maps_b[ngroups > 1 ? 1 : 0], *maps_b[ngroups > 2 ? 2 : 0], *maps_c[0], *maps_c[matrices > 1 ? 1 : 0], *maps_c[matrices > 2 ? 2 : 0],
                                      a, status, budget);
  if (e != cudaSuccess) { *err = std::string("gemm launch: ") + cudaGetErrorString(e); return QMK_ERR_CUDA; }
  return QMK_OK;
}

int launch_gemm(const CUtensorMap &map_a, const CUtensorMap &map_b, float *C, int M, int N, int K, int box_n,
                unsigned int *status, int timeout_ms, cudaStream_t stream, std::string *err, int live_rows, int a_box_rows,
                int wq, const void *raw) {
  const CUtensorMap *maps[1] = {&map_b};
  float *Cs[1] = {C};
  const int Ns[1] = {N};
  return launch_gemm_grouped(map_a, 1, maps, Cs, Ns, M, K, box_n, status, timeout_ms, stream, err, live_rows, a_box_rows, wq,
                             &raw);
}

}  // namespace qmk_tc

// ----------------------------------------------------------------------------- chunked prefill
namespace {

constexpr unsigned int PREFILL_RING_BYTES = 96 * 1024;
constexpr int PAIR_MIN_ROWS = 512;
constexpr int EXPAND_MIN_ROWS = 512;
constexpr int CHUNK = 4096;         // prompt tokens per pass over the weights (a multiple of the GEMM's 128)
constexpr int MAX_LAYERS = 48;

struct Workspace {                  // per device, allocated on first use, never freed (like the engine's scratch)
  bool ready = false;
  int *tokens = nullptr;
  float *x = nullptr, *q = nullptr, *k = nullptr, *v = nullptr, *qr = nullptr, *o = nullptr, *down = nullptr;
  __half *xn = nullptr, *attn = nullptr, *act = nullptr;
  unsigned int *status = nullptr;
  CUtensorMap map_xn, map_attn, map_act, map_qh;
  CUtensorMap map_cq, map_ck, map_cv, map_cact, map_co, map_cdown, map_cx;   // outputs of the pair GEMMs
  CUtensorMap map_xn2, map_attn2, map_act2;   // split activations: rows of hi and lo halves
  // batched decode: per-sequence state and the logits of one step
  bool decode_ready = false;
  int *positions = nullptr, *start_positions = nullptr;
  cudaStream_t gstream = nullptr;        // capture needs a non-default stream
  cudaEvent_t ev_in = nullptr, ev_out = nullptr;
  // One captured decode step per batch size (a serving loop's live count changes from round to round and
  // instantiating ~200 nodes costs tens of milliseconds); entry B is valid while its key matches.
  cudaGraphExec_t step_graph[129] = {};
  unsigned long long step_key[129][12] = {};
  unsigned long long graph_epoch = 1;    // bumped whenever tensor maps baked into the graphs are rebuilt
  __half **k_ptrs = nullptr, **v_ptrs = nullptr;
  CUtensorMap *kv_maps = nullptr;        // [128][2]: tiled-copy descriptors of every sequence's K and V cache (decode_attention_mma)
  unsigned char *packed = nullptr;       // tables of a packed prefill (row info, attention items, per-sequence descriptors and cache pointers)
  // pinned source of these tables and the pass's tokens, two that passes take in turn: a pass is prepared while the one before runs
  unsigned char *staging[2] = {nullptr, nullptr};
  cudaEvent_t staged[2] = {nullptr, nullptr};   // the copies out of it are done
  int **log_ptrs = nullptr;
  float *split_part = nullptr;            // partial attention states of split sequences (both decode attention kernels)
  qmk_pf::DamPlan *attn_plan = nullptr;   // the step's list of attention pieces (decode_attention_mma)
  unsigned int *split_count = nullptr;    // arrival counters, one per (sequence, kv head); zero between launches
  float *logits = nullptr;
  int logits_vocab = 0;
  float *amax_val = nullptr;              // [128][vocab / 128] pairs of the LM-head epilogue's greedy pick
  int *amax_idx = nullptr;
  const void *lm_ptr = nullptr;
  int lm_wq = 0;
  CUtensorMap map_lm;
  // A-operand maps that expose only the live rows: the rest of the 128-row box is zero-filled by the TMA unit
  // without being read, which cuts the activation traffic of a small batch by 128 / rows
  int a_rows = 0;
  CUtensorMap map_xn_b, map_attn_b, map_act_b;
  // weight maps of the layer table seen last (rebuilt when the table's contents change)
  unsigned long long table[MAX_LAYERS * 12] = {};
  int table_layers = 0;
  // packed weights, long prefill chunks: one layer's matrices as fp16 values, their row scales and maps
  __half *expanded = nullptr;
  float *expanded_scale = nullptr;
  CUtensorMap emap[7][2];              // boxes of 64 and 128 rows
  CUtensorMap emap32[7];
  int table_wq = 0;                    // weight format the maps below were made for
  CUtensorMap wmap[MAX_LAYERS][7][2];  // q, k, v, o, gate, up, down; boxes of 64 and 128 rows
  CUtensorMap wmap32[MAX_LAYERS][7];   // the same matrices in boxes of 32 rows (decode steps: more, smaller tiles)
};
// Prefill and batched decode keep separate workspaces and locks: a serving loop prefills the next request on one
// stream (and thread) while a decode step of the live sequences runs on another.
Workspace g_ws[16], g_ws_decode[16];
std::recursive_mutex g_ws_mu;   // (recursive: qmk_tc::prefill_split's caller holds it already, see prefill_lock)
std::atomic<int> g_ws_waiting{0};   // threads that wait for it
std::unique_lock<std::recursive_mutex> lock_workspace() {
  std::unique_lock<std::recursive_mutex> lock(g_ws_mu, std::try_to_lock);
  if (!lock) {
    ++g_ws_waiting;
    lock.lock();
    --g_ws_waiting;
  }
  return lock;
}
// Leaves the workspace to a thread that waits for it (a mutex that is released and taken again at once stays with its thread).
void let_another_in(std::unique_lock<std::recursive_mutex> &lock) {
  const int seen = g_ws_waiting.load();
  lock.unlock();
  for (int i = 0; i < 200 && seen > 0 && g_ws_waiting.load() >= seen; ++i) std::this_thread::sleep_for(std::chrono::microseconds(10));
  lock = lock_workspace();
}
std::mutex g_ws_decode_mu;

#define PF_CUDA(call)                                                                             \
  do {                                                                                            \
    cudaError_t err__ = (call);                                                                   \
    if (err__ != cudaSuccess)                                                                     \
      return qmk_internal::report(QMK_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(err__)); \
  } while (0)

cudaError_t device_memory(void **at, size_t bytes) { return cudaMalloc(at, bytes); }

// `rows`: activation rows the buffers hold (CHUNK for prefill, four 128-row tiles of partial sums for the batched decode).  All or nothing:
// buffers that were made are given back when a later one does not fit.  `no_room`: set (and nothing reported) where the
// reason is memory, for callers with another way.
int ensure_workspace(Workspace &w, int rows, bool *no_room = nullptr) {
  if (w.ready) return QMK_OK;
  using namespace qmk_pf;
  const size_t C = static_cast<size_t>(rows);
  const qmk_tc::Buffer buffers[] = {
      {reinterpret_cast<void **>(&w.tokens), sizeof(int) * C},
      {reinterpret_cast<void **>(&w.x), sizeof(float) * C * H},
      {reinterpret_cast<void **>(&w.q), sizeof(float) * C * QS},
      {reinterpret_cast<void **>(&w.k), sizeof(float) * C * KVS},
      {reinterpret_cast<void **>(&w.v), sizeof(float) * C * KVS},
      {reinterpret_cast<void **>(&w.qr), sizeof(float) * C * QS},
      {reinterpret_cast<void **>(&w.o), sizeof(float) * 2 * C * H},      // (two split-K partial matrices of a prefill chunk)
      {reinterpret_cast<void **>(&w.down), sizeof(float) * 2 * C * H},
      // (room for the hi and lo halves of split activations, [C][2 x width])
      {reinterpret_cast<void **>(&w.xn), sizeof(__half) * C * 2 * H},
      {reinterpret_cast<void **>(&w.attn), sizeof(__half) * C * 2 * QS},
      {reinterpret_cast<void **>(&w.act), sizeof(__half) * C * 2 * I},
      {reinterpret_cast<void **>(&w.status), 16}};
  cudaError_t e = qmk_tc::make_all(buffers, cudaSuccess, device_memory, cudaFree);
  // GEMM operand rows beyond a short chunk are read: zeros at first, later what earlier passes left there (any bits: a pass with
  // split activations uses the same memory in another layout).  They reach their own rows of a product only, which nobody uses.
  for (const qmk_tc::Buffer &b : buffers)
    if (e == cudaSuccess) e = cudaMemset(*b.at, 0, b.bytes);
  if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);   // (a caller's stream may not wait for the legacy one)
  std::string err;
  int rc = e == cudaSuccess ? QMK_OK : QMK_ERR_CUDA;
  if (rc != QMK_OK) err = std::string("workspace of the tensor-core path: ") + cudaGetErrorString(e);
  if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&w.map_xn, w.xn, C, H, qmk_gemm::BM, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&w.map_attn, w.attn, C, QS, qmk_gemm::BM, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&w.map_act, w.act, C, I, qmk_gemm::BM, &err);
  // the rotated queries as fp16 (the first half of the fp32 buffer), read by the attention kernel in 128-row boxes
  if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&w.map_qh, w.qr, C, QS, qmk_gemm::BM, &err);
  // the same buffers as [C][hi | lo]
  if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&w.map_xn2, w.xn, C, 2 * H, qmk_gemm::BM, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&w.map_attn2, w.attn, C, 2 * QS, qmk_gemm::BM, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&w.map_act2, w.act, C, 2 * I, qmk_gemm::BM, &err);
  // outputs of the pair GEMMs: q, k, v as fp16, the SwiGLU, fp32 sums (or partial matrices)
  if (rc == QMK_OK) rc = qmk_tc::make_map_c(&w.map_cq, w.q, C, QS, true, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_c(&w.map_ck, w.k, C, KVS, true, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_c(&w.map_cv, w.v, C, KVS, true, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_c(&w.map_cact, w.act, C, I, true, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_c(&w.map_co, w.o, 2 * C, H, false, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_c(&w.map_cdown, w.down, 2 * C, H, false, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_c(&w.map_cx, w.x, C, H, false, &err);
  if (rc != QMK_OK) {
    qmk_tc::drop_all(buffers, cudaFree);
    cudaGetLastError();
    if (no_room && e == cudaErrorMemoryAllocation) { *no_room = true; return rc; }
    return qmk_internal::report(rc, err);
  }
  w.ready = true;
  return QMK_OK;
}

// q, k, v, o, gate, up, down of a layer
constexpr int MAT_ROWS[7] = {qmk_pf::QS, qmk_pf::KVS, qmk_pf::KVS, qmk_pf::H, qmk_pf::I, qmk_pf::I, qmk_pf::H};
constexpr int MAT_COLS[7] = {qmk_pf::H, qmk_pf::H, qmk_pf::H, qmk_pf::QS, qmk_pf::H, qmk_pf::H, qmk_pf::I};

size_t weight_bytes(int j, int wq) { return static_cast<size_t>(MAT_ROWS[j]) * (wq ? qmk_tc::packed_row(wq, MAT_COLS[j]).pitch : 2u * MAT_COLS[j]); }

// Buffers of the expanded layer (32 MB), on first use.  Where they do not fit in memory `expanded` stays null.
int ensure_expanded(Workspace &w) {
  if (w.expanded) return QMK_OK;
  size_t values = 0, rows = 0;
  for (int j = 0; j < 7; ++j) { values += static_cast<size_t>(MAT_ROWS[j]) * MAT_COLS[j]; rows += MAT_ROWS[j]; }
  __half *buf = nullptr;
  float *scale = nullptr;
  if (cudaMalloc(&buf, values * sizeof(__half)) != cudaSuccess || cudaMalloc(&scale, rows * sizeof(float)) != cudaSuccess) {
    cudaGetLastError();
    if (buf) cudaFree(buf);
    return QMK_OK;
  }
  std::string err;
  int rc = QMK_OK;
  size_t at = 0;
  for (int j = 0; j < 7 && rc == QMK_OK; ++j) {
    rc = qmk_tc::make_map_f16(&w.emap32[j], buf + at, MAT_ROWS[j], MAT_COLS[j], 32, &err);
    for (int b = 0; b < 2 && rc == QMK_OK; ++b) rc = qmk_tc::make_map_f16(&w.emap[j][b], buf + at, MAT_ROWS[j], MAT_COLS[j], 64 << b, &err);
    at += static_cast<size_t>(MAT_ROWS[j]) * MAT_COLS[j];
  }
  if (rc != QMK_OK) { cudaFree(buf); cudaFree(scale); return qmk_internal::report(rc, err); }
  w.expanded = buf;
  w.expanded_scale = scale;
  return QMK_OK;
}

// Tensor maps of the seven projection matrices of every layer.  The layer table lives in device memory
// (the reference's packed pointer records): it is read back and the maps are rebuilt only when it changed.
int ensure_weight_maps(Workspace &w, const LDGLayerWeight *layers_dev, int num_layers, int wq, cudaStream_t stream) {
  using namespace qmk_pf;
  std::vector<unsigned long long> host(static_cast<size_t>(num_layers) * 12);
  PF_CUDA(cudaMemcpyAsync(host.data(), layers_dev, host.size() * 8, cudaMemcpyDeviceToHost, stream));
  PF_CUDA(cudaStreamSynchronize(stream));
  if (w.table_layers == num_layers && w.table_wq == wq && memcmp(host.data(), w.table, host.size() * 8) == 0) return QMK_OK;
  // record order: in_ln, wq, wk, wv, q_norm, k_norm, wo, post_ln, gate, up, down, pad
  static const int slot[7] = {1, 2, 3, 6, 8, 9, 10};
  std::string err;
  w.table_layers = 0;   // (until all maps are made: a table that is refused below has replaced some)
  for (int l = 0; l < num_layers; ++l)
    for (int j = 0; j < 7; ++j) {
      const void *ptr = reinterpret_cast<const void *>(host[static_cast<size_t>(l) * 12 + slot[j]]);
      if (!ptr) return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "prefill: null weight pointer in the layer table");
      {
        const int rc = qmk_tc::make_map_b(&w.wmap32[l][j], ptr, MAT_ROWS[j], MAT_COLS[j], 32, wq, &err);
        if (rc != QMK_OK) return qmk_internal::report(rc, err);
      }
      for (int b = 0; b < 2; ++b) {
        const int rc = qmk_tc::make_map_b(&w.wmap[l][j][b], ptr, MAT_ROWS[j], MAT_COLS[j], 64 << b, wq, &err);
        if (rc != QMK_OK) return qmk_internal::report(rc, err);
      }
    }
  memcpy(w.table, host.data(), host.size() * 8);
  w.table_layers = num_layers;
  w.table_wq = wq;
  ++w.graph_epoch;   // captured decode steps hold the old maps
  return QMK_OK;
}

}  // namespace

namespace {
// Several prompts in one pass: sequence s holds lens[s] tokens (concatenated in token_ids_host) and owns the caches
// k_caches[s] / v_caches[s]; every sequence starts at position 0.
struct PackedSeqs {
  int num_seqs;
  const int *lens;
  void *const *k_caches, *const *v_caches;
};
// One of the passes of a call: the first one under a hold of the workspace reads the layer table and clears the status, the last one
// waits and reports.  All of a call run with the options that pass 0 found: the maps are those of its weight format.
struct Pass { bool first = true, last = true; int index = 0; qmk_internal::WeightOptions *options = nullptr; };
constexpr int MAX_PACKED_SEQS = 64;
constexpr size_t PK_ROWS_OFF = 0, PK_ITEMS_OFF = 32768, PK_MAPS_OFF = 49152, PK_PTRS_OFF = 65536, PK_BYTES = 66560;

// Null where pinned memory is refused: pageable memory serves then, whose copies may hold the host up.
unsigned char *staging_slot(Workspace &w, int slot) {
  if (!w.staging[slot]) {
    void *at = nullptr;
    cudaEvent_t done = nullptr;
    if (cudaHostAlloc(&at, PK_BYTES + sizeof(int) * CHUNK, cudaHostAllocDefault) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    if (cudaEventCreateWithFlags(&done, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); cudaFreeHost(at); return nullptr; }
    w.staging[slot] = static_cast<unsigned char *>(at);
    w.staged[slot] = done;
  }
  return w.staging[slot];
}

int prefill_impl(const int *token_ids_host, int num_tokens, const void *embed_weight, const LDGLayerWeight *layer_weights,
                 const void *cos_table, const void *sin_table, void *k_cache, void *v_cache, int num_layers,
                 int start_position, int max_seq_len, float attn_scale, cudaStream_t stream, const PackedSeqs *pk, bool split,
                 bool *take_steps = nullptr, const Pass &pass = Pass()) {
  using namespace qmk_pf;
  if (num_tokens <= 0) return QMK_OK;
  qmk_internal::PrefillEnv env;
  int rc = qmk_internal::prefill_env(max_seq_len, stream, &env, pass.options, pass.index == 0);
  if (rc != QMK_OK) return rc;
  if (split) env.attn_tc = 0;   // (split operands have an attention kernel of their own)
  if (!token_ids_host || !embed_weight || !layer_weights || (!pk && (!k_cache || !v_cache)))
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "prefill: null pointer argument");
  const int wfmt = env.wfmt;   // 0 fp16, 1 FP8-E4M3 rows, 2 NVFP4 rows
  int wq = wfmt;               // the format the GEMMs of a chunk read: packed matrices are expanded inside them, or per layer (long chunks)
  if (num_layers < 1 || num_layers > MAX_LAYERS)
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "num_layers must be in [1, 48]");
  if (!pk && (start_position < 0 || start_position + num_tokens > max_seq_len))
    return qmk_internal::report(QMK_ERR_POSITION, "start_position + steps exceeds max_seq_len");
  if (pk) {
    if (pk->num_seqs < 1 || pk->num_seqs > MAX_PACKED_SEQS || !pk->lens || !pk->k_caches || !pk->v_caches || start_position != 0)
      return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "packed prefill: 1 to 64 sequences, each from position 0");
    int total = 0;
    for (int s = 0; s < pk->num_seqs; ++s) {
      if (pk->lens[s] < 1 || !pk->k_caches[s] || !pk->v_caches[s])
        return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "packed prefill: empty sequence or null cache");
      if (pk->lens[s] > max_seq_len) return qmk_internal::report(QMK_ERR_POSITION, "a prompt exceeds max_seq_len");
      total += pk->lens[s];
    }
    if (total != num_tokens) return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "packed prefill: lengths do not add up to num_tokens");
  }
  if (env.rope_from_table && (!cos_table || !sin_table))
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "rope_from_table needs cos/sin tables");
  for (int i = 0; i < num_tokens; ++i)
    if (token_ids_host[i] < 0 || token_ids_host[i] >= env.vocab)
      return qmk_internal::report(QMK_ERR_BAD_TOKEN, "prompt token outside [0, vocab)");
  int dev = 0;
  PF_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 16) return qmk_internal::report(QMK_ERR_CUDA, "device index out of range");
  const auto lock = lock_workspace();
  Workspace &w = g_ws[dev];
  rc = ensure_workspace(w, CHUNK, take_steps);
  if (rc == QMK_OK && pass.first) rc = ensure_weight_maps(w, layer_weights, num_layers, wq, stream);
  if (rc != QMK_OK) return rc;
  // ---- packed prompts: rows = the sequences one after the other, each padded to whole 128-row tiles
  std::vector<unsigned char> pageable;
  const int slot = pass.index & 1;
  int pk_items = 0;
  if (pk) {
    if (!env.attn_tc) return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "packed prefill needs the tcgen05 attention kernel");
    if (!w.packed) PF_CUDA(cudaMalloc(&w.packed, PK_BYTES));
    unsigned char *host = staging_slot(w, slot);
    if (host) {
      PF_CUDA(cudaEventSynchronize(w.staged[slot]));      // (two passes back)
    } else {
      pageable.resize(PK_BYTES + sizeof(int) * CHUNK);
      host = pageable.data();
    }
    memset(host, 0, PK_BYTES);
    int *const padded_tokens = reinterpret_cast<int *>(host + PK_BYTES);
    int2 *rows = reinterpret_cast<int2 *>(host + PK_ROWS_OFF);
    int4 *items = reinterpret_cast<int4 *>(host + PK_ITEMS_OFF);
    CUtensorMap *maps = reinterpret_cast<CUtensorMap *>(host + PK_MAPS_OFF);
    unsigned long long *ptrs = reinterpret_cast<unsigned long long *>(host + PK_PTRS_OFF);
    int total_rows = 0;
    for (int s = 0; s < pk->num_seqs; ++s) total_rows += (pk->lens[s] + qmk_gemm::BM - 1) / qmk_gemm::BM * qmk_gemm::BM;
    if (total_rows > CHUNK) return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "packed prefill: more than 4096 padded rows");
    for (int i = 0; i < total_rows; ++i) { padded_tokens[i] = 0; rows[i] = make_int2(0, -1); }
    std::vector<std::pair<int, int4>> order;   // (key tiles, item)
    std::string merr;
    int row0 = 0, tok0 = 0;
    for (int s = 0; s < pk->num_seqs; ++s) {
      const int len = pk->lens[s];
      for (int i = 0; i < len; ++i) {
        padded_tokens[row0 + i] = token_ids_host[tok0 + i];
        rows[row0 + i] = make_int2(s, i);
      }
      ptrs[2 * s] = reinterpret_cast<unsigned long long>(pk->k_caches[s]);
      ptrs[2 * s + 1] = reinterpret_cast<unsigned long long>(pk->v_caches[s]);
      int mrc = qmk_tc::make_map_kv(&maps[2 * s], pk->k_caches[s], static_cast<uint64_t>(len), static_cast<uint64_t>(max_seq_len),
                                    static_cast<uint64_t>(num_layers) * NKV, &merr);
      if (mrc == QMK_OK)
        mrc = qmk_tc::make_map_kv(&maps[2 * s + 1], pk->v_caches[s], static_cast<uint64_t>(len), static_cast<uint64_t>(max_seq_len),
                                  static_cast<uint64_t>(num_layers) * NKV, &merr);
      if (mrc != QMK_OK) return qmk_internal::report(mrc, merr);
      for (int qt = 0; qt * qmk_attn::TQ < len; ++qt) {
        const int last = (qt + 1) * qmk_attn::TQ < len ? (qt + 1) * qmk_attn::TQ - 1 : len - 1;
        for (int h = 0; h < NQ; ++h)
          order.push_back({last / qmk_attn::TK + 1, make_int4(s, row0 + qt * qmk_attn::TQ, qt * qmk_attn::TQ, h | (len << 8))});
      }
      row0 += (len + qmk_gemm::BM - 1) / qmk_gemm::BM * qmk_gemm::BM;
      tok0 += len;
    }
    std::stable_sort(order.begin(), order.end(), [](const auto &a, const auto &b) { return a.first > b.first; });   // longest job first
    pk_items = static_cast<int>(order.size());
    for (int i = 0; i < pk_items; ++i) items[i] = order[i].second;
    // Both copies out of the staging memory, then its event: whatever fails behind them, the pass that takes the slot next waits.
    cudaError_t copied = cudaMemcpyAsync(w.packed, host, PK_BYTES, cudaMemcpyHostToDevice, stream);
    if (copied == cudaSuccess) copied = cudaMemcpyAsync(w.tokens, padded_tokens, sizeof(int) * total_rows, cudaMemcpyHostToDevice, stream);
    if (pageable.empty()) PF_CUDA(cudaEventRecord(w.staged[slot], stream));
    PF_CUDA(copied);
    num_tokens = total_rows;      // (one chunk)
  }
  std::vector<unsigned long long> rec(w.table, w.table + static_cast<size_t>(num_layers) * 12);
  const float *rope = env.rope_from_table ? nullptr : env.rope;
  const __half *cosv = static_cast<const __half *>(cos_table), *sinv = static_cast<const __half *>(sin_table);
  const size_t layer_stride = static_cast<size_t>(NKV) * max_seq_len * D;
  if (pass.first) PF_CUDA(cudaMemsetAsync(w.status, 0, 16, stream));
  std::string err;
  // weight matrix j of layer l in boxes of `box_n` rows
  auto wmap_for = [&](int l, int j, int box_n) -> const CUtensorMap & {
    if (wq != wfmt) return box_n == 32 ? w.emap32[j] : w.emap[j][box_n == 64 ? 0 : 1];
    return box_n == 32 ? w.wmap32[l][j] : w.wmap[l][j][box_n == 64 ? 0 : 1];
  };
  static const int rec_slot[7] = {1, 2, 3, 6, 8, 9, 10};   // q, k, v, o, gate, up, down inside a layer record
  auto wptr = [&](int l, int j) { return reinterpret_cast<const void *>(rec[static_cast<size_t>(l) * 12 + rec_slot[j]]); };
  // row scales of expanded matrices for the next launch
  auto row_scales = [&](const int *js, int n) {
    for (int i = 0; i < 3; ++i) qmk_tc::t_row_scale[i] = nullptr;
    if (wq == wfmt) return;
    for (int i = 0; i < n; ++i) {
      int first = 0;
      for (int j = 0; j < js[i]; ++j) first += MAT_ROWS[j];
      qmk_tc::t_row_scale[i] = w.expanded_scale + first;
    }
  };
  struct ClearScales { ~ClearScales() { for (int i = 0; i < 3; ++i) qmk_tc::t_row_scale[i] = nullptr; } } clear_scales;   // on every way out
  // packed weights with split activations take narrower tiles
  auto split_box = [&](int box_n, int widest) { return split && wq != 0 && box_n > widest ? widest : box_n; };
  bool by_pairs = false;   // this chunk's GEMMs run on pairs of CTAs
  // several matrices against the same activations in one launch (q/k/v)
  auto gemm_group = [&](const CUtensorMap &a, int l, int n, const int *js, float *const *cs, const int *ns, int M, int K,
                        int live, const qmk_pair::Heads *heads) {
    int total = 0;
    for (int i = 0; i < n; ++i) total += ns[i];
    if (by_pairs) {
      const CUtensorMap *maps[3];
      for (int i = 0; i < n; ++i) maps[i] = &wmap_for(l, js[i], 128);
      const CUtensorMap *const out[3] = {&w.map_cq, &w.map_ck, &w.map_cv};
      row_scales(js, n);
      return qmk_tc::launch_gemm_pair(heads ? 4 : 1, a, n, maps, out, ns, M, K, 1, w.status, env.timeout_ms, stream, &err, heads);
    }
    const int box_n = split_box(qmk_tc::gemm_box_n(M, total), 64);
    const CUtensorMap *maps[3];
    const void *raws[3] = {nullptr, nullptr, nullptr};
    for (int i = 0; i < n; ++i) { maps[i] = &wmap_for(l, js[i], box_n); raws[i] = wptr(l, js[i]); }
    row_scales(js, n);
    return qmk_tc::launch_gemm_grouped(a, n, maps, cs, ns, M, K, box_n, w.status, env.timeout_ms, stream, &err, live, 0, wq,
                                       raws);
  };
  if ((rc = qmk_tc::ensure_gemm_attrs(&err)) != QMK_OK) return qmk_internal::report(rc, err);
  for (int c0 = 0; c0 < num_tokens; c0 += CHUNK) {
    const int T = (num_tokens - c0 < CHUNK) ? num_tokens - c0 : CHUNK;
    const int M = (T + qmk_gemm::BM - 1) / qmk_gemm::BM * qmk_gemm::BM;
    const int pos0 = start_position + c0;
    // Packed weights, long chunks: a GEMM expands its weight tile once per 128 rows; from EXPAND_MIN_ROWS rows on it is
    // cheaper to expand the layer's matrices once and run the fp16 form, on pairs of CTAs above 512 rows.  FP8 / NVFP4, in the
    // GEMMs -> expanded: 250 tokens 1.42 / 1.44 -> 1.60 / 1.57 ms, 380: 1.73 / 1.72 -> 1.85 / 1.82, 500: 2.02 / 1.98 -> 1.92 (NVFP4),
    // 1000: 3.35 / 3.19 -> 2.40 / 2.41, 4000: 10.6 / 10.1 -> 7.1 / 7.1.
    wq = wfmt;
    if (wfmt != 0 && !split && M >= EXPAND_MIN_ROWS) {
      rc = ensure_expanded(w);
      if (rc != QMK_OK) return rc;
      if (w.expanded) wq = 0;
    }
    // Chunks of more than four row tiles run on pairs of CTAs (fp16 weights, expanded packed ones).  760 / 1000 / 1500 / 2000 /
    // 4000 / 8191 tokens, single CTAs -> pairs: 2.01 / 2.10 / 3.17 / 3.74 / 8.10 / 20.4 -> 1.79 / 2.03 / 2.55 / 3.28 / 6.77 /
    // 17.6 ms; 500 tokens 1.56 -> 1.61, 250 tokens 1.21 -> 1.40 (a 256 x 256 tile for each pair leaves most pairs idle).
    by_pairs = wq == 0 && !split && M > PAIR_MIN_ROWS;
    // The O and down projections have only 1024 output columns.  K is split so that their tiles fill the SMs; the partial
    // matrices are added by the residual + RMSNorm kernel that follows anyway (or by the pairs, below).  Four parts below 1024 rows (M = 512: 32 tiles x
    // 4 = 128 CTAs with K loops of 8 / 12 blocks; unsplit, the narrowest tiles gave 128 CTAs with loops of 32 / 48 blocks of N =
    // 32 MMAs and these two products were 41 % of the pass), two above: the sums, and with them the last bits of every row behind,
    // do not depend on which kernel made them.  (One part where the pairs would fill the SMs without
    // a split: 4000 tokens 6.59 -> 6.50 ms, and NVFP4 batches whose picks were ties to 1e-3 went another way.)
    // Packed weights split only short chunks: a CTA expands its weight tile itself, so two CTAs with half a K loop each beat
    // one only while there are too few tiles (93 tokens 2.06 -> 1.75 ms; 1023 tokens measured 1 % slower with two splits).
    const int od_splits = M < 1024 ? 4 : wq == 0 ? 2 : 1;
    // Two parts whose 128-wide tiles all find an SM of their own (1024 and 1152 rows) stay with single CTAs: 32 or 40 tiles of
    // 256 x 256 leave half of the pairs idle (1000 tokens, with four parts to fill them, 2.03 ms; here 2.02).
    const bool od_pairs = by_pairs && (M < 1024 || static_cast<long>(M / qmk_gemm::BM) * (H / 128) * od_splits > qmk_tc::gemm_sm_count());
    // Where the two parts of all tiles are more than one round of the pairs anyway (ten row tiles, 2305 tokens, on 148 SMs), a pair makes
    // both parts of a tile and adds them to the residual rows itself, in the order in which the RMSNorm kernel added them: the same
    // bits without writing and reading two matrices of partial sums (32 MB each way at 4096 rows; a row kernel 12 -> 5 us, a product
    // 19 -> 21).  2400 / 3000 / 3500 / 4096 / 8191 tokens 4.23 / 5.02 / 5.93 / 6.83 / 17.67 -> 4.00 / 4.74 / 5.55 / 6.53 / 17.05 ms, NVFP4
    // 4096 6.69 -> 6.28.  Below the line half as many pairs work twice as long: 1300 / 1700 / 2048 / 2300 tokens 2.43 / 2.81 / 3.03 /
    // 3.43 ms with partial sums, 2.73 / 3.10 / 3.27 / 3.54 without.
    const bool od_adds = od_pairs && od_splits == 2 && static_cast<long>((M + qmk_pair::TM - 1) / qmk_pair::TM) * (H / qmk_pair::TN) * 2 > qmk_tc::gemm_sm_count() / 2;
    const size_t od_stride = static_cast<size_t>(od_pairs ? (M + qmk_pair::TM - 1) / qmk_pair::TM * qmk_pair::TM : M) * H;
    auto gemm_od = [&](const CUtensorMap &a, int l, int j, float *c, int Mrows, int K, int live) {
      row_scales(&j, 1);
      if (od_pairs) {
        const CUtensorMap *const map = &wmap_for(l, j, 128);
        const CUtensorMap *const out = od_adds ? &w.map_cx : c == w.o ? &w.map_co : &w.map_cdown;
        const int n = H;
        return qmk_tc::launch_gemm_pair(od_adds ? 3 : 0, a, 1, &map, &out, &n, Mrows, K, od_splits, w.status, env.timeout_ms, stream, &err);
      }
      if (od_splits == 1) {
        const int box_n = split_box(qmk_tc::gemm_box_n(Mrows, H), 64);
        return qmk_tc::launch_gemm(a, wmap_for(l, j, box_n), c, Mrows, H, K, box_n, w.status, env.timeout_ms, stream, &err, live, 0, wq,
                                   wptr(l, j));
      }
      // the narrowest tile whose CTAs fit on the SMs at once: a 128-row chunk has 32 CTAs of 128 columns, whose epilogues alone
      // took 2.1 us (31 / 109 / 250 tokens 0.91 / 1.06 / 1.27 -> 0.85 / 0.94 / 1.21 ms; from 500 tokens on the tile is the same)
      int box_n = 32;
      while (box_n < split_box(128, 64) && static_cast<long>(Mrows / qmk_gemm::BM) * (H / box_n) * od_splits > qmk_tc::gemm_sm_count()) box_n *= 2;
      return qmk_tc::launch_gemm_splitk(a, wmap_for(l, j, box_n), c, Mrows, H, K, od_splits, w.status, env.timeout_ms, stream, &err, box_n,
                                        live, 0, wq, wptr(l, j));
    };
    // Weights for the launches of this chunk to bring into L2 (single CTAs multiplying a layer's matrices as they are).
    auto ahead_of = [&](int l, std::initializer_list<int> js) {
      qmk_tc::PrefetchList list;
      int i = 0;
      for (int j : js)
        if (!by_pairs && wq == wfmt && l < num_layers) {
          list.ptr[i] = wptr(l, j);
          list.bytes[i++] = weight_bytes(j, wq);
        }
      return list;
    };
    CUtensorMap map_kc, map_vc;   // the caches up to this chunk's last position, all layers
    memset(&map_kc, 0, sizeof(map_kc));
    memset(&map_vc, 0, sizeof(map_vc));
    if (env.attn_tc && !pk) {
      rc = qmk_tc::make_map_kv(&map_kc, k_cache, static_cast<uint64_t>(pos0 + T), static_cast<uint64_t>(max_seq_len),
                               static_cast<uint64_t>(num_layers) * NKV, &err);
      if (rc == QMK_OK)
        rc = qmk_tc::make_map_kv(&map_vc, v_cache, static_cast<uint64_t>(pos0 + T), static_cast<uint64_t>(max_seq_len),
                                 static_cast<uint64_t>(num_layers) * NKV, &err);
      if (rc != QMK_OK) break;
    }
    if (!pk) PF_CUDA(cudaMemcpyAsync(w.tokens, token_ids_host + c0, sizeof(int) * T, cudaMemcpyHostToDevice, stream));
    // Every kernel behind the first launches as a programmatic dependent: its set-up (and a GEMM's first ring fill of WEIGHT
    // tiles) runs under the tail of the kernel before it.  In order are, with each kernel waiting for its predecessor before
    // its first dependent read and any write: the residual rows and sums; the expanded matrices of a packed layer
    // (expand_packed_rows waits for the last GEMM that multiplies them, and the first GEMM that requests tiles of them ahead
    // of its own wait is launched after the row kernel between has seen the expansion complete).  109 / 1000 / 2000 tokens,
    // GEMMs alone dependent -> all: 1.41 / 2.59 / 3.80 -> 1.24 / 2.42 / 3.74 ms.
    qmk_tc::PdlScope pdl_scope(env.pdl != 0);
    qmk_tc::SplitActScope split_scope(split);
    const CUtensorMap &map_xn = split ? w.map_xn2 : w.map_xn, &map_attn = split ? w.map_attn2 : w.map_attn,
                      &map_act = split ? w.map_act2 : w.map_act;
    // two GEMM CTAs per SM: one's epilogue under the other's main loop (split activations take the SM's whole TMEM: one CTA)
    qmk_tc::RingBudgetScope ring_scope(split ? 0 : PREFILL_RING_BYTES);
    {
      qmk_tc::PdlScope first(false);            // (follows a copy, not a kernel)
      PF_CUDA(qmk_tc::launch_kernel(embed_rows, dim3(T), dim3(256), 0, stream, w.tokens, embed_weight, wfmt, w.x));
    }
    // residual add (+ split-K partials) and RMSNorm: a warp per row for long chunks, a block per row for short ones
    auto norm_rows = [&](const float *add, const __half *g) {
      if (od_adds) add = nullptr;
      if (T >= 256 && od_splits <= 2)
        return qmk_tc::launch_kernel(split ? add_rmsnorm_rows_wide<true> : add_rmsnorm_rows_wide<false>, dim3((T + 7) / 8), dim3(256), 0,
                                     stream, w.x, add, od_splits, od_stride, g, w.xn, T, w.status + qmk_gemm::STATUS_BEYOND);
      return qmk_tc::launch_kernel(split ? add_rmsnorm_rows<true> : add_rmsnorm_rows<false>, dim3(T), dim3(256), 0, stream, w.x, add, od_splits, od_stride, g, w.xn,
                                   w.status + qmk_gemm::STATUS_BEYOND);
    };
    for (int l = 0; l < num_layers; ++l) {
      const unsigned long long *r = rec.data() + static_cast<size_t>(l) * 12;
      __half *kc = pk ? nullptr : static_cast<__half *>(k_cache) + l * layer_stride;
      __half *vc = pk ? nullptr : static_cast<__half *>(v_cache) + l * layer_stride;
      if (wq != wfmt) {
        qmk_gemm::ExpandArgs a;
        size_t at = 0;
        a.first_row[0] = 0;
        for (int j = 0; j < 7; ++j) {
          const qmk_tc::PackedRow pr = qmk_tc::packed_row(wfmt, MAT_COLS[j]);
          a.src[j] = static_cast<const unsigned char *>(wptr(l, j));
          a.dst[j] = w.expanded + at;
          a.scale[j] = w.expanded_scale + a.first_row[j];
          a.first_row[j + 1] = a.first_row[j] + MAT_ROWS[j];
          a.K[j] = MAT_COLS[j];
          a.pitch[j] = pr.pitch; a.bs_off[j] = pr.bs_off; a.scale_off[j] = pr.scale_off;
          at += static_cast<size_t>(MAT_ROWS[j]) * MAT_COLS[j];
        }
        // (the last layer stops after its q/k/v product)
        if (l == num_layers - 1) for (int j = 4; j < 8; ++j) a.first_row[j] = a.first_row[3];
        const dim3 grid((a.first_row[7] + qmk_gemm::EXPAND_THREADS / 32 - 1) / (qmk_gemm::EXPAND_THREADS / 32));
        PF_CUDA(qmk_tc::launch_kernel(wfmt == 1 ? qmk_gemm::expand_packed_rows<1> : qmk_gemm::expand_packed_rows<2>, grid,
                                      dim3(qmk_gemm::EXPAND_THREADS), 0, stream, a));
      }
      PF_CUDA(norm_rows(l > 0 ? w.down : nullptr, reinterpret_cast<const __half *>(r[0])));
      // On pairs of CTAs the product's epilogue normalises, rotates and stores the heads (fp16 queries, as the tcgen05 attention
      // kernel reads them).  520 / 777 / 1024 / 1300 / 2200 / 3500 / 6000 / 8191 tokens, with a kernel of its own -> in the epilogue:
      // 1.697 / 1.922 / 2.046 / 2.43 / 3.21 / 5.55 / 11.4 / 16.95 -> 1.70 / 1.91 / 2.02 / 2.35 / 3.08 / 5.35 / 10.9 / 16.4 ms.  (On single CTAs,
      // 128 threads walking TMEM eight columns at a time, slower than 2300 x 4 parallel blocks.)
      const bool heads_in_gemm = by_pairs && env.attn_tc;
      {
        qmk_pair::Heads heads;
        heads.q_norm = reinterpret_cast<const __half *>(r[4]);
        heads.k_norm = reinterpret_cast<const __half *>(r[5]);
        heads.rope = rope; heads.cos_table = cosv; heads.sin_table = sinv;
        heads.queries = reinterpret_cast<__half *>(w.qr);
        heads.k_cache = kc; heads.v_cache = vc;
        heads.row_info = pk ? reinterpret_cast<const int2 *>(w.packed + PK_ROWS_OFF) : nullptr;
        heads.kv_ptrs = pk ? reinterpret_cast<const unsigned long long *>(w.packed + PK_PTRS_OFF) : nullptr;
        heads.layer_off = static_cast<size_t>(l) * layer_stride;
        heads.rows = T; heads.pos0 = pos0; heads.max_seq_len = max_seq_len;
        heads.q_scale = attn_scale * 1.4426950408889634f;
        const int js[3] = {0, 1, 2};
        float *const cs[3] = {w.q, w.k, w.v};
        const int ns[3] = {QS, KVS, KVS};
        // fp16 q / k / v: every CTA of this launch reaches its epilogue at the same time, and the burst of stores set
        // its length (9.8 of 26 us at 2048 rows with fp32); the consumer below rounds to fp16 anyway
        // (split activations: fp32, the operands downstream are not rounded to fp16)
        qmk_tc::set_out_f16(!split);
        const qmk_tc::PrefetchScope ahead(l + 1 < num_layers ? ahead_of(l, {3}) : qmk_tc::PrefetchList());   // (the last layer ends here)
        rc = gemm_group(map_xn, l, 3, js, cs, ns, M, H, T, heads_in_gemm ? &heads : nullptr);
        qmk_tc::set_out_f16(false);
        if (rc != QMK_OK) break;
      }
      if (!heads_in_gemm)
        PF_CUDA(qmk_tc::launch_kernel(qk_norm_rope_cache, dim3(T), dim3(256), 0, stream, w.q, w.k, w.v, split ? 0 : 1,
                                    reinterpret_cast<const __half *>(r[4]), reinterpret_cast<const __half *>(r[5]), rope, cosv, sinv,
                                    w.qr, kc, vc, pos0, max_seq_len,
                                    pk ? reinterpret_cast<const int2 *>(w.packed + PK_ROWS_OFF) : nullptr,
                                    pk ? reinterpret_cast<const unsigned long long *>(w.packed + PK_PTRS_OFF) : nullptr,
                                    static_cast<size_t>(l) * layer_stride,
                                    env.attn_tc ? attn_scale * 1.4426950408889634f : 0.f));
      if (l == num_layers - 1) break;   // the cache is complete; nothing downstream of the last layer is kept
      if (env.attn_tc)
        PF_CUDA(qmk_tc::launch_kernel(qmk_attn::causal_attention_tc<>, dim3(pk ? pk_items : (T + qmk_attn::TQ - 1) / qmk_attn::TQ * NQ),
                                      dim3(qmk_attn::THREADS), qmk_attn::SMEM_BYTES, stream, w.map_qh, map_kc, map_vc, l * NKV, w.attn, T,
                                      pos0, attn_scale, w.status, static_cast<unsigned long long>(env.timeout_ms) * 1000000ull,
                                      pk ? reinterpret_cast<const int4 *>(w.packed + PK_ITEMS_OFF) : nullptr,
                                      pk ? reinterpret_cast<const CUtensorMap *>(w.packed + PK_MAPS_OFF) : nullptr));
      else if (split) {
        const int qtiles = (T + ATM_Q - 1) / ATM_Q, ktiles = (pos0 + T + ATM_KEYS - 1) / ATM_KEYS;
        // Two CTAs fit on an SM: fewer query tiles than that share out their keys, down to four key tiles each.  The partial
        // outputs go where q, k and v were (their values are in the cache and in qr by now).
        int splits = 2 * qmk_tc::gemm_sm_count() / (qtiles * NKV);
        if (splits > ktiles / 4) splits = ktiles / 4;
        if (splits > ATS_MAX_SPLITS) splits = ATS_MAX_SPLITS;
        if (splits < 1 || static_cast<size_t>(splits) * T * NQ * ATS_PART > static_cast<size_t>(CHUNK) * QS) splits = 1;
        PF_CUDA(qmk_tc::launch_kernel(causal_attention_split, dim3(qtiles, NKV, splits), dim3(ATM_THREADS), ATM_SMEM_BYTES, stream, w.qr,
                                      kc, vc, w.attn, w.q, T, pos0, max_seq_len, attn_scale));
        if (splits > 1)
          PF_CUDA(qmk_tc::launch_kernel(merge_attention_splits, dim3(T), dim3(512), 0, stream, w.q, splits, w.attn, T));
      } else
        PF_CUDA(qmk_tc::launch_kernel(causal_attention_mma, dim3((T + ATM_Q - 1) / ATM_Q, NKV), dim3(ATM_THREADS), ATM_SMEM_BYTES, stream,
                                      w.qr, kc, vc, w.attn, T, pos0, max_seq_len, attn_scale));
      {
        const qmk_tc::PrefetchScope ahead(ahead_of(l, {4, 5, 6}));
        rc = gemm_od(map_attn, l, 3, w.o, M, QS, T);
      }
      if (rc != QMK_OK) break;
      PF_CUDA(norm_rows(w.o, reinterpret_cast<const __half *>(r[7])));
      {
        const int box_gu = split_box(qmk_tc::gemm_box_n_fused(M, I), 32);
        const int js[2] = {4, 5};
        row_scales(js, 2);
        if (by_pairs) {
          const CUtensorMap *const maps[2] = {&wmap_for(l, 4, 128), &wmap_for(l, 5, 128)};
          const CUtensorMap *const out = &w.map_cact;
          const int n = I;
          rc = qmk_tc::launch_gemm_pair(2, map_xn, 2, maps, &out, &n, M, H, 1, w.status, env.timeout_ms, stream, &err);
        } else {
          rc = qmk_tc::launch_gemm_swiglu(map_xn, wmap_for(l, 4, box_gu), wmap_for(l, 5, box_gu), w.act, M, I, H, w.status,
                                          env.timeout_ms, stream, &err, box_gu, T, 0, wq, wptr(l, 4), wptr(l, 5));
        }
        if (rc != QMK_OK) break;
      }
      const qmk_tc::PrefetchScope ahead(ahead_of(l + 1, {0, 1, 2}));
      rc = gemm_od(map_act, l, 6, w.down, M, I, T);
      if (rc != QMK_OK) break;
    }
    if (rc != QMK_OK) break;
    PF_CUDA(cudaGetLastError());     // (the next chunk's token copy is stream-ordered behind this chunk's kernels)
  }
  if (rc != QMK_OK) return qmk_internal::report(rc, err);
  if (!pass.last) return QMK_OK;
  unsigned int host_status[4] = {0, 0, 0, 0};
  PF_CUDA(cudaMemcpyAsync(host_status, w.status, 16, cudaMemcpyDeviceToHost, stream));
  PF_CUDA(cudaStreamSynchronize(stream));
  if (host_status[0] != 0)
    return qmk_internal::report(static_cast<int>(host_status[0]) == 5 ? QMK_ERR_CUDA : static_cast<int>(host_status[0]),
                                host_status[0] == 5 ? "prefill: dynamic shared memory of the attention kernel is not 1024-byte aligned"
                                                    : "prefill: a bounded device wait ran out");
  if (split && host_status[qmk_gemm::STATUS_BEYOND] != 0) *take_steps = true;
  return QMK_OK;
}
}  // namespace

extern "C" int qmk_prefill_chunked(const int *token_ids_host, int num_tokens, const void *embed_weight,
                                   const LDGLayerWeight *layer_weights, const void *cos_table, const void *sin_table,
                                   void *k_cache, void *v_cache, int num_layers, int start_position, int max_seq_len,
                                   float attn_scale, cudaStream_t stream) {
  qmk_internal::begin_call();
  return prefill_impl(token_ids_host, num_tokens, embed_weight, layer_weights, cos_table, sin_table, k_cache, v_cache, num_layers,
                      start_position, max_seq_len, attn_scale, stream, nullptr, false);
}

namespace qmk_tc {
// The chunked pass with split activations, for qmk_prefill (fp32 activations at the precision of the token-serial kernels).
// Locks: the caller takes prefill_lock() BEFORE the engine's lock and holds both - the order in which every other path
// meets them (prefill_impl reports errors to the engine while it holds the workspace).  `take_steps`: set, with
// nothing reported, where the pass is not the way: the workspace does not fit in memory, or an activation exceeded the range
// of its halves (65504; the cache rows are then to be written again).
std::unique_lock<std::recursive_mutex> prefill_lock() { return lock_workspace(); }
int prefill_split(const int *token_ids_host, int num_tokens, const void *embed_weight, const LDGLayerWeight *layer_weights,
                  const void *cos_table, const void *sin_table, void *k_cache, void *v_cache, int num_layers, int start_position,
                  int max_seq_len, float attn_scale, cudaStream_t stream, bool *take_steps) {
  return prefill_impl(token_ids_host, num_tokens, embed_weight, layer_weights, cos_table, sin_table, k_cache, v_cache, num_layers,
                      start_position, max_seq_len, attn_scale, stream, nullptr, true, take_steps);
}
}  // namespace qmk_tc

extern "C" int qmk_prefill_packed(const int *token_ids_host, int num_seqs, const int *seq_lens, const void *embed_weight,
                                  const LDGLayerWeight *layer_weights, const void *cos_table, const void *sin_table,
                                  void *const *k_caches, void *const *v_caches, int num_layers, int max_seq_len, float attn_scale,
                                  cudaStream_t stream) {
  qmk_internal::begin_call();
  if (num_seqs <= 0) return QMK_OK;
  if (!seq_lens) return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "packed prefill: null lengths");
  long total = 0;
  for (int s = 0; s < num_seqs && s < MAX_PACKED_SEQS; ++s) total += seq_lens[s] > 0 ? seq_lens[s] : 0;
  const PackedSeqs pk = {num_seqs, seq_lens, k_caches, v_caches};
  return prefill_impl(token_ids_host, static_cast<int>(total), embed_weight, layer_weights, cos_table, sin_table, nullptr, nullptr,
                      num_layers, 0, max_seq_len, attn_scale, stream, &pk, false);
}

extern "C" int qmk_prefill_packed_passes(const int *token_ids_host, int num_passes, const int *seqs_per_pass, const int *seq_lens,
                                         const void *embed_weight, const LDGLayerWeight *layer_weights, const void *cos_table,
                                         const void *sin_table, void *const *k_caches, void *const *v_caches, int num_layers,
                                         int max_seq_len, float attn_scale, cudaStream_t stream) {
  qmk_internal::begin_call();
  if (num_passes <= 0) return QMK_OK;
  if (!token_ids_host || !seqs_per_pass || !seq_lens || !k_caches || !v_caches)
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "packed prefill: null array argument");
  for (int p = 0; p < num_passes; ++p)
    if (seqs_per_pass[p] < 1 || seqs_per_pass[p] > MAX_PACKED_SEQS)
      return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "packed prefill: 1 to 64 sequences a pass, each from position 0");
  // The passes share one workspace and one status, so the lock is held over them - until another thread wants it: the pass that is
  // being sent then ends as the last one of a call does, and the others follow behind that thread's.
  auto lock = lock_workspace();
  bool first = true;
  qmk_internal::WeightOptions options;
  int rc = QMK_OK;
  for (int p = 0, s0 = 0; p < num_passes && rc == QMK_OK; s0 += seqs_per_pass[p++]) {
    long total = 0;
    for (int s = 0; s < seqs_per_pass[p]; ++s) total += seq_lens[s0 + s] > 0 ? seq_lens[s0 + s] : 0;
    const PackedSeqs pk = {seqs_per_pass[p], seq_lens + s0, k_caches + s0, v_caches + s0};
    Pass pass;
    pass.first = first;
    pass.last = first = p + 1 == num_passes || g_ws_waiting.load() > 0;
    pass.index = p;
    pass.options = &options;
    rc = total < 1 ? qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "packed prefill: empty sequence or null cache")
                   : prefill_impl(token_ids_host, static_cast<int>(total), embed_weight, layer_weights, cos_table, sin_table, nullptr, nullptr,
                                  num_layers, 0, max_seq_len, attn_scale, stream, &pk, false, nullptr, pass);
    if (rc == QMK_OK && pass.last && p + 1 < num_passes) let_another_in(lock);
    if (rc != QMK_OK && p > 0) cudaStreamSynchronize(stream);   // the passes before it are done, as behind calls of their own
    token_ids_host += total;
  }
  return rc;
}

// ----------------------------------------------------------------------------- batched decode on the GEMM path
namespace {
unsigned int __float_as_uint_host(float f) {
  unsigned int u;
  memcpy(&u, &f, 4);
  return u;
}

constexpr int MAX_BATCH = 128;      // one 128-row GEMM tile of sequences

constexpr int MAX_ATTN_SPLITS = 8;
constexpr size_t SPLIT_PART_FLOATS = static_cast<size_t>(MAX_BATCH) * qmk_pf::NKV * MAX_ATTN_SPLITS * 2 * (qmk_pf::D + 2);
constexpr int MAX_ATTN_CTAS = 1024;
static_assert(qmk_pf::dam_max_states(MAX_BATCH, MAX_ATTN_CTAS) * qmk_pf::DAM_PART <= SPLIT_PART_FLOATS &&
                  MAX_BATCH <= qmk_pf::DAM_MAX_BATCH && MAX_LAYERS <= qmk_pf::DAM_MAX_LAYERS, "partial states of decode_attention_mma");
int ensure_decode_workspace(Workspace &w, const void *lm_head, int vocab, int wq) {
  if (!w.decode_ready) {
    const qmk_tc::Buffer buffers[] = {
        {reinterpret_cast<void **>(&w.positions), sizeof(int) * MAX_BATCH},
        {reinterpret_cast<void **>(&w.start_positions), sizeof(int) * MAX_BATCH},
        {reinterpret_cast<void **>(&w.k_ptrs), sizeof(void *) * MAX_BATCH},
        {reinterpret_cast<void **>(&w.v_ptrs), sizeof(void *) * MAX_BATCH},
        {reinterpret_cast<void **>(&w.log_ptrs), sizeof(void *) * MAX_BATCH},
        {reinterpret_cast<void **>(&w.kv_maps), sizeof(CUtensorMap) * 2 * MAX_BATCH},
        {reinterpret_cast<void **>(&w.split_part), sizeof(float) * SPLIT_PART_FLOATS},
        {reinterpret_cast<void **>(&w.attn_plan), sizeof(qmk_pf::DamPlan) + sizeof(qmk_pf::DamPiece) * qmk_pf::dam_max_pieces(MAX_BATCH, MAX_ATTN_CTAS)},
        {reinterpret_cast<void **>(&w.split_count), sizeof(unsigned int) * MAX_BATCH * qmk_pf::NKV}};
    if (!w.gstream) PF_CUDA(cudaStreamCreateWithFlags(&w.gstream, cudaStreamNonBlocking));
    if (!w.ev_in) PF_CUDA(cudaEventCreateWithFlags(&w.ev_in, cudaEventDisableTiming));
    if (!w.ev_out) PF_CUDA(cudaEventCreateWithFlags(&w.ev_out, cudaEventDisableTiming));
    const cudaError_t e = qmk_tc::make_all(buffers, cudaSuccess, device_memory, cudaFree);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return qmk_internal::report(QMK_ERR_CUDA, std::string("workspace of the batched decode: ") + cudaGetErrorString(e));
    }
    w.decode_ready = true;
  }
  if (w.logits_vocab < vocab) {
    if (w.logits) cudaFree(w.logits);
    w.logits = nullptr;
    w.logits_vocab = 0;
    PF_CUDA(cudaMalloc(&w.logits, sizeof(float) * static_cast<size_t>(MAX_BATCH) * vocab));
    if (w.amax_val) cudaFree(w.amax_val);
    if (w.amax_idx) cudaFree(w.amax_idx);
    w.amax_val = nullptr;
    w.amax_idx = nullptr;
    PF_CUDA(cudaMalloc(&w.amax_val, sizeof(float) * static_cast<size_t>(MAX_BATCH) * (vocab / 128)));
    PF_CUDA(cudaMalloc(&w.amax_idx, sizeof(int) * static_cast<size_t>(MAX_BATCH) * (vocab / 128)));
    w.logits_vocab = vocab;
    w.lm_ptr = nullptr;
  }
  if (w.lm_ptr != lm_head || w.lm_wq != wq) {
    std::string err;
    const int rc = qmk_tc::make_map_b(&w.map_lm, lm_head, vocab, qmk_pf::H, 128, wq, &err);
    if (rc != QMK_OK) return qmk_internal::report(rc, err);
    w.lm_ptr = lm_head;
    w.lm_wq = wq;
    ++w.graph_epoch;
  }
  return QMK_OK;
}
}  // namespace

extern "C" int qmk_decode_batched(int num_sequences, const int *first_token_ids, const int *start_positions, int num_steps,
                                  const void *embed_weight, const LDGLayerWeight *layer_weights,
                                  const void *final_norm_weight, const void *lm_head_weight, const void *cos_table,
                                  const void *sin_table, void *const *k_caches, void *const *v_caches,
                                  int *const *output_logs, int num_layers, int max_seq_len, float attn_scale,
                                  cudaStream_t stream) {
  qmk_internal::begin_call();
  using namespace qmk_pf;
  if (num_steps <= 0) return QMK_OK;
  qmk_internal::PrefillEnv env;
  int rc = qmk_internal::prefill_env(max_seq_len, stream, &env);
  if (rc != QMK_OK) return rc;
  if (num_sequences < 1 || num_sequences > MAX_BATCH)
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "qmk_decode_batched: num_sequences must be in [1, 128]");
  if (!first_token_ids || !start_positions || !k_caches || !v_caches || !output_logs || !embed_weight || !layer_weights ||
      !final_norm_weight || !lm_head_weight)
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "qmk_decode_batched: null pointer argument");
  const int wq = env.wfmt;   // packed FP8 / NVFP4 matrices stay packed in HBM and are expanded inside the GEMMs
  if (env.vocab % 128 != 0)
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "qmk_decode_batched needs a vocabulary that is a multiple of 128");
  if (num_layers < 1 || num_layers > MAX_LAYERS)
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "num_layers must be in [1, 48]");
  if (env.rope_from_table && (!cos_table || !sin_table))
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "rope_from_table needs cos/sin tables");
  const int B = num_sequences;
  for (int b = 0; b < B; ++b) {
    if (!k_caches[b] || !v_caches[b] || !output_logs[b])
      return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "qmk_decode_batched: null cache or log pointer");
    if (start_positions[b] < 0 || start_positions[b] + num_steps > max_seq_len)
      return qmk_internal::report(QMK_ERR_POSITION, "start_position + steps exceeds max_seq_len");
    if (first_token_ids[b] < 0 || first_token_ids[b] >= env.vocab)
      return qmk_internal::report(QMK_ERR_BAD_TOKEN, "first token outside [0, vocab)");
    for (int a = 0; a < b; ++a)
      if (k_caches[a] == k_caches[b] || v_caches[a] == v_caches[b] || output_logs[a] == output_logs[b])
        return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "qmk_decode_batched: two sequences share a cache or an output log");
  }
  int dev = 0;
  PF_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 16) return qmk_internal::report(QMK_ERR_CUDA, "device index out of range");
  std::lock_guard<std::mutex> lock(g_ws_decode_mu);
  Workspace &w = g_ws_decode[dev];
  rc = ensure_workspace(w, 512);   // room for the split-K partial matrices (4 x 128 rows)
  if (rc == QMK_OK) rc = ensure_weight_maps(w, layer_weights, num_layers, wq, stream);
  if (rc == QMK_OK) rc = ensure_decode_workspace(w, lm_head_weight, env.vocab, wq);
  if (rc != QMK_OK) return rc;
  std::vector<unsigned long long> rec(w.table, w.table + static_cast<size_t>(num_layers) * 12);
  const float *rope = env.rope_from_table ? nullptr : env.rope;
  const __half *cosv = static_cast<const __half *>(cos_table), *sinv = static_cast<const __half *>(sin_table);
  const size_t layer_stride = static_cast<size_t>(NKV) * max_seq_len * D;
  PF_CUDA(cudaMemsetAsync(w.status, 0, 16, stream));
  // (the attention kernels leave their arrival counters at zero; a call that failed half-way may not have)
  PF_CUDA(cudaMemsetAsync(w.split_count, 0, sizeof(unsigned int) * MAX_BATCH * NKV, stream));
  PF_CUDA(cudaMemcpyAsync(w.tokens, first_token_ids, sizeof(int) * B, cudaMemcpyHostToDevice, stream));
  PF_CUDA(cudaMemcpyAsync(w.positions, start_positions, sizeof(int) * B, cudaMemcpyHostToDevice, stream));
  PF_CUDA(cudaMemcpyAsync(w.start_positions, start_positions, sizeof(int) * B, cudaMemcpyHostToDevice, stream));
  PF_CUDA(cudaMemcpyAsync(w.k_ptrs, k_caches, sizeof(void *) * B, cudaMemcpyHostToDevice, stream));
  PF_CUDA(cudaMemcpyAsync(w.v_ptrs, v_caches, sizeof(void *) * B, cudaMemcpyHostToDevice, stream));
  PF_CUDA(cudaMemcpyAsync(w.log_ptrs, output_logs, sizeof(void *) * B, cudaMemcpyHostToDevice, stream));
  std::string err;
  std::vector<CUtensorMap> host_maps;
  if (env.attn_mma) {   // per-sequence descriptors of the whole [layer][kv head][position] caches, boxes of 16 rows x 64 dims
    host_maps.resize(2 * static_cast<size_t>(B));
    const uint64_t cache_rows = static_cast<uint64_t>(num_layers) * NKV * static_cast<uint64_t>(max_seq_len);
    for (int b = 0; b < B && rc == QMK_OK; ++b) {
      rc = qmk_tc::make_map_f16(&host_maps[2 * b], k_caches[b], cache_rows, D, 16, &err);
      if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&host_maps[2 * b + 1], v_caches[b], cache_rows, D, 16, &err);
    }
    if (rc != QMK_OK) return qmk_internal::report(rc, err);
    PF_CUDA(cudaMemcpyAsync(w.kv_maps, host_maps.data(), sizeof(CUtensorMap) * host_maps.size(), cudaMemcpyHostToDevice, stream));
    PF_CUDA(cudaStreamSynchronize(stream));   // (the pageable host vector must outlive the copy)
  }
  if ((rc = qmk_tc::ensure_gemm_attrs(&err)) != QMK_OK) return qmk_internal::report(rc, err);
  (void)qmk_tc::gemm_box_n(128, 128);   // caches the SM count before any capture
  {
    const int rows = (B + 7) / 8 * 8;
    if (w.a_rows != rows) {
      // boxes of just the live rows: the rest of the 128-row tile in shared memory is never written (nor needed)
      rc = qmk_tc::make_map_f16(&w.map_xn_b, w.xn, rows, H, rows, &err);
      if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&w.map_attn_b, w.attn, rows, QS, rows, &err);
      if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&w.map_act_b, w.act, rows, I, rows, &err);
      if (rc != QMK_OK) return qmk_internal::report(rc, err);
      w.a_rows = rows;   // (graphs captured earlier keep their own copies of the maps they were captured with)
    }
  }
  const int M = qmk_gemm::BM;   // one tile of rows; rows >= B are computed and ignored
  // One decode step for all sequences, enqueued on `s`.  Everything that changes from step to step (tokens,
  // positions) or from call to call (cache and log pointers) lives in device arrays at fixed addresses, so the
  // same sequence of launches - and a graph captured from it - serves every step.
  // The O (K = 2048) and down (K = 3072) projections have only 1024 output columns: K is split four ways and the
  // following RMSNorm adds the partial matrices.
  // N tiles of 32 columns: 128 (q/k/v), 96 (gate/up) and, with K split four ways, 128 CTAs (O, down) per GEMM
  // instead of 64 / 48 / 32-48 with 64-wide tiles; a decode step is bound by how many SMs pull weights at once.
  // The epilogues store only the B live rows of the 128-row tile (the LM head alone would otherwise write
  // 78 MB of padding logits per step).  Measured: 6.5 k -> 7.5 k tok/s at B = 16, 18.3 k -> 21.0 k at B = 64.
  constexpr int TILE_N = 32, O_SPLITS = 4, DOWN_SPLITS = 4;
  const int live = B, a_box = w.a_rows;
  // decode_attention_mma shares all cache rows out among two CTAs per SM.
  const int attn_ctas = std::min(2 * qmk_tc::g_sms[dev], MAX_ATTN_CTAS);
  // decode_attention_ring, few sequences: split every sequence's cache rows over several CTAs so that the attention fills the device
  // (two CTAs fit on an SM): 8 B CTAs otherwise, each streaming a whole sequence through one ring.
  int attn_splits = (2 * qmk_tc::g_sms[dev]) / (B * NKV);   // (gemm_box_n above cached the SM count of this device)
  attn_splits = attn_splits < 1 ? 1 : attn_splits > MAX_ATTN_SPLITS ? MAX_ATTN_SPLITS : attn_splits;
  const size_t PART = static_cast<size_t>(M) * H;
  auto enqueue_step = [&](cudaStream_t s) -> int {
    int r2 = QMK_OK;
    qmk_tc::PdlScope pdl_scope(env.pdl != 0);   // every launch below may start behind its predecessor's tail
    {
      qmk_tc::PdlScope first(false);            // (the first kernel of a step has no predecessor inside the step)
      PF_CUDA(qmk_tc::launch_kernel(embed_rows_and_plan, dim3(B + 1), dim3(256), 0, s, w.tokens, embed_weight, wq, env.vocab, w.x, w.positions,
                                    attn_ctas, w.attn_plan, w.status));
    }
    for (int l = 0; l < num_layers; ++l) {
      const unsigned long long *r = rec.data() + static_cast<size_t>(l) * 12;
      const size_t layer_off = l * layer_stride;
      auto wm = [&](int j) -> const CUtensorMap & { return w.wmap32[l][j]; };
      static const int rec_slot[7] = {1, 2, 3, 6, 8, 9, 10};   // q, k, v, o, gate, up, down inside a layer record
      auto wp = [&](int j) { return reinterpret_cast<const void *>(r[rec_slot[j]]); };
      auto ahead_of = [&](int layer, std::initializer_list<int> js) {
        qmk_tc::PrefetchList list;
        list.behind = true;
        int i = 0;
        for (int j : js)
          if (layer < num_layers) {
            list.ptr[i] = reinterpret_cast<const void *>(rec[static_cast<size_t>(layer) * 12 + rec_slot[j]]);
            list.bytes[i++] = weight_bytes(j, wq);
          }
        return list;
      };
      PF_CUDA(qmk_tc::launch_kernel(add_rmsnorm_rows<false>, dim3(B), dim3(256), 0, s, w.x, l > 0 ? w.down : nullptr, DOWN_SPLITS, PART,
                                    reinterpret_cast<const __half *>(r[0]), w.xn, nullptr));
      {
        const CUtensorMap *maps[3] = {&wm(0), &wm(1), &wm(2)};
        float *const cs[3] = {w.q, w.k, w.v};
        const int ns[3] = {QS, KVS, KVS};
        const void *raws[3] = {wp(0), wp(1), wp(2)};
        const qmk_tc::PrefetchScope ahead(ahead_of(l, {3}));
        if ((r2 = qmk_tc::launch_gemm_grouped(w.map_xn_b, 3, maps, cs, ns, M, H, TILE_N, w.status, env.timeout_ms, s, &err,
                                              live, a_box, wq, raws)) != QMK_OK)
          return r2;
      }
      if (env.attn_mma)
        PF_CUDA(qmk_tc::launch_kernel(decode_attention_mma<>, dim3(attn_ctas), dim3((DAM_WARPS + 1) * 32), DAM_SMEM_BYTES, s,
                                      w.q, w.k, w.v, reinterpret_cast<const __half *>(r[4]), reinterpret_cast<const __half *>(r[5]),
                                      rope, cosv, sinv, w.k_ptrs, w.v_ptrs, layer_off, w.attn_plan, l, w.attn, max_seq_len, attn_scale,
                                      w.status, static_cast<unsigned long long>(env.timeout_ms) * 1000000ull, w.split_part,
                                      w.split_count, w.kv_maps));
      else
        PF_CUDA(qmk_tc::launch_kernel(decode_attention_ring, dim3(B, NKV, attn_splits), dim3((DAR_WARPS + 1) * 32), DAR_SMEM_BYTES, s,
                                      w.q, w.k, w.v, reinterpret_cast<const __half *>(r[4]), reinterpret_cast<const __half *>(r[5]),
                                      rope, cosv, sinv, w.k_ptrs, w.v_ptrs, layer_off, w.positions, w.attn, max_seq_len, attn_scale,
                                      w.status, static_cast<unsigned long long>(env.timeout_ms) * 1000000ull, w.split_part,
                                      w.split_count));
      {
        const qmk_tc::PrefetchScope ahead(ahead_of(l, {4, 5, 6}));
        if ((r2 = qmk_tc::launch_gemm_splitk(w.map_attn_b, wm(3), w.o, M, H, QS, O_SPLITS, w.status, env.timeout_ms, s, &err,
                                             TILE_N, live, a_box, wq, wp(3))) != QMK_OK)
          return r2;
      }
      PF_CUDA(qmk_tc::launch_kernel(add_rmsnorm_rows<false>, dim3(B), dim3(256), 0, s, w.x, w.o, O_SPLITS, PART,
                                    reinterpret_cast<const __half *>(r[7]), w.xn, nullptr));
      if ((r2 = qmk_tc::launch_gemm_swiglu(w.map_xn_b, wm(4), wm(5), w.act, M, I, H, w.status, env.timeout_ms, s, &err, TILE_N,
                                           live, a_box, wq, wp(4), wp(5))) != QMK_OK)
        return r2;
      const qmk_tc::PrefetchScope ahead(ahead_of(l + 1, {0, 1, 2}));
      if ((r2 = qmk_tc::launch_gemm_splitk(w.map_act_b, wm(6), w.down, M, H, I, DOWN_SPLITS, w.status, env.timeout_ms, s, &err,
                                           TILE_N, live, a_box, wq, wp(6))) != QMK_OK)
        return r2;
    }
    PF_CUDA(qmk_tc::launch_kernel(add_rmsnorm_rows<false>, dim3(B), dim3(256), 0, s, w.x, w.down, DOWN_SPLITS, PART,
                                  static_cast<const __half *>(final_norm_weight), w.xn, nullptr));
    // Without a logits dump the LM head's epilogue picks the largest logit of each 128-column tile itself and the
    // rows of logits (B x 608 KB per step) are never written
    const bool fused_pick = env.logits_out == nullptr;
    if (fused_pick) qmk_tc::set_argmax_target(w.amax_val, w.amax_idx);
    qmk_tc::RingBudgetScope lm_scope(PREFILL_RING_BYTES);   // 1187 tiles: two CTAs per SM, four waves instead of eight
    r2 = qmk_tc::launch_gemm(w.map_xn_b, w.map_lm, w.logits, M, env.vocab, H, 128, w.status, env.timeout_ms, s, &err, live, a_box,
                             wq, lm_head_weight);
    qmk_tc::set_argmax_target(nullptr, nullptr);
    if (r2 != QMK_OK) return r2;
    if (fused_pick)
      PF_CUDA(qmk_tc::launch_kernel(argmax_pairs, dim3(B), dim3(256), 0, s, w.amax_val, w.amax_idx, env.vocab / 128, w.tokens,
                                    w.log_ptrs, w.start_positions, w.positions));
    else
      PF_CUDA(qmk_tc::launch_kernel(argmax_rows, dim3(B), dim3(1024), 0, s, w.logits, env.vocab, w.tokens, w.log_ptrs,
                                    w.start_positions, w.positions));
    return QMK_OK;
  };

  if (env.logits_out) {
    // debug dump [sequence][step][vocab]: plain launches with a copy after every step
    for (int step = 0; step < num_steps && rc == QMK_OK; ++step) {
      rc = enqueue_step(stream);
      if (rc != QMK_OK) break;
      PF_CUDA(cudaGetLastError());
      for (int b = 0; b < B; ++b)
        PF_CUDA(cudaMemcpyAsync(env.logits_out + (static_cast<size_t>(b) * num_steps + step) * env.vocab,
                                w.logits + static_cast<size_t>(b) * env.vocab, sizeof(float) * env.vocab,
                                cudaMemcpyDeviceToDevice, stream));
    }
  } else {
    // One step costs about 400 launches: capture it once as a CUDA graph (kept while nothing it bakes in
    // changes) and replay it num_steps times.
    const unsigned long long key[12] = {
        w.graph_epoch, static_cast<unsigned long long>(B) | (static_cast<unsigned long long>(wq) << 32), static_cast<unsigned long long>(num_layers),
        static_cast<unsigned long long>(max_seq_len), static_cast<unsigned long long>(env.vocab),
        static_cast<unsigned long long>(__float_as_uint_host(attn_scale)), reinterpret_cast<unsigned long long>(embed_weight),
        reinterpret_cast<unsigned long long>(final_norm_weight), reinterpret_cast<unsigned long long>(lm_head_weight),
        reinterpret_cast<unsigned long long>(rope), reinterpret_cast<unsigned long long>(cos_table),
        reinterpret_cast<unsigned long long>(sin_table) ^ (static_cast<unsigned long long>(env.timeout_ms) << 48) ^
            (static_cast<unsigned long long>(env.pdl != 0) << 63) ^ (static_cast<unsigned long long>(env.attn_mma != 0) << 62)};
    if (memcmp(key, w.step_key[B], sizeof(key)) != 0) {
      if (w.step_graph[B]) { cudaGraphExecDestroy(w.step_graph[B]); w.step_graph[B] = nullptr; }
      w.step_key[B][0] = 0;
      cudaGraph_t graph = nullptr;
      PF_CUDA(cudaStreamBeginCapture(w.gstream, cudaStreamCaptureModeThreadLocal));
      rc = enqueue_step(w.gstream);
      cudaError_t ce = cudaStreamEndCapture(w.gstream, &graph);   // always end the capture, also after an error
      if (rc == QMK_OK && ce != cudaSuccess) { rc = QMK_ERR_CUDA; err = std::string("graph capture: ") + cudaGetErrorString(ce); }
      if (rc == QMK_OK) {
        ce = cudaGraphInstantiate(&w.step_graph[B], graph, 0);
        if (ce != cudaSuccess) { rc = QMK_ERR_CUDA; err = std::string("cudaGraphInstantiate: ") + cudaGetErrorString(ce); }
      }
      if (graph) cudaGraphDestroy(graph);
      if (rc == QMK_OK) memcpy(w.step_key[B], key, sizeof(key));
    }
    if (rc == QMK_OK) {
      PF_CUDA(cudaEventRecord(w.ev_in, stream));          // the graph stream starts after the caller's stream
      PF_CUDA(cudaStreamWaitEvent(w.gstream, w.ev_in, 0));
      for (int step = 0; step < num_steps; ++step) PF_CUDA(cudaGraphLaunch(w.step_graph[B], w.gstream));
      PF_CUDA(cudaEventRecord(w.ev_out, w.gstream));
      PF_CUDA(cudaStreamWaitEvent(stream, w.ev_out, 0));  // ... and the caller's stream continues after it
    }
  }
  if (rc != QMK_OK) return qmk_internal::report(rc, err);
  unsigned int host_status[4] = {0, 0, 0, 0};
  PF_CUDA(cudaMemcpyAsync(host_status, w.status, 16, cudaMemcpyDeviceToHost, stream));
  PF_CUDA(cudaStreamSynchronize(stream));
  if (host_status[0] != 0)
    return qmk_internal::report(static_cast<int>(host_status[0]),
                                host_status[0] == QMK_ERR_BAD_TOKEN ? "decode_batched: a pick outside [0, vocab) (logits without a largest value)"
                                                                    : "decode_batched: a bounded device wait ran out");
  return QMK_OK;
}

// Bounded-wait self test of the GEMM kernel: one 128 x 128 tile whose loads are never issued.  The MMA thread's
// wait on the first stage runs out after budget_us, every role leaves its loop, TMEM is freed and the kernel
// returns status 4 with the context intact.
extern "C" int qmk_selftest_gemm_wait_timeout(int budget_us) {
  qmk_internal::begin_call();
  std::string err;
  if (budget_us < 1 || budget_us > 1000000) return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "budget_us must be in [1, 1e6]");
  int rc = qmk_tc::ensure_gemm_attrs(&err);
  if (rc != QMK_OK) return qmk_internal::report(rc, err);
  __half *ab = nullptr;
  float *c = nullptr;
  unsigned int *status = nullptr;
  PF_CUDA(cudaMalloc(&ab, sizeof(__half) * 128 * 64));
  PF_CUDA(cudaMalloc(&c, sizeof(float) * 128 * 128));
  PF_CUDA(cudaMalloc(&status, 16));
  PF_CUDA(cudaMemset(ab, 0, sizeof(__half) * 128 * 64));
  PF_CUDA(cudaMemset(status, 0, 16));
  CUtensorMap m;
  rc = qmk_tc::make_map_f16(&m, ab, 128, 64, 128, &err);
  if (rc == QMK_OK) {
    qmk_gemm::Groups gr;
    gr.C[0] = c; gr.C[1] = nullptr; gr.C[2] = nullptr;
    gr.N[0] = 128; gr.N[1] = 0; gr.N[2] = 0;
    gr.kblocks_per_split = 0;
    gr.split_stride = 0;
    gr.a_box_bytes = 0;
    for (int g = 0; g < qmk_gemm::MAX_GROUPS; ++g) gr.braw[g] = nullptr;
    gr.raw_pitch = gr.raw_bs_off = gr.raw_scale_off = 0;
    gr.amax_val = nullptr;
    gr.out_f16 = 0;
    gr.amax_idx = nullptr;
    const size_t smem = qmk_tc::selftest_ring(&gr);
    qmk_gemm::gemm_f16_tn_kernel<128><<<dim3(1, 1), qmk_gemm::THREADS, smem>>>(
        m, m, m, m, gr, 128, 64, status, static_cast<unsigned long long>(budget_us) * 1000ull, 1);
    unsigned int host[4] = {0, 0, 0, 0};
    cudaError_t e = cudaMemcpy(host, status, 16, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) { rc = QMK_ERR_CUDA; err = std::string("gemm self test: ") + cudaGetErrorString(e); }
    else rc = static_cast<int>(host[0]);
  }
  cudaFree(ab);
  cudaFree(c);
  cudaFree(status);
  if (rc != QMK_OK && rc != QMK_ERR_WAIT_TIMEOUT) return qmk_internal::report(rc, err);
  return rc;
}

// The same of the attention kernel: a query tile at position 512 whose score products stop behind the first, with keys and values
// in flight.
extern "C" int qmk_selftest_attention_wait_timeout(int budget_us) {
  qmk_internal::begin_call();
  using qmk_pf::QS;
  using qmk_pf::NKV;
  std::string err;
  if (budget_us < 1 || budget_us > 1000000) return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "budget_us must be in [1, 1e6]");
  int rc = QMK_OK;
  constexpr int T = qmk_attn::TQ, POS = 512, ROWS = POS + T;
  constexpr size_t q_bytes = sizeof(__half) * T * QS, kv_bytes = sizeof(__half) * NKV * ROWS * 128;
  unsigned char *buf = nullptr;            // queries, keys, values, outputs, status
  PF_CUDA(cudaMalloc(&buf, 2 * q_bytes + 2 * kv_bytes + 16));
  cudaError_t e = cudaMemset(buf, 0, 2 * q_bytes + 2 * kv_bytes + 16);
  unsigned char *const k = buf + q_bytes, *const v = k + kv_bytes, *const out = v + kv_bytes, *const status = out + q_bytes;
  CUtensorMap mq, mk, mv;
  rc = qmk_tc::make_map_f16(&mq, buf, T, QS, qmk_gemm::BM, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_kv(&mk, k, ROWS, ROWS, NKV, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_kv(&mv, v, ROWS, ROWS, NKV, &err);
  if (rc == QMK_OK && e == cudaSuccess) {
    e = cudaFuncSetAttribute(qmk_attn::causal_attention_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(qmk_attn::SMEM_BYTES));
    qmk_attn::causal_attention_tc<true><<<dim3(qmk_pf::NQ), qmk_attn::THREADS, qmk_attn::SMEM_BYTES>>>(
        mq, mk, mv, 0, reinterpret_cast<__half *>(out), T, POS, 1.0f, reinterpret_cast<unsigned int *>(status),
        static_cast<unsigned long long>(budget_us) * 1000ull, nullptr, nullptr);
    unsigned int host[4] = {0, 0, 0, 0};
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(host, status, 16, cudaMemcpyDeviceToHost);
    rc = static_cast<int>(host[0]);
  }
  if (e != cudaSuccess) { rc = QMK_ERR_CUDA; err = std::string("attention self test: ") + cudaGetErrorString(e); }
  cudaFree(buf);
  if (rc != QMK_OK && rc != QMK_ERR_WAIT_TIMEOUT) return qmk_internal::report(rc, err);
  return rc;
}

// The same of a decode step's attention: one CTA, one sequence at position 900, the chains of each kv head in two pieces (16 pieces, more
// than the producer may be ahead).  what = 1: nothing is loaded, so that consumers wait for chunks, then for pieces, and the
// producer for finished ones; 2: one chunk's copies are missing among a ring of others in flight.
extern "C" int qmk_selftest_decode_attention_wait_timeout(int budget_us, int what) {
  qmk_internal::begin_call();
  using namespace qmk_pf;
  std::string err;
  if (budget_us < 1 || budget_us > 1000000 || what < DAM_NO_LOADS || what > DAM_LOST_COPY)
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "budget_us must be in [1, 1e6], what in [1, 2]");
  constexpr int ROWS = 1024, POS = 900, CHUNKS = (POS + DAM_ROWS - 1) / DAM_ROWS, PARTS = 2, PIECES = NKV * PARTS;
  constexpr size_t kv_bytes = sizeof(__half) * NKV * ROWS * D, plan_bytes = sizeof(DamPlan) + sizeof(DamPiece) * PIECES;
  constexpr size_t at_v = kv_bytes, at_q = 2 * kv_bytes, at_new = at_q + sizeof(float) * QS, at_norm = at_new + 2 * sizeof(float) * KVS,
                   at_rope = at_norm + sizeof(__half) * D, at_out = at_rope + sizeof(float) * ROWS * D, at_maps = at_out + sizeof(__half) * QS,
                   at_plan = at_maps + 2 * sizeof(CUtensorMap), at_part = at_plan + (plan_bytes + 127) / 128 * 128,
                   at_count = at_part + sizeof(float) * NKV * DAM_CHAINS * DAM_PART, at_ptrs = at_count + sizeof(unsigned int) * NKV,
                   at_status = at_ptrs + 2 * sizeof(void *), total = at_status + 16;
  static_assert(at_maps % 128 == 0 && at_plan % 128 == 0 && at_ptrs % 8 == 0, "alignment of the self test's buffers");
  unsigned char *buf = nullptr;
  PF_CUDA(cudaMalloc(&buf, total));
  cudaError_t e = cudaMemset(buf, 0, total);
  CUtensorMap maps[2];
  int rc = qmk_tc::make_map_f16(&maps[0], buf, NKV * ROWS, D, DAM_ROWS, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&maps[1], buf + at_v, NKV * ROWS, D, DAM_ROWS, &err);
  std::vector<unsigned char> plan_bytes_host(plan_bytes, 0);
  DamPlan *const plan = reinterpret_cast<DamPlan *>(plan_bytes_host.data());
  plan->total = PIECES;
  for (int i = 0; i < PIECES; ++i) plan->pieces[i] = {0, POS, 0, CHUNKS, i / PARTS, 0, i % PARTS, 1 | (PARTS << 8)};
  const void *const ptrs[2] = {buf, buf + at_v};
  if (rc == QMK_OK && e == cudaSuccess) {
    e = cudaMemcpy(buf + at_maps, maps, sizeof(maps), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(buf + at_plan, plan, plan_bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(buf + at_ptrs, ptrs, sizeof(ptrs), cudaMemcpyHostToDevice);
    auto *const kernel = what == DAM_NO_LOADS ? decode_attention_mma<DAM_NO_LOADS> : decode_attention_mma<DAM_LOST_COPY>;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DAM_SMEM_BYTES);
    unsigned int host[4] = {0, 0, 0, 0};
    if (e == cudaSuccess) {
      const __half *const norm = reinterpret_cast<const __half *>(buf + at_norm);
      const float *const q = reinterpret_cast<const float *>(buf + at_q), *const fresh = reinterpret_cast<const float *>(buf + at_new);
      __half *const *const caches = reinterpret_cast<__half *const *>(buf + at_ptrs);
      kernel<<<dim3(1), (DAM_WARPS + 1) * 32, DAM_SMEM_BYTES>>>(
          q, fresh, fresh + KVS, norm, norm, reinterpret_cast<const float *>(buf + at_rope), nullptr, nullptr, caches, caches + 1, 0,
          reinterpret_cast<DamPlan *>(buf + at_plan), 0, reinterpret_cast<__half *>(buf + at_out), ROWS, 1.0f,
          reinterpret_cast<unsigned int *>(buf + at_status), static_cast<unsigned long long>(budget_us) * 1000ull,
          reinterpret_cast<float *>(buf + at_part), reinterpret_cast<unsigned int *>(buf + at_count), reinterpret_cast<const CUtensorMap *>(buf + at_maps));
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaMemcpy(host, buf + at_status, 16, cudaMemcpyDeviceToHost);
      rc = static_cast<int>(host[0]);
    }
  }
  if (e != cudaSuccess) { rc = QMK_ERR_CUDA; err = std::string("attention self test: ") + cudaGetErrorString(e); }
  cudaFree(buf);
  if (rc != QMK_OK && rc != QMK_ERR_WAIT_TIMEOUT) return qmk_internal::report(rc, err);
  return rc;
}

// The same of the pair kernel: one pair, two 256 x 256 tiles of eight K blocks.  Beside loads that are never issued: the second CTA's
// alone (the first has a ring of copies in flight whose barriers cannot complete), and an issuer that gives up behind the first
// tile (MMAs and a ring of copies in flight).  All end in status 4 with the pair's copies and MMAs drained.
extern "C" int qmk_selftest_gemm_pair_wait_timeout(int budget_us, int what) {
  qmk_internal::begin_call();
  std::string err;
  if (budget_us < 1 || budget_us > 1000000 || what < qmk_pair::NO_LOADS || what > qmk_pair::SECOND_CTA_NO_LOADS)
    return qmk_internal::report(QMK_ERR_BAD_ARGUMENT, "budget_us must be in [1, 1e6], what in [1, 3]");
  int rc = qmk_tc::ensure_gemm_attrs(&err);
  if (rc != QMK_OK) return qmk_internal::report(rc, err);
  constexpr int M = 2 * qmk_pair::TM, N = qmk_pair::TN, K = 8 * qmk_pair::BK;
  unsigned char *buf = nullptr;            // A, B, C, status
  constexpr size_t at_b = sizeof(__half) * M * K, at_c = at_b + sizeof(__half) * N * K, at_status = at_c + sizeof(float) * M * N;
  PF_CUDA(cudaMalloc(&buf, at_status + 16));
  cudaError_t e = cudaMemset(buf, 0, at_status + 16);
  CUtensorMap ma, mb, mc;
  rc = qmk_tc::make_map_f16(&ma, buf, M, K, 128, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&mb, buf + at_b, N, K, 128, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_c(&mc, buf + at_c, M, N, false, &err);
  if (rc == QMK_OK && e == cudaSuccess) {
    qmk_pair::Args a;
    a.heads = qmk_pair::Heads{};
    for (int g = 0; g < 3; ++g) { a.N[g] = g == 0 ? N : 0; a.row_scale[g] = nullptr; }
    a.m_tiles = 2; a.n_tiles = 1; a.splits = 1;
    a.kblocks = K / qmk_pair::BK;
    auto *const kernel = what == qmk_pair::NO_LOADS       ? qmk_pair::gemm_pair_kernel<0, false, qmk_pair::NO_LOADS>
                         : what == qmk_pair::ISSUER_STOPS ? qmk_pair::gemm_pair_kernel<0, false, qmk_pair::ISSUER_STOPS>
                                                          : qmk_pair::gemm_pair_kernel<0, false, qmk_pair::SECOND_CTA_NO_LOADS>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(qmk_pair::SMEM_BYTES));
    kernel<<<dim3(2), qmk_pair::THREADS, qmk_pair::SMEM_BYTES>>>(
        ma, mb, mb, mb, mc, mc, mc, a, reinterpret_cast<unsigned int *>(buf + at_status), static_cast<unsigned long long>(budget_us) * 1000ull);
    unsigned int host[4] = {0, 0, 0, 0};
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(host, buf + at_status, 16, cudaMemcpyDeviceToHost);
    rc = static_cast<int>(host[0]);
  }
  if (e != cudaSuccess) { rc = QMK_ERR_CUDA; err = std::string("gemm self test: ") + cudaGetErrorString(e); }
  cudaFree(buf);
  if (rc != QMK_OK && rc != QMK_ERR_WAIT_TIMEOUT) return qmk_internal::report(rc, err);
  return rc;
}

extern "C" int qmk_gemm_f16_tn(const void *a, const void *b, float *c, int m, int n, int k, cudaStream_t stream) {
  qmk_internal::begin_call();
  std::string err;
  CUtensorMap ma, mb;
  unsigned int *status = nullptr;
  int rc = qmk_tc::make_map_f16(&ma, a, m, k, qmk_gemm::BM, &err);
  const bool by_pairs = m > PAIR_MIN_ROWS && n > 0 && n % qmk_pair::TN == 0;
  const int box_n = (!by_pairs && m > 0 && n > 0 && m % 128 == 0 && n % 128 == 0) ? qmk_tc::gemm_box_n(m, n) : 128;
  if (rc == QMK_OK) rc = qmk_tc::make_map_f16(&mb, b, n, k, box_n, &err);
  if (rc == QMK_OK && cudaMalloc(&status, 16) != cudaSuccess) { rc = QMK_ERR_CUDA; err = "cudaMalloc failed"; }
  if (rc == QMK_OK) {
    cudaMemsetAsync(status, 0, 16, stream);
    if (by_pairs) {
      CUtensorMap mc;
      const CUtensorMap *const maps_b[1] = {&mb}, *const maps_c[1] = {&mc};
      rc = qmk_tc::make_map_c(&mc, c, m, n, false, &err);
      if (rc == QMK_OK) rc = qmk_tc::launch_gemm_pair(0, ma, 1, maps_b, maps_c, &n, m, k, 1, status, 2000, stream, &err);
    } else {
      rc = qmk_tc::launch_gemm(ma, mb, c, m, n, k, box_n, status, 2000, stream, &err);
    }
  }
  if (rc == QMK_OK) {
    unsigned int host[4] = {0, 0, 0, 0};
    cudaError_t e = cudaMemcpyAsync(host, status, 16, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) { rc = QMK_ERR_CUDA; err = std::string("gemm: ") + cudaGetErrorString(e); }
    else if (host[0] != 0) { rc = static_cast<int>(host[0]); err = "gemm: a bounded device wait ran out"; }
  }
  if (status) cudaFree(status);
  if (rc != QMK_OK) {
    qmk_internal::note_error(err);
    fprintf(stderr, "[qwen_megakernel] error %d: %s\n", rc, err.c_str());
  }
  return rc;
}

// The same GEMM with B in a packed weight format (1: FP8-E4M3 rows, 2: NVFP4 rows).  `mode` 0: C fp32 [m x n];
// mode 1: split-K in four parts, C holds the four partial matrices; mode 2: `b` is a gate matrix and `b2` an up
// matrix, C receives fp16 silu(A gate^T) * (A up^T) - the three forms the decode step uses.
extern "C" int qmk_gemm_packed_tn(const void *a, const void *b, const void *b2, void *c, int m, int n, int k, int weight_format,
                                  int mode, int box_n, cudaStream_t stream) {
  qmk_internal::begin_call();
  std::string err;
  CUtensorMap ma, mb, mb2;
  unsigned int *status = nullptr;
  if (weight_format < 1 || weight_format > 2 || mode < 0 || mode > 2 || m <= 0 || n <= 0 || m % 128 || n % 128 ||
      (mode == 2 && !b2) || !a || !b || !c) {
    qmk_internal::note_error("qmk_gemm_packed_tn: bad argument");
    fprintf(stderr, "[qwen_megakernel] error %d: qmk_gemm_packed_tn: bad argument\n", QMK_ERR_BAD_ARGUMENT);
    return QMK_ERR_BAD_ARGUMENT;
  }
  if (box_n <= 0) box_n = mode == 2 ? qmk_tc::gemm_box_n_fused(m, n) : mode == 1 ? 32 : qmk_tc::gemm_box_n(m, n);
  int rc = qmk_tc::make_map_f16(&ma, a, m, k, qmk_gemm::BM, &err);
  if (rc == QMK_OK) rc = qmk_tc::make_map_packed(&mb, b, n, k, box_n, weight_format, &err);
  if (rc == QMK_OK && mode == 2) rc = qmk_tc::make_map_packed(&mb2, b2, n, k, box_n, weight_format, &err);
  if (rc == QMK_OK && cudaMalloc(&status, 16) != cudaSuccess) { rc = QMK_ERR_CUDA; err = "cudaMalloc failed"; }
  if (rc == QMK_OK) {
    cudaMemsetAsync(status, 0, 16, stream);
    if (mode == 0)
      rc = qmk_tc::launch_gemm(ma, mb, static_cast<float *>(c), m, n, k, box_n, status, 2000, stream, &err, 0, 0, weight_format, b);
    else if (mode == 1)
      rc = qmk_tc::launch_gemm_splitk(ma, mb, static_cast<float *>(c), m, n, k, 4, status, 2000, stream, &err, box_n, 0, 0,
                                      weight_format, b);
    else
      rc = qmk_tc::launch_gemm_swiglu(ma, mb, mb2, static_cast<__half *>(c), m, n, k, status, 2000, stream, &err, box_n, 0, 0,
                                      weight_format, b, b2);
  }
  if (rc == QMK_OK) {
    unsigned int host[4] = {0, 0, 0, 0};
    cudaError_t e = cudaMemcpyAsync(host, status, 16, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) { rc = QMK_ERR_CUDA; err = std::string("gemm: ") + cudaGetErrorString(e); }
    else if (host[0] != 0) { rc = static_cast<int>(host[0]); err = "gemm: a bounded device wait ran out"; }
  }
  if (status) cudaFree(status);
  if (rc != QMK_OK) {
    qmk_internal::note_error(err);
    fprintf(stderr, "[qwen_megakernel] error %d: %s\n", rc, err.c_str());
  }
  return rc;
}
