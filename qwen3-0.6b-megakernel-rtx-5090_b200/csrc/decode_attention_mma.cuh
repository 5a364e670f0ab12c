// Batched decode attention on mma.sync (see the comment at the kernel).
#ifndef QMK_DECODE_ATTENTION_MMA_CUH_
#define QMK_DECODE_ATTENTION_MMA_CUH_

#include <cuda.h>
#include "prefill_kernels.cuh"

namespace qmk_pf {

// Decode-step attention for a batch of sequences on the tensor cores, with the per-head preparation fused in.
// Block = 288 = 8 consumer warps + 1 producer warp, two CTAs per SM, and the grid is what the device holds at once,
// whatever the batch (nine ring slots each: with eleven the CTAs nearest to memory finish so much earlier that the others
// set the time, with six the stream is short of copies in flight).  The work is a list of pieces, longest first (plan_pieces
// below); a CTA takes piece blockIdx.x, then whatever is next on the list.  A step's attention is bound by reading the cache (64
// sequences of 128 to 2048 tokens: 285 MB a layer, 43 us at the copy rate); with the same number of CTAs for every (sequence,
// kv head) item and nothing behind them, the longest sequences set the time.
//
// How an item is summed up does not depend on who does it: its chunks fall into `splits` equal ranges (as many as give every
// item's ranges a CTA; one for 19 sequences and more), a range into eight chains of every eighth chunk, each an online softmax of its
// own.  The chains are merged in order, then the ranges.  A piece is a whole range, or half or a quarter of the chains of a
// long one.
//
// The producer runs ahead across pieces: rows written by earlier steps do not depend on the kernel before, so its first
// ring fill overlaps that kernel's tail, and the next piece streams in while this one is merged.  Per piece the
// consumers prepare the heads (QK-norm, RoPE; one piece of an item writes the new cache row, whose score its last range takes),
// go over the chunks, a chain a warp, and merge.  An item of several pieces is finished by whichever CTA arrives last (a counter
// per item, nobody waits).
//
// Decode steps, a CTA per item and range -> pieces (with the GEMMs' 64-row tiles and prefetch): 64 NVFP4 sequences of 128 to 2048
// tokens 2710 -> 2120 us, 16 fp16 ones of 64 to 1024 1026 -> 932, 32 of 64 to 2048 1771 -> 1400; 16 and 32 of 1024, which were even
// before, 1053 -> 1042 and 1285 -> 1288, 30 of 300 to 320 887 -> 877.
//
// A chunk is four tiled TMA boxes of 16 rows x 128 bytes with the 128-byte swizzle, through per-sequence tensor maps kept
// in device memory, and a warp handles it with 16 mma.sync.m16n8k16: scores = K[16 x 128] . q[128 x 4] (columns: head 0
// hi / lo, head 1 hi / lo of the fp32 query split into two fp16 numbers), online softmax on the accumulator fragments
// (log2 domain), then out[128 x 4] += V^T[128 x 16] . p[16 x 4] with V read through ldmatrix.trans and p split like q -
// about 75 instructions per 16 rows.
//
// Waits are bounded.  On a time-out the CTA sets *status = 4, which the call returns: what it has written is then not valid.  It goes
// on through the pieces at hand without waiting and leaves at the first one it is not handed; pieces that it had taken from the list stay
// undone and their items' counters behind (the next call clears them).  A slot whose copy was given up is not loaded again, and the
// CTA stays until its copies have landed (whoever gives up waits for them, and the producer if it is still there).
constexpr int DAM_WARPS = 8, DAM_SLOTS = 9, DAM_ROWS = 16;
constexpr int DAM_BOX = DAM_ROWS * 128;                // one box: 16 rows x 64 dims
constexpr int DAM_SLOT_BYTES = 4 * DAM_BOX;            // 8 KB: K dims 0..63, K dims 64..127, V dims 0..63, V dims 64..127
constexpr int DAM_SMEM_BYTES = DAM_SLOTS * DAM_SLOT_BYTES + 2 * DAM_SLOTS * 8 + 16;   // ring, barriers, abort flag + issued counter
constexpr int DAM_QPITCH = 2 * D + 16;                 // bytes between the four query-operand rows (conflict-free ldmatrix)
constexpr int DAM_AHEAD = 4;                            // pieces the producer may be ahead of the consumers
constexpr float DAM_LO_SCALE = 2048.0f, DAM_LO_INV = 1.0f / 2048.0f;

__device__ __forceinline__ void dam_ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void dam_ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// fp32 -> fp16 operand half: the value rounded to fp16 (lo = false) or its scaled remainder (lo = true)
__device__ __forceinline__ __half dam_split(float x, bool lo) {
  const __half h = __float2half_rn(x);
  return lo ? __float2half_rn((x - __half2float(h)) * DAM_LO_SCALE) : h;
}
__device__ __forceinline__ uint32_t dam_pack(__half a, __half b) {
  return static_cast<uint32_t>(__half_as_ushort(a)) | (static_cast<uint32_t>(__half_as_ushort(b)) << 16);
}

// One piece: of the 16-row chunks [first, first + chunks) of sequence b's old rows, kv head g - range `split` of `splits` -
// the chains [8 part / parts, 8 (part + 1) / parts).
struct __align__(16) DamPiece {
  int b, pos, first, chunks;         // chunks < 0: no piece
  int g_single, split, part, splits_parts;   // g, + 256 where no CTA has more than one piece; splits, + 256 x parts
};
constexpr int DAM_CHAINS = DAM_WARPS;
constexpr int DAM_PART = 2 * (D + 2);                  // floats per partial state: two heads of A[128], M, L
constexpr int DAM_MAX_BATCH = 128, DAM_MAX_LAYERS = 48, DAM_MAX_SPLITS = 8;
__host__ __device__ inline int dam_splits(int batch, int grid) {
  const int s = grid / (batch * NKV);
  return s < 1 ? 1 : s > DAM_MAX_SPLITS ? DAM_MAX_SPLITS : s;
}
constexpr int dam_max_pieces(int batch, int grid) { return 4 * (NKV * batch + grid); }
// partial states: [item][split][chain]
constexpr size_t dam_max_states(int batch, int grid) { return static_cast<size_t>(NKV * batch > grid ? NKV * batch : grid) * DAM_CHAINS; }
struct DamPlan {
  int total;                               // pieces
  unsigned int next[DAM_MAX_LAYERS];       // pieces taken beyond the first of every CTA, per layer
  int pad[3];
  DamPiece pieces[1];                      // [dam_max_pieces]
};

// Once per step (every layer has the same rows): the pieces of all sequences, longest first.  One block of 256 threads.
//
// Ranges of more than 7/4 fair shares of all chunks (19 sequences and more, one range an item) are cut in two or four: the
// short ones even out by themselves behind them, and a CTA left with few others streams more than twice as fast as one of 296.  28
// NVFP4 sequences of 381 to 909 tokens, cut from 5/4 / 7/4 / 9/4 shares on: 1444 / 1233 / 1239 us a step, uncut 1335; 23 fp16 ones of 385
// to 1797: 1540 / 1250 / 1335, uncut 1580.  Fewer sequences have several ranges to an item already, whose merge the cuts lengthen:
// three shares (6 sequences of 128 to 2048 tokens, 7/4 / 9/4: 988 / 881; 12 of 100 to 800: 930 / 877).
constexpr int DAM_CUT_ONE = 7, DAM_CUT_SEVERAL = 12, DAM_WHOLE = 16;
__device__ inline void plan_pieces(const int *positions, int batch, int grid, DamPlan *plan) {
  __shared__ int s_n[DAM_MAX_BATCH], s_k[DAM_MAX_BATCH], s_at[DAM_MAX_BATCH];
  __shared__ __align__(16) int s_len[DAM_MAX_BATCH];
  __shared__ int s_by_rank[DAM_MAX_BATCH], s_total;
  const int tid = threadIdx.x, lane = tid & 31, splits = dam_splits(batch, grid);
  if (tid < DAM_MAX_LAYERS) plan->next[tid] = 0u;
  if (tid < 32) {                          // (batch <= 128: four sequences per lane)
    int n[4], sum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      n[i] = 4 * lane + i < batch ? (positions[4 * lane + i] + DAM_ROWS - 1) / DAM_ROWS : -1;
      sum += max(n[i], 0);
    }
    sum = NKV * __reduce_add_sync(0xffffffffu, sum);
    const int len = max(DAM_WHOLE, (sum / 4 * (splits == 1 ? DAM_CUT_ONE : DAM_CUT_SEVERAL)) / grid);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int range = (n[i] + splits - 1) / splits, parts = n[i] < 0 ? 0 : range <= len ? 1 : range <= 2 * len ? 2 : 4;
      s_n[4 * lane + i] = n[i];
      s_k[4 * lane + i] = parts;
      s_len[4 * lane + i] = parts > 0 ? (range + parts - 1) / parts : -1;
    }
  }
  __syncthreads();
  {                                        // rank of every sequence by the length of its pieces: two threads each
    const int b = tid >> 1, half = tid & 1, mine = s_len[b];
    int rank = 0;
#pragma unroll
    for (int i = 0; i < DAM_MAX_BATCH / 8; ++i) {
      const int j = half * (DAM_MAX_BATCH / 2) + 4 * i;
      const int4 v = *reinterpret_cast<const int4 *>(s_len + j);
      rank += (v.x > mine || (v.x == mine && j < b)) + (v.y > mine || (v.y == mine && j + 1 < b)) +
              (v.z > mine || (v.z == mine && j + 2 < b)) + (v.w > mine || (v.w == mine && j + 3 < b));
    }
    rank += __shfl_xor_sync(0xffffffffu, rank, 1);
    if (half == 0) s_by_rank[rank] = b;
  }
  __syncthreads();
  if (tid < 32) {                          // first piece of every sequence, in order of rank
    int k[4], sum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) { k[i] = NKV * splits * s_k[s_by_rank[4 * lane + i]]; sum += k[i]; }
    int at = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, at, o);
      if (lane >= o) at += up;
    }
    if (lane == 31) s_total = at;
    at -= sum;
#pragma unroll
    for (int i = 0; i < 4; ++i) { s_at[4 * lane + i] = at; at += k[i]; }
  }
  __syncthreads();
  const int total = s_total, single = total <= grid ? 256 : 0;
  if (tid == 0) plan->total = total;
  for (int i = total + tid; i < grid; i += blockDim.x) {    // CTAs without a piece
    reinterpret_cast<int4 *>(plan->pieces + i)[0] = make_int4(0, 0, 0, -1);
    reinterpret_cast<int4 *>(plan->pieces + i)[1] = make_int4(256, 0, 0, 257);
  }
  for (int i = tid; i < total; i += blockDim.x) {
    int lo = 0, hi = batch;                // (ranks batch .. 127 are the sequences that are not there)
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_at[mid] <= i) lo = mid; else hi = mid;
    }
    const int b = s_by_rank[lo], parts = s_k[b], n = s_n[b], j = i - s_at[lo];
    const int g = j / (splits * parts), sp = j / parts - g * splits, part = j % parts, first = n * sp / splits;
    reinterpret_cast<int4 *>(plan->pieces + i)[0] = make_int4(b, positions[b], first, n * (sp + 1) / splits - first);
    reinterpret_cast<int4 *>(plan->pieces + i)[1] = make_int4(g | single, sp, part, splits | (parts << 8));
  }
}
// Block b < batch: embedding row of sequence b's token (embed_row); the last block: the step's attention pieces.
// A row of logits without a largest value (all NaN, or all -inf) leaves 0x7fffffff as its pick.  As in the persistent kernels such a
// token is an error of the step that reads it (*status = 5, which the call returns), and no address is made of it.
__global__ void __launch_bounds__(256) embed_rows_and_plan(const int *tokens, const void *embed, int wq, int vocab, float *x, const int *positions,
                                                          int grid, DamPlan *plan, unsigned int *status) {
  pdl_wait();
  pdl_trigger();
  const int batch = static_cast<int>(gridDim.x) - 1;
  if (static_cast<int>(blockIdx.x) >= batch) { plan_pieces(positions, batch, grid, plan); return; }
  int token = tokens[blockIdx.x];
  if (token < 0 || token >= vocab) {
    if (threadIdx.x == 0) atomicCAS(status, 0u, 5u);
    token = 0;
  }
  embed_row(token, embed, wq, x, blockIdx.x);
}

// TEST (bounded waits only): 1: nothing is loaded or announced; 2: the third chunk's copies are not issued, those around it are.
enum { DAM_NO_LOADS = 1, DAM_LOST_COPY = 2 };
template <int TEST = 0>
__global__ void __launch_bounds__((DAM_WARPS + 1) * 32, 2) decode_attention_mma(
    const float *q, const float *k, const float *v, const __half *q_norm, const __half *k_norm, const float *rope,
    const __half *cos_table, const __half *sin_table, __half *const *k_ptrs, __half *const *v_ptrs, size_t layer_off,
    DamPlan *plan, int layer, __half *out, int max_seq_len, float scale, unsigned int *status, unsigned long long budget_ns,
    float *split_part, unsigned int *split_count, const CUtensorMap *kv_maps) {
  extern __shared__ __align__(128) unsigned char dam_smem[];
  __shared__ __align__(16) unsigned char s_qf[4 * DAM_QPITCH];   // fp16 query operand: q0 hi, q0 lo, q1 hi, q1 lo
  __shared__ float sknew[D], svnew[D], snew_score[2];
  __shared__ __align__(16) float s_raw[4][D], s_rope[4][D];         // the next piece's heads (q0, q1, k, v) and rotary row, as fetched
  __shared__ __half s_norm[3][D];                                   // their norm weights, each warp's own
  __shared__ float sm[DAM_WARPS][2], sl[DAM_WARPS][2];
  __shared__ __align__(16) float sacc[DAM_WARPS][2][D];
  __shared__ unsigned int s_last;
  __shared__ DamPiece s_piece[DAM_AHEAD];                           // pieces taken, in turn
  __shared__ volatile int s_taken, s_done;                          // pieces taken (the last one: none left, chunks = -1) and finished
  uint64_t *full = reinterpret_cast<uint64_t *>(dam_smem + DAM_SLOTS * DAM_SLOT_BYTES);
  uint64_t *empty = full + DAM_SLOTS;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(empty + DAM_SLOTS);
  // Chunks issued so far.  A parity wait can only tell two consecutive uses of a slot apart, and a warp's first chunk
  // in a slot may already be a second use (the tenth, in slot 0): consumers wait for "issued" first.
  volatile int *issued_ctr = abort_flag + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto s32 = [](const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); };
  auto try_wait = [&](uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(s32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
  };
  auto wait = [&](uint64_t *bar, uint32_t parity) {   // bounded
    if (try_wait(bar, parity)) return true;
    unsigned long long t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (uint32_t it = 1;; ++it) {
      if (try_wait(bar, parity)) return true;
      if ((it & 63u) == 0u) {
        if (*abort_flag) return false;
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > budget_ns) { *abort_flag = 1; atomicCAS(status, 0u, 4u); return false; }
      }
    }
  };
  if (threadIdx.x == 0) {
    for (int i = 0; i < DAM_SLOTS; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(full + i)), "r"(1) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(empty + i)), "r"(1) : "memory");
    }
    *abort_flag = 0;
    *issued_ctr = 0;
    // (The plan was written, like all old rows, before the kernel that this one may overlap had its inputs: see pdl_wait.)
    reinterpret_cast<int4 *>(&s_piece[0])[0] = __ldcg(reinterpret_cast<const int4 *>(plan->pieces + blockIdx.x));
    reinterpret_cast<int4 *>(&s_piece[0])[1] = __ldcg(reinterpret_cast<const int4 *>(plan->pieces + blockIdx.x) + 1);
    s_taken = 1;
    s_done = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // (weights: from DRAM; on its way while everything else is set up)
  __half norm_weights[4];                            // (q0, q1, k: warps 0, 1, 2; the vectors need not be aligned)
#pragma unroll
  for (int i = 0; i < 4; ++i) norm_weights[i] = warp < 3 ? (warp < 2 ? q_norm : k_norm)[lane + 32 * i] : __half(0.0f);
  __syncthreads();
  // a volatile counter of this CTA to pass `seen`, bounded
  auto wait_past = [&](volatile int *counter, int seen) {
    if (*counter > seen) return true;
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (uint32_t it = 1; *counter <= seen; ++it) {
      if ((it & 63u) == 0u) {
        if (*abort_flag) return false;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > budget_ns) { *abort_flag = 1; atomicCAS(status, 0u, 4u); return false; }
      }
    }
    return true;
  };
  // after a time-out: the copies of the `issued` chunks must land before the CTA may exit
  auto drain = [&](int issued) {
    for (int c = (issued > DAM_SLOTS ? issued - DAM_SLOTS : 0); c < issued; ++c) {
      unsigned long long t0, t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
      while (!try_wait(full + c % DAM_SLOTS, (c / DAM_SLOTS) & 1)) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > (budget_ns > 2000000ull ? budget_ns : 2000000ull)) break;
      }
    }
  };
  if (warp == DAM_WARPS) {            // ---- producer: takes pieces, streams their old rows in chunks of 16
    if (qmk_gemm::elect_one()) {      // (a thread picked by `lane == 0` takes 500 cycles to issue a chunk's copies: 8 sequences 653 -> 676 us a step)
      int issued = 0, slot = 0, mapped = -1;
      uint32_t parity = 1;                             // of the use before the one at hand
      const CUtensorMap *kmap = nullptr, *vmap = nullptr;
      int4 p0 = reinterpret_cast<const int4 *>(&s_piece[0])[0], p1 = reinterpret_cast<const int4 *>(&s_piece[0])[1];
      bool ok = true;
      for (int taken = 1; ok && p0.w >= 0; ++taken) {
        if (mapped != p0.x) {
          mapped = p0.x;
          kmap = kv_maps + 2 * mapped;
          vmap = kmap + 1;
          // the maps were written by the host into device memory before this launch
          asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(kmap)) : "memory");
          asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(vmap)) : "memory");
        }
        const int row0 = layer * NKV * max_seq_len + (p1.x & 255) * max_seq_len + p0.z * DAM_ROWS;   // in the sequence's [layer][head][pos] cache
        const int chains = DAM_CHAINS / (p1.w >> 8), chain0 = p1.z * chains;
        for (int c = 0; c < p0.w; ++c) {
          if (static_cast<unsigned int>((c & (DAM_CHAINS - 1)) - chain0) >= static_cast<unsigned int>(chains) || TEST == DAM_NO_LOADS) continue;
          const int row = row0 + c * DAM_ROWS;
          if (issued >= DAM_SLOTS && !wait(empty + slot, parity)) { ok = false; break; }
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(full + slot)), "r"(DAM_SLOT_BYTES) : "memory");
          const uint32_t dst = s32(dam_smem + slot * DAM_SLOT_BYTES);
#pragma unroll
          for (int sub = TEST == DAM_LOST_COPY && issued == 2 ? 4 : 0; sub < 4; ++sub)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                         ::"r"(dst + sub * DAM_BOX), "l"(sub < 2 ? kmap : vmap), "r"((sub & 1) * 64), "r"(row), "r"(s32(full + slot))
                         : "memory");
          ++issued;
          if (++slot == DAM_SLOTS) { slot = 0; parity ^= 1u; }
          __threadfence_block();
          *issued_ctr = issued;
        }
        // the next piece, taken when this one's last chunk is under way: a ring's worth of copies covers the round trip
        if (!ok || (p1.x & 256)) break;
        p0.w = -1;
        const int total = __ldcg(&plan->total), id = static_cast<int>(gridDim.x + atomicAdd(&plan->next[layer], 1u));
        if (id < total) {
          p0 = __ldcg(reinterpret_cast<const int4 *>(plan->pieces + id));
          p1 = __ldcg(reinterpret_cast<const int4 *>(plan->pieces + id) + 1);
        }
        if (taken >= DAM_AHEAD && !wait_past(&s_done, taken - DAM_AHEAD)) break;
        reinterpret_cast<int4 *>(&s_piece[taken % DAM_AHEAD])[0] = p0;
        reinterpret_cast<int4 *>(&s_piece[taken % DAM_AHEAD])[1] = p1;
        __threadfence_block();
        s_taken = taken + 1;
      }
      // (either this look finds the flag, or whoever sets it later finds the last chunk announced)
      __threadfence_block();
      if (*abort_flag) drain(issued);
    }
    return;
  }
  // ---- consumers: eight warps, whose barriers leave the producer out (it waits for slots that they free)
  auto sync_consumers = []() { asm volatile("bar.sync 1, %0;" ::"n"(DAM_WARPS * 32) : "memory"); };
  auto any_consumer = [](bool p) {
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(any) : "r"(p ? 1u : 0u), "n"(DAM_WARPS * 32) : "memory");
    return any != 0;
  };
  const float sc = scale * 1.4426950408889634f;
  const int quad = lane & 3, rowq = lane >> 2;     // accumulator fragment: rows rowq, rowq + 8; columns 2 quad, 2 quad + 1
  const int lr = (lane & 7) + ((lane >> 3) & 1) * 8;
  // Warps 0..3 prepare query heads 0 and 1, K and V, which they fetch to shared memory (no registers to spare) under the merge
  // of the piece before, where the next one is known by then.
  auto fetch16 = [&](const void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s32(dst)), "l"(src) : "memory");
  };
  auto fetch_heads = [&](const DamPiece &p) {
    const int g = p.g_single & 255;
    // (through L1: three warps and two CTAs an SM want the row, and every CTA of the device where all sequences are as long; past
    // it, the row's four lines answered the last CTA 5 us late)
    if (warp < 3 && rope)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(s32(&s_rope[warp][4 * lane])), "l"(rope + static_cast<size_t>(p.pos) * D + 4 * lane) : "memory");
    if (warp < 4)
      fetch16(&s_raw[warp][4 * lane], (warp < 2 ? q + static_cast<size_t>(p.b) * QS + (2 * g + warp) * D
                                                : (warp == 2 ? k : v) + static_cast<size_t>(p.b) * KVS + g * D) + 4 * lane);
  };
  // The producer streams cache rows written by EARLIER steps and started at once; the others read what the q/k/v GEMM
  // launched just before wrote, and write (cache row, output, split partials) only after it completed.
  pdl_wait();
  if (threadIdx.x == 0) pdl_trigger();   // (after the wait: at most two kernels of a chain overlap)
  const bool idle = s_piece[0].chunks < 0;           // (fewer pieces than CTAs)
  const bool single = (s_piece[0].g_single & 256) != 0;
  bool fetched = true;
  if (!idle) fetch_heads(s_piece[0]);
  if (warp < 3) {
#pragma unroll
    for (int i = 0; i < 4; ++i) s_norm[warp][lane + 32 * i] = norm_weights[i];
  }
  int ring = 0;                                      // ring chunks of the pieces before
  for (int j = 0;; ++j) {
    if (j > 0 && single) break;
    // (after a time-out some warps may see a piece here and some not: all go on, or none)
    if (j > 0 && any_consumer(!wait_past(&s_taken, j))) break;
    if (threadIdx.x == 0) s_done = j;      // behind that barrier nobody needs the piece before
    const DamPiece &piece = s_piece[j % DAM_AHEAD];
    const int nchunks = piece.chunks, pos = piece.pos, b = piece.b, g = piece.g_single & 255;
    if (nchunks < 0) break;
    const int splits = piece.splits_parts & 255, parts = piece.splits_parts >> 8, chains = DAM_CHAINS / parts;
    const bool last_split = piece.split == splits - 1;
    const bool owner = last_split && piece.part == parts - 1;      // writes the new cache row
    if (!fetched) fetch_heads(piece);
    float y[4] = {0.f, 0.f, 0.f, 0.f};
    if (warp < 4) {                   // ---- head preparation
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) y[i] = s_raw[warp][lane + 32 * i];
      if (warp < 3) {
        float ss = y[0] * y[0] + y[1] * y[1] + y[2] * y[2] + y[3] * y[3];
        ss = warp_sum(ss);
        const float rstd = 1.0f / sqrtf(ss * (1.0f / D) + RMS_EPS);
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = y[i] * rstd * __half2float(s_norm[warp][lane + 32 * i]);
        float c0, s0, c1, s1;
        if (rope) {
          c0 = s_rope[warp][lane]; c1 = s_rope[warp][lane + 32]; s0 = s_rope[warp][64 + lane]; s1 = s_rope[warp][96 + lane];
        } else {
          const __half *ct = cos_table + static_cast<size_t>(pos) * D, *st = sin_table + static_cast<size_t>(pos) * D;
          c0 = __half2float(ct[lane]); c1 = __half2float(ct[lane + 32]);
          s0 = __half2float(st[lane]); s1 = __half2float(st[lane + 32]);
        }
        const float r0 = y[0] * c0 - y[2] * s0, r2 = y[0] * s0 + y[2] * c0;
        const float r1 = y[1] * c1 - y[3] * s1, r3 = y[1] * s1 + y[3] * c1;
        y[0] = r0; y[1] = r1; y[2] = r2; y[3] = r3;
      }
      if (warp < 2) {
        __half *qh = reinterpret_cast<__half *>(s_qf + (2 * warp) * DAM_QPITCH);
        __half *ql = reinterpret_cast<__half *>(s_qf + (2 * warp + 1) * DAM_QPITCH);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          qh[lane + 32 * i] = dam_split(y[i], false);
          ql[lane + 32 * i] = dam_split(y[i], true);
        }
      } else {
        float *snew = warp == 2 ? sknew : svnew;
        __half *dst = (warp == 2 ? k_ptrs : v_ptrs)[b] + layer_off + (static_cast<size_t>(g) * max_seq_len + pos) * D;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __half hv = __float2half_rn(y[i]);
          if (owner) dst[lane + 32 * i] = hv;
          snew[lane + 32 * i] = __half2float(hv);
        }
      }
    }
    sync_consumers();
    if (warp < 2) {   // score of the new row for query head `warp`
      float d = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) d = fmaf(y[i], sknew[lane + 32 * i], d);
      d = warp_sum(d);
      if (lane == 0) snew_score[warp] = d * sc;
    }
    const int last_rows = pos - (piece.first + nchunks - 1) * DAM_ROWS;   // rows of the last chunk (or more)
    float acc[8][4];
#pragma unroll
    for (int t = 0; t < 8; ++t) { acc[t][0] = 0.f; acc[t][1] = 0.f; acc[t][2] = 0.f; acc[t][3] = 0.f; }
    float m = -INFINITY, l = 0.f;                    // running max / sum of this lane's head (quad = head, quads 2, 3 idle)
    uint32_t qf[4][4];                               // query operand fragments of the four 32-dim groups
    {
      const uint32_t q_addr = s32(s_qf + (lane & 3) * DAM_QPITCH) + (lane >> 3) * 16;   // rows 4..7 repeat 0..3
#pragma unroll
      for (int p = 0; p < 4; ++p) dam_ldsm_x4(q_addr + p * 64, qf[p]);
    }
    // warp w takes chain chain0 + w (where the piece has that many): the ring holds the piece's chunks in order
    const int chain0 = piece.part * chains;
    for (int c = warp < chains ? chain0 + warp : nchunks; c < nchunks; c += DAM_CHAINS) {
      const int rc = ring + (c >> 3) * chains + warp, slot = rc % DAM_SLOTS;
      bool mine = true;
      if (*issued_ctr <= rc) {           // bounded wait for the producer to reach this chunk
        unsigned long long t0, t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        for (uint32_t it = 1; *issued_ctr <= rc; ++it) {
          if ((it & 63u) == 0u) {
            if (*abort_flag) { mine = false; break; }
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t - t0 > budget_ns) { *abort_flag = 1; atomicCAS(status, 0u, 4u); mine = false; break; }
          }
        }
      }
      const bool ok = __all_sync(0xffffffffu, mine && wait(full + slot, (rc / DAM_SLOTS) & 1));
      const int nrow = c == nchunks - 1 ? min(DAM_ROWS, last_rows) : DAM_ROWS;
      if (ok) {   // warp-uniform
        unsigned char *slot_ptr = dam_smem + slot * DAM_SLOT_BYTES;
        const uint32_t base = s32(slot_ptr);
        if (nrow < DAM_ROWS) {   // rows past the sequence's end hold whatever the cache holds there: p = 0 for them, but 0 x NaN must not happen
          unsigned char *vrows = slot_ptr + 2 * DAM_BOX;
          const int pieces = (DAM_ROWS - nrow) * 8;      // 16-byte pieces per box
          for (int i = lane; i < 2 * pieces; i += 32)
            reinterpret_cast<uint4 *>(vrows + (i >= pieces ? DAM_BOX : 0) + nrow * 128)[i >= pieces ? i - pieces : i] = make_uint4(0u, 0u, 0u, 0u);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // these stores precede the slot's next tiled copy
          __syncwarp();
        }
        float sc4[4] = {0.f, 0.f, 0.f, 0.f}, sc4b[4] = {0.f, 0.f, 0.f, 0.f};   // two chains of four dependent MMAs instead of one of eight
        const uint32_t k_row = base + lr * 128;                        // this lane's K row in box 0
        const uint32_t k_xor = ((k_row >> 7) & 7u) << 4;               // swizzle of that row (the same in box 1: boxes are 2048 bytes)
        const uint32_t k_off = (lane >> 4) * 16;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          uint32_t a0[4], a1[4];
          dam_ldsm_x4(k_row + (p >> 1) * DAM_BOX + ((((p & 1) * 64) + k_off) ^ k_xor), a0);
          dam_ldsm_x4(k_row + (p >> 1) * DAM_BOX + ((((p & 1) * 64) + 32 + k_off) ^ k_xor), a1);
          mma_16816(sc4, a0, qf[p][0], qf[p][1]);
          mma_16816(sc4b, a1, qf[p][2], qf[p][3]);
        }
        float s_top = fmaf(sc4[1] + sc4b[1], DAM_LO_INV, sc4[0] + sc4b[0]) * sc, s_bot = fmaf(sc4[3] + sc4b[3], DAM_LO_INV, sc4[2] + sc4b[2]) * sc;
        if (rowq >= nrow) s_top = -INFINITY;
        if (rowq + 8 >= nrow) s_bot = -INFINITY;
        float cm = fmaxf(s_top, s_bot);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
        const float mn = fmaxf(m, cm);                    // finite: row 0 of a chunk always exists
        const float corr = exp2f(m - mn);
        const float p_top = exp2f(s_top - mn), p_bot = exp2f(s_bot - mn);
        float ps = p_top + p_bot;
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
        l = fmaf(l, corr, ps);
        m = mn;
        if (__any_sync(0xffffffffu, corr != 1.0f)) {
#pragma unroll
          for (int t = 0; t < 8; ++t) { acc[t][0] *= corr; acc[t][1] *= corr; acc[t][2] *= corr; acc[t][3] *= corr; }
        }
        // p as the B operand: column n = lane / 4 (0: head 0 hi, 1: head 0 lo, 2: head 1 hi, 3: head 1 lo, 4..7: zero),
        // rows 2 quad, 2 quad + 1 (b0) and + 8 (b1); p(head h, row r) lives in lane 4 (r % 8) + h
        const int n = lane >> 2, src_lane = (2 * quad) * 4 + ((n >> 1) & 1);
        const float pta = __shfl_sync(0xffffffffu, p_top, src_lane), ptb = __shfl_sync(0xffffffffu, p_top, src_lane + 4);
        const float pba = __shfl_sync(0xffffffffu, p_bot, src_lane), pbb = __shfl_sync(0xffffffffu, p_bot, src_lane + 4);
        uint32_t b0 = 0u, b1 = 0u;
        if (n < 4) {
          const bool lo = (n & 1) != 0;
          b0 = dam_pack(dam_split(pta, lo), dam_split(ptb, lo));
          b1 = dam_pack(dam_split(pba, lo), dam_split(pbb, lo));
        }
        const uint32_t v_row = base + 2 * DAM_BOX + ((lane & 7) + 8 * (lane >> 4)) * 128;
        const uint32_t v_xor = ((v_row >> 7) & 7u) << 4;
        const uint32_t v_off = ((lane >> 3) & 1) * 16;
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          uint32_t a[4];
          dam_ldsm_x4_trans(v_row + (t >> 2) * DAM_BOX + ((((t & 3) * 32) + v_off) ^ v_xor), a);
          mma_16816(acc[t], a, b0, b1);
        }
      }
      __syncwarp();
      if (!ok) break;
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(empty + slot)) : "memory");
    }
    ring += (nchunks >> 3) * chains + min(max((nchunks & (DAM_CHAINS - 1)) - chain0, 0), chains);
    fetched = s_taken > j + 1;
    asm volatile("" ::: "memory");       // (the piece is read behind the counter that says it is there)
    if (fetched && s_piece[(j + 1) % DAM_AHEAD].chunks >= 0) fetch_heads(s_piece[(j + 1) % DAM_AHEAD]);
    // this chain's partial state: lanes of quad h hold head h (columns hi, lo of the accumulator fragments)
    float *const item_states = split_part + static_cast<size_t>((b * NKV + g) * splits) * DAM_CHAINS * DAM_PART;
    float *const my_states = item_states + static_cast<size_t>(piece.split) * DAM_CHAINS * DAM_PART;
    const int h = threadIdx.x >> 7, d = threadIdx.x & (D - 1);
    __half *o = out + static_cast<size_t>(b) * QS + (2 * g + h) * D + d;
    if (parts == 1) {
      if (quad < 2) {
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          sacc[warp][quad][t * 16 + rowq] = fmaf(acc[t][1], DAM_LO_INV, acc[t][0]);
          sacc[warp][quad][t * 16 + rowq + 8] = fmaf(acc[t][3], DAM_LO_INV, acc[t][2]);
        }
        if (rowq == 0) { sm[warp][quad] = m; sl[warp][quad] = l; }
      }
      sync_consumers();
      // the range's state per (head, dim): maximum M, sum L, unnormalised output A
      float M = -INFINITY, L = 0.f, A = 0.f;
      if (last_split) M = snew_score[h];     // the new row is always there
#pragma unroll
      for (int w = 0; w < DAM_CHAINS; ++w) M = fmaxf(M, sm[w][h]);
      if (last_split) { L = exp2f(snew_score[h] - M); A = L * svnew[d]; }
#pragma unroll
      for (int w = 0; w < DAM_CHAINS; ++w) {
        const float mw = sm[w][h];
        const float s = (mw == -INFINITY) ? 0.f : exp2f(mw - M);
        L = fmaf(sl[w][h], s, L);
        A = fmaf(sacc[w][h][d], s, A);
      }
      if (splits == 1) {
        *o = __float2half_rn(A / L);
        continue;
      }
      my_states[h * (D + 2) + d] = A;
      if (d == 0) { my_states[h * (D + 2) + D] = M; my_states[h * (D + 2) + D + 1] = L; }
    } else if (warp < chains && quad < 2) {
      float *st = my_states + static_cast<size_t>(chain0 + warp) * DAM_PART + quad * (D + 2);
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        st[t * 16 + rowq] = fmaf(acc[t][1], DAM_LO_INV, acc[t][0]);
        st[t * 16 + rowq + 8] = fmaf(acc[t][3], DAM_LO_INV, acc[t][2]);
      }
      if (rowq == 0) { st[D] = m; st[D + 1] = l; }
    }
    // An item of several pieces: every CTA leaves its states in global memory and counts itself; the last one adds them up in
    // order and resets the counter.
    __threadfence();
    sync_consumers();
    if (threadIdx.x == 0) s_last = atomicAdd(split_count + b * NKV + g, 1u) == static_cast<unsigned int>(splits * parts - 1);
    sync_consumers();
    if (!s_last) continue;
    __threadfence();
    float ms[DAM_MAX_SPLITS], ls[DAM_MAX_SPLITS], as[DAM_MAX_SPLITS];
    if (parts == 1) {
#pragma unroll
      for (int sp = 0; sp < DAM_MAX_SPLITS; ++sp) {      // all loads first: one L2 round trip
        const float *st = item_states + static_cast<size_t>(sp) * DAM_CHAINS * DAM_PART + h * (D + 2);
        const bool have = sp < splits;
        ms[sp] = have ? __ldcg(st + D) : -INFINITY;
        ls[sp] = have ? __ldcg(st + D + 1) : 0.f;
        as[sp] = have ? __ldcg(st + d) : 0.f;
      }
    } else {
#pragma unroll
      for (int sp = 0; sp < DAM_MAX_SPLITS; ++sp) {
        ms[sp] = -INFINITY; ls[sp] = 0.f; as[sp] = 0.f;
        if (sp < splits) {
          float mw[DAM_CHAINS], lw[DAM_CHAINS], aw[DAM_CHAINS];
          const float *st = item_states + static_cast<size_t>(sp) * DAM_CHAINS * DAM_PART + h * (D + 2);
#pragma unroll
          for (int w = 0; w < DAM_CHAINS; ++w) {
            mw[w] = __ldcg(st + w * DAM_PART + D);
            lw[w] = __ldcg(st + w * DAM_PART + D + 1);
            aw[w] = __ldcg(st + w * DAM_PART + d);
          }
          float M = sp == splits - 1 ? snew_score[h] : -INFINITY, L = 0.f, A = 0.f;
#pragma unroll
          for (int w = 0; w < DAM_CHAINS; ++w) M = fmaxf(M, mw[w]);
          if (sp == splits - 1) { L = exp2f(snew_score[h] - M); A = L * svnew[d]; }
#pragma unroll
          for (int w = 0; w < DAM_CHAINS; ++w) {
            const float s = (mw[w] == -INFINITY) ? 0.f : exp2f(mw[w] - M);
            L = fmaf(lw[w], s, L);
            A = fmaf(aw[w], s, A);
          }
          ms[sp] = M; ls[sp] = L; as[sp] = A;
        }
      }
    }
    float Mt = -INFINITY;
#pragma unroll
    for (int sp = 0; sp < DAM_MAX_SPLITS; ++sp) Mt = fmaxf(Mt, ms[sp]);
    float Lt = 0.f, At = 0.f;
#pragma unroll
    for (int sp = 0; sp < DAM_MAX_SPLITS; ++sp) {
      const float s = (ms[sp] == -INFINITY) ? 0.f : exp2f(ms[sp] - Mt);
      Lt = fmaf(ls[sp], s, Lt);
      At = fmaf(as[sp], s, At);
    }
    *o = __float2half_rn(At / Lt);
    if (threadIdx.x == 0) split_count[b * NKV + g] = 0u;   // ready for the next launch (stream order)
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (*abort_flag) {
    __threadfence_block();
    drain(*issued_ctr);
  }
}

}  // namespace qmk_pf
#endif  // QMK_DECODE_ATTENTION_MMA_CUH_
