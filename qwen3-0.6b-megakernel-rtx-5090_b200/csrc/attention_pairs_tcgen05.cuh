// Causal attention of a long prefill chunk on the sm_100a tensor cores: the two query heads of a kv head in one CTA.
//
// A CTA works on two SLOTS of 128 query rows: one 128-query tile of the two heads that share a kv head, and so every key and value
// tile.  Keys and values come from the fp16 cache in tiles of 128 rows through two-stage rings fed by 3-D tiled TMA loads (no
// multicast; rows past the end of the sequence are outside the tensor map's extent and arrive as zeros).  Per slot h and tile u
//   S_h[128 x 128]  = Q_h . K_u^T    tcgen05.mma from shared memory, fp32 scores in 128 TMEM columns
//   P_h             = exp2(S_h - m)  four warps, one query row per thread: tcgen05.ld, causal mask, row maximum, exp2; P as
//                                    fp16 pairs back into the first 64 of the slot's score columns (tcgen05.st)
//   O_h[128 x 128] += P_h . V_u      tcgen05.mma with A in TMEM, B read MN-major from the [key][dim] rows
// A 128 x 128 tile of one slot is 2 x 512 cycles of tensor arithmetic and 16384 exponentials, 1024 cycles of the SM's MUFU: the
// slots take turns, one's products under the other's softmax (128 keys of both take about 3600 cycles: 1900 of a slot's softmax,
// 270 until its P is seen, 1200 of products).  causal_attention_tc - one head, 64-key tiles, P through shared memory as the A
// operand, keys and values brought once per head - takes 5400: prompts of 4000 / 8191 tokens 6.77 / 17.6 -> 6.59 / 16.8 ms.
// The products of one thread execute in issue order: "S_h of tile u is complete" also says that O_h is at rest and P_h consumed
// (P . V of u - 1 went before it), so a slot needs two barriers, scores ready and P ready.  Tried and slower: an issuing thread per
// slot with P handed over in halves (the tensor pipe then changes accumulators more often, at about 100 cycles a time);
// sub-tiles of 64 keys with two score buffers per slot (as fast, and further from float64); two loading threads.
// The running row maximum is only raised when it grew by more than 2^8 (P stays below 256, far inside fp16), so the accumulator
// in TMEM is rescaled a handful of times per row instead of once per tile; the row sums follow the same stale maximum and the
// final division makes the result exact again.  CTAs are numbered from the heaviest query tile down: longest job first.  The
// query tiles arrive by TMA as fp16 (the kernel before this one stores the rotated queries that way, pre-scaled); their shared
// memory takes the fp16 outputs at the end, which leave by tiled stores.  One CTA per SM (all 512 TMEM columns).  Every wait is
// bounded (status 4).
#ifndef QMK_ATTENTION_PAIRS_TCGEN05_CUH_
#define QMK_ATTENTION_PAIRS_TCGEN05_CUH_

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "attention_tcgen05.cuh"
#include "gemm_pair_tcgen05.cuh"

namespace qmk_attn_pairs {

using qmk_attn::fast_exp2;
using qmk_attn::smem_desc_mn_sw128;
using qmk_attn::tma_load_3d;

constexpr int D = 128, NQ = 16, NKV = 8;         // head dimension, query heads, kv heads
constexpr int TQ = 128, TK = 128;                // query rows per slot, keys per tile
constexpr int THREADS = 320;                     // warp 0 loads, warp 1 issues the MMAs, warps 2..5 / 6..9 own the query rows of slot 0 / 1
constexpr int STAGES = 2;
constexpr uint32_t HALF_BYTES = 128 * 128;       // 128 rows x 64 dims, swizzled
constexpr uint32_t TILE_BYTES = 2 * HALF_BYTES;  // a Q, K or V tile: two halves of the head dimension
constexpr uint32_t OFF_K = 2 * TILE_BYTES, OFF_V = OFF_K + STAGES * TILE_BYTES, OFF_BARS = OFF_V + STAGES * TILE_BYTES;
constexpr size_t SMEM_BYTES = OFF_BARS + 256;
constexpr uint32_t TMEM_COLS = 512;              // scores (then P) of slot h in columns [128 h, +128), O in [256 + 128 h, +128)
constexpr float RESCALE_THRESHOLD = 8.0f;        // log2 units

constexpr uint32_t IDESC_S = (1u << 4) | (static_cast<uint32_t>(TK >> 3) << 17) | (static_cast<uint32_t>(TQ >> 4) << 24);
constexpr uint32_t IDESC_PV = (1u << 4) | (1u << 16) /* B MN-major */ | (static_cast<uint32_t>(D >> 3) << 17) |
                              (static_cast<uint32_t>(TQ >> 4) << 24);
// D += A . B with A in TMEM: row = lane, two fp16 values of K per column.
__device__ __forceinline__ void mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t accumulate, uint32_t idesc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// map_q: 2-D map of the fp16 queries [rows][16 heads x 128] (normalised, rotated, times scale * log2 e), boxes of
// {64, 128}, 128-byte swizzle; query t sits at position pos0 + t and sees cache rows 0 .. pos0 + t.  map_k / map_v: 3-D maps
// {128 dims, pos0 + T rows, layers x 8 kv heads} of the fp16 caches, boxes of {64, 128, 1}, 128-byte swizzle.  map_out: the
// fp16 outputs [rows][2048] in blocks of 32 x 64 (whole query tiles are stored: rows past the live ones hold values that
// nothing reads).  grid = ceil(T / 128) * 8 CTAs in one dimension, numbered from the heaviest (last) query tile down.
__global__ void __launch_bounds__(THREADS, 1)
causal_attention_pairs(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                       const __grid_constant__ CUtensorMap map_out, int layer_head0, int T, int pos0, unsigned int *status,
                       unsigned long long budget_ns) {
  using namespace qmk_gemm;
  extern __shared__ __align__(1024) unsigned char attn_smem[];
  const uint32_t base = s32(attn_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total = static_cast<int>(gridDim.x), id = static_cast<int>(blockIdx.x);
  const int kv_head = id % NKV, head0 = 2 * kv_head;
  const int q0 = (total / NKV - 1 - id / NKV) * TQ;
  const int pbase = pos0 + q0;                 // position of the tile's first query
  const int last_q = (q0 + TQ < T ? q0 + TQ : T) - 1;                                        // last live query of the tile
  const int ntiles = (pbase + last_q - q0) / TK + 1;                                        // key tiles it can see
  const uint32_t bars = base + OFF_BARS;
  auto k_full = [&](int s) { return bars + 8u * s; };
  auto k_empty = [&](int s) { return bars + 8u * (2 + s); };
  auto v_full = [&](int s) { return bars + 8u * (4 + s); };
  auto v_empty = [&](int s) { return bars + 8u * (6 + s); };
  auto s_full = [&](int h) { return bars + 8u * (8 + h); };        // scores of slot h complete; behind its last tile: O complete
  auto p_ready = [&](int h) { return bars + 8u * (10 + h); };      // P of slot h stored
  const uint32_t q_full = bars + 8u * 12;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(attn_smem + OFF_BARS + 8 * 13);
  static_assert(STAGES == 2, "barrier layout above");
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  if ((base & 1023u) != 0u) {   // the swizzled tiles need a 1024-byte aligned window: report instead of computing garbage
    if (threadIdx.x == 0) atomicCAS(status, 0u, 5u);
    return;
  }
  if (warp == 0 && elect_one()) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_q)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_k)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_v)) : "memory");
    for (int s = 0; s < STAGES; ++s) {
      bar_init(k_full(s), 1); bar_init(v_full(s), 1); bar_init(k_empty(s), 1); bar_init(v_empty(s), 1);
    }
    for (int h = 0; h < 2; ++h) {
      bar_init(s_full(h), 1);
      bar_init(p_ready(h), 4);        // one arrival per softmax warp of the slot
    }
    bar_init(q_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_wait();   // queries and this chunk's cache rows come from the kernel launched just before
  auto load_tile = [&](const CUtensorMap *map, uint32_t dst, int j, uint32_t full) {
    bar_expect_tx(full, TILE_BYTES);
    tma_load_3d(dst, map, 0, j * TK, layer_head0 + kv_head, full);
    tma_load_3d(dst + HALF_BYTES, map, 64, j * TK, layer_head0 + kv_head, full);
  };
  const int prefilled = ntiles < STAGES ? ntiles : STAGES;
  if (warp == 0) {
    __syncwarp();
    // the query tiles and the rings' first fill go out at once; a CTA's fixed costs weigh as much as its first key tiles
    if (elect_one()) {
      // fp16, already times scale * log2 e (the softmax is an exp2), as [128 x 64] boxes in the K-major 128-byte-swizzled layout
      // the score MMAs read; rows past the live ones hold other tokens' or stale values
      bar_expect_tx(q_full, 2 * TILE_BYTES);
#pragma unroll
      for (int i = 0; i < 4; ++i) tma_load_2d(base + i * HALF_BYTES, &map_q, head0 * D + i * 64, q0, q_full);
      for (int j = 0; j < prefilled; ++j) {
        load_tile(&map_k, base + OFF_K + j * TILE_BYTES, j, k_full(j));
        load_tile(&map_v, base + OFF_V + j * TILE_BYTES, j, v_full(j));
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // behind the TMEM allocation: the next kernel's CTAs allocate too, and hold what they have while they wait for this kernel
  pdl_trigger();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {                     // ---- producer (V of a tile is asked for behind its K: the issuer needs them in that order)
      int issued_k = prefilled, issued_v = prefilled;
      for (int j = prefilled; j < ntiles; ++j) {
        const int s = j & 1;
        const uint32_t parity = ((j >> 1) - 1) & 1;
        if (!bar_wait(k_empty(s), parity, abort_flag, status, budget_ns)) break;
        load_tile(&map_k, base + OFF_K + s * TILE_BYTES, j, k_full(s));
        issued_k = j + 1;
        if (!bar_wait(v_empty(s), parity, abort_flag, status, budget_ns)) break;
        load_tile(&map_v, base + OFF_V + s * TILE_BYTES, j, v_full(s));
        issued_v = j + 1;
      }
      if (*abort_flag) {                   // copies already issued must land before the CTA may exit
        auto landed = [&](uint32_t bar, uint32_t parity) {
          const unsigned long long t0 = gtime();
          while (!bar_try(bar, parity))
            if (gtime() - t0 > (budget_ns > 2000000ull ? budget_ns : 2000000ull)) break;
        };
        landed(q_full, 0);
        for (int j = (issued_k > STAGES ? issued_k - STAGES : 0); j < issued_k; ++j) landed(k_full(j & 1), (j >> 1) & 1);
        for (int j = (issued_v > STAGES ? issued_v - STAGES : 0); j < issued_v; ++j) landed(v_full(j & 1), (j >> 1) & 1);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {                     // ---- MMA issuer: S_0 S_1 | PV_0 S_0 | PV_1 S_1 | ...
      const uint64_t dq = smem_desc_sw128(base), dk = smem_desc_sw128(base + OFF_K), dv0 = smem_desc_mn_sw128(base + OFF_V, HALF_BYTES);
      bool ok = bar_wait(q_full, 0, abort_flag, status, budget_ns);
      auto scores = [&](int h, int u) {
        const int s = u & 1;
        if (h == 0) ok = ok && bar_wait(k_full(s), (u >> 1) & 1, abort_flag, status, budget_ns);
        if (!ok) return;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t da = dq + h * (TILE_BYTES >> 4), db = dk + s * (TILE_BYTES >> 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {      // 16 of the 128 dims; the second half of them HALF_BYTES further on
          const uint64_t o = (i >> 2) * (HALF_BYTES >> 4) + 2u * (i & 3);
          mma_f16_ss(tmem_base + 128u * h, da + o, db + o, i > 0 ? 1u : 0u, IDESC_S);
        }
        mma_commit(s_full(h));
        if (h == 1) mma_commit(k_empty(s));
      };
      scores(0, 0);
      scores(1, 0);
      for (int u = 0; u < ntiles && ok; ++u) {
        const int s = u & 1;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          ok = ok && bar_wait(p_ready(h), u & 1, abort_flag, status, budget_ns) &&
               (h == 1 || bar_wait(v_full(s), (u >> 1) & 1, abort_flag, status, budget_ns));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // O_h += P_h . V_u: eight steps of 16 keys; V rows are [key][dim], i.e. MN-major for the B operand
          const uint64_t dv = dv0 + s * (TILE_BYTES >> 4);
#pragma unroll
          for (int i = 0; i < 8; ++i)
            mma_f16_ts(tmem_base + 256u + 128u * h, tmem_base + 128u * h + 8u * i, dv + static_cast<uint64_t>(i * (16 * 128 >> 4)),
                       (u > 0 || i > 0) ? 1u : 0u, IDESC_PV);
          if (h == 1) mma_commit(v_empty(s));
          if (u + 1 < ntiles) scores(h, u + 1);
          else mma_commit(s_full(h));       // O_h is complete
        }
      }
    }
  } else {                                 // ---- softmax: slot = warp group, thread = query row = TMEM lane
    const int h = (warp - 2) >> 2;
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const int qpos = pbase + row;          // (rows past T compute on values that nothing reads)
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tmem_s = tmem_base + lane_base + 128u * h, tmem_o = tmem_base + lane_base + 256u + 128u * h;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int u = 0; u < ntiles; ++u) {
      ok = __all_sync(0xffffffffu, bar_wait(s_full(h), u & 1, abort_flag, status, budget_ns));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t s[4][32];
#pragma unroll
      for (int q = 0; q < 4; ++q) tmem_ld32(tmem_s + 32u * q, s[q]);
      tmem_ld_wait();
      const int k0 = u * TK;
      if (k0 + TK - 1 > pbase) {            // some key of the tile is ahead of some query of the CTA
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (k0 + 32 * q + c > qpos) s[q][c] = __float_as_uint(-INFINITY);
      }
      // (four independent chains: a single running maximum would be 64 dependent instructions)
      float mx4[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        mx4[q] = fmaxf(__uint_as_float(s[q][0]), __uint_as_float(s[q][1]));
#pragma unroll
        for (int c = 2; c < 32; c += 2) mx4[q] = max3(mx4[q], __uint_as_float(s[q][c]), __uint_as_float(s[q][c + 1]));
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // raise the maximum in use only when it is far behind (always from -inf)
      const bool raise = mx > m_used + RESCALE_THRESHOLD;
      if (__any_sync(0xffffffffu, raise)) {
        const float m_new = raise ? mx : m_used;
        const float alpha = raise ? exp2f(m_used - m_new) : 1.0f;     // from -inf: exp2(-inf) = 0, l and O hold zeros at most
        if (u > 0) {
#pragma unroll 1
          for (int c = 0; c < D / 16; ++c) {
            uint32_t o[16];
            tmem_ld16(tmem_o + 16u * c, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st16(tmem_o + 16u * c, o);
          }
        }
        l *= alpha;
        m_used = m_new;
      }
      const float m_sub = m_used == -INFINITY ? 0.f : m_used;   // every score so far -inf: P = exp2(-inf - 0) = 0, not NaN
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < 8; ++q) {         // (eight columns at a time: sixteen spilled)
        uint32_t p[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float a = fast_exp2(__uint_as_float(s[q >> 1][16 * (q & 1) + 2 * i]) - m_sub),
                      b = fast_exp2(__uint_as_float(s[q >> 1][16 * (q & 1) + 2 * i + 1]) - m_sub);
          sum4[i & 3] += a + b;
          p[i] = qmk_pair::half2_bits(a, b);
        }
        tmem_st8(tmem_s + 8u * q, p);
      }
      l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(p_ready(h)) : "memory");
    }
    if (ok) ok = __all_sync(0xffffffffu, bar_wait(s_full(h), ntiles & 1, abort_flag, status, budget_ns));
    // outputs as fp16 through the query tiles' shared memory
    if (ok) {                             // (every product that reads this slot's query tile has finished)
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float inv = 1.0f / l;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t packed[32];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t o[32];
          tmem_ld32(tmem_o + 64u * half + 32u * c, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) packed[16 * c + i] = qmk_pair::half2_bits(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
        }
        const uint32_t block = base + h * TILE_BYTES + half * HALF_BYTES + quarter * 4096u;
        qmk_pair::stage_row(block, lane, packed);
        qmk_pair::store_block(&map_out, block, (head0 + h) * D + 64 * half, q0 + quarter * 32);
      }
    }
    __syncwarp();
    if (elect_one()) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

}  // namespace qmk_attn_pairs
#endif  // QMK_ATTENTION_PAIRS_TCGEN05_CUH_
