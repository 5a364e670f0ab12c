// C[M x N] = A[M x K] * B[N x K]^T (fp16 operands, fp32 accumulation) for long chunks: pairs of CTAs on one 256 x 256 tile.
//
// With tcgen05.mma.cta_group::2 each CTA of a pair brings its own 128 rows of A and HALF of the 256 rows of B, and both halves feed
// both tensor cores: 32 KB for 512 cycles of arithmetic per 64-wide K block.  Measured per K block, from the cycles of 4096 x 4096
// products of K = 1536 and 3072: 525 (operands zero) to 555 (random).  A launch's remaining time is its start, its last
// epilogue and the pairs without a tile in the last round (2048 rows: tensor pipe 57 and 64 % active in the q/k/v and gate/up
// products, 40 and 51 % in O and down, whose 64 tiles are one for each of 64 pairs).
// What single-CTA tiles of 128 x 256 lose is not their main loop: stand-alone, with every SM at work on operands in L2, loads of
// 48 KB take 458 cycles (107 bytes per cycle and SM; 32 KB 367; one SM alone 125 bytes per cycle), N = 256 MMAs of resident
// operands 512, and both together 513.  What is left is that they start and end a CTA once per tile.
//
// Persistent: a pair takes tiles pair, pair + pairs, ... (m fastest), and the accumulator has two buffers of 256 TMEM columns,
// so the epilogue of one tile runs under the main loop of the next.  Roles per CTA: warp 0 loads (one thread), warp 1 of
// the pair's first CTA issues the MMAs of both (one thread), warps 2..9 store: warp w holds TMEM lanes 32 * (w % 4) .. and one
// half of the columns; they go through a 4 KB block per warp to tiled bulk stores (a thread holds a row: 32-byte pieces straight
// from registers took 4096 LSU cycles a tile, the last epilogue of an fp32 product 4.6 us).  The full barriers live in the first CTA - the second CTA's copies complete there too
// (.cta_group::2) - the empty and accumulator-full barriers in both (multicast commit).  No multicast loads.
//
// MODE 0: C fp32; 1: C fp16; 2: fp16 silu(gate) * up, where the pair's first CTA brings 128 gate rows and the second the 128 up
// rows of the same columns.  3: fp32, added to C: a pair makes the two parts of K of a tile one after the other and adds each to
// the matrix with bulk reductions, in order, the first under the main loop of the second. At 4096 rows a product of 1024 columns
// takes 21 us (19 with two matrices of partial sums, whose row kernel then takes 12 instead of 5).
// 4: q, k and v with QK norm, rotation and cache write in the epilogue (store_heads): 43 -> 34 us a layer at 4096 rows.
// RS: every B row has an fp32 scale (expanded packed matrices).
// Every wait is bounded (status 4).  After a time-out of whatever role the issuing thread gives up too, or is through: it then waits
// for the MMAs issued and the copies of both CTAs in flight, which complete on its barriers (`drain`), or its readers wait for the
// accumulator it has completed, before both CTAs meet at the cluster barrier, free TMEM and leave.  All of it in the roles' cold
// exits: a look at a flag behind the barriers, with a second meeting for the drain, made prompts of 513 to 760 tokens 1.2 % longer.
#ifndef QMK_GEMM_PAIR_TCGEN05_CUH_
#define QMK_GEMM_PAIR_TCGEN05_CUH_

#include "gemm_tcgen05.cuh"
#include "prefill_kernels.cuh"

namespace qmk_pair {

using qmk_gemm::BK;
constexpr int TM = 256, TN = 256;                      // tile of a pair
constexpr int THREADS = 320;
constexpr int STAGES = 6;
constexpr uint32_t TILE_BYTES = 128 * BK * 2;          // 128 rows of A, or of B, per CTA and K block
constexpr uint32_t STAGE_BYTES = 2 * TILE_BYTES;
constexpr uint32_t RING_BYTES = STAGES * STAGE_BYTES;
constexpr uint32_t BLOCK_BYTES = 32 * 128;             // an epilogue warp's staging block: 32 rows of 32 floats or 64 halves
constexpr uint32_t OFF_BARS = RING_BYTES + 8 * BLOCK_BYTES;
constexpr size_t SMEM_BYTES = 1024 + OFF_BARS + 256;
static_assert(SMEM_BYTES <= 232448, "over the 227 KB shared-memory limit of one CTA");
constexpr uint32_t IDESC = (1u << 4) | (static_cast<uint32_t>(TN >> 3) << 17) | (static_cast<uint32_t>(TM >> 4) << 24);

// MODE 4: where the rows of q, k and v go.
struct Heads {
  const __half *q_norm, *k_norm;
  const float *rope;                          // fp32 rows, or null: the fp16 tables
  const __half *cos_table, *sin_table;
  __half *queries;                            // [row][16][128], times q_scale
  __half *k_cache, *v_cache;                  // one layer's rows [head][max_seq_len][128] (packed prompts: kv_ptrs + layer_off)
  const int2 *row_info;                       // packed prompts: (sequence, position or < 0) of each row; a prompt begins with a row tile of 128
  const unsigned long long *kv_ptrs;
  size_t layer_off;
  int rows, pos0, max_seq_len;
  float q_scale;
};
struct Args {
  Heads heads;
  int N[3];                      // columns of the groups' matrices (multiples of 256; MODE 2: of 128, group 0 only)
  const float *row_scale[3];     // RS: scales of the groups' B rows (MODE 2: [0] gate, [1] up)
  int m_tiles, n_tiles, splits;  // tiles of 256 rows / 256 columns (MODE 2: 128 outputs) over all groups, parts of K
  int kblocks;                   // K blocks of 64 of a part; the partial matrices (MODE 0) are m_tiles * 256 rows apart
};

enum SelfTest { NO_LOADS = 1, ISSUER_STOPS = 2, SECOND_CTA_NO_LOADS = 3 };   // of the bounded waits (the issuer: behind a pair's first tile)

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t in_first_cta(uint32_t addr) {   // the same shared-memory address in the pair's first CTA
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// (does not wait for this thread's stores)
__device__ __forceinline__ void cluster_leave() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap *map, int c0, int c1, uint32_t first_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(first_bar)
      : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(IDESC), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void commit_pair(uint32_t bar) {   // arrives on this barrier of both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(static_cast<unsigned short>(3)) : "memory");
}
// The issuing thread's way out after a time-out: the MMAs issued so far end, and so do the copies of the ring of K blocks
// [next, next + STAGES) below `end` that either loader may have asked for.  (Where one CTA has asked for its half of a block and
// the other has not, the barrier does not complete and the wait takes its whole limit.)
__device__ __noinline__ void drain(uint32_t full0, uint32_t stopped, int next, int end, unsigned long long budget_ns) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(stopped) : "memory");
  qmk_gemm::bar_drain(stopped, 0, budget_ns);
  for (int i = next; i < end && i < next + STAGES; ++i)
    qmk_gemm::bar_drain(full0 + 8u * static_cast<uint32_t>(i % STAGES), static_cast<uint32_t>(i / STAGES) & 1u, budget_ns);
}
// One row of 128 bytes of a warp's 32 x 128-byte block, in the 128-byte swizzle its store expects (conflict-free).
__device__ __forceinline__ void stage_row(uint32_t block, int lane, const uint32_t (&v)[32]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(block + static_cast<uint32_t>(lane * 128 + ((i ^ (lane & 7)) << 4))),
                 "r"(v[4 * i]), "r"(v[4 * i + 1]), "r"(v[4 * i + 2]), "r"(v[4 * i + 3]) : "memory");
}
// The staged block to (ADD: added to) columns c0 .., rows c1 .. of the matrix (rows past its end are not written).
template <bool ADD = false>
__device__ __forceinline__ void store_block(const CUtensorMap *map, uint32_t block, int c0, int c1) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (qmk_gemm::elect_one()) {
    if (ADD)
      asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%1, %2}], [%3];"
                   ::"l"(map), "r"(c0), "r"(c1), "r"(block) : "memory");
    else
      asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
                   ::"l"(map), "r"(c0), "r"(c1), "r"(block) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
}
// The block may be written again.
__device__ __forceinline__ void block_free() {
  if (qmk_gemm::elect_one()) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  __syncwarp();
}
__device__ __forceinline__ float2 as_floats(uint32_t bits) { return __half22float2(*reinterpret_cast<const __half2 *>(&bits)); }
// MODE 4, a warp's 32 rows of one head (group 0 q, 1 k, 2 v) from row t0, packed halves of row `lane` in `row`: QK norm and rotation with
// the operations of qk_norm_rope_cache, bit for bit.  The squares are added by the thread that holds the row, in the order of that
// kernel's shuffles; the rest goes row by row through the warp's 4 KB, 16 rows at a time, so that tables, cache and queries are read
// and written in whole lines: lane l has dims 2 l, 2 l + 1 and their partners 64 behind, no value crosses lanes.  The tables'
// rows of the next step are asked for ahead (1500 / 2200 / 4096 tokens 2.456 / 3.14 / 6.28 -> 2.40 / 3.08 / 6.22 ms).  A first form, that
// kernel's lanes and shuffles as they are, took 51 us a product at 4096 rows; this one 34, the product and the kernel in turn 43.
// Storing plain halves takes 26.6: with heads an epilogue (86 instructions a row of a head on average, two warps on each scheduler) is
// longer than the main loop it runs under.
__device__ __forceinline__ void store_heads(const Heads &a, uint32_t block, int lane, const uint32_t (&row)[64], int grp, int head, int t0) {
  using qmk_pf::D;
  int live = min(max(a.rows - t0, 0), 32), pos = a.pos0 + t0;
  __half *kc = a.k_cache, *vc = a.v_cache;
  if (a.row_info) {
    const int2 info = lane < live ? a.row_info[t0 + lane] : make_int2(0, -1);
    live = __popc(__ballot_sync(0xffffffffu, info.y >= 0));      // (rows of one prompt, then padding)
    const int seq = __shfl_sync(0xffffffffu, info.x, 0);
    pos = __shfl_sync(0xffffffffu, info.y, 0);
    kc = reinterpret_cast<__half *>(a.kv_ptrs[2 * seq]) + a.layer_off;
    vc = reinterpret_cast<__half *>(a.kv_ptrs[2 * seq + 1]) + a.layer_off;
  }
  if (live == 0) return;
  __half *const out = (grp == 0 ? a.queries + (static_cast<size_t>(t0) * qmk_pf::NQ + head) * D
                                : (grp == 1 ? kc : vc) + (static_cast<size_t>(head) * a.max_seq_len + pos) * D) + 2 * lane;
  const size_t pitch = grp == 0 ? qmk_pf::QS : D;
  const bool first = (lane & 1) == 0;      // this lane's first dim is that of a four (see qk_norm_rope_cache)
  float2 w0 = make_float2(0.f, 0.f), w1 = w0;
  float rstd = 0.f;
  if (grp < 2) {
    const __half *const norm = (grp == 0 ? a.q_norm : a.k_norm) + 2 * lane;
    w0 = __half22float2(*reinterpret_cast<const __half2 *>(norm));
    w1 = __half22float2(*reinterpret_cast<const __half2 *>(norm + 64));
    auto squares4 = [&](int i) {           // dims 4 i .. 4 i + 3
      const float2 x = as_floats(row[2 * i]), y = as_floats(row[2 * i + 1]);
      return fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(y.x, y.x, y.y * y.y)));
    };
    float t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) t[i] = squares4(i) + squares4(i + 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < o; ++i) t[i] += t[i + o];
    rstd = 1.0f / sqrtf(t[0] * (1.0f / D) + qmk_pf::RMS_EPS);
  }
  constexpr int ROWS = 4;                  // in flight together
  float2 cs_next[ROWS], sn_next[ROWS];
  auto ask = [&](int first) {
    if (grp == 2) return;
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const size_t at = static_cast<size_t>(pos + min(first + j, live - 1)) * D + 2 * lane;
      if (a.rope) {
        cs_next[j] = *reinterpret_cast<const float2 *>(a.rope + at);
        sn_next[j] = *reinterpret_cast<const float2 *>(a.rope + at + 64);
      } else {
        cs_next[j] = __half22float2(*reinterpret_cast<const __half2 *>(a.cos_table + at));
        sn_next[j] = __half22float2(*reinterpret_cast<const __half2 *>(a.sin_table + at));
      }
    }
  };
  ask(0);
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    if (hh * 16 >= live) break;
    __syncwarp();
    if ((lane >> 4) == hh) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(block + static_cast<uint32_t>((lane & 15) * 256 + ((i ^ (lane & 7)) << 4))),
                     "r"(row[4 * i]), "r"(row[4 * i + 1]), "r"(row[4 * i + 2]), "r"(row[4 * i + 3]) : "memory");
    }
    __syncwarp();
#pragma unroll 1
    for (int i0 = 0; i0 < 16 && hh * 16 + i0 < live; i0 += ROWS) {
      float2 cs[ROWS], sn[ROWS];
      uint32_t lo[ROWS], hi[ROWS];
#pragma unroll
      for (int j = 0; j < ROWS; ++j) { cs[j] = cs_next[j]; sn[j] = sn_next[j]; }
      ask(hh * 16 + i0 + ROWS);
#pragma unroll
      for (int j = 0; j < ROWS; ++j) {
        const int i = i0 + j;
        const uint32_t at = block + static_cast<uint32_t>(i * 256 + (((lane >> 2) ^ (i & 7)) << 4) + (lane & 3) * 4);
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(lo[j]) : "r"(at));
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(hi[j]) : "r"(at + 128));
      }
      if (grp < 2) {
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
          const float rs = __shfl_sync(0xffffffffu, rstd, hh * 16 + i0 + j);
          float2 l = as_floats(lo[j]), h = as_floats(hi[j]);
          l.x = l.x * rs * w0.x; l.y = l.y * rs * w0.y;
          h.x = h.x * rs * w1.x; h.y = h.y * rs * w1.y;
          float2 rl = make_float2(fmaf(l.x, cs[j].x, -__fmul_rn(h.x, sn[j].x)), fmaf(l.y, cs[j].y, -__fmul_rn(h.y, sn[j].y)));
          float2 rh = make_float2(first ? fmaf(l.x, sn[j].x, __fmul_rn(h.x, cs[j].x)) : fmaf(h.x, cs[j].x, __fmul_rn(l.x, sn[j].x)),
                                  fmaf(h.y, cs[j].y, __fmul_rn(l.y, sn[j].y)));
          if (grp == 0) { rl.x *= a.q_scale; rl.y *= a.q_scale; rh.x *= a.q_scale; rh.y *= a.q_scale; }
          const __half2 pl = __floats2half2_rn(rl.x, rl.y), ph = __floats2half2_rn(rh.x, rh.y);
          lo[j] = *reinterpret_cast<const uint32_t *>(&pl);
          hi[j] = *reinterpret_cast<const uint32_t *>(&ph);
        }
      }
#pragma unroll
      for (int j = 0; j < ROWS; ++j)
        if (hh * 16 + i0 + j < live) {
          uint32_t *const at = reinterpret_cast<uint32_t *>(out + (hh * 16 + i0 + j) * pitch);
          at[0] = lo[j];
          at[32] = hi[j];
        }
    }
  }
  __syncwarp();
}
__device__ __forceinline__ uint32_t half2_bits(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}

template <int MODE, bool RS, int TEST = 0>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b0,
                 const __grid_constant__ CUtensorMap map_b1, const __grid_constant__ CUtensorMap map_b2, const __grid_constant__ CUtensorMap map_c0,
                 const __grid_constant__ CUtensorMap map_c1, const __grid_constant__ CUtensorMap map_c2, const Args args,
                 unsigned int *status, unsigned long long budget_ns) {
  using namespace qmk_gemm;
  extern __shared__ unsigned char pair_smem_raw[];
  const uint32_t raw = s32(pair_smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t bars = base + OFF_BARS;
  auto full = [&](int s) { return bars + 8u * s; };                       // (in the first CTA)
  auto empty = [&](int s) { return bars + 8u * (STAGES + s); };
  auto acc_full = [&](int b) { return bars + 8u * (2 * STAGES + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (2 * STAGES + 2 + b); };   // (in the first CTA)
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(pair_smem_raw + (base - raw) + OFF_BARS + 8 * (2 * STAGES + 4));
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const uint32_t stopped = bars + 8u * (2 * STAGES + 6);                     // after a time-out: the MMAs issued have ended
  static_assert(8 * (2 * STAGES + 7) <= 256, "barriers, TMEM address and flag fit behind the ring");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int mn_tiles = args.m_tiles * args.n_tiles, tiles = mn_tiles * args.splits;
  const int kblocks = args.kblocks;
  // the pair's n-th tile, of `count`
  const int count = MODE == 3 ? (mn_tiles - pair + pairs - 1) / pairs * 2 : (tiles - pair + pairs - 1) / pairs;
  auto tile_of = [&](int n) { return MODE == 3 ? (n & 1) * mn_tiles + pair + (n >> 1) * pairs : pair + n * pairs; };

  if (warp == 0 && elect_one()) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_b0)) : "memory");
    if (MODE == 2) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_b1)) : "memory");
    for (int s = 0; s < STAGES; ++s) { bar_init(full(s), 1); bar_init(empty(s), 1); }
    for (int b = 0; b < 2; ++b) { bar_init(acc_full(b), 1); bar_init(acc_empty(b), 16); }   // eight warps of either CTA
    bar_init(stopped, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();                          // both CTAs' barriers are initialised
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  // tile -> group, first row, first column within the group's matrix, part of K
  auto locate = [&](int tile, int &grp, int &mt, int &nt, int &z) {
    z = tile / mn_tiles;
    tile -= z * mn_tiles;
    nt = tile / args.m_tiles;
    mt = tile - nt * args.m_tiles;
    grp = 0;
    if (MODE != 2) {
      if (nt >= args.N[0] / TN) { nt -= args.N[0] / TN; grp = 1; }
      if (grp == 1 && nt >= args.N[1] / TN) { nt -= args.N[1] / TN; grp = 2; }
    }
  };

  if (warp == 0) {
    if (elect_one()) {                     // ---- producer: this CTA's rows of A and its half of B
      int s = 0;
      uint32_t parity = 1;                 // (the first pass over the ring finds it empty)
      bool ok = !(TEST == NO_LOADS || (TEST == SECOND_CTA_NO_LOADS && rank == 1)), waited = false;
      for (int n = 0; n < count && ok; ++n) {
        int grp, mt, nt, z;
        locate(tile_of(n), grp, mt, nt, z);
        const CUtensorMap *map_b = MODE == 2 ? (rank == 0 ? &map_b0 : &map_b1) : grp == 0 ? &map_b0 : grp == 1 ? &map_b1 : &map_b2;
        const int arow = mt * TM + static_cast<int>(rank) * 128;
        const int brow = MODE == 2 ? nt * 128 : nt * TN + static_cast<int>(rank) * 128;
        int b_ahead = 0;
        if (!waited) {
          // B is a weight matrix: the first fill of the ring is requested before the wait for the kernel that writes A
          for (; b_ahead < STAGES && b_ahead < kblocks; ++b_ahead) {
            if (rank == 0) bar_expect_tx(full(b_ahead), 2 * STAGE_BYTES);
            tma_load_pair(base + b_ahead * STAGE_BYTES + TILE_BYTES, map_b, (z * kblocks + b_ahead) * BK, brow, in_first_cta(full(b_ahead)));
          }
          pdl_wait();
          pdl_trigger();                   // (behind the TMEM allocation)
          waited = true;
        }
        for (int kb = 0; kb < kblocks; ++kb) {
          const uint32_t fbar = in_first_cta(full(s)), dst = base + s * STAGE_BYTES;
          const int kcol = (z * kblocks + kb) * BK;
          if (kb >= b_ahead) {
            ok = bar_wait(empty(s), parity, abort_flag, status, budget_ns);
            if (!ok) break;
            if (rank == 0) bar_expect_tx(full(s), 2 * STAGE_BYTES);
            tma_load_pair(dst + TILE_BYTES, map_b, kcol, brow, fbar);
          }
          tma_load_pair(dst, &map_a, kcol, arow, fbar);
          if (++s == STAGES) { s = 0; parity ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {        // ---- MMA issuer of the pair
      int s = 0, n = 0;
      uint32_t parity = 0;
      bool ok = true;
      auto give_up = [&](int next) { drain(full(0), stopped, next, count * kblocks, budget_ns); };
      for (; n < count && ok; ++n) {
        const int buf = n & 1;
        ok = n < 2 || bar_wait(acc_empty(buf), ((n >> 1) - 1) & 1, abort_flag, status, budget_ns);
        if (TEST == ISSUER_STOPS && n == 1) ok = bar_wait(stopped, 0, abort_flag, status, budget_ns);   // (nothing arrives)
        if (!ok) { give_up(n * kblocks); break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem_base + static_cast<uint32_t>(buf) * TN;
        for (int kb = 0; kb < kblocks; ++kb) {
          ok = bar_wait(full(s), parity, abort_flag, status, budget_ns);
          if (!ok) { give_up(n * kblocks + kb); break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t da = smem_desc_sw128(base + s * STAGE_BYTES), db = smem_desc_sw128(base + s * STAGE_BYTES + TILE_BYTES);
#pragma unroll
          for (int j = 0; j < BK / 16; ++j) mma_pair(d, da + 2u * j, db + 2u * j, (kb > 0 || j > 0) ? 1u : 0u);
          commit_pair(empty(s));
          if (++s == STAGES) { s = 0; parity ^= 1u; }
        }
        if (ok) commit_pair(acc_full(buf));
      }
    }
  } else {                                 // ---- epilogue
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t block = base + RING_BYTES + static_cast<uint32_t>(warp - 2) * BLOCK_BYTES;
    for (int n = 0; n < count; ++n) {
      const int buf = n & 1;
      int grp, mt, nt, z;
      locate(tile_of(n), grp, mt, nt, z);
      const bool ok = __all_sync(0xffffffffu, bar_wait(acc_full(buf), (n >> 1) & 1, abort_flag, status, budget_ns));
      if (!ok) {
        bar_drain(acc_full(buf), (n >> 1) & 1, budget_ns);
        if (n + 1 < count) bar_drain(acc_full(buf ^ 1), ((n + 1) >> 1) & 1, budget_ns);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem_base + static_cast<uint32_t>(buf) * TN + (static_cast<uint32_t>(quarter * 32) << 16);
      const int row = (MODE == 3 ? 0 : z * args.m_tiles * TM) + mt * TM + static_cast<int>(rank) * 128 + quarter * 32;   // first of the warp's 32
      const bool reused = n + 2 < count;
      auto release = [&]() {               // the buffer has been read
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (reused && lane == 0) arrive_cluster(in_first_cta(acc_empty(buf)));
      };
      if (MODE == 2) {
        const int col = nt * 128 + half * 64;
        uint32_t out[32];
#pragma unroll
        for (int c = 0; c < 4; ++c) {       // 16 gate columns and the same 16 up columns
          uint32_t g[16], u[16];
          tmem_ld16(acc + half * 64 + c * 16, g);
          tmem_ld16(acc + 128 + half * 64 + c * 16, u);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float g0 = __uint_as_float(g[2 * i]), g1 = __uint_as_float(g[2 * i + 1]);
            float u0 = __uint_as_float(u[2 * i]), u1 = __uint_as_float(u[2 * i + 1]);
            if (RS) {
              const float2 sg = __ldg(reinterpret_cast<const float2 *>(args.row_scale[0] + col + c * 16) + i);
              const float2 su = __ldg(reinterpret_cast<const float2 *>(args.row_scale[1] + col + c * 16) + i);
              g0 *= sg.x; g1 *= sg.y; u0 *= su.x; u1 *= su.y;
            }
            out[c * 8 + i] = half2_bits(__fdividef(g0, 1.0f + __expf(-g0)) * u0, __fdividef(g1, 1.0f + __expf(-g1)) * u1);
          }
        }
        release();
        block_free();
        stage_row(block, lane, out);
        store_block(&map_c0, block, col, row);
      } else if (MODE == 4) {               // a warp's 128 columns are a head
        const float *scale = RS ? (grp == 0 ? args.row_scale[0] : grp == 1 ? args.row_scale[1] : args.row_scale[2]) + nt * TN + half * 128 : nullptr;
        uint32_t head[64];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          tmem_ld32(acc + half * 128 + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float lo = __uint_as_float(r[2 * i]), hi = __uint_as_float(r[2 * i + 1]);
            if (RS) {
              const float2 sc = __ldg(reinterpret_cast<const float2 *>(scale + c * 32) + i);
              lo *= sc.x; hi *= sc.y;
            }
            head[c * 16 + i] = half2_bits(lo, hi);
          }
        }
        release();
        store_heads(args.heads, block, lane, head, grp, nt * 2 + half, row);
      } else {
        const int col = nt * TN + half * 128;
        const CUtensorMap *map_c = grp == 0 ? &map_c0 : grp == 1 ? &map_c1 : &map_c2;
        const float *scale = RS ? (grp == 0 ? args.row_scale[0] : grp == 1 ? args.row_scale[1] : args.row_scale[2]) + col : nullptr;
        // (the part before has been added: this warp's, to the same elements)
        if (MODE == 3 && z > 0 && elect_one()) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        uint32_t out[32];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          tmem_ld32(acc + half * 128 + c * 32, r);
          tmem_ld_wait();
          if (c == 3) release();
          if (RS) {
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const float4 sc = __ldg(reinterpret_cast<const float4 *>(scale + c * 32 + i));
              r[i] = __float_as_uint(__uint_as_float(r[i]) * sc.x);
              r[i + 1] = __float_as_uint(__uint_as_float(r[i + 1]) * sc.y);
              r[i + 2] = __float_as_uint(__uint_as_float(r[i + 2]) * sc.z);
              r[i + 3] = __float_as_uint(__uint_as_float(r[i + 3]) * sc.w);
            }
          }
          if (MODE == 1) {                 // 64 halves are a row of the block
#pragma unroll
            for (int i = 0; i < 16; ++i) out[(c & 1) * 16 + i] = half2_bits(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
            if (c & 1) {
              block_free();
              stage_row(block, lane, out);
              store_block(map_c, block, col + (c >> 1) * 64, row);
            }
          } else {                         // 32 floats
            block_free();
            stage_row(block, lane, r);
            store_block<MODE == 3>(map_c, block, col + c * 32, row);
          }
        }
      }
    }
    if (elect_one()) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // (and no block is read after the CTA has left)
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_leave();                         // neither CTA leaves while the other's copies, MMAs or arrivals reach into it (the
                                           // arrivals are waited for: a buffer's last read is not announced)
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

}  // namespace qmk_pair
#endif  // QMK_GEMM_PAIR_TCGEN05_CUH_
