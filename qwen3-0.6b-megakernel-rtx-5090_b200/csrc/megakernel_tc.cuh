// Fused single-sequence decode kernel whose row products run on the tensor cores (fp16 weights; FP8-E4M3 rows with
// QMK_TC_FP8).
//
// Same layer structure as megakernel_fused.cuh (four cross-CTA hand-overs per layer, integer all-reduced residual
// sums) and the same attention items, merge and exchange code.  What changes is how a CTA multiplies its weight
// rows with the activation vector.  Measured with cycle stamps, every phase of the CUDA-core version ran at 10-20
// cycles per instruction per warp: a phase executes once per layer, the layer's code (150 KB) does not stay in the
// 32 KB an SM can loop in at full fetch rate, and a 1024-wide fp16 row costs 68 instructions per warp (one
// convert and one FMA per weight).  So the goal here is few instructions:
//   * a 16-row x 16-input tile of weights is one ldmatrix.x4 and one mma.sync.m16n8k16; the activation vector is
//     the B operand with its fp32 value split over two fp16 columns (hi = fp16(x), lo = fp16((x - hi) * 2048); the
//     row result is acc_hi + acc_lo / 2048, exact products, fp32 accumulation, relative error ~2^-22), i.e. about
//     5 instructions per row instead of 68;
//   * RMSNorm is applied once per CTA (each thread normalises the three values it fetched, the hi/lo halves go to
//     shared memory) instead of once per warp;
//   * the producer is one loop over four-row chunks for every tensor.
// Ring chunk = four consecutive rows of one matrix, each copied by its own cp.async.bulk to a 2064-byte pitch (and
// chunks in odd slots start 64 bytes in), so that the eight row addresses of an ldmatrix phase fall into different
// banks (2048-byte pitch: 8-way conflict).  Cache chunks (16 K rows + 16 V rows) arrive as four tiled TMA boxes of
// 16 rows x 128 bytes with the 128-byte swizzle, which does the same for 256-byte rows with 4 copies instead of 32
// (one bulk copy per padded 256-byte row was tried: the copy engine takes ~30 cycles per copy whatever its size,
// and 480 copies per layer made the attention phase slower than the CUDA-core loop).
// CTAs own whole chunks: rows of the fused q|k|v matrix, of gate/up and of the LM head are split in units of four.
//
// FP8 rows (QMK_TC_FP8): the four hand-overs of a layer, not bytes, are most of the time, so what the format can gain
// over fp16 rows is the difference in bytes and no more - as long as its row products are not slower.  In the CUDA-core
// kernel they were (one convert and one FMA per weight): 724 us per token at a 1024-token context.
// Here the tiles take the fp16 form's few instructions: one ldmatrix.x4 brings 16 rows x 32 weights, eight
// cvt.rn.f16x2.e4m3x2 (exact) make the A operands of two MMAs of it.  A lane's register holds four consecutive inputs,
// an MMA fragment wants inputs 2q, 2q + 1 and 2q + 8, 2q + 9: the activations are stored in the permuted order instead
// (xf_offset).  A packed row is 1040 bytes in memory, which is a conflict-free pitch in shared memory too: a chunk
// is eight rows and ONE bulk copy (four 2 KB rows: four copies).  Row scales multiply the finished sums (they sit in
// the rows' trailers); the per-output scales of the K-major O / down copies travel as one more chunk of those phases.
// Measured after: 493 us per token (128 tokens from a 1024-token context; 416 with what is described below).  Against float64 the cache rows are nearer than the
// CUDA-core kernel's (later layers' values that round differently: 0.149 % and 0.167 %).

namespace QMK_NS {
#if QMK_MAX_SEQ == 1 && defined(QMK_TC_BUILD)

#ifndef QMK_TC_SEQS
#define QMK_TC_SEQS 1
#endif
constexpr int TC_SEQS = QMK_TC_SEQS;           // sequences a launch can carry (2 and 4: megakernel_tc_multi.cuh)
static_assert(TC_SEQS == 1 || TC_SEQS == 2 || TC_SEQS == 4, "two of the eight columns of an MMA per sequence");
// smallest grid: down slices of <= 32 rows, O slices of <= 88 whose merge is two quads of outputs per warp and one for the last two; four
// sequences: phases of at most as many chunks as their shorter ring has slots
constexpr int TC_MIN_CTAS = TC_SEQS == 4 ? 112 : 96;
static_assert(TC_MIN_CTAS >= FUSED_MIN_CTAS, "the tensor-core kernel shares the fused kernel's slice layout");
#ifdef QMK_TC_FP8
constexpr bool FP8_ROWS = true;
#else
constexpr bool FP8_ROWS = false;
#endif
constexpr int ROW_BYTES = FP8_ROWS ? FP8_PITCH : 2 * H;          // bytes of a weight row in memory (fp8: scale trailer included)
constexpr int ROW_PITCH = FP8_ROWS ? FP8_PITCH : 2 * H + 16;     // bytes between the rows of a chunk in shared memory
constexpr int CH_ROWS = FP8_ROWS ? 8 : 4;
constexpr int TILE_CH = 16 / CH_ROWS;          // chunks of a 16-row tile
constexpr int SCALE_CH = FP8_ROWS ? 1 : 0;     // an O / down slice is followed by a chunk of its 1024 output scales
// weight rows of fp16 chunks in odd slots start four 16-byte bank groups later (an ldmatrix phase reads two chunks)
constexpr int ODD_SLOT_SKEW = FP8_ROWS ? 0 : 64;
static_assert(SLOT_BYTES >= ODD_SLOT_SKEW + CH_ROWS * ROW_PITCH, "a slot holds a chunk of padded rows");
static_assert(ROW_PITCH % 128 == 16, "eight consecutive rows of a chunk fall into different bank groups");
static_assert(I % CH_ROWS == 0 && QS % CH_ROWS == 0 && KVS % CH_ROWS == 0, "a chunk lies in one matrix");
// The O projection.  A CTA that merged its own 14 of the 2048 attention outputs multiplied them into all 1024 outputs: 148
// contributions to every word of the sum x1, which a word's L2 slice adds one after the other, and six tiles of fixed-point
// conversions a warp.  Here O_GROUP = 4 CTAs (4 g .. 4 g + 3) merge the SAME slice of 52 to 56 attention outputs and each
// multiplies it into its quarter of the outputs: the bytes of the K-major matrix and the MMAs are what they were, contributions to a
// word are 37, a CTA's words 256.  What it costs is a merge of four times the words, whose loads take whole 32-byte sectors now.
// Mean step of five placements of the buffers, us, before / after (with wait_chunks): one fp16 sequence at 64 / 1024 / 4096 tokens 430 / 443 /
// 488 -> 432 / 443 / 478, one FP8 at 1024 428 -> 411, two fp16 at 512 531 -> 530, four at 1024 747 -> 733, four FP8 801 -> 728.
// Grids that are no multiple of four leave the last CTAs without a slice (see tc_grid).
using qmkp::O_GROUP;
using qmkp::O_COLS;
constexpr int O_TILES = O_COLS / 16;
constexpr int O_PITCH = (FP8_ROWS ? 1 : 2) * O_COLS + qmkp::O_PAD;   // conflict-free, in memory as in shared memory
constexpr int O_CH_ROWS = FP8_ROWS ? 32 : 16;                        // rows of a chunk: what one ldmatrix.x4 takes
constexpr int TILE_STEP = O_CH_ROWS / 16;                            // k-steps of an ldmatrix.x4
constexpr int O_MAX_QUADS = (QS / 4 + TC_MIN_CTAS / O_GROUP - 1) / (TC_MIN_CTAS / O_GROUP);   // a slice is whole quads of rows
constexpr int O_KPAIRS = (4 * O_MAX_QUADS + 31) / 32;
static_assert(TC_MIN_CTAS % O_GROUP == 0 && O_TILES <= 2 * CONS_WARPS, "at most two output tiles per warp");
static_assert(O_PITCH % 128 == 16, "eight consecutive rows of an O chunk fall into different bank groups");
static_assert(SLOT_BYTES >= ODD_SLOT_SKEW + O_CH_ROWS * O_PITCH, "a slot holds a chunk of O rows");
static_assert(O_MAX_QUADS <= 2 * CONS_WARPS - 2, "merge: two quads per warp, one for the last two");
static_assert(4 * O_MAX_QUADS <= D, "a slice lies in at most two query heads");
// Chunks that CTA `cta` of `ncta` reads of a layer: of the q|k|v rows, of its slice of the attention outputs (scales included; none
// past the last whole group), of the gate (= up, down) rows.  The counts of tc_setup, for the host: called there too, this
// function cost four FP8 sequences 0.7 % of a step (the code around it comes out differently).
constexpr int QKV_CHUNKS = QKV_ROWS / CH_ROWS, GU_CHUNKS = I / CH_ROWS;
struct LayerChunks { int nq, no, ng; };
constexpr LayerChunks layer_chunks(int ncta, int cta) {
  LayerChunks s = {};
  int a = 0, b = 0;
  split_rows(QKV_CHUNKS, ncta, cta, a, b); s.nq = b - a;
  split_rows(GU_CHUNKS, ncta, cta, a, b); s.ng = b - a;
  if (cta / O_GROUP < ncta / O_GROUP) {
    split_rows(QS / 4, ncta / O_GROUP, cta / O_GROUP, a, b);
    s.no = (4 * (b - a) + O_CH_ROWS - 1) / O_CH_ROWS + SCALE_CH;
  }
  return s;
}
// The norm vectors of layer L go into the buffer of layer L - 2 as soon as the ring has room for the last chunk of layer L - 1,
// i.e. when the chunk NSLOTS before it was handed back.  That must be a gate/up chunk of layer L - 2 or a later one: every warp is
// past its last use of L - 2's norm vectors (post_ln, before the gate/up rows) by then.  So layer L - 1 and what follows the O chunks
// of L - 2 have to be more chunks than the ring has slots, on every CTA; an attention item only adds to L - 1.  fp16 layers are long
// enough on all grids.  FP8 layers are not on a CTA without an O slice, and up to 160 CTAs on the others.
constexpr bool norms_outlive_use(int ncta) {
  for (int cta = 0; cta < ncta; ++cta) {
    const LayerChunks s = layer_chunks(ncta, cta);
    if (s.nq + s.no + 2 * (3 * s.ng + SCALE_CH) <= NSLOTS) return false;
  }
  return true;
}
// One sequence: the last two warps make the split weights of a merge, and take part in it where the slice has a quad for them (merge_o;
// with the test taken out there, 777 tokens took 0.6 % longer).  That is every slice up to 171 CTAs.
constexpr bool slices_reach_last_warp(int ncta) { return TC_SEQS > 1 || QS / 4 / (ncta / O_GROUP) >= CONS_WARPS; }
// The grid of this kernel where `ctas` CTAs are there: the largest that holds in both ways, 0 (another kernel runs) outside
// [TC_MIN_CTAS, TC_MAX_CTAS].
constexpr int TC_MAX_CTAS = FP8_ROWS ? 160 : MAX_CTAS;
inline int tc_grid(int ctas) {
  struct Table { short largest[TC_MAX_CTAS + 1]; };
  static const Table table = [] {
    Table t = {};
    for (int n = TC_MIN_CTAS; n <= TC_MAX_CTAS; ++n) t.largest[n] = norms_outlive_use(n) && slices_reach_last_warp(n) ? static_cast<short>(n) : t.largest[n - 1];
    return t;
  }();
  return ctas < 0 || ctas > TC_MAX_CTAS ? 0 : table.largest[ctas];
}
inline void tc_ring(int ncta, int cta, int (&out)[5]) {
  const LayerChunks s = layer_chunks(ncta, cta);
  const int counts[5] = {NSLOTS, s.nq, s.no, 2 * s.ng, s.ng + SCALE_CH};
  for (int i = 0; i < 5; ++i) out[i] = counts[i];
}
// (Grids without a CTA that has no O slice all hold for the norm vectors: at most three CTAs stay idle because of them.)
constexpr bool whole_groups_hold() {
  for (int n = TC_MIN_CTAS; n <= TC_MAX_CTAS; n += O_GROUP)
    if (!norms_outlive_use(n)) return false;
  return true;
}
static_assert(whole_groups_hold(), "norm vectors overwritten in use");
static_assert(SLOT_BYTES % 128 == 0 && NSLOTS % 2 == 0, "swizzled boxes need 128-byte aligned slots; slot parity = chunk parity");
static_assert(EMPTY_UNITS == 12, "1, 2, 3, 4, 6 or 12 warps share a chunk");
constexpr float LO_SCALE = 2048.0f, LO_INV = 1.0f / 2048.0f;
// Cache chunk in a slot: four boxes of 16 rows x 128 bytes: K dims 0..63, K dims 64..127, V dims 0..63, V dims 64..127.
// Within a box the 16-byte piece j of row r sits at piece j ^ ((address >> 7) & 7) (128-byte swizzle on address bits).
constexpr int KV_BOX = KV_ROWS_PER_CHUNK * 128;
constexpr int KV_V_OFF = 2 * KV_BOX;
constexpr int KV_PITCH = 2 * D + 16;           // pitch of the four query-operand rows (plain padded rows)
static_assert(SLOT_BYTES >= 4 * KV_BOX, "a slot holds the four boxes of a cache chunk");
static_assert(CH_ROWS * ((GU_CHUNKS + TC_MIN_CTAS - 1) / TC_MIN_CTAS) <= 32, "slice_cols takes two k-steps");
constexpr int KPAIRS = H / 32;                 // pairs of 16-input k-steps in a row
constexpr int ACT16_PITCH = 32 * O_KPAIRS + 8; // halves between the hi and the lo row of a slice's activations (other banks)
static_assert(32 * O_KPAIRS >= 64, "the gate/up phase writes 64");

// Extra shared memory of this kernel, behind the single-sequence layout.
// Normalised activations as the B operand of the row products, in MMA fragment order: 128 bytes per pair of
// k-steps (32 inputs) = [hi: 4 lanes x 16 bytes][lo: 4 lanes x 16 bytes]; the 16 bytes of lane kq are the halves
// {b0, b1} of the first k-step (inputs 2kq, 2kq+1, 2kq+8, 2kq+9) and of the second (the same + 16).  Lanes 0..7 of a
// warp fetch a pair's operand with ONE 128-byte wavefront (ldmatrix.x4 over plain hi / lo rows takes four; the row
// products are bound by shared-memory bandwidth, where that is a third of the traffic).
constexpr size_t OFF_XF = (SMEM_BYTES + 127) / 128 * 128;
constexpr int XF_PAIR = 128 * TC_SEQS;                         // bytes of a pair's operand: [sequence][hi, lo]
constexpr int PART_TASK = 16 * TC_SEQS;                        // floats of a tile task's partials
constexpr size_t OFF_PART = OFF_XF + 4 * H * TC_SEQS;          // fp32 tile partials [2][12 tasks][sequence][16 rows]
constexpr size_t OFF_QF = OFF_PART + 2 * 12 * PART_TASK * 4;   // fp16 query operand [4: q0 hi, q0 lo, q1 hi, q1 lo][128], rows at KV_PITCH
constexpr size_t OFF_ACT16 = OFF_QF + 4 * KV_PITCH;            // fp16 hi row, scaled-lo row of a slice's activations (merge / gate-up outputs), per sequence
constexpr size_t OFF_TCTAB = OFF_ACT16 + ((TC_SEQS * 2 * ACT16_PITCH * 2 + 15) / 16) * 16;
struct alignas(16) TileTask { int active, first, valid, p0, p1, units, pad0, pad1; };   // see build_tile_tasks
struct alignas(16) TcTab {
  int q0, nq, g0, ng, lm0, nlm;    // first chunk / chunks of this CTA: q|k|v rows, gate (= up) rows, LM-head rows
  int nkb_qkv, nkb_gu;             // warps per tile in the two row-product phases
  TileTask qkv[12], gu[12];        // each warp's tile task in those phases
  int e0, ne, no, oq;              // this CTA's slice of the attention outputs, its ring chunks, its quarter of the outputs
  int n0, n1, groups, early;       // outputs whose residuals this CTA adds; groups of CTAs that share a slice; see EARLY_ROWS
  int s_cap, seq, local, pad;      // several sequences: most splits of one, the sequence of this CTA's attention item, the item
};
// Several sequences: previous contributions to the residual sums [x1, x2][sequence][1024] (sequences 0 and 1 where the
// single-sequence kernel has its fp32 vectors; the pitch puts the four sequences of a fragment into different banks),
// residuals of the outputs this CTA owns, split weights of the merge, sums of squares, tokens, splits.
constexpr int PREV_PITCH = H + 8, RESID_PITCH = 12;
static_assert(4 * PREV_PITCH <= FF_SPLITW, "sequences 0 and 1 fit in front of the weight arrays");
constexpr size_t OFF_PREV2 = OFF_TCTAB + (sizeof(TcTab) + 15) / 16 * 16;
constexpr size_t OFF_RESID = OFF_PREV2 + (TC_SEQS > 2 ? 4 * PREV_PITCH * 4 : 0);
constexpr size_t OFF_SPLITW = OFF_RESID + 2 * TC_SEQS * RESID_PITCH * 4;
constexpr size_t OFF_REDM = OFF_SPLITW + 2 * 32 * 4;
constexpr size_t OFF_TOKENS = OFF_REDM + TC_SEQS * CONS_WARPS * 4;
constexpr size_t TC_SMEM_BYTES = TC_SEQS > 1 ? OFF_TOKENS + 2 * TC_SEQS * 4 : OFF_TCTAB + sizeof(TcTab);
static_assert(TC_SMEM_BYTES <= 232448, "over the 227 KB shared-memory limit of one CTA");
static_assert(OFF_XF % 128 == 0 && OFF_QF % 16 == 0, "operand rows are 16-byte aligned, a pair's 128 bytes one wavefront");
// Byte offset in the fragment-order array of input i's hi (lo = 0) or lo (1) half, sequence b.
__device__ __forceinline__ int xf_offset(int i, int lo, int b = 0) {
  const int kk = i & 31, rem = kk & 15, r8 = rem & 7;
  if (FP8_ROWS) return (i >> 5) * XF_PAIR + b * 128 + lo * 64 + (rem >> 2) * 16 + (kk >> 4) * 8 + (i & 3) * 2;   // lane kq: inputs 4 kq .. 4 kq + 3
  return (i >> 5) * XF_PAIR + b * 128 + lo * 64 + (r8 >> 1) * 16 + ((kk >> 4) * 4 + (rem >> 3) * 2 + (r8 & 1)) * 2;
}

__device__ __forceinline__ const TcTab *tctab(const Ctx &c) { return reinterpret_cast<const TcTab *>(c.smem + OFF_TCTAB); }
__device__ __forceinline__ float *tc_part(const Ctx &c) { return reinterpret_cast<float *>(c.smem + OFF_PART); }

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// d = A . B of a 16 x 16 tile, from a zero accumulator.
__device__ __forceinline__ void mma_16816_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// c += A . B in the tensor core.  It truncates the accumulator it is given after every step, always towards zero: a long
// chain of MMAs loses more of a sum than rounded fp32 adds of the same products do.  So a chain is at most four MMAs long (64
// products), and the chains are added up in registers.  Four MMAs of 11-bit operands take 0.75 * 2^-23 off their sum on
// average (one 0.32, eight 1.3; measured on random operands, the scatter around it is 0.5): the adds multiply by
// UNSHRINK_F16.  e4m3 weights (0.06 per MMA) are best off with one product per add.
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c += A . B in registers.
__device__ __forceinline__ void mma_add_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float d[4];
  mma_16816_zero(d, a, b0, b1);
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] += d[i];
}
constexpr float UNSHRINK_F16 = 1.0f + 1.0f / 8388608.0f;

__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// fp32 -> fp16 operand half: the value rounded to fp16 (lo = false) or its scaled remainder (lo = true)
__device__ __forceinline__ __half split_half(float x, bool lo) {
  const __half h = __float2half_rn(x);
  return lo ? __float2half_rn((x - __half2float(h)) * LO_SCALE) : h;
}
// Range: a half ends at 65504, the fp32 values do not.  Operands that may lie above are divided by a power of two first and
// the finished sums multiplied by it (both exact; 1 for everything a usual model holds, and then nothing changes):
//   * SwiGLU outputs: by the largest of the CTA's slice (at most 32 rows: one warp holds them all);
//   * rotated queries: by the largest of the head;
//   * RMS-normalised activations, which stay below 32 x |norm weight|: by 64 where a weight of the vector exceeds 2040.
// Attention outputs need none: they are averages of fp16 cache rows.
constexpr int M_XSCALE = 24, M_QSCALE = 26, M_ASCALE = 20;   // words of F_MISC: activations, query heads [2], SwiGLU slice [sequence]
constexpr float NORM_W_LIMIT = 2040.0f, NORM_DOWN = 1.0f / 64.0f, NORM_UP = 64.0f;
// Exponent k >= 0 with |v| * 2^-k < 2^15 in every lane of the warp (infinities and NaN stay what they are).
__device__ __forceinline__ uint32_t operand_exponent(float v) {
  const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(v) & 0x7fffffffu) >> 23;
  return top > 141u ? top - 141u : 0u;
}
__device__ __forceinline__ float exp2_down(uint32_t k) { return __uint_as_float((127u - k) << 23); }
__device__ __forceinline__ float exp2_up(uint32_t k) { return __uint_as_float((127u + k) << 23); }
__device__ __forceinline__ uint32_t pack_half2(__half a, __half b) {
  return static_cast<uint32_t>(__half_as_ushort(a)) | (static_cast<uint32_t>(__half_as_ushort(b)) << 16);
}

// Activation operand of k-step pair p for this lane: column n = lane / 4 of B is the hi (even n) or the lo vector of
// sequence n / 2, or zero; {x, y} = fragments of the first k-step, {z, w} of the second.
__device__ __forceinline__ uint4 b_pair(const Ctx &c, int p) {
  return c.lane < 8 * TC_SEQS ? *reinterpret_cast<const uint4 *>(c.smem + OFF_XF + p * XF_PAIR + c.lane * 16) : make_uint4(0u, 0u, 0u, 0u);
}

// Shared-window address of row 0 of the weight chunk with ring index idx.
__device__ __forceinline__ uint32_t weight_rows(const Ctx &c, uint32_t idx) {
  return smem_u32(c.slot(idx)) + (idx & 1u) * ODD_SLOT_SKEW;
}
__device__ __forceinline__ void tma_box_2d(uint32_t dst, const void *map, int c0, int c1, uint64_t *bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar)) : "memory");
}

// A register of four e4m3 values as two fp16 pairs.
__device__ __forceinline__ void e4m3x4_half2x2(uint32_t four, uint32_t &first, uint32_t &second) {
  asm("{\n\t.reg .b16 l, u;\n\tmov.b32 {l, u}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, l;\n\tcvt.rn.f16x2.e4m3x2 %1, u;\n\t}"
      : "=r"(first), "=r"(second) : "r"(four));
}

// Waits for ring chunks [first, first + n), 1 <= n <= 32.  Lanes past the last one ask for it too, so that the warp asks once and
// votes without branching (a diverging wait took 370 cycles of chunks that were there, of an LM head tile with FP8 rows a sixth:
// 51.5 -> 44 us).  The vote orders the copied bytes before every lane's loads.
__device__ __forceinline__ bool wait_chunks(const Params &P, const Ctx &c, uint32_t first, int n) {
  const uint32_t idx = first + static_cast<uint32_t>(min(c.lane, n - 1));
  uint64_t *bar = c.full(idx % NSLOTS);
  const uint32_t parity = (idx / NSLOTS) & 1u;
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return __all_sync(0xffffffffu, mbar_wait(P, c, bar, parity, WHERE_FULL, false));
}

// One warp: rows of the 16-row tile that starts at ring chunk `first` (valid rows <= 16), k-step pairs [p0, p1).
// Operands come in front of the products they feed.  An MMA takes 8.5 cycles of a sub-partition (stand-alone, 4 to 12 warps;
// 21 from one to the next that depends on it), a ldmatrix 48 cycles until its data can be used and four of the SM's
// shared-memory port: asked for one after the other, in between the MMAs, a tile waited for its operands (26 cycles per MMA).
// With the attention's and the slices' operands ahead too: two fp16 sequences 570 -> 549 us per step, four 796 -> 780 (1024
// tokens), one 490 -> 486, one with FP8 rows 491 -> 482.  What bounds the phase now is the port: 48 rows of gate and up are
// 768 cycles of it.
// Leaves the 16 row sums of that k range in part[0..15] (sequence b: part[16 b..]) and hands the tile's chunks back with `units` each.
// Lanes 0..3 each wait for one of the tile's chunks (the vote that follows orders the copied bytes before every
// lane's loads).
struct RowTile { uint32_t first, a_addr; int valid, p0, p1, units; bool ok; };
__device__ __forceinline__ RowTile prepare_tile(const Params &P, const Ctx &c, uint32_t first, int valid_rows, int p0, int p1, int units) {
  RowTile r;
  r.first = first;
  r.valid = valid_rows;
  r.p0 = p0;
  r.p1 = p1;
  r.units = units;
  r.ok = wait_chunks(P, c, first, (valid_rows + CH_ROWS - 1) / CH_ROWS);
  int lr = (c.lane & 7) + ((c.lane >> 3) & 1) * 8;      // tile row whose address this lane supplies
  if (lr >= valid_rows) lr = 0;                         // rows past the end repeat row 0 (their sums are not used)
  r.a_addr = weight_rows(c, first + static_cast<uint32_t>(lr / CH_ROWS)) + (lr % CH_ROWS) * ROW_PITCH + (c.lane >> 4) * 16;
  return r;
}
__device__ __forceinline__ void run_tile(const Ctx &c, const RowTile &r, float *part, int fslot = 70) {
  const bool ok = r.ok;
  const uint32_t first = r.first, a_addr = r.a_addr;
  const int valid_rows = r.valid, p0 = r.p0, p1 = r.p1, units = r.units, nch = (valid_rows + CH_ROWS - 1) / CH_ROWS;
  float sum[4] = {0.f, 0.f, 0.f, 0.f};
  if (ok && FP8_ROWS) {   // r: rows 0..7 / 8..15 x inputs 0..15, then inputs 16..31; four consecutive inputs per lane
    float odd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
    for (int p = p0; p < p1; ++p) {
      uint32_t a0[4], a1[4], r[4];
      const uint4 b = b_pair(c, p);
      ldsm_x4(a_addr + p * 32, r);
      e4m3x4_half2x2(r[0], a0[0], a0[2]);
      e4m3x4_half2x2(r[1], a0[1], a0[3]);
      e4m3x4_half2x2(r[2], a1[0], a1[2]);
      e4m3x4_half2x2(r[3], a1[1], a1[3]);
      mma_add_16816(sum, a0, b.x, b.y);
      mma_add_16816(odd, a1, b.z, b.w);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[i] += odd[i];
  } else if (ok) {
#pragma unroll 1
    for (int p = p0; p < p1; p += 2) {     // all operands of a chain before its first MMA
      uint32_t a[4][4];
      const uint4 b0 = b_pair(c, p), b1 = b_pair(c, p + 1);
#pragma unroll
      for (int u = 0; u < 4; ++u) ldsm_x4(a_addr + p * 64 + u * 32, a[u]);
      float acc[4];
      mma_16816_zero(acc, a[0], b0.x, b0.y);
      mma_16816(acc, a[1], b0.z, b0.w);
      mma_16816(acc, a[2], b1.x, b1.y);
      mma_16816(acc, a[3], b1.z, b1.w);
#pragma unroll
      for (int i = 0; i < 4; ++i) sum[i] = fmaf(acc[i], UNSHRINK_F16, sum[i]);
    }
  }
  QMK_FINE(fslot + 5);
  float sc_top = 1.f, sc_bot = 1.f;                     // row scales, read before the rows are handed back
  if (FP8_ROWS && (c.lane & 3) < TC_SEQS) {
    const int r0 = c.lane >> 2, r1 = r0 + 8;
    if (r0 < valid_rows) sc_top = *reinterpret_cast<const float *>(c.slot(first + static_cast<uint32_t>(r0 / CH_ROWS)) + (r0 % CH_ROWS) * ROW_PITCH + H);
    if (r1 < valid_rows) sc_bot = *reinterpret_cast<const float *>(c.slot(first + static_cast<uint32_t>(r1 / CH_ROWS)) + (r1 % CH_ROWS) * ROW_PITCH + H);
  }
  __syncwarp();
  if (c.lane < nch) mbar_arrive_n(c.empty((first + static_cast<uint32_t>(c.lane)) % NSLOTS), static_cast<uint32_t>(units));
  if ((c.lane & 3) < TC_SEQS) {   // quad b of a fragment: the hi and lo columns of sequence b
    part += (c.lane & 3) * 16;
    part[c.lane >> 2] = fmaf(sum[1], LO_INV, sum[0]) * sc_top;
    part[(c.lane >> 2) + 8] = fmaf(sum[3], LO_INV, sum[2]) * sc_bot;
  }
}

// First k-step pair of part i of n of a row.  fp16: whole chains of four MMAs (two pairs), so that tile_task has no odd pair to
// look out for (the branches cost the kernel 120 bytes of spills).
__device__ __forceinline__ int k_split(int i, int n) { return FP8_ROWS ? KPAIRS * i / n : KPAIRS / 2 * i / n * 2; }

// Per-warp work of a layer phase, fixed for the launch (computed once: the integer divisions behind it cost more
// than the MMAs).  Phase rows = `groups` runs of `nch` consecutive chunks (q|k|v: one run; gate/up: the gate rows'
// chunks, then the up rows'); tiles of 16 rows; when there are fewer tiles than warps, nkb warps share a tile's
// 1024 inputs.  Grids of at least FUSED_MIN_CTAS CTAs have at most 6 tiles per phase: one task per warp.
// fp16 rows: the tiles run on from the gate into the up rows (148 CTAs: 40 to 48 rows are three tiles, where the gate and
// the up rows by themselves were two each, the second of them half empty; shared memory hands out a padded tile like a full one):
// 523 / 535 / 568 -> 518 / 531 / 563 us per token at 64 / 1024 / 4096-token contexts (both with full lines of sums, see
// RED_GROUP).  fp8 rows gained nothing at 1024 and lost 1 % at 64 and stay apart (their row conversions weigh more than the
// MMAs).
constexpr bool GU_ONE_RUN = !FP8_ROWS;
__device__ inline void build_tile_tasks(TileTask *tasks, int *nkb_out, int groups, int nch) {
  const int tpg = (nch + TILE_CH - 1) / TILE_CH, T = groups * tpg;
  const int nkb = T >= CONS_WARPS ? 1 : CONS_WARPS / T;   // 12, 6, 4, 3, 2, 2, 1: divides EMPTY_UNITS
  *nkb_out = nkb;
  for (int w = 0; w < CONS_WARPS; ++w) {
    TileTask &t = tasks[w];
    t.active = w < T * nkb ? 1 : 0;
    const int tile = w / nkb, kb = w - tile * nkb, grp = tile / tpg, tt = tile - grp * tpg;
    t.first = grp * nch + tt * TILE_CH;
    t.valid = min(16, (nch - tt * TILE_CH) * CH_ROWS);
    t.p0 = k_split(kb, nkb);
    t.p1 = k_split(kb + 1, nkb);
    t.units = EMPTY_UNITS / nkb;
    t.pad0 = t.pad1 = 0;
  }
}
// Row of the gate/up phase's tiles that holds the up row of gate row r.
__device__ __forceinline__ int up_row(int nch, int r) { return r + (GU_ONE_RUN ? nch * CH_ROWS : (nch + TILE_CH - 1) / TILE_CH * 16); }
// FP8 rows, several sequences: what a phase's first MMA waits for besides the activations - the task, the chunks' arrival, addresses -
// is done in front of the wait for these, which is long there (sums drain for longer): two / three / four sequences at 1024 tokens
// 560 / 633 / 710 -> 553 / 607 / 680 us per step.  One sequence 412 / 414; fp16 rows, whose phases take most of the ring, lose 4 %.
// All warps then wait for their chunks before the first one hands any back: the phase and what a group of eight issues
// with its last chunk must fit into the ring (TcTab::early).  The slots were last used two phases before, so the parity is that
// of this use (every warp waits for all chunks of an O or down phase, and the row phases end with a barrier).
constexpr bool EARLY_ROWS = FP8_ROWS && TC_SEQS > 1;
__device__ __forceinline__ RowTile prepare_rows(const Params &P, const Ctx &c, const TileTask *tasks) {
  const int4 a = reinterpret_cast<const int4 *>(tasks + c.warp)[0], b = reinterpret_cast<const int4 *>(tasks + c.warp)[1];
  // a = {active, first, valid, p0}, b = {p1, units, -, -}
  if (a.x) return prepare_tile(P, c, c.chunk + static_cast<uint32_t>(a.y), a.z, a.w, b.x, b.y);
  RowTile none = {};
  return none;
}
__device__ __forceinline__ void run_rows(const Ctx &c, const RowTile &rows, int fslot) {
  if (rows.valid > 0) run_tile(c, rows, tc_part(c) + c.warp * PART_TASK, fslot);
}

// The phases are inlined into the kernel's layer loop.  As functions of their own they cost a call and its register moves (160
// cycles, ten times a layer) and read every launch parameter through memory; inlined, parameters are constant-bank operands and
// a phase keeps 128 registers for itself: a step of one fp16 sequence at 64 / 1024 / 4096 tokens 486 / 491 / 518 -> 433 / 446 / 492
// us, one with FP8 rows at 1024 491 -> 430, two fp16 at 512 568 -> 525, four at 1024 795 -> 748, four FP8 820 -> 781.  (The two call sites of slice_cols and red_wait_norm
// do not hurt: a phase repeated at once, its code hot, takes as long as the first time.)
#if QMK_TC_SEQS == 1
// q|k|v rows of this CTA -> exchange words (megakernel_5090.cu:251-302).
__device__ __forceinline__ uint32_t qkv_phase(const Params &P, Ctx c, uint32_t tag) {
  const TcTab *t = tctab(c);
  const int nch = t->nq, nkb = t->nkb_qkv;
  QMK_FINE(0);
  run_rows(c, prepare_rows(P, c, t->qkv), 0);
  QMK_FINE(2);
  cons_sync();
  if (c.tid < nch * CH_ROWS) {
    const int r = c.tid;
    const float *p = tc_part(c) + (r >> 4) * nkb * 16 + (r & 15);
    float v = 0.f;
#pragma unroll
    for (int kb = 0; kb < CONS_WARPS; ++kb)
      if (kb < nkb) v += p[kb * 16];
    ll_store(P.ll + LL_QKV + t->q0 * CH_ROWS + r, v * c.f(F_MISC)[M_XSCALE], tag);
  }
  QMK_FINE(4);
  return c.chunk + static_cast<uint32_t>(nch);
}

// gate/up rows of this CTA -> silu(gate) * up in shared memory (megakernel_5090.cu:653-685, SiLU in fp32).
__device__ __forceinline__ uint32_t gateup_phase(const Params &P, Ctx c) {
  const TcTab *t = tctab(c);
  const int nch = t->ng, nkb = t->nkb_gu;
  QMK_FINE(10);
  run_rows(c, prepare_rows(P, c, t->gu), 10);
  QMK_FINE(12);
  cons_sync();
  if (c.warp < 2) {          // warp 0 holds the slice; rows past it multiply stale bytes: zero activations
    const int r = c.tid, ru = up_row(nch, r);
    float a = 0.f;
    if (r < nch * CH_ROWS) {
      const float *pg = tc_part(c) + (r >> 4) * nkb * 16 + (r & 15);
      const float *pu = tc_part(c) + (ru >> 4) * nkb * 16 + (ru & 15);
      float g = 0.f, u = 0.f;
#pragma unroll
      for (int kb = 0; kb < CONS_WARPS; ++kb)
        if (kb < nkb) { g += pg[kb * 16]; u += pu[kb * 16]; }
      const float up = c.f(F_MISC)[M_XSCALE];
      g *= up;
      a = g / (1.0f + expf(-g)) * (u * up);
    }
    const uint32_t k = operand_exponent(a);
    if (c.tid == 0) c.f(F_MISC)[M_ASCALE] = exp2_up(k);
    a *= exp2_down(k);
    __half *act16 = reinterpret_cast<__half *>(c.smem + OFF_ACT16);
    act16[r] = split_half(a, false);
    act16[ACT16_PITCH + r] = split_half(a, true);
  }
  QMK_FINE(14);
  return c.chunk + static_cast<uint32_t>(2 * nch);
}

#endif  // QMK_TC_SEQS == 1

// The exchange area of the sequence this CTA attends for.
__device__ __forceinline__ unsigned long long *tc_ll(const Params &P, const Ctx &c) {
  return TC_SEQS == 1 ? P.ll : P.ll + static_cast<size_t>(tctab(c)->seq) * LL_WORDS;
}
// attn_item (megakernel_device.cuh); several sequences: of the sequence the CTA belongs to, with at most s_cap splits.
__device__ __forceinline__ AttnItem tc_item(const Params &P, const Ctx &c, int pos) {
  if (TC_SEQS == 1) return attn_item(P, c, 0, 1, CONS_WARPS, pos);
  const int local = tctab(c)->local;
  AttnItem it;
  it.S = max(1, min(pos / max(1, P.split_len), tctab(c)->s_cap));
  it.active = local < NKV * it.S;
  it.g = local % NKV;
  it.s = local / NKV;
  it.p0 = it.active ? static_cast<int>(static_cast<unsigned>(pos * it.s) / static_cast<unsigned>(it.S)) : 0;
  it.p1 = it.active ? static_cast<int>(static_cast<unsigned>(pos * (it.s + 1)) / static_cast<unsigned>(it.S)) : 0;
  it.rpc = KV_ROWS_PER_CHUNK;
  it.nchunks = (it.p1 - it.p0 + KV_ROWS_PER_CHUNK - 1) / KV_ROWS_PER_CHUNK;
  return it;
}

// Attention work item (kv head g, split s) of this CTA on the tensor cores.  Same contract as attention_phase
// (megakernel_device.cuh): old cache rows [p0, p1) arrive as ring chunks of 16 K rows + 16 V rows (272-byte pitch),
// warp w takes chunks w, w + 12, ...; the last split also normalises, rotates and stores the new K/V row and folds
// it in; unnormalised partials (acc[128], max, sum per query head) are published for the merge.
// Per chunk: scores = K[16 x 128] . q[128 x 4] (columns: head 0 hi/lo, head 1 hi/lo of the fp32 query) as 8 MMAs,
// online softmax on the accumulator fragments (log2 domain), then out[128 x 4] += V^T[128 x 16] . p[16 x 4] as 8
// MMAs with V read through ldmatrix.trans and p split into hi/lo fp16 columns like q: ~75 instructions per 16
// rows where the CUDA-core loop needs ~480.
__device__ __forceinline__ uint32_t attention_tc(const Params &P, Ctx c, const __half *nv, int layer, int pos, uint32_t tag) {
  const AttnItem it = tc_item(P, c, pos);
  float *s_q = c.f(F_Q), *s_knew = c.f(F_KNEW), *s_vnew = c.f(F_VNEW), *s_wpart = c.f(F_WPART), *s_misc = c.f(F_MISC);
  const float *s_cs = c.f(F_CS);
  const unsigned long long *qkv = c.llr + LL_QKV;
  if (!it.active) return c.chunk;
  const int S = it.S, g = it.g, s = it.s;
  const bool owner = (s == S - 1);
  const int nrows_item = it.p1 - it.p0;
  const size_t head_base = (static_cast<size_t>(layer) * NKV + g) * static_cast<size_t>(P.max_seq_len) * D;

  QMK_FINE(60);
  // (1) head preparation: warps 0,1 = the two query heads; owner: warp 2 = K, warp 3 = V
  if (c.warp < 2 || (owner && c.warp < 4)) {
    const int w = c.warp, lane = c.lane;
    const unsigned long long *src = (w < 2) ? qkv + (2 * g + w) * D : (w == 2) ? qkv + QS + g * D : qkv + QS + KVS + g * D;
    float nw[4] = {1.f, 1.f, 1.f, 1.f};
    if (w < 3) {
      const __half *nwp = nv + ((w < 2) ? NB_QNORM : NB_KNORM);   // shared memory
#pragma unroll
      for (int i = 0; i < 4; ++i) nw[i] = __half2float(nwp[lane + 32 * i]);
    }
    float v[4];
    {
      const unsigned long long *wp[4] = {src + lane, src + lane + 32, src + lane + 64, src + lane + 96};
      // (a sentinel poll first, as in the residual-sum wait, costs its extra round trip here: 4.05 -> 4.34 us)
      ll_wait_many<4>(P, c, wp, 0xfu, tag, v);
    }
    if (w < 3) {
      float ss = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
      ss = warp_sum(ss);
      const float rstd = 1.0f / sqrtf(ss * (1.0f / D) + RMS_EPS);
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = v[i] * rstd * nw[i];
      // rotate-half: element i pairs with i+64 and both use frequency i (i < 64)
      const float c0 = s_cs[lane], s0 = s_cs[64 + lane];
      const float c1 = s_cs[lane + 32], s1 = s_cs[64 + lane + 32];
      const float r0 = v[0] * c0 - v[2] * s0, r2 = v[0] * s0 + v[2] * c0;
      const float r1 = v[1] * c1 - v[3] * s1, r3 = v[1] * s1 + v[3] * c1;
      v[0] = r0; v[1] = r1; v[2] = r2; v[3] = r3;
    }
    if (w < 2) {
      __half *qh = reinterpret_cast<__half *>(c.smem + OFF_QF + (2 * w) * KV_PITCH);
      __half *ql = reinterpret_cast<__half *>(c.smem + OFF_QF + (2 * w + 1) * KV_PITCH);
      const uint32_t k = operand_exponent(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
      if (lane == 0) s_misc[M_QSCALE + w] = exp2_up(k);
      const float down = exp2_down(k);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        s_q[w * D + lane + 32 * i] = v[i];
        qh[lane + 32 * i] = split_half(v[i] * down, false);
        ql[lane + 32 * i] = split_half(v[i] * down, true);
      }
    } else {
      // the new row takes part in this step's attention as the fp16 value the cache will hold
      float *snew = (w == 2) ? s_knew : s_vnew;
#pragma unroll
      for (int i = 0; i < 4; ++i) snew[lane + 32 * i] = __half2float(__float2half_rn(v[i]));
    }
  }
  QMK_FINE(61);
  cons_sync();
  QMK_FINE(62);

  const float sc_log2 = P.attn_scale * 1.4426950408889634f;
  if (owner && c.warp < 2) {   // score of the new row
    float d = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) d = fmaf(s_q[c.warp * D + c.lane + 32 * i], s_knew[c.lane + 32 * i], d);
    d = warp_sum(d);
    if (c.lane == 0) s_misc[c.warp] = d * sc_log2;
  }

  // (2) stream the old rows
  const int quad = c.lane & 3, rowq = c.lane >> 2;     // accumulator fragment: rows rowq, rowq + 8; columns 2 quad, 2 quad + 1
  const float sc_quad = sc_log2 * s_misc[M_QSCALE + (quad & 1)];
  float acc[8][4];
#pragma unroll
  for (int t = 0; t < 8; ++t) { acc[t][0] = 0.f; acc[t][1] = 0.f; acc[t][2] = 0.f; acc[t][3] = 0.f; }
  float m = -INFINITY, l = 0.f;                        // running max / sum of this lane's head (quad = head, quads 2, 3 idle)
  const uint32_t q_addr = smem_u32(c.smem + OFF_QF + (c.lane & 3) * KV_PITCH) + (c.lane >> 3) * 16;   // rows 4..7 repeat 0..3
  const int lr = (c.lane & 7) + ((c.lane >> 3) & 1) * 8;
  const bool pass_gate = it.nchunks > NSLOTS;   // see attention_phase
#pragma unroll 1
  for (int j0 = 0; j0 < it.nchunks; j0 += CONS_WARPS) {
    const int j = j0 + c.warp;
    if (j >= it.nchunks) {
      if (pass_gate) cons_sync();
      continue;
    }
    const uint32_t idx = c.chunk + static_cast<uint32_t>(j);
    const int nrow = min(KV_ROWS_PER_CHUNK, nrows_item - j * KV_ROWS_PER_CHUNK);
    if (__all_sync(0xffffffffu, mbar_wait(P, c, c.full(idx % NSLOTS), (idx / NSLOTS) & 1u, WHERE_FULL, false))) {
      const uint32_t base = smem_u32(c.slot(idx));
      if (nrow < KV_ROWS_PER_CHUNK) {   // rows past the item's end hold other rows of the cache: p = 0 for them, but 0 x NaN must not happen
        unsigned char *vrows = c.slot(idx) + KV_V_OFF;
        const int pieces = (KV_ROWS_PER_CHUNK - nrow) * 8;      // 16-byte pieces per box
        for (int i = c.lane; i < 2 * pieces; i += 32)
          reinterpret_cast<uint4 *>(vrows + (i >= pieces ? KV_BOX : 0) + nrow * 128)[i >= pieces ? i - pieces : i] = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // these stores precede the slot's next tiled copy
        __syncwarp();
      }
      float sc[4] = {0.f, 0.f, 0.f, 0.f}, sc2[4] = {0.f, 0.f, 0.f, 0.f};   // two chains of four dependent MMAs instead of one of eight
      const uint32_t k_row = base + lr * 128;                        // this lane's K row in box 0
      const uint32_t k_xor = ((k_row >> 7) & 7u) << 4;               // swizzle of that row (the same in box 1: boxes are 2048 bytes)
      const uint32_t k_off = (c.lane >> 4) * 16;
#pragma unroll
      for (int h = 0; h < 2; ++h) {       // a half's operands (the query's too: kept across chunks they cost 16 registers behind the softmax), then its products
        uint32_t qf[2][4], ka[2][2][4];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          ldsm_x4(q_addr + (2 * h + p) * 64, qf[p]);
          ldsm_x4(k_row + h * KV_BOX + ((p * 64 + k_off) ^ k_xor), ka[p][0]);
          ldsm_x4(k_row + h * KV_BOX + ((p * 64 + 32 + k_off) ^ k_xor), ka[p][1]);
        }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          mma_16816(sc, ka[p][0], qf[p][0], qf[p][1]);
          mma_16816(sc2, ka[p][1], qf[p][2], qf[p][3]);
        }
      }
      // V operand of the first half: requested here, needed behind the softmax
      const uint32_t v_row = base + KV_V_OFF + ((c.lane & 7) + 8 * (c.lane >> 4)) * 128;
      const uint32_t v_xor = ((v_row >> 7) & 7u) << 4;
      const uint32_t v_off = ((c.lane >> 3) & 1) * 16;
      uint32_t va[4][4];
#pragma unroll
      for (int t = 0; t < 4; ++t) ldsm_x4_trans(v_row + ((t * 32 + v_off) ^ v_xor), va[t]);
      float s_top = fmaf(sc[0] + sc2[0], UNSHRINK_F16, (sc[1] + sc2[1]) * LO_INV) * sc_quad,
            s_bot = fmaf(sc[2] + sc2[2], UNSHRINK_F16, (sc[3] + sc2[3]) * LO_INV) * sc_quad;
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
      const int n = c.lane >> 2, src_lane = (2 * quad) * 4 + ((n >> 1) & 1);
      const float pta = __shfl_sync(0xffffffffu, p_top, src_lane), ptb = __shfl_sync(0xffffffffu, p_top, src_lane + 4);
      const float pba = __shfl_sync(0xffffffffu, p_bot, src_lane), pbb = __shfl_sync(0xffffffffu, p_bot, src_lane + 4);
      uint32_t b0 = 0u, b1 = 0u;
      if (n < 4) {
        const bool lo = (n & 1) != 0;
        b0 = pack_half2(split_half(pta, lo), split_half(ptb, lo));
        b1 = pack_half2(split_half(pba, lo), split_half(pbb, lo));
      }
#pragma unroll
      for (int t0 = 0; t0 < 8; t0 += 4) {   // four products in flight, then their adds
        float d[4][4];
#pragma unroll
        for (int t = 0; t < 4; ++t) mma_16816_zero(d[t], va[t], b0, b1);
        if (t0 == 0) {
#pragma unroll
          for (int t = 0; t < 4; ++t) ldsm_x4_trans(v_row + KV_BOX + ((t * 32 + v_off) ^ v_xor), va[t]);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[t0 + t][i] += d[t][i];
      }
    }
    __syncwarp();
    if (c.lane == 0) mbar_arrive_n(c.empty(idx % NSLOTS), EMPTY_UNITS);
    if (pass_gate) cons_sync();
  }
  c.chunk += static_cast<uint32_t>(it.nchunks);
  QMK_FINE(63);
  // (3) this warp's partial state -> shared memory: lanes of quad h hold head h (columns hi, lo)
  if (quad < 2) {
    float *wp = s_wpart + (c.warp * 2 + quad) * PART_STRIDE;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      wp[t * 16 + rowq] = fmaf(acc[t][1], LO_INV, acc[t][0]);
      wp[t * 16 + rowq + 8] = fmaf(acc[t][3], LO_INV, acc[t][2]);
    }
    if (rowq == 0) { wp[D] = m; wp[D + 1] = l; }
  }
  QMK_FINE(64);
  cons_sync();
  QMK_FINE(65);
  // (4) merge the warps (+ the new row).  First the 2 x 13 weights exp2(max_w - max) and the head's (max, sum), by
  // warps 0 and 1 (one head each, lane = contributing warp, lane 12 = the new row); then every (head, dim) is a
  // weighted sum of 13 independent loads (a running max + rescale per thread took 1180 cycles here).
  // (an array of its own: the merge that follows writes its split weights without a barrier in between, and its last two
  // warps may get there while other warps of a CTA that is late still read these)
  float *s_scale = c.f(FF_ATTNW);                        // [2][16]
  if (c.warp < 2) {
    const int h = c.warp;
    float mw = -INFINITY, lw = 0.f;
    if (c.lane < CONS_WARPS) {
      mw = s_wpart[(c.lane * 2 + h) * PART_STRIDE + D];
      lw = s_wpart[(c.lane * 2 + h) * PART_STRIDE + D + 1];
    } else if (c.lane == CONS_WARPS && owner) {
      mw = s_misc[h];
      lw = 1.f;
    }
    const float M = warp_max(mw);
    const float scw = (mw == -INFINITY) ? 0.f : exp2f(mw - M);
    const float L = warp_sum(lw * scw);
    if (c.lane < 16) s_scale[h * 16 + c.lane] = scw;
    if (c.lane == 0) {
      unsigned long long *part = tc_ll(P, c) + LL_PART + static_cast<size_t>((2 * g + h) * MAX_SPLITS + s) * PART_STRIDE;
      ll_store(part + D, M, tag);
      ll_store(part + D + 1, L, tag);
    }
  }
  cons_sync();
  if (c.tid < 2 * D) {
    const int h = c.tid >> 7, d = c.tid & (D - 1);
    // (not a zero weight: on a CTA that does not own the new row s_vnew holds what an earlier kernel left in shared memory,
    // and 0 x NaN is NaN - which the integer sums then took for 0, a wrong first layer after some prefills)
    float A = owner ? s_vnew[d] * s_scale[h * 16 + CONS_WARPS] : 0.f;
#pragma unroll
    for (int w = 0; w < CONS_WARPS; ++w) A = fmaf(s_wpart[(w * 2 + h) * PART_STRIDE + d], s_scale[h * 16 + w], A);
    ll_store(tc_ll(P, c) + LL_PART + static_cast<size_t>((2 * g + h) * MAX_SPLITS + s) * PART_STRIDE + d, A, tag);
  }
  QMK_FINE(66);
  // New K,V row -> cache (megakernel_5090.cu:392-397), off the critical path.  The fence orders the row before the
  // exchange words this CTA publishes later; readers fence once per step.
  if (owner && (c.warp == 2 || c.warp == 3)) {
    __half *const k_cache = TC_SEQS == 1 ? P.k_cache : per_seq(P.k_caches, tctab(c)->seq);
    __half *const v_cache = TC_SEQS == 1 ? P.v_cache : per_seq(P.v_caches, tctab(c)->seq);
    __half *cache = ((c.warp == 2) ? k_cache : v_cache) + head_base + static_cast<size_t>(pos) * D;
    const float *snew = (c.warp == 2) ? s_knew : s_vnew;
#pragma unroll
    for (int i = 0; i < 4; ++i) cache[c.lane + 32 * i] = __float2half_rn(snew[c.lane + 32 * i]);
    __threadfence();
  }
  return c.chunk;
}

#if QMK_TC_SEQS == 1
// 1 / sqrt(mean of squares + eps) over the 1024 values whose squares the consumer threads hold in `ss`; one barrier, which
// also tells whether `big` holds in any thread.  (rsqrt.approx: 2 ulp; the sum's order is fixed.)
__device__ __forceinline__ float block_rstd(const Ctx &c, float ss, bool &big) {
  ss = warp_sum(ss);
  float *red = c.f(F_RED);
  if (c.lane == 0) red[c.warp] = ss;
  big = cons_any(big);
  const float4 r0 = reinterpret_cast<const float4 *>(red)[0], r1 = reinterpret_cast<const float4 *>(red)[1],
               r2 = reinterpret_cast<const float4 *>(red)[2];
  const float tot = (((r0.x + r0.y) + (r0.z + r0.w)) + ((r1.x + r1.y) + (r1.z + r1.w))) + ((r2.x + r2.y) + (r2.z + r2.w));
  return rsqrtf(tot * (1.0f / H) + RMS_EPS);
}

// fp32 vector value -> residual stream (fp32) and the hi/lo fp16 halves of its RMS-normalised form times `down`.
__device__ __forceinline__ void store_normalised(const Ctx &c, int n, float v, float rstd, float w, float down, float *dst) {
  dst[n] = v;
  const float xn = v * rstd * w * down;
  *reinterpret_cast<__half *>(c.smem + OFF_XF + xf_offset(n, 0)) = split_half(xn, false);
  *reinterpret_cast<__half *>(c.smem + OFF_XF + xf_offset(n, 1)) = split_half(xn, true);
}

// Waits until use number `use` (1-based) of a sum is complete (see megakernel_fused.cuh), writes the 1024 values
// to shared memory (which = 0: x1; 1: x, the next input) and RMS-normalises them with `norm_w` (fp16[1024], shared
// or global) into the hi/lo halves the tile products read.  emit: CTA 0 also writes the reference-signature outputs
// (final-norm result fp32, last hidden state fp16).  Ends with a consumer barrier.
__device__ __forceinline__ void red_wait_norm(const Params &P, const Ctx c, int which, uint32_t use, const __half *norm_w, int emit) {
  constexpr int PT = (H + CONS_THREADS - 1) / CONS_THREADS;
  const unsigned long long *buf = P.red + (which ? RED_X2 : RED_X1);
  float *dst = c.f(which ? F_X : F_X1);
  const int R = P.red_copies;
  QMK_FINE(which ? 44 : 40);
  long long vi[PT];
#pragma unroll
  for (int j = 0; j < PT; ++j) vi[j] = 0;
  uint32_t valid = 0;
#pragma unroll
  for (int j = 0; j < PT; ++j)
    if (c.tid + j * CONS_THREADS < H) valid |= 1u << j;
#pragma unroll 1
  for (int r = 0; r < R; ++r) {
    const unsigned long long base = static_cast<unsigned long long>(use) * red_contributors(which ? c.ncta : tctab(c)->groups, R, r);
    const unsigned long long *src = buf + r * RED_SUM_WORDS + red_index(c.tid);
    {
      // one lane per warp watches one word until it is complete, then the warp fetches its words: 32x fewer polls
      // hitting the lines the adds are draining into, at the price of one more L2 round trip at the end (measured at
      // 4096-token context: 1714 -> 1784 tok/s; one lane per CTA + a barrier: the same; a pause between polls: slower)
      if (c.lane == 0) {
        uint32_t n = 0;
        while (((ll_load(src) - base) & RED_CNT_MASK) != 0ull) {
          if ((++n & 1023u) == 0u && (c.flags()[0] || ld_relaxed_u32(P.status) != 0u)) break;   // the full wait below reports time-outs
          if (n > (1u << 22)) break;
        }
      }
      __syncwarp();
    }
    unsigned long long w[PT];
#pragma unroll
    for (int j = 0; j < PT; ++j)
      if (valid & (1u << j)) w[j] = ll_load(src + j * RED_STEP);
    uint32_t pending = valid;
    unsigned long long t0 = 0;
    uint32_t it = 0;
    for (;;) {
#pragma unroll
      for (int j = 0; j < PT; ++j)
        if ((pending & (1u << j)) && ((w[j] - base) & RED_CNT_MASK) == 0ull) pending &= ~(1u << j);
      if (pending == 0u) break;
      if (P.spin_sleep_ns) __nanosleep(P.spin_sleep_ns);
#pragma unroll
      for (int j = 0; j < PT; ++j)
        if (pending & (1u << j)) w[j] = ll_load(src + j * RED_STEP);
      if ((++it & 255u) == 0u) {
        if (c.flags()[0]) break;
        if (ld_relaxed_u32(P.status) != 0u) { c.flags()[0] = 1; break; }
        const unsigned long long t = now_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > P.timeout_ns) { raise_error(P, c, QMK_ERR_WAIT_TIMEOUT, WHERE_LL); break; }
      }
    }
#pragma unroll
    for (int j = 0; j < PT; ++j)
      if (valid & (1u << j)) vi[j] += static_cast<long long>(w[j] - base) >> RED_CNT_BITS;   // exact
  }
  QMK_FINE(which ? 45 : 41);
  float v[PT], w[PT], ss = 0.f;
  bool big = false;
#pragma unroll
  for (int j = 0; j < PT; ++j) {
    v[j] = (valid & (1u << j)) ? static_cast<float>(vi[j]) * RED_INV_SCALE : 0.f;
    w[j] = (valid & (1u << j)) ? __half2float(norm_w[c.tid + j * CONS_THREADS]) : 0.f;
    ss = fmaf(v[j], v[j], ss);
    big |= fabsf(w[j]) > NORM_W_LIMIT;
  }
  const float rstd = block_rstd(c, ss, big), down = big ? NORM_DOWN : 1.f;
  if (c.tid == 0) c.f(F_MISC)[M_XSCALE] = big ? NORM_UP : 1.f;
#pragma unroll
  for (int j = 0; j < PT; ++j)
    if (valid & (1u << j)) {
      const int n = c.tid + j * CONS_THREADS;
      store_normalised(c, n, v[j], rstd, w[j], down, dst);
      if (emit && c.cta == 0) {
        if (P.normalized_out) P.normalized_out[n] = v[j] * rstd * w[j];
        if (P.hidden_out) P.hidden_out[n] = __float2half_rn(v[j]);
      }
    }
  cons_sync();
  QMK_FINE(which ? 46 : 42);
}

#endif  // QMK_TC_SEQS == 1

// Element n of an embedding row.
__device__ __forceinline__ float embed_value(const unsigned char *erow, int n) {
  if (FP8_ROWS) {
    const __half_raw hr = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(__ldg(erow + n)), __NV_E4M3);
    return __half2float(*reinterpret_cast<const __half *>(&hr)) * __ldg(reinterpret_cast<const float *>(erow + H));
  }
  return __half2float(__ldg(reinterpret_cast<const __half *>(erow) + n));
}

#if QMK_TC_SEQS == 1
// Embedding row of `token` (megakernel_5090.cu:825-830) -> residual stream, normalised with layer 0's input norm.
__device__ __forceinline__ void embed_norm(const Params &P, const Ctx c, int token, const __half *norm_w) {
  constexpr int PT = (H + CONS_THREADS - 1) / CONS_THREADS;
  const unsigned char *erow = reinterpret_cast<const unsigned char *>(P.embed) + static_cast<size_t>(token) * ROW_BYTES;
  float v[PT], w[PT], ss = 0.f;
  bool big = false;
#pragma unroll
  for (int j = 0; j < PT; ++j) {
    const int n = c.tid + j * CONS_THREADS;
    v[j] = n < H ? embed_value(erow, n) : 0.f;
    w[j] = n < H ? __half2float(norm_w[n]) : 0.f;
    ss = fmaf(v[j], v[j], ss);
    big |= fabsf(w[j]) > NORM_W_LIMIT;
  }
  const float rstd = block_rstd(c, ss, big), down = big ? NORM_DOWN : 1.f;
  if (c.tid == 0) c.f(F_MISC)[M_XSCALE] = big ? NORM_UP : 1.f;
#pragma unroll
  for (int j = 0; j < PT; ++j) {
    const int n = c.tid + j * CONS_THREADS;
    if (n < H) store_normalised(c, n, v[j], rstd, w[j], down, c.f(F_X));
  }
  cons_sync();
}

#endif  // QMK_TC_SEQS == 1

// A operand of a slice's tiles: this lane's row of each k-step (rows past the slice repeat row 0: their activations are
// zero).  fp8: one ldmatrix.x4 takes 32 rows x 16 outputs, a lane's register holds outputs 2j, 2j + 1 of rows 2q and
// 2q + 1 (j = lane / 4); fragment rows j, j + 8 are those two outputs.
__device__ __forceinline__ void slice_row_addresses(const Ctx &c, int nrows, uint32_t (&arow)[2]) {
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) {
    int row = FP8_ROWS ? c.lane : ks * 16 + (c.lane & 7) + 8 * (c.lane >> 4);
    if (row >= nrows) row = 0;
    arow[ks] = weight_rows(c, c.chunk + static_cast<uint32_t>(row / CH_ROWS)) + (row % CH_ROWS) * ROW_PITCH + (FP8_ROWS ? 0 : ((c.lane >> 3) & 1) * 16);
  }
}
// Output tiles t0, t0 + 12, ... of a slice (past the end: the last tile again, for the caller to ignore): all operands
// first, then all products, then the sums.
constexpr int SLICE_TILES = (H / 16 + CONS_WARPS - 1) / CONS_WARPS;
__device__ __forceinline__ void slice_tiles(const uint32_t (&arow)[2], const uint32_t (&bq)[4], int t0, bool two, float (&acc)[SLICE_TILES][4]) {
  uint32_t a[SLICE_TILES][4];
#pragma unroll
  for (int u = 0; u < SLICE_TILES; ++u) {
    const int tile = min(t0 + u * CONS_WARPS, H / 16 - 1);
    ldsm_x4_trans(arow[0] + tile * (FP8_ROWS ? 16 : 32), a[u]);
  }
  if (FP8_ROWS) {
#pragma unroll
    for (int u = 0; u < SLICE_TILES; ++u) {
      uint32_t r[4], a0[4], a1[4];
      float d[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = __byte_perm(a[u][i], 0u, 0x3120);   // {row 2q, 2q + 1} of the first output, then of the second
      e4m3x4_half2x2(r[0], a0[0], a0[1]);
      e4m3x4_half2x2(r[1], a0[2], a0[3]);
      e4m3x4_half2x2(r[2], a1[0], a1[1]);
      e4m3x4_half2x2(r[3], a1[2], a1[3]);
      mma_16816_zero(acc[u], a0, bq[0], bq[1]);
      if (two) {
        mma_16816_zero(d, a1, bq[2], bq[3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[u][i] += d[i];
      }
    }
  } else {
#pragma unroll
    for (int u = 0; u < SLICE_TILES; ++u) mma_16816_zero(acc[u], a[u], bq[0], bq[1]);
    if (two) {
#pragma unroll
      for (int u = 0; u < SLICE_TILES; ++u) ldsm_x4_trans(arow[1] + min(t0 + u * CONS_WARPS, H / 16 - 1) * 32, a[u]);
      float d[SLICE_TILES][4];
#pragma unroll
      for (int u = 0; u < SLICE_TILES; ++u) mma_16816_zero(d[u], a[u], bq[2], bq[3]);
#pragma unroll
      for (int u = 0; u < SLICE_TILES; ++u)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[u][i] += d[u][i];
    }
  }
}

// What an O slice multiplies: this lane's row address in act16 and in the first four k-steps of 16 weight rows (fp8: two pairs).
// k-steps past the slice repeat its first row: their activations are zero.
constexpr int O_LOADS = 4 / TILE_STEP;         // ldmatrix.x4 of four k-steps
struct OSlice { uint32_t act, row[O_LOADS]; int ne; };
__device__ __forceinline__ uint32_t o_row(const Ctx &c, int ne, int k) {
  const int r = FP8_ROWS ? c.lane : (c.lane & 7) + 8 * (c.lane >> 4);
  const bool in = O_CH_ROWS * k + r < ne;
  return weight_rows(c, c.chunk + static_cast<uint32_t>(in ? k : 0)) + (in ? r : 0) * O_PITCH + (FP8_ROWS ? 0 : ((c.lane >> 3) & 1) * 16);
}
__device__ __forceinline__ OSlice o_slice(const Ctx &c, uint32_t act, int ne) {
  OSlice o;
  o.act = act;
  o.ne = ne;
#pragma unroll
  for (int k = 0; k < O_LOADS; ++k) o.row[k] = o_row(c, ne, k);
  return o;
}
// s + e = a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
  s = a + b;
  const float z = s - a;
  e = (a - (s - z)) + (b - z);
}
// Products of two k-steps: d0, d1 = their sums.  a0 (fp8: the packed bytes of both), a1: ldmatrix results.
__device__ __forceinline__ void o_products(uint32_t (&a0)[4], uint32_t (&a1)[4], const uint32_t (&bq)[4], float (&d0)[4], float (&d1)[4]) {
  if (FP8_ROWS) {
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = __byte_perm(a0[i], 0u, 0x3120);   // as in slice_tiles
    e4m3x4_half2x2(r[0], a0[0], a0[1]);
    e4m3x4_half2x2(r[1], a0[2], a0[3]);
    e4m3x4_half2x2(r[2], a1[0], a1[1]);
    e4m3x4_half2x2(r[3], a1[2], a1[3]);
  }
  mma_16816_zero(d0, a0, bq[0], bq[1]);
  mma_16816_zero(d1, a1, bq[2], bq[3]);
}
// One 16-output tile of an O slice: v[0], v[1] = this lane's two rows of the fragment (quad b: sequence b's hi and lo columns).
// A k-step's products come out of one MMA; the hi sums of the k-steps are added with their rounding errors kept, so that a
// contribution is rounded once, as it was with one k-step per CTA.
__device__ __forceinline__ void slice_o_tile(const Ctx &c, const OSlice &o, int tile, float (&v)[2]) {
  const uint32_t col = tile * (FP8_ROWS ? 16 : 32);
  uint32_t a[4][4], bq[2][4];
  float d[4][4], lo[2], s[2], e[2];
#pragma unroll
  for (int k = 0; k < O_LOADS; ++k) ldsm_x4_trans(o.row[k] + col, a[k * TILE_STEP]);
  ldsm_x4(o.act, bq[0]);
  ldsm_x4(o.act + 64, bq[1]);
  o_products(a[0], a[1], bq[0], d[0], d[1]);
  o_products(a[2], a[3], bq[1], d[2], d[3]);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float s0, s1, e0, e1;
    two_sum(d[0][2 * h], d[1][2 * h], s0, e0);
    two_sum(d[2][2 * h], d[3][2 * h], s1, e1);
    two_sum(s0, s1, s[h], e[h]);
    e[h] += e0 + e1;
    lo[h] = (d[0][2 * h + 1] + d[1][2 * h + 1]) + (d[2][2 * h + 1] + d[3][2 * h + 1]);
  }
#pragma unroll 1
  for (int k = 2; 32 * k < o.ne; ++k) {          // grids of up to 124 CTAs: more than 64 rows
    ldsm_x4_trans(o_row(c, o.ne, k * 2 / TILE_STEP) + col, a[0]);
    if (!FP8_ROWS) ldsm_x4_trans(o_row(c, o.ne, k * 2 + 1) + col, a[1]);
    ldsm_x4(o.act + k * 64, bq[0]);
    o_products(a[0], a[1], bq[0], d[0], d[1]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float s0, e0, e1;
      two_sum(d[0][2 * h], d[1][2 * h], s0, e0);
      two_sum(s[h], s0, s[h], e1);
      e[h] += e0 + e1;
      lo[h] += d[0][2 * h + 1] + d[1][2 * h + 1];
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) v[h] = s[h] + fmaf(lo[h], LO_INV, e[h]);
}

#if QMK_TC_SEQS == 1
// Merge of the attention partials for this CTA's slice of outputs [e0, e0 + ne): the unnormalised outputs of an element's S
// splits, weighted with exp2(max_s - max) / sum, go to act16 as the hi / lo halves of the O slice's operand.  A warp takes quads
// of four consecutive elements (a 32-byte sector of every split's partial): lane 4 k + i holds element i, splits k, k + 8 and k + 16.
// The last two warps also fetch the (max, sum) pairs of the slice's (at most two) heads, in the same round of polls, and share
// the weights through a barrier: polled by every warp they cost 2 us a layer.
constexpr int MERGE_QUADS = 2, MERGE_SPLITS = (MAX_SPLITS + 7) / 8;
__device__ __forceinline__ void merge_o(const Params &P, const Ctx &c, int S, uint32_t tag) {
  const TcTab *t = tctab(c);
  const int e0 = t->e0, ne = t->ne, h0 = e0 >> 7, el = c.lane & 3, sl = c.lane >> 2;
  float *s_wt = c.f(FF_SPLITW);
  constexpr int NW = MERGE_QUADS * MERGE_SPLITS;
  const unsigned long long *words = c.llr + LL_PART;
  uint32_t wp[NW], valid = 0;
#pragma unroll
  for (int i = 0; i < MERGE_QUADS; ++i) {
    const int q = c.warp + i * CONS_WARPS, e = e0 + (4 * q < ne ? 4 * q : 0) + el;
    const uint32_t head = (e >> 7) * (MAX_SPLITS * PART_STRIDE) + (e & (D - 1));
#pragma unroll
    for (int k = 0; k < MERGE_SPLITS; ++k) {
      wp[i * MERGE_SPLITS + k] = head + min(sl + 8 * k, S - 1) * PART_STRIDE;
      if (4 * q < ne && sl + 8 * k < S) valid |= 1u << (i * MERGE_SPLITS + k);
    }
  }
  QMK_FINE(50);
  float a[NW];
  if (4 * c.warp < ne) {
    // the owner split (the last one) also handles the new row: its words arrive last.  (Without this watch where there are one or
    // two splits, words polled at once: 432 -> 448 us per step at 64 tokens; polls slow the attention CTAs.)
    const int e = e0 + 4 * c.warp;
    ll_sentinel(P, c, words + ((e >> 7) * MAX_SPLITS + S - 1) * PART_STRIDE + (e & (D - 1)), tag);
    const int hw = h0 + (c.warp - (CONS_WARPS - 2));                      // head whose split weights this warp makes
    if (c.warp >= CONS_WARPS - 2 && hw <= ((e0 + ne - 1) >> 7)) {         // warp-uniform
      uint32_t wl[MERGE_SPLITS + 2];
      float v[MERGE_SPLITS + 2];
#pragma unroll
      for (int k = 0; k < MERGE_SPLITS; ++k) wl[k] = wp[k];
      wl[MERGE_SPLITS] = (hw * MAX_SPLITS + min(c.lane, S - 1)) * PART_STRIDE + D;
      wl[MERGE_SPLITS + 1] = wl[MERGE_SPLITS] + 1;
      ll_wait_words<MERGE_SPLITS + 2>(P, c, words, wl, (valid & ((1u << MERGE_SPLITS) - 1u)) | (c.lane < S ? 3u << MERGE_SPLITS : 0u), tag, v);
#pragma unroll
      for (int k = 0; k < NW; ++k) a[k] = k < MERGE_SPLITS ? v[k] : 0.f;
      const float m = c.lane < S ? v[MERGE_SPLITS] : -INFINITY, l = c.lane < S ? v[MERGE_SPLITS + 1] : 0.f;
      const float M = warp_max(m);
      const float sc = (m == -INFINITY) ? 0.f : exp2f(m - M);
      const float L = warp_sum(l * sc);
      s_wt[(hw - h0) * 32 + c.lane] = sc / L;
    } else {
      ll_wait_words<NW>(P, c, words, wp, valid, tag, a);
    }
    QMK_FINE(51);
  }
  cons_sync();
  QMK_FINE(52);
  __half *act16 = reinterpret_cast<__half *>(c.smem + OFF_ACT16);
  float A[MERGE_QUADS];
#pragma unroll
  for (int i = 0; i < MERGE_QUADS; ++i) {
    const int q = c.warp + i * CONS_WARPS, e = e0 + (4 * q < ne ? 4 * q : 0) + el;
    A[i] = 0.f;
#pragma unroll
    for (int k = 0; k < MERGE_SPLITS; ++k)
      if (valid & (1u << (i * MERGE_SPLITS + k))) A[i] = fmaf(a[i * MERGE_SPLITS + k], s_wt[((e >> 7) - h0) * 32 + sl + 8 * k], A[i]);
  }
#pragma unroll
  for (int o = 16; o > 2; o >>= 1)
#pragma unroll
    for (int i = 0; i < MERGE_QUADS; ++i) A[i] += __shfl_xor_sync(0xffffffffu, A[i], o);
#pragma unroll
  for (int i = 0; i < MERGE_QUADS; ++i) {
    const int q = c.warp + i * CONS_WARPS;
    if (4 * q < ne && sl < 2) act16[sl * ACT16_PITCH + 4 * q + el] = split_half(A[i], sl != 0);
  }
  if (c.tid >= ne && c.tid < 32 * O_KPAIRS) { act16[c.tid] = __float2half_rn(0.f); act16[ACT16_PITCH + c.tid] = __float2half_rn(0.f); }
}

// O slice: this CTA's merged attention outputs times its quarter of the outputs -> sum x1.
__device__ __forceinline__ uint32_t slice_o(const Params &P, Ctx c) {
  const TcTab *t = tctab(c);
  const int ne = t->ne, nch = t->no;
  if (nch == 0) return c.chunk;
  const float *resid = c.f(F_X);
  float *prev = c.f(FF_PREV);
  unsigned long long *mine = P.red + RED_X1 + ((c.cta / O_GROUP) & (P.red_copies - 1)) * RED_SUM_WORDS;   // one or two copies
  QMK_FINE(20);
  const bool ok = wait_chunks(P, c, c.chunk, nch);
  if (ok) {
    const OSlice o = o_slice(c, smem_u32(c.smem + OFF_ACT16) + (c.lane & 1) * (ACT16_PITCH * 2) + (c.lane >> 3) * 16, ne);
    const int n0 = t->n0, n1 = t->n1, out0 = t->oq * O_COLS;
    const int src = FP8_ROWS ? ((c.lane & 15) >> 1) * 4 : (c.lane & 7) * 4;      // as in slice_cols
    const bool second = (c.lane & (FP8_ROWS ? 1 : 8)) != 0;
    float v0[2], v1[2] = {0.f, 0.f};
    slice_o_tile(c, o, c.warp, v0);
    if (c.warp + CONS_WARPS < O_TILES) slice_o_tile(c, o, c.warp + CONS_WARPS, v1);
    const float s0 = __shfl_sync(0xffffffffu, v0[0], src), s1 = __shfl_sync(0xffffffffu, v0[1], src);
    const float s2 = __shfl_sync(0xffffffffu, v1[0], src), s3 = __shfl_sync(0xffffffffu, v1[1], src);
    const int tile = c.warp + (c.lane >> 4) * CONS_WARPS;
    if (tile < O_TILES) {
      const int j = tile * 16 + (c.lane & 15), n = out0 + j;
      float v = (c.lane & 16) ? (second ? s3 : s2) : (second ? s1 : s0);
      if (FP8_ROWS) v *= reinterpret_cast<const float *>(c.smem + (weight_rows(c, c.chunk + static_cast<uint32_t>(nch - 1)) - smem_u32(c.smem)))[j];
      if (n >= n0 && n < n1) v += resid[n];
      const long long fx = __float2ll_rn(v * RED_SCALE), fx_prev = __float2ll_rn(prev[j] * RED_SCALE);
      prev[j] = v;
      red_add_u64(mine + red_index(n), (static_cast<unsigned long long>(fx - fx_prev) << RED_CNT_BITS) + 1ull);
    }
  }
  __syncwarp();
  if (c.lane < nch) mbar_arrive_n(c.empty((c.chunk + static_cast<uint32_t>(c.lane)) % NSLOTS), EMPTY_UNITS / CONS_WARPS);
  QMK_FINE(23);
  return c.chunk + static_cast<uint32_t>(nch);
}

// Split-K slice of the down projection (see slice_colgemv of megakernel_fused.cuh) on the
// tensor cores: partial[n] = sum_i act[i] * Wt[first + i][n] with the K-major rows as the A operand read through
// ldmatrix.trans (tile = 16 outputs x 16 rows, at most two k-steps: slices of at most 32 rows), the slice's
// activations as B (hi / lo columns, from act16).  Warp w takes output tiles w, w + 12, ... over ALL rows of the
// slice, so a partial is complete when it leaves the warp: after each pair of tiles the 32 sums are spread over
// the 32 lanes (four shuffles) and every lane adds its one output into the residual sum - no staging in shared
// memory, no barrier, and the adds of early tiles drain while later tiles are computed.
__device__ __forceinline__ uint32_t slice_cols(const Params &P, Ctx c) {
  const TcTab *t = tctab(c);
  const int nrows = t->ng * CH_ROWS;
  const float *resid = c.f(F_X1);
  float *prev = c.f(FF_PREV) + H;
  unsigned long long *mine = P.red + RED_X2 + (c.cta & (P.red_copies - 1)) * RED_SUM_WORDS;   // one or two copies
  const int nch = (nrows + CH_ROWS - 1) / CH_ROWS + SCALE_CH;
  [[maybe_unused]] const float *scales = FP8_ROWS ? reinterpret_cast<const float *>(c.slot(c.chunk + static_cast<uint32_t>(nch - 1))) : nullptr;
  const bool two = nrows > 16;
  QMK_FINE(30);
  const bool ok = wait_chunks(P, c, c.chunk, nch);
  if (ok) {
    // B: the slice's activations; row n of B^T = hi (even n) / lo (odd n) vector; one ldmatrix.x4 = two k-steps
    uint32_t bq[4];
    ldsm_x4(smem_u32(c.smem + OFF_ACT16) + (c.lane & 1) * (ACT16_PITCH * 2) + (c.lane >> 3) * 16, bq);
    uint32_t arow[2];
    slice_row_addresses(c, nrows, arow);
    const int n0 = t->n0, n1 = t->n1;
    const float up = c.f(F_MISC)[M_ASCALE];
    // lane that holds this lane's output (fragment row = lane / 4), and whether it is its second row
    const int src = FP8_ROWS ? ((c.lane & 15) >> 1) * 4 : (c.lane & 7) * 4;
    const bool second = (c.lane & (FP8_ROWS ? 1 : 8)) != 0;
    float acc[SLICE_TILES][4];
    slice_tiles(arow, bq, c.warp, two, acc);
    static_assert(SLICE_TILES % 2 == 0, "tiles leave in pairs");
    // All sums on their lanes first, then all fixed-point values, then the adds (a pair of tiles after the other took 200 cycles each:
    // 435 / 446 -> 433 / 444 us per step at 64 / 1024 tokens).
    float v[SLICE_TILES / 2];
    unsigned long long add[SLICE_TILES / 2];
#pragma unroll
    for (int u = 0; u < SLICE_TILES; u += 2) {
      // lanes of quad 0 hold (hi, lo) sums of fragment rows lane / 4 and lane / 4 + 8 of both tiles; lane L takes output
      // L % 16 of tile L / 16
      const float s0 = __shfl_sync(0xffffffffu, fmaf(acc[u][1], LO_INV, acc[u][0]), src);
      const float s1 = __shfl_sync(0xffffffffu, fmaf(acc[u][3], LO_INV, acc[u][2]), src);
      const float s2 = __shfl_sync(0xffffffffu, fmaf(acc[u + 1][1], LO_INV, acc[u + 1][0]), src);
      const float s3 = __shfl_sync(0xffffffffu, fmaf(acc[u + 1][3], LO_INV, acc[u + 1][2]), src);
      v[u / 2] = ((c.lane & 16) ? (second ? s3 : s2) : (second ? s1 : s0)) * up;
    }
#pragma unroll
    for (int u = 0; u < SLICE_TILES / 2; ++u) {
      const int tile = c.warp + (2 * u + (c.lane >> 4)) * CONS_WARPS, n = (tile < H / 16 ? tile : c.warp) * 16 + (c.lane & 15);
      if (FP8_ROWS) v[u] *= scales[n];
      if (n >= n0 && n < n1) v[u] += resid[n];
      const long long fx = __float2ll_rn(v[u] * RED_SCALE), fx_prev = __float2ll_rn(prev[n] * RED_SCALE);
      add[u] = (static_cast<unsigned long long>(fx - fx_prev) << RED_CNT_BITS) + 1ull;
    }
#pragma unroll
    for (int u = 0; u < SLICE_TILES / 2; ++u) {
      const int tile = c.warp + (2 * u + (c.lane >> 4)) * CONS_WARPS, n = tile * 16 + (c.lane & 15);
      if (tile < H / 16) {
        prev[n] = v[u];
        red_add_u64(mine + red_index(n), add[u]);
      }
    }
  }
  __syncwarp();
  if (c.lane < nch) mbar_arrive_n(c.empty((c.chunk + static_cast<uint32_t>(c.lane)) % NSLOTS), EMPTY_UNITS / CONS_WARPS);
  QMK_FINE(33);
  return c.chunk + static_cast<uint32_t>(nch);
}

// Tied LM head + per-CTA argmax (megakernel_5090.cu:1024-1132).  One 16-row tile per round, its 1024 inputs split
// over the twelve warps; the partial sums go through a double-buffered shared array, so one barrier per round;
// threads 0..15 finish one row each and keep a running (max, lowest index).  A round consumes four of the ring's
// twenty chunks, which leaves sixteen in flight (the stream needs bandwidth x latency = ~130 KB per SM in flight;
// rounds of three tiles left eight and ran at 3.4 TB/s).  Leaves the per-warp results that argmax_exchange()
// expects in s_misc[32..43] / s_misc[48..59].
__device__ __forceinline__ uint32_t lm_head_tc(const Params &P, Ctx c, float *dump) {
  const TcTab *t = tctab(c);
  const int nch = t->nlm, ntiles = (nch + TILE_CH - 1) / TILE_CH;
  float *part = tc_part(c), *s_misc = c.f(F_MISC);
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  const int p0 = k_split(c.warp, CONS_WARPS), p1 = k_split(c.warp + 1, CONS_WARPS);
  const float up = s_misc[M_XSCALE];
#pragma unroll 1
  for (int tile = 0; tile < ntiles; ++tile) {
    float *pr = part + (tile & 1) * (CONS_WARPS * 16);
    run_tile(c, prepare_tile(P, c, c.chunk + static_cast<uint32_t>(tile * TILE_CH), min(16, (nch - tile * TILE_CH) * CH_ROWS), p0, p1,
                             EMPTY_UNITS / CONS_WARPS), pr + c.warp * 16);
    cons_sync();
    if (c.tid < 16) {
      const int row = tile * 16 + c.tid;
      if (row < nch * CH_ROWS) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < CONS_WARPS; ++w) v += pr[w * 16 + c.tid];
        v *= up;
        const int o = t->lm0 * CH_ROWS + row;
        if (v > best) { best = v; best_i = o; }     // rows ascend per thread: strict > keeps the lowest index
        if (dump) dump[o] = v;
      }
    }
  }
  if (c.warp == 0) {   // threads 0..15 hold candidates
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
      if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
  }
  if (c.lane == 0) {
    s_misc[32 + c.warp] = c.warp == 0 ? best : -INFINITY;
    s_misc[48 + c.warp] = __int_as_float(c.warp == 0 ? best_i : 0x7fffffff);
  }
  return c.chunk + static_cast<uint32_t>(nch);
}

#endif  // QMK_TC_SEQS == 1

// ----------------------------------------------------------------------------- producer (one warp)
// The warp issues eight chunks at a time: lanes 4g..4g+3 own chunk g of the group of eight, lane 4g waits for
// the slot and announces the bytes, lane 4g + r copies row r (one cp.async.bulk per row, 2064-byte pitch).  Per
// chunk, wait + announce + copy are ~800 cycles of dependent latency; one chunk at a time capped the stream at
// 19 GB/s per SM (LM head 2.8 TB/s), eight at a time keep that latency off the stream.
// A layer's chunks in ring order: q|k|v rows, this CTA's old K/V rows, K-major O rows [e0, e1), gate rows, up
// rows, K-major down rows (fp8: the output scales behind the O and the down rows); after the last layer the LM-head rows.
// kv_row >= 0 marks a cache chunk: 16 rows of the K and of the V cache from that row on (rows of the caches seen as
// [layers * 8 * max_seq_len][128]); lane r of the group copies box r (K low dims, K high dims, V low, V high).
struct ChunkSrc { const unsigned char *src; size_t src_pitch; uint32_t rows, row_bytes, dst_pitch; int kv_row; };

__device__ __forceinline__ bool tc_issue8(const Params &P, const Ctx &c, uint32_t ci, bool active, const ChunkSrc &d, uint64_t pol,
                                          const void *kmap, const void *vmap) {
  if (__any_sync(0xffffffffu, (c.flags()[0] | c.flags()[1]) != 0)) return false;   // the warp leaves as a whole
  const uint32_t slot = ci % NSLOTS;
  bool ok = true;
  if (active && ci >= NSLOTS) ok = mbar_wait(P, c, c.empty(slot), ((ci / NSLOTS) - 1u) & 1u, WHERE_EMPTY, true);
  if (!__all_sync(0xffffffffu, ok)) return false;
  const int sub = c.lane & 3;
  if (active && sub == 0) mbar_arrive_expect_tx(c.full(slot), d.kv_row >= 0 ? 4u * KV_BOX : d.rows * d.row_bytes);
  __syncwarp();
  if (active && d.kv_row >= 0) {
    tma_box_2d(smem_u32(c.slot(ci)) + sub * KV_BOX, sub < 2 ? kmap : vmap,
               (sub & 1) * 64, d.kv_row, c.full(slot));
  } else if (active && sub < static_cast<int>(d.rows)) {
    bulk_g2s(c.slot(ci) + (ci & 1u) * ODD_SLOT_SKEW + sub * d.dst_pitch, d.src + sub * d.src_pitch, d.row_bytes, c.full(slot), pol);
  }
  return true;
}
// A chunk's rows of a row-major matrix with 1024 inputs (or of a K-major copy), starting at `row`; fp8 rows are
// contiguous at the pitch they have in shared memory: one copy.
__device__ __forceinline__ ChunkSrc matrix_chunk(const void *base, int row, int rows) {
  ChunkSrc d;
  d.src = reinterpret_cast<const unsigned char *>(base) + static_cast<size_t>(row) * ROW_BYTES;
  d.src_pitch = ROW_BYTES;
  d.rows = static_cast<uint32_t>(FP8_ROWS ? 1 : rows);
  d.row_bytes = static_cast<uint32_t>(FP8_ROWS ? rows * ROW_BYTES : ROW_BYTES);
  d.dst_pitch = ROW_PITCH;
  d.kv_row = -1;
  return d;
}

// The 1024 fp32 output scales of a K-major fp8 copy with `rows` rows (they follow the last one).
__device__ __forceinline__ ChunkSrc scale_chunk(const void *base, int rows) {
  ChunkSrc d = matrix_chunk(base, rows, 0);
  d.rows = 1u;
  d.row_bytes = 4 * H;
  return d;
}

// (A function of its own for one sequence, inlined for several: 434 against 442 us per step of one fp16 sequence at 64 tokens, 812
// against 748 of four at 1024.)
#if QMK_TC_SEQS == 1
__device__ __noinline__
#else
__device__ __forceinline__
#endif
void producer_main_tc(const Params &P, const Ctx c) {
  const uint64_t pol = P.l2_evict_first ? l2_evict_first_policy() : l2_evict_normal_policy();
  const TcTab *tt = tctab(c);
  const int grp = c.lane >> 2;
  // the caches this CTA attends to
  const int seq = TC_SEQS == 1 ? 0 : tt->seq;
  const void *kmap = P.kmaps[0], *vmap = P.vmaps[0];
  if (TC_SEQS > 1) {
#pragma unroll
    for (int b = 1; b < TC_SEQS; ++b)
      if (seq == b) { kmap = P.kmaps[b]; vmap = P.vmaps[b]; }
  }
  const int start = TC_SEQS == 1 ? P.start_position : per_seq(P.start_positions, seq);
  const int nq = tt->nq, ng = tt->ng, ne = tt->ne, no = tt->no;
  uint32_t idx = 0, issued = 0;   // first chunk of the current layer / chunks issued so far
  bool ok = true;
#pragma unroll 1
  for (int step = 0; ok && step < P.num_steps; ++step) {
    const AttnItem it = tc_item(P, c, start + step);
    const int s1 = nq, s2 = s1 + it.nchunks, s3 = s2 + no, s4 = s3 + ng, s5 = s4 + ng, per_layer = s5 + ng + SCALE_CH;
#pragma unroll 1
    for (int l = 0; ok && l < P.num_layers; ++l) {
      const unsigned long long *rec = c.layer_rec(l);
      const unsigned long long *rect = c.layer_rec_t(l);
      if (c.lane == 0) {   // this layer's norm vectors (see producer_main)
        const uint32_t L = static_cast<uint32_t>(step) * static_cast<uint32_t>(P.num_layers) + static_cast<uint32_t>(l);
        const uint32_t b = L & 1u;
        __half *dst = c.norms(b);
        c.flags()[4 + b] = static_cast<int>(L + 1u);
        mbar_arrive_expect_tx(c.nfull(b), NORM_HALVES * 2);
        bulk_g2s(dst + NB_IN_LN, reinterpret_cast<const void *>(rec[REC_IN_LN]), H * 2, c.nfull(b), l2_evict_normal_policy());
        bulk_g2s(dst + NB_POST_LN, reinterpret_cast<const void *>(rec[REC_POST_LN]), H * 2, c.nfull(b), l2_evict_normal_policy());
        bulk_g2s(dst + NB_QNORM, reinterpret_cast<const void *>(rec[REC_QNORM]), D * 2, c.nfull(b), l2_evict_normal_policy());
        bulk_g2s(dst + NB_KNORM, reinterpret_cast<const void *>(rec[REC_KNORM]), D * 2, c.nfull(b), l2_evict_normal_policy());
      }
      __syncwarp();
#pragma unroll 1
      for (int j0 = 0; ok && j0 < per_layer; j0 += 8) {
        const int j = j0 + grp;
        ChunkSrc d = matrix_chunk(nullptr, 0, 0);
        if (j < s1) {            // q|k|v: a chunk lies in one tensor (2048 and 3072 are multiples of 4)
          const int row = (tt->q0 + j) * CH_ROWS;
          const int sel = row < QS ? 0 : row < QS + KVS ? 1 : 2;
          d = matrix_chunk(reinterpret_cast<const void *>(rec[REC_WQ + sel]), row - (sel == 0 ? 0 : sel == 1 ? QS : QS + KVS), CH_ROWS);
        } else if (j < s2) {     // old K rows (lane 4g) and V rows (lane 4g + 1) of the attention item
          d.kv_row = (l * NKV + it.g) * P.max_seq_len + it.p0 + (j - s1) * it.rpc;
        } else if (j < s3) {
          const int r = (j - s2) * O_CH_ROWS;
          const unsigned char *base = reinterpret_cast<const unsigned char *>(rect[0]);
          d.rows = 1u;
          if (r < ne) {
            d.src = base + static_cast<size_t>(tt->oq * QS + tt->e0 + r) * O_PITCH;
            d.row_bytes = static_cast<uint32_t>(min(O_CH_ROWS, ne - r) * O_PITCH);
          } else {               // fp8: the scales of the quarter's outputs
            d.src = base + static_cast<size_t>(O_GROUP * QS) * O_PITCH + tt->oq * O_COLS * 4;
            d.row_bytes = 4 * O_COLS;
          }
        } else if (j < s4) {
          d = matrix_chunk(reinterpret_cast<const void *>(rec[REC_GATE]), (tt->g0 + j - s3) * CH_ROWS, CH_ROWS);
        } else if (j < s5) {
          d = matrix_chunk(reinterpret_cast<const void *>(rec[REC_UP]), (tt->g0 + j - s4) * CH_ROWS, CH_ROWS);
        } else if (j < s5 + ng) {
          d = matrix_chunk(reinterpret_cast<const void *>(rect[1]), (tt->g0 + j - s5) * CH_ROWS, CH_ROWS);
        } else if (j < per_layer) {
          d = scale_chunk(reinterpret_cast<const void *>(rect[1]), I);
        }
        ok = tc_issue8(P, c, idx + static_cast<uint32_t>(j), j < per_layer, d, pol, kmap, vmap);   // issues all eight or none
        if (ok) issued = idx + static_cast<uint32_t>(min(j0 + 8, per_layer));
      }
      idx += static_cast<uint32_t>(per_layer);
    }
    if (!P.prefill) {
#pragma unroll 1
      for (int j0 = 0; ok && j0 < tt->nlm; j0 += 8) {
        const int j = j0 + grp;
        const ChunkSrc d = matrix_chunk(P.lm_head, (tt->lm0 + j) * CH_ROWS, CH_ROWS);
        ok = tc_issue8(P, c, idx + static_cast<uint32_t>(j), j < tt->nlm, d, pol, kmap, vmap);
        if (ok) issued = idx + static_cast<uint32_t>(min(j0 + 8, tt->nlm));
      }
      idx += static_cast<uint32_t>(tt->nlm);
    }
  }
  if (c.lane == 0) c.flags()[2] = static_cast<int>(issued);
}

// Barriers, tables and pointer records of a CTA; the caller synchronises the block.
__device__ __forceinline__ void tc_setup(const Params &P, const Ctx &c) {
  if (c.tid == 0) {
    for (int i = 0; i < NSLOTS; ++i) { mbar_init(c.full(i), 1); mbar_init(c.empty(i), EMPTY_UNITS); }
    mbar_init(c.nfull(0), 1);
    mbar_init(c.nfull(1), 1);
    volatile int *fl = c.flags();
    fl[0] = 0; fl[1] = 0; fl[2] = 0; fl[3] = 0; fl[4] = 0; fl[5] = 0; fl[6] = 0; fl[8] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (c.tid == 32) {
    build_segtab(reinterpret_cast<SegTab *>(c.smem + OFF_SEGS), c.cta, c.ncta, P.vocab);
    TcTab *tt = reinterpret_cast<TcTab *>(c.smem + OFF_TCTAB);
    int a, b;
    split_rows(QKV_CHUNKS, c.ncta, c.cta, a, b); tt->q0 = a; tt->nq = b - a;
    split_rows(GU_CHUNKS, c.ncta, c.cta, a, b); tt->g0 = a; tt->ng = b - a;
    split_rows(P.vocab / CH_ROWS, c.ncta, c.cta, a, b); tt->lm0 = a; tt->nlm = b - a;
    tt->early = EARLY_ROWS && max(tt->nq, 2 * tt->ng) + 7 <= NSLOTS;
    tt->groups = c.ncta / O_GROUP;
    const int grp = c.cta / O_GROUP;
    tt->oq = c.cta % O_GROUP;
    tt->e0 = tt->ne = tt->no = tt->n0 = tt->n1 = 0;   // (chunks as in layer_chunks)
    if (grp < tt->groups) {
      split_rows(QS / 4, tt->groups, grp, a, b); tt->e0 = 4 * a; tt->ne = 4 * (b - a);
      split_rows(O_COLS, tt->groups, grp, a, b); tt->n0 = tt->oq * O_COLS + a; tt->n1 = tt->oq * O_COLS + b;
      tt->no = (tt->ne + O_CH_ROWS - 1) / O_CH_ROWS + SCALE_CH;
    }
    build_tile_tasks(tt->qkv, &tt->nkb_qkv, 1, tt->nq);
    build_tile_tasks(tt->gu, &tt->nkb_gu, GU_ONE_RUN ? 1 : 2, GU_ONE_RUN ? 2 * tt->ng : tt->ng);
  }
  {
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(P.layers);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(c.smem + OFF_LAYERS);
    for (int i = c.tid; i < P.num_layers * 12; i += THREADS) dst[i] = src[i];
    const unsigned long long *srct = reinterpret_cast<const unsigned long long *>(P.layers_t);
    unsigned long long *dstt = reinterpret_cast<unsigned long long *>(c.smem + OFF_LAYERS_T);
    for (int i = c.tid; i < P.num_layers * 2; i += THREADS) dstt[i] = srct[i];
  }
}

// Bulk copies issued but never consumed must land before the CTA exits.
__device__ __forceinline__ void tc_drain(const Params &P, const Ctx &c) {
  if (c.tid == CONS_THREADS) {
    const uint32_t issued = static_cast<uint32_t>(c.flags()[2]);
#pragma unroll 1
    for (uint32_t i = (issued > NSLOTS ? issued - NSLOTS : 0u); i < issued; ++i) {
      uint64_t *bar = c.full(i % NSLOTS);
      const uint32_t parity = (i / NSLOTS) & 1u;
      const unsigned long long t0 = now_ns();
      while (!mbar_try_wait(bar, parity)) {
        if (now_ns() - t0 > P.timeout_ns) { raise_error(P, c, QMK_ERR_WAIT_TIMEOUT, WHERE_DRAIN); break; }
      }
    }
    for (uint32_t b = 0; b < 2; ++b) {
      const int v = c.flags()[4 + b];
      if (v == 0) continue;
      const uint32_t parity = ((static_cast<uint32_t>(v) - 1u) >> 1) & 1u;
      const unsigned long long t0 = now_ns();
      while (!mbar_try_wait(c.nfull(b), parity)) {
        if (now_ns() - t0 > P.timeout_ns) { raise_error(P, c, QMK_ERR_WAIT_TIMEOUT, WHERE_DRAIN); break; }
      }
    }
  }
}

#if QMK_TC_SEQS == 1
__global__ void __launch_bounds__(THREADS, 1) qwen3_decode_megakernel_tc(const __grid_constant__ Params P) {
  extern __shared__ __align__(128) unsigned char smem[];
  Ctx c;
  c.smem = smem;
  c.tid = threadIdx.x;
  c.warp = threadIdx.x >> 5;
  c.lane = threadIdx.x & 31;
  c.cta = blockIdx.x;
  c.ncta = gridDim.x;
  c.chunk = 0;
  c.repl = 1;
  c.llr = P.ll;

  tc_setup(P, c);
  for (int i = c.tid; i < 2 * H; i += THREADS) c.f(FF_PREV)[i] = 0.f;
  __syncthreads();

  if (c.warp == CONS_WARPS) {
    producer_main_tc(P, c);
    __syncwarp();
  } else {
    float *s_misc = c.f(F_MISC);
    int token = P.prefill ? P.token_ids[0] : P.first_token;
#pragma unroll 1
    for (int step = 0; step < P.num_steps; ++step) {
      const int pos = P.start_position + step;
      const uint32_t tag_base = (P.seq_base + static_cast<uint32_t>(step)) * 64u;
      if (token < 0 || token >= P.vocab) { if (c.tid == 0) raise_error(P, c, QMK_ERR_BAD_TOKEN, WHERE_TOKEN); token = 0; }
      if (c.tid < D / 2) {
        float cs, sn;
        if (P.rope_from_table) {
          cs = __half2float(P.cos_table[static_cast<size_t>(pos) * D + c.tid]);
          sn = __half2float(P.sin_table[static_cast<size_t>(pos) * D + c.tid]);
        } else {
          cs = __ldg(P.rope + static_cast<size_t>(pos) * D + c.tid);
          sn = __ldg(P.rope + static_cast<size_t>(pos) * D + 64 + c.tid);
        }
        c.f(F_CS)[c.tid] = cs;
        c.f(F_CS)[64 + c.tid] = sn;
      }
      __threadfence();  // acquire side of the KV-row ordering (rows written in earlier steps)
      const int S_step = max(1, min(pos / max(1, P.split_len), min(MAX_SPLITS, max(1, c.ncta / NKV))));  // as attn_item
      {
        const uint32_t L0 = static_cast<uint32_t>(step) * static_cast<uint32_t>(P.num_layers);
        mbar_wait(P, c, c.nfull(L0 & 1u), (L0 >> 1) & 1u, WHERE_FULL, false);
        embed_norm(P, c, token, c.norms(L0 & 1u) + NB_IN_LN);
      }
#pragma unroll 1
      for (int layer = 0; layer < P.num_layers; ++layer) {
        const uint32_t tag = tag_base + static_cast<uint32_t>(layer) + 1u;
        const uint32_t Lg = static_cast<uint32_t>(step) * static_cast<uint32_t>(P.num_layers) + static_cast<uint32_t>(layer);
        const __half *nv = c.norms(Lg & 1u);
        const uint32_t use = Lg + 1u;
#ifdef QMK_FINE_PROF
        if (c.tid == 0) c.flags()[8] = (step == P.num_steps - 1 && layer == 5) ? 1 : 0;
#endif
        QMK_STAMP(layer * 12 + 0);
        c.chunk = qkv_phase(P, c, tag);
        QMK_STAMP(layer * 12 + 1);
        c.chunk = attention_tc(P, c, nv, layer, pos, tag);
        QMK_STAMP(layer * 12 + 2);
        merge_o(P, c, S_step, tag);
        QMK_STAMP(layer * 12 + 3);
        cons_sync();
        c.chunk = slice_o(P, c);
        QMK_STAMP(layer * 12 + 4);
        red_wait_norm(P, c, 0, use, nv + NB_POST_LN, 0);
        QMK_STAMP(layer * 12 + 5);
        c.chunk = gateup_phase(P, c);
        QMK_STAMP(layer * 12 + 6);
        cons_sync();
        c.chunk = slice_cols(P, c);
        QMK_STAMP(layer * 12 + 7);
        const bool last = layer == P.num_layers - 1;
        if (!last) mbar_wait(P, c, c.nfull((Lg + 1u) & 1u), ((Lg + 1u) >> 1) & 1u, WHERE_FULL, false);
        // the next consumer of x: the following layer's input norm, or the final norm before the LM head (a prefill
        // pass ends here: any vector will do)
        const __half *next_norm = !last ? c.norms((Lg + 1u) & 1u) + NB_IN_LN : P.prefill ? nv + NB_IN_LN : P.final_norm;
        red_wait_norm(P, c, 1, use, next_norm, (last && !P.prefill) ? 1 : 0);
        QMK_STAMP(layer * 12 + 8);
        if (cons_any(c.flags()[0] != 0)) break;
      }
      if (cons_any(c.flags()[0] != 0)) break;
      if (P.prefill) {
        if (step + 1 < P.num_steps) token = P.token_ids[step + 1];
        continue;
      }
      QMK_STAMP(P.num_layers * 12 + 0);
      c.chunk = lm_head_tc(P, c, P.logits_out ? P.logits_out + static_cast<size_t>(step) * P.vocab : nullptr);
      QMK_STAMP(P.num_layers * 12 + 1);
      cons_sync();
      argmax_exchange(P, c, tag_base + 63u);
      const bool aborted = cons_any(c.flags()[0] != 0);
      QMK_STAMP(P.num_layers * 12 + 2);
      token = __float_as_int(s_misc[16]);
      if (aborted) break;
      if (c.cta == 0 && c.tid == 0) {
        if (P.output_log) P.output_log[step] = token;
        if (P.output_token) *P.output_token = token;
      }
      if (token == P.eos) break;
    }
    if (c.tid == 0) { c.flags()[3] = static_cast<int>(c.chunk); c.flags()[1] = 1; }
  }
  __syncthreads();
  tc_drain(P, c);
}
#endif  // QMK_TC_SEQS == 1

#endif  // QMK_MAX_SEQ == 1 && QMK_TC_BUILD
}  // namespace QMK_NS
