// Multi-sequence form of the tensor-core decode megakernel: up to QMK_TC_SEQS (2 or 4) sequences per launch.
//
// The B operand of an mma.sync.m16n8k16 has eight columns and the single-sequence kernel fills two of them (the hi and
// the lo half of the activations).  Here sequence b has columns 2b and 2b + 1, so the row products of all sequences are
// the SAME ldmatrix and MMA instructions as of one, and thread quad q of a fragment holds sequence q's sums.  The layer
// keeps the four hand-overs of the fused kernel; a sequence has its own exchange words (one copy of the exchange area
// each) and its own residual sums.  Attention items are (sequence, kv head, split): a CTA has at most one, the splits
// per sequence shrink instead (grid / (8 * sequences)).  What grows with the sequences: adds into the residual sums,
// words read back, cache rows.
// The launch it replaces (megakernel_batch.cuh, which stays for grids outside this kernel's range) gives each sequence a
// group of warps that convert and multiply every weight for themselves, and has six hand-overs per layer.
// Measured, us per step at 64 / 1024 / 2048-token contexts, means of five placements of the buffers: two fp16 sequences 485 / 514 /
// 566, three 625 / 694 / 756, four 642 / 728 / 819 (a placement within 1 %; three sequences 3 %), four with FP8 rows 589 / 688 / 793 (5 %),
// two 516 / 559 at 64 / 1024 (7 %).  (The group launch: two 1137 / 1317 at 64 / 1024; four 1655 / 1942; the GEMM step: four fp16 758 /
// 804 / 870, four FP8 904 / 959 / 1019, with fp16-rounded activations.)  Share of later layers' cache values
// that round to another fp16 than float64's, 1024 tokens: two and four fp16 sequences 0.155 and 0.157 % (group launch 0.147
// and 0.150), two with FP8 rows 0.149 (0.151).

namespace QMK_NS {
#if QMK_MAX_SEQ == 1 && defined(QMK_TC_BUILD) && QMK_TC_SEQS > 1

constexpr int LPS = 32 / TC_SEQS;              // lanes per sequence in the merge = most splits of a sequence
constexpr int TPS = CONS_THREADS / TC_SEQS;    // threads per sequence where a thread finishes one row
static_assert(LPS <= MAX_SPLITS, "exchange area");
static_assert(CH_ROWS * ((QKV_CHUNKS + TC_MIN_CTAS - 1) / TC_MIN_CTAS) <= TPS && TPS >= 64, "one row per thread");
// Every phase but attention has at most as many chunks as the ring has slots (see the ring's parity rule).
static_assert(2 * ((GU_CHUNKS + TC_MIN_CTAS - 1) / TC_MIN_CTAS) <= NSLOTS && (QKV_CHUNKS + TC_MIN_CTAS - 1) / TC_MIN_CTAS <= NSLOTS,
              "a phase exceeds the ring");
static_assert(TC_SEQS * 2 * MAX_CTAS <= CONS_WARPS * 2 * PART_STRIDE, "argmax words alias the attention partials");
static_assert((O_COLS + TC_MIN_CTAS / O_GROUP - 1) / (TC_MIN_CTAS / O_GROUP) <= RESID_PITCH, "outputs of a CTA");

__device__ __forceinline__ float *tc_prev(const Ctx &c, int which, int b) {
  return (b < 2 ? c.f(F_X) : reinterpret_cast<float *>(c.smem + OFF_PREV2)) + (which * 2 + (b & 1)) * PREV_PITCH;
}
__device__ __forceinline__ float *tc_resid(const Ctx &c, int which, int b) {
  return reinterpret_cast<float *>(c.smem + OFF_RESID) + (which * TC_SEQS + b) * RESID_PITCH;
}
__device__ __forceinline__ int *tc_tokens(const Ctx &c) { return reinterpret_cast<int *>(c.smem + OFF_TOKENS); }
__device__ __forceinline__ int *tc_splits(const Ctx &c) { return reinterpret_cast<int *>(c.smem + OFF_TOKENS) + TC_SEQS; }   // of each sequence's attention in this step

__device__ __forceinline__ uint32_t qkv_phase_seqs(const Params &P, Ctx c, const RowTile &rows, uint32_t tag) {
  const TcTab *t = tctab(c);
  const int nch = t->nq, nkb = t->nkb_qkv;
  run_rows(c, rows, 0);
  cons_sync();
  const int b = c.tid / TPS, r = c.tid % TPS;
  if (b < P.nseq && r < nch * CH_ROWS) {
    const float *p = tc_part(c) + (r >> 4) * nkb * PART_TASK + b * 16 + (r & 15);
    float v = 0.f;
#pragma unroll
    for (int kb = 0; kb < CONS_WARPS; ++kb)
      if (kb < nkb) v += p[kb * PART_TASK];
    ll_store(P.ll + static_cast<size_t>(b) * LL_WORDS + LL_QKV + t->q0 * CH_ROWS + r, v * c.f(F_MISC)[M_XSCALE], tag);
  }
  return c.chunk + static_cast<uint32_t>(nch);
}

__device__ __forceinline__ uint32_t gateup_phase_seqs(const Params &P, Ctx c, const RowTile &rows) {
  const TcTab *t = tctab(c);
  const int nch = t->ng, nkb = t->nkb_gu;
  run_rows(c, rows, 10);
  cons_sync();
  const int b = c.tid / TPS, r = c.tid % TPS;
  __half *act16 = reinterpret_cast<__half *>(c.smem + OFF_ACT16) + 2 * b * ACT16_PITCH;
  if (r < 64) {          // a sequence's first warp holds its slice; rows past it multiply stale bytes: zero activations
    float a = 0.f;
    if (r < nch * CH_ROWS) {
      const int ru = up_row(nch, r);
      const float *pg = tc_part(c) + (r >> 4) * nkb * PART_TASK + b * 16 + (r & 15);
      const float *pu = tc_part(c) + (ru >> 4) * nkb * PART_TASK + b * 16 + (ru & 15);
      float g = 0.f, u = 0.f;
#pragma unroll
      for (int kb = 0; kb < CONS_WARPS; ++kb)
        if (kb < nkb) { g += pg[kb * PART_TASK]; u += pu[kb * PART_TASK]; }
      const float up = c.f(F_MISC)[M_XSCALE];
      g *= up;
      a = g / (1.0f + expf(-g)) * (u * up);
    }
    const uint32_t k = operand_exponent(a);
    if (r == 0) c.f(F_MISC)[M_ASCALE + b] = exp2_up(k);
    a *= exp2_down(k);
    act16[r] = split_half(a, false);
    act16[ACT16_PITCH + r] = split_half(a, true);
  }
  return c.chunk + static_cast<uint32_t>(2 * nch);
}

// merge_o for all sequences at once: a warp takes (quad of elements, sequence) pairs, lane 4 k + i element i and splits k, k + 8.
constexpr int SEQ_TASKS = (O_MAX_QUADS * TC_SEQS + CONS_WARPS - 1) / CONS_WARPS, SEQ_SPLITS = (LPS + 7) / 8;
static_assert(O_MAX_QUADS * TC_SEQS <= SEQ_TASKS * CONS_WARPS - 2, "the last two warps have a task less and fetch split weights instead");
__device__ __forceinline__ void merge_seqs(const Params &P, const Ctx &c, uint32_t tag) {
  const TcTab *t = tctab(c);
  float *s_wt = reinterpret_cast<float *>(c.smem + OFF_SPLITW);      // [2 heads][sequence][LPS splits]
  const int e0 = t->e0, ne = t->ne, h0 = e0 >> 7, el = c.lane & 3, sl = c.lane >> 2;
  constexpr int NW = SEQ_TASKS * SEQ_SPLITS;
  const unsigned long long *words = P.ll + LL_PART;
  uint32_t wp[NW], valid = 0;
#pragma unroll
  for (int i = 0; i < SEQ_TASKS; ++i) {
    const int task = c.warp + i * CONS_WARPS, q = task / TC_SEQS, b = min(task % TC_SEQS, P.nseq - 1), S = tc_splits(c)[b];
    const bool mine = task % TC_SEQS < P.nseq && 4 * q < ne;
    const int e = e0 + (4 * q < ne ? 4 * q : 0) + el;
    const uint32_t head = b * LL_WORDS + (e >> 7) * (MAX_SPLITS * PART_STRIDE) + (e & (D - 1));
#pragma unroll
    for (int k = 0; k < SEQ_SPLITS; ++k) {
      wp[i * SEQ_SPLITS + k] = head + min(sl + 8 * k, S - 1) * PART_STRIDE;
      if (mine && sl + 8 * k < S) valid |= 1u << (i * SEQ_SPLITS + k);
    }
  }
  float a[NW];
  if (ne > 0) {
    {   // one lane per warp watches the last split's word of the last sequence first (see merge_o)
      const int e = e0 + min(4 * c.warp, ne - 1);
      ll_sentinel(P, c, words + (P.nseq - 1) * LL_WORDS + ((e >> 7) * MAX_SPLITS + tc_splits(c)[P.nseq - 1] - 1) * PART_STRIDE + (e & (D - 1)), tag);
    }
    const int hw = h0 + (c.warp - (CONS_WARPS - 2));                // head whose split weights this warp makes (last two warps)
    if (c.warp >= CONS_WARPS - 2 && hw <= ((e0 + ne - 1) >> 7)) {   // warp-uniform
      const int b = c.lane / LPS, s = c.lane % LPS, S = tc_splits(c)[min(b, P.nseq - 1)];
      const bool mine = b < P.nseq && s < S;
      constexpr int NL = NW - SEQ_SPLITS;
      uint32_t wl[NL + 2];
      float v[NL + 2];
#pragma unroll
      for (int k = 0; k < NL; ++k) wl[k] = wp[k];
      wl[NL] = min(b, P.nseq - 1) * LL_WORDS + (hw * MAX_SPLITS + min(s, S - 1)) * PART_STRIDE + D;
      wl[NL + 1] = wl[NL] + 1;
      ll_wait_words<NL + 2>(P, c, words, wl, valid | (mine ? 3u << NL : 0u), tag, v);
#pragma unroll
      for (int k = 0; k < NW; ++k) a[k] = k < NL ? v[k] : 0.f;
      const float m = mine ? v[NL] : -INFINITY, l = mine ? v[NL + 1] : 0.f;
      float M = m;
#pragma unroll
      for (int o = LPS / 2; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
      const float sc = (m == -INFINITY) ? 0.f : exp2f(m - M);
      float L = l * sc;
#pragma unroll
      for (int o = LPS / 2; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
      s_wt[(hw - h0) * 32 + c.lane] = mine ? sc / L : 0.f;
    } else {
      ll_wait_words<NW>(P, c, words, wp, valid, tag, a);
    }
  }
  cons_sync();
  __half *act16 = reinterpret_cast<__half *>(c.smem + OFF_ACT16);
  float A[SEQ_TASKS];
#pragma unroll
  for (int i = 0; i < SEQ_TASKS; ++i) {
    const int task = c.warp + i * CONS_WARPS, q = task / TC_SEQS, b = task % TC_SEQS;
    const int e = e0 + (4 * q < ne ? 4 * q : 0) + el;
    A[i] = 0.f;
#pragma unroll
    for (int k = 0; k < SEQ_SPLITS; ++k)
      if (valid & (1u << (i * SEQ_SPLITS + k))) A[i] = fmaf(a[i * SEQ_SPLITS + k], s_wt[((e >> 7) - h0) * 32 + b * LPS + sl + 8 * k], A[i]);
  }
#pragma unroll
  for (int o = 16; o > 2; o >>= 1)
#pragma unroll
    for (int i = 0; i < SEQ_TASKS; ++i) A[i] += __shfl_xor_sync(0xffffffffu, A[i], o);
#pragma unroll
  for (int i = 0; i < SEQ_TASKS; ++i) {     // (columns of sequences that do not exist: zero)
    const int task = c.warp + i * CONS_WARPS, q = task / TC_SEQS, b = task % TC_SEQS;
    if (4 * q < ne && sl < 2) act16[(2 * b + sl) * ACT16_PITCH + 4 * q + el] = split_half(A[i], sl != 0);
  }
  if (c.tid >= ne && c.tid < 32 * O_KPAIRS) {
#pragma unroll
    for (int r = 0; r < 2 * TC_SEQS; ++r) act16[r * ACT16_PITCH + c.tid] = __float2half_rn(0.f);
  }
}

// slice_o for all sequences: quad q of a fragment holds sequence q's sums.
__device__ __forceinline__ uint32_t slice_o_seqs(const Params &P, Ctx c) {
  const TcTab *t = tctab(c);
  const int ne = t->ne, nch = t->no;
  if (nch == 0) return c.chunk;
  const bool ok = wait_chunks(P, c, c.chunk, nch);
  if (ok) {
    const OSlice o = o_slice(c, smem_u32(c.smem + OFF_ACT16) + ((c.lane & 7) % (2 * TC_SEQS)) * (ACT16_PITCH * 2) + (c.lane >> 3) * 16, ne);
    const int b = c.lane & 3, j = c.lane >> 2;
    const bool live = b < P.nseq;
    const int n0 = t->n0, n1 = t->n1, out0 = t->oq * O_COLS;
    [[maybe_unused]] const float *scales = reinterpret_cast<const float *>(c.smem + (weight_rows(c, c.chunk + static_cast<uint32_t>(nch - 1)) - smem_u32(c.smem)));
    const float *resid = tc_resid(c, 1, live ? b : 0);
    float *prev = tc_prev(c, 0, live ? b : 0);
    unsigned long long *sum = P.red + (live ? b : 0) * RED_SUM_WORDS;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int tile = c.warp + u * CONS_WARPS;
      if (tile >= O_TILES) break;
      float v[2];
      slice_o_tile(c, o, tile, v);
      if (live) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int i = tile * 16 + (FP8_ROWS ? 2 * j + k : j + 8 * k), n = out0 + i;
          if (FP8_ROWS) v[k] *= scales[i];
          if (n >= n0 && n < n1) v[k] += resid[n - n0];
          const long long fx = __float2ll_rn(v[k] * RED_SCALE), fx_prev = __float2ll_rn(prev[i] * RED_SCALE);
          prev[i] = v[k];
          red_add_u64(sum + red_index(n), (static_cast<unsigned long long>(fx - fx_prev) << RED_CNT_BITS) + 1ull);
        }
      }
    }
  }
  __syncwarp();
  if (c.lane < nch) mbar_arrive_n(c.empty((c.chunk + static_cast<uint32_t>(c.lane)) % NSLOTS), EMPTY_UNITS / CONS_WARPS);
  return c.chunk + static_cast<uint32_t>(nch);
}

// slice_cols for all sequences: quad q of a fragment holds sequence q's hi and lo sums of two outputs, which its lanes
// scale and add into that sequence's residual sum where they are.
__device__ __forceinline__ uint32_t slice_cols_seqs(const Params &P, Ctx c) {
  const TcTab *t = tctab(c);
  const int nrows = t->ng * CH_ROWS;
  const int nch = (nrows + CH_ROWS - 1) / CH_ROWS + SCALE_CH;
  [[maybe_unused]] const float *scales = FP8_ROWS ? reinterpret_cast<const float *>(c.slot(c.chunk + static_cast<uint32_t>(nch - 1))) : nullptr;
  const bool two = nrows > 16;
  const bool ok = wait_chunks(P, c, c.chunk, nch);
  if (ok) {
    uint32_t bq[4];
    ldsm_x4(smem_u32(c.smem + OFF_ACT16) + ((c.lane & 7) % (2 * TC_SEQS)) * (ACT16_PITCH * 2) + (c.lane >> 3) * 16, bq);
    uint32_t arow[2];
    slice_row_addresses(c, nrows, arow);
    const int b = c.lane & 3, j = c.lane >> 2;
    const bool live = b < P.nseq;
    const int n0 = t->n0, n1 = t->n1;
    const float up = c.f(F_MISC)[M_ASCALE + (live ? b : 0)];
    const float *resid = tc_resid(c, 0, live ? b : 0);
    float *prev = tc_prev(c, 1, live ? b : 0);
    unsigned long long *sum = P.red + (TC_SEQS + (live ? b : 0)) * RED_SUM_WORDS;
    float acc[SLICE_TILES][4];
    slice_tiles(arow, bq, c.warp, two, acc);
#pragma unroll
    for (int u = 0; u < SLICE_TILES; ++u) {
      const int tile = c.warp + u * CONS_WARPS;
      if (live && tile < H / 16) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int n = tile * 16 + (FP8_ROWS ? 2 * j + k : j + 8 * k);
          float v = fmaf(acc[u][2 * k + 1], LO_INV, acc[u][2 * k]) * up;
          if (FP8_ROWS) v *= scales[n];
          if (n >= n0 && n < n1) v += resid[n - n0];
          const long long fx = __float2ll_rn(v * RED_SCALE), fx_prev = __float2ll_rn(prev[n] * RED_SCALE);
          prev[n] = v;
          red_add_u64(sum + red_index(n), (static_cast<unsigned long long>(fx - fx_prev) << RED_CNT_BITS) + 1ull);
        }
      }
    }
  }
  __syncwarp();
  if (c.lane < nch) mbar_arrive_n(c.empty((c.chunk + static_cast<uint32_t>(c.lane)) % NSLOTS), EMPTY_UNITS / CONS_WARPS);
  return c.chunk + static_cast<uint32_t>(nch);
}

// The 1024 values per sequence that the consumer threads hold (v[b][j] = element tid + 384 j) -> RMS-normalised operand
// halves; the residual stream keeps the outputs this CTA owns.  Two consumer barriers.
constexpr int VPT = (H + CONS_THREADS - 1) / CONS_THREADS;
__device__ __forceinline__ void normalise_seqs(const Ctx &c, const float (&v)[TC_SEQS][VPT], int which, const __half *norm_w) {
  float *red = reinterpret_cast<float *>(c.smem + OFF_REDM);
#pragma unroll
  for (int b = 0; b < TC_SEQS; ++b) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) ss = fmaf(v[b][j], v[b][j], ss);
    ss = warp_sum(ss);
    if (c.lane == 0) red[b * CONS_WARPS + c.warp] = ss;
  }
  const int n0 = tctab(c)->n0, n1 = tctab(c)->n1;
  float w[VPT];
  bool big = false;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int n = c.tid + j * CONS_THREADS;
    w[j] = n < H ? __half2float(norm_w[n]) : 0.f;
    big |= fabsf(w[j]) > NORM_W_LIMIT;
  }
  big = cons_any(big);
  if (c.tid == 0) c.f(F_MISC)[M_XSCALE] = big ? NORM_UP : 1.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) w[j] *= big ? NORM_DOWN : 1.f;
#pragma unroll
  for (int b = 0; b < TC_SEQS; ++b) {
    const float4 *r = reinterpret_cast<const float4 *>(red + b * CONS_WARPS);
    const float4 r0 = r[0], r1 = r[1], r2 = r[2];
    const float tot = (((r0.x + r0.y) + (r0.z + r0.w)) + ((r1.x + r1.y) + (r1.z + r1.w))) + ((r2.x + r2.y) + (r2.z + r2.w));
    const float rstd = rsqrtf(tot * (1.0f / H) + RMS_EPS);
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int n = c.tid + j * CONS_THREADS;
      if (n < H) {
        const float xn = v[b][j] * rstd * w[j];
        *reinterpret_cast<__half *>(c.smem + OFF_XF + xf_offset(n, 0, b)) = split_half(xn, false);
        *reinterpret_cast<__half *>(c.smem + OFF_XF + xf_offset(n, 1, b)) = split_half(xn, true);
        if (n >= n0 && n < n1) tc_resid(c, which, b)[n - n0] = v[b][j];
      }
    }
  }
  cons_sync();
}

// Contributions that may still be missing from the watched word when a warp goes on to fetch all its words: with several
// sequences the adds drain for longer, and the fetch's round trip fits into the rest of it (four sequences, us per step at
// 64 / 1024 / 2048 tokens: 0: 812 / 932 / 1034, 16: 771 / 896 / 981, 48: 725 / 844 / 953, with the watch in front of the merge 712 / 812 / 928; 147: no better; all with full lines of sums, see RED_GROUP).
// One sequence gains nothing.  (Those figures are from sums of one contribution per CTA; a word of x1 has a quarter of that now, so that
// only x2 is watched.)
constexpr unsigned long long SUM_SLACK = 48;
// red_wait_norm for all sequences: which = 0: x1, 1: x2 (kept as the residual of the next layer's O slice, x).
__device__ __forceinline__ void red_wait_norm_seqs(const Params &P, const Ctx c, int which, uint32_t use, const __half *norm_w) {
  const unsigned long long base = static_cast<unsigned long long>(use) * static_cast<unsigned long long>(which ? c.ncta : tctab(c)->groups);
  const unsigned long long *src = P.red + static_cast<size_t>(which) * TC_SEQS * RED_SUM_WORDS + red_index(c.tid);
  if (c.lane == 0) {   // one lane per warp watches one word (see red_wait_norm)
    const unsigned long long *p = src + static_cast<size_t>(P.nseq - 1) * RED_SUM_WORDS;
    uint32_t n = 0;
    while (((base - ll_load(p)) & RED_CNT_MASK) > SUM_SLACK) {
      if ((++n & 1023u) == 0u && (c.flags()[0] || ld_relaxed_u32(P.status) != 0u)) break;   // the full wait below reports time-outs
      if (n > (1u << 22)) break;
    }
  }
  __syncwarp();
  unsigned long long w[TC_SEQS * VPT];
  uint32_t valid = 0;
#pragma unroll
  for (int b = 0; b < TC_SEQS; ++b)
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = b * VPT + j;
      w[i] = base;
      if (b < P.nseq && c.tid + j * CONS_THREADS < H) { valid |= 1u << i; w[i] = ll_load(src + b * RED_SUM_WORDS + j * RED_STEP); }
    }
  uint32_t pending = valid, it = 0;
  unsigned long long t0 = 0;
  for (;;) {
#pragma unroll
    for (int i = 0; i < TC_SEQS * VPT; ++i)
      if ((pending & (1u << i)) && ((w[i] - base) & RED_CNT_MASK) == 0ull) pending &= ~(1u << i);
    if (pending == 0u) break;
#pragma unroll
    for (int b = 0; b < TC_SEQS; ++b)
#pragma unroll
      for (int j = 0; j < VPT; ++j)
        if (pending & (1u << (b * VPT + j))) w[b * VPT + j] = ll_load(src + b * RED_SUM_WORDS + j * RED_STEP);
    if ((++it & 255u) == 0u) {
      if (c.flags()[0]) break;
      if (ld_relaxed_u32(P.status) != 0u) { c.flags()[0] = 1; break; }
      const unsigned long long t = now_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > P.timeout_ns) { raise_error(P, c, QMK_ERR_WAIT_TIMEOUT, WHERE_LL); break; }
    }
  }
  float v[TC_SEQS][VPT];
#pragma unroll
  for (int b = 0; b < TC_SEQS; ++b)
#pragma unroll
    for (int j = 0; j < VPT; ++j)   // words that are not this thread's stayed at `base`: zero
      v[b][j] = static_cast<float>(static_cast<long long>(w[b * VPT + j] - base) >> RED_CNT_BITS) * RED_INV_SCALE;
  normalise_seqs(c, v, which, norm_w);
}

__device__ __forceinline__ void embed_norm_seqs(const Params &P, const Ctx c, const __half *norm_w) {
  float v[TC_SEQS][VPT];
#pragma unroll
  for (int b = 0; b < TC_SEQS; ++b) {
    const unsigned char *erow = reinterpret_cast<const unsigned char *>(P.embed) + static_cast<size_t>(tc_tokens(c)[b]) * ROW_BYTES;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int n = c.tid + j * CONS_THREADS;
      v[b][j] = (n < H && b < P.nseq) ? embed_value(erow, n) : 0.f;
    }
  }
  normalise_seqs(c, v, 1, norm_w);
}

// lm_head_tc for all sequences: thread 16 b + r finishes row r of every tile for sequence b and keeps its running best;
// the sixteen lanes of a sequence then agree and publish the CTA's pair.
__device__ __forceinline__ uint32_t lm_head_seqs(const Params &P, Ctx c, int step, uint32_t atag) {
  const TcTab *t = tctab(c);
  const int nch = t->nlm, ntiles = (nch + TILE_CH - 1) / TILE_CH;
  float *part = tc_part(c);
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  const int p0 = k_split(c.warp, CONS_WARPS), p1 = k_split(c.warp + 1, CONS_WARPS);
  const int b = c.tid >> 4, r = c.tid & 15;
  const float up = c.f(F_MISC)[M_XSCALE];
  float *dump = (P.logits_out && b < P.nseq) ? P.logits_out + (static_cast<size_t>(b) * P.num_steps + step) * P.vocab : nullptr;
#pragma unroll 1
  for (int tile = 0; tile < ntiles; ++tile) {
    float *pr = part + (tile & 1) * (CONS_WARPS * PART_TASK);
    run_tile(c, prepare_tile(P, c, c.chunk + static_cast<uint32_t>(tile * TILE_CH), min(16, (nch - tile * TILE_CH) * CH_ROWS), p0, p1,
                             EMPTY_UNITS / CONS_WARPS), pr + c.warp * PART_TASK);
    cons_sync();
    if (b < P.nseq) {
      const int row = tile * 16 + r;
      if (row < nch * CH_ROWS) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < CONS_WARPS; ++w) v += pr[w * PART_TASK + c.tid];
        v *= up;
        const int o = t->lm0 * CH_ROWS + row;
        if (v > best) { best = v; best_i = o; }     // rows ascend per thread: strict > keeps the lowest index
        if (dump) dump[o] = v;
      }
    }
  }
  if (c.warp < TC_SEQS / 2) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
      if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    if (r == 0 && b < P.nseq) {
      unsigned long long *words = P.ll + static_cast<size_t>(b) * LL_WORDS + LL_AMAX + 2 * c.cta;
      ll_store(words, best, atag);
      ll_store(words + 1, __int_as_float(best_i), atag);
    }
  }
  return c.chunk + static_cast<uint32_t>(nch);
}

// argmax_exchange for all sequences: the winning rows end up in tc_tokens().
__device__ __forceinline__ void argmax_seqs(const Params &P, const Ctx c, uint32_t atag) {
  float *s_amax = c.f(F_WPART);                     // [sequence][2 * MAX_CTAS], free outside the attention phase
  const int b = c.tid / TPS;
  if (b < P.nseq) {
#pragma unroll 1
    for (int i = c.tid % TPS; i < 2 * c.ncta; i += TPS)
      s_amax[b * 2 * MAX_CTAS + i] = ll_wait(P, c, P.ll + static_cast<size_t>(b) * LL_WORDS + LL_AMAX + i, atag);
  }
  cons_sync();
  if (c.warp < P.nseq) {
    const float *am = s_amax + c.warp * 2 * MAX_CTAS;
    float bv = -INFINITY;
    int bi = 0x7fffffff;
#pragma unroll 1
    for (int k = c.lane; k < c.ncta; k += 32) {
      const float v = am[2 * k];
      const int vi = __float_as_int(am[2 * k + 1]);
      if (v > bv || (v == bv && vi < bi)) { bv = v; bi = vi; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (c.lane == 0) tc_tokens(c)[c.warp] = bi;
  }
}

__global__ void __launch_bounds__(THREADS, 1) qwen3_decode_megakernel_tc_seqs(const __grid_constant__ Params P) {
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
  tc_setup(P, c);
  if (c.tid == 64) {
    // sequence b owns CTAs [8 s_cap b, 8 s_cap (b + 1)): one attention item per CTA at most; the CTAs behind the last
    // sequence's have none
    TcTab *tt = reinterpret_cast<TcTab *>(smem + OFF_TCTAB);
    const int s_cap = max(1, min(LPS, c.ncta / (NKV * P.nseq)));
    const int b = c.cta / (NKV * s_cap);
    tt->s_cap = s_cap;
    tt->seq = min(b, P.nseq - 1);
    tt->local = b < P.nseq ? c.cta - b * NKV * s_cap : NKV * MAX_SPLITS;
    for (int i = 0; i < TC_SEQS; ++i) tc_tokens(c)[i] = per_seq(P.first_tokens, min(i, P.nseq - 1));
  }
  for (int i = c.tid; i < 2 * 2 * PREV_PITCH; i += THREADS) {
    c.f(F_X)[i] = 0.f;
    if (TC_SEQS > 2) reinterpret_cast<float *>(smem + OFF_PREV2)[i] = 0.f;
  }
  __syncthreads();
  c.llr = tc_ll(P, c);

  if (c.warp == CONS_WARPS) {
    producer_main_tc(P, c);
    __syncwarp();
  } else {
    const int start = per_seq(P.start_positions, tctab(c)->seq);
#pragma unroll 1
    for (int step = 0; step < P.num_steps; ++step) {
      const int pos = start + step;                      // of the sequence whose attention item this CTA has
      const uint32_t tag_base = (P.seq_base + static_cast<uint32_t>(step)) * 64u;
      if (c.tid < TC_SEQS) {
        const int token = tc_tokens(c)[c.tid];
        if (token < 0 || token >= P.vocab) { raise_error(P, c, QMK_ERR_BAD_TOKEN, WHERE_TOKEN); tc_tokens(c)[c.tid] = 0; }
        tc_splits(c)[c.tid] = max(1, min((per_seq(P.start_positions, min(c.tid, P.nseq - 1)) + step) / max(1, P.split_len), tctab(c)->s_cap));
      }
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
      cons_sync();      // tokens
      {
        const uint32_t L0 = static_cast<uint32_t>(step) * static_cast<uint32_t>(P.num_layers);
        mbar_wait(P, c, c.nfull(L0 & 1u), (L0 >> 1) & 1u, WHERE_FULL, false);
        embed_norm_seqs(P, c, c.norms(L0 & 1u) + NB_IN_LN);
      }
      RowTile rows = {};
      const bool early = EARLY_ROWS && tctab(c)->early;
#pragma unroll 1
      for (int layer = 0; layer < P.num_layers; ++layer) {
        const uint32_t tag = tag_base + static_cast<uint32_t>(layer) + 1u;
        const uint32_t Lg = static_cast<uint32_t>(step) * static_cast<uint32_t>(P.num_layers) + static_cast<uint32_t>(layer);
        const __half *nv = c.norms(Lg & 1u);
        const uint32_t use = Lg + 1u;
        QMK_STAMP(layer * 12 + 0);
        if (!early || layer == 0) rows = prepare_rows(P, c, tctab(c)->qkv);
        c.chunk = qkv_phase_seqs(P, c, rows, tag);
        QMK_STAMP(layer * 12 + 1);
        c.chunk = attention_tc(P, c, nv, layer, pos, tag);
        QMK_STAMP(layer * 12 + 2);
        merge_seqs(P, c, tag);
        QMK_STAMP(layer * 12 + 3);
        cons_sync();
        c.chunk = slice_o_seqs(P, c);
        QMK_STAMP(layer * 12 + 4);
        if (early) rows = prepare_rows(P, c, tctab(c)->gu);
        red_wait_norm_seqs(P, c, 0, use, nv + NB_POST_LN);
        QMK_STAMP(layer * 12 + 5);
        if (!early) rows = prepare_rows(P, c, tctab(c)->gu);
        c.chunk = gateup_phase_seqs(P, c, rows);
        QMK_STAMP(layer * 12 + 6);
        cons_sync();
        c.chunk = slice_cols_seqs(P, c);
        QMK_STAMP(layer * 12 + 7);
        const bool last = layer == P.num_layers - 1;
        if (!last) mbar_wait(P, c, c.nfull((Lg + 1u) & 1u), ((Lg + 1u) >> 1) & 1u, WHERE_FULL, false);
        if (early && !last) rows = prepare_rows(P, c, tctab(c)->qkv);
        red_wait_norm_seqs(P, c, 1, use, last ? P.final_norm : c.norms((Lg + 1u) & 1u) + NB_IN_LN);
        QMK_STAMP(layer * 12 + 8);
        if (cons_any(c.flags()[0] != 0)) break;
      }
      if (cons_any(c.flags()[0] != 0)) break;
      QMK_STAMP(P.num_layers * 12 + 0);
      c.chunk = lm_head_seqs(P, c, step, tag_base + 63u);
      QMK_STAMP(P.num_layers * 12 + 1);
      argmax_seqs(P, c, tag_base + 63u);
      const bool aborted = cons_any(c.flags()[0] != 0);
      QMK_STAMP(P.num_layers * 12 + 2);
      if (aborted) break;
      if (c.cta == 0 && c.tid < P.nseq) {
        int *log = per_seq(P.output_logs, c.tid);
        if (log) log[step] = tc_tokens(c)[c.tid];
      }
    }
    if (c.tid == 0) { c.flags()[3] = static_cast<int>(c.chunk); c.flags()[1] = 1; }
  }
  __syncthreads();
  tc_drain(P, c);
}

#endif
}  // namespace QMK_NS
