// Paged GQA decode attention over packed INT2/INT4 KV at head_dim 128, sm_100a.
//
// What it computes follows the reference decode's semantics (src/foscar/wrapper.py:1153-1171;
// fold algebra src/foscar/_sm100/int_fold_decode.py:5-22, 378-434): codes are never
// dequantized. For token t and query head h
//     score = s_k[t] * (q_h . c_k[t]) + z_k[t] * sum(q_h)          (times sm_scale)
//     out_h = ( sum_t w[t,h] c_v[t]  +  sum_t p[t,h] z_v[t] ) / sum_t p[t,h]
// with w = p * s_v * 2^lp stored as two E4M3 planes (hi + lo/16).
// The structure is this library's own. One persistent CTA per SM, 20 warps, 128-token tiles:
//
//   warps 16, 19  producers on alternate tiles: page ids fetched 32 at a time a chunk ahead; a
//                 tile's two pages (K codes, V codes, scale records) as 16-byte cp.async copies
//                 from all lanes into a deep shared-memory ring, completion on an mbarrier. The
//                 first producer also stages each work item's query rows.
//   warps 0-15    four worker groups, tile i -> group i % 4. A group carries its tile through
//                 every stage: thread t unpacks token t's K row to exact E4M3 bytes
//                 (code * 2^-9) straight into TENSOR MEMORY as the S MMA's A operand, unpacks its
//                 V row into the group's 128-byte-swizzled shared-memory stage, folds the scales
//                 into S row t, joins the group's column max, writes its P row; one tile later
//                 thread d adds channel d of the tile's O to the group's accumulators. Each
//                 group keeps its own running (m, l, c, O); they are merged once per work item.
//   warp 17       S issuer:  S[128 tok x 16] = C_K . Q^T   (A from tensor memory)
//   warp 18       PV issuer: O^T[128 ch x 16] = C_V^T . [P_hi | P_lo]
//
// Why one group per tile rather than a role per stage: the kernel is bound by instruction issue
// and by hand-off latency, not by arithmetic. With separate unpack and softmax roles every tile
// crossed seven mbarrier hand-offs per warp and 28 warps walked the tile list; measured with all
// arithmetic removed, that skeleton alone took 70% of the launch time. Here a tile costs each of
// its four warps three waits (codes landed, S done, previous PV done) and three arrivals, the
// group's K stage, S, V stage, P rows and O need no barrier of their own (the group itself was
// their last reader), and a group's chain of dependent latencies (~2600 cycles a tile)
// overlaps with the other three groups'.
// The hand-offs are kept to few instructions: every role runs as whole converged warps, waits vote
// so that their branch is uniform, single-lane work (arrivals, MMAs, commits) is predicated by
// elect.sync inside one asm block, ring stages and barriers sit at compile-time offsets, and values
// that are the same in a warp are told to the compiler (uniform()), because tensor-memory, barrier
// and descriptor operands have to be in uniform registers. A tile took 1930 warp instructions with
// lane-0 branches and run-time offsets and takes 1575; side by side 32 requests of 4K-32K tokens (INT2,
// 32/8 heads) went from 107.7 to 98.9 us, 16 requests of 8K-16K with two query tokens from 67.8 to
// 57.4. Three, five and six groups measure the same or slower (the registers they cost), and so does
// one MMA in place of a chain of four: what is left is the instructions' own latency at five warps a
// scheduler.
// Every role walks the same list of work items, so the pipeline never drains inside an item.
// Byte-expansion yields channels in a fixed permuted order; Q is loaded in that order and O is
// stored through it, so no per-element fix-up exists anywhere.
//
// Variants of the same code (template parameters):
//   KG == 2       K quantized over two 64-channel groups: query rows 0-7 carry the heads against
//                 the first group's half of the row, rows 8-15 against the second's, which puts
//                 each group's partial score in its own column.
//   KG == 3       whole-head K with bf16 record pairs (8 bytes a token) instead of f32 (16).
// Split units are merged inside this launch: a piece that wrote partials is counted in on its
// unit's counter one tile into the CTA's next item (or after its last), once every worker warp
// has reported its stores of the piece on a barrier, and the CTA that completes the count merges
// the unit (merge_unit_partials).
// The ring's stage count is even, so that each stage belongs to one of the two producers.
#include "decode.cuh"

namespace fq {

namespace {

// Barrier words of a CTA, at fixed offsets: one per ring stage and direction, one per query stage
// and direction, and per worker group
//   k_ready : the tile's K operand is in tensor memory (the group's four warps)
//   s_done  : the tile's S MMA is complete (commit)
//   pv_ready: the tile's V operand and P rows are in shared memory (the group's four warps); the
//             group has by then read the O of its previous tile
//   pv_done : the tile's PV MMA is complete (commit): O can be read, and the group's V stage and P
//             rows are free
// A group's n-th tile uses phase n & 1. stored: every worker warp has issued its output or partial
// stores of the work item (one phase per item): what orders a split piece's partials before its
// count-in. Every hand-off between roles is one of these words, so that its wait is bounded and a
// role that gave up cannot keep another from ending. (Named barriers, whose waits nothing can end,
// stay among the worker groups: those execute the same ones whatever their waits returned. With one
// for the K operand a group that had given up could arrive twice before the issuer did once, which
// was then a warp short for good.)
template <int G, int NS>
struct Bars {
  uint32_t base;
  __device__ uint32_t ring_full(int s) const { return base + 8u * s; }
  __device__ uint32_t ring_empty(int s) const { return base + 8u * (NS + s); }
  __device__ uint32_t q_full(int s) const { return base + 8u * (2 * NS + s); }
  __device__ uint32_t q_empty(int s) const { return base + 8u * (2 * NS + 2 + s); }
  __device__ uint32_t s_done(int g) const { return base + 8u * (2 * NS + 4 + g); }
  __device__ uint32_t pv_done(int g) const { return base + 8u * (2 * NS + 4 + G + g); }
  __device__ uint32_t pv_ready(int g) const { return base + 8u * (2 * NS + 4 + 2 * G + g); }
  __device__ uint32_t k_ready(int g) const { return base + 8u * (2 * NS + 4 + 3 * G + g); }
  __device__ uint32_t stored() const { return base + 8u * (2 * NS + 4 + 4 * G); }
  static constexpr int WORDS = 2 * NS + 5 + 4 * G;
};
// Named barriers: 0 the CTA, 1 .. G inside a group, 1 + G all groups.

// INT2 with whole-head K at head_dim 128: the K rows are unpacked like the V rows, at five instead
// of seven instructions a packed word (odd operand words hold 4 * code), and the idle half of the
// sixteen query rows takes the odd words' products into score columns 8-15.
__host__ __device__ constexpr bool odd_columns(int bits, int head_dim, int kg) {
  return bits == 2 && head_dim == 128 && kg != 2;
}

// Tensor-memory column plan (f32 columns): per worker group one K operand stage (a 128-byte row
// per lane), one S buffer and one O buffer of 16 columns.
template <int BITS, int D>
struct TmemPlan {
  static constexpr int G = WORKER_GROUPS;
  static constexpr int KOP_COLS = 32;
  static constexpr int S_COLS = 16;
  static constexpr int O_COLS = 16;
  static constexpr int KOP = 0;
  static constexpr int S = G * KOP_COLS;
  static constexpr int O = S + G * S_COLS;
  static constexpr int USED = O + G * O_COLS;
  static constexpr int ALLOC = USED <= 128 ? 128 : (USED <= 256 ? 256 : 512);
  static_assert(USED <= 512, "tensor memory plan exceeds 512 columns");
};

// The request's last tile with several query tokens per request: column h sees positions below
// len - lag(h) only. Out of line, so that this rare path (and column_lag's division) costs the
// tile loop nothing: the scores pass through local memory here and nowhere else. `pos` is the
// thread's token position. Returns, in `over`, the largest visible score.
template <int GP>
__device__ __noinline__ void mask_lagged_columns(const DecodeParams& P, int len, int ht, int pos,
                                                 float (&x)[GP], float& over) {
  float top = -INFINITY;
  for (int h = 0; h < GP; ++h) {
    if (pos >= len - column_lag(P, ht * 8 + h)) x[h] = -INFINITY;
    top = fmaxf(top, x[h]);
  }
  over = top;
}

// Worker role: one of four 128-thread groups. Group `wg` takes the tiles whose running index is
// `wg` modulo 4 and carries each of them through every stage itself: unpack K into tensor memory,
// unpack V into shared memory, fold the scales into the raw scores, softmax, write the P rows,
// and (one of its own tiles later) add the tile's O to its accumulators. The group keeps its own
// running (m, l, c, O); the four groups are merged once per work item.
template <int BITS, int D, int GP, int KG, bool MQ>
__device__ __forceinline__ void worker_role(const DecodeParams& P, uint8_t* smem, uint32_t smem0,
                                            uint32_t tmem,
                                            const Bars<SmemPlan<BITS, D>::G, SmemPlan<BITS, D>::NS>& bars,
                                            volatile int* abort_flag, const ItemRange items) {
  using SP = SmemPlan<BITS, D>;
  using TP = TmemPlan<BITS, D>;
  constexpr int G = SP::G, NS = SP::NS;
  const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int wg = warp >> 2, wq = warp & 3;
  const int t = threadIdx.x & 127;  // token row while unpacking and in softmax, channel in O
  int* status = P.a.status;
  const uint32_t lane_base = static_cast<uint32_t>(32 * wq) << 16;
  const uint32_t k_dst = tmem + lane_base + TP::KOP + wg * TP::KOP_COLS;
  const uint32_t s_src = tmem + lane_base + TP::S + wg * TP::S_COLS;
  constexpr bool ODD = odd_columns(BITS, D, KG);
  const uint32_t o_src = tmem + lane_base + TP::O + wg * TP::O_COLS;
  // (rows are 128 bytes at a 1024-byte aligned base: piece cc of the swizzled row is an xor away)
  const uint32_t v_row = (smem0 + SP::VOP_OFF + wg * SP::VOP_STAGE + t * SP::ROW) | ((t & 7) << 4);
  const uint32_t p_row = smem0 + SP::P_OFF + wg * SP::P_BYTES + t * 16;
  // the thread's code row in a ring stage, at its piece 0: piece v is an xor away
  const uint32_t code_row = t * SP::RB + (SP::row_swizzle(t) << 4);
  float* red_max = reinterpret_cast<float*>(smem + SP::RED_OFF);              // [wg][buf][warp][8]
  float* red_sum = reinterpret_cast<float*>(smem + SP::RED_OFF + 256 * G);    // [wg][warp][16]
  // this warp's copy of the item's per-head constants: sm_scale*log2e*q_descale, and that times
  // the sum of the head's query values
  float* head_k = reinterpret_cast<float*>(smem + SP::HEADK_OFF) + warp * 24;
  // written per work item by thread 0 of group 0: {pieces, request, KV head, head tile} of the
  // unit this CTA must merge (pieces 0: none)
  volatile int* merge_info = reinterpret_cast<volatile int*>(smem + SP::INFO_OFF);
  const volatile float* head_const =
      reinterpret_cast<const volatile float*>(smem + SP::HEADC_OFF);  // [2][24]
  constexpr float LN2 = 0.6931471805599453f;

  // pool-wide P-scale exponent from the count table: lp = 135 - max(top nonzero bin, 27)
  int lp;
  {
    int top = 0;
    if (P.p.v_max_hist != nullptr) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int bin = lane * 8 + i;
        if (__ldg(P.p.v_max_hist + bin) != 0u) top = bin;
      }
    }
    top = __reduce_max_sync(0xFFFFFFFFu, top);
    lp = 135 - max(top, 27);
  }
  // w = p * s_v * 2^lp must stay inside E4M3 with p up to 2^MAX_LAG (see the softmax below). A raised
  // reference is the maximum itself: every log2 unit above it would raise more seldom (three of them:
  // 97.2 us instead of 98.8 on 32 requests of 4K-32K tokens, INT2) but put all weights a bit lower in
  // the E4M3 window, whose step ends at 2^-13 (hi + lo/16): 16 x 100K tokens at INT4, against 64 bits,
  // 0.0219 with three units, 0.0077 with one, 0.0048 with none.
  constexpr float MAX_LAG = 3.f;
  lp -= static_cast<int>(MAX_LAG);
  // Below 2^NO_WEIGHT of the reference w is less than 56 * 2^-20 < 2^-14 and rounds to zero. Such a
  // token's z_v is left out with its codes (l keeps its p): value = s_v c + z_v has mean zero where
  // z_v alone, the row's minimum, has not, and 100K such tokens add up (0.0048 -> 0.0033 above).
  constexpr float NO_WEIGHT = -20.f;
  const float p2lp = exp2f(static_cast<float>(lp));
  const float o_mul = exp2f(static_cast<float>(9 - lp));

  auto merge_unit = [&](int k, int b, int kvh, int ht, int h0, int hstep) {
    merge_unit_partials<MQ, 1>(P, D, GP, channel_of_expanded_pos<BITS>(t), t == 0, k, b, kvh, ht, h0,
                          hstep);
  };
  // the split piece this CTA has written but not yet counted in (thread 0 of group 0 only)
  int pend_k = 0, pend_unit = 0, pend_b = 0, pend_kvh = 0, pend_ht = 0;
  uint32_t pend_phase = 0;   // phase of the `stored` barrier that covers the pending piece
  int seen = -1;        // the pending piece's count-in result; -1: not counted in yet
  bool count_due = false;    // (warp 0) a piece is pending and not counted in
  int this_k = 0;       // pieces of the current item's unit (fetched at the item's start)
  auto count_in = [&]() {
    count_due = false;
    if (lane == 0) {
      mbar_wait(bars.stored(), pend_phase, abort_flag, status);
      __threadfence();
      seen = atomicAdd(P.a.unit_counters + pend_unit, 1);
    }
    __syncwarp();
  };

  int qi = 0;       // non-empty items so far: which query stage holds the item's rows
  int it0 = 0;      // running index of the current item's first tile (every role counts alike)
  int mine = wg;    // running index of this group's next tile
  uint32_t ph = 0;  // phase of the group's barriers: flips with every tile
  // ring position of tile `mine`
  uint32_t stage = smem0 + SP::RING_OFF + wg * SP::STAGE;
  uint32_t full = bars.ring_full(wg), ring_ph = 0;
  const WorkItem* const item_cache = reinterpret_cast<const WorkItem*>(smem + SP::ITEM_OFF);
  const WorkItem* const item_more =
      reinterpret_cast<const WorkItem*>(smem + SP::RING_OFF + NS * SP::STAGE);
  for (int wi = items.begin, ik = 0; wi < items.end; wi += items.step, ++ik) {
    const WorkItem w = uniform_item(item_at(P, item_cache, item_more, SP::ITEM_SLOTS, ik, wi));
    const int nt = max(w.t1 - w.t0, 0);
    float m[GP], l[GP], c[GP], oacc[GP];
#pragma unroll
    for (int h = 0; h < GP; ++h) { m[h] = 0.f; l[h] = 0.f; c[h] = 0.f; oacc[h] = 0.f; }
    uint32_t unset = (1u << GP) - 1u;   // heads without a finite score so far: m is no reference
    // The item's per-head constants (score scale, and score scale times the sum of the head's
    // query values) were computed by the first producer when it staged the query rows, well
    // ahead of the tiles; the warp keeps its own copy, read back from shared memory each tile
    // instead of living in 16 registers of every thread.
    __syncwarp();   // the warp's reads of the previous item's values are over
    if (nt > 0) {
      // Only a group with a tile in the item waits for the item's query stage: the stage cannot
      // be restaged before that group's K row has gone through the S MMA. A group without a tile
      // would have nothing holding the producer back, and a phase-parity wait that falls two
      // stagings behind never returns.
      if (mine < it0 + nt) {
        const int qb = qi & 1;
        mbar_wait(bars.q_full(qb), (qi >> 1) & 1, abort_flag, status);
        if (lane < 24) head_k[lane] = head_const[qb * 24 + lane];
      }
      ++qi;
    }
    __syncwarp();
    bool pending = false;
    if (wg == 0 && t == 0 && w.slot >= 0 && P.a.unit_counters != nullptr) {
      const int unit = (w.b * P.p.num_kv_heads + w.kvh) * P.head_tiles + w.ht;
      this_k = P.a.split_counts != nullptr ? __ldg(P.a.split_counts + unit) : P.a.kv_splits;
    }

    // Add the group's previous tile's O (its PV MMA has had most of a tile's time to finish).
    // The wait also frees the group's V stage and P rows for the tile in hand.
    auto accumulate = [&]() {
      mbar_wait_warp(bars.pv_done(wg), ph ^ 1u, abort_flag, status);
      tc_fence_after();
      uint32_t r[16];
      tmem_ld16(o_src, r);
      tmem_ld_wait();
#pragma unroll
      for (int h = 0; h < GP; ++h)
        oacc[h] += fmaf(__uint_as_float(r[8 + h]), 0.0625f, __uint_as_float(r[h]));
    };

    // first position of the thread's row in the group's next tile; tiles up to `whole` lie
    // entirely inside what every column sees
    int pos0 = (w.t0 + (mine - it0)) * SP::TT + t;
    const int whole = w.len - (MQ ? P.q_len - 1 : 0) - SP::TT + t;
#pragma unroll 1
    for (; mine < it0 + nt; mine += G, pos0 += G * SP::TT) {
      mbar_wait_warp(full, ring_ph, abort_flag, status);
      // ---- K row -> tensor memory (the S MMA's A operand). The stage is free: this group read the
      // S of its previous tile, so that tile's MMA, the stage's last reader, is complete.
      {
        uint32_t wk[D * BITS / 32], op[D / 4];
        load_code_row<BITS, D>(stage + SP::K_OFF + code_row, wk);
        if constexpr (ODD) expand_words_v<BITS, D>(wk, op);
        else expand_words<BITS, D>(wk, op);
        tmem_st32(k_dst, op);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      mbar_arrive_elect(bars.k_ready(wg));
      if (pending) accumulate();
      // ---- V row -> the group's 128-byte-swizzled shared-memory stage (the PV MMA's A operand)
      {
        uint32_t wv[D * BITS / 32], op[D / 4];
        load_code_row<BITS, D>(stage + SP::V_OFF + code_row, wv);
        expand_words_v<BITS, D>(wv, op);
#pragma unroll
        for (int cc = 0; cc < D / 16; ++cc)
          st_shared_v4(v_row ^ (cc << 4), op[4 * cc], op[4 * cc + 1], op[4 * cc + 2], op[4 * cc + 3]);
      }
      // the token's record; then the ring stage goes back to the producers
      float sk, zk, sv, zv;
      float sk1 = 0.f, zk1 = 0.f;         // the second K group's pair (KG == 2)
      if constexpr (KG == 2) {            // K ring: (s, z) of both groups; V ring after the page's K ring
        uint32_t k0, k1, vr;
        const uint32_t slot = stage + SP::S_OFF + (t >> 6) * SP::SCALE_PAGE;
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(k0), "=r"(k1)
                     : "r"(slot + (t & 63) * 8));
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(vr) : "r"(slot + 8 * PAGE + (t & 63) * 4));
        sk = __uint_as_float(k0 << 16); zk = __uint_as_float(k0 & 0xFFFF0000u);
        sk1 = __uint_as_float(k1 << 16); zk1 = __uint_as_float(k1 & 0xFFFF0000u);
        sv = __uint_as_float(vr << 16); zv = __uint_as_float(vr & 0xFFFF0000u);
      } else if constexpr (KG != 3) {     // KG == 1: f32 records; KG == 3: bf16 pairs
        ld_shared_f4(stage + SP::S_OFF + t * 16, sk, zk, sv, zv);
      } else {   // (s, z) as bf16 pairs, 8 bytes a token, each page at its f32-sized slot
        uint32_t kr, vr;
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];"
                     : "=r"(kr), "=r"(vr)
                     : "r"(stage + SP::S_OFF + (t >> 6) * SP::SCALE_PAGE + (t & 63) * 8));
        sk = __uint_as_float(kr << 16); zk = __uint_as_float(kr & 0xFFFF0000u);
        sv = __uint_as_float(vr << 16); zv = __uint_as_float(vr & 0xFFFF0000u);
      }
      __syncwarp();
      mbar_arrive_elect(full + 8 * NS);   // ring_empty of the stage
      stage += G * SP::STAGE;
      full += 8 * G;
      if (full >= bars.ring_full(NS)) {
        stage -= NS * SP::STAGE;
        full -= 8 * NS;
        ring_ph ^= 1u;
      }
      // ---- raw scores: columns [0, GP), and [8, 8 + GP) where the rows' halves are split
      mbar_wait_warp(bars.s_done(wg), ph, abort_flag, status);
      tc_fence_after();
      uint32_t raw[(KG == 2 || ODD) ? 16 : GP];
      if constexpr (KG == 2 || ODD) tmem_ld16(s_src, raw);
      else if constexpr (GP == 4) tmem_ld4(s_src, raw);
      else tmem_ld8(s_src, raw);
      tmem_ld_wait();
      // Only a request's last tile has positions past its length: their scores become -inf and
      // their records are neutralised, so stale shared memory can never reach the output.
      // Scores are taken relative to the group's running reference m, which may lag the true
      // maximum by up to MAX_LAG (p <= 2^MAX_LAG; the P scale leaves that headroom below the E4M3
      // range). Only when some score of the tile exceeds that does the group exchange the exact
      // column maxima and rescale; the common tile costs one reducing barrier.
      float x[GP];
      float over = -INFINITY;
      // with several query tokens a column stops short of the request's last positions
      const bool inside = pos0 <= whole;   // (the same for the whole group)
      float hk[GP], hz[GP];
#pragma unroll
      for (int h = 0; h < GP; h += 4) {
        ld_shared_f4(smem_u32(head_k + h), hk[h], hk[h + 1], hk[h + 2], hk[h + 3]);
        ld_shared_f4(smem_u32(head_k + 8 + h), hz[h], hz[h + 1], hz[h + 2], hz[h + 3]);
      }
      const bool valid = inside || pos0 < w.len;
      float wsc = sv * p2lp;
      if (!valid) { wsc = 0.f; zv = 0.f; }
#pragma unroll
      for (int h = 0; h < GP; ++h) {
        float xv, s = __uint_as_float(raw[h]);
        if constexpr (ODD) s = fmaf(0.25f, __uint_as_float(raw[8 + h]), s);
        if constexpr (KG == 2)
          xv = fmaf(hk[h] * sk, s,
                    fmaf(hk[h] * sk1, __uint_as_float(raw[8 + h]),
                         fmaf(hz[h], zk, fmaf(head_k[16 + h], zk1, -m[h]))));
        else
          xv = fmaf(hk[h] * sk, s, fmaf(hz[h], zk, -m[h]));
        x[h] = valid ? xv : -INFINITY;
        over = fmaxf(over, x[h]);
      }
      if constexpr (MQ) {
        if (!inside) mask_lagged_columns<GP>(P, w.len, w.ht, pos0, x, over);
      }
      if (named_barrier_or(1 + wg, 128, over > (unset ? -INFINITY : MAX_LAG))) {
        float* wmax = red_max + ((wg * 2 + ph) * 4 + wq) * 8;
#pragma unroll
        for (int h = 0; h < GP; ++h) {
          const float wm = warp_max_f32(x[h]);
          if (lane == 0) wmax[h] = wm;
        }
        named_barrier(1 + wg, 128);
        const float* gm = red_max + (wg * 2 + ph) * 4 * 8;
#pragma unroll
        for (int h = 0; h < GP; ++h) {
          const float top = fmaxf(fmaxf(gm[h], gm[8 + h]), fmaxf(gm[16 + h], gm[24 + h]));
          const bool first = (unset >> h) & 1u;
          if (top > (first ? -INFINITY : MAX_LAG)) {   // (the same for the whole group)
            const float delta = top;
            // (a head's first reference: its sums are zero)
            const float corr = first ? 1.f : fast_exp2(-delta);
            unset &= ~(1u << h);
            m[h] += delta;
            l[h] *= corr;
            c[h] *= corr;
            oacc[h] *= corr;   // holds every earlier tile's O (added above)
            x[h] -= delta;
          }
        }
      }
      // p = 2^x, w = p * s_v 2^lp, four heads at a time as E4M3 hi + lo/16. (ex2 on f32: the
      // f16x2 form takes twice as long per instruction on this part, so it saves nothing.)
      uint32_t pw[4] = {};
#pragma unroll
      for (int h = 0; h < GP; h += 4) {
        __half2 w2[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int a = h + 2 * i;
          const float p0 = fast_exp2(x[a]), p1 = fast_exp2(x[a + 1]);
          l[a] += p0;
          l[a + 1] += p1;
          c[a] = fmaf(x[a] < NO_WEIGHT ? 0.f : p0, zv, c[a]);
          c[a + 1] = fmaf(x[a + 1] < NO_WEIGHT ? 0.f : p1, zv, c[a + 1]);
          w2[i] = __floats2half2_rn(p0 * wsc, p1 * wsc);
        }
        split_e4m3x4(w2[0], w2[1], pw[h >> 2], pw[2 + (h >> 2)]);
      }
      // the P row: bytes [hi_0..hi_7 | lo_0..lo_7]; with the V rows above they complete the PV MMA's
      // operands
      st_shared_v4(p_row, pw[0], pw[1], pw[2], pw[3]);
      fence_proxy_async();
      tc_fence_before();   // (orders the O read above before the PV MMA)
      __syncwarp();
      mbar_arrive_elect(bars.pv_ready(wg));
      pending = true;
      ph ^= 1u;
      // The previous split piece of this CTA is counted in here, a tile into the next item: its
      // partials have drained, and the fence and the atomic's round trip cost one thread of
      // one group a microsecond in mid-stream instead of stalling an item boundary. The wait
      // (long satisfied) is what orders every worker warp's partial stores before this
      // thread's release fence and atomic.
      if (count_due) count_in();
    }
    it0 += nt;
    if (pending) accumulate();

    // ---- item epilogue. First, the count-in of the previous split piece (see step 1 below)
    if (count_due) count_in();   // group 0 had no tile in this item
    // group sums, then the groups' states through shared memory
    float* rs = red_sum + (wg * 4 + wq) * 16;
#pragma unroll
    for (int h = 0; h < GP; ++h) {
      float ls = l[h], cs = c[h];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        ls += __shfl_xor_sync(0xFFFFFFFFu, ls, o);
        cs += __shfl_xor_sync(0xFFFFFFFFu, cs, o);
      }
      if (lane == 0) { rs[h] = ls; rs[8 + h] = cs; }
    }
    named_barrier(1 + wg, 128);
    const float* gs = red_sum + wg * 4 * 16;
#pragma unroll
    for (int h = 0; h < GP; ++h) {
      l[h] = (gs[h] + gs[16 + h]) + (gs[32 + h] + gs[48 + h]);
      c[h] = (gs[8 + h] + gs[24 + h]) + (gs[40 + h] + gs[56 + h]);
    }
    {   // every group leaves its state in shared memory
      float* xo = reinterpret_cast<float*>(smem + SP::XCHG_OFF + wg * SP::XCHG_STRIDE);
      float* xmeta = xo + TILE * 8;
#pragma unroll
      for (int h = 0; h < GP; ++h) xo[h * TILE + t] = oacc[h];   // head-major: no bank conflicts
      if (t == 0) {
#pragma unroll
        for (int h = 0; h < GP; ++h) {
          xmeta[h] = (unset >> h) & 1u ? -INFINITY : m[h];
          xmeta[8 + h] = l[h];
          xmeta[16 + h] = c[h];
        }
      }
    }
    named_barrier(1 + G, 128 * G);
    // The groups' states are merged in fixed order (group 0, then 1, 2, 3), each group taking a
    // share of the heads; the loop over the groups is unrolled so that its loads go out together.
    // (The results go to global memory only after the barrier below: a barrier that follows
    // global stores waits for them to be acknowledged, about 2 us under this load.)
    constexpr int HPG = (GP + G - 1) / G;   // heads a group merges
    float rM[HPG], rL[HPG], rO[HPG];
#pragma unroll
    for (int i = 0; i < HPG; ++i) {
      const int h = wg + i * G;
      float M = -INFINITY, L = 0.f, C = 0.f, O = 0.f;
      if (h < GP) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float* xo = reinterpret_cast<const float*>(smem + SP::XCHG_OFF +
                                                           g * SP::XCHG_STRIDE);
          const float* xmeta = xo + TILE * 8;
          const float m1 = xmeta[h], l1 = xmeta[8 + h], c1 = xmeta[16 + h];
          const float o1 = xo[h * TILE + t];
          const float Mn = fmaxf(M, m1);
          const float f0 = M == -INFINITY ? 0.f : exp2f(M - Mn);
          const float f1 = m1 == -INFINITY ? 0.f : exp2f(m1 - Mn);
          L = L * f0 + l1 * f1;
          C = C * f0 + c1 * f1;
          O = O * f0 + o1 * f1;
          M = Mn;
        }
        O = O * (o_mul * v_position_scale<BITS>(t)) + C;
      }
      rM[i] = M; rL[i] = L; rO[i] = O;
    }
    // ---- in-kernel merge, step 1. A split piece is counted in (release fence + one atomic on
    // its unit's counter) not here but a tile into the NEXT item (above), or after the last
    // item. Whoever finds the count complete makes the CTA merge that unit after the barrier
    // below.
    if (wg == 0 && t == 0) {
      int km = 0;
      if (pend_k > 0 && seen == pend_k - 1) {
        P.a.unit_counters[pend_unit] = 0;   // nobody touches it again before the next launch
        km = pend_k;
      }
      merge_info[0] = km; merge_info[1] = pend_b; merge_info[2] = pend_kvh; merge_info[3] = pend_ht;
      pend_k = 0;
      seen = -1;
      if (w.slot >= 0 && P.a.unit_counters != nullptr) {
        pend_unit = (w.b * P.p.num_kv_heads + w.kvh) * P.head_tiles + w.ht;
        pend_k = this_k;
        pend_b = w.b; pend_kvh = w.kvh; pend_ht = w.ht;
        pend_phase = static_cast<uint32_t>(ik & 1);
      }
    }
    if (warp == 0) count_due = w.slot >= 0 && P.a.unit_counters != nullptr;
    // the exchange buffers are reused by the next item
    named_barrier(1 + G, 128 * G);
    // ---- in-kernel merge, step 2: every group takes its share of the unit's heads (the words
    // are next written after the next item's first all-group barrier, which this read precedes)
    if (w.slot != -2) {
      const int ch = channel_of_expanded_pos<BITS>(t);
#pragma unroll
      for (int i = 0; i < HPG; ++i) {
        const int h = wg + i * G;
        const int hl = w.ht * 8 + h;
        if (h >= GP || hl >= P.heads_per_kv) continue;
        const float M = rM[i], L = rL[i], O = rO[i];
        const long long head = static_cast<long long>(w.kvh) * P.heads_per_kv + hl;
        const long long row = static_cast<long long>(w.b) * P.a.num_qo_heads + head;
        if (w.slot < 0) {
          const long long orow = caller_row<MQ>(P, w.b, w.kvh, hl);
          const float val = L > 0.f ? O / L * P.a.o_scale : 0.f;
          store_value(P.a.out, P.a.out_dtype, orow * D + ch, val);
          if (t == 0 && P.a.lse != nullptr)
            P.a.lse[orow] = L > 0.f ? (M + log2f(L)) * LN2 : -INFINITY;
        } else {
          const long long prow =
              static_cast<long long>(w.slot) * P.a.batch * P.a.num_qo_heads + row;
          P.a.o_partial[prow * D + ch] = O;
          if (t == 0) { P.a.l_partial[prow] = L; P.a.m_partial[prow] = M; }
        }
      }
    }
    // this warp's stores of the item are issued
    __syncwarp();
    if (lane == 0) mbar_arrive(bars.stored());
    if (merge_info[0] > 0)
      merge_unit(merge_info[0], merge_info[1], merge_info[2], merge_info[3], wg, G);
  }
  // The last split piece of this CTA is counted in here; if that completes its unit, the CTA
  // merges it (every group its share of the heads, as above).
  {
    volatile int* last_info = merge_info + 4;   // slow groups may still be reading merge_info
    if (wg == 0 && t == 0) {
      int km = 0;
      if (pend_k > 0) {
        if (seen < 0) {
          mbar_wait(bars.stored(), pend_phase, abort_flag, status);
          __threadfence();
          seen = atomicAdd(P.a.unit_counters + pend_unit, 1);
        }
        if (seen == pend_k - 1) {
          P.a.unit_counters[pend_unit] = 0;
          km = pend_k;
        }
      }
      last_info[0] = km; last_info[1] = pend_b; last_info[2] = pend_kvh; last_info[3] = pend_ht;
    }
    named_barrier(1 + G, 128 * G);
    if (last_info[0] > 0)
      merge_unit(last_info[0], last_info[1], last_info[2], last_info[3], wg, G);
  }
}

}  // namespace

template <int BITS, int D, int GP, int KG, bool MQ>
__global__ void __launch_bounds__(DECODE_THREADS, 1)
decode_kernel(const __grid_constant__ DecodeParams P) {
  // KG: 1 whole-head K with f32 records, 3 the same with bf16 pairs, 2 two 64-channel K groups
  static_assert(KG >= 1 && KG <= 3 && D == 128, "head_dim 128");
  using SP = SmemPlan<BITS, D>;
  using TP = TmemPlan<BITS, D>;
  constexpr int G = SP::G, NS = SP::NS;
  constexpr int W_PRODUCER = 4 * G, W_S = W_PRODUCER + 1, W_PV = W_PRODUCER + 2,
                W_PRODUCER2 = W_PRODUCER + 3;
  static_assert(DECODE_THREADS == 32 * (W_PRODUCER2 + 1), "warp roles and block size disagree");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* const smem = smem_raw + (smem0 - smem_u32(smem_raw));
  const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const Bars<G, NS> bars{smem0 + SP::BAR_OFF};
  static_assert(8 * Bars<G, NS>::WORDS <= 1016, "barrier words");
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SP::BAR_OFF + 1024);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SP::BAR_OFF + 1016);
  int* status = P.a.status;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    set_wait_budget(abort_flag, P.wait_budget);
    for (int s = 0; s < NS; ++s) {
      mbar_init(bars.ring_full(s), 32);  // one cp.async arrival per producer lane
      mbar_init(bars.ring_empty(s), 4);  // the four warps of the group that took the tile
    }
    for (int g = 0; g < G; ++g) {
      mbar_init(bars.k_ready(g), 4);
      mbar_init(bars.s_done(g), 1);
      mbar_init(bars.pv_done(g), 1);
      mbar_init(bars.pv_ready(g), 4);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bars.q_full(s), 1);
      mbar_init(bars.q_empty(s), 1);
    }
    mbar_init(bars.stored(), 4 * G);   // one arrival per worker warp
    fence_barrier_init();
  }
  if (warp == W_S) tmem_alloc(smem_u32(tmem_slot), TP::ALLOC);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(*tmem_slot);

  // Everything above touched only this CTA's shared and tensor memory. Under a programmatic
  // launch it may have run while the launch before this one in the stream was still finishing:
  // wait for that launch (complete and flushed) before the first global access, and let the
  // launch after this one start its own set-up as SMs free up. Both are no-ops otherwise.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  const ItemRange items = uniform_range(item_range(P));
  // The CTA's first items, decoded by one thread each: their dependent loads (row, length, table
  // offset) go out side by side, once, instead of in every role at every item boundary.
  WorkItem* const item_cache = reinterpret_cast<WorkItem*>(smem + SP::ITEM_OFF);
  WorkItem* const item_more = reinterpret_cast<WorkItem*>(smem + SP::RING_OFF + NS * SP::STAGE);
  {
    const int k = threadIdx.x;
    const long long wi = items.begin + static_cast<long long>(k) * items.step;
    if (k < P.item_slots && wi < items.end) {
      const WorkItem w = decode_item(P, static_cast<int>(wi));
      if (k < SP::ITEM_SLOTS) item_cache[k] = w;
      else item_more[k - SP::ITEM_SLOTS] = w;
    }
  }
  __syncthreads();
  const uint32_t ring0 = smem0 + SP::RING_OFF;

  if (warp == W_PRODUCER || warp == W_PRODUCER2) {
    // ------------------------------------------------------------------ producers
    // Two warps take alternate tiles. A tile's two pages (K codes, V codes, scale records of
    // one KV head) arrive as 16-byte cp.async copies issued by all 32 lanes: measured on B200,
    // a cp.async.bulk costs its issuing warp ~200 cycles whatever its size, so six 1-2 KB bulk
    // copies per tile cap the ring near 2.5 TB/s, while 20 cp.async per lane cost ~370 cycles.
    // Page ids are fetched 32 at a time, one per lane, a chunk ahead of the tiles that use them.
    // The first producer also stages each item's query rows, in expansion order, as the S MMA's
    // B operand; it runs a ring's depth ahead of the MMAs, which hides the load.
    const int pi = warp == W_PRODUCER ? 0 : 1;
    const uint64_t stream_policy = l2_evict_first_policy();
    // (the stage count is even: a producer's own tiles are two stages apart)
    uint32_t stage = ring0 + pi * SP::STAGE, full = bars.ring_full(pi), empty_ph = 1;
    // code chunks go to their swizzled place in the row (SmemPlan::row_swizzle); a lane's
    // 16 bytes are chunk lane % CHUNKS of row lane / CHUNKS (+ a multiple of 8 rows)
    const uint32_t code_lane = 16u * ((lane & ~(SP::CHUNKS - 1)) |
                                      ((lane & (SP::CHUNKS - 1)) ^ SP::row_swizzle(lane / SP::CHUNKS)));
    const uint64_t lane16 = 16u * lane;
    int it = 0, qi = 0;
    for (int wi = items.begin, ik = 0; wi < items.end; wi += items.step, ++ik) {
      const WorkItem w = uniform_item(item_at(P, item_cache, item_more, SP::ITEM_SLOTS, ik, wi));
      if (w.t1 <= w.t0) continue;
      constexpr int PPT = SP::PPT;   // pages per tile
      const int npages = (w.len + PAGE - 1) / PAGE;
      const int pend = min(PPT * w.t1, npages);
      auto fetch = [&](int pg0) {
        const int pg = pg0 + lane;
        int id = -1;
        if (pg < pend) {
          const long long e = static_cast<long long>(w.table_off) + pg;
          if (e >= 0 && e < P.a.table_len) id = __ldg(P.a.page_table + e);
          if (id < 0 || id >= P.p.num_pages) {
            id = -1;
            if (status) atomicOr(status, FQ_STATUS_BAD_PAGE);
          }
        }
        return id;
      };
      // (requested before the query rows are staged: the two global round trips overlap)
      int cur = fetch(PPT * w.t0);
      if (pi == 0) {
        const int qb = qi & 1;
        mbar_wait(bars.q_empty(qb), ((qi >> 1) & 1) ^ 1, abort_flag, status);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int chunk = lane + 32 * j;      // 16 rows of eight 16-byte chunks
          const int r = chunk >> 3, cc = chunk & 7;
          uint4 v = make_uint4(0, 0, 0, 0);
          // With two K groups of 64 channels rows 0-7 carry the heads against the first group's
          // half of the K row (bytes 0-63) and rows 8-15 the same heads against the second's.
          // INT2 with whole-head K: rows 0-7 carry the heads against the even operand words, rows
          // 8-15 the same heads against the odd ones, which hold 4 * code (expand_words_v).
          constexpr bool SPLIT = KG == 2, ODD = odd_columns(BITS, D, KG);
          const int hl = w.ht * 8 + (r & 7);        // head inside the KV head's group
          const bool live = (SPLIT || ODD || r < 8) && hl < P.heads_per_kv;
          const long long qrow = live ? caller_row<MQ>(P, w.b, w.kvh, hl) : 0;
          const bool mine = !SPLIT || (r < 8) == (cc < 4);
          float qsum = 0.f;
          if (live && mine) {
            const uint4 in = __ldg(reinterpret_cast<const uint4*>(
                static_cast<const uint8_t*>(P.a.q) +
                qrow * D + 16 * cc));
            const uint32_t words[4] = {in.x, in.y, in.z, in.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 lo = e4m3x2_to_f32x2(words[i] & 0xFFFF);
              const float2 hi = e4m3x2_to_f32x2(words[i] >> 16);
              qsum += (lo.x + lo.y) + (hi.x + hi.y);
            }
            if (BITS == 2) {
              v.x = __byte_perm(in.x, in.y, 0x6420);
              v.y = __byte_perm(in.z, in.w, 0x6420);
              v.z = __byte_perm(in.x, in.y, 0x7531);
              v.w = __byte_perm(in.z, in.w, 0x7531);
              if (ODD && r < 8) v.y = v.w = 0u;
              if (ODD && r >= 8) v.x = v.z = 0u;
            } else {
              v = in;
            }
          }
          *reinterpret_cast<uint4*>(smem + SP::Q_OFF + qb * SP::Q_BYTES + r * 128 +
                                    ((cc ^ (r & 7)) << 4)) = v;
          if (j < 2 || KG == 2) {
            // the row's eight chunks sit in eight neighbouring lanes: per-head constants
            // (rows 8-15: the second K group's query sums)
            qsum += __shfl_xor_sync(0xFFFFFFFFu, qsum, 1);
            qsum += __shfl_xor_sync(0xFFFFFFFFu, qsum, 2);
            qsum += __shfl_xor_sync(0xFFFFFFFFu, qsum, 4);
            if (cc == 0) {
              float scale = 0.f;
              if (live) {
                scale = P.a.sm_scale * 1.4426950408889634f;
                if (P.a.q_descale != nullptr)
                  scale *= caller_descale<MQ>(P, w.b, w.kvh, hl);
              }
              float* hc = reinterpret_cast<float*>(smem + SP::HEADC_OFF) + qb * 24;
              if (r < 8) {
                hc[r] = scale * 512.f;   // (a code byte is code * 2^-9)
                hc[8 + r] = scale * qsum;
              } else {
                hc[16 + (r - 8)] = scale * qsum;
              }
            }
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(bars.q_full(qb));
      }
      ++qi;
      // this producer's tiles of the item: every other one
      int k = (it ^ pi) & 1;
      it += w.t1 - w.t0;
      for (int base = PPT * w.t0; base < PPT * w.t1; base += 32) {
        const int nxt = base + 32 < PPT * w.t1 ? fetch(base + 32) : -1;
        const int stop = min(32, PPT * w.t1 - base);
#pragma unroll 1
        for (int pg = PPT * k; pg < stop; pg += 2 * PPT) {
          mbar_wait_warp(full + 8 * NS, empty_ph, abort_flag, status);
#pragma unroll
          for (int j = 0; j < PPT; ++j) {
            const int id = __shfl_sync(0xFFFFFFFFu, cur, pg + j);
            if (id < 0) continue;
            // (blocks are numbered below 2^32: one is at least 2.5 KB)
            const uint32_t blk = static_cast<uint32_t>(id) * P.p.num_kv_heads + w.kvh;
            const uint64_t off = static_cast<uint64_t>(blk) * SP::CODE_PAGE + lane16;
            const uint8_t* ks = P.p.k_codes + off;
            const uint8_t* vs = P.p.v_codes + off;
            // records: 16 B per token in an f32 pool, 8 B in a bf16 pool (same slot in the ring)
            // (with two K groups: 8 B of K pairs per token, then 4 B of V pairs per token)
            constexpr int scale_page =
                KG == 2 ? 12 * PAGE : (KG == 3 ? SP::SCALE_PAGE / 2 : SP::SCALE_PAGE);
            const uint8_t* ss = static_cast<const uint8_t*>(P.p.scales) +
                                (static_cast<uint64_t>(blk) * scale_page + lane16);
            const uint32_t dst = stage + code_lane, dst_rec = stage + 16 * lane;
#pragma unroll
            for (int c = 0; c < SP::CODE_PAGE; c += 512)
              cp_async16_stream(dst + SP::K_OFF + j * SP::CODE_PAGE + c, ks + c, stream_policy);
#pragma unroll
            for (int c = 0; c < SP::CODE_PAGE; c += 512)
              cp_async16_stream(dst + SP::V_OFF + j * SP::CODE_PAGE + c, vs + c, stream_policy);
#pragma unroll
            for (int c = 0; c < SP::SCALE_PAGE; c += 512)
              if (c + 512 <= scale_page || c + 16 * lane < scale_page)
                cp_async16_stream(dst_rec + SP::S_OFF + j * SP::SCALE_PAGE + c, ss + c,
                                  stream_policy);
          }
          cp_async_arrive(full);
          stage += 2 * SP::STAGE;
          full += 16;
          if (full >= bars.ring_full(NS)) {
            stage -= NS * SP::STAGE;
            full -= 8 * NS;
            empty_ph ^= 1u;
          }
        }
        cur = nxt;
      }
    }
    // every copy this warp issued has landed before the CTA's shared memory is released
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == W_S) {
    // ------------------------------------------------------------------ S issuer
    // The whole warp walks the tiles; one elected lane issues S = C_K . Q^T. The group index is
    // a counter, descriptor high words, the instruction descriptor and the accumulate flags are
    // immediates.
    constexpr uint32_t IDESC_S = make_idesc_e4m3(128, 16, 0, 0);
    constexpr uint32_t Q_HI = smem_desc_hi(1024, 2);
    int qi = 0, g = 0;   // tiles go to the groups in turn
    uint32_t gph = 0;    // phase of the groups' barriers: flips once per round of G tiles
    for (int wi = items.begin, ik = 0; wi < items.end; wi += items.step, ++ik) {
      const WorkItem w = uniform_item(item_at(P, item_cache, item_more, SP::ITEM_SLOTS, ik, wi));
      if (w.t1 <= w.t0) continue;
      const int qb = qi & 1;
      mbar_wait_warp(bars.q_full(qb), (qi >> 1) & 1, abort_flag, status);
      const uint32_t q_lo = smem_desc_lo(smem0 + SP::Q_OFF + qb * SP::Q_BYTES, 16);
#pragma unroll 1
      for (int t = w.t0; t < w.t1; ++t) {
        mbar_wait_warp(bars.k_ready(g), gph, abort_flag, status);
        tc_fence_after();
        umma_ts_chain4<Q_HI, IDESC_S>(tmem + TP::S + g * TP::S_COLS, tmem + TP::KOP + g * TP::KOP_COLS,
                                      q_lo, bars.s_done(g));
        if (++g == G) { g = 0; gph ^= 1u; }
      }
      tc_commit_elect(bars.q_empty(qb));   // after the item's last chain
      ++qi;
    }
  } else if (warp == W_PV) {
    // ------------------------------------------------------------------ PV issuer
    constexpr uint32_t IDESC_PV = make_idesc_e4m3(128, 16, 1, 1);
    constexpr uint32_t V_HI = smem_desc_hi(1024, 2), P_HI = smem_desc_hi(128, 0);
    const uint32_t v_lo0 = smem_desc_lo(smem0 + SP::VOP_OFF, 16);
    const uint32_t p_lo0 = smem_desc_lo(smem0 + SP::P_OFF, 128);
    int g = 0;
    uint32_t gph = 0;    // phase of the groups' barriers: flips once per round of G tiles
    for (int wi = items.begin, ik = 0; wi < items.end; wi += items.step, ++ik) {
      const WorkItem w = uniform_item(item_at(P, item_cache, item_more, SP::ITEM_SLOTS, ik, wi));
#pragma unroll 1
      for (int t = w.t0; t < w.t1; ++t) {
        mbar_wait_warp(bars.pv_ready(g), gph, abort_flag, status);
        tc_fence_after();
        const uint32_t v_lo = v_lo0 + g * (SP::VOP_STAGE >> 4);
        const uint32_t p_lo = p_lo0 + g * (SP::P_BYTES >> 4);
        const uint32_t od = tmem + TP::O + g * TP::O_COLS;
        umma_ss_chain4<V_HI, P_HI, IDESC_PV, (32 * SP::ROW >> 4), (32 * 16 >> 4)>(od, v_lo, p_lo);
        tc_commit_elect(bars.pv_done(g));
        if (++g == G) { g = 0; gph ^= 1u; }
      }
    }
  } else {
    // ------------------------------------------------------------------ workers
    worker_role<BITS, D, GP, KG, MQ>(P, smem, smem0, tmem, bars, abort_flag, items);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == W_S) {
    tc_fence_after();
    tmem_dealloc(tmem, TP::ALLOC);
  }
}

// Tensor-core self test (see foscar_b200.h): one tile of both contractions on given operands.
__global__ void __launch_bounds__(128, 1)
umma_selftest_kernel(int mode, const uint8_t* k_bytes, const uint8_t* q_bytes,
                     const uint8_t* v_bytes, const uint8_t* p_bytes, float* s_out, float* o_out,
                     int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* const smem = smem_raw + (smem0 - smem_u32(smem_raw));
  constexpr int KOFF = 0, VOFF = 16384, QOFF = 32768, POFF = 34816, MISC = 36864;   // MISC: barrier, tensor-memory slot, abort flag + wait budget
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + MISC + 16);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + MISC + 8);
  const uint32_t bar = smem0 + MISC;
  if (t == 0) {
    *abort_flag = 0;
    set_wait_budget(abort_flag, WAIT_BUDGET_CYCLES);
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  if (warp == 0) tmem_alloc(smem_u32(tmem_slot), 128);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lane_base = static_cast<uint32_t>(32 * warp) << 16;
  // operands: K row t (128 bytes), V row t, P row t, Q chunk
  uint32_t kr[32];
  for (int i = 0; i < 32; ++i) kr[i] = reinterpret_cast<const uint32_t*>(k_bytes + t * 128)[i];
  if (mode == 0) {
    for (int v = 0; v < 4; ++v) tmem_st8(tmem + lane_base + 8 * v, kr + 8 * v);
    tmem_st_wait();
  } else {
    for (int c = 0; c < 8; ++c)
      *reinterpret_cast<uint4*>(smem + KOFF + t * 128 + ((c ^ (t & 7)) << 4)) =
          make_uint4(kr[4 * c], kr[4 * c + 1], kr[4 * c + 2], kr[4 * c + 3]);
  }
  for (int c = 0; c < 8; ++c)
    *reinterpret_cast<uint4*>(smem + VOFF + t * 128 + ((c ^ (t & 7)) << 4)) =
        reinterpret_cast<const uint4*>(v_bytes + t * 128)[c];
  *reinterpret_cast<uint4*>(smem + POFF + t * 16) = reinterpret_cast<const uint4*>(p_bytes)[t];
  {
    const int r = t >> 3, c = t & 7;
    *reinterpret_cast<uint4*>(smem + QOFF + r * 128 + ((c ^ (r & 7)) << 4)) =
        reinterpret_cast<const uint4*>(q_bytes + r * 128)[c];
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  if (t == 0) {
    tc_fence_after();
    constexpr uint32_t IDESC_S = make_idesc_e4m3(128, 16, 0, 0);
    constexpr uint32_t IDESC_PV = make_idesc_e4m3(128, 16, 1, 1);
    for (int k = 0; k < 4; ++k) {
      const uint64_t bd = make_smem_desc(smem0 + QOFF + k * 32, 16, 1024, 2);
      if (mode == 0) {
        umma_ts(tmem + 32, tmem + k * 8, bd, IDESC_S, k > 0);
      } else {
        const uint64_t ad = make_smem_desc(smem0 + KOFF + k * 32, 16, 1024, 2);
        umma_ss(tmem + 32, ad, bd, IDESC_S, k > 0);
      }
    }
    for (int k = 0; k < 4; ++k) {
      const uint64_t ad = make_smem_desc(smem0 + VOFF + k * 4096, 16, 1024, 2);
      const uint64_t bd = make_smem_desc(smem0 + POFF + k * 512, 128, 128, 0);
      umma_ss(tmem + 48, ad, bd, IDESC_PV, k > 0);
    }
    tc_commit(bar);
  }
  mbar_wait(bar, 0, abort_flag, status);
  tc_fence_after();
  uint32_t r16[16];
  tmem_ld16(tmem + lane_base + 32, r16);
  tmem_ld_wait();
  for (int i = 0; i < 16; ++i) s_out[t * 16 + i] = __uint_as_float(r16[i]);
  tmem_ld16(tmem + lane_base + 48, r16);
  tmem_ld_wait();
  for (int i = 0; i < 16; ++i) o_out[t * 16 + i] = __uint_as_float(r16[i]);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 128);
  }
}

// Wait self test (see foscar_b200.h): every form of wait that the decode kernels' roles use, one
// after the other, each with the given cycle budget and for something that never comes: a barrier
// phase that nothing completes, waited for by single threads; a hand-off that is two of its four
// arrivals short, waited for by whole warps; and a shared-memory word that neither reaches nor equals
// what one thread of a warp waits for. The first waiter to run out raises the CTA's abort flag
// and FQ_STATUS_TIMEOUT; the others fall through; the kernel returns.
__global__ void __launch_bounds__(64, 1) wait_selftest_kernel(long long budget, int* status,
                                                              int* gave_up) {
  __shared__ __align__(8) unsigned long long bar_words[2];
  __shared__ __align__(8) int ctl_words[4];
  __shared__ int word;
  volatile int* abort_flag = ctl_words;
  const uint32_t alone = smem_u32(&bar_words[0]), handoff = smem_u32(&bar_words[1]);
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    set_wait_budget(abort_flag, budget);
    mbar_init(alone, 1);
    mbar_init(handoff, 4);
    word = 1;
    fence_barrier_init();
  }
  __syncthreads();
  int all = 1;
  auto next_form = [&]() {   // was the flag raised? down again for the next form
    __syncthreads();
    all &= *abort_flag;
    __syncthreads();
    if (threadIdx.x == 0) *abort_flag = 0;
    __syncthreads();
  };
  mbar_wait(alone, 0, abort_flag, status);    // runs out
  mbar_wait(alone, 0, abort_flag, status);    // returns at once: the CTA has given up
  next_form();
  mbar_arrive_elect(handoff);                 // (one a warp: two of four)
  mbar_wait_warp(handoff, 0, abort_flag, status);
  next_form();
  if (threadIdx.x % 32 == 0) count_wait<true>(&word, 2, abort_flag, status);
  next_form();
  if (threadIdx.x % 32 == 0) count_wait<false>(&word, 0, abort_flag, status);
  next_form();
  if (threadIdx.x == 0 && gave_up != nullptr) *gave_up = all;
}

}  // namespace fq

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
#include <algorithm>
#include <cstdlib>

namespace fq {

static int device_sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return sms > 0 ? sms : 148;
}

template <int BITS, int D, int GP, int KG = 1, bool MQ = false>
static int launch_decode(DecodeParams& P, cudaStream_t stream) {
  using SP = SmemPlan<BITS, D>;
  constexpr int THREADS = DECODE_THREADS, LIMIT = SMEM_LIMIT;
  P.tile_tokens = SP::TT;
  P.wait_budget = P.a.wait_budget_cycles > 0 ? P.a.wait_budget_cycles : WAIT_BUDGET_CYCLES;
  // Shared memory the ring leaves over holds more decoded work items (32 bytes each), up to
  // one per thread of the CTA's start-up pass.
  constexpr int spare = LIMIT - 1024 - SP::RING_OFF - SP::NS * SP::STAGE;
  constexpr int more = std::max(0, std::min(spare / 32, THREADS - SP::ITEM_SLOTS));
  P.item_slots = SP::ITEM_SLOTS + more;
  constexpr int smem = SP::RING_OFF + SP::NS * SP::STAGE + more * 32 + 1024;
  static bool configured[64] = {};  // per (BITS, D, GP) instantiation and device
  auto kernel = decode_kernel<BITS, D, GP, KG, MQ>;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         LIMIT);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  int ctas = P.a.max_ctas > 0 ? P.a.max_ctas : device_sm_count();
  int grid = P.a.worklist ? ctas : std::min(ctas, P.num_items);
  if (grid < 1) grid = 1;
  if (P.a.flags & 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, P));
  }
  kernel<<<grid, THREADS, smem, stream>>>(P);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace fq


using namespace fq;

extern "C" int fq_ctas_per_sm(int32_t bits, int32_t head_dim) {
  if ((bits != 2 && bits != 4) || (head_dim != 64 && head_dim != 128 && head_dim != 256))
    return FQ_ERR_UNSUPPORTED;
  return 1;
}

extern "C" int fq_tile_tokens(int32_t bits, int32_t head_dim) {
  if ((bits != 2 && bits != 4) || (head_dim != 64 && head_dim != 128 && head_dim != 256))
    return FQ_ERR_UNSUPPORTED;
  return tile_tokens(bits, head_dim);
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

extern "C" int fq_decode(const fq_pools* pools, const fq_decode_args* args, void* stream) {
  if (!pools || !args) return FQ_ERR_BAD_ARG;
  if (!pools->k_codes || !pools->v_codes || !pools->scales) return FQ_ERR_BAD_ARG;
  if (pools->num_kv_heads <= 0 || pools->num_pages <= 0) return FQ_ERR_BAD_ARG;
  // the kernels read these with 16-byte vector loads and copies
  if (!aligned16(pools->k_codes) || !aligned16(pools->v_codes) || !aligned16(pools->scales) ||
      !aligned16(args->q) || (args->worklist && !aligned16(args->worklist)))
    return FQ_ERR_BAD_ARG;
  // sub-head K groups: 64-channel groups at head_dim 128 (bf16 pair rings)
  if (pools->k_groups != 1 &&
      !(pools->k_groups == 2 && pools->head_dim == 128 && pools->scale_bf16))
    return FQ_ERR_UNSUPPORTED;
  if (pools->head_dim != 64 && pools->head_dim != 128 && pools->head_dim != 256)
    return FQ_ERR_UNSUPPORTED;
  if (pools->head_dim == 256 && pools->k_groups != 1) return FQ_ERR_UNSUPPORTED;
  if (pools->bits != 2 && pools->bits != 4) return FQ_ERR_UNSUPPORTED;
  const fq_decode_args& a = *args;
  if (a.batch <= 0 || a.num_qo_heads <= 0 || a.num_qo_heads % pools->num_kv_heads) return FQ_ERR_BAD_ARG;
  if (!a.seq_lens || !a.page_table || !a.table_offsets || !a.q || !a.out) return FQ_ERR_BAD_ARG;
  if (a.out_dtype < 0 || a.out_dtype > 2) return FQ_ERR_BAD_ARG;
  DecodeParams P{};
  P.p = *pools;
  P.a = a;
  // several query tokens per request ride as further columns of their KV head's unit
  P.q_len = a.q_len > 1 ? a.q_len : 1;
  if (P.q_len > 64) return FQ_ERR_BAD_ARG;
  P.gqa = a.num_qo_heads / pools->num_kv_heads;
  P.gqa_inv = ((1 << 20) + P.gqa - 1) / P.gqa;
  P.hq = a.num_qo_heads;
  if (P.gqa * P.q_len > 512) return FQ_ERR_TOO_LARGE;   // (column_token's range)
  P.heads_per_kv = P.gqa * P.q_len;
  P.a.num_qo_heads = a.num_qo_heads * P.q_len;
  P.head_tiles = (P.heads_per_kv + 7) / 8;
  // the separate merge launch writes rows in [B, HQ] order only
  if (P.q_len > 1 && (a.worklist ? a.max_splits > 1 : a.kv_splits > 1) && !a.unit_counters)
    return FQ_ERR_UNSUPPORTED;
  const long long units = static_cast<long long>(a.batch) * pools->num_kv_heads * P.head_tiles;
  if (a.worklist) {
    if (a.num_work <= 0 || a.max_splits < 1) return FQ_ERR_BAD_ARG;
    if (!a.o_partial || !a.l_partial || !a.m_partial) return FQ_ERR_BAD_ARG;
    P.num_items = a.num_work;  // capacity; the live row count is read from the list's header
  } else {
    if (a.kv_splits < 1) return FQ_ERR_BAD_ARG;
    if (a.kv_splits > 1 && (!a.o_partial || !a.l_partial || !a.m_partial ||
                            a.kv_splits > a.max_splits))
      return FQ_ERR_BAD_ARG;
    if (units * a.kv_splits > 0x7FFFFFFFLL) return FQ_ERR_TOO_LARGE;
    P.num_items = static_cast<int>(units * a.kv_splits);
  }
  const int gp = std::min(P.heads_per_kv, 8) <= 4 ? 4 : 8;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (pools->head_dim == 256) return launch_decode_wide(P, s);
  if (pools->head_dim == 64) {
    if (pools->k_groups != 1) return FQ_ERR_UNSUPPORTED;
    return launch_decode_stream(P, std::min(P.heads_per_kv, 8), s);
  }
#define FQ_DISPATCH(DD, KK, MM)                                                               \
  do {                                                                                        \
    if (pools->bits == 2)                                                                     \
      return gp == 4 ? launch_decode<2, DD, 4, KK, MM>(P, s)                                  \
                     : launch_decode<2, DD, 8, KK, MM>(P, s);                                 \
    return gp == 4 ? launch_decode<4, DD, 4, KK, MM>(P, s)                                    \
                   : launch_decode<4, DD, 8, KK, MM>(P, s);                                   \
  } while (0)
  // several query tokens per request: builds of their own for whole-head K (f32 or bf16
  // records), so that the one-token builds stay as they are
  if (P.q_len > 1) {
    if (pools->k_groups != 1) return FQ_ERR_UNSUPPORTED;
    if (pools->scale_bf16) FQ_DISPATCH(128, 3, true);
    FQ_DISPATCH(128, 1, true);
  }
  if (pools->k_groups == 2) FQ_DISPATCH(128, 2, false);
  if (pools->scale_bf16) FQ_DISPATCH(128, 3, false);
  FQ_DISPATCH(128, 1, false);
#undef FQ_DISPATCH
}

// ---------------------------------------------------------------------------------------------
// Split decode for callers that cannot allocate device memory
// ---------------------------------------------------------------------------------------------
namespace fq {
// Scratch for the split partials (o, l, m) of fq_decode_split_static. It lives in the library
// image: every GPU that loads the library holds these bytes until the process exits.
static __device__ __align__(256) float g_static_partials[FQ_STATIC_SCRATCH_BYTES / 4];
}  // namespace fq

extern "C" int fq_decode_split_static(const fq_pools* pools, const fq_decode_args* args,
                                      void* stream) {
  if (!pools || !args) return FQ_ERR_BAD_ARG;
  if (args->worklist != nullptr || args->kv_splits < 1) return FQ_ERR_BAD_ARG;
  if (args->batch <= 0 || args->num_qo_heads <= 0) return FQ_ERR_BAD_ARG;
  if (args->q_len > 1) return FQ_ERR_UNSUPPORTED;   // fq_merge below writes [B, HQ] rows
  const long long rows = static_cast<long long>(args->kv_splits) * args->batch * args->num_qo_heads;
  const long long need = rows * (pools->head_dim + 2) * 4;
  if (need > static_cast<long long>(FQ_STATIC_SCRATCH_BYTES)) return FQ_ERR_SCRATCH_TOO_SMALL;
  // In host code the array's name is only a handle: the device address is asked for once per
  // device, with that device current, and cached.
  static float* base_of_device[64] = {};
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 0 || dev >= 64) return FQ_ERR_UNSUPPORTED;
  if (base_of_device[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, fq::g_static_partials);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (p == nullptr) return FQ_ERR_UNSUPPORTED;
    base_of_device[dev] = static_cast<float*>(p);
  }
  fq_decode_args a = *args;
  a.unit_counters = nullptr;  // partials are merged by fq_merge below
  a.split_counts = nullptr;
  a.max_splits = a.kv_splits;
  a.o_partial = base_of_device[dev];
  a.l_partial = a.o_partial + rows * pools->head_dim;
  a.m_partial = a.l_partial + rows;
  const int rc = fq_decode(pools, &a, stream);
  if (rc != 0 || a.kv_splits == 1) return rc;
  return fq_merge(a.o_partial, a.l_partial, a.m_partial, nullptr, a.kv_splits, a.kv_splits,
                  a.batch, a.num_qo_heads, pools->num_kv_heads, pools->head_dim, a.o_scale, a.out,
                  a.out_dtype, a.lse, stream);
}


extern "C" int fq_umma_selftest(int32_t mode, const uint8_t* k_bytes, const uint8_t* q_bytes,
                                const uint8_t* v_bytes, const uint8_t* p_bytes, float* s_out,
                                float* o_out, int32_t* status, void* stream) {
  if (!k_bytes || !q_bytes || !v_bytes || !p_bytes || !s_out || !o_out) return FQ_ERR_BAD_ARG;
  const int smem = 36864 + 64 + 1024;
  cudaError_t e = cudaFuncSetAttribute(umma_selftest_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return static_cast<int>(e);
  umma_selftest_kernel<<<1, 128, smem, static_cast<cudaStream_t>(stream)>>>(
      mode, k_bytes, q_bytes, v_bytes, p_bytes, s_out, o_out, status);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int fq_wait_selftest(int64_t budget_cycles, int32_t* status, int32_t* gave_up,
                                void* stream) {
  if (budget_cycles < 1 || budget_cycles > WAIT_BUDGET_CYCLES) return FQ_ERR_BAD_ARG;
  wait_selftest_kernel<<<1, 64, 0, static_cast<cudaStream_t>(stream)>>>(budget_cycles, status,
                                                                         gave_up);
  return static_cast<int>(cudaGetLastError());
}
