// Paged GQA decode attention over packed INT2/INT4 KV at head_dim 64, sm_100a.
//
// Same arithmetic as the head_dim 128 kernel (decode.cu; reference semantics
// src/foscar/wrapper.py:1153-1171, fold algebra src/foscar/_sm100/int_fold_decode.py:5-22,
// 378-434), another structure: one persistent CTA per SM whose sixteen warps each stream their own
// chunks of 32 tokens, with no hand-off between warps until a work item ends.
//
//   chunks     the CTA's work items are one running list of chunks; chunk i goes to warp i % W.
//              A warp keeps a private ring of chunks in shared memory, filled by its own 16-byte
//              cp.async copies (K codes, V codes, records), page ids looked up sixteen and more
//              chunks ahead.
//   scores     S[16 tokens x 8 heads] = C_K . Q^T with the warp-level mma m16n8k16 on f16. ldmatrix
//              hands a lane packed words of its tokens, and a field masked out in place is an f16
//              subnormal, exactly code * 2^(position - 24); the place is divided out of the query
//              operand (exact: powers of two), which holds the query row in the fields' order.
//   softmax    a lane holds two heads' scores of its tokens. The heads' running references may lag
//              the true maxima by up to MAX_LAG (log2 units), so a chunk usually costs one vote.
//   output     O^T[16 channels x 8 heads] += C_V^T . W with the same mma: ldmatrix.trans delivers
//              pairs of tokens of one 16-bit piece of the code row, masked out as above; the
//              weights, p * s_v * 2^lp in f16, become its B operand by one 8 x 8 transpose.
//
// Four or fewer columns (GP == 4): columns 4-7 of a score tile are idle, so their lanes take tokens
// 8-15's scores and every lane works on half as many; the two token halves keep references of their
// own in O's columns 0-3 and 4-7 and become one when the item ends.
//
// Why warp-level mma here and tcgen05 at head_dim 128: a decode has at most eight columns, so the
// matrix work is small and the cost lies in feeding it. tcgen05 reads its operands from shared or
// tensor memory, so unpacked codes are written there and handed to an issuing warp; the warp-level
// form takes them from the unpacking registers, but on this part it is slow (m16n8k16 every 2.7 SM
// cycles, hardly overlapping other instructions) and its cost grows with the row: 32 of them per 32
// tokens at head_dim 128, 16 at head_dim 64, while softmax and hand-offs cost the same. Measured,
// start of either form against the other: 256 requests of 64-131072 tokens (INT2, 64/8 heads x 64)
// 517 us here and 595 us with tcgen05; at head_dim 128 32 requests of 4K-32K tokens (INT2) 115 and
// 97 us. Against the tcgen05 form's last build here one request of 4000 tokens (64/8 heads) takes 19.7
// us (18.3), 16 of 2000-16000 37.8 (45.0), 64 of 16384 132 (174).
//
// A work item ends with the warps' states (m, l, c, O) merged in the order of its first chunks'
// warps: each leaves its state in its shared-memory slot, counts itself in and goes on with its
// chunks of the next items; the warp that completes the count merges. A piece of a split unit is
// counted in on the unit's counter, and the piece that completes the unit merges it.
// Which warp takes which chunk depends on the plan alone, so results are reproducible bit by bit.
#include <algorithm>

#include "decode.cuh"

namespace fq {
namespace stream {

namespace {

constexpr int D = 64;              // head_dim
constexpr int CHUNK = 32;          // tokens of a chunk
// A warp's chunks looked up ahead: a ring of {page id, 2 * KV head + page half}, or {-1, NO_CHUNK}:
// no such chunk, or nothing valid in it (the page id is the caller's word as it stands, so no value
// of it can be the mark); then what the lanes remember of their walks over the items.
constexpr int AHEAD = 64;
constexpr int NO_CHUNK = -1;
constexpr int TABLE_BYTES = AHEAD * 8 + 32 * 12;
constexpr int SLOTS = 32;          // items that may be waiting for their last warps, by item % SLOTS
// A head's running reference may lag the true maximum by up to MAX_LAG (log2 units); when it is
// raised it is set HEADROOM above the maximum of the chunk, so that few chunks raise it.
constexpr float MAX_LAG = 3.f, HEADROOM = 3.f;

// Shared-memory plan. All offsets from a 128-byte aligned base.
template <int BITS, int GP>
struct StreamPlan {
  static constexpr int W = 16;                         // warps
  static constexpr int RB = D * BITS / 8;              // code row bytes
  static constexpr int CHUNKS = RB / 16;               // 16-byte pieces of a row
  static constexpr int CODE = CHUNK * RB;              // a chunk's K (or V) codes
  static constexpr int K_OFF = 0, V_OFF = CODE, R_OFF = 2 * CODE;
  static constexpr int STAGE = 2 * CODE + CHUNK * 16;
  static constexpr int MT = D / 16;                    // m-tiles of O^T
  static constexpr int QR = D / 8;                     // query operand registers
  static constexpr int NST = GP == 4 ? 2 * MT : 4 * MT;   // state registers of a lane
  static constexpr int STATE = NST * 128;              // a warp's O: GP heads x D, f32
  static_assert(CHUNKS == 1 || CHUNKS == 2, "one piece a row at INT2, two at INT4");
  // 16-byte piece c of ring row r sits at piece c ^ row_swizzle(r): the eight rows an ldmatrix
  // matrix reads at the same piece then fall on different banks
  __host__ __device__ static constexpr int row_swizzle(int row) {
    return CHUNKS == 2 ? (row >> 2) & 1 : 0;
  }
  static constexpr int CTL_OFF = 0;                    // abort flag and wait budget, counters
  static constexpr int META_OFF = 512;                 // per warp m, l, c of eight columns
  static constexpr int TABLE_OFF = META_OFF + W * 96;  // per warp: chunks looked up ahead
  static constexpr int ITEM_OFF = TABLE_OFF + W * TABLE_BYTES;
  static constexpr int ITEM_SLOTS = 16;
  static constexpr int STATE_OFF = (ITEM_OFF + ITEM_SLOTS * 32 + 127) / 128 * 128;
  static constexpr int RING_OFF = STATE_OFF + W * STATE;
  static constexpr int stages() {
    int s = (SMEM_LIMIT - 128 - RING_OFF) / (W * STAGE);
    return s < 6 ? s : 6;   // (the first sixteen page ids are waited for; later ones land in time up to 8)
  }
  static constexpr int S = stages();
  static_assert(S >= 2, "a warp's ring needs two stages");
  static constexpr int MORE_OFF = RING_OFF + W * S * STAGE;
};

// Words of the control block (32-bit indices).
constexpr int CTL_BUSY = 8;                 // per warp: its state slot waits to be merged
constexpr int CTL_COUNT = 32;               // per item slot: warps that left their state
constexpr int CTL_DONE = CTL_COUNT + SLOTS; // per item slot: items completed
static_assert((CTL_DONE + SLOTS) * 4 <= 512, "control block");

__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                        uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                              uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// 8 x 8 f16 matrix, row r in the lanes 4r .. 4r+3, transposed.
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t x) {
  uint32_t y;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t& a, uint32_t& b, uint32_t& c,
                                      uint32_t& d) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t& a, uint32_t& b, uint32_t& c,
                                        uint32_t& d) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm2(uint32_t addr, uint32_t& a, uint32_t& b) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(a), "=r"(b) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm2_t(uint32_t addr, uint32_t& a, uint32_t& b) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(a), "=r"(b) : "r"(addr) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// A field of the packed words as f16 subnormals: the 16-bit halves' field f (of NF) at its own bit
// position while that stays inside the 10 mantissa bits, else after one shift of the whole word.
template <int BITS>
struct Field {
  static constexpr int NF = 16 / BITS;                      // fields of a 16-bit piece
  static constexpr int LOW = BITS == 2 ? 5 : 2;             // fields read in place
  static constexpr int SHIFT = BITS * LOW;                  // 10 or 8
  static constexpr uint32_t MASK = BITS == 2 ? 0x00030003u : 0x000F000Fu;
  __device__ static __forceinline__ uint32_t get(uint32_t w, uint32_t shifted, int f) {
    return f < LOW ? (w & (MASK << (BITS * f))) : (shifted & (MASK << (BITS * (f - LOW))));
  }
  // what the field's values are too large by, as a power of two (on top of 2^-24)
  __device__ static __forceinline__ int bits_up(int f) { return BITS * (f < LOW ? f : f - LOW); }
};

// Where O^T's rows sit: (m-tile f, row half hi, lane row r) -> channel and field.
template <int BITS>
__device__ __forceinline__ int o_field(int f, int hi) {
  return BITS == 2 ? 2 * f + hi : f;
}
template <int BITS>
__device__ __forceinline__ int o_channel(int f, int hi, int r) {
  constexpr int NF = Field<BITS>::NF, WC = 32 / BITS;
  const int piece = BITS == 2 ? r : 8 * hi + r;
  const int F = (piece & 1) * NF + o_field<BITS>(f, hi);
  return WC * (piece >> 1) + F / 2 + (WC / 2) * (F % 2);
}

// Bounded wait until a word of shared memory satisfies a condition; all lanes follow lane 0.
// (the abort flag and the cycle budget sit at the start of the control block)
template <bool AT_LEAST>
__device__ __forceinline__ void warp_wait(volatile int* word, int want, volatile int* abort_flag,
                                          int* status) {
  if ((threadIdx.x & 31) == 0) {
    if (AT_LEAST ? *word < want : *word != want)
      count_wait<AT_LEAST>(word, want, abort_flag, status);
  }
  __syncwarp();
}

// Merge of a split unit's partials by one warp: the arithmetic and slot order of merge_kernel. All
// heads at once, a head's channels dealt to 32 / HP lanes (HP: 1, 4 or 8 heads), so that a merge
// costs a memory round trip for every SB slots: at most 32 values a lane. (One head after the other,
// lane by channel, costs two for every head; 64 values a lane in flight, or two or four heads at a
// time, cost registers of the chunk loop around the call or instructions that a short launch fetches
// for the first time. One request of 4000 tokens, INT2, 64/8 heads: 19.7 us, 22.9 a head at a time,
// 13.9 without any merge.)
// `rows_out`: HP x D floats of the warp's shared memory, through which whole rows are stored.
template <int HP>
__device__ __noinline__ void merge_unit_warp(const DecodeParams& P, int k, int b, int kvh, int ht,
                                             float* rows_out) {
  constexpr float LN2 = 0.6931471805599453f;
  constexpr int LPH = 32 / HP, CH = D / LPH;
  constexpr int SB = CH < 4 ? 8 : 32 / CH;    // slots requested together
  const long long rows = static_cast<long long>(P.a.batch) * P.a.num_qo_heads;
  const int lane = threadIdx.x & 31, part = lane % LPH;
  const bool on = ht * 8 + lane / LPH < P.heads_per_kv;
  const long long row = static_cast<long long>(b) * P.a.num_qo_heads +
                        static_cast<long long>(kvh) * P.heads_per_kv + ht * 8 + lane / LPH;
  if (k > 64) k = 64;
  float os[SB][CH], ms[SB], ls[SB];
  auto fetch = [&](int s0) {
#pragma unroll
    for (int i = 0; i < SB; ++i) {
      const bool have = on && s0 + i < k;
      const long long at = (s0 + i) * rows + row;
      ms[i] = have ? __ldcg(P.a.m_partial + at) : -INFINITY;
      ls[i] = have ? __ldcg(P.a.l_partial + at) : 0.f;
#pragma unroll
      for (int c = 0; c < CH; ++c)
        os[i][c] = have ? __ldcg(P.a.o_partial + at * D + part + LPH * c) : 0.f;
    }
  };
  fetch(0);
  float M = ms[0];
#pragma unroll
  for (int i = 1; i < SB; ++i) M = fmaxf(M, ms[i]);
#pragma unroll 1
  for (int s0 = SB; s0 < k; s0 += 4 * LPH) {
    float further[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int s = s0 + part + LPH * i;
      further[i] = on && s < k ? __ldcg(P.a.m_partial + s * rows + row) : -INFINITY;
    }
    M = fmaxf(M, fmaxf(fmaxf(further[0], further[1]), fmaxf(further[2], further[3])));
  }
#pragma unroll
  for (int o = LPH / 2; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xFFFFFFFFu, M, o));
  float den = 0.f, acc[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) acc[c] = 0.f;
#pragma unroll 1
  for (int s0 = 0; s0 < k; s0 += SB) {
    if (s0 > 0) fetch(s0);
#pragma unroll
    for (int i = 0; i < SB; ++i) {            // (past the last slot: o, l and the weight are zero)
      const float wgt = M > -INFINITY ? exp2f(ms[i] - M) : 0.f;
      den += wgt * ls[i];
#pragma unroll
      for (int c = 0; c < CH; ++c) acc[c] += wgt * os[i][c];
    }
  }
#pragma unroll
  for (int c = 0; c < CH; ++c) rows_out[(lane / LPH) * D + part + LPH * c] = acc[c];
  __syncwarp();
#pragma unroll 1
  for (int h = 0; h < HP; ++h) {
    const int hl = ht * 8 + h;
    if (hl >= P.heads_per_kv) break;
    const float den_h = __shfl_sync(0xFFFFFFFFu, den, h * LPH);
    const float M_h = __shfl_sync(0xFFFFFFFFu, M, h * LPH);
    const bool live = den_h > 0.f;
    const long long orow = caller_row<true>(P, b, kvh, hl);
#pragma unroll
    for (int c = 0; c < D; c += 32)
      store_value(P.a.out, P.a.out_dtype, orow * D + lane + c,
                  live ? rows_out[h * D + lane + c] / den_h * P.a.o_scale : 0.f);
    if (lane == 0 && P.a.lse != nullptr)
      P.a.lse[orow] = live ? (M_h + log2f(den_h)) * LN2 : -INFINITY;
  }
  __syncwarp();
}

// Chunks of an item; an empty one counts as one (nothing valid in it), so that its rows are
// written like any other's.
__device__ __forceinline__ int chunks_of(const WorkItem& w, int tile) {
  const int n = min(w.t1 * tile, w.len) - w.t0 * tile;
  return n > 0 ? (n + CHUNK - 1) / CHUNK : 1;
}

// Looks up chunks of the warp, one per lane from lane `from` on: the lane walks the items to its
// chunk and has the page id copied to the chunk's table entry (asynchronously: it has landed when
// the copies of the chunk being issued have). Out of line, with the walks in shared memory, so
// that the chunk loop holds none of it in registers.
// A chunk that the page table has no entry for gets -1, like any page id outside the pool.
__device__ __noinline__ void look_up_chunks(const DecodeParams& P, const WorkItem* cached,
                                            const WorkItem* more, int slots, const ItemRange items,
                                            int warps, uint8_t* table, int at, int from, int to) {
  const int lane = threadIdx.x & 31;
  if (lane >= from && lane < to) {
    int* const walk = reinterpret_cast<int*>(table + AHEAD * 8) + 3 * lane;
    int k = walk[0], base = walk[1];
    const int g = walk[2];
    int half = NO_CHUNK;
    int2* const place = reinterpret_cast<int2*>(table) + ((at + lane) & (AHEAD - 1));
    for (int wi = items.begin + k * items.step; wi < items.end; wi += items.step, ++k) {
      const WorkItem w = item_at(P, cached, more, slots, k, wi);
      const int n = chunks_of(w, P.tile_tokens);
      if (g >= base + n) {
        base += n;
        continue;
      }
      const int pos = w.t0 * P.tile_tokens + CHUNK * (g - base);
      if (pos < min(w.t1 * P.tile_tokens, w.len)) {
        half = 2 * w.kvh + (pos & (PAGE - 1)) / CHUNK;
        const long long e = static_cast<long long>(w.table_off) + pos / PAGE;
        if (e >= 0 && e < P.a.table_len)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(place)),
                       "l"(P.a.page_table + e) : "memory");
        else
          place->x = -1;
      }
      break;
    }
    walk[0] = k;
    walk[1] = base;
    walk[2] = g + 32 * warps;
    if (half == NO_CHUNK) place->x = -1;
    place->y = half;
  }
}

// A chunk whose page id is not in the pool: reported, and its records are zeroed, so that the
// chunk's result is finite (its tokens' scores count as zero).
__device__ __noinline__ void bad_page(uint32_t records, int* status) {
  const int lane = threadIdx.x & 31;
  if (lane == 0 && status != nullptr) atomicOr(status, FQ_STATUS_BAD_PAGE);
  asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(records + 16 * lane), "r"(0) : "memory");
}

}  // namespace

template <int BITS, int GP, bool HALF>
__global__ void __launch_bounds__(32 * StreamPlan<BITS, GP>::W, 1)
stream_decode_kernel(const __grid_constant__ DecodeParams P) {
  // HALF: the records are bf16 pairs, not f32
  using SP = StreamPlan<BITS, GP>;
  using FD = Field<BITS>;
  constexpr int W = SP::W, CHUNKS = SP::CHUNKS, RB = SP::RB, MT = SP::MT;
  constexpr int NT = GP == 4 ? 1 : 2;         // tokens of a lane in a group of sixteen
  constexpr int NG = CHUNK / 16;
  constexpr float LN2 = 0.6931471805599453f;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem0 = (smem_u32(smem_raw) + 127u) & ~127u;
  uint8_t* const smem = smem_raw + (smem0 - smem_u32(smem_raw));
  volatile int* const ctl = reinterpret_cast<volatile int*>(smem + SP::CTL_OFF);
  volatile int* const abort_flag = ctl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = lane >> 2, j = lane & 3;      // mma fragment row and column group
  int* const status = P.a.status;

  for (int i = threadIdx.x; i < 128; i += 32 * W) ctl[i] = 0;
  __syncthreads();
  if (threadIdx.x == 0) set_wait_budget(abort_flag, P.wait_budget);

  // Everything above touched only this CTA's shared memory. Under a programmatic launch it may
  // have run while the launch before this one in the stream was still finishing: wait for that
  // launch (complete and flushed) before the first global access, and let the launch after this
  // one start its own set-up as SMs free up. Both are no-ops otherwise.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // the pool's P-scale exponent, from the count table's top nonzero bin (requested first, used
  // after the items are decoded)
  uint32_t bins[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    bins[i] = P.p.v_max_hist != nullptr ? __ldg(P.p.v_max_hist + lane * 8 + i) : 0u;

  const ItemRange items = item_range(P);
  // The CTA's first items, decoded by one thread each: their dependent loads (row, length, table
  // offset) go out side by side, once.
  WorkItem* const item_cache = reinterpret_cast<WorkItem*>(smem + SP::ITEM_OFF);
  WorkItem* const item_more = reinterpret_cast<WorkItem*>(smem + SP::MORE_OFF);
  for (int k = threadIdx.x; k < P.item_slots; k += 32 * W) {
    const long long wi = items.begin + static_cast<long long>(k) * items.step;
    if (wi < items.end) {
      const WorkItem w = decode_item(P, static_cast<int>(wi));
      if (k < SP::ITEM_SLOTS) item_cache[k] = w;
      else item_more[k - SP::ITEM_SLOTS] = w;
    }
  }
  // w = p * s_v * 2^lp stays inside f16 with p up to 2^MAX_LAG: lp = 135 - bin is the exponent
  // that takes the pool's largest s_v below 448 = 7 * 2^6; 6 - MAX_LAG more still fit
  int top = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (bins[i] != 0u) top = lane * 8 + i;
  top = __reduce_max_sync(0xFFFFFFFFu, top);
  const int lp = 135 - max(top, 27) + 6 - static_cast<int>(MAX_LAG);
  const float p2lp = exp2f(static_cast<float>(lp));
  const float o_mul = exp2f(static_cast<float>(24 - lp));
  __syncthreads();

  // ------------------------------------------------------------------ the warp's copies
  constexpr int NS = SP::S;
  const uint32_t ring = smem0 + SP::RING_OFF + warp * SP::S * SP::STAGE;
  const uint64_t stream_policy = l2_evict_first_policy();
  uint8_t* const table = smem + SP::TABLE_OFF + warp * TABLE_BYTES;
  auto look_up = [&](int at, int from, int to) {
    look_up_chunks(P, item_cache, item_more, SP::ITEM_SLOTS, items, W, table, at, from, to);
  };
  {
    int* const walk = reinterpret_cast<int*>(table + AHEAD * 8) + 3 * lane;
    walk[0] = walk[1] = 0;
    walk[2] = warp + W * lane;
  }
  look_up(0, 0, 16);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  int issued = 0;
  uint32_t issue_to = ring;
  const uint64_t lane16 = 16u * lane;
  const uint32_t kv2 = 2u * P.p.num_kv_heads;
  // a lane's 16 bytes are piece lane % CHUNKS of row lane / CHUNKS (and of rows further on)
  const uint32_t code_lane =
      16u * ((lane & ~(CHUNKS - 1)) | ((lane & (CHUNKS - 1)) ^ SP::row_swizzle(lane / CHUNKS)));
  auto issue = [&]() {
    const int2 entry = reinterpret_cast<const int2*>(table)[issued & (AHEAD - 1)];
    if (static_cast<uint32_t>(entry.x) < static_cast<uint32_t>(P.p.num_pages)) {
      // half pages are numbered 2 * (page * HKV + head) + half (below 2^32: a half page of one
      // head is at least 1.25 KB)
      const uint32_t blk2 = static_cast<uint32_t>(entry.x) * kv2 + entry.y;
      const uint64_t off = static_cast<uint64_t>(blk2) * SP::CODE + lane16;
      const uint8_t* ks = P.p.k_codes + off;
      const uint8_t* vs = P.p.v_codes + off;
      const uint32_t dst = issue_to;
#pragma unroll
      for (int c = 0; c < SP::CODE; c += 512) {   // (a step of 16 rows keeps the swizzle)
        cp_async16_stream(dst + SP::K_OFF + c + code_lane, ks + c, stream_policy);
        cp_async16_stream(dst + SP::V_OFF + c + code_lane, vs + c, stream_policy);
      }
      const uint8_t* ss = static_cast<const uint8_t*>(P.p.scales) + lane16;
      if constexpr (!HALF) {             // 16 bytes a token
        ss += static_cast<uint64_t>(blk2) * (16 * CHUNK);
        cp_async16_stream(dst + SP::R_OFF + 16 * lane, ss, stream_policy);
      } else {                           // 8 bytes a token
        ss += static_cast<uint64_t>(blk2) * (8 * CHUNK);
        if (lane < 16) cp_async16_stream(dst + SP::R_OFF + 16 * lane, ss, stream_policy);
      }
    } else if (entry.y != NO_CHUNK) {   // (no chunk: nothing to copy)
      bad_page(issue_to + SP::R_OFF, status);
    }
    cp_async_commit();
    issue_to += SP::STAGE;
    if (issue_to == ring + NS * SP::STAGE) issue_to = ring;
    ++issued;
  };
  for (int a = 1; a < NS; ++a) issue();
  look_up(0, 16, 32);

  // ------------------------------------------------------------------ the warp's chunks
  // ldmatrix row of this lane: token (lane / 16) * 8 + lane % 8 of a group of sixteen, piece
  // (lane / 8) % 2 of a pair (rows of one piece: token lane % 16)
  const int lrow = CHUNKS == 1 ? (lane & 15) : ((lane >> 4) << 3) + (lane & 7);
  const uint32_t lm_off = lrow * RB +
      (CHUNKS == 1 ? 0 : ((((lane >> 3) & 1) ^ SP::row_swizzle(lrow)) << 4));
  const bool upper = GP == 4 && j >= 2;       // four columns: this lane takes tokens 8-15's scores
  const int tok0 = r + (upper ? 8 : 0);       // the lane's (first) token of a group of sixteen
  const int h0 = GP == 4 ? 2 * (j & 1) : 2 * j;   // its two heads of the head tile: h0, h0 + 1

  float O[MT][4];
  uint32_t qr[SP::QR];
  float hs[2], hq[2];                         // score scale; sum of the query row
  float m[2], l[2], c[2];
  float thr[2];                               // excess that raises m; -inf: no finite score yet
  int lim[2];                                 // the heads' first invisible position
  int c_k = 0, c_base = 0, c_n = 0;           // item of the CTA, its first chunk, its chunks
  WorkItem w;

  auto begin_item = [&]() {
    // the query operand: column r's quarter of the row, words 4c + j, in the order a packed word's
    // fields are taken, each field's place in the word divided out (exact: powers of two)
    const int hl = w.ht * 8 + r;
    const bool live = r < GP && hl < P.heads_per_kv;
    const long long qrow = live ? caller_row<true>(P, w.b, w.kvh, hl) : 0;
    const uint8_t* q = static_cast<const uint8_t*>(P.a.q) + qrow * D;
    float scale = live ? P.a.sm_scale * 1.4426950408889634f : 0.f;
    if (live && P.a.q_descale != nullptr) scale *= caller_descale<true>(P, w.b, w.kvh, hl);
    float sum = 0.f;
#pragma unroll
    for (int cc = 0; cc < CHUNKS; ++cc) {
      constexpr int NB = 32 / BITS / 4;       // 4-byte words of the q bytes against one packed word
      uint32_t raw[NB];
      if constexpr (BITS == 2) {
        const uint4 v = live ? __ldg(reinterpret_cast<const uint4*>(q) + 4 * cc + j)
                             : make_uint4(0, 0, 0, 0);
        raw[0] = v.x; raw[1] = v.y; raw[2] = v.z; raw[3] = v.w;
      } else {
        const uint2 v = live ? __ldg(reinterpret_cast<const uint2*>(q) + 4 * cc + j)
                             : make_uint2(0, 0);
        raw[0] = v.x; raw[1] = v.y;
      }
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const float2 a = e4m3x2_to_f32x2(raw[i] & 0xFFFF), b = e4m3x2_to_f32x2(raw[i] >> 16);
        s += (a.x + a.y) + (b.x + b.y);
      }
      sum += s;
#pragma unroll
      for (int f = 0; f < FD::NF; ++f) {
        // channels of fields f and NF + f
        constexpr int HW = 16 / BITS;
        const int lo = f / 2 + HW * (f & 1), hi = lo + HW / 2;
        const uint32_t pair = ((raw[lo / 4] >> (8 * (lo & 3))) & 0xFFu) |
                              (((raw[hi / 4] >> (8 * (hi & 3))) & 0xFFu) << 8);
        const __half2 v = __hmul2(e4m3x2_to_f16x2(pair),
                                  __float2half2_rn(1.f / static_cast<float>(1 << FD::bits_up(f))));
        qr[cc * FD::NF + f] = *reinterpret_cast<const uint32_t*>(&v);
      }
    }
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
#pragma unroll
    for (int i = 0; i < 2; ++i) {             // from the operand's columns to the lane's heads
      // (a code is code * 2^-24: the scores' scale makes up for it, the query sums are divided)
      hs[i] = __shfl_sync(0xFFFFFFFFu, scale, 4 * (h0 + i)) * 16777216.f;
      hq[i] = __shfl_sync(0xFFFFFFFFu, sum, 4 * (h0 + i)) * (1.f / 16777216.f);
      m[i] = l[i] = c[i] = 0.f;
      thr[i] = -INFINITY;
      lim[i] = (w.t1 > w.t0 ? w.len : 0) -
               (P.q_len > 1 ? column_lag(P, w.ht * 8 + h0 + i) : 0);
    }
#pragma unroll
    for (int f = 0; f < MT; ++f)
#pragma unroll
      for (int i = 0; i < 4; ++i) O[f][i] = 0.f;
  };

  // The warp's share of the item is done: its state goes to its slot, and the last warp to get
  // here merges the slots, in the order of the chunks the warps began with.
  auto finish_item = [&]() {
    float M[2], st[SP::NST];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        l[i] += __shfl_xor_sync(0xFFFFFFFFu, l[i], o);
        c[i] += __shfl_xor_sync(0xFFFFFFFFu, c[i], o);
      }
      M[i] = thr[i] == -INFINITY ? -INFINITY : m[i];
    }
    if constexpr (GP == 4) {                  // the two token halves of a head become one
      float f[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float Mn = fmaxf(M[i], __shfl_xor_sync(0xFFFFFFFFu, M[i], 2));
        f[i] = M[i] == -INFINITY ? 0.f : exp2f(M[i] - Mn);
        M[i] = Mn;
        l[i] *= f[i];
        c[i] *= f[i];
        l[i] += __shfl_xor_sync(0xFFFFFFFFu, l[i], 2);
        c[i] += __shfl_xor_sync(0xFFFFFFFFu, c[i], 2);
      }
#pragma unroll
      for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float lo = O[t][i] * f[i], hi = O[t][2 + i] * f[i];
          const float got = __shfl_xor_sync(0xFFFFFFFFu, j < 2 ? hi : lo, 2);
          st[2 * t + i] = (j < 2 ? lo : hi) + got;
        }
    } else {
#pragma unroll
      for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) st[4 * t + i] = O[t][i];
    }
    const int slot = c_k % SLOTS;
    const int parts = min(c_n, W), first = c_base % W;
    float* const mine = reinterpret_cast<float*>(smem + SP::STATE_OFF + warp * SP::STATE);
    warp_wait<false>(ctl + CTL_BUSY + warp, 0, abort_flag, status);
    bool last = true;
    // The items of a slot complete in turn: DONE[slot] counts them, and one that counts its parts in,
    // or itself done, waits for all the slot's earlier items first. (That holds for an item of one
    // part too: its early count would pass for an earlier item that is still open, and the item
    // between them would then count on that one's parts. It waits for earlier items only, so the
    // waits end.)
    if (parts > 1) {
#pragma unroll
      for (int q = 0; q < SP::NST / 4; ++q)
        reinterpret_cast<float4*>(mine)[q * 32 + lane] =
            make_float4(st[4 * q], st[4 * q + 1], st[4 * q + 2], st[4 * q + 3]);
      float* const meta = reinterpret_cast<float*>(smem + SP::META_OFF + warp * 96);
      if (lane < GP / 2)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          meta[h0 + i] = M[i];
          meta[8 + h0 + i] = l[i];
          meta[16 + h0 + i] = c[i];
        }
      if (lane == 0) ctl[CTL_BUSY + warp] = 1;
      warp_wait<true>(ctl + CTL_DONE + slot, c_k / SLOTS, abort_flag, status);
      __threadfence_block();
      int seen = 0;
      if (lane == 0) seen = atomicAdd(const_cast<int*>(ctl) + CTL_COUNT + slot, 1);
      seen = __shfl_sync(0xFFFFFFFFu, seen, 0);
      last = seen == parts - 1;
      if (last) {
        __threadfence_block();
        M[0] = M[1] = -INFINITY;
        for (int p = 0; p < parts; ++p) {
          const volatile float* meta_p = reinterpret_cast<const volatile float*>(
              smem + SP::META_OFF + ((first + p) % W) * 96);
          M[0] = fmaxf(M[0], meta_p[h0]);
          M[1] = fmaxf(M[1], meta_p[h0 + 1]);
        }
        l[0] = l[1] = c[0] = c[1] = 0.f;
#pragma unroll
        for (int i = 0; i < SP::NST; ++i) st[i] = 0.f;
#pragma unroll 1
        for (int p = 0; p < parts; ++p) {
          const int wp = (first + p) % W;
          const volatile float* meta_p =
              reinterpret_cast<const volatile float*>(smem + SP::META_OFF + wp * 96);
          float f[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float mp = meta_p[h0 + i];
            f[i] = mp == -INFINITY ? 0.f : exp2f(mp - M[i]);
            l[i] += f[i] * meta_p[8 + h0 + i];
            c[i] += f[i] * meta_p[16 + h0 + i];
          }
          const float4* sp = reinterpret_cast<const float4*>(smem + SP::STATE_OFF + wp * SP::STATE);
#pragma unroll
          for (int q = 0; q < SP::NST / 4; ++q) {
            const float4 v = sp[q * 32 + lane];
            st[4 * q] += f[0] * v.x;
            st[4 * q + 1] += f[1] * v.y;
            st[4 * q + 2] += f[0] * v.z;
            st[4 * q + 3] += f[1] * v.w;
          }
        }
        __syncwarp();
        __threadfence_block();
        if (lane < parts && (first + lane) % W != warp) ctl[CTL_BUSY + (first + lane) % W] = 0;
        if (lane == 0) {
          ctl[CTL_COUNT + slot] = 0;
          __threadfence_block();
          atomicAdd(const_cast<int*>(ctl) + CTL_DONE + slot, 1);
        }
      }
    } else {
      warp_wait<true>(ctl + CTL_DONE + slot, c_k / SLOTS, abort_flag, status);
      if (lane == 0) atomicAdd(const_cast<int*>(ctl) + CTL_DONE + slot, 1);
    }
    if (!last) return;
    if (w.slot != -2) {
      // rows through the warp's slot, so that the stores are whole rows
#pragma unroll
      for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int i = 0; i < SP::NST / MT; ++i) {
          const int hi = GP == 4 ? (j >> 1) : (i >> 1);
          const float unit =
              1.f / static_cast<float>(1 << FD::bits_up(o_field<BITS>(t, hi)));
          mine[(h0 + (i & 1)) * D + o_channel<BITS>(t, hi, r)] =
              fmaf(st[(SP::NST / MT) * t + i], o_mul * unit, c[i & 1]);
        }
      __syncwarp();
#pragma unroll 1
      for (int h = 0; h < GP; ++h) {
        const int hl = w.ht * 8 + h;
        if (hl >= P.heads_per_kv) break;
        const float Lh = __shfl_sync(0xFFFFFFFFu, h & 1 ? l[1] : l[0], h >> 1);
        const float Mh = __shfl_sync(0xFFFFFFFFu, h & 1 ? M[1] : M[0], h >> 1);
        const float* row = mine + h * D;
        if (w.slot < 0) {
          const long long orow = caller_row<true>(P, w.b, w.kvh, hl);
#pragma unroll
          for (int i = 0; i < D / 32; ++i)
            store_value(P.a.out, P.a.out_dtype, orow * D + lane + 32 * i,
                        Lh > 0.f ? row[lane + 32 * i] / Lh * P.a.o_scale : 0.f);
          if (lane == 0 && P.a.lse != nullptr)
            P.a.lse[orow] = Lh > 0.f ? (Mh + log2f(Lh)) * LN2 : -INFINITY;
        } else {
          const long long prow = static_cast<long long>(w.slot) * P.a.batch * P.a.num_qo_heads +
                                 static_cast<long long>(w.b) * P.a.num_qo_heads +
                                 (static_cast<long long>(w.kvh) * P.heads_per_kv + hl);
#pragma unroll
          for (int i = 0; i < D / 32; ++i) P.a.o_partial[prow * D + lane + 32 * i] = row[lane + 32 * i];
          if (lane == 0) { P.a.l_partial[prow] = Lh; P.a.m_partial[prow] = Mh; }
        }
      }
      __syncwarp();
    }
    if (lane == 0) ctl[CTL_BUSY + warp] = 0;
    // a split piece is counted in on its unit; the piece that completes the unit merges it
    if (w.slot >= 0 && P.a.unit_counters != nullptr) {
      const int unit = (w.b * P.p.num_kv_heads + w.kvh) * P.head_tiles + w.ht;
      int k = 0;
      __threadfence();
      __syncwarp();
      if (lane == 0) {
        const int pieces = P.a.split_counts != nullptr ? __ldg(P.a.split_counts + unit) : P.a.kv_splits;
        if (atomicAdd(P.a.unit_counters + unit, 1) == pieces - 1) {
          P.a.unit_counters[unit] = 0;   // nobody touches it again before the next launch
          k = pieces;
        }
      }
      k = __shfl_sync(0xFFFFFFFFu, k, 0);
      if (k > 0) {
        __threadfence();
        if constexpr (GP == 8) {
          merge_unit_warp<8>(P, k, w.b, w.kvh, w.ht, mine);
        } else {
          if (P.heads_per_kv == 1) merge_unit_warp<1>(P, k, w.b, w.kvh, w.ht, mine);
          else merge_unit_warp<4>(P, k, w.b, w.kvh, w.ht, mine);
        }
      }
    }
  };

  int g = warp;                               // the warp's next chunk
  uint32_t sb = ring;                         // its ring stage
  for (int c_wi = items.begin; c_wi < items.end; c_wi += items.step, ++c_k, c_base += c_n) {
  w = item_at(P, item_cache, item_more, SP::ITEM_SLOTS, c_k, c_wi);
  c_n = chunks_of(w, P.tile_tokens);
  const int g_end = c_base + c_n;
  if (g >= g_end) continue;
  begin_item();
  int pos0 = w.t0 * P.tile_tokens + CHUNK * (g - c_base);
  const int end = w.t1 > w.t0 ? w.len : 0;      // (an empty piece's one chunk: nothing is valid)
  const int whole = end - (P.q_len - 1) - CHUNK;   // chunks up to here need no mask
#pragma unroll 1
  for (; g < g_end; g += W, pos0 += W * CHUNK) {
    __syncwarp();                             // the stage of the chunk before is read
    if ((issued & 31) == 16) look_up(issued + 16, 0, 32);
    issue();
    cp_async_wait<NS - 1>();
    __syncwarp();

    float x[NG][NT][2], zv[NG][NT], wsc[NG][NT];
    // ---- scores
#pragma unroll
    for (int tb = 0; tb < NG; ++tb) {
      const uint32_t ka = sb + SP::K_OFF + tb * 16 * RB;
      float acc[4];
      uint32_t kw[CHUNKS][2];                 // a piece's words of tokens r and r + 8
      if constexpr (CHUNKS == 1) ldsm2(ka + lm_off, kw[0][0], kw[0][1]);
      else ldsm4(ka + lm_off, kw[0][0], kw[CHUNKS - 1][0], kw[0][1], kw[CHUNKS - 1][1]);
#pragma unroll
      for (int cc = 0; cc < CHUNKS; ++cc) {
        const uint32_t k0 = kw[cc][0], k1 = kw[cc][1];
        const uint32_t s0 = k0 >> FD::SHIFT, s1 = k1 >> FD::SHIFT;
#pragma unroll
        for (int f = 0; f < FD::NF; f += 2) {
          const uint32_t a0 = FD::get(k0, s0, f), a1 = FD::get(k1, s1, f),
                         a2 = FD::get(k0, s0, f + 1), a3 = FD::get(k1, s1, f + 1);
          const uint32_t b0 = qr[cc * FD::NF + f], b1 = qr[cc * FD::NF + f + 1];
          if (f == 0 && cc == 0) mma_f16_first(acc, a0, a1, a2, a3, b0, b1);
          else mma_f16(acc, a0, a1, a2, a3, b0, b1);
        }
      }
      if constexpr (GP == 4) {                // columns 4-7 are idle: their lanes take tokens 8-15
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float got = __shfl_xor_sync(0xFFFFFFFFu, acc[2 + i], 2);
          if (upper) acc[i] = got;
        }
      }
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int tok = 16 * tb + 8 * t + tok0;
        float sk, zk, sv;
        if constexpr (!HALF) {
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                       : "=f"(sk), "=f"(zk), "=f"(sv), "=f"(zv[tb][t])
                       : "r"(sb + SP::R_OFF + 16 * tok));
        } else {
          uint32_t kr, vr;
          asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(kr), "=r"(vr)
                       : "r"(sb + SP::R_OFF + 8 * tok));
          sk = __uint_as_float(kr << 16); zk = __uint_as_float(kr & 0xFFFF0000u);
          sv = __uint_as_float(vr << 16); zv[tb][t] = __uint_as_float(vr & 0xFFFF0000u);
        }
        // (the bound keeps w inside f16 whatever the record says)
        wsc[tb][t] = fminf(sv * p2lp, 8000.f);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float s = fmaf(sk, acc[2 * t + i], zk * hq[i]);
          x[tb][t][i] = fmaf(hs[i], s, -m[i]);
        }
      }
    }
    // Positions past the request's end, or past what a head of several query tokens sees: their
    // scores become -inf and their records are neutralised, so stale shared memory never reaches
    // the output.
    if (pos0 > whole) {
#pragma unroll
      for (int tb = 0; tb < NG; ++tb)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int pos = pos0 + 16 * tb + 8 * t + tok0;
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (pos >= lim[i]) x[tb][t][i] = -INFINITY;
          if (pos >= end) { zv[tb][t] = 0.f; wsc[tb][t] = 0.f; }
        }
    }
    // ---- the heads' references: raised when a score exceeds one by more than MAX_LAG
    float over[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      over[i] = x[0][0][i];
#pragma unroll
      for (int e = 1; e < NG * NT; ++e) over[i] = fmaxf(over[i], x[e / NT][e % NT][i]);
    }
    if (__any_sync(0xFFFFFFFFu, over[0] > thr[0] || over[1] > thr[1])) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1)
          over[i] = fmaxf(over[i], __shfl_xor_sync(0xFFFFFFFFu, over[i], o));
        const bool first = thr[i] == -INFINITY, raise = over[i] > thr[i];
        const float delta = raise ? over[i] + HEADROOM : 0.f;
        const float corr = first ? 1.f : fast_exp2(-delta);   // (first: the sums are zero)
        if (raise) thr[i] = MAX_LAG;
        m[i] += delta;
        l[i] *= corr;
        c[i] *= corr;
#pragma unroll
        for (int e = 0; e < NG * NT; ++e) x[e / NT][e % NT][i] -= delta;
#pragma unroll
        for (int f = 0; f < MT; ++f) {
          O[f][i] *= corr;
          O[f][2 + i] *= corr;
        }
      }
    }
    // ---- weights, and O^T += C_V^T . W
#pragma unroll
    for (int tb = 0; tb < NG; ++tb) {
      uint32_t pw[NT];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        float p[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          p[i] = fast_exp2(x[tb][t][i]);
          l[i] += p[i];
          c[i] = fmaf(p[i], zv[tb][t], c[i]);
        }
        const __half2 h = __floats2half2_rn(p[0] * wsc[tb][t], p[1] * wsc[tb][t]);
        pw[t] = transpose_8x8(*reinterpret_cast<const uint32_t*>(&h));
      }
      // (four columns: rows 0-3 of the transposed tile are tokens 0-7's weights, rows 4-7 tokens
      // 8-15's; each goes to its own columns of O)
      uint32_t b0, b1;
      if constexpr (GP == 4) { b0 = r < 4 ? pw[0] : 0u; b1 = r < 4 ? 0u : pw[0]; }
      else { b0 = pw[0]; b1 = pw[NT - 1]; }
      const uint32_t va = sb + SP::V_OFF + tb * 16 * RB;
      if constexpr (CHUNKS == 1) {
        uint32_t v0, v1;
        ldsm2_t(va + lm_off, v0, v1);
        const uint32_t s0 = v0 >> FD::SHIFT, s1 = v1 >> FD::SHIFT;
#pragma unroll
        for (int f = 0; f < MT; ++f)
          mma_f16(O[f], FD::get(v0, s0, 2 * f), FD::get(v0, s0, 2 * f + 1), FD::get(v1, s1, 2 * f),
                  FD::get(v1, s1, 2 * f + 1), b0, b1);
      } else {
        uint32_t v0, v1, v2, v3;
        ldsm4_t(va + lm_off, v0, v1, v2, v3);
        const uint32_t s0 = v0 >> FD::SHIFT, s1 = v1 >> FD::SHIFT, s2 = v2 >> FD::SHIFT,
                       s3 = v3 >> FD::SHIFT;
#pragma unroll
        for (int f = 0; f < MT; ++f)
          mma_f16(O[f], FD::get(v0, s0, f), FD::get(v1, s1, f), FD::get(v2, s2, f),
                  FD::get(v3, s3, f), b0, b1);
      }
    }
    sb += SP::STAGE;
    if (sb == ring + NS * SP::STAGE) sb = ring;
  }
  finish_item();
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int BITS, int GP, bool HALF>
static int launch(DecodeParams& P, cudaStream_t stream) {
  using SP = StreamPlan<BITS, GP>;
  P.tile_tokens = tile_tokens(BITS, D);
  P.wait_budget = P.a.wait_budget_cycles > 0 ? P.a.wait_budget_cycles : WAIT_BUDGET_CYCLES;
  // Shared memory the rings leave over holds more decoded work items (32 bytes each)
  constexpr int more = std::max(0, std::min((SMEM_LIMIT - 128 - SP::MORE_OFF) / 32, 512));
  P.item_slots = SP::ITEM_SLOTS + more;
  constexpr int smem = SP::MORE_OFF + more * 32 + 128;
  static_assert(smem <= SMEM_LIMIT, "shared-memory plan");
  static bool configured[64] = {};  // per instantiation and device
  auto kernel = stream_decode_kernel<BITS, GP, HALF>;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  int sms = 148;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    sms = 148;
  const int ctas = P.a.max_ctas > 0 ? P.a.max_ctas : sms;
  int grid = P.a.worklist ? ctas : std::min(ctas, P.num_items);
  if (grid < 1) grid = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(32 * SP::W);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (P.a.flags & 1) ? 1 : 0;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, P));
}

}  // namespace stream

// head_dim 64 with whole-head K, f32 or bf16 records; columns: the unit's columns, at most 8.
int launch_decode_stream(DecodeParams& P, int columns, cudaStream_t s) {
  const bool two = P.p.bits == 2, half = P.p.scale_bf16 != 0;
  if (columns <= 4) {
    if (two) return half ? stream::launch<2, 4, true>(P, s) : stream::launch<2, 4, false>(P, s);
    return half ? stream::launch<4, 4, true>(P, s) : stream::launch<4, 4, false>(P, s);
  }
  if (two) return half ? stream::launch<2, 8, true>(P, s) : stream::launch<2, 8, false>(P, s);
  return half ? stream::launch<4, 8, true>(P, s) : stream::launch<4, 8, false>(P, s);
}

}  // namespace fq
