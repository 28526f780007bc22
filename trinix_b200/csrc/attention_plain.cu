// Attention forward without a dense mask or dropout: softmax(scale * Q K^T - ALiBi) V, online softmax
// (but few query rows: attention_decode.cuh, and a single KV tile in one wave of CTAs: attention.cu).
//
// A work item is two 128-row Q tiles: the same 128 query rows of two query heads that share a kv head
// (GQA / MQA: both tiles then see exactly the same keys), or 256 consecutive rows of one head
// otherwise. A CTA (one per SM) works on the item of its own block index and then on further ones
// that the hardware hands it (cluster launch control), so that set-up is paid once per SM and the next
// item's copies, first Q K^T and softmax run under the epilogue of the last; launches of one item per CTA
// have instantiations of their own. 16 warps:
//   warps 0-3, 4-7  softmax of Q tile 0 and 1, a thread per row (TMEM lane): no shuffles
//   warps 8-11      epilogue: O / l -> global
//   warp 12         TMA producer: Q, then K and V tiles of 128 keys through a 4-stage ring, across
//                   items (128-byte swizzle, no multicast); asks for and describes the next item
//   warps 13, 14    MMA issue of Q tile 0 and 1: S = Q K^T (both operands from shared memory) and
//                   O += P V (P from TMEM, V from shared memory, MN-major)
// TMEM (512 columns): S0 | S1 | O0 | O1; P (16-bit) overwrites the first half of its S. Softmax in the
// log2 domain (scale * log2e in one FMA, ALiBi as one more), O rescaled only when a row maximum grew
// by more than 2^8. KV tiles outside the causal / window range of a Q tile are never visited; tiles
// that the range cuts are masked 32 columns at a time by a bit mask. Query head h reads kv head
// h / (Hq / Hk). With ALiBi under a causal mask the KV tiles of a row block are visited from the
// diagonal backwards: the first tile then holds the row maximum and O is never rescaled again.
//
// What bounds it: per Q tile a chain scores -> softmax (about 2000 cycles, of them 1024 on the
// special-function unit) -> P V -> next Q K^T (1032 cycles at the MMA rate) -> scores; two of them
// share the SM, the tensor and the special-function pipe are each busy 55 to 60 % of the time (2 x 4096
// causal 56.5 and 56.5 %, ncu), under the power cap. What mattered (16 x 4096 causal, 32 / 8 heads x 128
// unless said otherwise; here and below single kernels timed in short bursts: call after call, where the
// power cap holds the clock down, the same shape takes 2120 to 2180 us for 1900 there):
//   * the issuing warps stay converged and elect a lane, and every branch goes by a vote: descriptors
//     are then uniform registers (from one lane in divergent code 4 x 4096 full: 1142 us, so 991);
//   * one issuing warp per Q tile: a wait on a ready barrier costs such a warp some 200 cycles, and
//     with one warp for both the P of one tile waits behind the MMAs of the other (1978 us, so 1904,
//     with its registers 1874 to 1910; window 1024: 1304, 1097; 8 x 2048 causal, 16 heads x 64: 188, 137);
//   * cut tiles: one uniform test per visit, then bit masks (2900 -> 600 cycles for such a tile).
// Measured and not taken: S shared by both tiles with P beside it (1016-1200 us on 4 x 4096 full
// against 868-990), 64-key tiles with two S buffers each (1059; an MMA with N = 64 is bound by shared
// memory, 48 cycles instead of 32), exponentials of the two tiles in forced turns (2064).
// Every wait is bounded: 400 ms, counted from the CTA's last progress where it may last an item.
#include "attention_common.cuh"
#include "attention_issue.cuh"

namespace trx {

constexpr int AP_THREADS = 512;
// P is handed over in two pieces: the P V of the first 96 keys runs while the last 32 are
// exponentiated (causal 16 x 4096: 1994 us in one piece, 1904 so, 2064 in halves).
constexpr int AP_REST = 2;  // of the 8 MMAs of a P V, those of the second piece
// Cycles by which Q tile 1's first softmax waits in a launch of one item per CTA. Both Q tiles' first
// scores are ready at the same time, and tiles in step stay so: both wait for the special-function
// unit, then both for the tensor pipe, 2.3 us a visit instead of 1.6 (512 queries x 8192 keys, 32 / 8
// heads x 128: 152 us, so 108; x 4096 84, 58; 1 x 1000 27.3, 22.0; 2 x 256 12.1, 11.1; a window of
// 256 on 1024 15.6, 15.2). 1000 / 1250 / 1750 cycles: 109.3 / 108.5 / 108.7, 1 x 1000 25.4 / 22.9 /
// 21.8, 2 x 256 11.5 / 11.2 / 11.2. The same in launches of several items per CTA gained 1 to 3 % on
// some and lost as much on others. A single visit (up to 128 keys) has nobody to get out of step with.
// A bias makes the softmax, and so half a visit, longer: 1500 / 1900 / 2200 / 2600 cycles, causal with
// ALiBi 1 x 1000 26.5 / 25.1 / 24.5 / 24.6, 4 x 512 18.7 / 17.4 / 17.1 / 17.2, both sides 1 x 2048,
// 8 heads 51.3 / 50.0 / 49.3 / 50.3.
constexpr unsigned AP_LAG = 1500, AP_LAG_BIAS = 2200;

// What is added to the scaled scores: nothing; ALiBi as one ramp per row (every visible key at or
// before its query); ALiBi on either side of the query, or a scale that is not positive. Of the last,
// a KV tile that lies on one side of its Q tile is a ramp as well, up or down, added to the raw score by
// one packed FMA for two, counted from its key next to the queries (its last, AP_RAMP_TO_LAST, or its
// first), so that the keys that weigh most carry the least rounding; only those in between take a
// difference, a product and an FMA for each score (for all tiles: 4 x 2048, 32 / 8 heads x 128 382 us,
// so 323; 16 heads x 64 172, 148).
enum AttnBias { AP_NONE = 0, AP_RAMP = 1, AP_GENERAL = 2, AP_RAMP_TO_LAST = 3 };

// Registers per thread after the split. The four warpgroups' shares sum to what the launch gives
// (4 x 128). The softmax loop holds 128 scores and does not fit 168 (16 x 4096 causal 2111 us against
// 1947 with 176); with 176 and 184 a few values around the loop and in the epilogue are spilled.
// Beyond that the register allocator's schedule decides, measured with 176 / 184: plain scores at head
// dim 128: causal 1947 / 1874 us, window 1024 1189 / 1044, 2 x 8192 full 1953 / 1731; ALiBi on both
// sides (ramps from column 0) 4 x 2048 339 / 313, but one item per CTA 51.3 / 55.5; ALiBi under a causal
// mask 2153 / 2345; head dim 64, 8 x 2048 x 16 heads 226 / 239, causal 146 / 151.
template <int D, int BIAS, bool SINGLE>
struct PlainRegs {
  static constexpr bool WIDE = D == 128 && (BIAS == AP_NONE || (BIAS == AP_GENERAL && !SINGLE));
  static constexpr int SOFTMAX = WIDE ? 184 : 176;
  static constexpr int EPILOGUE = 256 - SOFTMAX, OTHER = 256 - SOFTMAX;
  static_assert(2 * SOFTMAX + EPILOGUE + OTHER <= 512, "register split");
};

// Column numbers of a KV tile in pairs, for ALiBi's ramp: as immediates they cost two moves a pair
// (16 x 4096 causal with ALiBi: 2490 us against 2262).
struct ColumnPairs {
  float2 v[ATT_BN / 2];
};
constexpr ColumnPairs column_pairs(int first) {
  ColumnPairs t{};
  for (int i = 0; i < ATT_BN / 2; ++i) {
    t.v[i].x = static_cast<float>(first + 2 * i);
    t.v[i].y = static_cast<float>(first + 2 * i + 1);
  }
  return t;
}
static __constant__ ColumnPairs g_columns = column_pairs(0);
static __constant__ ColumnPairs g_columns_to_last = column_pairs(1 - ATT_BN);

template <int D>
struct PlainSmem {
  static constexpr int CHUNKS = D / 64;
  static constexpr int CHUNK_BYTES = ATT_BN * 128;  // 64 columns of a tile
  static constexpr int TILE_BYTES = CHUNKS * CHUNK_BYTES;
  static constexpr int Q_OFF = 0;
  static constexpr int KV_OFF = ATT_NQ * TILE_BYTES;
  static constexpr int BAR_OFF = KV_OFF + AP_STAGES * TILE_BYTES;
  static constexpr int NUM_BARS = 2 * AP_STAGES + 2 * 12 + 1;
  static constexpr int CTRL_OFF = BAR_OFF + NUM_BARS * 8;
  static constexpr int NEXT_OFF = (CTRL_OFF + 64 + 15) / 16 * 16;  // the answer: 16 bytes
  static constexpr int ITEM_OFF = NEXT_OFF + 16;                   // [2] PlainItem
  static constexpr int STAT_OFF = ITEM_OFF + 2 * 64;               // [2 tiles][sum, max][128]
  static constexpr int TOTAL = STAT_OFF + 2 * 2 * ATT_BM * 4;
  static constexpr int DYN_BYTES = TOTAL + 1024;  // slack for 1024-byte alignment
  static_assert(DYN_BYTES <= 232448, "shared memory");
};

// Visits count an item's KV tiles in visiting order: visit r is KV tile first + r * step. Q tile t
// takes part in visits [lo[t], hi[t]); its rows are m0 + t * t_rows .. of query head h + t * t_head.
struct PlainItem {
  int valid, b, h, m0;
  int n, first;
  int lo[ATT_NQ], hi[ATT_NQ];
};
static_assert(sizeof(PlainItem) <= 64, "shared memory slot");
// Which of a block index's x, y, z are the row block, the head (or pair of heads) and the batch; x runs
// fastest. Row blocks first: the K and V of few heads are at work at a time. Under a causal mask row
// blocks differ in length: with the heads of a batch, or all heads of all batches, running faster than
// the row blocks the heaviest come first and the CTAs end together.
enum PlainOrder { AP_MHB = 0, AP_HMB = 1, AP_HBM = 2 };
__device__ __forceinline__ PlainItem plain_item(const AttnParams& p, int x, int y, int z) {
  PlainItem w;
  w.valid = 1;
  const int mi = p.order == AP_MHB ? x : p.order == AP_HMB ? y : z;
  const int hi = p.order == AP_MHB ? y : x;
  w.b = p.order == AP_HBM ? y : z;
  const int m_blocks = p.order == AP_MHB ? gridDim.x : p.order == AP_HMB ? gridDim.y : gridDim.z;
  const int mblk = p.reverse_m ? m_blocks - 1 - mi : mi;
  w.h = hi * (p.pair_heads ? 2 : 1);
  w.m0 = mblk * (p.pair_heads ? ATT_BM : ATT_NQ * ATT_BM);
  TileRange r[ATT_NQ];
  int jlo = 1 << 30, jhi = 0;
#pragma unroll
  for (int t = 0; t < ATT_NQ; ++t) {
    r[t] = tile_range(p, w.m0 + (p.pair_heads ? 0 : t * ATT_BM));
    if (r[t].jhi > r[t].jlo) {
      jlo = min(jlo, r[t].jlo);
      jhi = max(jhi, r[t].jhi);
    }
  }
  w.n = max(0, jhi - jlo);
  w.first = p.reverse_kv ? jhi - 1 : jlo;
#pragma unroll
  for (int t = 0; t < ATT_NQ; ++t) {
    const bool any = r[t].jhi > r[t].jlo;
    w.lo[t] = !any ? 0 : p.reverse_kv ? jhi - r[t].jhi : r[t].jlo - jlo;
    w.hi[t] = !any ? 0 : w.lo[t] + r[t].jhi - r[t].jlo;
  }
  return w;
}

// Without the suspension of try_wait: whether the phase is complete now.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// mbar_wait for a whole converged warp, whose lanes all poll: every branch here goes by a vote, so
// that the compiler knows that the warp stays together and keeps what follows in uniform registers.
__device__ __forceinline__ bool mbar_poll_warp(uint32_t bar, uint32_t parity,
                                               volatile int* abort_flag, unsigned int* status,
                                               unsigned code) {
  uint64_t t0 = 0;
#pragma unroll 1
  for (uint32_t i = 0; i < ATT_WAIT_LIMIT; ++i) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((i & 63u) == 63u) {
      if (t0 == 0) t0 = global_ns();
      if (__any_sync(0xffffffffu, *abort_flag != 0)) return false;
      if (__any_sync(0xffffffffu, global_ns() - t0 > ATT_WAIT_NS)) break;
    }
  }
  *abort_flag = 1;
  atomicOr(status, code);
  return false;
}
static __device__ __noinline__ bool mbar_poll_warp_call(uint32_t bar, uint32_t parity,
                                                        volatile int* abort_flag,
                                                        unsigned int* status, unsigned code) {
  return mbar_poll_warp(bar, parity, abort_flag, status, code);
}
// `INLINE` false: out of line but for the first poll (which the hardware suspends for a while), for
// roles with few live registers: the code of a role that has to react fast stays small.
template <bool INLINE>
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity,
                                               volatile int* abort_flag, unsigned int* status,
                                               unsigned code) {
  if constexpr (INLINE) return mbar_poll_warp(bar, parity, abort_flag, status, code);
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return __any_sync(0xffffffffu, mbar_poll_warp_call(bar, parity, abort_flag, status, code));
}
// A wait for something that takes as long as a whole work item (its row statistics, the next item): an
// item may have any number of KV tiles, so the time counts from the last `progress` of the CTA.
__device__ __forceinline__ bool mbar_poll_item(uint32_t bar, uint32_t parity,
                                               volatile int* abort_flag, unsigned int* status,
                                               unsigned code, volatile int* progress) {
  uint64_t t0 = 0;
  int seen = 0;
#pragma unroll 1
  for (uint32_t i = 0; i < ATT_WAIT_LIMIT; ++i) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((i & 63u) == 63u) {
      if (__any_sync(0xffffffffu, *abort_flag != 0)) return false;
      const int now = *progress;
      if (__any_sync(0xffffffffu, t0 == 0 || now != seen)) {
        seen = now;
        t0 = global_ns();
        i = 0;
      } else if (__any_sync(0xffffffffu, global_ns() - t0 > ATT_WAIT_NS)) {
        break;
      }
    }
  }
  *abort_flag = 1;
  atomicOr(status, code);
  return false;
}
static __device__ __noinline__ bool mbar_poll_item_call(uint32_t bar, uint32_t parity,
                                                        volatile int* abort_flag,
                                                        unsigned int* status, unsigned code,
                                                        volatile int* progress) {
  return mbar_poll_item(bar, parity, abort_flag, status, code, progress);
}
template <bool INLINE>
__device__ __forceinline__ bool mbar_wait_item(uint32_t bar, uint32_t parity,
                                               volatile int* abort_flag, unsigned int* status,
                                               unsigned code, volatile int* progress) {
  if constexpr (INLINE) return mbar_poll_item(bar, parity, abort_flag, status, code, progress);
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return __any_sync(0xffffffffu,
                    mbar_poll_item_call(bar, parity, abort_flag, status, code, progress));
}
// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t is;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(is));
  return is != 0;
}
// Cluster launch control: ask the hardware for the block index of a CTA of this grid that has not
// been launched yet (it then never will be); the 16-byte answer arrives on an mbarrier.
__device__ __forceinline__ void request_block(uint32_t dst, uint32_t bar) {
  asm volatile(
      "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], "
      "[%1];" ::"r"(dst), "r"(bar)
      : "memory");
}
// Whether the answer is a block index, and which.
__device__ __forceinline__ bool requested_block(uint32_t src, int& x, int& y, int& z) {
  uint32_t ok, a, b, c;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 h;\n\t.reg .b32 w;\n\t"
      "ld.shared.b128 h, [%4];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t"
      "mov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, w}, h;\n\t}"
      : "=r"(ok), "=r"(a), "=r"(b), "=r"(c)
      : "r"(src)
      : "memory");
  x = a;
  y = b;
  z = c;
  return ok != 0;
}
// tcgen05.wait::ld that the loaded registers pass through, so that no use of them moves above it.
template <int OFF, int N>
__device__ __forceinline__ void tmem_wait_ld32(uint32_t (&r)[N]) {
  asm volatile(
      "tcgen05.wait::ld.sync.aligned;"
      : "+r"(r[OFF + 0]), "+r"(r[OFF + 1]), "+r"(r[OFF + 2]), "+r"(r[OFF + 3]), "+r"(r[OFF + 4]),
        "+r"(r[OFF + 5]), "+r"(r[OFF + 6]), "+r"(r[OFF + 7]), "+r"(r[OFF + 8]), "+r"(r[OFF + 9]),
        "+r"(r[OFF + 10]), "+r"(r[OFF + 11]), "+r"(r[OFF + 12]), "+r"(r[OFF + 13]),
        "+r"(r[OFF + 14]), "+r"(r[OFF + 15]), "+r"(r[OFF + 16]), "+r"(r[OFF + 17]),
        "+r"(r[OFF + 18]), "+r"(r[OFF + 19]), "+r"(r[OFF + 20]), "+r"(r[OFF + 21]),
        "+r"(r[OFF + 22]), "+r"(r[OFF + 23]), "+r"(r[OFF + 24]), "+r"(r[OFF + 25]),
        "+r"(r[OFF + 26]), "+r"(r[OFF + 27]), "+r"(r[OFF + 28]), "+r"(r[OFF + 29]),
        "+r"(r[OFF + 30]), "+r"(r[OFF + 31])
      :
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
        "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
        "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ float2 pair_of(const uint32_t* r) {
  return make_float2(__uint_as_float(r[0]), __uint_as_float(r[1]));
}
__device__ __forceinline__ void put_pair(uint32_t* r, float2 v) {
  r[0] = __float_as_uint(v.x);
  r[1] = __float_as_uint(v.y);
}

// SINGLE: the launch has no more CTAs than the GPU has SMs, so that each has one item: no request for
// another, no answer to wait for, nothing to hand over, all known at compile time. Decided at run time
// by the producer alone the other roles still waited for an item that says that there is none: 4 x 128
// causal, 16 / 2 heads x 128 10.7 us, so 10.2; 8 x 128 full, 16 heads x 64 7.6, 7.1.
template <int D, bool BF16, int BIAS, bool SINGLE>
__global__ void __launch_bounds__(AP_THREADS, 1)
    attn_plain_kernel(const __grid_constant__ AttnParams p) {
  using L = PlainSmem<D>;
  constexpr int STAGES = AP_STAGES, BN = ATT_BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + L::BAR_OFF;
  auto bar = [&](int i) { return bar0 + 8u * i; };
  constexpr int B_QFULL = 0;                    // [2] Q tile loaded
  constexpr int B_QEMPTY = 2;                   // [2] last Q K^T of the item done with it
  constexpr int B_SFULL = 4;                    // [2] scores ready
  constexpr int B_PFULL = 6;                    // [2] first piece of P in TMEM
  constexpr int B_PREST = 8;                    // [2] and the rest
  constexpr int B_ODONE = 10;                   // [2] last P V of the item done
  constexpr int B_STAT = 12;                    // [2] row sums and maxima in shared memory
  constexpr int B_STATFREE = 14;                // [2] and read
  constexpr int B_ITEM = 16;                    // [2] an item is described in shared memory
  constexpr int B_ITEMFREE = 18;                // [2] and has been read by every role
  constexpr int B_OFREE = 20;                   // [2] O of an item with keys read
  constexpr int B_KVFULL = 22;                  // [STAGES]
  constexpr int B_KVEMPTY = B_KVFULL + STAGES;  // [STAGES]
  constexpr int B_DRAIN = B_KVEMPTY + STAGES;   // [2]
  constexpr int B_NEXT = B_DRAIN + 2;           // the next block index is there
  static_assert(B_NEXT + 1 == L::NUM_BARS, "barrier count");
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + L::CTRL_OFF);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  int* fills_issued = reinterpret_cast<int*>(tmem_holder + 2);  // [STAGES]
  int* q_issued = fills_issued + STAGES;                        // [2]
  volatile PlainItem* items = reinterpret_cast<volatile PlainItem*>(smem + L::ITEM_OFF);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int t_rows = p.pair_heads ? 0 : ATT_BM;  // Q tile 1 against tile 0
  const int t_head = p.pair_heads ? 1 : 0;
  const int kv_step = p.reverse_kv ? -1 : 1;

  // A launch that follows a recorded failure does no work: the host must read and clear
  // the status word first.
  __shared__ int skip_launch;

  // One K or V tile of an item into ring stage g % STAGES, g counting the fills of all items. An
  // item's tiles in the order of their first use: K(0), K(1), V(0), K(2), V(1), .. V(n - 1).
  auto issue_fill = [&](const PlainItem& w, int kh, int vh, int fill, int g) {
    const int s = g % STAGES;
    const bool is_k = fill == 0 || ((fill & 1) != 0 && fill != 2 * w.n - 1);
    const int v = is_k ? (fill + 1) >> 1 : fill == 2 * w.n - 1 ? w.n - 1 : (fill >> 1) - 1;
    const int j = w.first + v * kv_step;
    mbar_expect_tx(bar(B_KVFULL + s), L::TILE_BYTES);
    fills_issued[s] = g / STAGES + 1;
    const CUtensorMap* tm = is_k ? &p.tm_k : &p.tm_v;
    const int hh = is_k ? kh : vh;
    const int bb = w.b * (is_k ? p.k_bmul : p.v_bmul);
#pragma unroll
    for (int c = 0; c < L::CHUNKS; ++c)
      tma_load_4d(sbase + L::KV_OFF + s * L::TILE_BYTES + c * L::CHUNK_BYTES, tm,
                  bar(B_KVFULL + s), c * 64, j * BN, hh, bb);
  };
  auto kv_heads = [&](const PlainItem& w, int& kh, int& vh) {  // of an item
    kh = w.h / p.k_hdiv;
    vh = p.v_hdiv == p.k_hdiv ? kh : w.h / p.v_hdiv;
  };
  auto issue_q = [&](const PlainItem& w, int t) {
    mbar_expect_tx(bar(B_QFULL + t), L::TILE_BYTES);
    q_issued[t] += 1;
#pragma unroll
    for (int c = 0; c < L::CHUNKS; ++c)
      tma_load_4d(sbase + L::Q_OFF + t * L::TILE_BYTES + c * L::CHUNK_BYTES, &p.tm_q,
                  bar(B_QFULL + t), c * 64, w.m0 + t * t_rows, w.h + t * t_head, w.b);
  };
  auto publish = [&](const PlainItem& w, int q) {  // item q, for the other roles
    volatile PlainItem& o = items[q & 1];
    o.valid = w.valid;
    if (w.valid) {
      o.b = w.b;
      o.h = w.h;
      o.m0 = w.m0;
      o.n = w.n;
      o.first = w.first;
#pragma unroll
      for (int t = 0; t < ATT_NQ; ++t) {
        o.lo[t] = w.lo[t];
        o.hi[t] = w.hi[t];
      }
    }
    mbar_arrive(bar(B_ITEM + (q & 1)));
  };

  if (warp == 12 && lane == 0) {
    skip_launch = (*reinterpret_cast<volatile unsigned int*>(p.status) != 0u) ? 1 : 0;
  }
  if (warp == 12 && lane == 0 && !skip_launch) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar(B_KVFULL + s), 1);
      mbar_init(bar(B_KVEMPTY + s), 2);  // one arrival per Q tile
      fills_issued[s] = 0;
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(bar(B_QFULL + t), 1);
      mbar_init(bar(B_QEMPTY + t), 1);
      mbar_init(bar(B_SFULL + t), 1);
      mbar_init(bar(B_PFULL + t), 4);  // one arrival per softmax warp
      mbar_init(bar(B_PREST + t), 4);
      mbar_init(bar(B_ODONE + t), 1);
      mbar_init(bar(B_STAT + t), 4);
      mbar_init(bar(B_STATFREE + t), 4);  // one per epilogue warp
      mbar_init(bar(B_OFREE + t), 4);
      mbar_init(bar(B_ITEM + t), 1);
      mbar_init(bar(B_ITEMFREE + t), 8 + 4 + 2);  // softmax, epilogue and issuing warps
      mbar_init(bar(B_DRAIN + t), 1);
      q_issued[t] = 0;
    }
    mbar_init(bar(B_NEXT), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // the first copies run under the TMEM allocation and the CTA-wide sync
    const PlainItem w = plain_item(p, blockIdx.x, blockIdx.y, blockIdx.z);
    if (w.n > 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_q) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_k) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_v) : "memory");
#pragma unroll
      for (int t = 0; t < ATT_NQ; ++t)
        if (w.hi[t] > w.lo[t]) issue_q(w, t);
      int kh, vh;
      kv_heads(w, kh, vh);
      const int first_round = min(STAGES, 2 * w.n);  // the ring is empty: nobody to wait for
      for (int fill = 0; fill < first_round; ++fill) issue_fill(w, kh, vh, fill, fill);
    }
    publish(w, 0);
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_holder)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  // TMEM columns (the allocation is all 512, so it starts at 0): S0 | S1 | O0 | O1
  constexpr uint32_t S_COL = 0, O_COL = ATT_NQ * BN;  // P (16-bit) over the first half of its S
  if (skip_launch) {  // nothing was started: give the TMEM columns back and leave
    if (threadIdx.x == 0) report_status(p.status);
    if (warp == 0)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                   "r"(512u)
                   : "memory");
    return;
  }
  // What takes as long as a work item is waited for while the ring is being filled.
  auto wait_item = [&](auto inline_tag, int i, uint32_t parity) -> bool {
    return mbar_wait_item<decltype(inline_tag)::value>(bar(i), parity, abort_flag, p.status,
                                                       ATT_ST_SOFTMAX, fills_issued);
  };
  // an item has been read: a warp's arrival
  auto item_read = [&](int q) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_ITEMFREE + (q & 1)));
  };

  // O / l of this thread's row of Q tile t (TMEM lane) to global memory, and its log sum
  auto store_rows = [&](int t, bool any, float l_row, float m_row, int b, int hq, int row,
                        auto&& o_is_read) {
    tc_fence_after();
    const float inv = (any && l_row > 0.0f) ? __fdividef(1.0f, l_row) : 0.0f;
    const uint32_t o_addr = (static_cast<uint32_t>((warp & 3) * 32) << 16) + O_COL + t * D;
    uint8_t* orow = reinterpret_cast<uint8_t*>(p.out) +
                    2ll * (b * p.o_stride_b + static_cast<long long>(row) * p.o_stride_s +
                           hq * p.o_stride_h);
#pragma unroll 1
    for (int cc = 0; cc < D; cc += 32) {
      uint32_t orr[32];
      if (any) {
        tmem_ld32<0>(o_addr + cc, orr);
        tmem_wait_ld32<0>(orr);
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) orr[e] = 0u;
      }
      if (cc == D - 32) o_is_read();
      if (row < p.Sq) {
#pragma unroll
        for (int e = 0; e < 32; e += 8) {
          uint4 v;
          uint32_t* vv = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            vv[i] = pack16<BF16>(__uint_as_float(orr[e + 2 * i]) * inv,
                                 __uint_as_float(orr[e + 2 * i + 1]) * inv);
          *reinterpret_cast<uint4*>(orow + 2 * (cc + e)) = v;
        }
      }
      __syncwarp();
    }
    if (p.lse && row < p.Sq)
      p.lse[b * p.lse_stride_b + hq * p.lse_stride_h + row] =
          (any && l_row > 0.0f) ? (m_row + log2f(l_row)) * 0.6931471805599453f : -INFINITY;
  };

  if (warp >= 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PlainRegs<D, BIAS, SINGLE>::OTHER));
    if (warp == 12) {
      // =========================== TMA producer =======================================
      if (lane == 0) {
        auto wait = [&](int i, uint32_t parity) {
          return mbar_wait(bar(i), parity, abort_flag, p.status, ATT_ST_PRODUCER);
        };
        PlainItem w = plain_item(p, blockIdx.x, blockIdx.y, blockIdx.z);
        int kh, vh;
        kv_heads(w, kh, vh);
        int base = 0;                        // fills of the items before this one
        int start = min(STAGES, 2 * w.n);    // of this one, issued before the CTA-wide sync
        bool ok = true, asked = false;
        int q = 0;
        auto fill_one = [&](int fill) {
          const int g = base + fill;
          if (g >= STAGES) ok = wait(B_KVEMPTY + g % STAGES, ((g / STAGES) & 1) ^ 1);
          if (ok) issue_fill(w, kh, vh, fill, g);
        };
#pragma unroll 1
        while (true) {
          const int total = 2 * w.n;
#pragma unroll 1
          for (int fill = start; fill < total && ok; ++fill) fill_one(fill);
          base += total;
          start = 0;
          if (!ok) break;
          if constexpr (SINGLE) break;  // no other item, and no answer to wait for
          // The next item is asked for when this one's last tiles have been: some visits before its
          // end, enough to hide the answer; earlier would take items from CTAs that are done sooner.
          mbar_expect_tx(bar(B_NEXT), 16);
          request_block(sbase + L::NEXT_OFF, bar(B_NEXT));
          asked = true;
          ok = wait(B_NEXT, q & 1);
          if (!ok) break;
          asked = false;
          int x, y, z;
          const bool more = requested_block(sbase + L::NEXT_OFF, x, y, z);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          if (more) {
            w = plain_item(p, x, y, z);
            kv_heads(w, kh, vh);
          } else {
            w.valid = 0;
          }
          ++q;
          if (q >= 2) ok = wait(B_ITEMFREE + (q & 1), ((q >> 1) & 1) ^ 1);
          if (!ok) break;
          publish(w, q);
          if (!more) break;
          if (w.n > 0) {  // its first K tile need not wait for the Q tiles to be free
            fill_one(0);
            start = 1;
          }
#pragma unroll
          for (int t = 0; t < ATT_NQ; ++t)
            if (ok && w.hi[t] > w.lo[t]) {
              if (q_issued[t] > 0) ok = wait(B_QEMPTY + t, (q_issued[t] - 1) & 1);
              if (ok) issue_q(w, t);
            }
          if (!ok) break;
        }
        if (asked) {  // gave up with an answer on its way into shared memory
          const uint64_t t0 = global_ns();
          while (!mbar_try_wait(bar(B_NEXT), q & 1) && global_ns() - t0 < ATT_WAIT_NS) {
          }
        }
      }
    } else if (warp <= 14) {
      // =========================== MMA issue ==========================================
      // One warp per Q tile, each between its softmax warps and the tensor pipe: every cycle it spends
      // between two groups of MMAs is one in which that tile's chain stands still. The warp stays
      // converged and one elected lane issues, so that addresses and descriptors are uniform
      // registers; a run of visits with nothing special has a loop of its own. The order of the work is
      // plain_issue's (attention_issue.cuh); here is what its steps are.
      const int t = warp - 13;
      const uint32_t idesc_qk = make_idesc(BF16 ? 1 : 0, ATT_BM, BN, 0, 0);
      const uint32_t idesc_pv = make_idesc(BF16 ? 1 : 0, ATT_BM, D, 0, 1);
      // Descriptors differ only in their 14-bit start-address field (address >> 4), the low part
      // of the low word.
      const uint64_t desc_k_major = make_desc(0, 16, 1024);               // K-major, SBO 1 KB
      const uint64_t desc_mn_major = make_desc(0, L::CHUNK_BYTES, 1024);  // MN-major V
      const uint32_t dk_hi = static_cast<uint32_t>(desc_k_major >> 32);
      const uint32_t dv_hi = static_cast<uint32_t>(desc_mn_major >> 32);
      constexpr uint32_t T16 = L::TILE_BYTES >> 4;
      const uint32_t q_lo = static_cast<uint32_t>(desc_k_major) + ((sbase + L::Q_OFF) >> 4);
      const uint32_t k_lo = static_cast<uint32_t>(desc_k_major) + ((sbase + L::KV_OFF) >> 4);
      const uint32_t v_lo = static_cast<uint32_t>(desc_mn_major) + ((sbase + L::KV_OFF) >> 4);
      auto desc_of = [](uint32_t lo, uint32_t hi) {
        return (static_cast<uint64_t>(hi) << 32) | lo;
      };
      auto wait = [&](int b, uint32_t parity) {
        return mbar_wait_warp<false>(bar(b), parity, abort_flag, p.status, ATT_ST_MMA);
      };
      uint32_t ppar = 0;  // parity of the next P
      const uint32_t d_o = O_COL + t * D, d_s = S_COL + t * BN, qst = q_lo + t * T16;

      // O_t += P_t V (P from TMEM, V MN-major from its ring stage); `acc` = 0 clears O first
      auto pv = [&](int vf, uint32_t acc) -> bool {
        const uint32_t vst = v_lo + (static_cast<uint32_t>(vf) & (STAGES - 1)) * T16;
        if (!wait(B_PFULL + t, ppar)) return false;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < BN / 16 - AP_REST; ++kk)
            mma_ts(d_o, d_s + kk * 8, desc_of(vst + kk * (2048 >> 4), dv_hi), idesc_pv,
                   kk == 0 ? acc : 1u);
        }
        const bool rest = wait(B_PREST + t, ppar);
        ppar ^= 1u;
        if (!rest) return false;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int kk = BN / 16 - AP_REST; kk < BN / 16; ++kk)
            mma_ts(d_o, d_s + kk * 8, desc_of(vst + kk * (2048 >> 4), dv_hi), idesc_pv, 1u);
        }
        return true;
      };
      // S = Q_t K^T (both operands K-major in shared memory), then announce it to the softmax warps.
      // The P V that reads the P in its columns is ahead of it in the pipe.
      auto qk = [&](int kf) {
        tc_fence_after();
        const uint32_t kst = k_lo + (static_cast<uint32_t>(kf) & (STAGES - 1)) * T16;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = ((kk / 4) * L::CHUNK_BYTES + (kk % 4) * 32) >> 4;
            if (kk == 0)
              mma_ss_first(d_s, desc_of(qst + off, dk_hi), desc_of(kst + off, dk_hi), idesc_qk);
            else
              mma_ss_acc(d_s, desc_of(qst + off, dk_hi), desc_of(kst + off, dk_hi), idesc_qk);
          }
          tc_commit(bar(B_SFULL + t));
        }
      };
      auto commit = [&](int b) {  // once this warp's MMAs are done
        if (elect_one()) tc_commit(bar(b));
      };
      // Whether a barrier's phase is complete, without waiting for it (try_wait would be suspended for
      // microseconds where only this warp's next step can complete it: 2 x 6000 full, 12 heads x 64,
      // whose last Q tile is empty, 547 us, now 307).
      auto ready = [&](int b, uint32_t parity) -> bool {
        return __all_sync(0xffffffffu, mbar_test(bar(b), parity));
      };
      // Values that are the same in every lane, in a way the compiler knows.
      auto uniform = [](int x) { return __reduce_max_sync(0xffffffffu, x); };
      auto open = [&](PlainCursor& c, int item, bool& ok) -> bool {  // false: there is no such item
        if (SINGLE && item > 0) return false;
        ok = wait(B_ITEM + (item & 1), (item >> 1) & 1);
        if (!ok) return false;
        volatile PlainItem& w = items[item & 1];
        const bool valid = __any_sync(0xffffffffu, w.valid != 0);
        if (valid) {
          c.lo = uniform(w.lo[t]);
          c.hi = uniform(w.hi[t]);
          c.n = uniform(w.n);
          c.item = item;
          c.v = 0;
        }
        item_read(item);
        return valid;
      };
      PlainSteps steps{
          open,
          [&](int i) { return SINGLE || ready(B_ITEM + (i & 1), (i >> 1) & 1); },
          [&](int f) { return wait(B_KVFULL + (f & (STAGES - 1)), (f / STAGES) & 1); },
          [&](int f) { return ready(B_KVFULL + (f & (STAGES - 1)), (f / STAGES) & 1); },
          [&](int f) { commit(B_KVEMPTY + (f & (STAGES - 1))); },
          [&](uint32_t parity) { return wait(B_QFULL + t, parity); },
          [&](uint32_t parity) { return ready(B_QFULL + t, parity); },
          qk,
          [&] { commit(B_QEMPTY + t); },
          [&](uint32_t parity) { return wait(B_OFREE + t, parity); },
          pv,
          [&] { commit(B_ODONE + t); }};
      const bool ok = plain_issue(steps);
      if (!ok && elect_one()) {
        // drain whatever was issued before giving up: a commit follows the MMAs of its own thread, and
        // which lane elect.sync takes is not specified
        tc_commit(bar(B_DRAIN + t));
        const uint64_t t0 = global_ns();
        while (!mbar_try_wait(bar(B_DRAIN + t), 0) && global_ns() - t0 < ATT_WAIT_NS) {
        }
      }
    }
  } else if (warp >= 8) {
    // =========================== epilogue =============================================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PlainRegs<D, BIAS, SINGLE>::EPILOGUE));
    const int wq = warp & 3;
    const int r = wq * 32 + lane;
    uint32_t opar[2] = {0u, 0u};  // parity of the next finished O
    auto wait = [&](int i, uint32_t parity) -> bool {
      return mbar_wait_warp<false>(bar(i), parity, abort_flag, p.status, ATT_ST_SOFTMAX);
    };
    struct Item {
      int q, b, h, m0;
      bool any0, any1;  // whether a Q tile has a key
    };
    auto finish = [&](const Item& w) -> bool {  // O and the row statistics of an item to global memory
      bool ok = true;
#pragma unroll
      for (int t = 0; t < ATT_NQ; ++t) {
        const bool any = t ? w.any1 : w.any0;
        if (ok) ok = wait_item(std::false_type{}, B_STAT + t, w.q & 1);
        if (ok && any) {
          ok = wait(B_ODONE + t, opar[t]);
          opar[t] ^= 1u;
        }
        if (!ok) break;
        const float* stat = reinterpret_cast<const float*>(smem + L::STAT_OFF) + t * 2 * ATT_BM;
        store_rows(t, any, stat[r], stat[ATT_BM + r], w.b, w.h + t * t_head, w.m0 + t * t_rows + r,
                   [&] {  // O and the statistics are read: the next item may write them
                     tc_fence_before();
                     __syncwarp();
                     if (lane == 0) {
                       if (any) mbar_arrive(bar(B_OFREE + t));
                       mbar_arrive(bar(B_STATFREE + t));
                     }
                   });
      }
      return ok;
    };
#pragma unroll 1
    for (int q = 0;; ++q) {
      if (!wait_item(std::false_type{}, B_ITEM + (q & 1), (q >> 1) & 1)) break;
      volatile PlainItem& w = items[q & 1];
      const bool valid = w.valid != 0;
      Item it;
      it.q = q;
      it.b = w.b;
      it.h = w.h;
      it.m0 = w.m0;
      it.any0 = w.hi[0] > w.lo[0];
      it.any1 = w.hi[1] > w.lo[1];
      item_read(q);
      if (!valid || !finish(it) || SINGLE) break;
    }
  } else {
    // =========================== softmax ==============================================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PlainRegs<D, BIAS, SINGLE>::SOFTMAX));
    const int t = warp >> 2;
    const int wq = warp & 3;
    const int rl = wq * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t s_addr = lanes + S_COL + t * BN;
    const uint32_t o_addr = lanes + O_COL + t * D;
    float* stat = reinterpret_cast<float*>(smem + L::STAT_OFF) + t * 2 * ATT_BM;
    const float sl2 = p.scale_log2;
    uint32_t s_par = 0;  // parity of the next S
    bool ok = true;
    auto wait = [&](int i, uint32_t parity) -> bool {
      return mbar_wait_warp<true>(bar(i), parity, abort_flag, p.status, ATT_ST_SOFTMAX);
    };
#pragma unroll 1
    for (int q = 0;; ++q) {
      ok = wait_item(std::true_type{}, B_ITEM + (q & 1), (q >> 1) & 1);
      if (!ok) break;
      volatile PlainItem& w = items[q & 1];
      const bool valid = w.valid != 0;
      const int row0 = w.m0 + t * t_rows;
      const int lo = w.lo[t], n_it = w.hi[t] - lo;
      int c0 = (w.first + lo * kv_step) * BN;  // first key of the visit
      float slope2 = 0.0f;
      if (BIAS != AP_NONE && valid && p.slopes)
        slope2 = p.slopes[w.h + t * t_head] * 1.4426950408889634f;
      item_read(q);
      if (!valid) break;
      const int row1 = min(p.Sq, row0 + ATT_BM) - 1;
      const int row = row0 + rl;
      int hi_i = p.Sk - 1, lo_i = 0;          // visible keys of this row
      int hi_min = p.Sk - 1, lo_max = 0;      // keys that every row of the tile sees
      if (p.causal) {
        hi_i = min(hi_i, row);
        hi_min = min(hi_min, row0);
      }
      if (p.win_right >= 0) {
        hi_i = min(hi_i, row + p.win_right);
        hi_min = min(hi_min, row0 + p.win_right);
      }
      if (p.win_left >= 0) {
        lo_i = max(0, row - p.win_left);
        lo_max = max(0, row1 - p.win_left);
      }
      const float kc = BIAS == AP_NONE ? 0.0f : __fdividef(slope2, sl2);
      // whether scores can carry the ramp: scaled by a positive number, and not too small a one
      const bool foldable = BIAS == AP_GENERAL && sl2 > 0.0f && fabsf(kc) < 1e30f;
      // The row sum in four shares, one of every fourth pair of columns; in a tile each is a chain of
      // the 16 even and one of the 16 odd columns. The order of attention.cu, whose rows are held by
      // four threads, so that the two agree to the last bit. Two chains and one share leave a relative
      // error of 1.4 / 2.0 x 2^-24 (rms, 4096 / 8192 keys), these 0.9 / 1.1, at the same speed within 1 to
      // 3 % either way (16 x 4096 causal 2147 / 2131 us, with ALiBi 2294 / 2333, 4 x 3001 window 1024 191.2
      // / 192.0, 2 x 2048 causal 74.0 / 76.6) as long as a pair is packed before it is added (else 2148,
      // 2374, 193.7, 76.7).
      float m_run = -INFINITY;
      float2 l_run[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
      float m_ref = 0.0f;  // m_run, or 0 while no key has been visible

#pragma unroll 1
      for (int itn = 0; itn < n_it; ++itn, c0 += kv_step * BN) {
        ok = wait(B_SFULL + t, s_par);
        if (!ok) break;
        s_par ^= 1u;
        if (SINGLE && t == 1 && itn == 0 && n_it > 1) {
          // half a visit behind the other Q tile, see AP_LAG
          constexpr unsigned LAG = BIAS == AP_NONE ? AP_LAG : AP_LAG_BIAS;
          const unsigned begin = static_cast<unsigned>(clock());
          for (int i = 0; i < 4096 && static_cast<unsigned>(clock()) - begin < LAG; ++i) {
          }
          __syncwarp();
        }
        tc_fence_after();
        // by a vote: a branch that the compiler knows to be uniform
        const bool cut = __any_sync(0xffffffffu, c0 + BN - 1 > hi_min || c0 < lo_max);
        // AP_GENERAL: a tile that lies on one side of its queries is a ramp too
        const bool up = BIAS == AP_GENERAL && __any_sync(0xffffffffu, foldable && c0 + BN - 1 <= row0);
        const bool down = BIAS == AP_GENERAL && __any_sync(0xffffffffu, foldable && c0 >= row1);
        const float unit = BIAS == AP_GENERAL && !up && !down ? 1.0f : sl2;
        uint32_t sr[BN];
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        // 32 columns: add the bias, hide what the row does not see, take the maximum
        auto take = [&](auto off_tag, auto cut_tag, auto bias_tag) {
          constexpr int OFF = decltype(off_tag)::value, TILE_BIAS = decltype(bias_tag)::value;
          if constexpr (TILE_BIAS == AP_GENERAL) {
            const float fi = static_cast<float>(row - c0);
#pragma unroll
            for (int c = OFF; c < OFF + 32; ++c)
              sr[c] = __float_as_uint(fmaf(-slope2, fabsf(fi - static_cast<float>(c)),
                                           __uint_as_float(sr[c]) * sl2));
          }
          if constexpr (TILE_BIAS == AP_RAMP || TILE_BIAS == AP_RAMP_TO_LAST) {
            const float kt = BIAS == AP_GENERAL && TILE_BIAS == AP_RAMP ? -kc : kc;
            const float2 kc2 = make_float2(kt, kt);
#pragma unroll
            for (int c = OFF; c < OFF + 32; c += 2)
              put_pair(sr + c, fma2(TILE_BIAS == AP_RAMP ? g_columns.v[c / 2] : g_columns_to_last.v[c / 2],
                                    kc2, pair_of(sr + c)));
          }
          if constexpr (decltype(cut_tag)::value) {
            const int hi_c = hi_i - c0 - OFF, lo_c = lo_i - c0 - OFF;
            if (__any_sync(0xffffffffu, hi_c < 31 || lo_c > 0)) {
              uint32_t keep = hi_c < 0 ? 0u : hi_c >= 31 ? 0xffffffffu : (2u << hi_c) - 1u;
              keep &= lo_c <= 0 ? 0xffffffffu : lo_c > 31 ? 0u : 0xffffffffu << lo_c;
#pragma unroll
              for (int c = 0; c < 32; ++c)
                if (!(keep & (1u << c))) sr[OFF + c] = 0xff800000u;
            }
          }
#pragma unroll
          for (int c = OFF; c < OFF + 32; c += 8)
#pragma unroll
            for (int i = 0; i < 4; ++i)
              mx[i] = max3(mx[i], __uint_as_float(sr[c + 2 * i]), __uint_as_float(sr[c + 2 * i + 1]));
        };
        auto take_all = [&](auto cut_tag, auto bias_tag) {
          tmem_wait_ld32<0>(sr);
          tmem_ld32<32>(s_addr + 32, sr);
          take(std::integral_constant<int, 0>{}, cut_tag, bias_tag);
          tmem_wait_ld32<32>(sr);
          tmem_ld32<64>(s_addr + 64, sr);
          take(std::integral_constant<int, 32>{}, cut_tag, bias_tag);
          tmem_wait_ld32<64>(sr);
          tmem_ld32<96>(s_addr + 96, sr);
          take(std::integral_constant<int, 64>{}, cut_tag, bias_tag);
          tmem_wait_ld32<96>(sr);
          take(std::integral_constant<int, 96>{}, cut_tag, bias_tag);
        };
        tmem_ld32<0>(s_addr, sr);
        auto take_tile = [&](auto bias_tag) {
          if (cut) take_all(std::true_type{}, bias_tag);
          else take_all(std::false_type{}, bias_tag);
        };
        if (BIAS == AP_GENERAL && up) take_tile(std::integral_constant<int, AP_RAMP_TO_LAST>{});
        else if (BIAS == AP_GENERAL && down) take_tile(std::integral_constant<int, AP_RAMP>{});
        else take_tile(std::integral_constant<int, BIAS>{});
        // the bias of the tile's column 0 (AP_RAMP_TO_LAST: of its last): slope_v * dist
        const float slope_v = BIAS == AP_GENERAL ? (up ? slope2 : down ? -slope2 : 0.0f) : slope2;
        const float dist = static_cast<float>((up ? c0 + BN - 1 : c0) - row);
        const float off = BIAS == AP_NONE ? 0.0f : slope_v * dist;
        const float m_raw = fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]);
        const float m_tile = fmaf(m_raw, unit, off);  // unit > 0: -inf stays -inf

        // lazy rescale: keep the old reference maximum unless the new one is much larger (or the
        // first). O is this thread's row; the commit behind S covers every P V before it.
        const bool grown = m_tile > m_run + ATT_LAZY_RESCALE;
        if (__any_sync(0xffffffffu, grown)) {
          const float factor = grown ? fast_exp2(m_run - m_tile) : 1.0f;  // 0 when m_run == -inf
          if (grown) m_run = m_ref = m_tile;
#pragma unroll
          for (int i = 0; i < 2; ++i)
            l_run[i] = make_float2(l_run[i].x * factor, l_run[i].y * factor);
          if (itn > 0) {
#pragma unroll 1
            for (int cc = 0; cc < D; cc += 32) {
              uint32_t orr[32];
              tmem_ld32<0>(o_addr + cc, orr);
              tmem_wait_ld32<0>(orr);
#pragma unroll
              for (int i = 0; i < 32; ++i)
                orr[i] = __float_as_uint(__uint_as_float(orr[i]) * factor);
              tmem_st32<0>(o_addr + cc, orr);
            }
          }
        }
        const float neg = BIAS == AP_NONE ? off - m_ref : fmaf(slope_v, dist, -m_ref);

        // P = exp2(x - m), 32 keys (16 packed columns) at a time, over the scores
        static_assert(AP_REST == 2, "the last 32 keys are two MMAs");
        const float2 unit2 = make_float2(unit, unit), neg2 = make_float2(neg, neg);
        float2 sum[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[i] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int g = 0; g < BN / 32; ++g) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int c = 32 * g + 2 * i;
            const float2 x = fma2(pair_of(sr + c), unit2, neg2);
            const float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
            pk[i] = pack16<BF16>(e.x, e.y);
            sum[i & 3] = add2(sum[i & 3], e);
          }
          tmem_st16(s_addr + 16 * g, pk);
          if (g >= BN / 32 - 2) {
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar((g == BN / 32 - 1 ? B_PREST : B_PFULL) + t));
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
          l_run[i] = add2(l_run[i], make_float2(sum[2 * i].x + sum[2 * i].y,
                                                sum[2 * i + 1].x + sum[2 * i + 1].y));
      }
      if (!ok) break;
      if (q > 0) {
        ok = wait(B_STATFREE + t, (q - 1) & 1);  // the last item's statistics have been read
        if (!ok) break;
      }
      stat[rl] = (l_run[0].x + l_run[0].y) + (l_run[1].x + l_run[1].y);
      stat[ATT_BM + rl] = m_run;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_STAT + t));
      if (SINGLE) break;
    }
  }

  // ------------------------------- teardown -------------------------------------------
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    // make sure no bulk copy of this CTA is still in flight before shared memory is released
    auto drain = [&](int i, int n) {
      if (n <= 0) return;
      bool done = false;
      const uint64_t t0 = global_ns();
      while (!(done = mbar_try_wait(bar(i), (n - 1) & 1)) && global_ns() - t0 < ATT_WAIT_NS) {
      }
      if (!done) atomicOr(p.status, ATT_ST_DRAIN);
    };
    for (int s = 0; s < STAGES; ++s) drain(B_KVFULL + s, fills_issued[s]);
    for (int t = 0; t < ATT_NQ; ++t) drain(B_QFULL + t, q_issued[t]);
    report_status(p.status);
  }
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(512u)
                 : "memory");
  }
}

template <int D, bool BF16, int BIAS, bool SINGLE>
static int launch_plain(const AttnParams& p, cudaStream_t stream) {
  // The attribute is set once per device; host threads that race on the first call each set
  // the same value (the call is idempotent) and publish the flag atomically.
  static std::atomic<bool> configured[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return TRX_ERR_CUDA;
  const bool cacheable = dev >= 0 && dev < 64;
  if (!cacheable || !configured[dev].load(std::memory_order_acquire)) {
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, attn_plain_kernel<D, BF16, BIAS, SINGLE>) != cudaSuccess)
      return TRX_ERR_CUDA;
    // the register split draws on what the block is launched with: never wait for more than that
    using Regs = PlainRegs<D, BIAS, SINGLE>;
    if (a.numRegs * 4 < 2 * Regs::SOFTMAX + Regs::EPILOGUE + Regs::OTHER) return TRX_ERR_UNSUPPORTED;
    if (cudaFuncSetAttribute(attn_plain_kernel<D, BF16, BIAS, SINGLE>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             PlainSmem<D>::DYN_BYTES) != cudaSuccess)
      return TRX_ERR_CUDA;
    if (cacheable) configured[dev].store(true, std::memory_order_release);
  }
  const int rows = p.pair_heads ? ATT_BM : ATT_NQ * ATT_BM;
  const unsigned m = (p.Sq + rows - 1) / rows, h = p.pair_heads ? p.Hq / 2 : p.Hq, b = p.B;
  const dim3 grid = p.order == AP_MHB ? dim3(m, h, b) : p.order == AP_HMB ? dim3(h, m, b) : dim3(h, b, m);
  attn_plain_kernel<D, BF16, BIAS, SINGLE><<<grid, AP_THREADS, PlainSmem<D>::DYN_BYTES, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? TRX_OK : TRX_ERR_CUDA;
}

template <int D, bool BF16, bool SINGLE>
static int launch_plain_bias(const AttnParams& p, cudaStream_t stream) {
  if (!(p.scale_log2 > 0.0f)) return launch_plain<D, BF16, AP_GENERAL, SINGLE>(p, stream);
  if (!p.slopes) return launch_plain<D, BF16, AP_NONE, SINGLE>(p, stream);
  // under a causal mask, or a window that ends at the query, every visible key is at or before it
  return p.causal || p.win_right == 0 ? launch_plain<D, BF16, AP_RAMP, SINGLE>(p, stream)
                                      : launch_plain<D, BF16, AP_GENERAL, SINGLE>(p, stream);
}

template <int D, bool BF16>
static int launch_plain_items(const AttnParams& p, bool single, cudaStream_t stream) {
  return single ? launch_plain_bias<D, BF16, true>(p, stream)
                : launch_plain_bias<D, BF16, false>(p, stream);
}

int launch_attn_plain(AttnParams& p, int64_t D, cudaStream_t stream) {
  const int rows = p.pair_heads ? ATT_BM : ATT_NQ * ATT_BM;
  const int64_t m = (p.Sq + rows - 1) / rows, h = p.pair_heads ? p.Hq / 2 : p.Hq;
  const bool single = m * h * p.B <= sm_count_of_current_device();
  p.order = AP_MHB;
  if (p.causal && m <= 65535) {
    // Heaviest row blocks first: over all heads of all batches while their keys and values are a third
    // of L2, over those of one batch up to 100 MB. One head after the other / one batch / all, us:
    // 4 x 2048, 32 / 8 heads x 128 (34 MB) 158 / 147 / 144, 2 x 4096 (34 MB) 269 / 248 / 248, 8 x 2048
    // (67 MB) 292 / 286 / 288, 16 x 4096 (268 MB, 17 of a batch) 2174 / 2166 / 2374. The upper line is
    // not fitted: 1 x 8192, 32 / 32 heads (134 MB) takes 546 / 490 / 489, 1 x 6144 (101 MB) 334 / 286 / 285.
    const double kv = 4.0 * p.Sk * static_cast<double>(D) * p.Hq / p.group;  // bytes of a batch
    if (kv * p.B <= 40e6) p.order = AP_HBM;
    else if (kv <= 100e6) p.order = AP_HMB;
  }
  if (D == 128)
    return p.is_bf16 ? launch_plain_items<128, true>(p, single, stream)
                     : launch_plain_items<128, false>(p, single, stream);
  return p.is_bf16 ? launch_plain_items<64, true>(p, single, stream)
                   : launch_plain_items<64, false>(p, single, stream);
}

}  // namespace trx
