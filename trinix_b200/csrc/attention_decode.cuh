// Attention forward for few query rows against many keys (decoding against a KV cache).
// Included by attention.cu, whose parameter block, barrier and TMA wrappers it uses.
//
// The work is reading K and V once: per key and kv head 4 * D bytes and, with `group` query heads
// of Sq rows on that kv head, only group * Sq rows of arithmetic. The tcgen05 kernel gives such a
// call one 128-row tile per query head, i.e. one serial chain over all keys per CTA, mostly on
// padding rows, and reads the keys of a kv head once per pair of query heads: 139.5 us for 16
// sequences of 4093 keys (32 / 8 heads, head dim 128), 1.9 TB/s; one sequence of 32768 keys
// 507 us. Here (45.0 us, 6.0 TB/s; 34.6 us)
//   * the query heads of a kv head and their rows are packed into tiles of 16 rows, the M of one
//     mma.sync.m16n8k16, one or two tiles to a warp: K and V are read once per 16 or 32 packed rows,
//     i.e. once for up to 32 of them (again for more, mostly from L2), and the padding is less than
//     one such tile and not 128 rows;
//   * the keys are split over the CTAs of a thread-block cluster and, inside a CTA, over its four
//     warps. Each warp owns a ring of 16-key K and V tiles (TMA, 128-byte swizzle, its own
//     mbarriers) and its own running maximum, sum and O accumulators, so no warp waits for
//     another one before the end;
//   * the partial results meet in shared memory, then over distributed shared memory inside the
//     cluster: no workspace, one launch, and sums in an order fixed by the shape of the whole call
//     (the number of splits goes by the batch, too) and the SM count of the device.
// Scores, sums and O are fp32, probabilities go into the second product in the activation dtype,
// as in the tcgen05 kernel; an mma.sync at M = 16 is issued 32 times per 8 KB of keys, so the
// tensor pipe idles beside the memory system either way.
#pragma once

#include <cooperative_groups.h>

namespace trx {

constexpr int DEC_WARPS = 4;
constexpr int DEC_THREADS = DEC_WARPS * 32;
constexpr int DEC_KEYS = 16;     // keys of one tile: the K of one mma
constexpr int DEC_STAGES = 3;    // tiles of a warp's ring
constexpr int DEC_CTAS_PER_SM = 2;
constexpr int DEC_MAX_SPLIT = 16;

template <int D, int MT>
struct DecSmem {
  static constexpr int CHUNKS = D / 64;
  static constexpr int CHUNK_BYTES = DEC_KEYS * 128;
  static constexpr int TILE_BYTES = CHUNKS * CHUNK_BYTES;             // K or V of 16 keys
  static constexpr int RING_BYTES = DEC_STAGES * 2 * TILE_BYTES;      // one warp's ring
  static constexpr int ROWS = 16 * MT;
  static_assert(ROWS * D * 4 <= RING_BYTES, "a warp's partial O reuses its ring");
  static constexpr int BAR_OFF = DEC_WARPS * RING_BYTES;
  static constexpr int ML_OFF = BAR_OFF + DEC_WARPS * DEC_STAGES * 8;  // max, sum per warp and row
  static constexpr int CTA_ML_OFF = ML_OFF + 2 * DEC_WARPS * ROWS * 4;
  static constexpr int FLAG_OFF = CTA_ML_OFF + 2 * ROWS * 4;
  static constexpr int TOTAL = FLAG_OFF + (DEC_WARPS + 1) * 4;  // a flag per warp, one of the CTA
  static constexpr int DYN_BYTES = TOTAL + 1024;  // slack for 1024-byte alignment
};

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                          uint32_t b1) {
  if constexpr (BF16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Grid (splits, kv units * row tiles, B), clusters of all the splits of one row tile. Packed row r
// of a kv unit is row r / group of query head unit * group + r % group.
template <int D, bool BF16, int MT>
__global__ void __launch_bounds__(DEC_THREADS, DEC_CTAS_PER_SM)
    attn_decode_kernel(const __grid_constant__ AttnParams p) {
  using L = DecSmem<D, MT>;
  namespace cg = cooperative_groups;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t sbase = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q4 = lane & 3, rl = lane >> 2;
  const int nsplit = gridDim.x, split = blockIdx.x, b = blockIdx.z;
  const int group = p.group, rows = group * p.Sq;
  const int row_tiles = (rows + L::ROWS - 1) / L::ROWS;
  const int unit = blockIdx.y / row_tiles;
  const int r0 = (blockIdx.y - unit * row_tiles) * L::ROWS;
  const int h0 = unit * group;

  // keys that any row of this tile sees, in tiles of 16, and this CTA's share of them
  const int s_min = r0 / group, s_max = min(rows - 1, r0 + L::ROWS - 1) / group;
  int hi = p.Sk - 1, lo = 0, hi_min = p.Sk - 1, lo_max = 0;
  if (p.causal) {
    hi = min(hi, s_max);
    hi_min = min(hi_min, s_min);
  }
  if (p.win_right >= 0) {
    hi = min(hi, s_max + p.win_right);
    hi_min = min(hi_min, s_min + p.win_right);
  }
  if (p.win_left >= 0) {
    lo = max(0, s_min - p.win_left);
    lo_max = max(0, s_max - p.win_left);
  }
  const int t_lo = lo / DEC_KEYS, n_tiles = hi < lo ? 0 : hi / DEC_KEYS + 1 - t_lo;
  const int share = (n_tiles + nsplit - 1) / nsplit;
  const int first = t_lo + min(n_tiles, split * share) + warp;
  const int last = t_lo + min(n_tiles, (split + 1) * share);
  int n_it = first < last ? (last - first + DEC_WARPS - 1) / DEC_WARPS : 0;

  const uint32_t ring = sbase + warp * L::RING_BYTES;
  const uint32_t bars = sbase + L::BAR_OFF + warp * DEC_STAGES * 8;
  int* no_result = reinterpret_cast<int*>(smem + L::FLAG_OFF);  // [DEC_WARPS], then the CTA's
  volatile int* abort_flag = no_result + warp;
  const int kh = h0 / p.k_hdiv, vh = h0 / p.v_hdiv, kb = b * p.k_bmul, vb = b * p.v_bmul;
  auto issue_fill = [&](int it) {  // one lane: K and V of the it-th tile of this warp
    const int s = it % DEC_STAGES, key0 = (first + it * DEC_WARPS) * DEC_KEYS;
    mbar_expect_tx(bars + 8 * s, 2 * L::TILE_BYTES);
#pragma unroll
    for (int c = 0; c < L::CHUNKS; ++c)
      tma_load_4d(ring + s * 2 * L::TILE_BYTES + c * L::CHUNK_BYTES, &p.tm_k, bars + 8 * s, c * 64,
                  key0, kh, kb);
#pragma unroll
    for (int c = 0; c < L::CHUNKS; ++c)
      tma_load_4d(ring + (s * 2 + 1) * L::TILE_BYTES + c * L::CHUNK_BYTES, &p.tm_v, bars + 8 * s,
                  c * 64, key0, vh, vb);
  };
  if (lane == 0) {
    for (int s = 0; s < DEC_STAGES; ++s) mbar_init(bars + 8 * s, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int it = 0; it < min(n_it, DEC_STAGES); ++it) issue_fill(it);
  }
  __syncwarp();
  // A launch that follows a recorded failure writes nothing; the copies above are waited for. The
  // word may turn non-zero at any time (another CTA, another stream), so one lane reads it for its
  // warp, whose trip count depends on it; what the other warps and CTAs read is settled at the end.
  unsigned int seen = 0;
  if (lane == 0) seen = *reinterpret_cast<volatile unsigned int*>(p.status);
  const bool skip = __shfl_sync(0xffffffffu, seen, 0) != 0u;
  if (skip) n_it = min(n_it, DEC_STAGES);

  // Q as mma A fragments: rows rl and rl + 8 of each 16-row tile
  uint32_t qf[MT][D / 16][4];
  int row_s[MT][2];  // query row of this thread's packed rows (clamped for the padding rows)
  float slope2[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = r0 + 16 * m + 8 * e + rl;
      const bool live = r < rows;
      const int s = (live ? r : rows - 1) / group, h = h0 + (live ? r : rows - 1) % group;
      row_s[m][e] = s;
      slope2[m][e] = p.slopes ? p.slopes[h] * 1.4426950408889634f : 0.0f;
      const uint16_t* qrow = reinterpret_cast<const uint16_t*>(p.q) + b * p.q_stride_b +
                             s * p.q_stride_s + h * p.q_stride_h + 2 * q4;
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          qf[m][ks][2 * c + e] =
              live ? __ldg(reinterpret_cast<const uint32_t*>(qrow + 16 * ks + 8 * c)) : 0u;
    }

  float o[MT][D / 8][4];
  float m_run[MT][2], l_run[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      m_run[m][e] = -INFINITY;
      l_run[m][e] = 0.0f;
    }
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) o[m][n][i] = 0.0f;
  }
  // ldmatrix row addresses. K (16 keys x 16 of D, not transposed): matrices keys 0-7 / 8-15 by
  // column halves; V (transposed): keys 0-7 / 8-15 first, then the column halves.
  const int k_key = ((lane >> 4) << 3) + (lane & 7), k_col = (lane >> 3) & 1;
  const int v_key = (((lane >> 3) & 1) << 3) + (lane & 7), v_col = lane >> 4;
  const float sl2 = p.scale_log2;
  const bool has_alibi = p.slopes != nullptr;
  bool ok = true;

  int it = 0;
#pragma unroll 1
  for (; it < n_it; ++it) {
    const int st = it % DEC_STAGES;
    ok = __all_sync(0xffffffffu, mbar_wait(bars + 8 * st, (it / DEC_STAGES) & 1, abort_flag,
                                           p.status, ATT_ST_SOFTMAX));
    if (!ok) break;
    const uint32_t kt = ring + st * 2 * L::TILE_BYTES, vt = kt + L::TILE_BYTES;
    const int c0 = (first + it * DEC_WARPS) * DEC_KEYS;
    float s[MT][2][4];  // [row tile][keys 0-7 / 8-15][row rl: keys 2 q4, 2 q4 + 1; row rl + 8]
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) s[m][n][i] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      uint32_t kf[4];
      const int col = (ks % 4) * 2 + k_col;
      ldsm_x4(kt + (ks / 4) * L::CHUNK_BYTES + k_key * 128 + ((col ^ (lane & 7)) << 4), kf);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        mma_16816<BF16>(s[m][0], qf[m][ks], kf[0], kf[1]);
        mma_16816<BF16>(s[m][1], qf[m][ks], kf[2], kf[3]);
      }
    }
    const bool need_mask = c0 + DEC_KEYS - 1 > hi_min || c0 < lo_max;
    uint32_t pf[MT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = row_s[m][e];
        int hi_i = p.Sk - 1, lo_i = 0;
        if (p.causal) hi_i = min(hi_i, i);
        if (p.win_right >= 0) hi_i = min(hi_i, i + p.win_right);
        if (p.win_left >= 0) lo_i = max(0, i - p.win_left);
        float x[4];  // keys 2 q4, 2 q4 + 1, 8 + 2 q4, 8 + 2 q4 + 1 of the tile
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int j = c0 + 8 * n + 2 * q4 + c;
            float v = s[m][n][2 * e + c] * sl2;
            if (has_alibi) v = fmaf(-slope2[m][e], fabsf(static_cast<float>(i - j)), v);
            if (need_mask && (j < lo_i || j > hi_i)) v = -INFINITY;
            x[2 * n + c] = v;
          }
        float mx = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        // the reference maximum follows only when it is far behind, as in the tcgen05 kernel
        if (mx > m_run[m][e] + ATT_LAZY_RESCALE || (m_run[m][e] == -INFINITY && mx > -INFINITY)) {
          const float f = fast_exp2(m_run[m][e] - mx);  // 0 when m_run == -inf
          m_run[m][e] = mx;
          l_run[m][e] *= f;
#pragma unroll
          for (int n = 0; n < D / 8; ++n) {
            o[m][n][2 * e] *= f;
            o[m][n][2 * e + 1] *= f;
          }
        }
        const float m_ref = m_run[m][e] == -INFINITY ? 0.0f : m_run[m][e];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = fast_exp2(x[k] - m_ref);
        l_run[m][e] += (x[0] + x[1]) + (x[2] + x[3]);
        pf[m][e] = pack16<BF16>(x[0], x[1]);
        pf[m][2 + e] = pack16<BF16>(x[2], x[3]);
      }
    }
#pragma unroll
    for (int dn = 0; dn < D / 16; ++dn) {
      uint32_t vf[4];
      const int col = (dn % 4) * 2 + v_col;
      ldsm_x4_trans(vt + (dn / 4) * L::CHUNK_BYTES + v_key * 128 + ((col ^ (lane & 7)) << 4), vf);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        mma_16816<BF16>(o[m][2 * dn], pf[m], vf[0], vf[1]);
        mma_16816<BF16>(o[m][2 * dn + 1], pf[m], vf[2], vf[3]);
      }
    }
    __syncwarp();  // every lane has read the tile
    if (lane == 0 && !skip && it + DEC_STAGES < n_it) issue_fill(it + DEC_STAGES);
  }
  if (!ok) {  // gave up on tile `it`: wait (bounded) for the copies still in flight
    for (int f = it; f < min(n_it, it + DEC_STAGES); ++f) {
      const uint64_t t0 = global_ns();
      bool done = false;
      while (!done && global_ns() - t0 < ATT_WAIT_NS)
        done = mbar_try_wait(bars + 8 * (f % DEC_STAGES), (f / DEC_STAGES) & 1);
      if (!done) atomicOr(p.status, ATT_ST_DRAIN);
    }
    __syncwarp();  // lane 0 reports what every lane has recorded
  }
  const bool has_result = ok && !skip;
  if (!has_result && lane == 0) {
    *abort_flag = 1;
    report_status(p.status);
  }

  // ---- this warp's partial result: O into its own ring, row maxima and sums beside it ----------
  // (not from a warp without one: a copy that was given up may still be writing the ring)
  float* ml = reinterpret_cast<float*>(smem + L::ML_OFF);        // [2][DEC_WARPS][ROWS]
  float* cta_ml = reinterpret_cast<float*>(smem + L::CTA_ML_OFF);  // [2][ROWS]
  float* ow = reinterpret_cast<float*>(smem + warp * L::RING_BYTES);
  __syncwarp();
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = 16 * m + 8 * e + rl;
      float l = l_run[m][e];
      l += __shfl_xor_sync(0xffffffffu, l, 1);
      l += __shfl_xor_sync(0xffffffffu, l, 2);
      if (q4 == 0) {
        ml[warp * L::ROWS + r] = m_run[m][e];
        ml[(DEC_WARPS + warp) * L::ROWS + r] = l;
      }
      if (has_result && r0 + r < rows)
#pragma unroll
        for (int n = 0; n < D / 8; ++n)
          *reinterpret_cast<float2*>(ow + r * D + 8 * n + 2 * q4) =
              make_float2(o[m][n][2 * e], o[m][n][2 * e + 1]);
    }
  __syncthreads();
  bool whole = true;  // every warp (below: of the cluster) has a result; else nothing is written
#pragma unroll
  for (int w = 0; w < DEC_WARPS; ++w) whole = whole && no_result[w] == 0;

  // out[row, 4 c4 ..] = acc / l, and the row's LSE
  auto emit = [&](int r, int c4, float4 acc, float mx, float l) {
    const int s = (r0 + r) / group, h = h0 + (r0 + r) % group;
    const float inv = l > 0.0f ? __fdividef(1.0f, l) : 0.0f;
    if (whole) {
      uint2 v;
      v.x = pack16<BF16>(acc.x * inv, acc.y * inv);
      v.y = pack16<BF16>(acc.z * inv, acc.w * inv);
      *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(p.out) + b * p.o_stride_b +
                                s * p.o_stride_s + h * p.o_stride_h + 4 * c4) = v;
      if (p.lse && c4 == 0)
        p.lse[b * p.lse_stride_b + h * p.lse_stride_h + s] =
            l > 0.0f ? (mx + log2f(l)) * 0.6931471805599453f : -INFINITY;
    }
  };
  // sum of n partial results of one row: weights 2^(m_i - max m), 0 for an empty part
  const int live_rows = min(L::ROWS, rows - r0);
  float* o0 = reinterpret_cast<float*>(smem);
  for (int idx = threadIdx.x; idx < live_rows * (D / 4); idx += DEC_THREADS) {
    const int r = idx / (D / 4), c4 = idx % (D / 4);
    float mx = -INFINITY, l = 0.0f;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) mx = fmaxf(mx, ml[w * L::ROWS + r]);
    const float m_ref = mx == -INFINITY ? 0.0f : mx;
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) {
      const float f = fast_exp2(ml[w * L::ROWS + r] - m_ref);
      const float4 v = *reinterpret_cast<const float4*>(
          reinterpret_cast<const float*>(smem + w * L::RING_BYTES) + r * D + 4 * c4);
      l = fmaf(f, ml[(DEC_WARPS + w) * L::ROWS + r], l);
      acc.x = fmaf(f, v.x, acc.x);
      acc.y = fmaf(f, v.y, acc.y);
      acc.z = fmaf(f, v.z, acc.z);
      acc.w = fmaf(f, v.w, acc.w);
    }
    if (nsplit == 1) {
      emit(r, c4, acc, mx, l);
    } else {
      *reinterpret_cast<float4*>(o0 + r * D + 4 * c4) = acc;  // this thread's own element
      if (c4 == 0) {
        cta_ml[r] = mx;
        cta_ml[L::ROWS + r] = l;
      }
    }
  }
  if (nsplit == 1) return;
  if (threadIdx.x == 0) no_result[DEC_WARPS] = whole ? 0 : 1;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  static_assert(DEC_MAX_SPLIT <= 32, "one lane per CTA");
  whole = __all_sync(0xffffffffu, lane >= nsplit ||
                                      cluster.map_shared_rank(no_result, lane)[DEC_WARPS] == 0);
  for (int idx = split * DEC_THREADS + threadIdx.x; idx < live_rows * (D / 4);
       idx += nsplit * DEC_THREADS) {
    const int r = idx / (D / 4), c4 = idx % (D / 4);
    float mx = -INFINITY, l = 0.0f;
    for (int k = 0; k < nsplit; ++k) mx = fmaxf(mx, cluster.map_shared_rank(cta_ml, k)[r]);
    const float m_ref = mx == -INFINITY ? 0.0f : mx;
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int k = 0; k < nsplit; ++k) {
      const float* kml = cluster.map_shared_rank(cta_ml, k);
      const float f = fast_exp2(kml[r] - m_ref);
      const float4 v =
          *reinterpret_cast<const float4*>(cluster.map_shared_rank(o0, k) + r * D + 4 * c4);
      l = fmaf(f, kml[L::ROWS + r], l);
      acc.x = fmaf(f, v.x, acc.x);
      acc.y = fmaf(f, v.y, acc.y);
      acc.z = fmaf(f, v.z, acc.z);
      acc.w = fmaf(f, v.w, acc.w);
    }
    emit(r, c4, acc, mx, l);
  }
  cluster.sync();  // no CTA leaves while another one reads its shared memory
}

// CTAs that share the keys of one row tile: the power of two that a cost, in quarters of the time
// of one 16-key tile (0.75 to 1.1 us), makes the cheapest. A CTA costs a start and an end (14), the merge of a
// cluster 10 more; a second CTA on an SM slows both down at either end (5, with two row tiles per
// warp 10); clusters of 8 and 16 wait for room in one GPC once there are many of them. Fitted to
// every split of 2624 shapes (1 to 16 rows, 64 to 32768 keys, 1 to 1536 units, both head dims): 1.7 %
// slower than the best split in the mean. Splitting wherever a warp keeps two tiles and the chip has
// room, and by two for every last wave that is under half full, is 6.0 % slower, and far off in
// single shapes (32 / 8 heads, head dim 128, that / this / the tcgen05 kernel): 24 x 256 keys, 16 rows
// 40.6 / 23.7 / 28.6 us; 8 x 256 keys, 16 rows 14.8 / 11.2 / 10.8 us; 2 x 4096 keys, 1 row 18.2 / 12.6
// / 69.5 us.
static int decode_splits(const AttnParams& p, int64_t units, bool wide) {
  int64_t keys = p.Sk;  // that some row sees
  if (p.causal && p.Sq < keys) keys = p.Sq;
  if (p.win_right >= 0 && static_cast<int64_t>(p.Sq) + p.win_right < keys) keys = p.Sq + p.win_right;
  if (p.win_left >= 0 && static_cast<int64_t>(p.Sq) + p.win_left + p.win_right < keys)
    keys = p.Sq + p.win_left + p.win_right;
  const int64_t sms = sm_count_of_current_device(), slots = sms * DEC_CTAS_PER_SM;
  const int64_t tiles = (keys + DEC_KEYS - 1) / DEC_KEYS;
  auto cost = [&](int64_t n) {
    const int64_t ctas = units * n, waves = (ctas + slots - 1) / slots;
    const int64_t chain = (tiles + n * DEC_WARPS - 1) / (n * DEC_WARPS);
    int64_t ends = 14;
    if (n > 1) ends += waves > 1 ? 13 : 10;
    if (ctas > sms) ends += wide ? 10 : 5;
    if (n >= 8 && ctas > 64) ends += n == 8 ? 4 : 6;
    if (n == 16) ends += 1;
    return waves * (ends + 4 * chain);
  };
  int best = 1;
  for (int n = 2; n <= DEC_MAX_SPLIT && tiles >= n * DEC_WARPS; n *= 2)
    if ((n == 2 || units * n <= slots) && cost(n) < cost(best)) best = n;
  return best;
}

template <int D, bool BF16, int MT>
static int launch_decode(const AttnParams& p, cudaStream_t stream) {
  using L = DecSmem<D, MT>;
  auto kernel = attn_decode_kernel<D, BF16, MT>;
  static std::atomic<bool> configured[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return TRX_ERR_CUDA;
  const bool cacheable = dev >= 0 && dev < 64;
  if (!cacheable || !configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::DYN_BYTES) !=
            cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
            cudaSuccess)
      return TRX_ERR_CUDA;
    if (cacheable) configured[dev].store(true, std::memory_order_release);
  }
  const int64_t units = static_cast<int64_t>(p.Hq / p.group) *
                        ((static_cast<int64_t>(p.group) * p.Sq + L::ROWS - 1) / L::ROWS);
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr{};
  const unsigned n = static_cast<unsigned>(decode_splits(p, units * p.B, MT == 2));
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = n;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3(n, static_cast<unsigned>(units), static_cast<unsigned>(p.B));
  cfg.blockDim = dim3(DEC_THREADS);
  cfg.dynamicSmemBytes = L::DYN_BYTES;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, p) == cudaSuccess ? TRX_OK : TRX_ERR_CUDA;
}

// Calls that take this kernel: up to 16 query rows. The tcgen05 kernels spend the same time on any
// Sq up to 128 (they work on whole 128-row tiles), this one works on tiles of 16 packed rows. Measured
// at 4096 keys, head dim 128, this / attention_plain.cu: Sq = 16, B = 16, 32 / 32 heads 160 / 198 us;
// 32 / 8 heads 94 / 139 us; 32 / 1 heads (512 packed rows) 90 / 138 us, B = 1 29 / 56 us; Sq = 32, B = 4,
// 32 / 8 heads 52 / 57, Sq = 64 89 / 57 us. The exception is a single key tile of attention.cu's kernel
// that is nearly full, in one wave of CTAs, at head dim 128, against two row tiles per warp here: 97 to
// 128 keys 8.4 to 8.7 / 7.3 to 7.8 us (96 keys 8.1 to 8.4 / 7.6 to 7.9, 64 keys 7.3 / 7.4; 129 keys 9.2 /
// 10.0).
static bool use_decode(const AttnParams& p, int64_t D) {
  const int64_t rows = static_cast<int64_t>(p.Sq) * p.group;
  if (p.Sq > 16 || (p.Hq / p.group) * ((rows + 15) / 16) > 65535) return false;
  const int64_t ctas = static_cast<int64_t>(p.B) * (p.pair_heads ? p.Hq / 2 : p.Hq);
  return !(D == 128 && rows > 16 && p.Sk > 96 && p.Sk <= ATT_BN && ctas <= sm_count_of_current_device());
}

}  // namespace trx
