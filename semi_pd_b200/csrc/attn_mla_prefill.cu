// Ragged prefill of multi-head latent attention (MLA) with the heads expanded, on tcgen05: K and V of every head are made
// from the cached latent rows by one GEMM per layer (spd_mla_gather brings the rows together, spd_gemm expands them), and
// the attention then runs at the heads' own widths, 192 (128 + 64 rotated) for the scores and 128 for the values.
//
// Reference: DeepseekV2AttentionMLA.forward_normal (python/sglang/srt/models/deepseek_v2.py:591-631), used there for
// prefill batches without a cached prefix; here it serves prefixes as well, as long as a latent row is met by enough
// queries to pay for its expansion.  The absorbed form (attn_mla.cu) needs 1088 multiply-adds per query, key and head and
// this one 320, plus 131072 per key and head.  4096 new tokens in 4 requests, two of them behind 515 cached tokens, 16
// heads, whole attention layer called after other work: 606 us absorbed, 185 here; warm and alone this kernel 67, the rows 6, the
// expanding GEMM 26.
//
// Items are two consecutive 128-query tiles of one head that share every K / V tile of 64 keys, one tile per softmax
// warpgroup; they are dealt to one persistent CTA per SM by weight (tile_list).  Roles as in attn_prefill.cu (384 threads):
//   warps 0-3 / 4-7  softmax warpgroups, one thread per query row, with the true running max (a reference that lags by up to
//                    2^8 rounds the largest probability of a row too: a layer's rms error was 0.2 % above the absorbed
//                    form's, so it is 0.6 % below, and no slower) and the sum of the
//                    rounded probabilities (see softmax_chunk).  O is rescaled after the unit's exponentials, when its last PV has long finished;
//   warp 8 / warp 9  K loader (two boxes of the expanded rows, one of the rotated latent part) / V loader, one lane each;
//   warp 10 / 11     MMA issuer of warpgroup 0 / 1: S(u) = Q K_u^T into one of two buffers, O += P(u) V_u with P from TMEM
//                    over the S it came from; PV(u), then S(u + 2).
// smem: Q 2 x 48 KB, three K slots of 24 KB and two V slots of 16 KB, 2.5 KB per softmax warp for its output rows.
// TMEM: S 2 x 2 x 64, O 2 x 128 columns.
// Every mbarrier wait is bounded (see mbar_wait_bounded, spd_wait_status).
#include <cuda.h>

#include "common.cuh"
#include "prefill_tiles.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace spd {

constexpr int kMpThreads = 384;
constexpr int kMpM = 128;                        // query rows per warpgroup
constexpr int kMpN = 64;                         // keys per tile
constexpr int kMpNope = 128, kMpRope = 64, kMpDV = 128, kMpRank = 512;
constexpr int kMpDQ = kMpNope + kMpRope;
constexpr int kMpHeadCols = kMpNope + kMpDV;     // columns of a head in an expanded row
constexpr int kMpQBytes = kMpM * kMpDQ * 2;      // three swizzle blocks of [128 rows x 128 bytes]
constexpr int kMpKBytes = kMpN * kMpDQ * 2;      // three of [64 rows x 128 bytes]
constexpr int kMpVBytes = kMpN * kMpDV * 2;      // two
constexpr int kMpK = 3, kMpV = 2;                // ring slots
constexpr int kMpRowBytes = 80;                  // 32 output columns of a row, and 16 bytes against bank conflicts
constexpr int kMpStage = 32 * kMpRowBytes;       // per softmax warp
constexpr int kMpBars = 512;
constexpr int kMpSmem = 2 * kMpQBytes + kMpK * kMpKBytes + kMpV * kMpVBytes + 8 * kMpStage + kMpBars + kTileList * 2 + 1024;
static_assert(kMpSmem <= 232448, "shared memory of one block");
static_assert(8 * kMpStage >= kTileList * 4, "the list is sorted in the staging area");

struct MlaPrefillParams {
  void* out;
  const void* q;
  const void* kv;    // [rows, H * 256]: a head's 128 key and 128 value columns
  const void* rows;  // [rows, 576]: the latent rows, their last 64 columns are the rotated part of every head's key
  const int32_t* kv_start;
  const int32_t* prefix_lens;
  const int32_t* extend_lens;
  const int32_t* extend_start_loc;
  int H, batch, tiles_x, total_items, sorted;
  uint32_t heads_m, heads_s, per_x_m, per_x_s, tiles_x_m, tiles_x_s;
  int64_t q_stride, out_stride;
  float scale_log2;
  unsigned* wait_expired;
};

struct MpRaw {
  int req, qx, head;
  int ext, pre, start, kv0;
};
struct MpItem {
  int head, kv0, n;             // first row of the request's keys; tiles of 64 keys (of the later query tile)
  int m0[2], rows[2], nt[2], q_row0[2], pre;
};

__device__ __forceinline__ MpRaw mp_raw(const MlaPrefillParams& p, const TileList& tl, int idx) {
  MpRaw r{0, 0, 0, 0, 0, 0, 0};
  if (idx < tl.items) {
    if (tl.list != nullptr) {
      const int e = fastdiv(idx, p.heads_m, p.heads_s);
      r.head = idx - e * p.H;
      const int slot = tl.list[e];
      r.req = fastdiv(slot, p.tiles_x_m, p.tiles_x_s);
      r.qx = slot - r.req * p.tiles_x;
    } else {
      const int ix = fastdiv(idx, p.per_x_m, p.per_x_s);
      const int rest = idx - ix * (p.H * p.batch);
      r.qx = p.tiles_x - 1 - ix;
      r.req = fastdiv(rest, p.heads_m, p.heads_s);
      r.head = rest - r.req * p.H;
    }
    r.ext = __ldg(p.extend_lens + r.req);
    r.pre = __ldg(p.prefix_lens + r.req);
    r.start = __ldg(p.extend_start_loc + r.req);
    r.kv0 = __ldg(p.kv_start + r.req);
  }
  return r;
}
// the same in every lane of a warp, and known to be
__device__ __forceinline__ MpRaw mp_raw_uniform(MpRaw r) {
  r.req = __shfl_sync(0xffffffffu, r.req, 0);
  r.qx = __shfl_sync(0xffffffffu, r.qx, 0);
  r.head = __shfl_sync(0xffffffffu, r.head, 0);
  r.ext = __shfl_sync(0xffffffffu, r.ext, 0);
  r.pre = __shfl_sync(0xffffffffu, r.pre, 0);
  r.start = __shfl_sync(0xffffffffu, r.start, 0);
  r.kv0 = __shfl_sync(0xffffffffu, r.kv0, 0);
  return r;
}
__device__ __forceinline__ MpItem mp_item(const MpRaw& raw) {
  MpItem it;
  it.head = raw.head;
  it.kv0 = raw.kv0;
  it.pre = raw.pre;
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    it.m0[w] = (2 * raw.qx + w) * kMpM;
    const int rows = min(kMpM, raw.ext - it.m0[w]);
    it.rows[w] = rows > 0 ? rows : 0;
    it.nt[w] = rows > 0 ? (raw.pre + it.m0[w] + rows + kMpN - 1) / kMpN : 0;  // keys that the tile's last row sees
    it.q_row0[w] = raw.start + it.m0[w];
  }
  it.n = max(it.nt[0], it.nt[1]);
  return it;
}

// Column c + lane of one query row's output by a warp, from the keys the row sees alone, before the division by the sum:
// for rows whose output is not finite, since the tiles hold keys that the row does not see, and their P of 0 times an
// infinite or NaN value is NaN.
template <typename T>
__device__ __noinline__ float mp_row_alone(const T* q, const T* kv, const T* rope, int64_t kv_stride, int keys, int c,
                                           float scale, float m_off) {
  const int lane = threadIdx.x & 31;
  float acc = 0.f;
#pragma unroll 1
  for (int j0 = 0; j0 < keys; j0 += 32) {
    const int j = j0 + lane;
    float prob = 0.f;
    if (j < keys) {
      float dot = 0.f;
#pragma unroll 1
      for (int d = 0; d < kMpDQ; d += 8) {
        const Vec16<T> a = ldv(q + d);
        const Vec16<T> b = ldv(d < kMpNope ? kv + j * kv_stride + d : rope + static_cast<int64_t>(j) * (kMpRank + kMpRope) + d - kMpNope);
#pragma unroll
        for (int e = 0; e < 8; ++e) dot = fmaf(to_f32<T>(a.e()[e]), to_f32<T>(b.e()[e]), dot);
      }
      prob = to_f32<T>(from_f32<T>(fast_exp2(fmaf(dot, scale, -m_off))));
    }
    const int n = min(32, keys - j0);
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const float pi = __shfl_sync(0xffffffffu, prob, i);
      acc = fmaf(pi, to_f32<T>(kv[(j0 + i) * kv_stride + kMpNope + c + lane]), acc);
    }
    if (__all_sync(0xffffffffu, isnan(acc))) break;  // nothing changes that any more
  }
  return acc;
}

template <typename T>
__global__ void __launch_bounds__(kMpThreads, 1)
attn_mla_prefill_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                        const __grid_constant__ CUtensorMap tmR, const MlaPrefillParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + 2 * kMpQBytes;
  uint8_t* sV = sK + kMpK * kMpKBytes;
  uint8_t* sO = sV + kMpV * kMpVBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sO + 8 * kMpStage);
  uint64_t* q_full = bars;               // 2
  uint64_t* k_full = q_full + 2;         // kMpK
  uint64_t* k_empty = k_full + kMpK;     // kMpK: both issuers
  uint64_t* v_full = k_empty + kMpK;     // kMpV
  uint64_t* v_empty = v_full + kMpV;     // kMpV: both issuers
  uint64_t* s_full = v_empty + kMpV;     // 4: [warpgroup][buffer]
  uint64_t* p_full = s_full + 4;         // 4
  uint64_t* pv_done = p_full + 4;        // 4
  uint64_t* o_free = pv_done + 4;        // 2
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_free + 2);
  uint32_t* n_tiles = tmem_slot + 1;
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 2);
  uint16_t* list = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(bars) + kMpBars);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const int cta = blockIdx.x, ncta = gridDim.x;

  if (warp == 10) {
    if (lane == 0) {
      for (int i = 0; i < 2; ++i) mbar_init(&q_full[i], 1);
      for (int i = 0; i < kMpK; ++i) {
        mbar_init(&k_full[i], 1);
        mbar_init(&k_empty[i], 2);
      }
      for (int i = 0; i < kMpV; ++i) {
        mbar_init(&v_full[i], 1);
        mbar_init(&v_empty[i], 2);
      }
      for (int i = 0; i < 4; ++i) {
        mbar_init(&s_full[i], 1);
        mbar_init(&p_full[i], 4);
        mbar_init(&pv_done[i], 1);
      }
      for (int i = 0; i < 2; ++i) mbar_init(&o_free[i], 4);
      *n_tiles = 0;
      *dead = 0;
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (warp == 8 && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmKV);
    tma_prefetch_desc(&tmR);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_S = *tmem_slot;       // [warpgroup][buffer] x 64 columns; P over the first 32 of a buffer
  const uint32_t tmem_O = tmem_S + 256;     // [warpgroup] x 128

  griddep_wait();
  TileList tl{p.total_items, nullptr};
  if (p.sorted)
    tl = tile_list<kMpThreads>(
        p.batch * p.tiles_x, p.H, p.total_items,
        [&](int slot) {
          MpRaw raw{};
          raw.req = fastdiv(slot, p.tiles_x_m, p.tiles_x_s);
          raw.qx = slot - raw.req * p.tiles_x;
          raw.ext = __ldg(p.extend_lens + raw.req);
          raw.pre = __ldg(p.prefix_lens + raw.req);
          const MpItem it = mp_item(raw);
          return (it.nt[0] + it.nt[1] + 1) / 2;
        },
        reinterpret_cast<uint32_t*>(sO), n_tiles, list);

  if (warp >= 10) {
    // ===================== MMA issuer of warpgroup 0 (warp 10) / 1 (warp 11) =====================
    const bool leader = elect_one();
    const int w = warp - 10;
    constexpr uint32_t idesc_qk = umma_idesc<T>(kMpM, kMpN, 0, 0);    // A, B K-major
    constexpr uint32_t idesc_pv = umma_idesc<T>(kMpM, kMpDV, 0, 1);   // A = P (TMEM), B = V MN-major
    const uint64_t qd = umma_desc_sw128(smem_u32(sQ + w * kMpQBytes), 16, 1024);
    const uint64_t kd = umma_desc_sw128(smem_u32(sK), 16, 1024);
    const uint64_t vd = umma_desc_sw128(smem_u32(sV), kMpN * 128, 1024);
    const uint32_t qk_hi = static_cast<uint32_t>(qd >> 32), v_hi = static_cast<uint32_t>(vd >> 32);
    RingSlot<kMpK> ks;  // the next S's K slot
    RingSlot<kMpV> vs;  // the next PV's V slot
    uint32_t su = 0;    // S units issued (all items): buffer su & 1
    uint32_t pu = 0;    // PV units issued
    uint32_t eq = 0;    // items of the warpgroup
    bool q_ahead = false;
    auto load_q = [&](const MpItem& it) {
      const int row0 = w == 0 ? it.q_row0[0] : it.q_row0[1];
      if (leader) {
        mbar_expect_tx(&q_full[w], kMpQBytes);
#pragma unroll
        for (int b = 0; b < 3; ++b)
          tma_load_2d(sQ + w * kMpQBytes + b * 16384, &tmQ, &q_full[w], it.head * kMpDQ + b * 64, row0, kEvictFirst);
      }
      __syncwarp();
    };
    int idx = pf_rank(0, cta, ncta);
    MpRaw raw = mp_raw_uniform(mp_raw(p, tl, idx));
    for (int kk = 0; idx < tl.items; ++kk) {
      const MpItem it = mp_item(raw);
      idx = pf_rank(kk + 1, cta, ncta);
      raw = mp_raw_uniform(mp_raw(p, tl, idx));
      if (it.n == 0) continue;
      const int nt = w == 0 ? it.nt[0] : it.nt[1];
      if (nt > 0) {
        if (!q_ahead) load_q(it);
        q_ahead = false;
        mbar_wait_bounded(&q_full[w], eq & 1, dead);
      }
      // S(j) of the warpgroup if it uses the tile, and K_j given back: by both issuers, also by one that does not use it,
      // which waits for the tile first so that its arrivals keep to the ring's rounds.  The buffer's previous P has been
      // consumed by PV(j - 2), issued earlier by this thread (tcgen05.mma executes in issue order).
      auto next_s = [&](int j) {
        mbar_wait_bounded(&k_full[ks.i], ks.round, dead);
        tc_fence_after_sync();
        if (j < nt) {
          uint32_t qa = static_cast<uint32_t>(qd), ka = static_cast<uint32_t>(kd) + ks.i * (kMpKBytes / 16);
          const uint32_t td = tmem_S + w * 128 + (su & 1) * kMpN;
#pragma unroll 1
          for (int k = 0; k < kMpDQ / 16; ++k) {
            umma_ss_if(leader, td, qa, ka, qk_hi, idesc_qk, k);
            const bool block = (k & 3) == 3;  // the next 64 channels
            qa += block ? (kMpM * 128 - 96) / 16 : 2;
            ka += block ? (kMpN * 128 - 96) / 16 : 2;
          }
          umma_commit_if(leader, &s_full[w * 2 + (su & 1)]);
          ++su;
        }
        umma_commit_if(leader, &k_empty[ks.i]);
        ks.next();
      };
      next_s(0);
      if (it.n > 1) next_s(1);
      for (int j = 0; j < it.n; ++j) {
        if (j < nt) {
          const uint32_t b = pu & 1;
          mbar_wait_bounded(&p_full[w * 2 + b], (pu >> 1) & 1, dead);
          mbar_wait_bounded(&v_full[vs.i], vs.round, dead);
          if (j == 0) mbar_wait_bounded(&o_free[w], (eq & 1) ^ 1, dead);  // previous item's O has been read
          if (j == nt - 1 && idx < tl.items) {
            // every S of the item is complete: its P has arrived.  Q's memory is free for the next item.
            const MpItem next = mp_item(raw);
            q_ahead = (w == 0 ? next.nt[0] : next.nt[1]) > 0;
            if (q_ahead) load_q(next);
          }
          tc_fence_after_sync();
          uint32_t va = static_cast<uint32_t>(vd) + vs.i * (kMpVBytes / 16);
          uint32_t pa = tmem_S + w * 128 + b * kMpN;
          uint32_t acc = j > 0 ? 1u : 0u;
#pragma unroll 1
          for (int k = 0; k < kMpN / 16; ++k) {
            umma_ts_if(leader, tmem_O + w * kMpDV, pa, va, v_hi, idesc_pv, acc);
            pa += 8;
            va += 2048 / 16;
            acc = 1;
          }
          umma_commit_if(leader, &pv_done[w * 2 + b]);
          ++pu;
        } else {
          mbar_wait_bounded(&v_full[vs.i], vs.round, dead);
        }
        umma_commit_if(leader, &v_empty[vs.i]);
        vs.next();
        if (j + 2 < it.n) next_s(j + 2);
      }
      if (nt > 0) ++eq;
    }
  } else if (warp >= 8) {
    // ===================== K loader (warp 8) / V loader (warp 9) =====================
    if (elect_one()) {
      RingSlot<kMpK> ks;
      RingSlot<kMpV> vs;
      int idx = pf_rank(0, cta, ncta);
      MpRaw raw = mp_raw(p, tl, idx);
      for (int k = 0; idx < tl.items; ++k) {
        const MpItem it = mp_item(raw);
        idx = pf_rank(k + 1, cta, ncta);
        raw = mp_raw(p, tl, idx);
        const int col = it.head * kMpHeadCols;
        for (int j = 0; j < it.n; ++j) {
          const int row = it.kv0 + j * kMpN;
          if (warp == 8) {
            uint8_t* dst = sK + ks.i * kMpKBytes;
            mbar_wait_bounded(&k_empty[ks.i], ks.round ^ 1, dead);
            mbar_expect_tx(&k_full[ks.i], kMpKBytes);
            tma_load_2d(dst, &tmKV, &k_full[ks.i], col, row, kEvictNormal);
            tma_load_2d(dst + kMpN * 128, &tmKV, &k_full[ks.i], col + 64, row, kEvictNormal);
            tma_load_2d(dst + 2 * kMpN * 128, &tmR, &k_full[ks.i], kMpRank, row, kEvictNormal);
            ks.next();
          } else {
            uint8_t* dst = sV + vs.i * kMpVBytes;
            mbar_wait_bounded(&v_empty[vs.i], vs.round ^ 1, dead);
            mbar_expect_tx(&v_full[vs.i], kMpVBytes);
            tma_load_2d(dst, &tmKV, &v_full[vs.i], col + kMpNope, row, kEvictNormal);
            tma_load_2d(dst + kMpN * 128, &tmKV, &v_full[vs.i], col + kMpNope + 64, row, kEvictNormal);
            vs.next();
          }
        }
      }
    }
  } else {
    // ===================== softmax warpgroups (one thread per query row) =====================
    const int w = warp >> 2;
    const int row = threadIdx.x & 127;  // == TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t ts = tmem_S + lane_base + w * 128;
    const uint32_t to = tmem_O + lane_base + w * kMpDV;
    uint8_t* stage = sO + warp * kMpStage;
    uint32_t u = 0;  // units of this warpgroup (all items)
    // PV of unit v has finished; at most that phase of its barrier is outstanding: S of unit v + 1 was issued after PV of
    // unit v - 1
    auto wait_pv = [&](uint32_t v) {
      mbar_wait_bounded(&pv_done[w * 2 + (v & 1)], (v >> 1) & 1, dead);
      tc_fence_after_sync();
    };
    int idx = pf_rank(0, cta, ncta);
    MpRaw raw = mp_raw(p, tl, idx);
    for (int k = 0; idx < tl.items; ++k) {
      const MpItem it = mp_item(raw);
      idx = pf_rank(k + 1, cta, ncta);
      raw = mp_raw(p, tl, idx);
      const int nt = w == 0 ? it.nt[0] : it.nt[1];
      if (nt == 0) continue;
      const int m0 = w == 0 ? it.m0[0] : it.m0[1];
      const int rows = w == 0 ? it.rows[0] : it.rows[1];
      const int q_row0 = w == 0 ? it.q_row0[0] : it.q_row0[1];
      const int limit = it.pre + m0 + row;  // last visible key
      const float scale = p.scale_log2;
      float m_used = -INFINITY, l = 0.f;
      for (int j = 0; j < nt; ++j, ++u) {
        const int kv = j * kMpN;
        const bool need_mask = kv + kMpN - 1 > it.pre + m0;
        const uint32_t tsh = ts + (u & 1) * kMpN;
        mbar_wait_bounded(&s_full[w * 2 + (u & 1)], (u >> 1) & 1, dead);
        tc_fence_after_sync();
        uint32_t ra[32], rb[32], pk[kMpN / 2];
        const float mx = need_mask ? softmax_load_max<true, false>(tsh, ra, rb, kv, limit, 0)
                                   : softmax_load_max<false, false>(tsh, ra, rb, kv, limit, 0);
        const bool raise = __any_sync(0xffffffffu, mx > m_used);
        float alpha = 1.f;
        if (raise) {
          const float m_new = fmaxf(m_used, mx);
          alpha = (m_used == -INFINITY) ? 0.f : fast_exp2((m_used - m_new) * scale);
          l *= alpha;
          m_used = m_new;
        }
        l += softmax_unit<T>(ra, rb, pk, scale, (m_used == -INFINITY) ? 0.f : m_used * scale);
        tmem_st_32x32b_x32(tsh, pk);
        if (raise && j > 0) {
          wait_pv(u - 1);
          rescale_row128(to, alpha);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[w * 2 + (u & 1)]);
      }
      // ---- O / l: TMEM -> registers -> 32 columns of 32 rows in shared memory -> global, 64 bytes per row and store ----
      wait_pv(u - 1);
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      const float m_off = (m_used == -INFINITY) ? 0.f : m_used * scale;
      const int row0 = row & ~31;  // the warp's rows of the tile
      T* dst = reinterpret_cast<T*>(p.out) + static_cast<int64_t>(q_row0 + row0) * p.out_stride +
               static_cast<int64_t>(it.head) * kMpDV;
#pragma unroll 1
      for (int c = 0; c < kMpDV; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(to + c, r);
        tmem_ld_wait();
        if (c + 32 == kMpDV) {
          // every O column of this warp is in registers: the next item's first PV may overwrite it
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&o_free[w]);
        }
        float z = 0.f;  // NaN when a value of these columns is infinite or NaN
#pragma unroll
        for (int i = 0; i < 32; ++i) z = fmaf(__uint_as_float(r[i]), 0.f, z);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint4 v;
          v.x = pack2<T>(__uint_as_float(r[8 * i]) * inv_l, __uint_as_float(r[8 * i + 1]) * inv_l);
          v.y = pack2<T>(__uint_as_float(r[8 * i + 2]) * inv_l, __uint_as_float(r[8 * i + 3]) * inv_l);
          v.z = pack2<T>(__uint_as_float(r[8 * i + 4]) * inv_l, __uint_as_float(r[8 * i + 5]) * inv_l);
          v.w = pack2<T>(__uint_as_float(r[8 * i + 6]) * inv_l, __uint_as_float(r[8 * i + 7]) * inv_l);
          *reinterpret_cast<uint4*>(stage + lane * kMpRowBytes + i * 16) = v;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int rr = i * 8 + (lane >> 2), piece = lane & 3;
          if (row0 + rr < rows)
            *reinterpret_cast<uint4*>(dst + rr * p.out_stride + c + piece * 8) =
                *reinterpret_cast<const uint4*>(stage + rr * kMpRowBytes + piece * 16);
        }
        __syncwarp();
        uint32_t todo = __ballot_sync(0xffffffffu, row < rows && isnan(z));
#pragma unroll 1
        for (; todo != 0; todo &= todo - 1) {
          const int src = __ffs(todo) - 1;
          const T* kv = reinterpret_cast<const T*>(p.kv) + static_cast<int64_t>(it.kv0) * p.H * kMpHeadCols + it.head * kMpHeadCols;
          const T* rope = reinterpret_cast<const T*>(p.rows) + static_cast<int64_t>(it.kv0) * (kMpRank + kMpRope) + kMpRank;
          const T* q = reinterpret_cast<const T*>(p.q) + static_cast<int64_t>(q_row0 + row0 + src) * p.q_stride + it.head * kMpDQ;
          const float f = mp_row_alone<T>(q, kv, rope, static_cast<int64_t>(p.H) * kMpHeadCols, it.pre + m0 + row0 + src + 1, c,
                                          scale, __shfl_sync(0xffffffffu, m_off, src));
          dst[src * p.out_stride + c + lane] = from_f32<T>(f * __shfl_sync(0xffffffffu, inv_l, src));
        }
      }
    }
  }

  griddep_launch_dependents();
  tc_fence_before_sync();
  __syncthreads();
  if (*dead) {
    wait_drain();
    if (threadIdx.x == 0) wait_report(p.wait_expired);
  }
  if (warp == 10) tmem_dealloc(tmem_S, 512);
}

// The latent rows of every request's keys, one request after another, and where each begins.  Block (request, 16 rows), a
// thread's pieces all in flight: latency is what it costs (5.2 k rows, 12 MB: 64 rows a block, piece after piece, 10.2 us;
// 5.7 here).
constexpr int kGatherRows = 16;
template <typename T>
__global__ void __launch_bounds__(256)
mla_gather_kernel(T* __restrict__ rows, int32_t* __restrict__ kv_start, const T* __restrict__ pool,
                  const int32_t* __restrict__ req_to_token, const int64_t* __restrict__ req_pool_indices,
                  const int32_t* __restrict__ prefix_lens, const int32_t* __restrict__ extend_lens, int64_t total,
                  int64_t rtt_stride) {
  constexpr int kChunks = (kMpRank + kMpRope) / 8;  // 16-byte pieces of a row
  __shared__ int part[8];
  __shared__ int slots[kGatherRows];
  griddep_wait();
  const int req = blockIdx.x, tid = threadIdx.x, at = blockIdx.y * kGatherRows;
  const int len = prefix_lens[req] + extend_lens[req];
  if (at >= len && blockIdx.y > 0) return;
  int before = 0;
  for (int r = tid; r < req; r += 256) before += prefix_lens[r] + extend_lens[r];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if ((tid & 31) == 0) part[tid >> 5] = before;
  if (tid < kGatherRows && at + tid < len) slots[tid] = req_to_token[req_pool_indices[req] * rtt_stride + at + tid];
  __syncthreads();
  int start = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) start += part[i];
  if (blockIdx.y == 0 && tid == 0) kv_start[req] = start;
  // (rows past `total`, what the caller says the lengths add up to, are not written)
  const int64_t n = min(static_cast<int64_t>(min(kGatherRows, len - at)), total - start - at);
  T* dst = rows + (static_cast<int64_t>(start) + at) * (kMpRank + kMpRope);
  constexpr int kPer = (kGatherRows * kChunks + 255) / 256;
  Vec16<T> v[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int i = tid + 256 * k, r = i / kChunks, c = i - r * kChunks;
    if (i < n * kChunks) v[k] = ldv(pool + static_cast<int64_t>(slots[r]) * (kMpRank + kMpRope) + c * 8);
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k)
    if (tid + 256 * k < n * kChunks) stv(dst + (tid + 256 * k) * 8, v[k]);
  griddep_launch_dependents();
}

}  // namespace spd

using namespace spd;

extern "C" {

int spd_mla_gather(void* rows, int32_t* kv_start, const void* kv_pool, const int32_t* req_to_token,
                   const int64_t* req_pool_indices, const int32_t* prefix_lens, const int32_t* extend_lens, int64_t batch,
                   int64_t total_kv, int64_t max_kv_len, int kv_lora_rank, int rope_dim, int64_t req_to_token_stride,
                   int dtype, spd_stream_t stream) {
  SPD_REQUIRE(rows && kv_start && kv_pool && req_to_token && req_pool_indices && prefix_lens && extend_lens, SPD_E_BADARG,
              "spd_mla_gather: null pointer");
  SPD_REQUIRE(kv_lora_rank == kMpRank && rope_dim == kMpRope, SPD_E_SHAPE,
              "spd_mla_gather: built for kv_lora_rank 512 + rope 64 (got %d + %d)", kv_lora_rank, rope_dim);
  SPD_REQUIRE(batch >= 0 && total_kv >= 0 && total_kv < (1ll << 31) && max_kv_len >= 0 && max_kv_len <= static_cast<int64_t>(kGatherRows) * 65535,
              SPD_E_BADARG, "spd_mla_gather: bad sizes");
  SPD_REQUIRE(aligned16(rows) && aligned16(kv_pool), SPD_E_ALIGN, "spd_mla_gather: pointers must be 16-B aligned");
  if (batch == 0) return 0;
  const unsigned chunks = static_cast<unsigned>((max_kv_len + kGatherRows - 1) / kGatherRows);
  SPD_DISPATCH_DTYPE(dtype, {
    SPD_CUDA(launch(mla_gather_kernel<T>, dim3((unsigned)batch, chunks > 0 ? chunks : 1), dim3(256), 0, as_stream(stream),
                    pdl_enabled(), (T*)rows, kv_start, (const T*)kv_pool, req_to_token, req_pool_indices, prefix_lens,
                    extend_lens, total_kv, req_to_token_stride));
  });
  return 0;
}

int spd_attn_mla_prefill(void* out, const void* q, const void* kv, const void* rows, const int32_t* kv_start,
                         const int32_t* prefix_lens, const int32_t* extend_lens, const int32_t* extend_start_loc,
                         int64_t batch, int64_t total_tokens, int64_t total_kv, int64_t max_extend_len, int64_t max_kv_len,
                         int num_heads, int nope_dim, int rope_dim, int v_dim, int64_t q_stride, int64_t out_stride,
                         float sm_scale, int dtype, int sm_budget, spd_stream_t stream) {
  SPD_REQUIRE(out && q && kv && rows && kv_start && prefix_lens && extend_lens && extend_start_loc, SPD_E_BADARG,
              "spd_attn_mla_prefill: null pointer");
  SPD_REQUIRE(nope_dim == kMpNope && rope_dim == kMpRope && v_dim == kMpDV, SPD_E_SHAPE,
              "spd_attn_mla_prefill: built for 128 + 64 key and 128 value channels (got %d + %d, %d)", nope_dim, rope_dim, v_dim);
  SPD_REQUIRE(num_heads > 0 && batch >= 0 && total_tokens >= 0 && total_kv >= 0 && max_extend_len >= 0 && sm_scale > 0.f &&
                  total_tokens < (1ll << 31) && total_kv < (1ll << 31) && max_kv_len < (1ll << 31),
              SPD_E_BADARG, "spd_attn_mla_prefill: bad sizes");
  SPD_REQUIRE(q_stride % 8 == 0 && out_stride % 8 == 0 && aligned16(out) && aligned16(q) && aligned16(kv) && aligned16(rows),
              SPD_E_ALIGN, "spd_attn_mla_prefill: strides must be multiples of 8 and pointers 16-B aligned");
  if (batch == 0 || total_tokens == 0 || max_extend_len == 0) return 0;
  MlaPrefillParams p{};
  if (int rc = wait_flag(&p.wait_expired)) return rc;
  p.out = out;
  p.q = q;
  p.kv = kv;
  p.rows = rows;
  p.kv_start = kv_start;
  p.prefix_lens = prefix_lens;
  p.extend_lens = extend_lens;
  p.extend_start_loc = extend_start_loc;
  p.H = num_heads;
  p.batch = static_cast<int>(batch);
  p.q_stride = q_stride;
  p.out_stride = out_stride;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
  const int64_t tiles_x = (max_extend_len + 2 * kMpM - 1) / (2 * kMpM);
  SPD_REQUIRE(tiles_x * num_heads * batch < (1ll << 30), SPD_E_SHAPE, "spd_attn_mla_prefill: too many work items");
  p.tiles_x = static_cast<int>(tiles_x);
  p.total_items = static_cast<int>(tiles_x * num_heads * batch);
  fastdiv_magic(static_cast<uint32_t>(num_heads), p.heads_m, p.heads_s);
  fastdiv_magic(static_cast<uint32_t>(num_heads) * static_cast<uint32_t>(batch), p.per_x_m, p.per_x_s);
  fastdiv_magic(static_cast<uint32_t>(tiles_x), p.tiles_x_m, p.tiles_x_s);
  const int device_sms = device_sm_count_cached();
  const int sms = sm_budget > 0 && sm_budget < device_sms ? sm_budget : device_sms;
  const int grid = p.total_items < sms ? p.total_items : sms;
  // the list serves where some CTA gets more than one item; 16 bits name its tiles and hold their weight
  p.sorted = p.total_items > grid && total_tokens / (2 * kMpM) + batch <= kTileList && batch * tiles_x <= 65536 &&
             max_kv_len < 65535ll * kMpN;
  CUtensorMap tq, tkv, tr;
  const uint64_t kv_cols = static_cast<uint64_t>(num_heads) * kMpHeadCols;
  if (int rc = get_tmap(&tq, q, static_cast<uint64_t>(total_tokens), static_cast<uint64_t>(num_heads) * kMpDQ,
                        static_cast<uint64_t>(q_stride), kMpM))
    return rc;
  if (int rc = get_tmap(&tkv, kv, static_cast<uint64_t>(total_kv), kv_cols, kv_cols, kMpN)) return rc;
  if (int rc = get_tmap(&tr, rows, static_cast<uint64_t>(total_kv), kMpRank + kMpRope, kMpRank + kMpRope, kMpN)) return rc;
  SPD_DISPATCH_DTYPE(dtype, {
    auto kern = attn_mla_prefill_kernel<T>;
    static bool configured = false;
    if (!configured) {
      SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMpSmem));
      configured = true;
    }
    SPD_CUDA(launch(kern, dim3(grid), dim3(kMpThreads), kMpSmem, as_stream(stream), pdl_enabled(), tq, tkv, tr, p));
  });
  return 0;
}

}  // extern "C"
