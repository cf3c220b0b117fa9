// Ragged chunked-prefill ("extend") attention on tcgen05: QK^T and PV both run on the tensor
// cores with S and O accumulators in TMEM.  One pass over [prefix pages || new tokens] with the
// causal mask applied only on the diagonal tiles — no separate ragged / paged kernels and no LSE
// merge as in the flashinfer backend (S/layers/attention/flashinfer_backend.py:425-445).
// Semantics: S/layers/attention/torch_native_backend.py:26-109.
//
// PERSISTENT CTAs, one per SM of the caller's partition, walk a static work list of ITEMS.  An
// item is TWO 128-row query tiles of one request that share every K/V tile:
//   * GQA with an even group (Llama: 4 query heads per KV head): the same 128 tokens of two query
//     heads of one KV head — identical causal range, perfectly balanced;
//   * otherwise: two consecutive 128-token tiles of one query head.
// Each query tile belongs to one softmax warpgroup (own S, P, O, running max and row sum), so a
// K/V tile staged once in shared memory feeds 2 x 128 query rows (half the L2->SM traffic per
// FLOP of a single-tile CTA).
// HALF-TILE UNITS.  A 128-token K/V tile is consumed as two independent 64-column halves a / b of
// the warpgroup's S tile (S_a = Q K[0:64]^T in TMEM columns 0-63, S_b in 64-127, each with its own
// full / P-ready barriers).  While a warpgroup exponentiates half b of tile j, the tensor core
// runs PV_a(j) and S_a(j+1) for it, so its softmax never waits for the S -> softmax -> PV -> S
// chain of the whole tile (ncu on the whole-tile version: softmax warps 50 % of their time on
// s_full, tensor pipe 44 %); the second warpgroup fills the remaining tensor time.
// Roles (384 threads):
//   warps 0-3 / 4-7  softmax warpgroup 0 / 1: one thread per query row, ONE pass per tile in the
//                    exp2 domain against a lazily raised reference max (O in TMEM is rescaled only
//                    when a row outgrows it by 2^8 — then the tile is redone; rare after tile 0).
//                    P never touches shared memory: the 16-bit probabilities are written back
//                    into TMEM over the first 32 columns of the S half they came from
//                    (tcgen05.st) and feed the PV MMA as its A operand from TMEM;
//                    epilogue O / l from TMEM through shared memory and TMA stores (a ragged last tile: from registers);
//   warp 8, warp 9   K / V loader into 128-byte-swizzled smem; one 4-slot ring K_j V_j K_{j+1} ...
//                    runs ahead of the consumer ACROSS items, so an item's first tiles are in
//                    flight while the previous item drains.  A tile whose 128 page-table entries
//                    are consecutive slots (what the run allocator produces, memory_pool.py) is a
//                    strided 2-D box of the pool and is fetched with two TMA tensor copies by one
//                    lane; any other tile (scattered slots, the ragged tail of a sequence) is
//                    gathered row by row through req_to_token with 16-byte cp.async, whose completion arrives on
//                    the slot's barrier by itself;
//   warp 10, warp 11 MMA issuer of warpgroup 0 / 1: S_h = Q K_j[h]^T (both K-major in smem), O += P_h V_j[h] (P
//                    from TMEM, V MN-major in smem); the order is PV(j,h) then S(j+1,h) (which overwrites the columns
//                    P(j,h) lives in; tcgen05.mma executes in order).  The next item's Q tile is fetched (TMA) when the
//                    item's last S is complete.
// The issuers' own time bounded the kernel while one lane of one warp issued for both warpgroups from unrolled code: 65 clk
// per MMA and 250 between two units.  Whole warps with uniform operands, short loops and an issuer per warpgroup (warm, the
// kernel alone): 8 requests of 1024 new tokens on average, half of them behind 1024 cached ones, 32 / 8 heads: 193 -> 176 us;
// 4 requests of 2048, 16 / 4 heads, window 1024: 142 -> 132 us.  Slower: S issued 128 keys wide with softmax and PV still
// per half and one issuer (160 / 128 us against 156 / 112 with the sorted items), or with two (250 us: both warpgroups in one phase).
// With an issuer each nothing keeps the warpgroups apart, and on half of the CTAs they fell into one phase: warpgroup 1
// starts every item behind warpgroup 0 (`turn`).  64 requests of 128 tokens, 32 / 8 heads: 36.1 us with one issuer, 41.5 with
// two, 36.2 here; 8 of 1024: 80.1, 82.8, 80.9; 16 of 500: 58.0, 62.1, 60.4 (of unequal lengths 96, 75, 74).
// Items are ordered heaviest first (pf_sort) and dealt to the CTAs in snake order.
// smem: Q0 Q1 + 4 K/V slots + output staging = 7 x 32 KB, the list of tiles.
// TMEM: S0a/P0a S0b/P0b | S1a/P1a S1b/P1b | O0 | O1 = 512 columns.
#include <cuda.h>

#include "common.cuh"
#include "prefill_tiles.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace spd {

constexpr int kPfThreads = 384;  // 12 warps -> 168 registers per thread
constexpr int kPfM = 128;    // query rows per warpgroup tile
constexpr int kPfN = 128;    // kv tokens per tile
constexpr int kPfH = 64;     // kv tokens per half-tile unit (columns of one S half)
constexpr int kPfD = 128;    // head dim
constexpr int kTileBytes = 128 * 128 * 2;  // one [128 x 128] 16-bit tile = two 16 KB swizzle blocks
constexpr int kPfSlots = 4;
constexpr int kPfStage = 2 * 16384;  // epilogue staging: one [128 x 64] 16-bit block per warpgroup
constexpr int kPfBars = 512;
constexpr int kPfSmem = kTileBytes * (2 + kPfSlots) + kPfStage + kPfBars + kTileList * 2 + 1024;
static_assert(kPfSmem <= 232448, "shared memory of one block");

struct PrefillParams {
  void* out;
  const void* k_pool;
  const void* v_pool;
  const int32_t* req_to_token;
  const int64_t* req_pool_indices;
  const int32_t* prefix_lens;
  const int32_t* extend_lens;
  const int32_t* extend_start_loc;
  int Hq, Hk;
  int64_t out_stride, rtt_stride;
  float scale_log2;
  int pair_heads;  // 1: the two tiles are two heads of one KV head; 0: two consecutive token tiles
  int tiles_x;     // item rows along the token axis
  int heads_x;     // item columns along the head axis
  int batch;
  int total_items;
  int sorted;      // 1: items are dealt from a list of the row tiles by weight (pf_sort)
  int use_tma;  // 0: always gather (SPD_ATTN_TMA=0)
  // n / d for the three launch-constant divisors of the item decode (per_x = heads_x * batch,
  // heads_x, GQA group) as multiply-high + shift: four dependent integer divisions sat on every
  // item boundary of every role
  uint32_t per_x_m, per_x_s, heads_x_m, heads_x_s, group_m, group_s, tiles_x_m, tiles_x_s;
  // kWin only: keys a query sees up to and with itself; a logit per head in the softmax denominator (nullptr: none); query
  // temperature 1 + coef ln(floor((pos + 1) / every) + 1) (every 0: none)
  int window, qtemp_every;
  const void* q;
  int64_t q_stride;
  const float* sinks;
  float qtemp_coef;
  long long* trace;  // debug timeline of CTA 0; kTrace builds only
  int trace_cap;
};

// timeline region r: (tag, clock64) pairs written by one thread of CTA 0
template <bool kTrace>
__device__ __forceinline__ void pf_trace(const PrefillParams& p, int region, uint32_t& n, long long tag) {
  if constexpr (kTrace) {
    if (blockIdx.x == 0 && (threadIdx.x & 31) == 0 && p.trace && static_cast<int>(n) < p.trace_cap) {
      long long* e = p.trace + (static_cast<size_t>(region) * p.trace_cap + n) * 2;
      e[0] = tag;
      e[1] = clock64();
      ++n;
    }
  }
}

struct PfItem {
  int req, pre, hk, n;         // n = end of the item's KV tiles (max over the two query tiles), j0 = the first of them
  int j0;
  int head[2], m0[2], rows[2], nt[2], q_row0[2];
  int kv_len;
};

// where an item lies, and the three per-request values it needs from global memory; loaded ONE ITEM AHEAD by every
// role (the dependent loads used to sit between two items: ~1000 clk per item boundary)
struct PfRaw {
  int req, qx, hx;
  int ext, pre, start;
};
__device__ __forceinline__ PfRaw pf_raw(const PrefillParams& p, const TileList& pl, int idx) {
  PfRaw r{0, 0, 0, 0, 0, 0};
  if (idx < pl.items) {
    if (pl.list != nullptr) {
      const int e = fastdiv(idx, p.heads_x_m, p.heads_x_s);
      r.hx = idx - e * p.heads_x;
      const int slot = pl.list[e];
      r.req = fastdiv(slot, p.tiles_x_m, p.tiles_x_s);
      r.qx = slot - r.req * p.tiles_x;
    } else {
      const int ix = fastdiv(idx, p.per_x_m, p.per_x_s);
      const int rest = idx - ix * (p.heads_x * p.batch);
      r.qx = p.tiles_x - 1 - ix;  // heaviest (latest) query tiles first
      r.req = fastdiv(rest, p.heads_x_m, p.heads_x_s);
      r.hx = rest - r.req * p.heads_x;
    }
    r.ext = __ldg(p.extend_lens + r.req);
    r.pre = __ldg(p.prefix_lens + r.req);
    r.start = __ldg(p.extend_start_loc + r.req);
  }
  return r;
}
// the same in every lane of a warp, and known to be
__device__ __forceinline__ PfRaw pf_raw_uniform(PfRaw r) {
  r.req = __shfl_sync(0xffffffffu, r.req, 0);
  r.qx = __shfl_sync(0xffffffffu, r.qx, 0);
  r.hx = __shfl_sync(0xffffffffu, r.hx, 0);
  r.ext = __shfl_sync(0xffffffffu, r.ext, 0);
  r.pre = __shfl_sync(0xffffffffu, r.pre, 0);
  r.start = __shfl_sync(0xffffffffu, r.start, 0);
  return r;
}

template <bool kWin>
__device__ __forceinline__ PfItem pf_item(const PrefillParams& p, const PfRaw& raw) {
  PfItem it;
  it.req = raw.req;
  if (p.pair_heads) {
    it.head[0] = 2 * raw.hx;
    it.head[1] = 2 * raw.hx + 1;
    it.m0[0] = it.m0[1] = raw.qx * kPfM;
  } else {
    it.head[0] = it.head[1] = raw.hx;
    it.m0[0] = 2 * raw.qx * kPfM;
    it.m0[1] = (2 * raw.qx + 1) * kPfM;
  }
  it.hk = fastdiv(it.head[0], p.group_m, p.group_s);
  const int ext = raw.ext;
  it.pre = raw.pre;
  const int start = raw.start;
  it.kv_len = 0;
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const int rows = min(kPfM, ext - it.m0[w]);
    it.rows[w] = rows > 0 ? rows : 0;
    const int kv = it.pre + it.m0[w] + it.rows[w];  // keys visible to the tile's last valid row
    it.nt[w] = rows > 0 ? (kv + kPfN - 1) / kPfN : 0;
    it.q_row0[w] = start + it.m0[w];
    if (rows > 0) it.kv_len = max(it.kv_len, kv);
  }
  it.n = max(it.nt[0], it.nt[1]);
  // first key that the first row sees (the later tile of an item, if any, sees no earlier one)
  it.j0 = 0;
  if constexpr (kWin) it.j0 = max(0, it.pre + it.m0[0] - p.window + 1) / kPfN;
  return it;
}

// The row tiles with any rows, by the K / V tiles they walk (see tile_list).  Request lengths differ, so the order by query
// tile alone leaves the CTAs with unequal shares: 8 requests of 512 - 1536 new tokens, four with a prefix of 1024, 102
// tiles on the busiest CTA against 79 on average; sorted 81 (176 -> 156 us; with the window, 50 and 37: 132 -> 112 us).
template <bool kWin>
__device__ __forceinline__ TileList pf_sort(const PrefillParams& p, uint32_t* keys, uint32_t* count, uint16_t* list) {
  if (!p.sorted) return TileList{p.total_items, nullptr};
  return tile_list<kPfThreads>(
      p.batch * p.tiles_x, p.heads_x, p.total_items,
      [&](int slot) {
        PfRaw raw{};
        raw.req = fastdiv(slot, p.tiles_x_m, p.tiles_x_s);
        raw.qx = slot - raw.req * p.tiles_x;
        raw.ext = __ldg(p.extend_lens + raw.req);
        raw.pre = __ldg(p.prefix_lens + raw.req);
        const PfItem it = pf_item<kWin>(p, raw);
        return it.n > 0 ? it.n - it.j0 : 0;
      },
      keys, count, list);
}

// byte offset of (row, 16-byte chunk) inside a [128 x 128] 16-bit tile stored as two
// [128 rows x 128 B] blocks with the 128-byte swizzle (chunk index XOR row%8)
__device__ __forceinline__ uint32_t tile_off(int row, int chunk16) {
  return (chunk16 >> 3) * 16384 + row * 128 + (((chunk16 & 7) ^ (row & 7)) << 4);
}

// Output of one query row by a warp, from the keys the row sees alone; before the division by the sum, columns
// c + 2 lane and c + 2 lane + 1.  (kWin, for rows whose output is not finite: the tiles hold keys that the row does not
// see, and their P of 0 times an infinite or NaN value is NaN.  Looking for them in the epilogue: 140.2 -> 142.7 us for
// 4 requests of 2048 new tokens, 16 / 4 heads, window 1024.)
template <typename T>
__device__ __noinline__ float2 pf_row_alone(const T* q, const T* k_pool, const T* v_pool, const int32_t* page,
                                            int64_t row_elems, int kv0, int kv1, int c, float scale, float m_off) {
  const int lane = threadIdx.x & 31;
  float2 acc = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int j0 = kv0; j0 < kv1; j0 += 32) {
    const int j = j0 + lane;
    int64_t at = 0;
    float prob = 0.f;
    if (j < kv1) {
      at = page[j] * row_elems;
      float dot = 0.f;
#pragma unroll 1
      for (int d = 0; d < kPfD; d += 8) {
        const Vec16<T> a = ldv(q + d), b = ldv(k_pool + at + d);
#pragma unroll
        for (int e = 0; e < 8; ++e) dot = fmaf(to_f32<T>(a.e()[e]), to_f32<T>(b.e()[e]), dot);
      }
      prob = to_f32<T>(from_f32<T>(fast_exp2(fmaf(dot, scale, -m_off))));
    }
    const int n = min(32, kv1 - j0);
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const float pi = __shfl_sync(0xffffffffu, prob, i);
      const T* v = v_pool + __shfl_sync(0xffffffffu, at, i) + c + 2 * lane;
      acc.x = fmaf(pi, to_f32<T>(v[0]), acc.x);
      acc.y = fmaf(pi, to_f32<T>(v[1]), acc.y);
    }
    if (__all_sync(0xffffffffu, isnan(acc.x) && isnan(acc.y))) break;  // nothing changes that any more
  }
  return acc;
}

// kWin: a sliding window (KV tiles before the item's first visible key are skipped), sinks and a query temperature — the
// general attention of the hybrid families at head size 128 (see spd::attn_prefill_window_try).
// 4 requests of 2048 new tokens, 16 / 4 heads, window 1024: 320 us on warp-level MMAs with 64 x 64 tiles, 101 us here,
// warm (60 GFLOP visible; a query tile of 128 meets nine key tiles, two of them masked).
template <typename T, bool kTrace, bool kWin>
__global__ void __launch_bounds__(kPfThreads, 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                    const PrefillParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;                     // 2 tiles (warpgroup 0 / 1)
  uint8_t* sKV = smem + 2 * kTileBytes;   // ring: position 2t = K of tile t, 2t+1 = V of tile t
  uint8_t* sO = smem + (2 + kPfSlots) * kTileBytes;  // epilogue staging, 16 KB per warpgroup
  uint64_t* bars = reinterpret_cast<uint64_t*>(sO + kPfStage);
  uint64_t* q_full = bars;                     // 2
  uint64_t* kv_full = bars + 2;                // kPfSlots
  uint64_t* kv_empty = kv_full + kPfSlots;     // kPfSlots
  uint64_t* s_full = kv_empty + kPfSlots;      // 4: [warpgroup][half]
  uint64_t* p_full = s_full + 4;               // 4: [warpgroup][half]
  uint64_t* pv_done = p_full + 4;              // 4: [warpgroup][half] (see the parity note in the softmax)
  uint64_t* o_free = pv_done + 4;              // 2
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_free + 2);
  uint32_t* n_tiles = tmem_slot + 1;
  volatile uint32_t* turn = tmem_slot + 2;  // items whose first S warpgroup 0's issuer has handed in
  uint16_t* list = reinterpret_cast<uint16_t*>(sO + kPfStage + kPfBars);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const int cta = blockIdx.x, ncta = gridDim.x;
  constexpr int kU = kPfH;        // columns of one softmax / MMA unit
  constexpr int kNU = kPfN / kU;  // units per K/V tile

  if (warp == 10) {
    if (lane == 0) {
      for (int i = 0; i < 2; ++i) mbar_init(&q_full[i], 1);
      for (int i = 0; i < kPfSlots; ++i) {
        mbar_init(&kv_full[i], 32);
        mbar_init(&kv_empty[i], 2);
      }
      for (int i = 0; i < 4; ++i) {
        mbar_init(&s_full[i], 1);
        mbar_init(&p_full[i], 4);
        mbar_init(&pv_done[i], 1);
      }
      for (int i = 0; i < 2; ++i) mbar_init(&o_free[i], 4);
      *n_tiles = 0;
      *turn = 0;
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (warp == 11 && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmO);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base;        // 2 x (64 + 64) columns (warpgroup 0 / 1, half a / b); P_h aliases
                                            // the first 32 columns of S_h
  const uint32_t tmem_O = tmem_base + 256;  // 2 x 128 columns

  griddep_wait();
  const TileList pl = pf_sort<kWin>(p, reinterpret_cast<uint32_t*>(sO), n_tiles, list);

  if (warp >= 10) {
    // ===================== MMA issuer of warpgroup 0 (warp 10) / 1 (warp 11) =====================
    // The whole warp walks the items and one lane issues: descriptors then stay in uniform registers.  Short loops, not
    // unrolled ones.
    const bool leader = elect_one();
    const int w = warp - 10;
    constexpr uint32_t idesc_qk = umma_idesc<T>(kPfM, kU, 0, 0);    // A, B K-major; N = one unit
    constexpr uint32_t idesc_pv = umma_idesc<T>(kPfM, kPfD, 0, 1);  // A = P (TMEM), B = V MN-major
    const uint64_t qd = umma_desc_sw128(smem_u32(sQ + w * kTileBytes), 16, 1024);
    const uint64_t kd0 = umma_desc_sw128(smem_u32(sKV), 16, 1024);
    const uint64_t vd0 = umma_desc_sw128(smem_u32(sKV), 16384, 1024);
    const uint32_t qk_hi = static_cast<uint32_t>(qd >> 32), v_hi = static_cast<uint32_t>(vd0 >> 32);
    uint32_t t_base = 0;  // tiles of all previous items (ring position / 2)
    uint32_t pq = 0;      // PV units issued (all items); unit of the tile = pq % kNU
    uint32_t eq = 0;      // items of the warpgroup (o_free phase)
    uint32_t items = 0;   // items begun
    uint32_t tn = 0;
    bool q_ahead = false;  // the next item's Q is already under way
    auto load_q = [&](const PfItem& it) {
      const int head = w == 0 ? it.head[0] : it.head[1], row0 = w == 0 ? it.q_row0[0] : it.q_row0[1];
      if (leader) {
        mbar_expect_tx(&q_full[w], kTileBytes);
        tma_load_2d(sQ + w * kTileBytes, &tmQ, &q_full[w], head * kPfD, row0, kEvictFirst);
        tma_load_2d(sQ + w * kTileBytes + 16384, &tmQ, &q_full[w], head * kPfD + 64, row0, kEvictFirst);
      }
      __syncwarp();
    };
    int idx = pf_rank(0, cta, ncta);
    PfRaw raw = pf_raw(p, pl, idx);
    for (int kk = 0; idx < pl.items; ++kk) {
      const PfItem it = pf_item<kWin>(p, pf_raw_uniform(raw));
      idx = pf_rank(kk + 1, cta, ncta);
      raw = pf_raw(p, pl, idx);
      if (it.n == 0) continue;
      const int nt = w == 0 ? it.nt[0] : it.nt[1];
      if (nt > 0) {
        if (!q_ahead) load_q(it);
        q_ahead = false;
        mbar_wait(&q_full[w], eq & 1);
      }
      // S(j, h): the warpgroup's previous P in these columns has been consumed by PV(j-1, h),
      // issued earlier by this thread — tcgen05.mma executes in issue order.
      auto issue_s = [&](int j, int h) {
        const uint32_t pos = 2 * (t_base + j - it.j0);
        mbar_wait(&kv_full[pos % kPfSlots], (pos / kPfSlots) & 1);
        if (h == 0) fence_proxy_async_smem();
        tc_fence_after_sync();
        uint32_t qa = static_cast<uint32_t>(qd);
        uint32_t ka = static_cast<uint32_t>(kd0) + (pos % kPfSlots) * (kTileBytes / 16) + h * (kU * 128 / 16);
        const uint32_t td = tmem_S + w * kPfN + h * kU;
#pragma unroll 1
        for (int k = 0; k < kPfD / 16; ++k) {
          umma_ss_if(leader, td, qa, ka, qk_hi, idesc_qk, k);
          const uint32_t step = k == 3 ? (16384 - 96) / 16 : 2;
          qa += step;
          ka += step;
        }
        umma_commit_if(leader, &s_full[w * 2 + h]);
      };
      // K_j (V_j) is released by both issuers, also by one whose warpgroup does not use the tile: it waits for the tile
      // first, so that its arrivals keep to the ring's phases
      auto release_k = [&](int j) {
        const uint32_t pos = 2 * (t_base + j - it.j0);
        if (j >= nt) mbar_wait(&kv_full[pos % kPfSlots], (pos / kPfSlots) & 1);
        umma_commit_if(leader, &kv_empty[pos % kPfSlots]);
      };
      // the epilogue of the previous item reads O, not S — and its last PVs (reading P in the S
      // columns) were issued before these, so S(0, .) may go out immediately
      // Warpgroup 1 starts an item behind the first S of warpgroup 0: in one phase the two meet at the exponentials and at
      // the output (5.7 us instead of 5.0 per item of one tile).  (The count only grows and warpgroup 0's issuer waits for
      // nothing that comes later here; a start that is not seen costs the phase, no result.)
      ++items;
      if (w == 1 && nt > 0) {
        for (int i = 0; i < 1024 && *turn < items; ++i) {}
        __syncwarp();
      }
      if (it.j0 < nt) {
#pragma unroll
        for (int h = 0; h < kNU; ++h) issue_s(it.j0, h);
        if (w == 0 && leader) *turn = items;
      }
      release_k(it.j0);
      for (int j = it.j0; j < it.n; ++j) {
        const uint32_t vpos = 2 * (t_base + j - it.j0) + 1;
        if (j < nt) {
#pragma unroll
          for (int h = 0; h < kNU; ++h) {
            if (j == nt - 1 && h == 0 && idx < pl.items) {
              // The item's last S is under way, and nothing goes out before P arrives: once it is complete, Q's memory
              // is free for the next item
              const PfItem next = pf_item<kWin>(p, pf_raw_uniform(raw));
              q_ahead = (w == 0 ? next.nt[0] : next.nt[1]) > 0;
              if (q_ahead) {
                mbar_wait(&s_full[w * 2 + kNU - 1], (pq / kNU) & 1);
                load_q(next);
              }
            }
            pf_trace<kTrace>(p, 2 + w, tn, 0x100 + w * 2 + h);  // waiting for P
            mbar_wait(&p_full[w * 2 + h], (pq / kNU) & 1);
            pf_trace<kTrace>(p, 2 + w, tn, 0x200 + w * 2 + h);  // P ready
            mbar_wait(&kv_full[vpos % kPfSlots], (vpos / kPfSlots) & 1);
            if (h == 0) fence_proxy_async_smem();
            if (j == it.j0 && h == 0) mbar_wait(&o_free[w], (eq & 1) ^ 1);  // previous item's O has been read
            tc_fence_after_sync();
            uint32_t va = static_cast<uint32_t>(vd0) + (vpos % kPfSlots) * (kTileBytes / 16) + h * (kU * 128 / 16);
            uint32_t pa = tmem_S + w * kPfN + h * kU;
            uint32_t acc = (j > it.j0 || h > 0) ? 1u : 0u;
#pragma unroll 1
            for (int k = 0; k < kU / 16; ++k) {
              // A = P[128 x 16 kv]: 8 TMEM columns per k-step; B = V[16 kv x 128 d] (MN-major: 2
              // blocks of 64 d, LBO = 16 KB; kv rows 128 B apart, 8-row groups SBO = 1 KB)
              umma_ts_if(leader, tmem_O + w * kPfD, pa, va, v_hi, idesc_pv, acc);
              pa += 8;
              va += 2048 / 16;
              acc = 1;
            }
            umma_commit_if(leader, &pv_done[w * 2 + h]);
            ++pq;
            if (j + 1 < nt) issue_s(j + 1, h);
            pf_trace<kTrace>(p, 2 + w, tn, 0x300 + w * 2 + h);  // PV (+ next S) issued
          }
        } else {
          mbar_wait(&kv_full[vpos % kPfSlots], (vpos / kPfSlots) & 1);
        }
        umma_commit_if(leader, &kv_empty[vpos % kPfSlots]);  // V_j: all PVs issued
        if (j + 1 < it.n) release_k(j + 1);
      }
      if (nt > 0) ++eq;
      t_base += it.n - it.j0;
    }
  } else if (warp >= 8) {
    // ===================== K loader (warp 8) / V loader (warp 9) =====================
    const int is_v = warp == 9 ? 1 : 0;
    const int chunk = lane & 15;   // 16-byte chunk of the 256-byte head row
    const int rsub = lane >> 4;    // 0..1
    const T* pool = reinterpret_cast<const T*>(is_v ? p.v_pool : p.k_pool);
    const int64_t row_elems = static_cast<int64_t>(p.Hk) * kPfD;
    uint32_t t = 0;        // tiles loaded so far (all items)
    int idx = pf_rank(0, cta, ncta);
    PfRaw raw = pf_raw(p, pl, idx);
    for (int k = 0; idx < pl.items; ++k) {
      const PfItem it = pf_item<kWin>(p, raw);
      idx = pf_rank(k + 1, cta, ncta);
      raw = pf_raw(p, pl, idx);
      if (it.n == 0) continue;
      const int32_t* rtt = p.req_to_token + p.req_pool_indices[it.req] * p.rtt_stride;
      const int64_t col = static_cast<int64_t>(it.hk) * kPfD + chunk * 8;
      for (int j = it.j0; j < it.n; ++j, ++t) {
        // page-table lookups first, all in flight together (the cp.async asm is a compiler
        // barrier; interleaving the lookups with it would serialise the dependent load latencies)
        int slot[64];
#pragma unroll
        for (int i = 0; i < 64; ++i) {
          const int kv = j * kPfN + i * 2 + rsub;
          slot[i] = kv < it.kv_len ? __ldg(rtt + kv) : -1;
        }
        // consecutive slots?  (full tile whose 128 entries are base, base+1, ...; warp vote)
        const int base = (p.use_tma && (j + 1) * kPfN <= it.kv_len) ? __ldg(rtt + j * kPfN) : -1;
        bool contig = base > 0;
#pragma unroll
        for (int i = 0; i < 64; ++i) contig &= (slot[i] == base + i * 2 + rsub);
        contig = __all_sync(0xffffffffu, contig);
        const uint32_t pos = 2 * t + is_v;
        const int st = pos % kPfSlots;
        const uint32_t epar = ((pos / kPfSlots) & 1) ^ 1;
        mbar_wait(&kv_empty[st], epar);
        if (contig) {
          // TMA: rows base .. base+127 of the pool, the 128 columns of kv head hk, as the slot's
          // two 16 KB swizzle blocks; the 32 KB are counted on the slot's barrier next to the
          // warp's 32 arrivals
          if (lane == 0) {
            uint8_t* dst = sKV + st * kTileBytes;
            fence_proxy_async_smem();  // the slot may last have been written by the gather path
            mbar_expect_tx_noarrive(&kv_full[st], kTileBytes);
            tma_load_2d(dst, is_v ? &tmV : &tmK, &kv_full[st], it.hk * kPfD, base, kEvictNormal);
            tma_load_2d(dst + 16384, is_v ? &tmV : &tmK, &kv_full[st], it.hk * kPfD + 64, base, kEvictNormal);
          }
          __syncwarp();
          mbar_arrive(&kv_full[st]);
          continue;
        }
        const uint32_t dst = smem_u32(sKV + st * kTileBytes);
#pragma unroll
        for (int i = 0; i < 64; ++i) {
          const int row = i * 2 + rsub;
          const bool valid = slot[i] >= 0;
          const int64_t s64 = valid ? slot[i] : 0;
          cp_async16(dst + tile_off(row, chunk), pool + s64 * row_elems + col, valid);
        }
        // each lane's arrival comes when its copies have landed: nothing here waits for them, and the next tile's lookups
        // and copies follow at once.  (The MMA issuers, who read what these wrote, fence between the two proxies.)  Handed
        // over by the loader, a tile waited for the next one's page-table lookups: 40 portions of 16 tokens 25.3 -> 23.7 us,
        // 16 of 500 61.4 -> 60.4, 8 of 250 18.1 -> 17.4.
        cp_async_mbar_arrive_noinc(&kv_full[st]);
      }
    }
  } else {
    // ===================== softmax warpgroups (one thread per query row) =====================
    const int w = warp >> 2;            // warpgroup == query tile of the item
    const int row = threadIdx.x & 127;  // == TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t ts = tmem_S + lane_base + w * kPfN;
    const uint32_t to = tmem_O + lane_base + w * kPfD;
    uint32_t u = 0;  // units processed by this warpgroup (all items); unit of the tile = u % kNU
    uint32_t tn = 0;
    const bool tracer = kTrace && (threadIdx.x & 127) == 0;
    // ---- epilogue: O / l, TMEM -> registers -> global ----
    // (Tried: DEFERRING it until the next item's first unit has been exponentiated, so
    // that the ~1500-1900 clk drain of the item's last PV is spent on useful work.  The drain wait
    // did shrink to ~700 clk, but o_free — and with it the next item's first PV — moved later by
    // a whole softmax pass, and the kernel got 5 % slower at 8 x 1024; not kept.)
    float e_l = 0.f;  // state of the item being written out
    int e_rows = 0, e_head = 0, e_q_row0 = 0;
    uint32_t e_u = 0;
    int e_req = 0, e_hk = 0, e_limit = 0;  // kWin
    float e_scale = 0.f, e_m_off = 0.f;
    // kWin: the warp's rows whose columns c .. c + 63 have a value that is not finite (z is NaN), again; into the staging
    // block or (nullptr) to global memory
    auto rows_alone = [&](float z, int c, float inv_l, uint8_t* stage) {
      uint32_t todo = __ballot_sync(0xffffffffu, isnan(z));
      if (todo == 0) return;
      __syncwarp();
      const int64_t col = static_cast<int64_t>(e_hk) * kPfD;
#pragma unroll 1
      for (; todo != 0; todo &= todo - 1) {
        const int src = __ffs(todo) - 1, r = (row & ~31) + src;
        const int lim = __shfl_sync(0xffffffffu, e_limit, src);
        const float2 f = pf_row_alone<T>(
            reinterpret_cast<const T*>(p.q) + static_cast<int64_t>(e_q_row0 + r) * p.q_stride +
                static_cast<int64_t>(e_head) * kPfD,
            reinterpret_cast<const T*>(p.k_pool) + col, reinterpret_cast<const T*>(p.v_pool) + col,
            p.req_to_token + p.req_pool_indices[e_req] * p.rtt_stride, static_cast<int64_t>(p.Hk) * kPfD,
            max(0, lim - p.window + 1), lim + 1, c, __shfl_sync(0xffffffffu, e_scale, src),
            __shfl_sync(0xffffffffu, e_m_off, src));
        const float inv = __shfl_sync(0xffffffffu, inv_l, src);
        const uint32_t pair = pack2<T>(f.x * inv, f.y * inv);
        if (stage != nullptr)
          *reinterpret_cast<uint32_t*>(stage + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4) = pair;
        else
          *reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(p.out) + static_cast<int64_t>(e_q_row0 + r) * p.out_stride +
                                       static_cast<int64_t>(e_head) * kPfD + c + 2 * lane) = pair;
      }
    };
    auto epilogue = [&]() {
      // last unit = half b of the last tile; S of that unit complete => PV(b) of the tile before is
      // complete, so only this one phase of pv_done[w][b] can be outstanding; PV(b) complete => PV(a)
      mbar_wait(&pv_done[w * 2 + (kNU - 1)], ((e_u - 1) / kNU) & 1);
      tc_fence_after_sync();
      if (tracer) pf_trace<kTrace>(p, w, tn, 0x500);  // last PV complete
      const float inv_l = e_l > 0.f ? 1.f / e_l : 0.f;
      // A full tile leaves through shared memory and one TMA store per 64-column block: with one
      // thread per row, direct 16-byte stores touch 32 different lines per warp instruction and
      // the 128 rows x 256 B took ~5900 clk per item (in-kernel timeline) — a quarter of
      // the kernel at 1024-token prompts.  A ragged last tile (fewer than 128 rows) must not write
      // the rows of the next request and keeps the direct path.
      const bool full_tile = e_rows == kPfM;
      uint8_t* stage = sO + w * (kPfStage / 2);
      T* dst = reinterpret_cast<T*>(p.out) + static_cast<int64_t>(e_q_row0 + row) * p.out_stride +
               static_cast<int64_t>(e_head) * kPfD;
#pragma unroll 1
      for (int c = 0; c < kPfD; c += 64) {
        uint32_t a[32], b[32];
        tmem_ld_32x32b_x32(to + c, a);
        tmem_ld_32x32b_x32(to + c + 32, b);
        tmem_ld_wait();
        if (c == 64) {
          // every O column of this warp is in registers: the next item's first PV may overwrite it
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&o_free[w]);
        }
        float z0 = 0.f, z1 = 0.f;  // kWin: NaN when a value of these columns is infinite or NaN
        if constexpr (kWin) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            z0 = fmaf(__uint_as_float(a[i]), 0.f, z0);
            z1 = fmaf(__uint_as_float(b[i]), 0.f, z1);
          }
        }
        uint4 v[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[i].x = pack2<T>(__uint_as_float(a[8 * i]) * inv_l, __uint_as_float(a[8 * i + 1]) * inv_l);
          v[i].y = pack2<T>(__uint_as_float(a[8 * i + 2]) * inv_l, __uint_as_float(a[8 * i + 3]) * inv_l);
          v[i].z = pack2<T>(__uint_as_float(a[8 * i + 4]) * inv_l, __uint_as_float(a[8 * i + 5]) * inv_l);
          v[i].w = pack2<T>(__uint_as_float(a[8 * i + 6]) * inv_l, __uint_as_float(a[8 * i + 7]) * inv_l);
          v[4 + i].x = pack2<T>(__uint_as_float(b[8 * i]) * inv_l, __uint_as_float(b[8 * i + 1]) * inv_l);
          v[4 + i].y = pack2<T>(__uint_as_float(b[8 * i + 2]) * inv_l, __uint_as_float(b[8 * i + 3]) * inv_l);
          v[4 + i].z = pack2<T>(__uint_as_float(b[8 * i + 4]) * inv_l, __uint_as_float(b[8 * i + 5]) * inv_l);
          v[4 + i].w = pack2<T>(__uint_as_float(b[8 * i + 6]) * inv_l, __uint_as_float(b[8 * i + 7]) * inv_l);
        }
        if (full_tile) {
          // the block's previous TMA store has finished READING the staging memory
          if (row == 0) bulk_wait_group_read0();
          asm volatile("bar.sync %0, 128;" ::"r"(2 + w) : "memory");
#pragma unroll
          for (int i = 0; i < 8; ++i)  // [128 rows x 128 B], 128-byte swizzle: chunk ^ (row % 8)
            *reinterpret_cast<uint4*>(stage + row * 128 + ((i ^ (row & 7)) << 4)) = v[i];
          if constexpr (kWin) rows_alone(z0 + z1, c, inv_l, stage);
          fence_proxy_async_smem();
          asm volatile("bar.sync %0, 128;" ::"r"(2 + w) : "memory");
          if (row == 0) {
            tma_store_2d(&tmO, stage, e_head * kPfD + c, e_q_row0);
            bulk_commit_group();
          }
        } else {
          if (row < e_rows) {
#pragma unroll
            for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(dst + c + 8 * i) = v[i];
          }
          if constexpr (kWin) rows_alone(row < e_rows ? z0 + z1 : 0.f, c, inv_l, nullptr);
        }
      }
      if (tracer) pf_trace<kTrace>(p, w, tn, 0x600);  // O stored
    };
    const auto rescale_o = [&](float alpha, uint32_t unit) {
      // O must be quiescent: S of this unit was issued after PV of unit u-kNU (so units
      // <= u-kNU are complete), but PV of the units in between (the other half) may still
      // be running.  pv_done is per unit-of-tile so that this wait cannot alias: on that
      // barrier at most the one phase we wait for is outstanding (a parity wait only tells
      // the current phase from the one before it).
      mbar_wait(&pv_done[w * 2 + ((unit - 1) % kNU)], ((unit - 1) / kNU) & 1);
      tc_fence_after_sync();
      rescale_row128(to, alpha);
    };
    int idx = pf_rank(0, cta, ncta);
    PfRaw raw = pf_raw(p, pl, idx);
    for (int k = 0; idx < pl.items; ++k) {
      const PfItem it = pf_item<kWin>(p, raw);
      idx = pf_rank(k + 1, cta, ncta);
      raw = pf_raw(p, pl, idx);
      const int nt = w == 0 ? it.nt[0] : it.nt[1];
      if (nt == 0) continue;
      const int m0 = w == 0 ? it.m0[0] : it.m0[1];
      const int rows_valid = w == 0 ? it.rows[0] : it.rows[1];
      const int head = w == 0 ? it.head[0] : it.head[1];
      const int q_row0 = w == 0 ? it.q_row0[0] : it.q_row0[1];
      const int limit = it.pre + m0 + row;  // last visible key of this row (causal)
      float scale = p.scale_log2;
      int span = 0;
      if constexpr (kWin) {
        span = p.window - 1;
        if (p.qtemp_every > 0)
          scale *= 1.f + p.qtemp_coef * logf(static_cast<float>((limit + 1) / p.qtemp_every + 1));
      }
      float m_used = -INFINITY;  // max currently folded into O and l (raw score units)
      float l = 0.f;
      for (int jh = 0; jh < kNU * (nt - it.j0); ++jh, ++u) {
        const int h = jh % kNU;
        const int kv0 = (it.j0 + jh / kNU) * kPfN + h * kU;
        // a row that does not see the whole unit: the first one past its end, or the last one with its window past its start
        const bool need_mask = (kv0 + kU - 1) > (it.pre + m0) || (kWin && kv0 < it.pre + m0 + kPfM - p.window);
        const uint32_t tsh = ts + h * kU;
        if (tracer) pf_trace<kTrace>(p, w, tn, 0x100 + h);  // waiting for S
        mbar_wait(&s_full[w * 2 + h], (u / kNU) & 1);
        tc_fence_after_sync();
        if (tracer) pf_trace<kTrace>(p, w, tn, 0x200 + h);  // S ready
        uint32_t pk[kU / 2];
        bool raise = false;  // kWin: the reference max has been raised, O is rescaled below
        float alpha = 1.f;
        if constexpr (kWin) {
          // The true running max: the largest P of a row is then exactly 1, as in the warp-level kernel that serves the
          // other calls.  (A reference that lags, as below, rounds that P too: 9 - 15 % more rms error against 64-bit results.)
          // One read of the unit for the max and the P, and O rescaled after the exponentials: 112 -> 101 us for 4
          // requests of 2048 new tokens, 16 / 4 heads, window 1024; the sum of the rounded P: 0.6 % less rms error.
          uint32_t ra[32], rb[32];
          const float mx = need_mask ? softmax_load_max<true, kWin>(tsh, ra, rb, kv0, limit, span)
                                     : softmax_load_max<false, kWin>(tsh, ra, rb, kv0, limit, span);
          raise = __any_sync(0xffffffffu, mx > m_used);
          if (raise) {
            const float m_new = fmaxf(m_used, mx);
            alpha = (m_used == -INFINITY) ? 0.f : fast_exp2((m_used - m_new) * scale);
            l *= alpha;
            m_used = m_new;
            raise = jh > 0;
          }
          l += softmax_unit<T>(ra, rb, pk, scale, (m_used == -INFINITY) ? 0.f : m_used * scale);
        } else {
          if (jh == 0)  // first unit of the item: establish the reference max with a max-only pre-pass
            m_used = need_mask ? softmax_row_max<true>(tsh, kv0, limit)
                               : softmax_row_max<false>(tsh, kv0, limit);
          float m_off = (m_used == -INFINITY) ? 0.f : m_used * scale;
          float psum = need_mask ? softmax_row_pass<T, true>(tsh, pk, scale, m_off, kv0, limit)
                                 : softmax_row_pass<T, false>(tsh, pk, scale, m_off, kv0, limit);
          // raise the reference max only when some row may have outgrown it by > 2^8 (an element
          // above 2^8 implies a row sum above 2^8; warp-uniform decision: tcgen05.ld/st are
          // warp-collective); S is still intact (P is stored below), so the unit is simply redone
          if (__any_sync(0xffffffffu, psum > kRescaleTrigger)) {
            const float mx = need_mask ? softmax_row_max<true>(tsh, kv0, limit)
                                       : softmax_row_max<false>(tsh, kv0, limit);
            const float m_new = fmaxf(m_used, mx);
            alpha = (m_used == -INFINITY) ? 0.f : fast_exp2((m_used - m_new) * scale);
            l *= alpha;
            m_used = m_new;
            m_off = (m_used == -INFINITY) ? 0.f : m_used * scale;
            if (jh > 0) rescale_o(alpha, u);
            psum = need_mask ? softmax_row_pass<T, true>(tsh, pk, scale, m_off, kv0, limit)
                             : softmax_row_pass<T, false>(tsh, pk, scale, m_off, kv0, limit);
          }
          l += psum;
        }
        // P over the first kU/2 columns of this S unit (every column of it is in registers by now)
        tmem_st_32x32b_x32(tsh, pk);
        if (kWin && raise) rescale_o(alpha, u);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[w * 2 + h]);
        if (tracer) pf_trace<kTrace>(p, w, tn, 0x300 + h);  // P published
      }
      if (tracer) pf_trace<kTrace>(p, w, tn, 0x400);  // item done
      if constexpr (kWin) {
        if (p.sinks != nullptr) l += fast_exp2(p.sinks[head] * 1.4426950408889634f - m_used * scale);
      }
      e_l = l;
      e_rows = rows_valid;
      e_head = head;
      e_q_row0 = q_row0;
      e_u = u;
      if constexpr (kWin) {
        e_req = it.req;
        e_hk = it.hk;
        e_limit = limit;
        e_scale = scale;
        e_m_off = m_used == -INFINITY ? 0.f : m_used * scale;
      }
      epilogue();
    }
  }

  if (warp < 8 && (threadIdx.x & 127) == 0) bulk_wait_group0();  // this thread's TMA stores have landed
  griddep_launch_dependents();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 10) tmem_dealloc(tmem_base, 512);
}

static int pf_setup(PrefillParams& p, CUtensorMap& tq, CUtensorMap& tk, CUtensorMap& tv, CUtensorMap& to, void* out,
                    const void* q, const void* k_pool, const void* v_pool, const int32_t* req_to_token,
                    const int64_t* req_pool_indices, const int32_t* prefix_lens, const int32_t* extend_lens,
                    const int32_t* extend_start_loc, int64_t batch, int64_t total_tokens, int64_t max_extend_len,
                    int num_q_heads, int num_kv_heads, int64_t q_stride, int64_t out_stride, int64_t req_to_token_stride,
                    float sm_scale) {
  p.out = out;
  p.k_pool = k_pool;
  p.v_pool = v_pool;
  p.req_to_token = req_to_token;
  p.req_pool_indices = req_pool_indices;
  p.prefix_lens = prefix_lens;
  p.extend_lens = extend_lens;
  p.extend_start_loc = extend_start_loc;
  p.Hq = num_q_heads;
  p.Hk = num_kv_heads;
  p.out_stride = out_stride;
  p.rtt_stride = req_to_token_stride;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
  const int q_tiles = static_cast<int>((max_extend_len + kPfM - 1) / kPfM);
  p.pair_heads = ((num_q_heads / num_kv_heads) % 2 == 0) ? 1 : 0;
  p.tiles_x = p.pair_heads ? q_tiles : (q_tiles + 1) / 2;
  p.heads_x = p.pair_heads ? num_q_heads / 2 : num_q_heads;
  p.batch = static_cast<int>(batch);
  const int64_t total = static_cast<int64_t>(p.tiles_x) * p.heads_x * batch;
  SPD_REQUIRE(total < (1ll << 30), SPD_E_SHAPE, "prefill attention: too many work items");
  p.total_items = static_cast<int>(total);
  fastdiv_magic(static_cast<uint32_t>(p.heads_x) * static_cast<uint32_t>(p.batch), p.per_x_m, p.per_x_s);
  fastdiv_magic(static_cast<uint32_t>(p.tiles_x), p.tiles_x_m, p.tiles_x_s);
  fastdiv_magic(static_cast<uint32_t>(p.heads_x), p.heads_x_m, p.heads_x_s);
  fastdiv_magic(static_cast<uint32_t>(num_q_heads / num_kv_heads), p.group_m, p.group_s);
  if (int rc = get_tmap(&tq, q, static_cast<uint64_t>(total_tokens),
                     static_cast<uint64_t>(num_q_heads) * kPfD, static_cast<uint64_t>(q_stride), kPfM))
    return rc;
  // the output as a TMA-store target: same geometry as Q (rows beyond total_tokens are clipped)
  if (int rc = get_tmap(&to, out, static_cast<uint64_t>(total_tokens),
                     static_cast<uint64_t>(num_q_heads) * kPfD, static_cast<uint64_t>(out_stride), kPfM))
    return rc;
  // K/V pools as [slots, Hk*D] tensors, box 128 rows x 64 columns (the row extent only bounds the
  // coordinates; they are slot ids taken from req_to_token)
  static const bool tma_on = []() { const char* e = getenv("SPD_ATTN_TMA"); return !(e && e[0] == '0'); }();
  p.use_tma = tma_on ? 1 : 0;
  const uint64_t row_elems = static_cast<uint64_t>(num_kv_heads) * kPfD;
  if (int rc = get_tmap(&tk, k_pool, 1ull << 31, row_elems, row_elems, kPfN)) return rc;
  if (int rc = get_tmap(&tv, v_pool, 1ull << 31, row_elems, row_elems, kPfN)) return rc;
  return 0;
}

// A list of the row tiles by weight serves where some CTA gets more than one item; it holds kTileList tiles, named by 16 bits
// (kv lengths below 2^23, so that a weight fits the key's other half).
static int pf_wants_list(const PrefillParams& p, int64_t total_tokens, int grid) {
  const int64_t rows = p.pair_heads ? kPfM : 2 * kPfM;
  return p.total_items > grid && total_tokens / rows + p.batch <= kTileList &&
                 static_cast<int64_t>(p.batch) * p.tiles_x <= 65536 && p.rtt_stride < (1 << 23)
             ? 1
             : 0;
}

// Ragged extend of the general attention at head size 128 with a window, sinks and a query temperature (no distance bias,
// score cap, pooled blocks or kept first tokens).  → 0 launched, 1 not applicable, else an error.
int attn_prefill_window_try(void* out, const void* q, const void* k_pool, const void* v_pool, const int32_t* req_to_token,
                            const int64_t* req_pool_indices, const int32_t* prefix_lens, const int32_t* extend_lens,
                            const int32_t* extend_start_loc, int64_t batch, int64_t total_tokens, int64_t max_extend_len,
                            int H, int G, int64_t q_stride, int64_t out_stride, int64_t r2t_stride, float sm_scale,
                            int window, const float* sinks, float qtemp_coef, int qtemp_every, int dtype, int sm_budget,
                            cudaStream_t stream) {
  // a max of raw scores serves the scaled ones only where the scale is positive
  if (!(sm_scale > 0.f) || !(qtemp_every <= 0 || qtemp_coef >= 0.f)) return 1;
  if (q_stride % 8 != 0 || out_stride % 8 != 0 || !aligned16(out) || !aligned16(q) || !aligned16(k_pool) || !aligned16(v_pool))
    return 1;
  const int64_t items = (max_extend_len + kPfM - 1) / kPfM * H * batch;
  if (total_tokens <= 0 || items >= (1ll << 30) || total_tokens >= (1ll << 31)) return 1;
  PrefillParams p{};
  CUtensorMap tq, tk, tv, to;
  if (int rc = pf_setup(p, tq, tk, tv, to, out, q, k_pool, v_pool, req_to_token, req_pool_indices, prefix_lens, extend_lens,
                        extend_start_loc, batch, total_tokens, max_extend_len, H, G, q_stride, out_stride, r2t_stride,
                        sm_scale))
    return rc;
  p.q = q;
  p.q_stride = q_stride;
  p.window = window > 0 && window < (1 << 30) ? window : 1 << 30;
  p.sinks = sinks;
  p.qtemp_coef = qtemp_coef;
  p.qtemp_every = qtemp_every > 0 ? qtemp_every : 0;
  const int sms = sm_budget > 0 ? sm_budget : device_sm_count_cached();  // items are dealt to the CTAs that run at once
  const int grid = p.total_items < sms ? p.total_items : sms;
  p.sorted = pf_wants_list(p, total_tokens, grid);
  SPD_DISPATCH_DTYPE(dtype, {
    auto kern = attn_prefill_kernel<T, false, true>;
    static bool configured = false;
    if (!configured) {
      SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPfSmem));
      configured = true;
    }
    SPD_CUDA(launch(kern, dim3(grid), dim3(kPfThreads), kPfSmem, stream, pdl_enabled(), tq, tk, tv, to, p));
  });
  return 0;
}

int check_attn_args(const char* fn, const void* out, const void* q, const void* k_pool,
                    const void* v_pool, const void* rtt, const void* rpi, int Hq, int Hk, int D,
                    int64_t q_stride, int64_t out_stride);

}  // namespace spd

using namespace spd;

// debug only (not part of include/spd.h): subsequent launches run the traced build and CTA 0 writes
// its timeline — 4 regions (softmax warpgroup 0, 1, MMA issuer 0, 1) of `cap` (tag, clock) pairs
static long long* g_pf_trace = nullptr;
static int g_pf_trace_cap = 0;
extern "C" int spd_debug_attn_prefill_trace(void* buf, int64_t cap) {
  g_pf_trace = static_cast<long long*>(buf);
  g_pf_trace_cap = static_cast<int>(cap);
  return 0;
}

extern "C" int spd_attn_prefill_ragged(void* out, const void* q, const void* k_pool,
                                       const void* v_pool, const int32_t* req_to_token,
                                       const int64_t* req_pool_indices, const int32_t* prefix_lens,
                                       const int32_t* extend_lens, const int32_t* extend_start_loc,
                                       int64_t batch, int64_t total_tokens, int64_t max_extend_len,
                                       int num_q_heads, int num_kv_heads, int head_dim,
                                       int64_t q_stride, int64_t out_stride,
                                       int64_t req_to_token_stride, float sm_scale, int dtype,
                                       int sm_budget, spd_stream_t stream) {
  int rc = check_attn_args("spd_attn_prefill_ragged", out, q, k_pool, v_pool, req_to_token,
                           req_pool_indices, num_q_heads, num_kv_heads, head_dim, q_stride, out_stride);
  if (rc) return rc;
  SPD_REQUIRE(prefix_lens && extend_lens && extend_start_loc && batch >= 0 && total_tokens >= 0 &&
                  max_extend_len >= 0,
              SPD_E_BADARG, "spd_attn_prefill_ragged: bad arguments");
  SPD_REQUIRE(head_dim == kPfD, SPD_E_SHAPE,
              "spd_attn_prefill_ragged: head_dim must be 128 on the tcgen05 path (got %d)", head_dim);
  if (batch == 0 || total_tokens == 0 || max_extend_len == 0) return 0;
  PrefillParams p{};
  CUtensorMap tq, tk, tv, to;
  if ((rc = pf_setup(p, tq, tk, tv, to, out, q, k_pool, v_pool, req_to_token, req_pool_indices, prefix_lens, extend_lens,
                     extend_start_loc, batch, total_tokens, max_extend_len, num_q_heads, num_kv_heads, q_stride, out_stride,
                     req_to_token_stride, sm_scale)))
    return rc;
  const int sms = sm_budget > 0 ? sm_budget : device_sm_count_cached();
  const int grid = p.total_items < sms ? p.total_items : sms;
  p.sorted = pf_wants_list(p, total_tokens, grid);
#define SPD_PF_LAUNCH(TR)                                                                              \
  do {                                                                                                 \
    auto kern = attn_prefill_kernel<T, TR, false>;                                                             \
    static bool configured = false;                                                                    \
    if (!configured) {                                                                                 \
      SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPfSmem));      \
      configured = true;                                                                               \
    }                                                                                                  \
    SPD_CUDA(launch(kern, dim3(grid), dim3(kPfThreads), kPfSmem, as_stream(stream), pdl_enabled(), tq, tk, tv, to, p)); \
  } while (0)
  SPD_DISPATCH_DTYPE(dtype, {
    if (g_pf_trace) {
      p.trace = g_pf_trace;
      p.trace_cap = g_pf_trace_cap;
      SPD_PF_LAUNCH(true);
    } else {
      SPD_PF_LAUNCH(false);
    }
  });
#undef SPD_PF_LAUNCH
  return 0;
}
