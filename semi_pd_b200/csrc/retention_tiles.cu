// Retention mixer over long prefill batches: tiles of 128 tokens that all run at the same time (retention_chunked.cu walks a
// portion 64 tokens after 64).  In the segmented form of the same sums, per request, head and tile of n tokens,
//     U     = sum_j (c d^(n-1-j) k_j) v_j^T                     retention_tile_sums_kernel: what a tile adds to the state
//     S'    = d^n S + U                                         retention_tile_scan_kernel: the state before every tile
//     A_ij  = (q_i . k_j) c d^(i-j) for j <= i                  retention_tile_kernel
//     o_i   = d^(i+1) q_i S + sum_j A_ij v_j
// Operands are fp32 as three bf16 parts (retention_parts.cuh), products of two split operands six part products, smallest
// first, accumulated in fp32 in tensor memory.  Decays go into k before it is split, so that v, a bf16 number, keeps its one
// part and U takes three part products.
//
// Why tiles: a chunk's MMAs of 64 rows run at half the tensor core's rate, its phases follow one another, both halves of a
// head's values split q and k again, and the longest portion decides (41 chunks of 5.6 us of the 8192 tokens below).  Tiles
// of 128 rows and 128 value columns are independent, q lies in tensor memory (its products read only their other operand
// from shared memory), and the state is split once per 128 tokens.  4 requests, 8192 tokens, 16 heads of 128 x 128, bf16:
// 240 us in chunks, 168 here (sums 46, scan 28, outputs 88); one request of 8000 tokens 242 -> 153.  Against 64 bits the
// outputs' error is 2.47e-7 -> 2.10e-7, the state's 2.18e-7 -> 1.21e-7 (300 tokens: 2.01e-7 -> 2.04e-7, 1.05e-7 -> 1.07e-7).
// What bounds it: an output tile's phases (16 k clk: splitting q and k 3.3, Q K^T 2.4, Q S with A's split beside it 3.3, A V
// 1.7, outputs 1.7) that still follow one another for want of shared memory, issue slots 36 % busy, tensor core 25 %
// (under ncu, 94 us); the sums likewise (42 %, 12 %); the scan HBM and the L2 (71 MB read, 107 written, of which 49 left it in time).
#include <math.h>

#include "retention_parts.cuh"

namespace spd {

double retention_chunked_us(int64_t batch, int64_t total_tokens, int H, int dv, int sms);  // retention_chunked.cu

constexpr int kRtTok = 128;
constexpr int kRtBlock = kRtTok * 128;  // [128 rows x 128 B]: one swizzle block of a tile's operand
constexpr int kRtPart = 2 * kRtBlock;   // one part of k, A: 128 columns
constexpr int kRtThreads = 512;  // and a warp that hands in the MMAs
constexpr int kRtSumThreads = 256;

struct RetTileParams {
  RetChunkParams c;
  int4* list;  // per tile: (request, tile of the portion, tiles of the portion, first tile of the portion in the list),
               // (tokens, tokens from the tile's first to the portion's end, position, row)
  int* odd;    // [request][head][dv / cols]: first tile whose k or v have no parts, -1: a wait ran out
  uint8_t* states;
  float* powers;  // [head][129] of the decay
  int cols, max_tiles;
};

// What a tile adds to the state, [dv / 64][128][64] fp32: all tiles of a head side by side (with all heads of a tile side by
// side the scan's steps were a megabyte apart).  The state before it: [dv / cols] [3 parts][cols / 64][128 x 128 B], as the
// products read it.
__device__ __forceinline__ float* rt_slot(const RetTileParams& t, int h, int tile) {
  return t.c.sums + (static_cast<int64_t>(h) * t.max_tiles + tile) * t.c.dv * kRcDk;
}
__device__ __forceinline__ uint8_t* rt_state(const RetTileParams& t, int h, int tile, int z) {
  return t.states + ((static_cast<int64_t>(h) * t.max_tiles + tile) * (t.c.dv / t.cols) + z) * (3ll * (t.cols / 64) * kRtBlock);
}
__device__ __forceinline__ double rt_power_f64(double b, int e) {
  double x = 1.0;
  for (; e > 0; e >>= 1) {
    if (e & 1) x *= b;
    b *= b;
  }
  return x;
}
__device__ __forceinline__ float rt_power(double b, int e) { return static_cast<float>(rt_power_f64(b, e)); }  // rounded once
__device__ __forceinline__ void rt_st_x4(uint32_t taddr, const uint32_t (&r)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3])
               : "memory");
}
// 16 lanes x 32 columns as mma fragments (rc_ld_frag)
__device__ __forceinline__ void rt_ld_frag(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void rt_floats4(const float4& a, const float4& b, float (&x)[8]) {
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
  x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
template <typename T>
__device__ __forceinline__ void rt_floats(const uint4& w, float (&x)[8]) {
  const uint32_t a[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = unpack2<T>(a[e]);
    x[2 * e] = f.x;
    x[2 * e + 1] = f.y;
  }
}
// the parts of eight numbers in registers
struct RtParts {
  uint32_t p[3][4];
};
__device__ __forceinline__ RtParts rt_split8(const float (&x)[8]) {
  RtParts r;
#pragma unroll
  for (int e = 0; e < 4; ++e) rc_split2(x[2 * e], x[2 * e + 1], r.p[0][e], r.p[1][e], r.p[2][e]);
  return r;
}

// U of every tile, [128 x NC] of a head, to its slot; the list of tiles; whether k and v have parts.  256 threads, two CTAs per
// SM, items one after another: one CTA splits while the other's MMAs run, and the next 64 tokens' rows are on their way to
// shared memory meanwhile.  64 tokens at a time, each half of a tile with an accumulator of its own (sums of more products in
// tensor memory lose bits), added in fp32.
template <typename T, int VS, int NC>
__global__ void __launch_bounds__(kRtSumThreads, 2)
retention_tile_sums_kernel(const __grid_constant__ RetTileParams t) {
  const RetChunkParams& p = t.c;
  constexpr int kBlocks = NC / 64, kV = kBlocks * kRcV;  // one part of v: [64 x 128 B] blocks of 64 columns
  extern __shared__ uint8_t rt_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(rt_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem;                // 3 parts
  uint8_t* sV = sK + 3 * kRcQ;       // bf16: two chunks' v; fp16: two parts
  uint8_t* raw = sV + 2 * kV;        // raw rows of k, 64 of 256 B; fp16: and of v
  constexpr int kRaw = kRcQ + (VS == 2 ? kV : 0);
  uint64_t* bar = reinterpret_cast<uint64_t*>(raw + kRaw);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* powers = reinterpret_cast<float*>(bar + 2);  // [2][132], items in turn

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const bool leader = elect_one();
  const int zs = p.dv / NC, per_tile = p.H * zs;
  const int step_tile = static_cast<int>(gridDim.x) / per_tile, step_hz = static_cast<int>(gridDim.x) - step_tile * per_tile;
  const int half = p.rot >> 1, groups = p.rot >> 4;
  const int kt = tid >> 3, u = tid & 7;  // this thread's pieces of k: u and u + 8 of rows kt and kt + 32
  int tile = static_cast<int>(blockIdx.x) / per_tile, hz = static_cast<int>(blockIdx.x) - tile * per_tile;
  // the chunk that is fetched: tokens from t0 of the item's n
  struct Chunk {
    int tile, h, z, n, t0, pos;
  } next{0, 0, 0, 0, 0, 0};
  int64_t row0 = 0;
  auto place = [&]() {  // item (tile, hz); its tile's list entry is written once, a portion's marks by its first tile's items
    next.n = next.t0 = 0;
    if (tile >= t.max_tiles) return;
    RcSegment sg{0, 0, 0, 0};
    const bool there = rc_segment(p, tile, sg);
    const int begin = sg.seg * kRtTok, all = there ? p.extend_lens[sg.r] : 0;
    row0 = there ? p.extend_start_loc[sg.r] + begin : 0;
    next.pos = there ? p.prefix_lens[sg.r] + begin : 0;
    next.n = min(kRtTok, all - begin);
    next.tile = tile;
    next.h = hz / zs;
    next.z = hz - next.h * zs;
    if (hz == 0 && tid == 0) {
      t.list[2 * tile] = make_int4(sg.r, sg.seg, sg.nseg, sg.first);
      t.list[2 * tile + 1] = make_int4(next.n, all - begin, next.pos, static_cast<int>(row0));
    }
    if (there && sg.seg == 0 && tid == 0) t.odd[static_cast<int64_t>(sg.r) * per_tile + hz] = 0x7fffffff;
  };
  auto fetch = [&](uint32_t buf) {  // zeros past the portion
    constexpr int kKRows = kRtSumThreads / 16, kVRows = kRtSumThreads / (NC / 8);  // rows that the CTA takes at once
    const int kr = tid >> 4, kc = tid & 15, vr = tid / (NC / 8), vc = tid % (NC / 8);
    const T* kg = reinterpret_cast<const T*>(p.k) + (row0 + next.t0 + kr) * p.k_stride + next.h * kRcDk + kc * 8;
    const T* vg = reinterpret_cast<const T*>(p.v) + (row0 + next.t0 + vr) * p.v_stride + next.h * p.dv + next.z * NC + vc * 8;
    const uint32_t kd = smem_u32(raw), vd = (VS == 1 ? smem_u32(sV) + buf * kV : kd + kRcQ) + (vc >> 3) * kRcV;
    const int left = next.n - next.t0;
#pragma unroll
    for (int r = 0; r < kRcTok; r += kKRows, kg += kKRows * p.k_stride)
      cp_async16(kd + rc_raw(kr + r, kc), kr + r < left ? kg : reinterpret_cast<const T*>(p.k), kr + r < left);
#pragma unroll
    for (int r = 0; r < kRcTok; r += kVRows, vg += kVRows * p.v_stride)
      cp_async16(vd + rc_off(vr + r, vc & 7), vr + r < left ? vg : reinterpret_cast<const T*>(p.v), vr + r < left);
    cp_async_commit();
  };
  float4 ang[2][4];  // cos and sin of the fetched rows' pieces u (of u and u + 8, where both are rotated: of u + 8 later)
  auto angles = [&](const Chunk& c, int r, int piece, float4 (&a)[4]) {
    const int64_t pos = min(static_cast<int64_t>(c.pos) + c.t0 + kt + 32 * r, p.max_positions - 1);
    const float* cp = p.cos_sin + pos * p.rot + 8 * (piece < groups ? piece : piece - groups);
    a[0] = __ldg(reinterpret_cast<const float4*>(cp));
    a[1] = __ldg(reinterpret_cast<const float4*>(cp) + 1);
    a[2] = __ldg(reinterpret_cast<const float4*>(cp + half));
    a[3] = __ldg(reinterpret_cast<const float4*>(cp + half) + 1);
  };
  uint32_t items = 0;  // whose powers have been written
  auto start = [&]() {  // of an item: d^0 .. d^128
    if (next.t0 == 0 && next.n > 0) {
      if (tid <= kRtTok) powers[(items & 1) * 132 + tid] = rt_power(static_cast<double>(p.decay[next.h]), tid);
      ++items;
    }
    if (next.n > 0 && u < 2 * groups)
#pragma unroll
      for (int r = 0; r < 2; ++r) angles(next, r, u, ang[r]);
  };
  place();
  if (next.n > 0) {
    fetch(0);
    start();
  }
  if (warp == 0) {
    if (lane == 0) {
      mbar_init(bar, 1);
      *dead = 0;
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, 2 * NC);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tU = *tmem_slot;
  uint32_t buf = 0, par = 1;  // (the wait before the first chunk's products passes)
  uint32_t z = 0;
  Chunk cur{0, 0, 0, 0, 0, 0};
  // the item of `cur` has been multiplied
  auto output = [&](int spoilt) {
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    float* sums = rt_slot(t, cur.h, cur.tile) + cur.z * NC * kRcDk;
    tc_fence_after_sync();
    // as fragments: four threads a 32-byte sector (rows of 16 bytes a thread, 32 lines an instruction, took 60 us for 58 tiles
    // of 16 heads)
#pragma unroll 1
    for (int i = 0; i < NC / 32; ++i) {
      const int hf = i & 1, col = (warp >> 2) * (NC / 2) + (i >> 1) * 32, row = (warp & 3) * 32 + hf * 16 + (lane >> 2);
      const uint32_t at = tU + lane_base + (static_cast<uint32_t>(hf * 16) << 16) + col;
      uint32_t x[16], y[16];
      rt_ld_frag(at, x);
      if (cur.n > kRcTok) rt_ld_frag(at + NC, y);
      tmem_ld_wait();
      float* dst = sums + ((col >> 6) * kRcDk + row) * kRcDv + (col & 63) + 2 * (lane & 3);
#pragma unroll
      for (int g = 0; g < 4; ++g)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float a = __uint_as_float(x[4 * g + 2 * e]), b = __uint_as_float(x[4 * g + 2 * e + 1]);
          if (cur.n > kRcTok) {
            a += __uint_as_float(y[4 * g + 2 * e]);
            b += __uint_as_float(y[4 * g + 2 * e + 1]);
          }
          *reinterpret_cast<float2*>(dst + 8 * e * kRcDv + 8 * g) = make_float2(a, b);
        }
    }
    tc_fence_before_sync();
    if (tid == 0) p.flags[(static_cast<int64_t>(cur.tile) * p.H + cur.h) * zs + cur.z] = *dead ? 2 : spoilt ? 1 : 0;
  };
  bool ends = false;  // cur is its item's last chunk
  while (next.n > 0) {
    if (warp == 0) mbar_wait_bounded(bar, par, dead);  // the products before: the operands' memory is free
    par ^= 1;
    cp_async_wait<0>();
    const int spoilt = __syncthreads_or(rc_spoilt(z));
    if (ends) {
      output(spoilt);
      z = 0;
    }
    cur = next;
    const float* pw = powers + ((items - 1) & 1) * 132;
    const int n = cur.n, t0 = cur.t0;
    ends = t0 + kRcTok >= n;
    float4 now[2][4];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) now[r][e] = ang[r][e];
    if (ends) {
      tile += step_tile;
      hz += step_hz;
      if (hz >= per_tile) {
        hz -= per_tile;
        ++tile;
      }
      place();
    } else {
      next.t0 += kRcTok;
    }
    // ---- k: rotate, scale, split ----
    const uint8_t* kr = raw;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = kt + 32 * r, tok = t0 + row;
      const float f = tok < n ? pw[n - 1 - tok] * p.k_scale : 0.f;
#pragma unroll
      for (int half8 = 0; half8 < 2; ++half8) {
        const int piece = u + 8 * half8;
        const bool first = piece < groups, rotated = piece < 2 * groups;
        float x[8];
        rc_load8<T>(reinterpret_cast<const T*>(kr + rc_raw(row, piece)), x);
        if (rotated) {
          float y[8], cs[8], sn[8];
          rc_load8<T>(reinterpret_cast<const T*>(kr + rc_raw(row, first ? piece + groups : piece - groups)), y);
          if (half8 == 1) angles(cur, r, piece, now[r]);
          rt_floats4(now[r][0], now[r][1], cs);
          rt_floats4(now[r][2], now[r][3], sn);
          const float sign = first ? -1.f : 1.f;
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = fmaf(x[e], cs[e], y[e] * (sign * sn[e]));
        }
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          rc_watch(pack2<__nv_bfloat16>(x[e], x[e + 1]), z);
          x[e] *= f;
          x[e + 1] *= f;
        }
        rc_split8(x, sK + half8 * kRcV + rc_off(row, u), kRcQ);
      }
    }
    // ---- v: bf16 numbers lie where they are read; fp16 ones have two parts ----
#pragma unroll
    for (int j = 0; j < kRcTok * (NC / 8) / kRtSumThreads; ++j) {
      const int i = j * kRtSumThreads + tid, r = i / (NC / 8), c = i % (NC / 8);
      const uint32_t off = (c >> 3) * kRcV + rc_off(r, c & 7);
      if constexpr (VS == 1) {
        const uint4 w = *reinterpret_cast<const uint4*>(sV + buf * kV + off);
        rc_watch(w.x, z);
        rc_watch(w.y, z);
        rc_watch(w.z, z);
        rc_watch(w.w, z);
      } else {
        float x[8];
        rc_load8<T>(reinterpret_cast<const T*>(kr + kRcQ + off), x);
        const RtParts q = rt_split8(x);
#pragma unroll
        for (int e = 0; e < 4; ++e) rc_watch(q.p[0][e], z);
#pragma unroll
        for (int e = 0; e < 2; ++e)
          *reinterpret_cast<uint4*>(sV + e * kV + off) = make_uint4(q.p[e][0], q.p[e][1], q.p[e][2], q.p[e][3]);
      }
    }
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    if (next.n > 0) fetch(buf ^ 1);
    if (warp == 0) {
      tc_fence_after_sync();
      constexpr uint32_t id_kv = umma_idesc<__nv_bfloat16>(128, NC, 1, 1);
      const uint64_t dk = umma_desc_sw128(smem_u32(sK), kRcV, 1024), dw = umma_desc_sw128(smem_u32(sV) + (VS == 1 ? buf * kV : 0), kRcV, 1024);
      const uint32_t hi = static_cast<uint32_t>(dk >> 32), d = tU + (t0 > 0 ? NC : 0);
      uint32_t acc = 0;
#pragma unroll 1
      for (int pr = 0; pr < 6; ++pr) {
        if (rc_pb(pr) >= VS) continue;
        const uint32_t a = static_cast<uint32_t>(dk) + rc_pa(pr) * (kRcQ >> 4), b = static_cast<uint32_t>(dw) + rc_pb(pr) * (kV >> 4);
#pragma unroll
        for (int s = 0; s < kRcTok / 16; ++s) {
          umma_ss_if(leader, d, a + s * 128, b + s * 128, hi, id_kv, acc);
          acc = 1;
        }
      }
      umma_commit_if(leader, bar);
    }
    __syncwarp();
    start();
    buf ^= 1;
  }
  if (warp == 0) mbar_wait_bounded(bar, par, dead);
  const int spoilt = __syncthreads_or(rc_spoilt(z));
  if (ends) output(spoilt);
  __syncthreads();
  if (*dead) {
    wait_drain();
    if (tid == 0) wait_report(p.wait_expired);
  }
  if (warp == 0) tmem_dealloc(tU, 2 * NC);
}

// The state before every tile of a portion, in parts, and the portion's last state: S' = d^n S + U.  A CTA takes 1024 values of a head through the tiles of its portion.  A portion that starts from a state without parts (or so
// large that sums with it may end) is marked odd from its first tile on: that tile's CTA then takes all of it.
__global__ void __launch_bounds__(256)
retention_tile_scan_kernel(const __grid_constant__ RetTileParams t) {
  const RetChunkParams& p = t.c;
  __shared__ float2 d_tile[2];  // d^128 and d^n of the last tile as two floats: their rounding would add up over the tiles
  const int r = blockIdx.y, lane = threadIdx.x & 31;
  const int64_t per_head = static_cast<int64_t>(p.dv) * kRcDk, at = blockIdx.x * 1024ll;  // (a multiple of 1024 floats a head)
  const int h = static_cast<int>(at / per_head), in_head = static_cast<int>(at % per_head) + threadIdx.x * 4;
  const int block = in_head / (kRcDk * kRcDv), sr = in_head % (kRcDk * kRcDv) / kRcDv, col = block * kRcDv + in_head % kRcDv;
  int first = 0, ntile = 0;
  for (int i = lane; i <= r; i += 32) {
    const int m = p.prefix_lens[i] >= 0 ? max(p.extend_lens[i], 0) : 0, ns = (m + kRtTok - 1) / kRtTok;
    if (i < r) first += ns;
    else ntile = ns;
  }
  const int pos0 = p.prefix_lens[r], n_last = p.extend_lens[r] - (p.extend_lens[r] - 1) / kRtTok * kRtTok;
  const double decay = static_cast<double>(p.decay[h]);
  float* st = p.state + (p.req_pool_indices[r] * p.H + h) * per_head + static_cast<int64_t>(sr) * p.dv + col;
  first = __reduce_add_sync(0xffffffffu, first);
  ntile = __reduce_add_sync(0xffffffffu, ntile);
  if (r == 0 && at == h * per_head && threadIdx.x <= kRtTok) t.powers[h * (kRtTok + 1) + threadIdx.x] = rt_power(decay, threadIdx.x);
  if (ntile == 0) return;
  const int64_t per_tile = per_head / 4;
  float4* slot = reinterpret_cast<float4*>(rt_slot(t, h, first) + in_head);
  const int part = t.cols / 64 * kRtBlock;
  const int64_t per_state = 3ll * (p.dv / kRcDv) * kRtBlock;
  uint8_t* parts = rt_state(t, h, first, col / t.cols) + (col % t.cols >> 6) * kRtBlock + rc_off(sr, (col & 63) >> 3) + (col & 7) * 2;
  constexpr int kAhead = 4;  // tiles whose sums come together, while the ones before are added
  float4 u[2][kAhead];
  auto load = [&](int i0, float4 (&x)[kAhead]) {
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
      if (i0 + j < ntile) x[j] = __ldcg(slot + (i0 + j) * per_tile);
  };
  load(0, u[0]);
  float4 S = pos0 > 0 ? *reinterpret_cast<const float4*>(st) : make_float4(0.f, 0.f, 0.f, 0.f);
  load(kAhead, u[1]);
  int odd = ntile, worst = 0;
  for (int i = lane; i < ntile; i += 32) {
    const int f = p.flags[((first + i) * static_cast<int64_t>(p.H) + h) * (p.dv / t.cols) + block * kRcDv / t.cols];
    worst = max(worst, f);
    if (f == 1) odd = min(odd, i);
  }
  if (threadIdx.x < 2) {
    const double x = rt_power_f64(decay, threadIdx.x == 0 ? kRtTok : n_last);
    const float hi = static_cast<float>(x);
    d_tile[threadIdx.x] = make_float2(hi, static_cast<float>(x - static_cast<double>(hi)));
  }
  odd = __reduce_min_sync(0xffffffffu, odd);
  worst = __reduce_max_sync(0xffffffffu, worst);
  const bool fine = fabsf(S.x) <= 0x1p64f && fabsf(S.y) <= 0x1p64f && fabsf(S.z) <= 0x1p64f && fabsf(S.w) <= 0x1p64f;
  // (several CTAs of a head write it; the sums of the portion's first tile have set it)
  int* mark = t.odd + (static_cast<int64_t>(r) * p.H + h) * (p.dv / t.cols) + block * kRcDv / t.cols;
  const int bad = __syncthreads_or(!fine);
  if (threadIdx.x == 0) atomicMin(mark, worst == 2 ? -1 : bad ? 0 : odd);
  const float2 d = d_tile[0], dl = d_tile[1];
  auto add = [&](int i0, const float4 (&x)[kAhead]) {
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      if (i0 + j >= ntile) break;
      uint32_t q[3][2];
      rc_split2(S.x, S.y, q[0][0], q[1][0], q[2][0]);
      rc_split2(S.z, S.w, q[0][1], q[1][1], q[2][1]);
#pragma unroll
      for (int e = 0; e < 3; ++e)
        *reinterpret_cast<uint2*>(parts + (i0 + j) * per_state + e * part) = make_uint2(q[e][0], q[e][1]);
      const float2 f = i0 + j == ntile - 1 ? dl : d;
      S.x = fmaf(f.x, S.x, fmaf(f.y, S.x, x[j].x));
      S.y = fmaf(f.x, S.y, fmaf(f.y, S.y, x[j].y));
      S.z = fmaf(f.x, S.z, fmaf(f.y, S.z, x[j].z));
      S.w = fmaf(f.x, S.w, fmaf(f.y, S.w, x[j].w));
    }
  };
  for (int i0 = 0; i0 < ntile; i0 += 2 * kAhead) {
    add(i0, u[0]);
    load(i0 + 2 * kAhead, u[0]);
    add(i0 + kAhead, u[1]);
    load(i0 + 3 * kAhead, u[1]);
  }
  if (worst != 2 && !bad) *reinterpret_cast<float4*>(st) = S;  // (bad: the first tile's CTA starts from what stands there)
}

// Among the 16 warps: a barrier; a wait by one warp, the others held at the barrier (sixteen polling warps take the issue slots
// that the MMAs' operands need); a warp's arrival on a barrier of the issuing warp
__device__ __forceinline__ void rt_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kRtThreads) : "memory"); }
__device__ __forceinline__ void rt_wait(uint64_t* bar, uint32_t parity, int warp, volatile int* dead) {
  if (warp == 0) mbar_wait_bounded(bar, parity, dead);
  rt_sync();
}
__device__ __forceinline__ void rt_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// Outputs of the tiles.  16 warps and one that hands in the MMAs, one CTA per SM, items (tile, head, NC value
// columns) one after another.
// Shared memory: X, k's parts, then A's; Y, raw q and k, then the state's parts; v.  Tensor memory: q's parts, A~ (then A V),
// q S.  While a phase's MMAs run the threads split what the next one needs.
template <typename T, int VS, int NC>
__global__ void __launch_bounds__(kRtThreads + 128, 1)
retention_tile_kernel(const __grid_constant__ RetTileParams t) {
  const RetChunkParams& p = t.c;
  constexpr int kBlocks = NC / 64, kS = kBlocks * kRtBlock;  // one part of the state, of v
  extern __shared__ uint8_t rt_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(rt_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sX = smem;                // 3 parts of 128 x 128
  uint8_t* sY = sX + 3 * kRtPart;    // 3 parts of 128 x NC; raw q, k: 128 rows of 256 B each
  constexpr int kYBytes = 3 * kS > 2 * kRtPart ? 3 * kS : 2 * kRtPart;
  uint8_t* sV = sY + kYBytes;        // VS parts of 128 x NC
  uint64_t* done = reinterpret_cast<uint64_t*>(sV + VS * kS);  // Q K^T, Q S, A V complete
  uint64_t* ready = done + 3;                                  // their operands are there, a warp at a time
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 6);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* spoilt = dead + 1;                     // [2] items in turn: q, k or v without parts
  float* powers = reinterpret_cast<float*>(done + 9);  // [2][132]

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const bool leader = elect_one();
  if (warp == 0) {
    if (lane == 0) {
      for (int i = 0; i < 3; ++i) {
        mbar_init(&done[i], 1);
        mbar_init(&ready[i], i == 1 ? 1 : kRtThreads / 32);
      }
      *dead = 0;
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = *tmem_slot, tQ = tm, tA = tm + 192, tO = tm + 320;
  const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const int row = (warp & 3) * 32 + lane, quarter = warp >> 2;
  const int half = p.rot >> 1, groups = p.rot >> 4, plain = (kRcDk - p.rot) >> 3;
  const int rot_steps = VS == 1 ? p.rot / 16 : kRcDk / 16;  // k-steps whose q, k need three parts
  const int zs = p.dv / NC, per_tile = p.H * zs;
  const int step_tile = static_cast<int>(gridDim.x) / per_tile, step_hz = static_cast<int>(gridDim.x) - step_tile * per_tile;

  // item: tile, head, value columns; the next one's list entry, rows, powers and angles are on their way early
  int tile = static_cast<int>(blockIdx.x) / per_tile, hz = static_cast<int>(blockIdx.x) - tile * per_tile;
  int h = hz / zs, col0 = (hz - h * zs) * NC;
  int4 a4 = make_int4(0, 0, 0, 0), b4 = a4;
  auto look = [&](int tl, int4& a, int4& b) {
    b.x = 0;
    if (tl < t.max_tiles) {
      a = t.list[2 * tl];
      b = t.list[2 * tl + 1];
    }
  };
  look(tile, a4, b4);
  uint32_t par = 0;

  // 640 threads start with 96 registers each; the issuing warp's group gives some to the four others (4 x 112 + 32 = 5 x 96)
  if (warp >= kRtThreads / 32) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    // The whole warp computes the operands, one lane issues; short loops (retention_chunked.cu).
    while (warp == kRtThreads / 32 && b4.x > 0) {
      mbar_wait_bounded(&ready[0], par, dead);
      tc_fence_after_sync();
      {
        constexpr uint32_t id = umma_idesc<__nv_bfloat16>(128, 128, 0, 0);
        const uint64_t dk = umma_desc_sw128(smem_u32(sX), 16, 1024);
        const uint32_t hi = static_cast<uint32_t>(dk >> 32);
        uint32_t acc = 0;
#pragma unroll 1
        for (int pr = 0; pr < 6; ++pr) {
          uint32_t a = tQ + rc_pa(pr) * 64, b = static_cast<uint32_t>(dk) + rc_pb(pr) * (kRtPart >> 4);
          const int steps = pr == 5 ? kRcDk / 16 : rot_steps;
#pragma unroll 1
          for (int s = 0; s < steps; s += 4) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              umma_ts_if(leader && s + e < steps, tA, a + e * 8, b + e * 2, hi, id, acc);
              acc = 1;
            }
            a += 32;
            b += kRtBlock >> 4;
          }
        }
        umma_commit_if(leader, &done[0]);
      }
      mbar_wait_bounded(&ready[1], par, dead);
      tc_fence_after_sync();
      {
        constexpr uint32_t id = umma_idesc<__nv_bfloat16>(128, NC, 0, 1);
        const uint64_t ds = umma_desc_sw128(smem_u32(sY), kRtBlock, 1024);
        const uint32_t hi = static_cast<uint32_t>(ds >> 32);
        uint32_t acc = 0;
#pragma unroll 1
        for (int pr = 0; pr < 6; ++pr) {
          uint32_t a = tQ + rc_pa(pr) * 64, b = static_cast<uint32_t>(ds) + rc_pb(pr) * (kS >> 4);
          const int steps = rc_pa(pr) == 0 ? kRcDk / 16 : rot_steps;
#pragma unroll 1
          for (int s = 0; s < steps; s += 4) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              umma_ts_if(leader && s + e < steps, tO, a + e * 8, b + e * 128, hi, id, acc);
              acc = 1;
            }
            a += 32;
            b += 512;
          }
        }
        umma_commit_if(leader, &done[1]);
      }
      mbar_wait_bounded(&ready[2], par, dead);
      tc_fence_after_sync();
      {
        constexpr uint32_t id = umma_idesc<__nv_bfloat16>(128, NC, 0, 1);
        const uint64_t da = umma_desc_sw128(smem_u32(sX), 16, 1024), dv = umma_desc_sw128(smem_u32(sV), kRtBlock, 1024);
        // (the two descriptors differ in the lower half only: the leading offset stands there)
        const uint32_t hi = static_cast<uint32_t>(da >> 32);
        // 64 keys an accumulator: A~'s place, and q's once Q S has read it (one of 128 keys had 5 % more error)
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          if (half == 1) {
            mbar_wait_bounded(&done[1], par, dead);
            tc_fence_after_sync();
          }
          uint32_t acc = 0;
#pragma unroll 1
          for (int pr = 0; pr < 6; ++pr) {
            if (rc_pb(pr) >= VS) continue;
            const uint32_t a = static_cast<uint32_t>(da) + rc_pa(pr) * (kRtPart >> 4) + half * (kRtBlock >> 4);
            const uint32_t b = static_cast<uint32_t>(dv) + rc_pb(pr) * (kS >> 4) + half * 512;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              umma_ss_if(leader, half ? tQ : tA, a + e * 2, b + e * 128, hi, id, acc);
              acc = 1;
            }
          }
        }
        umma_commit_if(leader, &done[2]);
      }
      tile += step_tile;
      hz += step_hz;
      if (hz >= per_tile) {
        hz -= per_tile;
        ++tile;
      }
      look(tile, a4, b4);
      par ^= 1;
    }
  } else {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
  auto fetch = [&](int h, const int4& b) {  // raw q, k; zeros past the portion
    constexpr int kRows = kRtThreads / 16;  // at once
    const int r0 = tid >> 4, c = tid & 15;
    const T* qg = reinterpret_cast<const T*>(p.q) + (b.w + r0) * p.q_stride + h * kRcDk + c * 8;
    const T* kg = reinterpret_cast<const T*>(p.k) + (b.w + r0) * p.k_stride + h * kRcDk + c * 8;
    const uint32_t dst = smem_u32(sY);
#pragma unroll
    for (int r = 0; r < kRtTok; r += kRows, qg += kRows * p.q_stride, kg += kRows * p.k_stride) {
      const bool ok = r0 + r < b.x;
      cp_async16(dst + rc_raw(r0 + r, c), ok ? qg : reinterpret_cast<const T*>(p.q), ok);
      cp_async16(dst + kRtPart + rc_raw(r0 + r, c), ok ? kg : reinterpret_cast<const T*>(p.k), ok);
    }
    cp_async_commit();
  };
  float power = 0.f;
  float4 ang[4];  // cos and sin of this thread's first pair of pieces
  auto angles = [&](int g) {
    int64_t pos = static_cast<int64_t>(b4.z) + row;
    pos = pos < p.max_positions ? pos : p.max_positions - 1;
    const float4* cp = reinterpret_cast<const float4*>(p.cos_sin + pos * p.rot + 8 * g);
    const float4* sp = reinterpret_cast<const float4*>(p.cos_sin + pos * p.rot + half + 8 * g);
    ang[0] = __ldg(cp);
    ang[1] = __ldg(cp + 1);
    ang[2] = __ldg(sp);
    ang[3] = __ldg(sp + 1);
  };
  auto early = [&]() {
    if (tid <= kRtTok) power = t.powers[h * (kRtTok + 1) + tid];
    if (quarter < groups) angles(quarter);
  };
  if (b4.x > 0) {
    fetch(h, b4);
    early();
  }
  while (b4.x > 0) {
    const int n = b4.x;
    const uint8_t* state = rt_state(t, h, tile, col0 / NC);
    // v's memory is free since the last A V
    constexpr int kVRows = kRtThreads / (NC / 8);
    const int vr = tid / (NC / 8), vc = tid % (NC / 8);
    const T* vg = reinterpret_cast<const T*>(p.v) + (b4.w + vr) * p.v_stride + h * p.dv + col0 + vc * 8;
    uint4 rv[VS == 2 ? kRtTok / kVRows : 1];
#pragma unroll
    for (int j = 0; j < kRtTok / kVRows; ++j, vg += kVRows * p.v_stride) {
      const int tok = vr + j * kVRows;
      if constexpr (VS == 1)
        cp_async16(smem_u32(sV) + (vc >> 3) * kRtBlock + rc_off(tok, vc & 7), tok < n ? vg : reinterpret_cast<const T*>(p.v), tok < n);
      else
        rv[j] = tok < n ? __ldg(reinterpret_cast<const uint4*>(vg)) : make_uint4(0, 0, 0, 0);
    }
    if constexpr (VS == 1) cp_async_commit();
    const int odd_tile = t.odd[(static_cast<int64_t>(a4.x) * p.H + h) * (p.dv / t.cols) + col0 / t.cols];
    float* pw = powers + par * 132;
    if (tid <= kRtTok) pw[tid] = power * p.k_scale;  // c d^i
    if (tid == 0) spoilt[par] = 0;
    if constexpr (VS == 1) cp_async_wait<1>();  // (v's copies may still be on their way)
    else cp_async_wait<0>();
    rt_sync();
    // ---- q to tensor memory, k to X: rotate, split ----
    uint32_t z = 0;
    auto put = [&](const float (&x)[8], int w, int piece) {
      const RtParts s = rt_split8(x);
#pragma unroll
      for (int e = 0; e < 4; ++e) rc_watch(s.p[0][e], z);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        if (w == 0) rt_st_x4(tQ + lane_base + q * 64 + piece * 4, s.p[q]);
        else *reinterpret_cast<uint4*>(sX + q * kRtPart + (piece >> 3) * kRtBlock + rc_off(row, piece & 7)) =
            make_uint4(s.p[q][0], s.p[q][1], s.p[q][2], s.p[q][3]);
      }
    };
#pragma unroll 1
    for (int g = quarter; g < groups; g += 4) {  // pairs of pieces g and g + groups
      float cs[8], sn[8];
      if (g != quarter) angles(g);
      rt_floats4(ang[0], ang[1], cs);
      rt_floats4(ang[2], ang[3], sn);
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        float x[8], y[8];
        rc_load8<T>(reinterpret_cast<const T*>(sY + w * kRtPart + rc_raw(row, g)), x);
        rc_load8<T>(reinterpret_cast<const T*>(sY + w * kRtPart + rc_raw(row, g + groups)), y);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float a = x[e], b = y[e];
          x[e] = fmaf(a, cs[e], -(b * sn[e]));
          y[e] = fmaf(b, cs[e], a * sn[e]);
        }
        put(x, w, g);
        put(y, w, g + groups);
      }
    }
#pragma unroll 1
    for (int i = quarter; i < plain; i += 4) {
      const int piece = 2 * groups + i;
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const uint8_t* raw = sY + w * kRtPart + rc_raw(row, piece);
        if constexpr (VS == 1) {  // a bf16 number that is not rotated has one part; the others' are not multiplied
          const uint4 x = *reinterpret_cast<const uint4*>(raw);
          const uint32_t r[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) rc_watch(r[e], z);
          if (w == 0) rt_st_x4(tQ + lane_base + piece * 4, r);
          else *reinterpret_cast<uint4*>(sX + (piece >> 3) * kRtBlock + rc_off(row, piece & 7)) = x;
        } else {
          float x[8];
          rc_load8<T>(reinterpret_cast<const T*>(raw), x);
          put(x, w, piece);
        }
      }
    }
    tmem_st_wait();
    fence_proxy_async_smem();
    tc_fence_before_sync();
    if (rc_spoilt(z)) spoilt[par] = 1;
    rt_arrive(&ready[0], lane);
    rt_sync();  // the raw rows have been read
    // ---- the state's parts over the raw rows; fp16 values' parts ----
    if (tid == 0) {
      fence_proxy_async_smem();
      mbar_expect_tx(&ready[1], 3 * kS);
#pragma unroll
      for (int q = 0; q < 3; ++q)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(sY + q * kS)),
                     "l"(state + q * kS), "r"(kS), "r"(smem_u32(&ready[1]))
                     : "memory");
    }
    if constexpr (VS == 2) {
#pragma unroll
      for (int j = 0; j < kRtTok * (NC / 8) / kRtThreads; ++j) {
        const int i = j * kRtThreads + tid, tok = i / (NC / 8), c = i % (NC / 8);
        float x[8];
        rt_floats<T>(rv[j], x);
        const RtParts s = rt_split8(x);
#pragma unroll
        for (int q = 0; q < VS; ++q)
          *reinterpret_cast<uint4*>(sV + q * kS + (c >> 3) * kRtBlock + rc_off(tok, c & 7)) =
              make_uint4(s.p[q][0], s.p[q][1], s.p[q][2], s.p[q][3]);
      }
    }
    int next_tile = tile + step_tile, next_hz = hz + step_hz;
    if (next_hz >= per_tile) {
      next_hz -= per_tile;
      ++next_tile;
    }
    int4 a_next = a4, b_next = b4;
    look(next_tile, a_next, b_next);
    float back[4];  // d^(i + 1) of the rows that this thread writes
#pragma unroll
    for (int e = 0; e < 4; ++e) back[e] = t.powers[h * (kRtTok + 1) + (warp & 3) * 32 + 8 * e + (lane >> 2) + 1];
    // ---- A: decay, mask, split, over k's parts ----
    rt_wait(&done[0], par, warp, dead);
    tc_fence_after_sync();
    // (rows of a warp: 32 from a multiple of 32 on; columns likewise: whole blocks above the diagonal are zeros)
    if (quarter > (warp & 3)) {
#pragma unroll
      for (int g = 0; g < 4; ++g)
#pragma unroll
        for (int q = 0; q < 3; ++q)
          *reinterpret_cast<uint4*>(sX + q * kRtPart + (quarter >> 1) * kRtBlock + rc_off(row, (quarter * 4 + g) & 7)) = make_uint4(0, 0, 0, 0);
    } else {
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        const int j0 = quarter * 32 + c * 16;
        uint32_t x[16];
        tmem_ld_32x32b_x16(tA + lane_base + j0, x);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          float y[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int age = row - j0 - 8 * g - e;
            y[e] = age >= 0 ? __uint_as_float(x[8 * g + e]) * pw[max(age, 0)] : 0.f;
          }
          rc_split8(y, sX + (quarter >> 1) * kRtBlock + rc_off(row, ((j0 >> 3) + g) & 7), kRtPart);
        }
      }
    }
    if constexpr (VS == 1) cp_async_wait<0>();  // v
    fence_proxy_async_smem();
    tc_fence_before_sync();
    rt_arrive(&ready[2], lane);
    // ---- outputs ----
    rt_wait(&done[1], par, warp, dead);
    tc_fence_after_sync();
    const int next_h = next_hz / zs;
    if (b_next.x > 0) fetch(next_h, b_next);  // the state's parts have been multiplied
    constexpr int kCols = NC / 4;  // of a warp: 32 or 16
    const int fr = lane >> 2, fc = quarter * kCols + 2 * (lane & 3);
    float* og = p.o + (static_cast<int64_t>(b4.w) * p.H + h) * static_cast<int64_t>(p.dv) + col0;
    const bool mine = odd_tile >= a4.y;  // else an earlier tile takes this one, or a wait ran out
#pragma unroll 1
    for (int hf = 0; hf < 2; ++hf) {
      const uint32_t at = lane_base + (static_cast<uint32_t>(hf * 16) << 16) + quarter * kCols;
      uint32_t x[kCols / 2], y[kCols / 2], w[kCols / 2];
      if constexpr (kCols == 32) rt_ld_frag(tO + at, x);
      else rc_ld_frag(tO + at, x);
      if (hf == 0) {
        rt_wait(&done[2], par, warp, dead);
        tc_fence_after_sync();
      }
      if constexpr (kCols == 32) {
        rt_ld_frag(tA + at, y);
        rt_ld_frag(tQ + at, w);
      } else {
        rc_ld_frag(tA + at, y);
        rc_ld_frag(tQ + at, w);
      }
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = (warp & 3) * 32 + hf * 16 + fr + 8 * e;
        if (i < n && mine) {
          const float f = hf == 0 ? back[e] : back[2 + e];
          float* dst = og + static_cast<int64_t>(i) * p.H * p.dv + fc;
#pragma unroll
          for (int g = 0; g < kCols / 8; ++g)
            *reinterpret_cast<float2*>(dst + 8 * g) =
                make_float2(fmaf(f, __uint_as_float(x[4 * g + 2 * e]), __uint_as_float(y[4 * g + 2 * e]) + __uint_as_float(w[4 * g + 2 * e])),
                            fmaf(f, __uint_as_float(x[4 * g + 2 * e + 1]),
                                 __uint_as_float(y[4 * g + 2 * e + 1]) + __uint_as_float(w[4 * g + 2 * e + 1])));
        }
      }
    }
    tc_fence_before_sync();
    if (mine && !*dead && (spoilt[par] || odd_tile == a4.y)) {
      // q, k or v without parts: this tile (all that follows, where the state behind it would not exist) token by token
      const bool rest = odd_tile == a4.y;
      const int sr = row, sc = quarter * 16;
      for (int blk = 0; blk < kBlocks; ++blk) {
        float* st = p.state + (p.req_pool_indices[a4.x] * p.H + h) * static_cast<int64_t>(kRcDk) * p.dv +
                    static_cast<int64_t>(sr) * p.dv + col0 + blk * kRcDv + sc;
        float from[16];  // the parts' sum is the state, to the bit
        for (int c = 0; c < 2; ++c) {
          float x[3][8];
          for (int q = 0; q < 3; ++q)
            rc_load8<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(state + q * kS + blk * kRtBlock + rc_off(sr, (sc >> 3) + c)), x[q]);
          for (int e = 0; e < 8; ++e) {
            const float sum = (x[0][e] + x[1][e]) + x[2][e];
            // (no parts: the portion's first state, which stands untouched.  Behind an earlier tile a state is finite and has
            // parts however large it is, and what stands in memory is the portion's last one.)
            from[8 * c + e] = a4.y > 0 || fabsf(sum) <= 0x1p64f ? sum : st[8 * c + e];
          }
        }
        rc_token_by_token<T, 1>(&p, 0, rest ? b4.y : n, b4.z, b4.w, reinterpret_cast<float*>(sX), from, rest ? st : nullptr, p.decay[h], h,
                                col0 + blk * kRcDv);
      }
    }
    par ^= 1;
    tile = next_tile;
    hz = next_hz;
    h = next_h;
    col0 = (hz - h * zs) * NC;
    a4 = a_next;
    b4 = b_next;
    if (b4.x > 0) early();
  }
  cp_async_wait<0>();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*dead) {
    wait_drain();
    if (tid == 0) wait_report(p.wait_expired);
  }
  if (warp == 0) tmem_dealloc(tm, 512);
}

template <typename T, int VS, int NC>
static int rt_launch(const RetTileParams& t, int sms, cudaStream_t stream) {
  constexpr int kS = NC / 64 * kRtBlock, kY = 3 * kS > 2 * kRtPart ? 3 * kS : 2 * kRtPart;
  constexpr int kV = (NC / 64) * kRcV, sum_smem = 3 * kRcQ + 2 * kV + kRcQ + (VS == 2 ? kV : 0) + 1024 + 1280, smem = 3 * kRtPart + kY + VS * kS + 1024 + 2048;
  static_assert(smem <= 232448 && 2 * (sum_smem + 1024) <= 233472, "shared memory of an SM");
  auto sums = retention_tile_sums_kernel<T, VS, NC>;
  auto kern = retention_tile_kernel<T, VS, NC>;
  static bool configured = false;  // per instantiation
  if (!configured) {
    SPD_CUDA(cudaFuncSetAttribute(sums, cudaFuncAttributeMaxDynamicSharedMemorySize, sum_smem));
    SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured = true;
  }
  const RetChunkParams& p = t.c;
  const int64_t items = static_cast<int64_t>(t.max_tiles) * p.H * (p.dv / NC);
  SPD_CUDA(launch(sums, dim3((unsigned)(items < 2 * sms ? items : 2 * sms)), dim3(kRtSumThreads), sum_smem, stream, /*pdl=*/false, t));
  SPD_CUDA(launch(retention_tile_scan_kernel, dim3((unsigned)(p.H * (p.dv / kRcDv) * (kRcDk * kRcDv / 1024)), (unsigned)p.batch),
                  dim3(256), 0, stream, /*pdl=*/false, t));
  SPD_CUDA(launch(kern, dim3((unsigned)(items < sms ? items : sms)), dim3(kRtThreads + 128), smem, stream, /*pdl=*/false, t));
  return 0;
}

// Estimated us: 11 and 18.5 a wave of tiles (its sums, its part of the scan, its outputs), 64 value columns at a time 12 and
// 15 (bf16) or 16 (fp16).  Taken where that is 7 % below the chunks' estimate (retention_chunked_us) and the portions of a single
// wave have more than four chunks in the mean.  16 heads of 128 x 128, chunks / tiles in us: 1 x 256 tokens 29.1 / 31.1 (not taken),
// 300 35.3 / 31.1, 1500 67.9 / 43.5, 8000 235 / 148; 2 x 250 29.8 / 33.2 (not taken), 2 x 450 52 / 35, 4 x 250 31 / 38 (not taken), 4 x
// 500 67 / 51, 8 x 300 69 / 77 (not taken), 8 x 1000 222 / 162; on 72 SMs 4 x 300 67 / 71 (not taken).  Of 2280 calls (1 - 64 portions of
// 64 - 8000 tokens, 4 - 32 heads, 64 - 256 value columns, both types, 148, 72 and 40 SMs) 8 take 2 - 6 % more than in chunks.
static bool rt_pays(int64_t batch, int64_t total_tokens, int H, int dv, bool half, int sms) {
  const int cols = !half && dv % 128 == 0 ? 128 : 64;
  const double items = (static_cast<double>(total_tokens) / kRtTok + 0.5 * static_cast<double>(batch)) * H * (dv / cols);
  const double waves = ceil(items / sms), us = cols == 128 ? 11 + 18.5 * waves : 12 + (half ? 16.0 : 15.0) * waves;
  if (waves <= 1 && total_tokens <= 2 * kRtTok * batch) return false;
  return us < 0.93 * retention_chunked_us(batch, total_tokens, H, dv, sms);
}

// A call's scratch at most, beyond which the chunks serve, which want far less or none: it is 10 bytes a state value and 128 tokens
// (4 x 2048 tokens, 16 heads of 128 x 128: 178 MB), and a server leaves little beside its caches.
constexpr int64_t kRtMaxScratch = 512ll << 20;

static int64_t rt_tiles(int64_t batch, int64_t total_tokens) { return total_tokens / kRtTok + batch; }
// fp32 sums, then the states' parts
static int64_t rt_state_bytes(int64_t tiles, int H, int dv, int bytes) { return tiles * H * static_cast<int64_t>(dv) * kRcDk * bytes; }

}  // namespace spd

using namespace spd;

extern "C" {

int64_t spd_retention_tiles_workspace_bytes(int64_t batch, int64_t total_tokens, int num_heads, int head_dim, int v_dim,
                                            int rot_dims, int in_act, int dtype, int sm_budget) {
  if (batch <= 0 || batch > 65535 || num_heads <= 0 || num_heads > 65535 || total_tokens <= 0) return 0;
  if (dtype == SPD_F32 || in_act != 0 || head_dim != kRcDk || v_dim <= 0 || v_dim % kRcDv != 0 || rot_dims < 0 || rot_dims > kRcDk ||
      rot_dims % 16 != 0 || v_dim / kRcDv > 65535 || total_tokens <= 40 * batch)
    return 0;
  if (!rt_pays(batch, total_tokens, num_heads, v_dim, dtype == SPD_F16, sm_budget > 0 ? sm_budget : device_sm_count_cached())) return 0;
  const int64_t tiles = rt_tiles(batch, total_tokens);
  const int64_t room = rt_state_bytes(tiles, num_heads, v_dim, 10) + tiles * 32 + ((tiles + batch) * (v_dim / kRcDv) + kRtTok + 1) * num_heads * 4;
  return room <= kRtMaxScratch ? room : 0;
}

int spd_retention_extend_tiles(float* o, const void* q, const void* k, const void* v, float* state,
                               const int64_t* req_pool_indices, const int32_t* prefix_lens, const int32_t* extend_lens,
                               const int32_t* extend_start_loc, int64_t batch, int64_t total_tokens, int num_heads, int head_dim,
                               int v_dim, int64_t q_stride, int64_t k_stride, int64_t v_stride, const float* decay,
                               const float* cos_sin, int rot_dims, int64_t max_positions, float k_scale, int in_act, int dtype,
                               void* workspace, int64_t workspace_bytes, int sm_budget, spd_stream_t stream) {
  SPD_REQUIRE(o && q && k && v && state && req_pool_indices && prefix_lens && extend_lens && extend_start_loc && decay && workspace,
              SPD_E_BADARG, "spd_retention_extend_tiles: null pointer");
  SPD_REQUIRE(dtype == SPD_BF16 || dtype == SPD_F16, SPD_E_BADARG, "spd_retention_extend_tiles: bad dtype %d", dtype);
  const int64_t room = spd_retention_tiles_workspace_bytes(batch, total_tokens, num_heads, head_dim, v_dim, rot_dims, in_act, dtype, sm_budget);
  SPD_REQUIRE(room > 0 && (rot_dims == 0 || (cos_sin && max_positions > 0)), SPD_E_SHAPE,
              "spd_retention_extend_tiles: sizes that spd_retention_tiles_workspace_bytes has no room for");
  SPD_REQUIRE(workspace_bytes >= room, SPD_E_WORKSPACE, "spd_retention_extend_tiles: workspace too small");
  SPD_REQUIRE(q_stride % 8 == 0 && k_stride % 8 == 0 && v_stride % 8 == 0 && aligned16(q) && aligned16(k) && aligned16(v) &&
                  aligned16(o) && aligned16(state) && aligned16(workspace) && (rot_dims == 0 || aligned16(cos_sin)),
              SPD_E_ALIGN, "spd_retention_extend_tiles: rows, tables and buffers must be 16-byte aligned");
  RetTileParams t{};
  RetChunkParams& p = t.c;
  p = RetChunkParams{o, q, k, v, state, req_pool_indices, prefix_lens, extend_lens, extend_start_loc, num_heads, v_dim, rot_dims,
                     q_stride, k_stride, v_stride, max_positions, decay, cos_sin, k_scale, nullptr, static_cast<int>(batch), kRtTok,
                     nullptr, nullptr, nullptr, 0};
  if (int rc = wait_flag(&p.wait_expired)) return rc;
  t.max_tiles = static_cast<int>(rt_tiles(batch, total_tokens));
  // 128 value columns at a time; fp16 values have two parts, which leaves room for 64
  t.cols = p.flag_cols = dtype == SPD_BF16 && v_dim % 128 == 0 ? 128 : 64;
  p.sums = static_cast<float*>(workspace);
  t.states = static_cast<uint8_t*>(workspace) + rt_state_bytes(t.max_tiles, num_heads, v_dim, 4);
  t.list = reinterpret_cast<int4*>(static_cast<uint8_t*>(workspace) + rt_state_bytes(t.max_tiles, num_heads, v_dim, 10));
  p.flags = reinterpret_cast<int*>(t.list + 2 * t.max_tiles);
  t.odd = p.flags + static_cast<int64_t>(t.max_tiles) * num_heads * (v_dim / kRcDv);
  t.powers = reinterpret_cast<float*>(t.odd + batch * num_heads * (v_dim / kRcDv));
  const int sms = sm_budget > 0 ? sm_budget : device_sm_count_cached();
  cudaStream_t st = as_stream(stream);
  if (dtype == SPD_F16) return rt_launch<__half, 2, 64>(t, sms, st);
  return t.cols == 128 ? rt_launch<__nv_bfloat16, 1, 128>(t, sms, st) : rt_launch<__nv_bfloat16, 1, 64>(t, sms, st);
}

}  // extern "C"
