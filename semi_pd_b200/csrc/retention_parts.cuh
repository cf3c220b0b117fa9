// What the chunked and the tiled retention prefill share (retention_chunked.cu, retention_tiles.cu): fp32 numbers as three
// bf16 parts, the watch over numbers that have none, segments of portions, the way on token by token.
#pragma once
#include "common.cuh"
#include "prefill_tiles.cuh"
#include "ptx.cuh"

namespace spd {

constexpr int kRcTok = 64;       // tokens per chunk
constexpr int kRcDk = 128;       // key channels
constexpr int kRcDv = 64;        // value columns per CTA
constexpr int kRcThreads = 512;
constexpr int kRcQ = 2 * kRcTok * 128;   // one part of q or k: two [64 x 128 B] swizzle blocks
constexpr int kRcS = kRcDk * 128;        // one part of S: [128 x 128 B]
constexpr int kRcV = kRcTok * 128;       // one part of v, v', A: [64 x 128 B]
constexpr int kRcMisc = 1024;

struct RetChunkParams {
  float* o;
  const void *q, *k, *v;
  float* state;
  const int64_t* req_pool_indices;
  const int32_t *prefix_lens, *extend_lens, *extend_start_loc;
  int H, dv, rot;
  int64_t q_stride, k_stride, v_stride, max_positions;
  const float* decay;
  const float* cos_sin;
  float k_scale;
  unsigned* wait_expired;
  // portions cut into segments of seg_tokens (a multiple of 64) that run at the same time; sums == nullptr: not cut
  int batch, seg_tokens;
  float* sums;  // [segment][head][64-column block][128][64]: what a segment adds to the state, then the state behind it; of a
                // portion's last segment: the state that the portion starts from
  float* keep;  // the same again: the state at a segment's first token that has no parts
  int* flags;   // [segment][head][dv / cols of retention_sums]: 0, 1 (k or v have no parts), 2 (a wait ran out)
  int flag_cols;
};

__device__ __forceinline__ uint32_t rc_off(int row, int c) { return row * 128 + ((c ^ (row & 7)) << 4); }

// the same for raw rows of 256 bytes: threads that take one piece of many rows meet no bank conflicts
__device__ __forceinline__ uint32_t rc_raw(int row, int c) { return row * 256 + (((c & 8) | ((c ^ row) & 7)) << 4); }

// x = h + m + l in bf16 (exact to 24 bits), two numbers at a time
__device__ __forceinline__ void rc_split2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  const uint64_t minus = pack_f32x2(-1.f, -1.f);
  h = pack2<__nv_bfloat16>(x0, x1);
  float2 f = unpack2<__nv_bfloat16>(h);
  unpack_f32x2(ffma2(pack_f32x2(f.x, f.y), minus, pack_f32x2(x0, x1)), x0, x1);  // x - h
  m = pack2<__nv_bfloat16>(x0, x1);
  f = unpack2<__nv_bfloat16>(m);
  unpack_f32x2(ffma2(pack_f32x2(f.x, f.y), minus, pack_f32x2(x0, x1)), x0, x1);
  l = pack2<__nv_bfloat16>(x0, x1);
}
// eight numbers -> one 16-byte chunk per part at dst, dst + part, dst + 2 part; the upper parts
struct RcUpper {
  uint32_t h[4];
};
__device__ __forceinline__ RcUpper rc_split8(const float (&x)[8], uint8_t* dst, int part) {
  uint32_t h[4], m[4], l[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) rc_split2(x[2 * e], x[2 * e + 1], h[e], m[e], l[e]);
  *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<uint4*>(dst + part) = make_uint4(m[0], m[1], m[2], m[3]);
  *reinterpret_cast<uint4*>(dst + 2 * part) = make_uint4(l[0], l[1], l[2], l[3]);
  return {{h[0], h[1], h[2], h[3]}};
}
template <typename T>
__device__ __forceinline__ void rc_load8(const T* p, float (&x)[8]) {
  const uint4 w = *reinterpret_cast<const uint4*>(p);
  const uint32_t a[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = unpack2<T>(a[e]);
    x[2 * e] = f.x;
    x[2 * e + 1] = f.y;
  }
}

// Keeps watch over numbers that have no three parts (an infinity or NaN: inf - inf), and over ones so large that A might
// overflow where the token-by-token sums do not: z + 2^96 h in bf16 is not finite any more once an |h| was 2^32 or more
// (from 2^26 on where many were), and stays so.  One instruction per two numbers.
__device__ __forceinline__ void rc_watch(uint32_t h, uint32_t& z) {
  asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(z) : "r"(h), "r"(0x6f806f80u));
}
__device__ __forceinline__ bool rc_spoilt(uint32_t z) {
  return (z & 0x7f80u) == 0x7f80u || (z & 0x7f800000u) == 0x7f800000u;
}

// 16 lanes x 16 columns as mma fragments: value 4 g + e is row (lane >> 2) + 8 (e >> 1), column 8 g + 2 (lane & 3) + (e & 1)
__device__ __forceinline__ void rc_ld_frag(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// For all warps but the issuing one: warp 1 polls, the others are held at a barrier.  (Sixteen polling warps took the issue
// slots that the MMAs' operands need: 64 clk per MMA instead of 32 - 48.)
__device__ __forceinline__ void rc_wait(uint64_t* bar, uint32_t parity, int warp, volatile int* dead) {
  if (warp <= 1) mbar_wait_bounded(bar, parity, dead);
  if (warp >= 1) asm volatile("bar.sync 1, %0;" ::"n"(kRcThreads - 32) : "memory");
}

// Segment b of the batch's list (every portion's, one portion after another): request, place in it, segments of the request
// and the first of them.  Collective over a warp.
struct RcSegment {
  int r, seg, nseg, first;
};
__device__ __forceinline__ bool rc_segment(const RetChunkParams& p, int b, RcSegment& out) {
  const int lane = threadIdx.x & 31;
  int base = 0;
  for (int r0 = 0; r0 < p.batch; r0 += 32) {
    const int r = r0 + lane;
    const int n = r < p.batch && p.prefix_lens[r] >= 0 ? max(p.extend_lens[r], 0) : 0;
    const int ns = (n + p.seg_tokens - 1) / p.seg_tokens;
    int incl = ns;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    const uint32_t past = __ballot_sync(0xffffffffu, b < base + incl);
    if (past != 0) {
      const int src = __ffs(past) - 1, nseg = __shfl_sync(0xffffffffu, ns, src);
      const int first = base + __shfl_sync(0xffffffffu, incl, src) - nseg;
      out = {r0 + src, b - first, nseg, first};
      return true;
    }
    base += __shfl_sync(0xffffffffu, incl, 31);
  }
  return false;
}

// Tokens t0 .. n - 1 of a portion one after another on the CUDA cores, as retention.cu takes them.  f: 96 KB for [64][128]
// rotated q, rotated and scaled k, [64][64] v and [2][4][64] partial sums; from, to: this thread's 16 values of the state
// (to: nullptr where another segment of the portion writes it); h, col0: head and first of its 64 value columns.  Behind the
// chunks' loop and not inside it: there the call (never made) took 40 us of 256.
template <typename T, int kBar = 0>  // the barrier of the 512 threads
__device__ __forceinline__ void rc_token_by_token(const RetChunkParams* p, int t0, int n, int64_t pos0, int64_t row0, float* f,
                                                  const float* from, float* to_state, float dec, int h, int col0) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, half = p->rot >> 1;
  const int sr = (warp & 3) * 32 + lane, sc = (warp >> 2) * 16;
  auto sync = []() { asm volatile("bar.sync %0, %1;" ::"n"(kBar), "n"(kRcThreads) : "memory"); };
  float *fq = f, *fk = fq + kRcTok * kRcDk, *fv = fk + kRcTok * kRcDk, *part = fv + kRcTok * kRcDv;
  float S[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) S[i] = from[i];
#pragma unroll 1
  for (; t0 < n; t0 += kRcTok) {
    const int nt = min(kRcTok, n - t0);
    sync();  // what stood in `f` has been read
#pragma unroll 1
    for (int i = tid; i < nt * kRcDk; i += kRcThreads) {
      const int t = i / kRcDk, d = i % kRcDk;
      const int64_t row = row0 + t0 + t;
      const T* qr = reinterpret_cast<const T*>(p->q) + row * p->q_stride + h * kRcDk;
      const T* kr = reinterpret_cast<const T*>(p->k) + row * p->k_stride + h * kRcDk;
      float q = to_f32<T>(qr[d]), k = to_f32<T>(kr[d]);
      if (d < p->rot) {
        int64_t pos = pos0 + t0 + t;
        pos = pos < p->max_positions ? pos : p->max_positions - 1;
        const int j = d < half ? d : d - half, other = d < half ? d + half : d - half;
        const float c = p->cos_sin[pos * p->rot + j], s = p->cos_sin[pos * p->rot + half + j];
        const float q2 = to_f32<T>(qr[other]), k2 = to_f32<T>(kr[other]);
        q = d < half ? q * c - q2 * s : q * c + q2 * s;
        k = d < half ? k * c - k2 * s : k * c + k2 * s;
      }
      fq[i] = q;
      fk[i] = k * p->k_scale;
    }
#pragma unroll 1
    for (int i = tid; i < nt * kRcDv; i += kRcThreads)
      fv[i] = to_f32<T>(reinterpret_cast<const T*>(p->v)[(row0 + t0 + i / kRcDv) * p->v_stride +
                                                         static_cast<int64_t>(h) * p->dv + col0 + i % kRcDv]);
    sync();
#pragma unroll 1
    for (int t = 0; t < nt; ++t) {
      const float kt = fk[t * kRcDk + sr], qt = fq[t * kRcDk + sr];
      float* to = part + (t & 1) * 4 * kRcDv;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        S[i] = fmaf(dec, S[i], kt * fv[t * kRcDv + sc + i]);
        const float sum = warp_sum(S[i] * qt);
        if (lane == 0) to[(warp & 3) * kRcDv + sc + i] = sum;
      }
      sync();
      if (tid < kRcDv)
        p->o[((row0 + t0 + t) * p->H + h) * static_cast<int64_t>(p->dv) + col0 + tid] =
            (to[tid] + to[kRcDv + tid]) + (to[2 * kRcDv + tid] + to[3 * kRcDv + tid]);
    }
  }
  if (to_state != nullptr) {
#pragma unroll
    for (int i = 0; i < 16; ++i) to_state[i] = S[i];
  }
}

// parts (a, b) of the six products, smallest first
__host__ __device__ constexpr int rc_pa(int i) { return (0x001102 >> (4 * i)) & 15; }  // 2 0 1 1 0 0
__host__ __device__ constexpr int rc_pb(int i) { return (0x010120 >> (4 * i)) & 15; }  // 0 2 1 0 1 0

}  // namespace spd
