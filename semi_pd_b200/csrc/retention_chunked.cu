// Retention mixer over prefill portions on tcgen05, in 32-bit arithmetic carried by 16-bit tensor cores.
//
// retention.cu walks a portion token by token on the CUDA cores: S_t = d S_(t-1) + k_t v_t^T, o_t = S_t^T q_t.  Here a CTA
// owns (request, head, 64 value columns) and takes 64 tokens at a time in the chunked form of the same sums:
//     A[i][j] = (q_i . k_j) c d^(i-j) for j <= i                  c: the key scale
//     o_i     = d^(i+1) q_i S + sum_j A[i][j] v_j
//     S       = d^n S + sum_j k_j (c d^(n-1-j) v_j)^T             n: tokens of the chunk
// All operands are fp32 (q and k are rotated in fp32, S and A are fp32) and stay so: each is split exactly into three
// bf16 parts x = h + m + l (24 bits), and a product of two split operands is the sum of the six part products down to
// 2^-16 of it (l m, m l and l l lie below fp32's last bit), accumulated in fp32 in TMEM.  What is a bf16 number anyway
// has one part: v (two parts for fp16 values), and the channels of bf16 q and k that are not rotated.  Against 64 bits
// the outputs' relative error is no larger than the recurrence's (tests).
//
// Per chunk (512 threads, one CTA per SM):
//   split q, k, v' = c d^(n-1-j) v into shared memory (128-byte swizzle); fetch the next chunk's raw rows (cp.async)
//   MMA  A~ = Q K^T [64 x 64], O1 = Q S [64 x 64], U = K^T V' [128 x 64]
//   A~ -> decay, mask, split -> shared memory (over Q);   MMA  O2 = A V [64 x 64]
//   S (fp32, 16 values per thread in registers) = d^n S + U -> split -> shared memory;   o = d^(i+1) O1 + O2
// K is stored once: rows of tokens serve Q K^T as K-major and K^T V' as MN-major operand.  Rows past the portion are
// zeros.  What bounds it: the chain of a chunk (split 2800 clk, Q K^T and
// Q S 3600, A 800, A V and the rest 3000), one after another in a CTA that fills an SM.  4 requests, 8192 tokens, 16 heads
// of 128 x 128: 875 us token by token, 265 us here (41 chunks of 6.4 us for the longest request; 256 without the watch for
// values that cannot be split, see rc_watch).
//
// The sums of a portion are cut every 64 tokens from its start, so results depend in their last bits on how a prompt is
// cut into portions (the token-by-token kernel's do not).
#include "common.cuh"
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
};

__device__ __forceinline__ uint32_t rc_off(int row, int c) { return row * 128 + ((c ^ (row & 7)) << 4); }

// x = h + m + l in bf16 (exact to 24 bits), two numbers at a time
__device__ __forceinline__ void rc_split2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack2<__nv_bfloat16>(x0, x1);
  float2 f = unpack2<__nv_bfloat16>(h);
  x0 -= f.x;
  x1 -= f.y;
  m = pack2<__nv_bfloat16>(x0, x1);
  f = unpack2<__nv_bfloat16>(m);
  l = pack2<__nv_bfloat16>(x0 - f.x, x1 - f.y);
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

// one warp polls, the others wait at a barrier
__device__ __forceinline__ void rc_wait(uint64_t* bar, uint32_t parity, int warp, volatile int* dead) {
  if (warp == 0) mbar_wait_bounded(bar, parity, dead);
  asm volatile("bar.sync 1, %0;" ::"n"(kRcThreads) : "memory");
}

// Tokens t0 .. n - 1 of a portion one after another on the CUDA cores, as retention.cu takes them.  f: 96 KB for [64][128]
// rotated q, rotated and scaled k, [64][64] v and [2][4][64] partial sums; state: this thread's 16 values.  Behind the
// chunks' loop and not inside it: there the call (never made) took 40 us of 256.
template <typename T>
__device__ __forceinline__ void rc_token_by_token(const RetChunkParams* p, int t0, int n, int64_t pos0, int64_t row0, float* f,
                                               float* state, float dec) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, half = p->rot >> 1, h = blockIdx.y;
  const int sr = (warp & 3) * 32 + lane, sc = (warp >> 2) * 16, col0 = blockIdx.z * kRcDv;
  float *fq = f, *fk = fq + kRcTok * kRcDk, *fv = fk + kRcTok * kRcDk, *part = fv + kRcTok * kRcDv;
  float S[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) S[i] = state[i];
#pragma unroll 1
  for (; t0 < n; t0 += kRcTok) {
    const int nt = min(kRcTok, n - t0);
    __syncthreads();  // what stood in `f` has been read
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
    __syncthreads();
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
      __syncthreads();
      if (tid < kRcDv)
        p->o[((row0 + t0 + t) * p->H + h) * static_cast<int64_t>(p->dv) + col0 + tid] =
            (to[tid] + to[kRcDv + tid]) + (to[2 * kRcDv + tid] + to[3 * kRcDv + tid]);
    }
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) state[i] = S[i];
}

// parts (a, b) of the six products, smallest first
__host__ __device__ constexpr int rc_pa(int i) { return (0x001102 >> (4 * i)) & 15; }  // 2 0 1 1 0 0
__host__ __device__ constexpr int rc_pb(int i) { return (0x010120 >> (4 * i)) & 15; }  // 0 2 1 0 1 0

template <typename T, int VS>  // VS: bf16 parts of a value as it is stored (1: bf16, 2: fp16)
__global__ void __launch_bounds__(kRcThreads, 1)
retention_chunked_kernel(const __grid_constant__ RetChunkParams p) {
  extern __shared__ uint8_t rc_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(rc_smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;               // 3 parts; A's three parts once Q has been read
  uint8_t* sK = sQ + 3 * kRcQ;      // 3 parts
  uint8_t* sS = sK + 3 * kRcQ;      // 3 parts
  uint8_t* sW = sS + 3 * kRcS;      // 3 parts of v'
  uint8_t* sV = sW + 3 * kRcV;      // VS parts of v
  T* rq = reinterpret_cast<T*>(sV + VS * kRcV);  // raw rows of the next chunk: q, k [64][128], v [64][64]
  T* rk = rq + kRcTok * kRcDk;
  T* rv = rk + kRcTok * kRcDk;
  uint8_t* misc = reinterpret_cast<uint8_t*>(rv + kRcTok * kRcDv);
  uint64_t* bars = reinterpret_cast<uint64_t*>(misc);  // A~ and O1 / U / O2 complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* pw = reinterpret_cast<float*>(misc + 64);  // [65] powers of the decay

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * kRcDv;
  const int n = p.extend_lens[r];
  const int64_t pos0 = p.prefix_lens[r], row0 = p.extend_start_loc[r];
  if (n <= 0 || pos0 < 0) return;
  if (warp == 0) {
    if (lane == 0) {
      for (int i = 0; i < 3; ++i) mbar_init(&bars[i], 1);
      *dead = 0;
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  if (tid <= kRcTok) {  // d^tid in double, rounded once
    double b = static_cast<double>(p.decay[h]), x = 1.0;
    for (int e = tid; e > 0; e >>= 1) {
      if (e & 1) x *= b;
      b *= b;
    }
    pw[tid] = static_cast<float>(x);
  }
  const T* qg = reinterpret_cast<const T*>(p.q) + static_cast<int64_t>(h) * kRcDk;
  const T* kg = reinterpret_cast<const T*>(p.k) + static_cast<int64_t>(h) * kRcDk;
  const T* vg = reinterpret_cast<const T*>(p.v) + static_cast<int64_t>(h) * p.dv + col0;
  auto fetch = [&](int t0) {  // raw rows t0 .. t0 + 63, zeros past the portion
    for (int i = tid; i < kRcTok * 16; i += kRcThreads) {
      const int t = i >> 4, ch = i & 15;
      const bool ok = t0 + t < n;
      const int64_t row = row0 + (ok ? t0 + t : 0);
      cp_async16(smem_u32(rq + t * kRcDk + ch * 8), qg + row * p.q_stride + ch * 8, ok);
      cp_async16(smem_u32(rk + t * kRcDk + ch * 8), kg + row * p.k_stride + ch * 8, ok);
    }
    for (int i = tid; i < kRcTok * 8; i += kRcThreads) {
      const int t = i >> 3, ch = i & 7;
      const bool ok = t0 + t < n;
      cp_async16(smem_u32(rv + t * kRcDv + ch * 8), vg + (row0 + (ok ? t0 + t : 0)) * p.v_stride + ch * 8, ok);
    }
    cp_async_commit();
  };
  fetch(0);

  // this thread's piece of the state: channel sr, value columns sc .. sc + 15
  const int sr = (warp & 3) * 32 + lane, sc = (warp >> 2) * 16;
  float* st = p.state + (p.req_pool_indices[r] * p.H + h) * static_cast<int64_t>(kRcDk) * p.dv +
              static_cast<int64_t>(sr) * p.dv + col0 + sc;
  float S[16];
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    const float4 x = pos0 > 0 ? *reinterpret_cast<const float4*>(st + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    S[i] = x.x; S[i + 1] = x.y; S[i + 2] = x.z; S[i + 3] = x.w;
  }
  // the same watch over the state a portion starts from; what inputs below 2^32 add to it stays far from fp32's end
  bool odd_state = false;
#pragma unroll
  for (int i = 0; i < 16; ++i) odd_state |= !(fabsf(S[i]) <= 0x1p64f);
  auto put_state = [&]() {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = S[8 * c + e];
      rc_split8(x, sS + rc_off(sr, (sc >> 3) + c), kRcS);
    }
  };
  put_state();
  const int half = p.rot >> 1;
  const int rot_steps = sizeof(T) == 2 && VS == 1 ? p.rot / 16 : kRcDk / 16;  // k-steps whose q, k need three parts
  const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const int ar = (warp & 3) * 16 + (lane >> 2), ac = (warp >> 2) * 16 + 2 * (lane & 3);  // fragment row (+ 8), column

  // this thread's part of a chunk's preparation: token ut; value columns 8 u ..; key channels d0 .. d0 + 7 and d1 .. d1 + 7,
  // the two halves of a rotation where they are rotated, neighbours elsewhere
  const int ut = tid >> 3, u = tid & 7;
  const int d0 = u * 16 < p.rot ? u * 8 : u * 16, d1 = u * 16 < p.rot ? d0 + half : d0 + 8;
  float cs[8], sn[8];
  auto angles = [&](int t0) {  // cos / sin of this thread's token and channels, loaded a chunk ahead
    if (d0 >= p.rot) return;
    int64_t pos = pos0 + t0 + ut;
    pos = pos < p.max_positions ? pos : p.max_positions - 1;
    const float4* cp = reinterpret_cast<const float4*>(p.cos_sin + pos * p.rot + d0);
    const float4* sp = reinterpret_cast<const float4*>(p.cos_sin + pos * p.rot + half + d0);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float4 a = __ldg(cp + e), b = __ldg(sp + e);
      cs[4 * e] = a.x; cs[4 * e + 1] = a.y; cs[4 * e + 2] = a.z; cs[4 * e + 3] = a.w;
      sn[4 * e] = b.x; sn[4 * e + 1] = b.y; sn[4 * e + 2] = b.z; sn[4 * e + 3] = b.w;
    }
  };
  angles(0);
  auto store_state = [&]() {
#pragma unroll
    for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(st + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
  };
  int t_odd = n;
  uint32_t par = 0;
  for (int t0 = 0; t0 < n; t0 += kRcTok, par ^= 1) {
    const int nt = min(kRcTok, n - t0);
    cp_async_wait<0>();
    tc_fence_before_sync();
    __syncthreads();  // raw rows visible; the previous chunk's operands and accumulators have been read
    uint32_t z = 0;
    {
      // ---- q, k: rotate, split: 16 channels of a token and of each ----
      const bool live = ut < nt;
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const T* raw = (w ? rk : rq) + ut * kRcDk;
        float x[8], y[8];
        rc_load8<T>(raw + d0, x);
        rc_load8<T>(raw + d1, y);
        if (d0 < p.rot) {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float a = x[e], b = y[e];
            x[e] = a * cs[e] - b * sn[e];
            y[e] = b * cs[e] + a * sn[e];
          }
        }
        if (!live) {
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = y[e] = 0.f;
        }
        uint8_t* dst = w ? sK : sQ;
        const RcUpper hx = rc_split8(x, dst + (d0 >> 6) * kRcV + rc_off(ut, (d0 >> 3) & 7), kRcQ);
        const RcUpper hy = rc_split8(y, dst + (d1 >> 6) * kRcV + rc_off(ut, (d1 >> 3) & 7), kRcQ);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          rc_watch(hx.h[e], z);
          rc_watch(hy.h[e], z);
        }
      }
      // ---- v, v' ----
      {
        float v8[8];
        rc_load8<T>(rv + ut * kRcDv + u * 8, v8);
        if (!live) {
#pragma unroll
          for (int e = 0; e < 8; ++e) v8[e] = 0.f;
        }
        const uint32_t off = rc_off(ut, u);
        uint32_t hh[4], mm[4], ll;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          rc_split2(v8[2 * e], v8[2 * e + 1], hh[e], mm[e], ll);
          rc_watch(hh[e], z);
        }
        *reinterpret_cast<uint4*>(sV + off) = make_uint4(hh[0], hh[1], hh[2], hh[3]);
        if constexpr (VS == 2) *reinterpret_cast<uint4*>(sV + kRcV + off) = make_uint4(mm[0], mm[1], mm[2], mm[3]);
        const float f = pw[max(nt - 1 - ut, 0)] * p.k_scale;
#pragma unroll
        for (int e = 0; e < 8; ++e) v8[e] *= f;
        rc_split8(v8, sW + off, kRcV);
      }
    }
    fence_proxy_async_smem();
    // the first chunk with a value that has no parts: it and what follows are done again, from this state, behind the loop
    if (__syncthreads_or(rc_spoilt(z) || odd_state) && t0 < t_odd) {
      t_odd = t0;
      store_state();
    }
    tc_fence_after_sync();
    const uint32_t tm = *tmem_slot;
    const uint32_t tA = tm, tO1 = tm + 64, tO2 = tm + 128, tU = tm + 192;
    // descriptors' lower halves (they move by 16-byte units); the upper half is the same for all
    const uint64_t dq = umma_desc_sw128(smem_u32(sQ), 16, 1024);
    const uint32_t hi = static_cast<uint32_t>(dq >> 32), q_lo = static_cast<uint32_t>(dq);
    if (warp == 0 && elect_one()) {
      constexpr uint32_t id_qk = umma_idesc<__nv_bfloat16>(64, 64, 0, 0);
      constexpr uint32_t id_kv = umma_idesc<__nv_bfloat16>(128, 64, 1, 1);
      constexpr uint32_t id_qs = umma_idesc<__nv_bfloat16>(64, 64, 0, 1);
      const uint32_t k_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sK), 16, 1024));
      const uint32_t s_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sS), 16, 1024));
      // everything but the number of rotated steps is known at compile time: an addition or two per MMA
      uint32_t acc = 0;
#pragma unroll
      for (int pr = 0; pr < 6; ++pr)
#pragma unroll
        for (int s = 0; s < kRcDk / 16; ++s)
          if (pr == 5 || s < rot_steps) {
            const uint32_t at = (s >> 2) * (kRcV >> 4) + (s & 3) * 2;
            umma_ss_lo(tA, q_lo + rc_pa(pr) * (kRcQ >> 4) + at, k_lo + rc_pb(pr) * (kRcQ >> 4) + at, hi, id_qk, acc);
            acc = 1;
          }
      acc = 0;
#pragma unroll
      for (int pr = 0; pr < 6; ++pr)
#pragma unroll
        for (int s = 0; s < kRcDk / 16; ++s)
          if (rc_pa(pr) == 0 || s < rot_steps) {
            umma_ss_lo(tO1, q_lo + rc_pa(pr) * (kRcQ >> 4) + (s >> 2) * (kRcV >> 4) + (s & 3) * 2,
                       s_lo + rc_pb(pr) * (kRcS >> 4) + s * 128, hi, id_qs, acc);
            acc = 1;
          }
      umma_commit(&bars[0]);
      const uint32_t km_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sK), kRcV, 1024));
      const uint32_t w_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sW), 16, 1024));
#pragma unroll
      for (int pr = 0; pr < 6; ++pr) {
        const uint32_t a = km_lo + rc_pa(pr) * (kRcQ >> 4), b = w_lo + rc_pb(pr) * (kRcV >> 4);
#pragma unroll
        for (int s = 0; s < kRcTok / 16; ++s) umma_ss_lo(tU, a + s * 128, b + s * 128, hi, id_kv, (pr | s) ? 1u : 0u);
      }
      umma_commit(&bars[1]);
    }
    __syncwarp();
    if (t0 + nt < n) {
      fetch(t0 + nt);
      angles(t0 + nt);
    }
    // ---- A: decay, mask, split (over Q, which the MMAs have read) ----
    mbar_wait_bounded(&bars[0], par, dead);  // (by every warp: warp 0 is still handing in U's MMAs)
    tc_fence_after_sync();
    {
      uint32_t a[8];
      rc_ld_frag(tA + lane_base + (warp >> 2) * 16, a);
      tmem_ld_wait();
#pragma unroll
      for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int i = ar + 8 * x, j = ac + 8 * g;
          const float a0 = j <= i ? __uint_as_float(a[4 * g + 2 * x]) * (pw[max(i - j, 0)] * p.k_scale) : 0.f;
          const float a1 = j < i ? __uint_as_float(a[4 * g + 2 * x + 1]) * (pw[max(i - j - 1, 0)] * p.k_scale) : 0.f;
          uint32_t hh, mm, ll;
          rc_split2(a0, a1, hh, mm, ll);
          uint8_t* dst = sQ + rc_off(i, j >> 3) + (j & 7) * 2;
          *reinterpret_cast<uint32_t*>(dst) = hh;
          *reinterpret_cast<uint32_t*>(dst + kRcV) = mm;
          *reinterpret_cast<uint32_t*>(dst + 2 * kRcV) = ll;
        }
    }
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 0 && elect_one()) {
      constexpr uint32_t id_av = umma_idesc<__nv_bfloat16>(64, 64, 0, 1);
      const uint32_t v_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sV), 16, 1024));
      uint32_t acc = 0;
#pragma unroll
      for (int pr = 0; pr < 6; ++pr) {
        if (rc_pb(pr) >= VS) continue;
        const uint32_t a = q_lo + rc_pa(pr) * (kRcV >> 4), b = v_lo + rc_pb(pr) * (kRcV >> 4);
#pragma unroll
        for (int s = 0; s < kRcTok / 16; ++s) {
          umma_ss_lo(tO2, a + s * 2, b + s * 128, hi, id_av, acc);
          acc = 1;
        }
      }
      umma_commit(&bars[2]);
    }
    __syncwarp();
    // ---- state ----
    rc_wait(&bars[1], par, warp, dead);
    tc_fence_after_sync();
    {
      uint32_t x[16];
      tmem_ld_32x32b_x16(tU + lane_base + sc, x);
      tmem_ld_wait();
      const float dn = pw[nt];
#pragma unroll
      for (int i = 0; i < 16; ++i) S[i] = fmaf(dn, S[i], __uint_as_float(x[i]));
    }
    if (t0 + nt < n) put_state();
    // ---- outputs ----
    rc_wait(&bars[2], par, warp, dead);
    tc_fence_after_sync();
    {
      uint32_t a[8], b[8];
      rc_ld_frag(tO1 + lane_base + (warp >> 2) * 16, a);
      rc_ld_frag(tO2 + lane_base + (warp >> 2) * 16, b);
      tmem_ld_wait();
      float* og = p.o + ((row0 + t0) * p.H + h) * static_cast<int64_t>(p.dv) + col0;
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int i = ar + 8 * x;
        if (i < nt) {
          const float f = pw[i + 1];
          float* dst = og + static_cast<int64_t>(i) * p.H * p.dv + ac;
#pragma unroll
          for (int g = 0; g < 2; ++g)
            *reinterpret_cast<float2*>(dst + 8 * g) =
                make_float2(fmaf(f, __uint_as_float(a[4 * g + 2 * x]), __uint_as_float(b[4 * g + 2 * x])),
                            fmaf(f, __uint_as_float(a[4 * g + 2 * x + 1]), __uint_as_float(b[4 * g + 2 * x + 1])));
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*dead) {  // the request keeps the state it had (or, stored above, had at its first token without parts)
    wait_drain();
    if (tid == 0) wait_report(p.wait_expired);
  } else if (t_odd < n) {
    rc_token_by_token<T>(&p, t_odd, n, pos0, row0, reinterpret_cast<float*>(sQ), st, pw[1]);
  } else {
    store_state();
  }
  __syncthreads();
  if (warp == 0) tmem_dealloc(*tmem_slot, 256);
}

template <typename T, int VS>
static int rc_launch(const RetChunkParams& p, int64_t batch, cudaStream_t stream) {
  constexpr int smem = 6 * kRcQ + 3 * kRcS + (3 + VS) * kRcV + (2 * kRcTok * kRcDk + kRcTok * kRcDv) * 2 + kRcMisc + 1024;
  static_assert(smem <= 232448, "does not fit an SM");
  auto kern = retention_chunked_kernel<T, VS>;
  static bool configured = false;  // per instantiation
  if (!configured) {
    SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured = true;
  }
  SPD_CUDA(launch(kern, dim3((unsigned)batch, (unsigned)p.H, (unsigned)(p.dv / kRcDv)), dim3(kRcThreads), smem, stream,
                  /*pdl=*/false, p));
  return 0;
}

// → 0 launched, 1 not applicable (the caller takes the token-by-token kernel), else an error
int retention_chunked_try(float* o, const void* q, const void* k, const void* v, float* state,
                          const int64_t* req_pool_indices, const int32_t* prefix_lens, const int32_t* extend_lens,
                          const int32_t* extend_start_loc, int64_t batch, int H, int dk, int dv, int64_t q_stride,
                          int64_t k_stride, int64_t v_stride, const float* decay, const float* cos_sin, int rot,
                          int64_t max_positions, float k_scale, int in_act, int dtype, int64_t total_tokens,
                          cudaStream_t stream) {
  // A chunk costs what some tens of tokens cost one by one, and its CTA takes a whole SM: 4 requests of 16 tokens 12.1 us
  // (token by token) / 11.8, of 64 tokens 32.9 / 17.6; 16 requests of 16 tokens 30 / 41 us, of 40 tokens 63 / 41.
  if (total_tokens <= 40 * batch) return 1;
  // 16-bit rows without an activation (their parts are what the split was counted for), 128 channels, whole 64-column
  // slices, a rotation in whole 16-byte pieces, 16-byte rows
  if (dtype == SPD_F32 || in_act != 0 || dk != kRcDk || dv % kRcDv != 0 || rot % 16 != 0) return 1;
  if (H > 65535 || dv / kRcDv > 65535) return 1;
  if (q_stride % 8 != 0 || k_stride % 8 != 0 || v_stride % 8 != 0 || !aligned16(q) || !aligned16(k) || !aligned16(v) ||
      !aligned16(o) || !aligned16(state) || (rot > 0 && !aligned16(cos_sin)))
    return 1;
  unsigned* wait_expired;
  if (int rc = wait_flag(&wait_expired)) return rc;
  const RetChunkParams p{o, q, k, v, state, req_pool_indices, prefix_lens, extend_lens, extend_start_loc, H, dv, rot,
                         q_stride, k_stride, v_stride, max_positions, decay, cos_sin, k_scale, wait_expired};
  return dtype == SPD_BF16 ? rc_launch<__nv_bfloat16, 1>(p, batch, stream) : rc_launch<__half, 2>(p, batch, stream);
}

}  // namespace spd
