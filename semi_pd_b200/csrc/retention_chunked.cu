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
// Per chunk (512 threads, one CTA per SM); S, and q, k, v, v' = c d^(n-1-j) v of the chunk stand split in shared memory
// (128-byte swizzle):
//   MMA  A~ = Q K^T [64 x 64], U = K^T V' [128 x 64], O1 = Q S [64 x 64]; fetch the next chunk's raw rows (cp.async)
//   S (fp32, 16 values per thread in registers) = d^n S + U;   A~ -> decay, mask, split -> over V'
//   MMA  O2 = A V [64 x 64];   S -> split -> shared memory;   the next chunk's q, k -> rotate, split
//   o = d^(i+1) O1 + O2;   the next chunk's v -> split
// K is stored once: rows of tokens serve Q K^T as K-major and K^T V' as MN-major operand.  Rows past the portion are
// zeros.  What bounds it: shared memory, 700 KB of operands and splits per chunk (5500 clk at 128 bytes a clk), and phases of
// MMAs (5500 clk) and of splitting (4900) that mostly follow one another.  4 requests, 8192 tokens, 16 heads of 128 x 128:
// 875 us token by token, 241 us here (41 chunks of 5.6 us for the longest request; 264 with the MMAs handed in by one lane
// from unrolled code, all warps polling, and a thread's rotated channels mixed with others in its warp).
//
// Long portions of few requests are cut into segments that run side by side (retention_sums_kernel, rc_seg_tokens): one
// request of 8000 tokens 728 -> 260 us.
//
// The sums of a portion are cut every 64 tokens from its start (and at segments), so results depend in their last bits on how a prompt is
// cut into portions (the token-by-token kernel's do not).
#include "retention_parts.cuh"

namespace spd {

// VS: bf16 parts of a value as it is stored (1: bf16, 2: fp16); kCut: portions in segments
template <typename T, int VS, bool kCut>
__global__ void __launch_bounds__(kRcThreads, 1)
retention_chunked_kernel(const __grid_constant__ RetChunkParams p) {
  extern __shared__ uint8_t rc_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(rc_smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;               // 3 parts
  uint8_t* sK = sQ + 3 * kRcQ;      // 3 parts
  uint8_t* sS = sK + 3 * kRcQ;      // 3 parts
  uint8_t* sW = sS + 3 * kRcS;      // 3 parts of v'; A's three parts once K^T V' has been read
  uint8_t* sV = sW + 3 * kRcV;      // VS parts of v
  T* rq = reinterpret_cast<T*>(sV + VS * kRcV);  // raw rows of the next chunk: q, k [64][128], v [64][64]
  T* rk = rq + kRcTok * kRcDk;
  T* rv = rk + kRcTok * kRcDk;
  uint8_t* misc = reinterpret_cast<uint8_t*>(rv + kRcTok * kRcDv);
  uint64_t* bars = reinterpret_cast<uint64_t*>(misc);  // A~ and O1 / U / O2 complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* pw = reinterpret_cast<float*>(misc + 64);  // [65] powers of the decay

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const bool leader = elect_one();
  const int h = blockIdx.y, col0 = blockIdx.z * kRcDv;
  RcSegment sg{static_cast<int>(blockIdx.x), 0, 1, 0};
  if constexpr (kCut) {
    if (!rc_segment(p, blockIdx.x, sg)) return;
  }
  const int r = sg.r, n_all = p.extend_lens[r];
  const int64_t pos0 = p.prefix_lens[r], row0 = p.extend_start_loc[r];
  if (n_all <= 0 || pos0 < 0) return;
  // this CTA's tokens: its segment, or all that follows from the first segment on whose k or v have no parts (later segments'
  // starting states do not exist then; they leave)
  const int begin = kCut ? sg.seg * p.seg_tokens : 0;
  bool last = !kCut || sg.seg == sg.nseg - 1;
  int n = last ? n_all : begin + p.seg_tokens;
  const int64_t per_seg = static_cast<int64_t>(p.H) * (p.dv / kRcDv) * kRcDk * kRcDv;  // floats of a segment in p.sums
  const int64_t own = (static_cast<int64_t>(h) * (p.dv / kRcDv) + blockIdx.z) * kRcDk * kRcDv;
  if (kCut && sg.nseg > 1) {
    int worst = 0, odd = sg.nseg;
    for (int i = lane; i < sg.nseg - 1; i += 32) {
      const int f = p.flags[((sg.first + i) * static_cast<int64_t>(p.H) + h) * (p.dv / p.flag_cols) + col0 / p.flag_cols];
      worst = max(worst, f);
      if (f == 1) odd = min(odd, i);
    }
    worst = __reduce_max_sync(0xffffffffu, worst);
    odd = __reduce_min_sync(0xffffffffu, odd);
    if (worst == 2 || sg.seg > odd) return;
    if (sg.seg == odd) {
      n = n_all;
      last = true;
    }
  }
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
    if (warp == 0) return;  // it hands in the MMAs
    for (int i = tid - 32; i < kRcTok * 16; i += kRcThreads - 32) {
      const int t = i >> 4, ch = i & 15;
      const bool ok = t0 + t < n;
      const int64_t row = row0 + (ok ? t0 + t : 0);
      cp_async16(smem_u32(rq) + rc_raw(t, ch), qg + row * p.q_stride + ch * 8, ok);
      cp_async16(smem_u32(rk) + rc_raw(t, ch), kg + row * p.k_stride + ch * 8, ok);
    }
    for (int i = tid - 32; i < kRcTok * 8; i += kRcThreads - 32) {
      const int t = i >> 3, ch = i & 7;
      const bool ok = t0 + t < n;
      cp_async16(smem_u32(rv + t * kRcDv + ch * 8), vg + (row0 + (ok ? t0 + t : 0)) * p.v_stride + ch * 8, ok);
    }
    cp_async_commit();
  };
  fetch(begin);

  // what the first chunk needs besides its rows, before anything waits for the state: what a CTA does before its first MMA
  // counts for short portions and for every wave of segments (60 tokens 12.9 us with the angles requested after the state had
  // arrived, 12.5 here; 8000 tokens of 4 heads in segments of two chunks 116, 82)
  const int half = p.rot >> 1;
  const int rot_steps = sizeof(T) == 2 && VS == 1 ? p.rot / 16 : kRcDk / 16;  // k-steps whose q, k need three parts
  const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const int ar = (warp & 3) * 16 + (lane >> 2), ac = (warp >> 2) * 16 + 2 * (lane & 3);  // fragment row (+ 8), column

  // this thread's part of a chunk's preparation: token t, eight pairs (8 g .., 8 g + half ..) of q or k where they are rotated
  // (of both, where more than 64 channels are), pieces of eight channels of what is not rotated, value columns 8 u ..
  const int t = tid & 63, t8 = tid >> 6, ut = tid >> 3, u = tid & 7;
  const int groups = p.rot >> 4;
  const bool both = groups > 4, rotates = t8 < (both ? groups : 2 * groups);
  const int w0 = !both && t8 >= groups ? 1 : 0, d0 = 8 * (t8 - w0 * groups), d1 = d0 + half;
  const int plain = (kRcDk - p.rot) >> 3;  // pieces of a row that are not rotated
  float cs[8], sn[8];
  auto angles = [&](int t0) {  // cos / sin of this thread's token and channels, loaded a chunk ahead; zeros past the portion
    if (!rotates) return;
    int64_t pos = pos0 + t0 + t;
    pos = pos < p.max_positions ? pos : p.max_positions - 1;
    const bool live = t0 + t < n;
    const float4* cp = reinterpret_cast<const float4*>(p.cos_sin + pos * p.rot + d0);
    const float4* sp = reinterpret_cast<const float4*>(p.cos_sin + pos * p.rot + half + d0);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), a = live ? __ldg(cp + e) : zero, b = live ? __ldg(sp + e) : zero;
      cs[4 * e] = a.x; cs[4 * e + 1] = a.y; cs[4 * e + 2] = a.z; cs[4 * e + 3] = a.w;
      sn[4 * e] = b.x; sn[4 * e + 1] = b.y; sn[4 * e + 2] = b.z; sn[4 * e + 3] = b.w;
    }
  };
  if constexpr (VS == 1) {
    // bf16 channels that are not rotated have one part: the others' rows in K^T V' are zeros
    for (int i = tid; i < 2 * kRcQ / 16; i += kRcThreads) reinterpret_cast<uint4*>(sK + kRcQ)[i] = make_uint4(0, 0, 0, 0);
  }
  angles(begin);

  // this thread's piece of the state: channel sr, value columns sc .. sc + 15
  const int sr = (warp & 3) * 32 + lane, sc = (warp >> 2) * 16;
  float* st = p.state + (p.req_pool_indices[r] * p.H + h) * static_cast<int64_t>(kRcDk) * p.dv +
              static_cast<int64_t>(sr) * p.dv + col0 + sc;
  float S[16];
  const float* from = kCut && sg.nseg > 1 ? p.sums + (sg.first + sg.nseg - 1) * per_seg + own + sr * kRcDv + sc : st;
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    const float4 x = pos0 > 0 ? *reinterpret_cast<const float4*>(from + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    S[i] = x.x; S[i + 1] = x.y; S[i + 2] = x.z; S[i + 3] = x.w;
  }
  // the same watch over the state a portion starts from; what inputs below 2^32 add to it stays far from fp32's end
  bool odd_state = false;
#pragma unroll
  for (int i = 0; i < 16; ++i) odd_state |= !(fabsf(S[i]) <= 0x1p64f);
  if (kCut && sg.nseg > 1) {
    if (__syncthreads_or(odd_state)) {  // the first segment's CTA takes the portion token by token
      if (sg.seg > 0) n = 0;
      else n = n_all;
      last = true;
    } else if (sg.seg > 0) {
      const float* start = p.sums + (sg.first + sg.seg - 1) * per_seg + own + sr * kRcDv + sc;
#pragma unroll
      for (int c = 0; c < 16; c += 4) {
        const float4 x = *reinterpret_cast<const float4*>(start + c);
        S[c] = x.x; S[c + 1] = x.y; S[c + 2] = x.z; S[c + 3] = x.w;
      }
    }
  }
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
  cp_async_wait<0>();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  auto store_state = [&](float* to) {
#pragma unroll
    for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(to + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
  };
  float* keep = kCut && sg.nseg > 1 ? p.keep + blockIdx.x * per_seg + own + tid * 16 : st;
  // the two halves of a chunk's preparation: q and k (their memory is free once Q K^T, Q S and K^T V' are done), v and v'
  // (once A V is, whose A lies over v')
  auto split_qk = [&](uint32_t& z) {
    // ---- q, k: rotate, split ----
    if (rotates) {
#pragma unroll 1
      for (int w = w0; w <= (both ? 1 : w0); ++w) {
        const uint8_t* raw = reinterpret_cast<const uint8_t*>(w ? rk : rq);
        float x[8], y[8];
        rc_load8<T>(reinterpret_cast<const T*>(raw + rc_raw(t, d0 >> 3)), x);
        rc_load8<T>(reinterpret_cast<const T*>(raw + rc_raw(t, d1 >> 3)), y);
#pragma unroll
        for (int e = 0; e < 8; e += 2) {  // rows past the portion are zeros already
          const uint64_t a = pack_f32x2(x[e], x[e + 1]), b = pack_f32x2(y[e], y[e + 1]);
          const uint64_t c2 = pack_f32x2(cs[e], cs[e + 1]), s2 = pack_f32x2(sn[e], sn[e + 1]);
          unpack_f32x2(ffma2(a, c2, fmul2(b, pack_f32x2(-sn[e], -sn[e + 1]))), x[e], x[e + 1]);
          unpack_f32x2(ffma2(b, c2, fmul2(a, s2)), y[e], y[e + 1]);
        }
        uint8_t* dst = w ? sK : sQ;
        const RcUpper hx = rc_split8(x, dst + (d0 >> 6) * kRcV + rc_off(t, (d0 >> 3) & 7), kRcQ);
        const RcUpper hy = rc_split8(y, dst + (d1 >> 6) * kRcV + rc_off(t, (d1 >> 3) & 7), kRcQ);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          rc_watch(hx.h[e], z);
          rc_watch(hy.h[e], z);
        }
      }
    }
    for (int i = t8; i < 2 * plain; i += kRcThreads / 64) {
      const int w = i >= plain ? 1 : 0, c = (p.rot >> 3) + i - w * plain;
      const uint8_t* raw = reinterpret_cast<const uint8_t*>(w ? rk : rq) + rc_raw(t, c);
      uint8_t* dst = (w ? sK : sQ) + (c >> 3) * kRcV + rc_off(t, c & 7);
      if constexpr (VS == 1) {  // (rows past the portion are zeros already)
        const uint4 x = *reinterpret_cast<const uint4*>(raw);
        *reinterpret_cast<uint4*>(dst) = x;
        rc_watch(x.x, z);
        rc_watch(x.y, z);
        rc_watch(x.z, z);
        rc_watch(x.w, z);
      } else {
        float x[8];
        rc_load8<T>(reinterpret_cast<const T*>(raw), x);
        const RcUpper hx = rc_split8(x, dst, kRcQ);
#pragma unroll
        for (int e = 0; e < 4; ++e) rc_watch(hx.h[e], z);
      }
    }
  };
  auto split_v = [&](int nt, uint32_t& z) {
    {
      float v8[8];
      rc_load8<T>(rv + ut * kRcDv + u * 8, v8);
      if (ut >= nt) {
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
  };
  const uint32_t tm = *tmem_slot;
  const uint32_t tA = tm, tO1 = tm + 64, tO2 = tm + 128, tU = tm + 192;
  // descriptors' lower halves (they move by 16-byte units); the upper half is the same for all
  const uint64_t dq = umma_desc_sw128(smem_u32(sQ), 16, 1024);
  const uint32_t hi = static_cast<uint32_t>(dq >> 32), q_lo = static_cast<uint32_t>(dq);
  int t_odd = n;
  uint32_t par = 0, z = 0;
  split_qk(z);
  split_v(min(kRcTok, n - begin), z);
  for (int t0 = begin; t0 < n; t0 += kRcTok, par ^= 1) {
    const int nt = min(kRcTok, n - t0), next = min(kRcTok, n - t0 - nt);  // tokens of this chunk and of the next
    fence_proxy_async_smem();
    tc_fence_before_sync();
    // the first chunk with a value that has no parts: it and what follows are done again, from this state, behind the loop
    if (__syncthreads_or(rc_spoilt(z) || odd_state) && t0 < t_odd) {
      t_odd = t0;
      store_state(keep);
    }
    tc_fence_after_sync();
    if (warp == 0) {
      // The whole warp computes the operands, one lane issues; short loops.  (Unrolled from one lane: 56 clk per MMA where
      // the tensor core takes 31.)  Q S goes last: the state's update and A's decay and split run under it.
      constexpr uint32_t id_qk = umma_idesc<__nv_bfloat16>(64, 64, 0, 0);
      constexpr uint32_t id_kv = umma_idesc<__nv_bfloat16>(128, 64, 1, 1);
      constexpr uint32_t id_qs = umma_idesc<__nv_bfloat16>(64, 64, 0, 1);
      const uint32_t k_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sK), 16, 1024));
      const uint32_t s_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sS), 16, 1024));
      uint32_t acc = 0;
#pragma unroll 1
      for (int pr = 0; pr < 6; ++pr) {
        uint32_t a = q_lo + rc_pa(pr) * (kRcQ >> 4), b = k_lo + rc_pb(pr) * (kRcQ >> 4);
        const int steps = pr == 5 ? kRcDk / 16 : rot_steps;
#pragma unroll 1
        for (int s = 0; s < steps; s += 4) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            umma_ss_if(leader && s + e < steps, tA, a + e * 2, b + e * 2, hi, id_qk, acc);
            acc = 1;
          }
          a += kRcV >> 4;
          b += kRcV >> 4;
        }
      }
      const uint32_t km_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sK), kRcV, 1024));
      const uint32_t w_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sW), 16, 1024));
      acc = 0;
#pragma unroll 1
      for (int pr = 0; pr < 6; ++pr) {
        const uint32_t a = km_lo + rc_pa(pr) * (kRcQ >> 4), b = w_lo + rc_pb(pr) * (kRcV >> 4);
#pragma unroll
        for (int s = 0; s < kRcTok / 16; ++s) {
          umma_ss_if(leader, tU, a + s * 128, b + s * 128, hi, id_kv, acc);
          acc = 1;
        }
      }
      umma_commit_if(leader, &bars[1]);
      acc = 0;
#pragma unroll 1
      for (int pr = 0; pr < 6; ++pr) {
        uint32_t a = q_lo + rc_pa(pr) * (kRcQ >> 4), b = s_lo + rc_pb(pr) * (kRcS >> 4);
        const int steps = rc_pa(pr) == 0 ? kRcDk / 16 : rot_steps;
#pragma unroll 1
        for (int s = 0; s < steps; s += 4) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            umma_ss_if(leader && s + e < steps, tO1, a + e * 2, b + e * 128, hi, id_qs, acc);
            acc = 1;
          }
          a += kRcV >> 4;
          b += 512;
        }
      }
      umma_commit_if(leader, &bars[0]);
    }
    __syncwarp();
    if (next > 0) {
      fetch(t0 + nt);
      angles(t0 + nt);
    }
    // ---- state ----
    rc_wait(&bars[1], par, warp, dead);  // (by every warp: warp 0 is still handing in Q S)
    tc_fence_after_sync();
    {
      uint32_t x[16];
      tmem_ld_32x32b_x16(tU + lane_base + sc, x);
      tmem_ld_wait();
      const float dn = pw[nt];
#pragma unroll
      for (int i = 0; i < 16; ++i) S[i] = fmaf(dn, S[i], __uint_as_float(x[i]));
    }
    // ---- A: decay, mask, split, over v' (rows 0 - 15 have columns 0 - 15 only: warp 4 takes them, warp 0 has been busy) ----
    if (warp != 0) {
      const int cg = warp == 4 ? 0 : warp >> 2;
      uint32_t a[8];
      rc_ld_frag(tA + lane_base + cg * 16, a);
      tmem_ld_wait();
#pragma unroll
      for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int i = ar + 8 * x, j = cg * 16 + 2 * (lane & 3) + 8 * g;
          const float a0 = j <= i ? __uint_as_float(a[4 * g + 2 * x]) * (pw[max(i - j, 0)] * p.k_scale) : 0.f;
          const float a1 = j < i ? __uint_as_float(a[4 * g + 2 * x + 1]) * (pw[max(i - j - 1, 0)] * p.k_scale) : 0.f;
          uint32_t hh, mm, ll;
          rc_split2(a0, a1, hh, mm, ll);
          uint8_t* dst = sW + rc_off(i, j >> 3) + (j & 7) * 2;
          *reinterpret_cast<uint32_t*>(dst) = hh;
          *reinterpret_cast<uint32_t*>(dst + kRcV) = mm;
          *reinterpret_cast<uint32_t*>(dst + 2 * kRcV) = ll;
          if (warp == 4) {  // its own columns 16 - 31
            uint8_t* zero = sW + rc_off(i, (j >> 3) + 2) + (j & 7) * 2;
            *reinterpret_cast<uint32_t*>(zero) = 0;
            *reinterpret_cast<uint32_t*>(zero + kRcV) = 0;
            *reinterpret_cast<uint32_t*>(zero + 2 * kRcV) = 0;
          }
        }
    }
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 0) {
      constexpr uint32_t id_av = umma_idesc<__nv_bfloat16>(64, 64, 0, 1);
      const uint32_t v_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sV), 16, 1024));
      const uint32_t a_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sW), 16, 1024));
      uint32_t acc = 0;
#pragma unroll 1
      for (int pr = 0; pr < 6; ++pr) {
        if (rc_pb(pr) >= VS) continue;
        const uint32_t a = a_lo + rc_pa(pr) * (kRcV >> 4), b = v_lo + rc_pb(pr) * (kRcV >> 4);
#pragma unroll
        for (int s = 0; s < kRcTok / 16; ++s) {
          umma_ss_if(leader, tO2, a + s * 2, b + s * 128, hi, id_av, acc);
          acc = 1;
        }
      }
      umma_commit_if(leader, &bars[2]);
    }
    __syncwarp();
    rc_wait(&bars[0], par, warp, dead);
    z = 0;
    if (next > 0) {
      put_state();
      cp_async_wait<0>();
      __syncthreads();  // the next chunk's raw rows are there
      split_qk(z);
    }
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
    if (next > 0) split_v(next, z);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*dead) {  // the request keeps the state it had (or, stored above, had at its first token without parts)
    wait_drain();
    if (tid == 0) wait_report(p.wait_expired);
  } else if (t_odd < n) {
    rc_token_by_token<T>(&p, t_odd, n, pos0, row0, reinterpret_cast<float*>(sQ), keep, last ? st : nullptr, pw[1], h, col0);
  } else if (last && n > 0) {
    store_state(st);
  }
  __syncthreads();
  if (warp == 0) tmem_dealloc(*tmem_slot, 256);
}

// What the segments of a portion but its last add to the state, [128 x NC] of a head: sum_j c d^(L - 1 - j) k_j v_j^T over the
// segment's L tokens.  With these (retention_scan_kernel), the segments' chunks run at the same time.  Also keeps the state that the portion starts from, which the last segment's CTA will
// overwrite.  Each chunk's products are folded into a second accumulator in fp32, as the chunks' loop does (tensor memory
// sums of a whole segment had four times the error).  256 threads, two CTAs per SM: one splits while the other's MMAs (1540
// clk per chunk at NC = 128, bounded by their operands in shared memory) run.
constexpr int kRsThreads = 256;
template <typename T, int NC>
__global__ void __launch_bounds__(kRsThreads, 2)
retention_sums_kernel(const __grid_constant__ RetChunkParams p) {
  constexpr int kBlocks = NC / 64, kW = kBlocks * kRcV;  // one part of v': [64 x 128 B] blocks of 64 columns
  extern __shared__ uint8_t rc_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(rc_smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem;           // 3 parts
  uint8_t* sW = sK + 3 * kRcQ;  // 3 parts
  uint64_t* bar = reinterpret_cast<uint64_t*>(sW + 3 * kW);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* pw = reinterpret_cast<float*>(bar + 4);  // [65] powers of the decay

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const bool leader = elect_one();
  const int h = blockIdx.y, col0 = blockIdx.z * NC;
  RcSegment sg;
  if (!rc_segment(p, blockIdx.x, sg) || sg.nseg == 1) return;
  const int64_t pos0 = p.prefix_lens[sg.r], row0 = p.extend_start_loc[sg.r];
  const int64_t blocks = p.dv / kRcDv;
  float* sums = p.sums + ((static_cast<int64_t>(blockIdx.x) * p.H + h) * blocks + col0 / kRcDv) * kRcDk * kRcDv;
  if (sg.seg == sg.nseg - 1) {
    const float* st = p.state + (p.req_pool_indices[sg.r] * p.H + h) * static_cast<int64_t>(kRcDk) * p.dv + col0;
    if (pos0 > 0)
      for (int i = tid; i < kRcDk * NC / 4; i += kRsThreads) {
        const int row = i / (NC / 4), c = i % (NC / 4) * 4;
        *reinterpret_cast<float4*>(sums + ((c >> 6) * kRcDk + row) * kRcDv + (c & 63)) =
            *reinterpret_cast<const float4*>(st + static_cast<int64_t>(row) * p.dv + c);
      }
    return;
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
  if (tid <= kRcTok) {
    double b = static_cast<double>(p.decay[h]), x = 1.0;
    for (int e = tid; e > 0; e >>= 1) {
      if (e & 1) x *= b;
      b *= b;
    }
    pw[tid] = static_cast<float>(x);
  }
  for (int i = tid; i < 3 * kRcQ / 16; i += kRsThreads) reinterpret_cast<uint4*>(sK)[i] = make_uint4(0, 0, 0, 0);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tU = *tmem_slot;

  const T* kg = reinterpret_cast<const T*>(p.k) + row0 * p.k_stride + static_cast<int64_t>(h) * kRcDk;
  const T* vg = reinterpret_cast<const T*>(p.v) + row0 * p.v_stride + static_cast<int64_t>(h) * p.dv + col0;
  const int begin = sg.seg * p.seg_tokens, half = p.rot >> 1, groups = p.rot >> 4;
  // k: eight threads a row, pieces u and u + 8 of rows kt and kt + 32 (whole lines in flight: one row per thread took three
  // times as long); a rotated piece meets its other half by shuffles.  v: rows vt, vt + 256 / (NC / 8) .., columns 8 vc ..
  const int kt = tid >> 3, u = tid & 7;
  const int vt = tid / (NC / 8), vc = tid % (NC / 8);
  constexpr int kVStep = kRsThreads / (NC / 8), kVN = kRcTok / kVStep;
  uint4 rk[2][2], rv[kVN];  // a chunk's rows, read a chunk ahead: [row][piece]
  float4 ang[2][4];         // cos and sin of the rows' pieces u
  // angles of a rotated piece: cos, sin of eight channels
  auto angles = [&](int t0, int row, int piece, float4 (&a)[4]) {
    const int64_t pos = min(pos0 + t0 + kt + 32 * row, p.max_positions - 1);
    const float* cp = p.cos_sin + pos * p.rot + 8 * (piece < groups ? piece : piece - groups);
    a[0] = __ldg(reinterpret_cast<const float4*>(cp));
    a[1] = __ldg(reinterpret_cast<const float4*>(cp) + 1);
    a[2] = __ldg(reinterpret_cast<const float4*>(cp + half));
    a[3] = __ldg(reinterpret_cast<const float4*>(cp + half) + 1);
  };
  auto read = [&](int t0) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint4* kr = reinterpret_cast<const uint4*>(kg + static_cast<int64_t>(t0 + kt + 32 * r) * p.k_stride);
      rk[r][0] = __ldg(kr + u);
      rk[r][1] = __ldg(kr + u + 8);
      if (u < 2 * groups) angles(t0, r, u, ang[r]);
    }
#pragma unroll
    for (int i = 0; i < kVN; ++i)
      rv[i] = __ldg(reinterpret_cast<const uint4*>(vg + static_cast<int64_t>(t0 + vt + i * kVStep) * p.v_stride + vc * 8));
  };
  auto floats = [](const uint4& w, float (&x)[8]) {
    const uint32_t a[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = unpack2<T>(a[e]);
      x[2 * e] = f.x;
      x[2 * e + 1] = f.y;
    }
  };
  read(begin);
  // chunk c has been multiplied: sum = d^64 sum + its products; after the last one to global memory
  uint32_t par = 0;
  auto fold = [&](int c) {
    if (warp == 0) mbar_wait_bounded(bar, par, dead);
    __syncthreads();
    par ^= 1;
    tc_fence_after_sync();
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int row = (warp & 3) * 32 + lane;
    const float dn = pw[kRcTok];
#pragma unroll 1
    for (int col = (warp >> 2) * (NC / 2); col < (warp >> 2) * (NC / 2) + NC / 2; col += 16) {
      uint32_t x[16];
      tmem_ld_32x32b_x16(tU + lane_base + col, x);
      if (c > 0) {
        uint32_t y[16];
        tmem_ld_32x32b_x16(tU + lane_base + NC + col, y);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = __float_as_uint(fmaf(dn, __uint_as_float(y[i]), __uint_as_float(x[i])));
      } else {
        tmem_ld_wait();
      }
      if (c + kRcTok < p.seg_tokens) {
        tmem_st_32x32b_x16(tU + lane_base + NC + col, x);
      } else {
        uint4* dst = reinterpret_cast<uint4*>(sums + ((col >> 6) * kRcDk + row) * kRcDv + (col & 63));
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = make_uint4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
      }
    }
    tmem_st_wait();
    tc_fence_before_sync();
  };
  uint32_t z = 0;
#pragma unroll 1
  for (int c = 0; c < p.seg_tokens; c += kRcTok) {
    const int t0 = begin + c;
    if (c > 0) fold(c - kRcTok);
    // ---- k ----
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int half8 = 0; half8 < 2; ++half8) {
        const int piece = u + 8 * half8, row = kt + 32 * r;
        const bool first = piece < groups, rotated = piece < 2 * groups;
        const uint4 w = rk[r][half8];
        uint4 o = w;  // the piece that it is rotated with: groups further on or back
        if (8 * half8 < 2 * groups) {
          const int with = first ? piece + groups : piece - groups, lane8 = (lane & 24) | (with & 7);
          const bool far = (with & 8) != 0;
          const uint4 &a = rk[r][0], &b = rk[r][1];
          const uint32_t lo[4] = {__shfl_sync(0xffffffffu, a.x, lane8), __shfl_sync(0xffffffffu, a.y, lane8),
                                  __shfl_sync(0xffffffffu, a.z, lane8), __shfl_sync(0xffffffffu, a.w, lane8)};
          o = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          if (groups > 4) {  // pairs reach into the other half of the row
            const uint32_t up[4] = {__shfl_sync(0xffffffffu, b.x, lane8), __shfl_sync(0xffffffffu, b.y, lane8),
                                    __shfl_sync(0xffffffffu, b.z, lane8), __shfl_sync(0xffffffffu, b.w, lane8)};
            if (far) o = make_uint4(up[0], up[1], up[2], up[3]);
          }
        }
        uint8_t* dst = sK + half8 * kRcV + rc_off(row, u);
        if (rotated || umma_fmt<T>::v == 0) {
          float x[8], y[8];
          floats(w, x);
          if (rotated) {
            float4 ca[4];
            if (half8 == 0) {
#pragma unroll
              for (int e = 0; e < 4; ++e) ca[e] = ang[r][e];
            } else {
              angles(t0, r, piece, ca);
            }
            const float cs[8] = {ca[0].x, ca[0].y, ca[0].z, ca[0].w, ca[1].x, ca[1].y, ca[1].z, ca[1].w};
            const float sn[8] = {ca[2].x, ca[2].y, ca[2].z, ca[2].w, ca[3].x, ca[3].y, ca[3].z, ca[3].w};
            const float sign = first ? -1.f : 1.f;
            floats(o, y);
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = fmaf(x[e], cs[e], y[e] * (sign * sn[e]));
          }
          const RcUpper hx = rc_split8(x, dst, kRcQ);
#pragma unroll
          for (int e = 0; e < 4; ++e) rc_watch(hx.h[e], z);
        } else {  // bf16: one part, the others' zeros stand since the start
          *reinterpret_cast<uint4*>(dst) = w;
          rc_watch(w.x, z);
          rc_watch(w.y, z);
          rc_watch(w.z, z);
          rc_watch(w.w, z);
        }
      }
    // ---- v' ----
#pragma unroll
    for (int i = 0; i < kVN; ++i) {
      const int tok = vt + i * kVStep;
      float x[8];
      floats(rv[i], x);
      if constexpr (umma_fmt<T>::v == 1) {
        rc_watch(rv[i].x, z);
        rc_watch(rv[i].y, z);
        rc_watch(rv[i].z, z);
        rc_watch(rv[i].w, z);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) rc_watch(pack2<__nv_bfloat16>(x[2 * e], x[2 * e + 1]), z);
      }
      const float f = pw[kRcTok - 1 - tok] * p.k_scale;
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] *= f;
      rc_split8(x, sW + (vc >> 3) * kRcV + rc_off(tok, vc & 7), kW);
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (warp == 0) {
      tc_fence_after_sync();
      constexpr uint32_t id_kv = umma_idesc<__nv_bfloat16>(128, NC, 1, 1);
      const uint64_t dk = umma_desc_sw128(smem_u32(sK), kRcV, 1024), dw = umma_desc_sw128(smem_u32(sW), kRcV, 1024);
      const uint32_t hi = static_cast<uint32_t>(dk >> 32);
      uint32_t acc = 0;
#pragma unroll 1
      for (int pr = 0; pr < 6; ++pr) {
        const uint32_t a = static_cast<uint32_t>(dk) + rc_pa(pr) * (kRcQ >> 4), b = static_cast<uint32_t>(dw) + rc_pb(pr) * (kW >> 4);
#pragma unroll
        for (int s = 0; s < kRcTok / 16; ++s) {
          umma_ss_if(leader, tU, a + s * 128, b + s * 128, hi, id_kv, acc);
          acc = 1;
        }
      }
      umma_commit_if(leader, bar);
    }
    __syncwarp();
    if (c + kRcTok < p.seg_tokens) read(t0 + kRcTok);
  }
  fold(p.seg_tokens - kRcTok);
  const int odd = __syncthreads_or(rc_spoilt(z));
  if (tid == 0) p.flags[(static_cast<int64_t>(blockIdx.x) * p.H + h) * (p.dv / NC) + blockIdx.z] = *dead ? 2 : odd ? 1 : 0;
  if (*dead) {
    wait_drain();
    if (tid == 0) wait_report(p.wait_expired);
  }
  if (warp == 0) tmem_dealloc(tU, 2 * NC);
}

// The state behind every segment but a portion's last, in place of what the segment adds: S = d^L S + U.  A thread takes four
// values of a head through the segments of its portion.
__global__ void __launch_bounds__(256)
retention_scan_kernel(const __grid_constant__ RetChunkParams p) {
  __shared__ float d_seg;
  const int r = blockIdx.y, lane = threadIdx.x & 31;
  const int64_t per_head = static_cast<int64_t>(p.dv) * kRcDk, at = blockIdx.x * 1024ll;  // (a multiple of 1024 floats a head)
  int first = 0, nseg = 0;
  for (int i = lane; i <= r; i += 32) {
    const int n = p.prefix_lens[i] >= 0 ? max(p.extend_lens[i], 0) : 0;
    const int ns = (n + p.seg_tokens - 1) / p.seg_tokens;
    if (i < r) first += ns;
    else nseg = ns;
  }
  first = __reduce_add_sync(0xffffffffu, first);
  nseg = __reduce_add_sync(0xffffffffu, nseg);
  if (nseg < 2) return;
  if (threadIdx.x == 0) {
    double b = static_cast<double>(p.decay[at / per_head]), x = 1.0;
    for (int e = p.seg_tokens; e > 0; e >>= 1) {
      if (e & 1) x *= b;
      b *= b;
    }
    d_seg = static_cast<float>(x);
  }
  __syncthreads();
  const float d = d_seg;
  const int64_t per_seg = p.H * per_head / 4;
  float4* slot = reinterpret_cast<float4*>(p.sums) + first * per_seg + at / 4 + threadIdx.x;
  float4 S = p.prefix_lens[r] > 0 ? slot[(nseg - 1) * per_seg] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int i = 0; i < nseg - 1; ++i) {
    const float4 u = slot[i * per_seg];
    S.x = fmaf(d, S.x, u.x);
    S.y = fmaf(d, S.y, u.y);
    S.z = fmaf(d, S.z, u.z);
    S.w = fmaf(d, S.w, u.w);
    slot[i * per_seg] = S;
  }
}

template <typename T, int NC>
static int rc_launch_sums(const RetChunkParams& p, int64_t segments, cudaStream_t stream) {
  constexpr int smem = 3 * kRcQ + 3 * (NC / 64) * kRcV + 1024 + 1024;
  auto kern = retention_sums_kernel<T, NC>;
  static bool configured = false;  // per instantiation
  if (!configured) {
    SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured = true;
  }
  SPD_CUDA(launch(kern, dim3((unsigned)segments, (unsigned)p.H, (unsigned)(p.dv / NC)), dim3(kRsThreads), smem, stream,
                  /*pdl=*/false, p));
  SPD_CUDA(launch(retention_scan_kernel, dim3((unsigned)(p.H * (p.dv / kRcDv) * (kRcDk * kRcDv / 1024)), (unsigned)p.batch),
                  dim3(256), 0, stream, /*pdl=*/false, p));
  return 0;
}

template <typename T, int VS, bool kCut>
static int rc_launch(const RetChunkParams& p, int64_t segments, cudaStream_t stream) {
  constexpr int smem = 6 * kRcQ + 3 * kRcS + (3 + VS) * kRcV + (2 * kRcTok * kRcDk + kRcTok * kRcDv) * 2 + kRcMisc + 1024;
  static_assert(smem <= 232448, "does not fit an SM");
  auto kern = retention_chunked_kernel<T, VS, kCut>;
  static bool configured = false;  // per instantiation
  if (!configured) {
    SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured = true;
  }
  if constexpr (kCut) {
    const int rc = p.flag_cols == 128 ? rc_launch_sums<T, 128>(p, segments, stream) : rc_launch_sums<T, 64>(p, segments, stream);
    if (rc) return rc;
  }
  SPD_CUDA(launch(kern, dim3((unsigned)segments, (unsigned)p.H, (unsigned)(p.dv / kRcDv)), dim3(kRcThreads), smem, stream,
                  /*pdl=*/false, p));
  return 0;
}

// Tokens of a segment (a multiple of 64), or 0: portions are not cut.  Estimates in us.  Not cut: the longest portion (which
// only the device knows: 1.25 times the mean) at 5.6 per chunk.  Cut: the waves of CTAs of the segments' sums (4.5 per chunk,
// two CTAs an SM, 128 columns each), 10 for the scan and the launches, the waves of the chunks' own CTAs and 6 for each
// but the first (a CTA begins when one before it has ended).  16 heads, not cut /
// cut: 1 x 500 tokens 52 / 37 (segments of 2 chunks), 1 x 1500 139 / 71 (3), 1 x 8000 728 / 241 (7), 2 x 1000 97 / 85 (4),
// 2 x 3000 277 / 208 (8), 3 x 2000 190 / 216 (6); 32 heads, 3 x 2000 377 / 418 (5), 371 (12).
static int rc_seg_tokens(int64_t batch, int64_t total_tokens, int H, int dv, int sms, double* us = nullptr) {
  const int64_t chunks = (total_tokens + kRcTok - 1) / kRcTok, ctas = static_cast<int64_t>(H) * (dv / kRcDv);
  auto waves = [](int64_t n, int64_t slots) { return static_cast<double>((n + slots - 1) / slots); };
  const double mean = static_cast<double>(chunks) / static_cast<double>(batch);
  const double whole = waves(batch * ctas, sms) * 5.6 * (batch > 1 ? 1.25 : 1.0) * mean + 4;
  double best = 0.9 * whole;
  int seg = 0;
  for (int n = 2; n <= 16; ++n) {
    const int64_t segs = (chunks + n - 1) / n + batch / 2;
    if (segs <= batch) break;
    const double w = waves(segs * ctas, sms);
    const double t = w * (5.6 * n + 4) + (w - 1) * 6 + 10 + waves((segs - batch) * ((ctas + 1) / 2), 2 * sms) * (4.5 * n + 5);
    if (t < best) {
      best = t;
      seg = n;
    }
  }
  if (us != nullptr) *us = seg > 0 ? best : whole;
  return seg * kRcTok;
}
// What the chunks take, in us.
double retention_chunked_us(int64_t batch, int64_t total_tokens, int H, int dv, int sms) {
  double us;
  rc_seg_tokens(batch, total_tokens, H, dv, sms, &us);
  return us;
}
static int64_t rc_segments(int64_t batch, int64_t total_tokens, int seg_tokens) { return total_tokens / seg_tokens + batch; }
static bool rc_applies(int64_t batch, int64_t total_tokens, int H, int dk, int dv, int rot, int in_act, int dtype) {
  // A chunk costs what some tens of tokens cost one by one, and its CTA takes a whole SM: 4 requests of 16 tokens 12.1 us
  // (token by token) / 11.8, of 64 tokens 32.9 / 17.6; 16 requests of 16 tokens 30 / 41 us, of 40 tokens 63 / 41.
  if (total_tokens <= 40 * batch) return false;
  // 16-bit rows without an activation (their parts are what the split was counted for), 128 channels, whole 64-column
  // slices, a rotation in whole 16-byte pieces
  return dtype != SPD_F32 && in_act == 0 && dk == kRcDk && dv > 0 && dv % kRcDv == 0 && rot % 16 == 0 && H <= 65535 &&
         dv / kRcDv <= 65535;
}
int64_t retention_chunked_workspace(int64_t batch, int64_t total_tokens, int H, int dk, int dv, int rot, int in_act, int dtype,
                                    int sms) {
  if (batch <= 0 || batch > 65535 || H <= 0 || sms <= 0 || !rc_applies(batch, total_tokens, H, dk, dv, rot, in_act, dtype)) return 0;
  const int seg = rc_seg_tokens(batch, total_tokens, H, dv, sms);
  if (seg == 0) return 0;
  const int64_t n = rc_segments(batch, total_tokens, seg);
  return n * H * (2ll * dv * kRcDk * 4 + dv / kRcDv * 4ll);
}

// → 0 launched, 1 not applicable (the caller takes the token-by-token kernel), else an error
int retention_chunked_try(float* o, const void* q, const void* k, const void* v, float* state,
                          const int64_t* req_pool_indices, const int32_t* prefix_lens, const int32_t* extend_lens,
                          const int32_t* extend_start_loc, int64_t batch, int H, int dk, int dv, int64_t q_stride,
                          int64_t k_stride, int64_t v_stride, const float* decay, const float* cos_sin, int rot,
                          int64_t max_positions, float k_scale, int in_act, int dtype, int64_t total_tokens,
                          void* workspace, int64_t workspace_bytes, int sms, cudaStream_t stream) {
  if (!rc_applies(batch, total_tokens, H, dk, dv, rot, in_act, dtype)) return 1;
  // 16-byte rows
  if (q_stride % 8 != 0 || k_stride % 8 != 0 || v_stride % 8 != 0 || !aligned16(q) || !aligned16(k) || !aligned16(v) ||
      !aligned16(o) || !aligned16(state) || (rot > 0 && !aligned16(cos_sin)))
    return 1;
  unsigned* wait_expired;
  if (int rc = wait_flag(&wait_expired)) return rc;
  RetChunkParams p{o, q, k, v, state, req_pool_indices, prefix_lens, extend_lens, extend_start_loc, H, dv, rot,
                   q_stride, k_stride, v_stride, max_positions, decay, cos_sin, k_scale, wait_expired,
                   static_cast<int>(batch), 1 << 30, nullptr, nullptr, nullptr, dv % 128 == 0 ? 128 : 64};
  int64_t segments = batch;
  const int seg = workspace != nullptr && aligned16(workspace) && sms > 0 && batch <= 65535 ? rc_seg_tokens(batch, total_tokens, H, dv, sms) : 0;
  if (seg > 0 && workspace_bytes >= retention_chunked_workspace(batch, total_tokens, H, dk, dv, rot, in_act, dtype, sms)) {
    segments = rc_segments(batch, total_tokens, seg);
    p.seg_tokens = seg;
    p.sums = static_cast<float*>(workspace);
    p.keep = p.sums + segments * H * static_cast<int64_t>(dv) * kRcDk;
    p.flags = reinterpret_cast<int*>(p.keep + segments * H * static_cast<int64_t>(dv) * kRcDk);
  }
  if (p.sums != nullptr)
    return dtype == SPD_BF16 ? rc_launch<__nv_bfloat16, 1, true>(p, segments, stream) : rc_launch<__half, 2, true>(p, segments, stream);
  return dtype == SPD_BF16 ? rc_launch<__nv_bfloat16, 1, false>(p, segments, stream) : rc_launch<__half, 2, false>(p, segments, stream);
}

}  // namespace spd
