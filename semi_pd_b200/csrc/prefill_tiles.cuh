// What the tcgen05 prefill attentions share: the work list of row tiles by weight, MMAs issued by a whole warp, a row pass of
// the softmax over one unit of 64 scores in tensor memory.
#pragma once
#include "ptx.cuh"

namespace spd {

// floor(n / d), n < 2^31, with (m, s) from fastdiv_magic(d)
__device__ __forceinline__ int fastdiv(int n, uint32_t m, uint32_t s) {
  return static_cast<int>((static_cast<uint64_t>(__umulhi(static_cast<uint32_t>(n), m)) + static_cast<uint32_t>(n)) >> s);
}
// Granlund-Montgomery round-up magic: s = ceil(log2 d), m = floor(2^32 * (2^s - d) / d) + 1
inline void fastdiv_magic(uint32_t d, uint32_t& m, uint32_t& s) {
  s = 0;
  while ((1ull << s) < d) ++s;
  m = static_cast<uint32_t>(((1ull << 32) * ((1ull << s) - d)) / d + 1);
}

// The row tiles of a launch that has more items than CTAs, heaviest first.  Every CTA makes the same list in its own
// shared memory.
constexpr int kTileList = 768;  // row tiles that it holds
struct TileList {
  int items;             // items to deal: row tiles x heads
  const uint16_t* list;  // nullptr: no list, items in the order of their position
};
// slots 0 .. n_slots - 1 with a weight (below 65536) other than 0, sorted, into `list`; keys: kTileList words of shared memory,
// 16-byte aligned, that nothing uses yet; count: zero before.  More of them than the list holds: no list, `all` items.
// It stands before a CTA's first load, so its own time counts: up to a slot per thread there is no compaction, and a rank is
// counted from four keys a read (64 slots: 1.3 us with an atomic per slot and a key per read, 1.1 here, most of it the
// loads of the lengths).
template <int kThreads, typename Weight>
__device__ __forceinline__ TileList tile_list(int n_slots, int heads, int all, Weight weight, uint32_t* keys, uint32_t* count,
                                              uint16_t* list) {
  auto place = [&](uint32_t key, int n) {  // keys differ: the order is the same in every CTA
    const uint4* k4 = reinterpret_cast<const uint4*>(keys);
    int rank = 0;
#pragma unroll 4
    for (int f = 0; f < n / 4; ++f) {
      const uint4 k = k4[f];
      rank += (k.x > key) + (k.y > key) + (k.z > key) + (k.w > key);
    }
    for (int f = n & ~3; f < n; ++f) rank += keys[f] > key;
    list[rank] = static_cast<uint16_t>(key);
  };
  static_assert(kThreads <= kTileList, "a slot per thread fits the list");
  if (n_slots <= kThreads) {
    const int slot = threadIdx.x, w = slot < n_slots ? weight(slot) : 0;
    const uint32_t key = w > 0 ? static_cast<uint32_t>(w) << 16 | static_cast<uint32_t>(slot) : 0u;  // (0: below all others)
    if (slot < n_slots) keys[slot] = key;
    const int n = __syncthreads_count(w > 0);
    if (w > 0) place(key, n_slots);
    __syncthreads();
    return TileList{n * heads, list};
  }
  for (int slot = threadIdx.x; slot < n_slots; slot += kThreads) {
    const int w = weight(slot);
    if (w > 0) {
      const uint32_t at = atomicAdd(count, 1u);
      if (at < kTileList) keys[at] = static_cast<uint32_t>(w) << 16 | static_cast<uint32_t>(slot);
    }
  }
  __syncthreads();
  const int n = static_cast<int>(*count);
  if (n > kTileList) return TileList{all, nullptr};
  for (int e = threadIdx.x; e < n; e += kThreads) place(keys[e], n);
  __syncthreads();
  return TileList{n * heads, list};
}

// k-th item of CTA c out of G CTAs, snake order over the heaviest-first list
__device__ __forceinline__ int pf_rank(int k, int c, int G) {
  return k * G + ((k & 1) ? (G - 1 - c) : c);
}

// a place in a ring and the parity of its current round
template <int n>
struct RingSlot {
  int i = 0;
  uint32_t round = 0;
  __device__ __forceinline__ void next() {
    if (++i == n) {
      i = 0;
      round ^= 1;
    }
  }
};

// MMAs and commits issued by the warp's lane for which `on` holds; every lane computes the operands.  Descriptors by
// halves, as in umma_ss_lo.  umma_ts_if: A (here the 16-bit probabilities, two per 32-bit column, row = TMEM lane) is read
// from tensor memory.
__device__ __forceinline__ void umma_ss_if(bool on, uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}\n" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate), "r"(static_cast<uint32_t>(on))
      : "memory");
}
__device__ __forceinline__ void umma_ts_if(bool on, uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi,
                                           uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}\n" ::"r"(tmem_d),
      "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(static_cast<uint32_t>(on))
      : "memory");
}
__device__ __forceinline__ void umma_commit_if(bool on, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(smem_u32(bar)),
      "r"(static_cast<uint32_t>(on))
      : "memory");
}

// Packed fp32 pairs (sm_100 FFMA2 / FADD2): one instruction per two elements.  The softmax warps
// are issue-bound around the MUFU stream (one warp per scheduler and warpgroup), so halving the
// FFMA / FADD count is what shortens a row pass.
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t fmul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fadd2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// key `kv` of a masked unit is visible: kv <= limit, and with a window (span = its size - 1) limit - kv <= span
template <bool kWin>
__device__ __forceinline__ bool pf_visible(int kv, int limit, int span) {
  if constexpr (kWin) return static_cast<uint32_t>(limit - kv) <= static_cast<uint32_t>(span);
  return kv <= limit;
}
// 32 columns of one tile row: p = exp2(s*scale - m_off), packed to 16 bits into pk[0..16), and their sum.
// kRound: the sum of the rounded p, the weights that the products use: sum(p v) / sum(p) is then a true mean of the v, and
// the rounding of a p that outweighs the others cancels.
template <typename T, bool kMask, bool kRound>
__device__ __forceinline__ void softmax_chunk(const uint32_t* r, int c, uint32_t* pk, uint64_t scale2,
                                              uint64_t neg_m2, int kv0, int limit, uint64_t& ps) {
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    float x0, x1;
    unpack_f32x2(ffma2(pack_f32x2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), scale2, neg_m2), x0, x1);
    float p0 = fast_exp2(x0);
    float p1 = fast_exp2(x1);
    if constexpr (kMask) {
      p0 = kv0 + c + i <= limit ? p0 : 0.f;
      p1 = kv0 + c + i + 1 <= limit ? p1 : 0.f;
    }
    pk[i >> 1] = pack2<T>(p0, p1);
    if constexpr (kRound) {
      const float2 f = unpack2<T>(pk[i >> 1]);
      p0 = f.x;
      p1 = f.y;
    }
    ps = fadd2(ps, pack_f32x2(p0, p1));
  }
}

// One row of one S unit (64 columns) for one thread: S (TMEM) -> 32 packed 16-bit
// pairs in registers.  Returns the row sum of p (masked entries excluded).  Two 32-column TMEM
// loads are in flight while the previous 32 columns are exponentiated.  kMask is a template
// parameter so that the unmasked units run the lean loop: FFMA + MUFU.EX2 + FADD + half an F2FP
// per element.
template <typename T, bool kMask>
__device__ __forceinline__ float softmax_row_pass(uint32_t ts, uint32_t* pk, float scale_log2, float m_off,
                                                  int kv0, int limit) {
  const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2);
  const uint64_t neg_m2 = pack_f32x2(-m_off, -m_off);
  uint64_t ps = pack_f32x2(0.f, 0.f);
  uint32_t ra[32], rb[32];
  tmem_ld_32x32b_x32(ts, ra);
  tmem_ld_32x32b_x32(ts + 32, rb);
  tmem_ld_wait();
  softmax_chunk<T, kMask, false>(ra, 0, pk, scale2, neg_m2, kv0, limit, ps);
  softmax_chunk<T, kMask, false>(rb, 32, pk + 16, scale2, neg_m2, kv0, limit, ps);
  float ps0, ps1;
  unpack_f32x2(ps, ps0, ps1);
  return ps0 + ps1;
}

// The same against the true running max, from one read of the unit: scores of keys that the row does not see become -inf
// (a scale above 0 then makes their p 0), the row's max, then the p.
template <bool kMask, bool kWin>
__device__ __forceinline__ float softmax_load_max(uint32_t ts, uint32_t* ra, uint32_t* rb, int kv0, int limit, int span) {
  tmem_ld_32x32b_x32(ts, ra);
  tmem_ld_32x32b_x32(ts + 32, rb);
  tmem_ld_wait();
  float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    if constexpr (kMask) {
      ra[i] = pf_visible<kWin>(kv0 + i, limit, span) ? ra[i] : 0xff800000u;
      rb[i] = pf_visible<kWin>(kv0 + 32 + i, limit, span) ? rb[i] : 0xff800000u;
    }
    m0 = fmaxf(m0, __uint_as_float(ra[i]));
    m1 = fmaxf(m1, __uint_as_float(rb[i]));
  }
  return fmaxf(m0, m1);
}
// kRound sums (see softmax_chunk) of a unit that softmax_load_max has read
template <typename T>
__device__ __forceinline__ float softmax_unit(const uint32_t* ra, const uint32_t* rb, uint32_t* pk, float scale_log2, float m_off) {
  const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2);
  const uint64_t neg_m2 = pack_f32x2(-m_off, -m_off);
  uint64_t ps = pack_f32x2(0.f, 0.f);
  softmax_chunk<T, false, true>(ra, 0, pk, scale2, neg_m2, 0, 0, ps);
  softmax_chunk<T, false, true>(rb, 32, pk + 16, scale2, neg_m2, 0, 0, ps);
  float ps0, ps1;
  unpack_f32x2(ps, ps0, ps1);
  return ps0 + ps1;
}
// a row's 128 fp32 sums in tensor memory times alpha (collective over the warp)
__device__ __forceinline__ void rescale_row128(uint32_t to, float alpha) {
  const uint64_t a2 = pack_f32x2(alpha, alpha);
#pragma unroll 1
  for (int c = 0; c < 128; c += 64) {
    uint32_t ra[32], rb[32];
    tmem_ld_32x32b_x32(to + c, ra);
    tmem_ld_32x32b_x32(to + c + 32, rb);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      float x, y;
      unpack_f32x2(fmul2(pack_f32x2(__uint_as_float(ra[i]), __uint_as_float(ra[i + 1])), a2), x, y);
      ra[i] = __float_as_uint(x);
      ra[i + 1] = __float_as_uint(y);
      unpack_f32x2(fmul2(pack_f32x2(__uint_as_float(rb[i]), __uint_as_float(rb[i + 1])), a2), x, y);
      rb[i] = __float_as_uint(x);
      rb[i + 1] = __float_as_uint(y);
    }
    tmem_st_32x32b_x32(to + c, ra);
    tmem_st_32x32b_x32(to + c + 32, rb);
  }
}

constexpr float kRescaleTrigger = 256.f;  // a row sum above 2^8 may hide an element above 2^8

// max of the visible raw scores of one row of an S unit (TMEM)
template <bool kMask>
__device__ __forceinline__ void rowmax_chunk(const uint32_t* r, int c, int kv0, int limit, float& m0, float& m1) {
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    float a = __uint_as_float(r[i]), b = __uint_as_float(r[i + 1]);
    if constexpr (kMask) {
      a = kv0 + c + i <= limit ? a : -INFINITY;
      b = kv0 + c + i + 1 <= limit ? b : -INFINITY;
    }
    m0 = fmaxf(m0, a);
    m1 = fmaxf(m1, b);
  }
}
template <bool kMask>
__device__ __forceinline__ float softmax_row_max(uint32_t ts, int kv0, int limit) {
  float m0 = -INFINITY, m1 = -INFINITY;
  uint32_t ra[32], rb[32];
  tmem_ld_32x32b_x32(ts, ra);
  tmem_ld_32x32b_x32(ts + 32, rb);
  tmem_ld_wait();
  rowmax_chunk<kMask>(ra, 0, kv0, limit, m0, m1);
  rowmax_chunk<kMask>(rb, 32, kv0, limit, m0, m1);
  return fmaxf(m0, m1);
}

}  // namespace spd
