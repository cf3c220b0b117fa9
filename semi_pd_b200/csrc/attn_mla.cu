// Absorbed multi-head latent attention (MLA) over the token-granular latent KV pool on tcgen05 — decode and ragged
// extend in one kernel.
//
// Reference: DeepseekV2AttentionMLA.forward_absorb (python/sglang/srt/models/deepseek_v2.py:633-706)
// over MLATokenToKVPool rows [kv_a_normed(kv_lora) || k_pe_roped(rope)] (mem_cache/memory_pool.py:
// 379-452), computed there by the Triton kernels decode_attention_fwd_grouped / extend_attention_fwd
// (layers/attention/triton_ops/decode_attention.py:235-470, extend_attention.py:291-410): all H
// query heads share ONE latent K/V stream (MQA), K = the whole latent row (DL = kv_lora + rope),
// V = its first DV = kv_lora columns.  The reference switches to a plain MHA (forward_normal) for
// prefill batches without a cached prefix; the absorbed form, the same function of the same inputs
// (oracle/deepseek_oracle.py checks both against each other), serves decode here and the prefill
// batches for which expanded heads (attn_mla_prefill.cu) would not be faster.
//
// Swap-AB formulation: an item is TQ query tokens x 16 heads = N columns (decode: 1 x 16, extend: 4 x 16),
//     S^T[64 kv x N]  = K_tile[64 x 576] * Q^T           (36 MMAs, M = 64)
//     O^T[512 x N]   += V_tile^T[512 x 64 kv] * P^T       (4 blocks of 128 value columns x 4 MMAs, M = 128)
// so a latent row enters an SM once per N columns, serves both products from the same shared memory, and the fp32
// output of a whole item (4 N columns of TMEM) stays on chip.  N = 64 is what fits: 72 KB of Q, two 72 KB K/V tiles
// and 8 KB of P are the 227 KB of an SM, 256 columns of O^T and two S^T in two halves the 512 of its TMEM.
//
// Work split.  The tiles of all items, one after another, are one list that the CTAs (one per SM) cut into equal
// contiguous ranges; lengths are read on the device, so nothing is planned on the host.  A CTA that starts or ends
// inside an item leaves a partial (max, sum, O^T) in the workspace and a second small kernel merges the parts of each
// such item; with many items per CTA the cuts are moved to item starts instead (`snap`) and nothing is merged.
//
// warps 0-3: softmax, O rescale, epilogue     warps 4-5: loaders     warp 6: MMA issuer + TMEM allocator.
// The K/V ring is made of slots of 16 KB (one pair of a tile's 64-column blocks, what one PV block reads) and of 8 KB
// (its rope block, free after S), each given back by itself: 2.75 tiles at N = 16, 2 at N = 64.  A tile's copies meet on
// one barrier.  Full tiles of 64 consecutive slots come by TMA (four boxes of 64 rows x 2 blocks and one of 64 x 1),
// anything else by 16-byte cp.async through req_to_token.  The
// softmax keeps the true running max per column (see there): scores are read from TMEM in the 16x256b fragment layout (all
// 32 lanes of a warp busy although M = 64 fills 16 lanes per warp), P goes back as stmatrix-transposed K-major rows.
//
// Decode streams each latent row once, 64 requests of 1088 keys (83 MB) in 26.3 us with the merge launch, 160 of 1000 in
// 44.5 in a row; one CTA per token, head group and split with warp-level MMAs took 62 us.  Start, last tile and merge are 14
// of the 26 us; between them a 72 KB tile takes 1.67 us per SM, which is what its copies alone take.  It took 2.7 us (34.3
// for the 64 requests) while a tile held its slots for 4000 clk after landing and its copies were issued one after the
// other: what counts is the time from landing to the last PV (S 1130 clk, softmax 600, PV 700), so the reference of the
// softmax lags in decode, the two parts of P are columns of one product (V passes once), and Q's copies and a tile's five
// go out in parallel.  MMAs (M = 64: 23 clk at N = 16, 31 at N = 64) are hidden as long as the issuer's code stays a
// short loop.  Extend, 4096 new tokens in 4 requests (two with 515 cached), whole layer: 1645 -> 600 us (a batch that takes
// expanded heads now: 185 us); bounded by the
// ring of two tiles (a tile's copies start when the PV before last has finished), by the rescale of O^T whenever a tile
// raises one of 64 columns, and by beginning and ending items, which therefore count in the split (without that, SMs with
// short items took twice as long).
//
// Every mbarrier wait is bounded: a wait that runs out marks the CTA dead, all later waits fall through, the kernel
// finishes without waiting and sets the word that spd_wait_status reads.
#include <cuda.h>

#include "common.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace spd {

constexpr int kMlaThreads = 224;
constexpr int kMlaTile = 64;     // kv tokens per tile
constexpr int kMlaHeads = 16;    // heads per item
constexpr int kMlaDL = 576, kMlaDV = 512;
constexpr int kMlaBlk = kMlaTile * 128;       // one [64 rows x 64 columns] swizzle block of a tile
constexpr int kMlaMisc = 2048;

struct MlaParams {
  void* out;             // [items, H, DV]
  const void* q;         // [items, H, DL]
  const void* kv_pool;   // [slots, DL]
  const int32_t* req_to_token;
  const int64_t* req_pool_indices;
  const int64_t* seq_lens;          // decode (extend: nullptr)
  const int32_t* prefix_lens;       // extend
  const int32_t* extend_start_loc;  // extend
  int batch, total, H, hgs;         // total: query tokens (extend); hgs: groups of 16 heads
  int64_t q_stride, out_stride, rtt_stride;
  int q_row0, q_dir;  // decode: token i is row q_row0 + q_dir i of Q's tensor map
  float scale_log2;
  int min_tiles;   // fewest tiles a CTA takes
  int snap;        // 1: CTA ranges start at item starts, nothing is split
  int cols;        // columns of a partial: TQ x min(H, 16)
  float* o_part;   // [2 * grid][cols][DV]
  float* ml_part;  // [2 * grid][cols][2]
  int by_item;     // 1: info by item (few of them, see mla_merge_many_kernel), not by the CTA that an item ends in
  int* info;       // [grid][8]: see mla_merge_kernel
  unsigned* wait_expired;
};

template <bool kExtend>
struct MlaShape {
  static constexpr int TQ = kExtend ? 4 : 1;
  static constexpr int N = TQ * kMlaHeads;
  static constexpr int E = kExtend ? 2 : 1;  // what beginning and ending an item costs, in tiles: it counts in the work split
  static constexpr int kQBytes = 9 * N * 128;
  // P as the sum of two 16-bit numbers (decode): rounded to one, its error grew 2.3 % over the warp-level kernel's, whose
  // shorter tiles and splits had more probabilities that are exactly 1 (extend: 0.1 % of a layer's, and no room for it)
  static constexpr int kPParts = kExtend ? 1 : 2;
  static constexpr float kLag = kExtend ? 0.f : 8.f;  // how far (log2) a score may exceed its column's reference
  static constexpr int kPPart = N * 128;
  static constexpr int kPBytes = kPParts * kPPart;
  static constexpr int kPairs = kExtend ? 8 : 11;  // ring slots of 16 KB: one pair of 64-column blocks of a tile
  static constexpr int kRopes = kExtend ? 2 : 3;   // ring slots of 8 KB: a tile's rope block
  static constexpr int kRing = kPairs * 2 * kMlaBlk + kRopes * kMlaBlk;
  static constexpr int kBars = kPairs + kRopes + 4 + 9;
  static constexpr int kSmem = kQBytes + kRing + kPBytes + kMlaMisc + 1024;
  static constexpr int kON = kPParts * N;          // columns of an O^T block: one set for each part of P
  static constexpr int kOCols = 4 * kON;           // TMEM columns of O^T, then two S^T of two halves
  static constexpr int kTmem = kExtend ? 512 : 256;
};
static_assert(MlaShape<true>::kSmem <= 232448 && MlaShape<false>::kSmem <= 232448 && MlaShape<true>::kTmem <= 512,
              "does not fit an SM");
static_assert(MlaShape<true>::kBars * 8 + 40 + 256 + 5 * 4 * 64 <= kMlaMisc &&
                  MlaShape<false>::kBars * 8 + 40 + 256 + 5 * 4 * 16 <= kMlaMisc,
              "misc area");

// a place in a ring and the parity of its current round
template <int n>
struct MlaSlot {
  int i = 0;
  uint32_t round = 0;
  __device__ __forceinline__ void next() {
    if (++i == n) {
      i = 0;
      round ^= 1;
    }
  }
};

// an item: one token (decode) or group of four tokens (extend) of a request, times 16 heads
struct MlaItem {
  int hg, r, j;                       // head group, request, token group
  int row0, ntok, p0, vis, load_end;  // first query row, tokens, position of the first, visible keys, loadable keys
  int ntiles, next_r;                 // next_r: 1 when the request has no further group
};

__device__ __forceinline__ void mla_request(const MlaParams& p, int r, int& start, int& ext, int& prefix) {
  start = p.extend_start_loc[r];
  ext = (r + 1 < p.batch ? p.extend_start_loc[r + 1] : p.total) - start;
  prefix = p.prefix_lens[r];
}

template <bool kExtend>
__device__ __forceinline__ void mla_set_item(const MlaParams& p, MlaItem& it) {
  if constexpr (kExtend) {
    constexpr int TQ = MlaShape<true>::TQ;
    int start, ext, prefix;
    mla_request(p, it.r, start, ext, prefix);
    const int i0 = it.j * TQ;
    it.ntok = min(TQ, ext - i0);
    it.row0 = start + i0;
    it.p0 = prefix + i0;
    it.vis = it.p0 + it.ntok;
    it.load_end = prefix + ext;
    it.next_r = i0 + TQ >= ext;
  } else {
    const int L = static_cast<int>(p.seq_lens[it.r]);
    it.ntok = 1;
    it.row0 = it.r;
    it.p0 = L - 1;
    it.vis = it.load_end = L;
    it.next_r = 1;
  }
  it.ntiles = max(1, (it.vis + kMlaTile - 1) / kMlaTile);
}

// tiles of the first n token groups of 4 with `prefix` cached tokens, all of them full:
// sum over k = 1..n of ceil((prefix + 4 k) / 64) = sum of floor((k + u) / 16), u = floor((prefix + 63) / 4)
__device__ __forceinline__ int mla_floor16_sum(int x) {  // sum of floor(i / 16), i = 0..x
  const int q = x >> 4;
  return 8 * q * (q - 1) + q * ((x & 15) + 1);
}
__device__ __forceinline__ int mla_group_tiles(int prefix, int n) {
  const int u = (prefix + 63) >> 2;
  return mla_floor16_sum(n + u) - mla_floor16_sum(u);
}
// units of a request in the work list: the tiles of its items, and E for each item (in front of its tiles)
template <bool kExtend>
__device__ __forceinline__ int mla_request_tiles(const MlaParams& p, int r) {
  if constexpr (kExtend) {
    int start, ext, prefix;
    mla_request(p, r, start, ext, prefix);
    if (ext <= 0) return 0;
    return mla_group_tiles(prefix, ext / 4) + (ext % 4 ? (prefix + ext + kMlaTile - 1) / kMlaTile : 0) +
           (ext + 3) / 4 * MlaShape<true>::E;
  } else {
    return max(1, (static_cast<int>(p.seq_lens[r]) + kMlaTile - 1) / kMlaTile) + MlaShape<false>::E;
  }
}

template <bool kExtend>
__device__ __forceinline__ void mla_next_item(const MlaParams& p, MlaItem& it) {
  if (!it.next_r) {
    ++it.j;
  } else {
    it.j = 0;
    do {
      if (++it.r == p.batch) {
        it.r = 0;
        if (++it.hg == p.hgs) return;  // past the end: the caller has no tiles left
      }
      if constexpr (kExtend) {
        int start, ext, prefix;
        mla_request(p, it.r, start, ext, prefix);
        if (ext > 0) break;
      } else {
        break;
      }
    } while (true);
  }
  mla_set_item<kExtend>(p, it);
}

// walks the CTA's tiles: every role keeps its own copy
template <bool kExtend>
struct MlaCursor {
  static constexpr int E = MlaShape<kExtend>::E;
  MlaItem it;
  int tile, left, seg;  // left: units of the CTA's range that remain, from this tile on; seg: items left behind so far
  bool valid;
  __device__ __forceinline__ void init(const MlaParams& p, const int* start, int count) {
    it.hg = start[0];
    it.r = start[1];
    it.j = start[2];
    const int at = start[3];  // units of the item before the range
    left = count;
    seg = tile = 0;
    valid = left > 0;
    if (!valid) return;
    mla_set_item<kExtend>(p, it);
    if (p.snap) {  // an item belongs to the CTA whose range holds its first unit
      if (at > 0) {
        left -= it.ntiles + E - at;
        valid = left > 0;
        if (valid) mla_next_item<kExtend>(p, it);
      }
      left -= E;
    } else if (at <= E) {
      left -= E - at;
      valid = left > 0;
    } else {
      tile = at - E;
    }
  }
  // whether this tile is the last of its item here
  __device__ __forceinline__ bool ends(const MlaParams& p) const {
    return tile + 1 == it.ntiles || (!p.snap && left == 1);
  }
  __device__ __forceinline__ void next(const MlaParams& p) {
    const bool e = ends(p);
    --left;
    if (!e) {
      ++tile;
      return;
    }
    ++seg;
    tile = 0;
    valid = p.snap ? left > 0 : left > E;
    left -= E;
    if (valid) mla_next_item<kExtend>(p, it);
  }
};

// [rows x 64 columns] 16-bit swizzle block: 16-byte chunk `c` (0..7) of row `row`
__device__ __forceinline__ uint32_t mla_off(int row, int c) { return row * 128 + ((c ^ (row & 7)) << 4); }

__device__ __forceinline__ bool mla_bar_or(bool pred) {  // barrier + OR over the 128 softmax threads
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "barrier.cta.red.or.pred p, 1, 128, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(out)
      : "r"(static_cast<uint32_t>(pred))
      : "memory");
  return out != 0;
}
__device__ __forceinline__ void mla_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
__device__ __forceinline__ void mla_loader_bar() { asm volatile("bar.sync 2, 64;" ::: "memory"); }  // the loader threads
__device__ __forceinline__ bool mla_loader_and(bool pred) {  // barrier + AND over the 64 loader threads
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "barrier.cta.red.and.pred p, 2, 64, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(out)
      : "r"(static_cast<uint32_t>(pred))
      : "memory");
  return out != 0;
}

// 16 lanes x N columns of fp32 accumulators as mma fragments: value 4 g + e of lane l is row (l >> 2) + 8 (e >> 1),
// column 8 g + 2 (l & 3) + (e & 1)
__device__ __forceinline__ void mla_ld_frag(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void mla_ld_frag(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// four 8 x 8 fragments stored transposed: lane i's address is row (i & 7) of matrix i >> 3
__device__ __forceinline__ void mla_stsm_x4_t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b),
               "r"(c), "r"(d)
               : "memory");
}

template <typename T, bool kExtend>
__global__ void __launch_bounds__(kMlaThreads, 1)
attn_mla_kernel(const __grid_constant__ CUtensorMap tmKV, const __grid_constant__ CUtensorMap tmR,
                const __grid_constant__ CUtensorMap tmQ, const MlaParams p) {
  using S = MlaShape<kExtend>;
  constexpr int N = S::N, TQ = S::TQ;
  extern __shared__ uint8_t mla_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(mla_smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem;                          // kPairs x 16 KB
  uint8_t* sR = sK + S::kPairs * 2 * kMlaBlk;  // kRopes x 8 KB
  uint8_t* sQ = sK + S::kRing;                 // 9 blocks of [N x 64]
  uint8_t* sP = sQ + S::kQBytes;               // [N x 64]
  uint64_t* t_full = reinterpret_cast<uint64_t*>(sP + S::kPBytes);  // [4]: tile t & 3 has landed
  uint64_t* k_empty = t_full + 4;                                   // [kPairs]
  uint64_t* r_empty = k_empty + S::kPairs;                          // [kRopes]
  uint64_t* s_full = r_empty + S::kRopes;                           // [2]
  uint64_t* s_empty = s_full + 2;                                   // [2]
  uint64_t* p_full = s_empty + 2;
  uint64_t* p_empty = p_full + 1;
  uint64_t* o_empty = p_full + 2;
  uint64_t* q_full = p_full + 3;
  uint64_t* q_empty = p_full + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(p_full + 5);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* s_start = reinterpret_cast<int*>(tmem_slot + 2);  // hg, r, j, units of the item before the range
  volatile int* s_gath = s_start + 4;                    // [4]: whether tile t & 3 was gathered
  int* s_slot = s_start + 8;                             // [64] slots of a gathered tile
  float* red = reinterpret_cast<float*>(s_slot + 64);    // [4][N]
  float* s_col = red + 4 * N;                            // [N]: rescale factors, then 1 / sum

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 6) {
    if (lane == 0) {
      for (int i = 0; i < 4; ++i) mbar_init(&t_full[i], 65);
      for (int i = 0; i < S::kPairs; ++i) mbar_init(&k_empty[i], 1);
      for (int i = 0; i < S::kRopes; ++i) mbar_init(&r_empty[i], 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(&s_full[i], 1);
        mbar_init(&s_empty[i], 4);
      }
      mbar_init(p_full, 128);
      mbar_init(p_empty, 1);
      mbar_init(o_empty, 4);
      mbar_init(q_full, kExtend ? 64 : 1);
      mbar_init(q_empty, 1);
      *dead = 0;
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, S::kTmem);
    tmem_relinquish();
  } else if (tid == 128) {
    tma_prefetch_desc(&tmKV);
    tma_prefetch_desc(&tmR);
    if constexpr (!kExtend) tma_prefetch_desc(&tmQ);
  }
  griddep_wait();

  // ---- this CTA's range of the tile list ----
  int* scan = reinterpret_cast<int*>(sK);
  const int per_thread = (p.batch + kMlaThreads - 1) / kMlaThreads;
  const int r0 = tid * per_thread, r1 = min(p.batch, r0 + per_thread);
  int sum = 0;
  for (int r = r0; r < r1; ++r) {
    prefetch_l2(p.req_pool_indices + r);  // read next, when the range is known
    sum += mla_request_tiles<kExtend>(p, r);
  }
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) scan[warp] = incl;
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // the merge's blocks wait for this grid's end beside its CTAs, instead of being launched then (from here on, since whatever
  // follows them may want tensor memory and this CTA has its own now)
  if (!p.snap) griddep_launch_dependents();
  int before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kMlaThreads / 32; ++w) {
    if (w < warp) before += scan[w];
    all += scan[w];
  }
  const int total = all * p.hgs;
  const int grid = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
  // Few units: two a CTA, but three where an item has just those and is not cut then (37 requests of 128 keys 12.7 -> 10.6 us,
  // 30 of 100 13.9 -> 11.8), and four where an item would have some 50 parts and their merge takes longer than two tiles (one
  // request of 8000 keys 18.8 -> 16.9, two 20.0 -> 17.2; three of 4000 keys with three a CTA 14.9 -> 17.7: not there).
  int least = p.min_tiles;
  if (!kExtend && !p.snap) least = all > 96 * p.batch ? 4 : all > 2 * p.batch && all <= 3 * p.batch ? 3 : least;
  const int per = max(least, (total + grid - 1) / grid);
  const int t_begin = min(total, per * cta), t_count = min(total, t_begin + per) - t_begin;
  if (t_count > 0) {
    const int hg = t_begin / all;
    int rem = t_begin - hg * all - (before + incl - sum);
    if (rem >= 0 && rem < sum) {  // exactly one thread: the one whose requests the range starts in
      int r = r0;
      for (;; ++r) {
        const int w = mla_request_tiles<kExtend>(p, r);
        if (rem < w) break;
        rem -= w;
      }
      int j = 0;
      if constexpr (kExtend) {
        int start, ext, prefix;
        mla_request(p, r, start, ext, prefix);
        int lo = 0, hi = (ext - 1) / TQ;  // last group that starts at or before unit `rem`
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (mla_group_tiles(prefix, mid) + mid * S::E <= rem) lo = mid; else hi = mid - 1;
        }
        j = lo;
        rem -= mla_group_tiles(prefix, j) + j * S::E;
      }
      s_start[0] = hg;
      s_start[1] = r;
      s_start[2] = j;
      s_start[3] = rem;
    }
  }
  fence_proxy_async_smem();  // the scan's generic writes to the tile area, before copies land there
  __syncthreads();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_O = tmem_base, tmem_S = tmem_base + S::kOCols;
  MlaCursor<kExtend> c;
  c.init(p, s_start, t_count);

  if (warp == 6) {
    // ===================== MMA issuer =====================
    // One copy of each step in one loop: straight-line code of 52 MMAs would stream through the instruction cache
    // (it ran at 190 clk per MMA).
    if (elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc<T>(64, N, 0, 0);   // A = K (K-major), B = Q (K-major)
      constexpr uint32_t idesc_o = umma_idesc<T>(128, S::kON, 1, 0);  // A = V^T (MN-major), B = P^T (K-major)
      // descriptors in halves: the upper one is a constant, the lower one moves by 16-byte units
      const uint64_t dk = umma_desc_sw128(smem_u32(sK), 16, 1024), dr = umma_desc_sw128(smem_u32(sR), 16, 1024);
      const uint32_t hi = static_cast<uint32_t>(dk >> 32), k_lo = static_cast<uint32_t>(dk), r_lo = static_cast<uint32_t>(dr);
      const uint32_t v_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sK), kMlaBlk, 1024));
      const uint32_t q_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sQ), 16, 1024));
      const uint32_t p_lo = static_cast<uint32_t>(umma_desc_sw128(smem_u32(sP), 16, 1024));
      int ts = 0, tp = 0;             // tiles whose S / PV has been issued
      uint32_t firsts = 0, segs = 0;  // bit (tile & 1): first tile of its item here; parity of its item's number
      bool cross = true;              // the next S belongs to another item than the last
      MlaSlot<S::kPairs> ks, kp;      // next pair of the S stream / of the PV stream
      MlaSlot<S::kRopes> rs;
      while (c.valid || tp < ts) {
        // S of the next tile goes before PV of this one if its rows have landed — and not across items, where its Q may
        // still be on the way: PV frees ring slots, so it never waits behind a copy
        if (c.valid && (ts == tp || (ts == tp + 1 && !cross && mbar_test(&t_full[ts & 3], (ts >> 2) & 1)))) {
          const int b = ts & 1;
          if (cross) mbar_wait_bounded(q_full, c.seg & 1, dead);
          firsts = (firsts & ~(1u << b)) | (cross ? 1u << b : 0u);
          segs = (segs & ~(1u << b)) | ((c.seg & 1) << b);
          mbar_wait_bounded(&s_empty[b], ((ts >> 1) & 1) ^ 1, dead);
          const uint32_t d = tmem_S + b * 2 * N;
          mbar_wait_bounded(&t_full[ts & 3], (ts >> 2) & 1, dead);
          if ((kExtend && cross) || s_gath[ts & 3]) fence_proxy_async_smem();  // extend's Q and gathered tiles come by cp.async
          tc_fence_after_sync();
          // two accumulators in turn; the softmax adds them
          uint32_t qa = q_lo;
#pragma unroll 1
          for (int i = 0; i < 4; ++i) {
            const uint32_t ka = k_lo + ks.i * (2 * kMlaBlk >> 4);
            ks.next();
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_ss_lo(d + (kk & 1) * N, ka + (kk >> 2) * (kMlaBlk >> 4) + (kk & 3) * 2,
                         qa + (kk >> 2) * (N * 128 >> 4) + (kk & 3) * 2, hi, idesc_s, (i > 0 || kk > 1) ? 1u : 0u);
            qa += 2 * (N * 128 >> 4);
          }
          const uint32_t ra = r_lo + rs.i * (kMlaBlk >> 4);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_ss_lo(d + (kk & 1) * N, ra + kk * 2, qa + kk * 2, hi, idesc_s, 1u);
          umma_commit(&r_empty[rs.i]);
          rs.next();
          umma_commit(&s_full[b]);
          cross = c.ends(p);
          if (cross) umma_commit(q_empty);
          ++ts;
          c.next(p);
          continue;
        }
        const int b = tp & 1;
        mbar_wait_bounded(p_full, tp & 1, dead);
        const bool first = (firsts >> b) & 1;
        if (first) mbar_wait_bounded(o_empty, ((segs >> b) & 1) ^ 1, dead);
        tc_fence_after_sync();  // (P's writers have fenced; the rows were fenced for S)
#pragma unroll 1
        for (int i = 0; i < 4; i += 2) {  // two blocks of 128 value columns in turn
          const int slot0 = kp.i;
          kp.next();
          const int slot1 = kp.i;
          kp.next();
          const uint32_t v0 = v_lo + slot0 * (2 * kMlaBlk >> 4), v1 = v_lo + slot1 * (2 * kMlaBlk >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t acc = (!first || k > 0) ? 1u : 0u;
            umma_ss_lo(tmem_O + i * S::kON, v0 + k * 128, p_lo + k * 2, hi, idesc_o, acc);
            umma_ss_lo(tmem_O + (i + 1) * S::kON, v1 + k * 128, p_lo + k * 2, hi, idesc_o, acc);
          }
          umma_commit(&k_empty[slot0]);
          umma_commit(&k_empty[slot1]);
        }
        umma_commit(p_empty);
        ++tp;
      }
    }
  } else if (!kExtend && warp >= 4) {
    // ===================== loaders, decode =====================
    // Each warp looks at all 64 rows of a tile: warp 4 copies full tiles, warp 5 an item's Q (which may
    // have to wait for the last S of the item before), both gather.  The five copies of a tile go out by five lanes, each
    // when its slot is free: one lane after the other took 3650 clk a tile, more than the tile's time in memory.
    const T* pool = reinterpret_cast<const T*>(p.kv_pool);
    const int half = warp - 4;
    // a row is read once unless there are more heads than an item has: first to leave the L2, 64 requests 27.2 -> 26.3 us
    const uint64_t policy = p.hgs == 1 ? kEvictFirst : kEvictNormal;
    int t = 0, gather_age = 4;  // gather_age: tiles since one was gathered
    const int32_t* page = nullptr;
    int page_r = -1;
    auto lookup = [&](const MlaCursor<kExtend>& cc, int& base, int& s0, int& s1) {
      if (cc.it.r != page_r) {
        page_r = cc.it.r;
        page = p.req_to_token + p.req_pool_indices[page_r] * p.rtt_stride;
      }
      const int pos = cc.tile * kMlaTile, end = cc.it.load_end;
      base = pos + kMlaTile <= end ? __ldg(page + pos) : -1;  // a full tile: candidate TMA row
      s0 = pos + lane < end ? __ldg(page + pos + lane) : -1;
      s1 = pos + 32 + lane < end ? __ldg(page + pos + 32 + lane) : -1;
    };
    MlaSlot<S::kPairs> ks;
    MlaSlot<S::kRopes> rs;
    int base = -1, s0 = -1, s1 = -1;
    if (c.valid) lookup(c, base, s0, s1);
    bool first = true;
    while (c.valid) {
      const int row0 = c.it.row0, hg = c.it.hg, seg = c.seg;
      const bool load_q = first;
      first = c.ends(p);
      c.next(p);
      int nbase = -1, n0 = -1, n1 = -1;
      if (c.valid) lookup(c, nbase, n0, n1);  // the next tile's page-table entries, off the critical path
      const bool contig = __all_sync(0xffffffffu, base >= 0 && s0 == base + lane && s1 == base + 32 + lane);
      // tile by tile together: a warp ahead or behind by two rounds of a slot would take one phase of its barrier for another
      mla_loader_bar();
      if (half == 1 && load_q && lane == 0) {
        mbar_wait_bounded(q_empty, (seg & 1) ^ 1, dead);
        mbar_expect_tx(q_full, S::kQBytes);
        tma_load_4d(sQ, &tmQ, q_full, 0, hg * kMlaHeads, p.q_row0 + p.q_dir * row0, 0, kEvictFirst);
      }
      __syncwarp();
      gather_age = contig ? gather_age + 1 : 0;
      uint64_t* full = &t_full[t & 3];
      if (contig) {
        if (half == 0) {
          if (lane == 0) {
            s_gath[t & 3] = 0;
            mbar_expect_tx(full, 9 * kMlaBlk);
          }
          __syncwarp();
          if (gather_age < 4) fence_proxy_async_smem();  // the slots may last have been written by the gather path
          int at = ks.i + lane;  // of lanes 0-3; lane 4: the rope block
          uint32_t round = ks.round;
          if (at >= S::kPairs) {
            at -= S::kPairs;
            round ^= 1;
          }
          uint64_t* empty = lane < 4 ? &k_empty[at] : &r_empty[rs.i];
          if (lane == 4) round = rs.round;
          bool todo = lane < 5;
#pragma unroll 1
          for (int i = 0; __any_sync(0xffffffffu, todo); ++i) {
            if (todo && (mbar_test(empty, round ^ 1) || *dead || i == kMbarWaitTries)) {
              if (i == kMbarWaitTries) *dead = 1;
              if (lane < 4)
                tma_load_3d(sK + at * 2 * kMlaBlk, &tmKV, full, 0, base, 2 * lane, policy);
              else
                tma_load_2d(sR + rs.i * kMlaBlk, &tmR, full, kMlaDV, base, policy);
              todo = false;
            }
          }
          if (lane == 0) mbar_arrive_n(full, 64);
        }
#pragma unroll
        for (int st = 0; st < 4; ++st) ks.next();
        rs.next();
      } else {
        if (half == 0 && lane == 0) s_gath[t & 3] = 1;
#pragma unroll 1
        for (int st = 0; st < 5; ++st) {
          uint8_t* dst = st < 4 ? sK + ks.i * 2 * kMlaBlk : sR + rs.i * kMlaBlk;
          mbar_wait_bounded(st < 4 ? &k_empty[ks.i] : &r_empty[rs.i], (st < 4 ? ks.round : rs.round) ^ 1, dead);
          __syncwarp();
          const int shift = st < 4 ? 4 : 3;  // log2 of the 16-byte chunks of a row in a pair / in the rope block
#pragma unroll 4
          for (int i = half * 32 + lane; i < kMlaTile << shift; i += 64) {
            const int row = i >> shift, ch = i - (row << shift);
            const int a = __shfl_sync(0xffffffffu, s0, row & 31), b = __shfl_sync(0xffffffffu, s1, row & 31);
            const int sl = row < 32 ? a : b;
            cp_async16(smem_u32(dst + (ch >> 3) * kMlaBlk + mla_off(row, ch & 7)),
                       pool + static_cast<int64_t>(sl < 0 ? 0 : sl) * kMlaDL + st * 128 + ch * 8, sl >= 0);
          }
          if (st < 4) ks.next(); else rs.next();
        }
        cp_async_mbar_arrive_noinc(full);
        if (half == 0 && lane == 0) mbar_arrive(full);
      }
      ++t;
      base = nbase;
      s0 = n0;
      s1 = n1;
    }
    cp_async_commit();
    cp_async_wait<0>();
  } else if (warp >= 4) {
    // ===================== loaders, extend =====================
    const int lt = tid - 128;  // 0..63: also the row of a tile this thread looks up
    const T* pool = reinterpret_cast<const T*>(p.kv_pool);
    int t = 0, gather_age = 4;  // gather_age: tiles since one was gathered
    auto lookup = [&](const MlaCursor<kExtend>& cc, int& base) {
      const int32_t* page = p.req_to_token + p.req_pool_indices[cc.it.r] * p.rtt_stride;
      const int pos = cc.tile * kMlaTile;
      base = pos + kMlaTile <= cc.it.load_end ? __ldg(page + pos) : -1;  // a full tile: candidate TMA row
      return pos + lt < cc.it.load_end ? __ldg(page + pos + lt) : -1;
    };
    MlaSlot<S::kPairs> ks;
    MlaSlot<S::kRopes> rs;
    int base = -1, slot = -1;
    if (c.valid) slot = lookup(c, base);
    bool first = true;
    while (c.valid) {
      const MlaItem it = c.it;
      const int seg = c.seg;
      const bool load_q = first;
      first = c.ends(p);
      c.next(p);
      int nbase = -1, nslot = -1;
      if (c.valid) nslot = lookup(c, nbase);  // the next tile's page-table entries, off the critical path
      const bool contig = mla_loader_and(base >= 0 && slot == base + lt);
      if (lt == 0) s_gath[t & 3] = !contig;  // published by this thread's extra arrival below
      gather_age = contig ? gather_age + 1 : 0;
      if (!contig) {
        s_slot[lt] = slot;  // (both warps have passed the barrier above: the previous tile's rows have been read)
        mla_loader_and(true);
      }
      uint64_t* full = &t_full[t & 3];
      if (contig) {
        if (lt == 0) {
          if (gather_age < 4) fence_proxy_async_smem();  // the slots may last have been written by the gather path
          mbar_expect_tx(full, 9 * kMlaBlk);
#pragma unroll 1
          for (int st = 0; st < 4; ++st) {
            mbar_wait_bounded(&k_empty[ks.i], ks.round ^ 1, dead);
            tma_load_3d(sK + ks.i * 2 * kMlaBlk, &tmKV, full, 0, base, 2 * st, kEvictNormal);
            ks.next();
          }
          mbar_wait_bounded(&r_empty[rs.i], rs.round ^ 1, dead);
          tma_load_2d(sR + rs.i * kMlaBlk, &tmR, full, kMlaDV, base, kEvictNormal);
          rs.next();
          mbar_arrive_n(full, 64);
        } else {
          for (int st = 0; st < 4; ++st) ks.next();
          rs.next();
        }
      } else {
#pragma unroll 1
        for (int st = 0; st < 5; ++st) {
          uint8_t* dst = st < 4 ? sK + ks.i * 2 * kMlaBlk : sR + rs.i * kMlaBlk;
          mbar_wait_bounded(st < 4 ? &k_empty[ks.i] : &r_empty[rs.i], (st < 4 ? ks.round : rs.round) ^ 1, dead);
          const int shift = st < 4 ? 4 : 3;  // log2 of the 16-byte chunks of a row in a pair / in the rope block
#pragma unroll 4
          for (int i = lt; i < kMlaTile << shift; i += 64) {
            const int row = i >> shift, ch = i - (row << shift);
            const int s = s_slot[row];
            cp_async16(smem_u32(dst + (ch >> 3) * kMlaBlk + mla_off(row, ch & 7)),
                       pool + static_cast<int64_t>(s < 0 ? 0 : s) * kMlaDL + st * 128 + ch * 8, s >= 0);
          }
          if (st < 4) ks.next(); else rs.next();
        }
        cp_async_mbar_arrive_noinc(full);
        if (lt == 0) mbar_arrive(full);
      }
      if (load_q) {
        // the item's N query rows (token, head), zero where there is none; the tile above is already on its way
        mbar_wait_bounded(q_empty, (seg & 1) ^ 1, dead);
        const T* qb = reinterpret_cast<const T*>(p.q);
        const int h0 = it.hg * kMlaHeads, nh = min(kMlaHeads, p.H - h0);
#pragma unroll 4
        for (int i = lt; i < N * 72; i += 64) {
          const int col = i / 72, ch = i - col * 72;
          const int tok = col >> 4, h = col & 15;
          const bool ok = tok < it.ntok && h < nh;
          cp_async16(smem_u32(sQ + (ch >> 3) * (N * 128) + mla_off(col, ch & 7)),
                     qb + (ok ? (it.row0 + tok) * p.q_stride + static_cast<int64_t>(h0 + h) * kMlaDL + ch * 8 : 0), ok);
        }
        cp_async_mbar_arrive_noinc(q_full);
      }
      ++t;
      base = nbase;
      slot = nslot;
    }
    cp_async_commit();
    cp_async_wait<0>();
  } else {
    // ===================== softmax / correction / epilogue =====================
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    constexpr int C = N / 4;  // columns of this thread: 8 (i >> 1) + 2 (lane & 3) + (i & 1)
    const int col0 = 2 * (lane & 3);
    if (tid == 0 && !p.snap) {
      // what the merge kernel needs of an item that began in an earlier CTA and ends here
      int* info = p.info + (p.by_item ? c.it.hg * p.batch + c.it.r : cta) * 8;
      const bool tail = t_count > 0 && c.tile > 0 && c.it.ntiles - c.tile <= t_count;
      if (tail || !p.by_item) info[0] = tail;
      if (tail) {
        info[1] = (t_begin - c.tile) / per;  // CTA of the item's first tile (tiles are consecutive units)
        info[2] = c.it.row0;
        info[3] = c.it.ntok;
        info[4] = c.it.hg * kMlaHeads;
        info[5] = cta;
      }
    }
    int t = 0;
    while (c.valid) {
      const MlaItem it = c.it;
      const int tile0 = c.tile;
      int tile_last = tile0;
      float m_ref[C], l_thr[C];
#pragma unroll
      for (int i = 0; i < C; ++i) { m_ref[i] = -INFINITY; l_thr[i] = 0.f; }
      bool end = false;
      while (!end) {
        end = c.ends(p);
        tile_last = c.tile;
        const int kv0 = c.tile * kMlaTile;
        const bool first = c.tile == tile0;
        c.next(p);
        const int sb = t & 1;
        mbar_wait_bounded(&s_full[sb], (t >> 1) & 1, dead);
        tc_fence_after_sync();
        uint32_t r[N / 2], r2[N / 2];
        mla_ld_frag(tmem_S + lane_base + sb * 2 * N, r);
        mla_ld_frag(tmem_S + lane_base + sb * 2 * N + N, r2);
        tmem_ld_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_empty[sb]);
        float s[N / 2];
        const int pos = kv0 + warp * 16 + (lane >> 2);
        const bool all_seen = kv0 + kMlaTile - 1 <= it.p0;  // every column sees the whole tile
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
          const float v = (__uint_as_float(r[i]) + __uint_as_float(r2[i])) * p.scale_log2;
          s[i] = all_seen || pos + 8 * ((i >> 1) & 1) <= it.p0 + (i >> 3) ? v : -INFINITY;  // i >> 3: the column's token
        }
        bool exceed = false;
#pragma unroll
        for (int i = 0; i < N / 2; ++i) exceed |= s[i] > m_ref[(i >> 2) * 2 + (i & 1)] + S::kLag;
        if (mla_bar_or(exceed)) {
          // The running max per column.  Where P has one part it is the true one, so that a column's largest P is exactly 1: a
          // reference that lags by up to 2^8 saves most of these rescales (900 of 1500 clk from S to P) but rounds that P
          // too (extend 548 instead of 600 us, but 6 - 14 % more rms error against 64-bit results).  With two parts
          // nothing is rounded that counts.
#pragma unroll
          for (int i = 0; i < C; ++i) {
            float m = fmaxf(s[(i >> 1) * 4 + (i & 1)], s[(i >> 1) * 4 + 2 + (i & 1)]);
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
            if (lane < 4) red[warp * N + (i >> 1) * 8 + col0 + (i & 1)] = m;
          }
          mla_bar();
#pragma unroll
          for (int i = 0; i < C; ++i) {
            const int col = (i >> 1) * 8 + col0 + (i & 1);
            const float mt = fmaxf(fmaxf(red[col], red[N + col]), fmaxf(red[2 * N + col], red[3 * N + col]));
            const float m_new = fmaxf(m_ref[i], mt);
            // (a column that has seen no key yet has nothing to scale; -inf - -inf stays out)
            const float alpha = m_ref[i] == -INFINITY ? 0.f : fast_exp2(m_ref[i] - m_new);
            l_thr[i] *= alpha;
            m_ref[i] = m_new;
            if (tid < 4) s_col[col] = alpha;
          }
          mla_bar();
          if (!first) {
            mbar_wait_bounded(p_empty, (t & 1) ^ 1, dead);  // PV of the previous tile has finished: O^T is stable
            tc_fence_after_sync();
#pragma unroll 1
            for (int cc = 0; cc < S::kOCols; cc += 16) {
              uint32_t o[16];
              tmem_ld_32x32b_x16(tmem_O + lane_base + cc, o);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * s_col[(cc & (N - 1)) + e]);
              tmem_st_32x32b_x16(tmem_O + lane_base + cc, o);
            }
            tmem_st_wait();
            tc_fence_before_sync();
          }
          mla_bar();  // red / s_col may be written again
        }
        // P^T -> shared memory (B operand, K-major: row = column of the item, 64 kv); sums of what is multiplied
        uint32_t pk[N / 4], pk2[S::kPParts == 2 ? N / 4 : 1];
#pragma unroll
        for (int g = 0; g < N / 8; ++g)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const float m0 = m_ref[2 * g] == -INFINITY ? 0.f : m_ref[2 * g];
            const float m1 = m_ref[2 * g + 1] == -INFINITY ? 0.f : m_ref[2 * g + 1];
            const float p0 = fast_exp2(s[4 * g + 2 * x] - m0), p1 = fast_exp2(s[4 * g + 2 * x + 1] - m1);
            pk[2 * g + x] = pack2<T>(p0, p1);
            const float2 v = unpack2<T>(pk[2 * g + x]);
            if constexpr (S::kPParts == 2) {
              pk2[2 * g + x] = pack2<T>(p0 - v.x, p1 - v.y);
              l_thr[2 * g] += p0;
              l_thr[2 * g + 1] += p1;
            } else {
              l_thr[2 * g] += v.x;
              l_thr[2 * g + 1] += v.y;
            }
          }
        mbar_wait_bounded(p_empty, (t & 1) ^ 1, dead);
#pragma unroll
        for (int g = 0; g < N / 8; g += 2) {
          // matrices: (columns 8 g.., kv 0-7), (8 g.., kv 8-15), (8 (g + 1).., kv 0-7), (8 (g + 1).., kv 8-15)
          const int row = 8 * (g + (lane >> 4)) + (lane & 7);
          const uint32_t at = smem_u32(sP + mla_off(row, warp * 2 + ((lane >> 3) & 1)));
          mla_stsm_x4_t(at, pk[2 * g], pk[2 * g + 1], pk[2 * g + 2], pk[2 * g + 3]);
          if constexpr (S::kPParts == 2)
            mla_stsm_x4_t(at + S::kPPart, pk2[2 * g], pk2[2 * g + 1], pk2[2 * g + 2], pk2[2 * g + 3]);
        }
        fence_proxy_async_smem();
        mbar_arrive(p_full);
        ++t;
      }
      // ---- epilogue: column sums over the kv rows of all tiles, then O^T / sum (or the partial as it is) ----
      const bool whole = tile0 == 0 && tile_last + 1 == it.ntiles;
      if (tid == 0 && whole && p.by_item) p.info[(it.hg * p.batch + it.r) * 8] = 0;
      const int h0 = it.hg * kMlaHeads, nh = min(kMlaHeads, p.H - h0), nhm = min(kMlaHeads, p.H);
      const int64_t part0 = static_cast<int64_t>(2 * cta + (tile0 > 0 ? 0 : 1)) * p.cols;
#pragma unroll
      for (int i = 0; i < C; ++i) {
        float l = l_thr[i];
        l += __shfl_xor_sync(0xffffffffu, l, 4);
        l += __shfl_xor_sync(0xffffffffu, l, 8);
        l += __shfl_xor_sync(0xffffffffu, l, 16);
        if (lane < 4) red[warp * N + (i >> 1) * 8 + col0 + (i & 1)] = l;
      }
      mla_bar();
      if (tid < 4) {
#pragma unroll
        for (int i = 0; i < C; ++i) {
          const int col = (i >> 1) * 8 + col0 + (i & 1);
          const float l = (red[col] + red[N + col]) + (red[2 * N + col] + red[3 * N + col]);
          s_col[col] = l > 0.f ? 1.f / l : 0.f;
          const int tok = col >> 4, h = col & 15;
          if (!whole && tok < it.ntok && h < nh) {
            float* ml = p.ml_part + (part0 + tok * nhm + h) * 2;
            ml[0] = m_ref[i];
            ml[1] = l;
          }
        }
      }
      mla_bar();
      mbar_wait_bounded(p_empty, (t - 1) & 1, dead);  // the last PV of the item has finished
      tc_fence_after_sync();
      T* out = reinterpret_cast<T*>(p.out) + it.row0 * p.out_stride + static_cast<int64_t>(h0) * kMlaDV + warp * 32;
      float z[2] = {0.f, 0.f};  // kExtend: NaN when an output is infinite or NaN
      if (whole) {
        // neighbouring lanes swap halves of two columns: 4-byte stores, 64 bytes of a row per half warp
        const bool odd = lane & 1;
        T* dst = out + (lane & ~1) + (odd ? kMlaDV : 0);
#pragma unroll 1
        for (int blk = 0; blk < 4; ++blk, dst += 128) {
          uint32_t o[N];
#pragma unroll
          for (int cc = 0; cc < N; cc += 16) tmem_ld_32x32b_x16(tmem_O + lane_base + blk * S::kON + cc, o + cc);
          if constexpr (S::kPParts == 2) {
            uint32_t lo[N];
            tmem_ld_32x32b_x16(tmem_O + lane_base + blk * S::kON + N, lo);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < N; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) + __uint_as_float(lo[e]));
          } else {
            tmem_ld_wait();
          }
#pragma unroll
          for (int cc = 0; cc < N; cc += 16) {
            if ((cc >> 4) >= it.ntok) break;
            if constexpr (kExtend) {
#pragma unroll
              for (int e = 0; e < 16; ++e) z[e & 1] = fmaf(__uint_as_float(o[cc + e]), 0.f, z[e & 1]);
            }
            T* row = dst + (cc >> 4) * p.out_stride;
#pragma unroll
            for (int e = 0; e < 16; e += 4) {
              const float4 f = *reinterpret_cast<const float4*>(s_col + cc + e);
              const float a0 = __uint_as_float(o[cc + e]) * f.x, a1 = __uint_as_float(o[cc + e + 1]) * f.y;
              const float b0 = __uint_as_float(o[cc + e + 2]) * f.z, b1 = __uint_as_float(o[cc + e + 3]) * f.w;
              const float ga = __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, 1);
              const float gb = __shfl_xor_sync(0xffffffffu, odd ? b0 : b1, 1);
              if (e + odd < nh) *reinterpret_cast<uint32_t*>(row + e * kMlaDV) = odd ? pack2<T>(ga, a1) : pack2<T>(a0, ga);
              if (e + 2 + odd < nh)
                *reinterpret_cast<uint32_t*>(row + (e + 2) * kMlaDV) = odd ? pack2<T>(gb, b1) : pack2<T>(b0, gb);
            }
          }
        }
      } else {
        float* dst = p.o_part + part0 * kMlaDV + warp * 32 + lane;
#pragma unroll 1
        for (int blk = 0; blk < 4; ++blk, dst += 128) {
          uint32_t o[N];
#pragma unroll
          for (int cc = 0; cc < N; cc += 16) tmem_ld_32x32b_x16(tmem_O + lane_base + blk * S::kON + cc, o + cc);
          if constexpr (S::kPParts == 2) {
            uint32_t lo[N];
            tmem_ld_32x32b_x16(tmem_O + lane_base + blk * S::kON + N, lo);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < N; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) + __uint_as_float(lo[e]));
          } else {
            tmem_ld_wait();
          }
#pragma unroll
          for (int cc = 0; cc < N; cc += 16) {
            if ((cc >> 4) >= it.ntok) break;
            if constexpr (kExtend) {
#pragma unroll
              for (int e = 0; e < 16; ++e) z[e & 1] = fmaf(__uint_as_float(o[cc + e]), 0.f, z[e & 1]);
            }
            float* row = dst + static_cast<int64_t>((cc >> 4) * nhm) * kMlaDV;
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (e < nh) row[e * kMlaDV] = __uint_as_float(o[cc + e]);
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(o_empty);
      if constexpr (kExtend) {
        // The tiles hold rows that some or all of the item's tokens may not see.  Their P is 0, but 0 times an infinite or
        // NaN value is NaN: an output that is not finite is computed again from the visible keys, where such a row was there.  (Looking at every output and the
        // barrier: 600 -> 603 us for a layer of 4096 new tokens.)
        if (mla_bar_or(isnan(z[0] + z[1]))) {
          if (tid < 4) {
#pragma unroll
            for (int i = 0; i < C; ++i) red[(i >> 1) * 8 + col0 + (i & 1)] = m_ref[i];
          }
          const int32_t* page = p.req_to_token + p.req_pool_indices[it.r] * p.rtt_stride;
          const T* pool = reinterpret_cast<const T*>(p.kv_pool);
          const int end_key = min(it.load_end, (tile_last + 1) * kMlaTile);
          const int hid0 = max(it.p0 + 1, tile0 * kMlaTile);  // from here on some token does not see the rows
          bool odd_v = false;
#pragma unroll 1
          for (int i = tid; i < (end_key - hid0) * (kMlaDV / 8); i += 128) {
            const Vec16<T> x = ldv(pool + static_cast<int64_t>(page[hid0 + i / (kMlaDV / 8)]) * kMlaDL + i % (kMlaDV / 8) * 8);
#pragma unroll
            for (int e = 0; e < 8; ++e) odd_v |= !(fabsf(to_f32<T>(x.e()[e])) <= 3.4028235e38f);
          }
          if (mla_bar_or(odd_v)) {
            float* pk_s = red + 2 * N;  // probabilities of 128 keys
            const T* qb = reinterpret_cast<const T*>(p.q) + it.row0 * p.q_stride + static_cast<int64_t>(h0) * kMlaDL;
#pragma unroll 1
            for (int col = 0; col < it.ntok * kMlaHeads; ++col) {
              const int tok = col >> 4, h = col & 15;
              if (h >= nh) continue;
              const T* qr = qb + tok * p.q_stride + h * kMlaDL;
              const int seen = min(end_key, it.p0 + tok + 1);
              const float m = red[col];
              float acc[4] = {0.f, 0.f, 0.f, 0.f};  // value columns 4 tid ..
#pragma unroll 1
              for (int k0 = tile0 * kMlaTile; k0 < seen; k0 += 128) {
                float dot = 0.f;
                if (k0 + tid < seen) {
                  const T* kr = pool + static_cast<int64_t>(page[k0 + tid]) * kMlaDL;
#pragma unroll 1
                  for (int d = 0; d < kMlaDL; d += 8) {
                    const Vec16<T> a = ldv(qr + d), b = ldv(kr + d);
#pragma unroll
                    for (int e = 0; e < 8; ++e) dot = fmaf(to_f32<T>(a.e()[e]), to_f32<T>(b.e()[e]), dot);
                  }
                }
                pk_s[tid] = to_f32<T>(from_f32<T>(fast_exp2(dot * p.scale_log2 - m)));
                mla_bar();
#pragma unroll 1
                for (int i = 0; i < min(128, seen - k0); ++i) {
                  const T* vr = pool + static_cast<int64_t>(page[k0 + i]) * kMlaDL + tid * 4;
#pragma unroll
                  for (int e = 0; e < 4; ++e) acc[e] = fmaf(pk_s[i], to_f32<T>(vr[e]), acc[e]);
                }
                mla_bar();
              }
              if (whole) {
                T* row = reinterpret_cast<T*>(p.out) + (it.row0 + tok) * p.out_stride +
                         static_cast<int64_t>(h0 + h) * kMlaDV + tid * 4;
#pragma unroll
                for (int e = 0; e < 4; ++e) row[e] = from_f32<T>(acc[e] * s_col[col]);
              } else {
                float* row = p.o_part + (part0 + tok * nhm + h) * kMlaDV + tid * 4;
#pragma unroll
                for (int e = 0; e < 4; ++e) row[e] = acc[e];
              }
            }
          }
        }
      }
      mla_bar();  // red / s_col belong to the next item
    }
  }

  if (p.snap) griddep_launch_dependents();
  tc_fence_before_sync();
  __syncthreads();
  if (*dead) {
    wait_drain();
    if (tid == 0) wait_report(p.wait_expired);
  }
  if (warp == 6) tmem_dealloc(tmem_base, S::kTmem);
}

// Merges the parts of the items that span several CTAs.  Block (c, 4 columns) serves the item that ends in CTA c after
// beginning in CTA info[1] < c: that CTA left its part in slot 2 info[1] + 1, the following ones up to c in slot 2 i.
// info: {any, first CTA, first query row, tokens, first head, last CTA}.
template <typename T>
__global__ void __launch_bounds__(512)
mla_merge_kernel(const MlaParams p) {
  griddep_launch_dependents();
  griddep_wait();
  const int c = blockIdx.x, nhm = min(kMlaHeads, p.H);
  const int* info = p.info + c * 8;
  if (!info[0]) return;
  const int col = blockIdx.y * 4 + (threadIdx.x >> 7), x = threadIdx.x & 127;
  const int tok = col / nhm, h = col % nhm;
  if (tok >= info[3] || info[4] + h >= p.H) return;
  const int c0 = info[1];
  auto at = [&](int i) { return static_cast<int64_t>(i == c0 ? 2 * i + 1 : 2 * i) * p.cols + col; };
  float M = -INFINITY;
  for (int i = c0; i <= c; ++i) M = fmaxf(M, p.ml_part[at(i) * 2]);  // (-inf where a part saw no key)
  float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
  float den = 0.f;
#pragma unroll 4
  for (int i = c0; i <= c; ++i) {
    const float2 ml = *reinterpret_cast<const float2*>(p.ml_part + at(i) * 2);
    const float4 o = *reinterpret_cast<const float4*>(p.o_part + at(i) * kMlaDV + x * 4);
    const float w = ml.y > 0.f ? fast_exp2(ml.x - M) : 0.f;
    num.x = fmaf(w, o.x, num.x);
    num.y = fmaf(w, o.y, num.y);
    num.z = fmaf(w, o.z, num.z);
    num.w = fmaf(w, o.w, num.w);
    den = fmaf(w, ml.y, den);
  }
  const float inv = den > 0.f ? 1.f / den : 0.f;
  T* dst = reinterpret_cast<T*>(p.out) + (static_cast<int64_t>(info[2]) + tok) * p.out_stride +
           static_cast<int64_t>(info[4] + h) * kMlaDV + x * 4;
  *reinterpret_cast<uint2*>(dst) = make_uint2(pack2<T>(num.x * inv, num.y * inv), pack2<T>(num.z * inv, num.w * inv));
}

// The same for few items, which then have many parts each (one request of 8000 keys: 63, read in 20 us by one thread after
// the other part).  Block (item, column): a warp takes 32 of the column's 512 values, each quarter of it every fourth part
// with eight on the way; the quarters meet by shuffles, since shared memory would keep the blocks from waiting beside the
// attention's CTAs.  (Where an item has two or three parts the shuffles cost more than they save: 27.2 -> 28.2 us for 64
// requests of 1088 keys.)
template <typename T>
__global__ void __launch_bounds__(512)
mla_merge_many_kernel(const MlaParams p) {
  griddep_launch_dependents();
  griddep_wait();
  const int* info = p.info + blockIdx.x * 8;
  const int col = blockIdx.y;  // a head of the item's one token
  if (!info[0] || info[4] + col >= p.H) return;
  const int lane = threadIdx.x & 31, g = lane >> 3, x = (threadIdx.x >> 5) * 8 + (lane & 7);
  const int c0 = info[1], c = info[5];
  auto at = [&](int i) { return static_cast<int64_t>(i == c0 ? 2 * i + 1 : 2 * i) * p.cols + col; };
  const float2* ml = reinterpret_cast<const float2*>(p.ml_part);
  const float4* o_part = reinterpret_cast<const float4*>(p.o_part) + x;
  float M = -INFINITY, den = 0.f;
  float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int i = c0 + g; i <= c; i += 4) M = fmaxf(M, ml[at(i)].x);  // (-inf where a part saw no key)
  M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, 8));
  M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, 16));
#pragma unroll 8
  for (int i = c0 + g; i <= c; i += 4) {
    const float2 v = ml[at(i)];
    const float4 o = o_part[at(i) * (kMlaDV / 4)];
    const float w = v.y > 0.f ? fast_exp2(v.x - M) : 0.f;
    num.x = fmaf(w, o.x, num.x);
    num.y = fmaf(w, o.y, num.y);
    num.z = fmaf(w, o.z, num.z);
    num.w = fmaf(w, o.w, num.w);
    den = fmaf(w, v.y, den);
  }
  auto all4 = [](float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
  };
  const float d = all4(den), n0 = all4(num.x), n1 = all4(num.y), n2 = all4(num.z), n3 = all4(num.w);
  const float inv = d > 0.f ? 1.f / d : 0.f;
  if (g == 0)
    *reinterpret_cast<uint2*>(reinterpret_cast<T*>(p.out) + static_cast<int64_t>(info[2]) * p.out_stride +
                              static_cast<int64_t>(info[4] + col) * kMlaDV + x * 4) =
        make_uint2(pack2<T>(n0 * inv, n1 * inv), pack2<T>(n2 * inv, n3 * inv));
}

// What stands between the fused q / latent projection and the attention, one CTA per token: the latent row (RMS norm of
// its 512 columns, rotation of its 64) goes to its cache slot, the rotated part of every query head to its place behind
// the absorbed part, or back to where it was (q_rot: head 0's, in either case).  Replaces four launches (norm in place, rotation in place, cache write, a strided copy of the rotated
// queries: 8.2 + 7.9 + 5.5 + 12.5 us at 4096 tokens); it moves 13 KB a token, what bounds it is latency at small batches.
template <typename T>
__global__ void __launch_bounds__(256)
mla_rotary_store_kernel(T* q_rot, const T* qa, T* __restrict__ pool, const T* __restrict__ w,
                        const float* __restrict__ cos_sin, const int64_t* __restrict__ positions,
                        const int64_t* __restrict__ loc, int H, int nope, int64_t qa_stride, int64_t q_rot_stride,
                        int q_head_stride, float eps) {
  constexpr int kRot = kMlaDL - kMlaDV;
  __shared__ float part[2];
  griddep_launch_dependents();
  griddep_wait();
  const int64_t t = blockIdx.x;
  const int tid = threadIdx.x, q_size = H * (nope + kRot);
  const T* row = qa + t * qa_stride;
  T* dst = pool + loc[t] * kMlaDL;
  if (tid < 64) {  // the norm: eight columns per thread of two warps
    const Vec16<T> x = ldv(row + q_size + tid * 8), wv = ldv(w + tid * 8);
    float f[8], ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      f[i] = to_f32<T>(x.e()[i]);
      ss += f[i] * f[i];
    }
    ss = warp_sum(ss);
    if ((tid & 31) == 0) part[tid >> 5] = ss;
    asm volatile("bar.sync 1, 64;" ::: "memory");
    const float inv = rsqrtf((part[0] + part[1]) / static_cast<float>(kMlaDV) + eps);
    Vec16<T> o;
#pragma unroll
    for (int i = 0; i < 8; ++i) o.e()[i] = from_f32<T>(f[i] * inv * to_f32<T>(wv.e()[i]));
    stv(dst + tid * 8, o);
    return;
  }
  const float* cs = cos_sin + positions[t] * kRot;  // cos of the 32 pairs, then sin
  for (int i = tid - 64; i < (H + 1) * (kRot / 8); i += 192) {
    const int h = i >> 3, c = i & 7;  // four (even, odd) pairs of head h, or of the latent's own rotated part
    const Vec16<T> x = ldv(h < H ? row + h * (nope + kRot) + nope + c * 8 : row + q_size + kMlaDV + c * 8);
    const float4 cv = *reinterpret_cast<const float4*>(cs + c * 4), sv = *reinterpret_cast<const float4*>(cs + kRot / 2 + c * 4);
    const float co[4] = {cv.x, cv.y, cv.z, cv.w}, si[4] = {sv.x, sv.y, sv.z, sv.w};
    Vec16<T> o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = to_f32<T>(x.e()[2 * j]), b = to_f32<T>(x.e()[2 * j + 1]);
      o.e()[2 * j] = from_f32<T>(a * co[j] - b * si[j]);
      o.e()[2 * j + 1] = from_f32<T>(b * co[j] + a * si[j]);
    }
    stv(h < H ? q_rot + t * q_rot_stride + static_cast<int64_t>(h) * q_head_stride + c * 8 : dst + kMlaDV + c * 8, o);
  }
}

template <typename T, bool kExtend>
static int mla_launch(MlaParams p, int grid, cudaStream_t st) {
  CUtensorMap tm, tr, tq{};
  // the C-ABI does not carry the pool's slot count: rows are slot ids read from req_to_token, so the maximum is declared
  if (int rc = make_tmap_blocks_sw128(&tm, p.kv_pool, 1ull << 31, 9, kMlaDL, kMlaTile, 2)) return rc;
  if (int rc = get_tmap(&tr, p.kv_pool, 1ull << 31, kMlaDL, kMlaDL, kMlaTile)) return rc;
  if constexpr (!kExtend) {
    // [64 columns, heads, tokens, 9 blocks] of Q: an item's 16 heads in one copy, zeros where there is no head.  A row
    // stride of zero or below is served from the lowest address.
    const int64_t stride = p.q_stride < 0 ? -p.q_stride : p.q_stride;
    p.q_dir = p.q_stride > 0 ? 1 : p.q_stride < 0 ? -1 : 0;
    p.q_row0 = p.q_stride < 0 ? p.batch - 1 : 0;
    const T* low = reinterpret_cast<const T*>(p.q) + (p.q_stride < 0 ? (p.batch - 1) * p.q_stride : 0);
    const uint64_t rows = p.q_stride == 0 ? 1 : p.batch;
    const uint64_t dims[4] = {64, static_cast<uint64_t>(p.H), rows, 9};
    const uint64_t strides[3] = {kMlaDL, static_cast<uint64_t>(stride > 0 ? stride : kMlaDL), 64};
    const uint32_t box[4] = {64, kMlaHeads, 1, 9};
    if (int rc = make_tmap_sw128(&tq, low, 4, dims, strides, box)) return rc;
  }
  auto kern = attn_mla_kernel<T, kExtend>;
  static bool configured = false;
  if (!configured) {
    SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MlaShape<kExtend>::kSmem));
    configured = true;
  }
  SPD_CUDA(launch(kern, dim3(grid), dim3(kMlaThreads), MlaShape<kExtend>::kSmem, st, pdl_enabled(), tm, tr, tq, p));
  if (p.by_item)
    SPD_CUDA(launch(mla_merge_many_kernel<T>, dim3(p.batch * p.hgs, p.cols), dim3(512), 0, st, pdl_enabled(), p));
  else if (!p.snap)
    SPD_CUDA(launch(mla_merge_kernel<T>, dim3(grid, (p.cols + 3) / 4), dim3(512), 0, st, pdl_enabled(), p));
  return 0;
}

}  // namespace spd

using namespace spd;

extern "C" {

static int mla_rotary_store(const char* fn, void* q_rot, int64_t q_rot_stride, int q_head_stride, const void* qa, void* kv_pool,
                            const void* norm_weight, const float* cos_sin_cache, const int64_t* positions,
                            const int64_t* loc, int64_t tokens, int num_heads, int nope_dim, int kv_lora_rank, int rope_dim,
                            int64_t qa_stride, float eps, int dtype, spd_stream_t stream) {
  SPD_REQUIRE(kv_lora_rank == kMlaDV && rope_dim == kMlaDL - kMlaDV, SPD_E_SHAPE,
              "%s: built for kv_lora_rank 512 + rope 64 (got %d + %d)", fn, kv_lora_rank, rope_dim);
  SPD_REQUIRE(tokens >= 0 && tokens < (1ll << 31) && num_heads > 0 && nope_dim >= 0, SPD_E_BADARG, "%s: bad sizes", fn);
  SPD_REQUIRE(nope_dim % 8 == 0 && qa_stride % 8 == 0 && q_rot_stride % 8 == 0 && aligned16(q_rot) && aligned16(qa) &&
                  aligned16(kv_pool) && aligned16(norm_weight) && aligned16(cos_sin_cache),
              SPD_E_ALIGN, "%s: strides must be multiples of 8 and pointers 16-B aligned", fn);
  if (tokens == 0) return 0;
  SPD_DISPATCH_DTYPE(dtype, {
    SPD_CUDA(launch(mla_rotary_store_kernel<T>, dim3((unsigned)tokens), dim3(256), 0, as_stream(stream), pdl_enabled(),
                    (T*)q_rot, (const T*)qa, (T*)kv_pool, (const T*)norm_weight, cos_sin_cache, positions, loc, num_heads,
                    nope_dim, qa_stride, q_rot_stride, q_head_stride, eps));
  });
  return 0;
}

int spd_mla_rotary_store(void* q_lat, const void* qa, void* kv_pool, const void* norm_weight, const float* cos_sin_cache,
                         const int64_t* positions, const int64_t* loc, int64_t tokens, int num_heads, int nope_dim,
                         int kv_lora_rank, int rope_dim, int64_t qa_stride, int64_t q_lat_stride, float eps, int dtype,
                         spd_stream_t stream) {
  SPD_REQUIRE(q_lat && qa && kv_pool && norm_weight && cos_sin_cache && positions && loc, SPD_E_BADARG,
              "spd_mla_rotary_store: null pointer");
  return mla_rotary_store("spd_mla_rotary_store", static_cast<char*>(q_lat) + 2 * kMlaDV, q_lat_stride, kMlaDL, qa, kv_pool,
                          norm_weight, cos_sin_cache, positions, loc, tokens, num_heads, nope_dim, kv_lora_rank, rope_dim,
                          qa_stride, eps, dtype, stream);
}

int spd_mla_rotary_store_inplace(void* qa, void* kv_pool, const void* norm_weight, const float* cos_sin_cache,
                                 const int64_t* positions, const int64_t* loc, int64_t tokens, int num_heads, int nope_dim,
                                 int kv_lora_rank, int rope_dim, int64_t qa_stride, float eps, int dtype,
                                 spd_stream_t stream) {
  SPD_REQUIRE(qa && kv_pool && norm_weight && cos_sin_cache && positions && loc, SPD_E_BADARG,
              "spd_mla_rotary_store_inplace: null pointer");
  SPD_REQUIRE(nope_dim >= 0 && rope_dim >= 0 && nope_dim < (1 << 20) && rope_dim < (1 << 20), SPD_E_BADARG,
              "spd_mla_rotary_store_inplace: bad sizes");
  return mla_rotary_store("spd_mla_rotary_store_inplace", static_cast<char*>(qa) + 2ll * nope_dim, qa_stride,
                          nope_dim + rope_dim, qa, kv_pool, norm_weight, cos_sin_cache, positions, loc, tokens, num_heads,
                          nope_dim, kv_lora_rank, rope_dim, qa_stride, eps, dtype, stream);
}

int64_t spd_attn_mla_workspace_bytes(int num_heads, int kv_lora_rank) {
  // two partials per CTA of up to 4 tokens x min(heads, 16) rows, and 32 bytes per CTA; 8 rows per head of two per SM
  // cover that for any number of heads
  const int64_t items = 2ll * device_sm_count_cached();
  return items * num_heads * 8 * (kv_lora_rank + 2) * 4 + 256;
}

// own_workspace: the workspace is this stream's alone at every batch size (spd_attn_mla_own); otherwise a call that need not
// bring one leaves it untouched.
static int attn_mla(void* out, const void* q, const void* kv_pool, const int32_t* req_to_token,
                    const int64_t* req_pool_indices, const int64_t* seq_lens, const int32_t* prefix_lens,
                    const int32_t* extend_start_loc, int64_t batch, int64_t total_tokens, int num_heads, int kv_lora_rank,
                    int rope_dim, int64_t q_stride, int64_t out_stride, int64_t req_to_token_stride, float sm_scale,
                    int dtype, void* workspace, int64_t workspace_bytes, bool own_workspace, int sm_budget,
                    spd_stream_t stream) {
  SPD_REQUIRE(out && q && kv_pool && req_to_token && req_pool_indices, SPD_E_BADARG, "spd_attn_mla: null pointer");
  const bool extend = seq_lens == nullptr;
  SPD_REQUIRE(!extend || (prefix_lens && extend_start_loc), SPD_E_BADARG,
              "spd_attn_mla: give seq_lens (decode) or prefix_lens + extend_start_loc (extend)");
  SPD_REQUIRE(kv_lora_rank == kMlaDV && rope_dim == kMlaDL - kMlaDV, SPD_E_SHAPE,
              "spd_attn_mla: built for kv_lora_rank 512 + rope 64 (got %d + %d)", kv_lora_rank, rope_dim);
  SPD_REQUIRE(num_heads > 0 && batch >= 0 && total_tokens >= 0, SPD_E_BADARG, "spd_attn_mla: bad sizes");
  SPD_REQUIRE(q_stride % 8 == 0 && out_stride % 8 == 0 && aligned16(out) && aligned16(q) && aligned16(kv_pool),
              SPD_E_ALIGN, "spd_attn_mla: strides must be multiples of 8 and pointers 16-B aligned");
  const int64_t items = extend ? total_tokens : batch;
  if (items == 0) return 0;
  SPD_REQUIRE(items < 65536, SPD_E_SHAPE, "spd_attn_mla: more than 65535 query tokens in one call");
  const int device_sms = device_sm_count_cached();
  const int sms = sm_budget > 0 ? sm_budget : device_sms;
  const int grid = sms < device_sms ? sms : device_sms;
  MlaParams p{};
  if (int rc = wait_flag(&p.wait_expired)) return rc;
  p.out = out;
  p.q = q;
  p.kv_pool = kv_pool;
  p.req_to_token = req_to_token;
  p.req_pool_indices = req_pool_indices;
  p.seq_lens = seq_lens;
  p.prefix_lens = prefix_lens;
  p.extend_start_loc = extend_start_loc;
  p.batch = static_cast<int>(batch);
  p.total = static_cast<int>(total_tokens);
  p.H = num_heads;
  p.hgs = (num_heads + kMlaHeads - 1) / kMlaHeads;
  p.q_stride = q_stride;
  p.out_stride = out_stride;
  p.rtt_stride = req_to_token_stride;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
  p.min_tiles = 2;
  const int tq = extend ? MlaShape<true>::TQ : MlaShape<false>::TQ;
  p.cols = tq * (num_heads < kMlaHeads ? num_heads : kMlaHeads);
  const int64_t rows = 2ll * grid * p.cols, need = rows * (kMlaDV + 2) * 4 + grid * 32ll;
  const int64_t groups = (items + tq - 1) / tq * p.hgs;
  // what a call has to bring: room for the partials of a fixed split by query tokens, or nothing where those alone fill
  // the SMs twice; a workspace of just that size still serves calls cut at item starts
  const int64_t ctas = items * p.hgs;
  int64_t splits = (2ll * sms + ctas - 1) / ctas;
  splits = splits < 8 ? splits : 8;
  const int64_t least = splits > 1 ? items * num_heads * splits * (kMlaDV + 2) * 4 : 0;
  SPD_REQUIRE(least == 0 || (workspace && workspace_bytes >= least), SPD_E_WORKSPACE,
              "spd_attn_mla: workspace too small (%lld < %lld)", (long long)workspace_bytes, (long long)least);
  if (least == 0 && !own_workspace) workspace = nullptr;
  p.snap = workspace == nullptr || workspace_bytes < need || groups >= 16ll * grid;
  if (!p.snap) {
    p.o_part = reinterpret_cast<float*>(workspace);
    p.ml_part = p.o_part + rows * kMlaDV;
    p.info = reinterpret_cast<int*>(p.ml_part + rows * 2);
    p.by_item = !extend && 4 * groups <= grid;
  }
  cudaStream_t st = as_stream(stream);
  SPD_DISPATCH_DTYPE(dtype, {
    return extend ? mla_launch<T, true>(p, grid, st) : mla_launch<T, false>(p, grid, st);
  });
  return 0;
}

int spd_attn_mla(void* out, const void* q, const void* kv_pool, const int32_t* req_to_token, const int64_t* req_pool_indices,
                 const int64_t* seq_lens, const int32_t* prefix_lens, const int32_t* extend_start_loc, int64_t batch,
                 int64_t total_tokens, int num_heads, int kv_lora_rank, int rope_dim, int64_t q_stride, int64_t out_stride,
                 int64_t req_to_token_stride, float sm_scale, int dtype, void* workspace, int64_t workspace_bytes,
                 int sm_budget, spd_stream_t stream) {
  return attn_mla(out, q, kv_pool, req_to_token, req_pool_indices, seq_lens, prefix_lens, extend_start_loc, batch, total_tokens,
                  num_heads, kv_lora_rank, rope_dim, q_stride, out_stride, req_to_token_stride, sm_scale, dtype, workspace,
                  workspace_bytes, false, sm_budget, stream);
}

int spd_attn_mla_own(void* out, const void* q, const void* kv_pool, const int32_t* req_to_token, const int64_t* req_pool_indices,
                     const int64_t* seq_lens, const int32_t* prefix_lens, const int32_t* extend_start_loc, int64_t batch,
                     int64_t total_tokens, int num_heads, int kv_lora_rank, int rope_dim, int64_t q_stride, int64_t out_stride,
                     int64_t req_to_token_stride, float sm_scale, int dtype, void* workspace, int64_t workspace_bytes,
                     int sm_budget, spd_stream_t stream) {
  return attn_mla(out, q, kv_pool, req_to_token, req_pool_indices, seq_lens, prefix_lens, extend_start_loc, batch, total_tokens,
                  num_heads, kv_lora_rank, rope_dim, q_stride, out_stride, req_to_token_stride, sm_scale, dtype, workspace,
                  workspace_bytes, true, sm_budget, stream);
}

}  // extern "C"
