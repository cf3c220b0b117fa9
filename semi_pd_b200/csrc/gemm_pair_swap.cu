// GEMM of prefill-sized batches with the operands swapped, on CTA PAIRS: D[256 weight rows x n tokens] = W A^T,
// C[token][column], n any multiple of 32 up to 256 from tile to tile.
//
// Why: the tiles of gemm_pair.cu and gemm.cu have 256 or 128 token rows, and what a batch (or, with experts, every expert's
// share of it) has beyond a multiple of that is work done for padding: 18 % at 1300 tokens, 17 % at 4096 tokens x 6 of 64
// experts, where single-CTA tiles also fetch 48 KB per k-block for the same MMAs (the L2 -> SM path moves about 16 TB/s).
// With the tokens on the MMA's N side a batch is cut into equal token tiles of 32-row units, and the weights, whose sizes
// are mostly multiples of 256, feed M.  What bounds it: the tensor cores under the power cap, then the operands' way from L2
// (16 KB + 64 n bytes per k-block and CTA).  Two Llama-3-8B layers on 1300 tokens 1249 -> 1097 us (gate / up 297 -> 236, down
// 146 -> 126); DeepSeek-V2-Lite's MoE layer on 4096 tokens 680 -> 614.
//
// Pipeline as in gemm_pair.cu (warp 0 TMA, warp 1 of the leader the MMAs, warps 4-7 of both the epilogue, two accumulators).
// With SiLU*mul the weight tile alternates 8 gate
// and 8 up rows (one 5-D box: columns, 8 rows, gate / up, row groups, expert), so that with the 16-lane form of tcgen05.ld a
// thread holds the gate and the up value of its outputs.  The epilogue transposes with stmatrix.trans: 64 tokens at a time
// are staged as rows of this CTA's 128 (SiLU: 64) columns and leave in pieces of 256 (128) contiguous bytes.
#include <cuda.h>
#include <stdlib.h>
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "pair.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace spd {

constexpr int kPsThreads = 256;
constexpr int kPsBK = 64;
constexpr int kPsStages = 12;                  // at most
constexpr int kPsHalfBytes = 128 * kPsBK * 2;  // 128 rows of one operand
constexpr int kPsTokens = 64;                  // tokens staged at a time
constexpr int kPsMaxTiles = 512;               // token tiles of a call
constexpr int kPsStageBytes = kPsTokens * (256 + 16);
struct PsControl {  // behind the list of token tiles
  uint64_t full[kPsStages], empty[kPsStages];  // (the leader's full are the live ones)
  uint64_t tfull[2], tempty[2];                // (the leader's tempty)
  uint32_t tmem;
  int dead;
  int warp_tiles[kPsThreads / 32];
};
constexpr int kPsFixedSmem = kPsStageBytes + (sizeof(PsControl) + 15) / 16 * 16 + 1024;  // beside the ring and the list
constexpr int kPsMaxSmem = 232448;
static_assert(6 * 2 * kPsHalfBytes + kPsMaxTiles * 16 + kPsFixedSmem <= kPsMaxSmem, "shared memory of a CTA");

struct SwapGemmParams {
  void* C;
  int64_t ldc;
  int n_cols;  // output columns (of a group)
  int w_tiles, kblocks;
  int rows;                    // of A
  int units, tok_tiles;        // one group: 32-row units, token tiles
  int stages, slot;            // ring: slots and bytes of each (128 weight rows, half of the widest token tile)
  int list;                    // token tiles that the list has room for
  int decode;                  // one group: a batch that streams the weights once (see the launch)
  int early;                   // one group: the first weights are fetched before the grid waits for its predecessor
  int panel;                   // one group: token tiles of a rasterisation panel
  const int2* group_rows;      // (first row, rows) of every group, null: one group
  int num_groups;
  int64_t w_group_rows, w_group_cols;  // plain weights: where a group's begin
  unsigned* wait_expired;
};

// token rows in boxes of 16, 32, .. 128 rows: half a token tile comes with one copy instruction (from boxes of 64, 32 and 16
// rows the tiles of 192 columns took 7 % longer)
struct TokenMaps {
  CUtensorMap rows[8];
};

// tcgen05.ld of 16 lanes x 64 columns: thread t has of every 8 columns those at 2 (t % 4) of lanes t / 4 (r[0], r[1]) and
// 8 + t / 4 (r[2], r[3])
__device__ __forceinline__ void tmem_ld_16x256b_x8(uint32_t taddr, uint32_t* r) {
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
// four 8 x 8 fragments of 16-bit pairs to shared memory, transposed; lane l gives the address of row l % 8 of fragment l / 8
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared::cta.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b),
               "r"(c), "r"(d)
               : "memory");
}
__device__ __forceinline__ void mbar_wait_cluster_bounded(uint64_t* bar, uint32_t parity, volatile int* dead) {
  for (int i = 0; i < kMbarWaitTries; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok || *dead) return;
  }
  *dead = 1;
}

// Token tile i of the `tiles` that `units` 32-row units are cut into: (first row, MMA columns, rows that exist, group)
__device__ __forceinline__ int4 token_tile(int i, int tiles, int units, int row0, int rows, int group) {
  const int base = units / tiles, more = units - base * tiles;
  const int at = 32 * (i * base + min(i, more)), n = 32 * (base + (i < more));
  return make_int4(row0 + at, n, min(n, rows - at), group);
}

template <typename T, bool kSilu>
__global__ void __launch_bounds__(kPsThreads, 1)
gemm_pair_swap_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ TokenMaps tmA, const SwapGemmParams p) {
  constexpr int kOut = kSilu ? 64 : 128;             // output columns of this CTA's half of a weight tile
  constexpr int kRow = kOut * 2 + 16;                // staged token row: 16 bytes more against bank conflicts
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sOut = smem + p.stages * p.slot;
  int4* tiles = reinterpret_cast<int4*>(sOut + kPsStageBytes);
  PsControl& control = *reinterpret_cast<PsControl*>(tiles + p.list);
  uint64_t *full = control.full, *empty = control.empty, *tfull = control.tfull, *tempty = control.tempty;
  uint32_t* tmem_slot = &control.tmem;
  volatile int* dead = &control.dead;
  int* warp_tiles = control.warp_tiles;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1;
  const int npairs = gridDim.x >> 1;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    *dead = 0;
  }
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < kPsStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 8);
    }
    fence_barrier_init();
  }
  if (warp == 2) {
    tmem_alloc_2cta(tmem_slot, 512);
    tmem_relinquish_2cta();
  }
  int tok_tiles = p.tok_tiles;
  for (int i = threadIdx.x; i < tok_tiles; i += kPsThreads) tiles[i] = token_tile(i, tok_tiles, p.units, 0, p.rows, 0);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before any cross-CTA signal
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (p.decode) griddep_launch_dependents();
  // (early: the weights are older than the kernel before, so the copies of the first ones precede the wait)
  if (!p.early || warp != 0) griddep_wait();
  // the token tiles of all groups, one behind the other
  if (p.group_rows) {
    const int g = threadIdx.x;
    int2 gr = g < p.num_groups ? p.group_rows[g] : make_int2(0, 0);
    gr.y = gr.x >= 0 && gr.x < p.rows ? max(0, min(gr.y, p.rows - gr.x)) : 0;  // (rows that A and C have)
    const int units = (gr.y + 31) >> 5, mine = (units + 7) >> 3;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tiles[warp] = incl;
    __syncthreads();
    int at = incl - mine;
    tok_tiles = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      if (w < warp) at += warp_tiles[w];
      tok_tiles += warp_tiles[w];
    }
    tok_tiles = min(tok_tiles, p.list);
    for (int i = 0; i < mine && at + i < p.list; ++i) tiles[at + i] = token_tile(i, mine, units, gr.x, gr.y, g);
    __syncthreads();
  }

  const int num_tiles = p.w_tiles * tok_tiles;
  // tile -> (weight tile, token tile).  Groups: a token tile's weight tiles before the next token tile, so that the pairs
  // work on a few neighbouring groups, whose weights and rows are read from HBM once.  One group: panels of token tiles
  // that stay in L2, within a panel all token tiles of a weight tile before the next.
  auto coords = [&](int tile, int& wt, int& tt) {
    if (p.group_rows) {
      tt = tile / p.w_tiles;
      wt = tile - tt * p.w_tiles;
      return;
    }
    const int per_panel = p.w_tiles * p.panel, pn = tile / per_panel, r = tile - pn * per_panel;
    const int q = min(p.panel, tok_tiles - pn * p.panel);
    wt = r / q;
    tt = pn * p.panel + r - wt * q;
  };

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0, phase = 0, ahead = 0;
      const uint64_t policy = p.decode ? kEvictFirst : kEvictNormal;  // of the weights
      auto load_w = [&](int slot, uint32_t lead_full, int kb, int wt, int group) {
        if constexpr (kSilu)
          tma_load_5d_2cta(smem + slot * p.slot, &tmW, lead_full, kb * kPsBK, 0, 0, wt * 16 + static_cast<int>(rank) * 8, group,
                           policy);
        else
          tma_load_2d_2cta(smem + slot * p.slot, &tmW, lead_full, static_cast<int>(group * p.w_group_cols) + kb * kPsBK,
                           static_cast<int>(group * p.w_group_rows) + wt * 256 + static_cast<int>(rank) * 128, policy);
      };
      if (p.early) {
        int wt, tt;
        coords(pair, wt, tt);
        const uint32_t bytes = 2 * (kPsHalfBytes + (tiles[tt].y >> 1) * (kPsBK * 2));
        for (; ahead < min(p.stages, p.kblocks); ++ahead) {
          if (rank == 0) mbar_expect_tx(&full[ahead], bytes);
          load_w(ahead, map_to_rank(smem_u32(&full[ahead]), 0), ahead, wt, 0);
        }
        griddep_wait();
      }
      for (int tile = pair; tile < num_tiles; tile += npairs) {
        int wt, tt;
        coords(tile, wt, tt);
        const int4 t = tiles[tt];
        const int half = t.y >> 1, a_row = t.x + static_cast<int>(rank) * half;
        const CUtensorMap* tm_tok = &tmA.rows[(half >> 4) - 1];
        for (int kb = 0; kb < p.kblocks; ++kb) {
          const uint32_t lead_full = map_to_rank(smem_u32(&full[stage]), 0);
          if (ahead > 0) {
            --ahead;  // its weights are on their way
          } else {
            mbar_wait_bounded(&empty[stage], phase ^ 1, dead);
            if (rank == 0) mbar_expect_tx(&full[stage], 2 * (kPsHalfBytes + half * (kPsBK * 2)));
            load_w(stage, lead_full, kb, wt, t.w);
          }
          tma_load_2d_2cta(smem + stage * p.slot + kPsHalfBytes, tm_tok, lead_full, kb * kPsBK, a_row, kEvictNormal);
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      int stage = 0, phase = 0, n = 0;
      for (int tile = pair; tile < num_tiles; tile += npairs) {
        int wt, tt;
        coords(tile, wt, tt);
        const uint32_t idesc = umma_idesc<T>(256, tiles[tt].y, 0, 0);
        const int as = n & 1, aphase = (n >> 1) & 1;
        ++n;
        mbar_wait_cluster_bounded(&tempty[as], aphase ^ 1, dead);  // both CTAs drained this accumulator
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + as * 256;
        for (int kb = 0; kb < p.kblocks; ++kb) {
          mbar_wait_bounded(&full[stage], phase, dead);
          tc_fence_after_sync();
          const uint32_t wa = smem_u32(smem + stage * p.slot), aa = wa + kPsHalfBytes;
#pragma unroll
          for (int k = 0; k < kPsBK / 16; ++k)
            umma_ss_2cta(d_tmem, umma_desc_sw128(wa + k * 32, 16, 1024), umma_desc_sw128(aa + k * 32, 16, 1024), idesc,
                         (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit_2cta_mc(&empty[stage], 0b11);  // both CTAs' slots are free once these MMAs are done
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
        umma_commit_2cta_mc(&tfull[as], 0b11);
      }
    }
  } else if (warp >= 4) {
    const int q = warp & 3, et = threadIdx.x - 128;
    const uint32_t lead_tempty0 = map_to_rank(smem_u32(&tempty[0]), 0);
    const uint32_t out = smem_u32(sOut);
    // this lane's row of the fragment it gives the address of: token (lane & 7) + 8 * (fragment's token block), column
    const int frag = lane >> 3;
    const uint32_t dst0 = kSilu ? out + (frag * 8 + (lane & 7)) * kRow + q * 32
                                : out + ((frag >> 1) * 8 + (lane & 7)) * kRow + q * 64 + (frag & 1) * 16;
    int n = 0;
    for (int tile = pair; tile < num_tiles; tile += npairs) {
      int wt, tt;
      coords(tile, wt, tt);
      const int4 t = tiles[tt];
      const int as = n & 1, aphase = (n >> 1) & 1;
      ++n;
      mbar_wait_bounded(&tfull[as], aphase, dead);
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + as * 256;
      const int n0 = wt * (2 * kOut) + static_cast<int>(rank) * kOut;
      T* C = reinterpret_cast<T*>(p.C) + static_cast<int64_t>(t.x) * p.ldc + n0;
#pragma unroll 1
      for (int c = 0; c < t.z; c += kPsTokens) {  // (the last 32 columns of an odd n: read, not stored)
        uint32_t r[2][32];
        tmem_ld_16x256b_x8(taddr + c, r[0]);
        tmem_ld_16x256b_x8(taddr + (16u << 16) + c, r[1]);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          auto f = [&](int i) { return __uint_as_float(r[h][i]); };
          if constexpr (kSilu) {
            auto one = [&](int i) {  // gate_up_proj's output is rounded to T before SiluAndMul reads it
              return silu_f32(to_f32<T>(from_f32<T>(f(i)))) * to_f32<T>(from_f32<T>(f(i + 2)));
            };
            auto two = [&](int b) { return pack2<T>(one(4 * b), one(4 * b + 1)); };
#pragma unroll
            for (int b = 0; b < 8; b += 4)
              stmatrix_x4_trans(dst0 + h * 16 + b * 8 * kRow, two(b), two(b + 1), two(b + 2), two(b + 3));
          } else {
#pragma unroll
            for (int b = 0; b < 8; b += 2)
              stmatrix_x4_trans(dst0 + h * 32 + b * 8 * kRow, pack2<T>(f(4 * b), f(4 * b + 1)), pack2<T>(f(4 * b + 2), f(4 * b + 3)),
                                pack2<T>(f(4 * b + 4), f(4 * b + 5)), pack2<T>(f(4 * b + 6), f(4 * b + 7)));
          }
        }
        if (c + kPsTokens >= t.z) {  // the accumulator has been read
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_remote_release(lead_tempty0 + as * 8);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        constexpr int kVecs = kOut / 8, kPer = 128 / kVecs;
        const int v = et % kVecs;
        if (n0 + v * 8 < p.n_cols) {
#pragma unroll
          for (int i = 0; i < kPsTokens; i += kPer) {
            const int tok = i + et / kVecs;
            if (c + tok < t.z)
              *reinterpret_cast<uint4*>(C + static_cast<int64_t>(c + tok) * p.ldc + v * 8) =
                  *reinterpret_cast<const uint4*>(sOut + tok * kRow + v * 16);
          }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
      }
    }
  }

  __syncwarp();  // the warps of the elected lanes come together before the barriers, which count whole warps
  if (!p.decode) griddep_launch_dependents();
  tc_fence_before_sync();
  __syncthreads();
  if (*dead) {
    wait_drain();
    if (threadIdx.x == 0) wait_report(p.wait_expired);
  }
  cluster_sync_all();  // the peer may still read this CTA's shared memory / signal its barriers
  if (warp == 2) tmem_dealloc_2cta(tmem_base, 512);
}

// Gate and up rows of all groups as [group][8-row group][gate / up][8 rows][64 columns]
int get_gate_up_tmap(CUtensorMap* out, const void* W, uint64_t groups, uint64_t inter, uint64_t cols, uint64_t ldw) {
  struct Key {
    const void* base;
    uint64_t groups, inter, cols, ldw;
    bool operator==(const Key& o) const {
      return base == o.base && groups == o.groups && inter == o.inter && cols == o.cols && ldw == o.ldw;
    }
  };
  struct Hash {
    size_t operator()(const Key& k) const {
      return reinterpret_cast<size_t>(k.base) ^ (k.groups * 0x9E3779B97F4A7C15ull) ^ (k.inter * 0xC2B2AE3D27D4EB4Full) ^
             (k.cols * 0x165667B19E3779F9ull) ^ (k.ldw << 7);
    }
  };
  static std::mutex mu;
  static std::unordered_map<Key, CUtensorMap, Hash> cache;
  const Key key{W, groups, inter, cols, ldw};
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it == cache.end()) {
    CUtensorMap m;
    const uint64_t dims[5] = {cols, 8, 2, inter / 8, groups};
    const uint64_t strides[4] = {ldw, inter * ldw, 8 * ldw, 2 * inter * ldw};
    const uint32_t box[5] = {kPsBK, 8, 2, 8, 1};
    if (int rc = make_tmap_sw128(&m, W, 5, dims, strides, box)) return rc;
    if (cache.size() > 8192) cache.clear();
    it = cache.emplace(key, m).first;
  }
  *out = it->second;
  return 0;
}

template <typename T, bool kSilu>
static int launch_swap(const CUtensorMap& tw, const TokenMaps& ta, const SwapGemmParams& p, int pairs, cudaStream_t stream) {
  auto kern = gemm_pair_swap_kernel<T, kSilu>;
  static bool configured = false;
  if (!configured) {
    SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPsMaxSmem));
    configured = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2 * pairs);
  cfg.blockDim = dim3(kPsThreads);
  cfg.dynamicSmemBytes = p.stages * p.slot + p.list * 16 + kPsFixedSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  SPD_CUDA(cudaLaunchKernelEx(&cfg, kern, tw, ta, p));
  return 0;
}

static int run_swap(SwapGemmParams& p, const void* A, int64_t rows, int64_t K, int64_t lda, const void* W, uint64_t groups,
                    int64_t ldw, bool silu, int64_t w_rows, int64_t w_cols, int widest, int dtype, int pairs, cudaStream_t stream) {
  p.slot = kPsHalfBytes + widest * kPsBK;
  const int fit = (kPsMaxSmem - kPsFixedSmem - p.list * 16) / p.slot;
  p.stages = fit < kPsStages ? fit : kPsStages;
  CUtensorMap tw;
  TokenMaps ta;
  for (int i = 0; i < 8; ++i)
    if (int rc = get_tmap(&ta.rows[i], A, rows, K, lda, 16 * (i + 1))) return rc;
  if (int rc = silu ? get_gate_up_tmap(&tw, W, groups, p.n_cols, K, ldw) : get_tmap(&tw, W, w_rows, w_cols, ldw, 128)) return rc;
  if (int rc = wait_flag(&p.wait_expired)) return rc;
  if (silu) SPD_DISPATCH_DTYPE(dtype, { return launch_swap<T, true>(tw, ta, p, pairs, stream); });
  SPD_DISPATCH_DTYPE(dtype, { return launch_swap<T, false>(tw, ta, p, pairs, stream); });
}

int gemm_pair_cols(int64_t M, int64_t N, int64_t K, int epilogue, int sms, int64_t* cost);

// Token tiles that a plain GEMM of these sizes is cut into, 0: the tiles of gemm_pair.cu / gemm.cu.  A wave of tiles of n
// columns takes about n + 100 units here as there (pair_tile_cols), so the fewer and narrower waves win; below 128
// columns a tile does not get shorter.  Where both count the same (M = 1600: seven tiles of 256 rows, or of 229) the
// rows saved still pay from three waves on, in power.  On both sides of the line, other tiles / these, us: 1300 tokens,
// K = 4096, N = 14336 with SiLU 297 / 236, 6144 59 / 53; 800: 201 / 153, 41 / 37; 512: 113 / 111, 22.8 / 23.1; K = 14336,
// N = 4096: 384 66 / 54, 700 76 / 77, 1100 111 / 121 (single CTAs), 1300 146 / 126, 2500 231 / 268 (not taken).  Single CTAs
// whose tiles are cut to 128 columns take a wave of those in 228 units: 64 x 2048, 1300 tokens 8.2 / 9.8, 640 on 72 SMs 8.3 / 10.2;
// 3648 x 2048, 640 11.2 / 12.7, 384 on 108 SMs 10.9 / 11.8; 264 x 1024, 513 6.2 / 7.7; 1000 x 192, 800 4.3 / 5.5 (not taken).
int gemm_swap_tiles(int64_t M, int64_t N, int64_t K, int epilogue, int sms) {
  if (M <= 256 || sms < 2 || (epilogue != SPD_EPI_NONE && epilogue != SPD_EPI_SILU_MUL) || M >= (1ll << 31) || N >= (1ll << 30))
    return 0;
  int64_t other;
  gemm_pair_cols(M, N, K, epilogue, sms, &other);
  if (other == 0) return 0;
  const int64_t units = (M + 31) / 32, w_tiles = epilogue == SPD_EPI_SILU_MUL ? (N + 127) / 128 : (N + 255) / 256;
  const int64_t pairs = sms / 2;
  int64_t best = 0, cost = 0, waves = 0;
  for (int64_t t = (units + 7) / 8; t <= (units + 3) / 4 && t <= kPsMaxTiles; ++t) {
    const int64_t n = 32 * ((units + t - 1) / t), w = (t * w_tiles + pairs - 1) / pairs, c = w * ((n < 128 ? 128 : n) + 100);
    if (best == 0 || c < cost) {
      best = t;
      cost = c;
      waves = w;
    }
  }
  const bool fewer_rows = waves >= 3 && 32 * units * 105 <= (M + 255) / 256 * 256 * 100;
  // (up to 16 k-blocks the tiles' ends decide, which take longer here: 5140 x 4096, K = 512 25.9 / 26.5 us for 6 % fewer units)
  if (K <= 16 * kPsBK) return cost * 10 < other * 9 ? static_cast<int>(best) : 0;
  return cost < other || (cost == other && fewer_rows) ? static_cast<int>(best) : 0;
}

int gemm_pair_swap(void* C, const void* A, const void* W, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldw, int64_t ldc,
                   int dtype, int epilogue, int sms, int tok_tiles, int panel_mb, bool early, cudaStream_t stream) {
  SwapGemmParams p{};
  const bool silu = epilogue == SPD_EPI_SILU_MUL;
  p.C = C;
  p.ldc = ldc;
  p.n_cols = static_cast<int>(N);
  p.w_tiles = static_cast<int>(silu ? (N + 127) / 128 : (N + 255) / 256);
  p.kblocks = static_cast<int>((K + kPsBK - 1) / kPsBK);
  p.rows = static_cast<int>(M);
  p.units = static_cast<int>((M + 31) / 32);
  p.tok_tiles = tok_tiles;
  const int64_t panel = (static_cast<int64_t>(panel_mb) << 20) / (((p.units + tok_tiles - 1) / tok_tiles) * 64 * K);
  p.panel = static_cast<int>(panel < 1 ? 1 : panel < tok_tiles ? panel : tok_tiles);
  const int64_t total = static_cast<int64_t>(p.w_tiles) * tok_tiles;
  const int pairs = static_cast<int>(total < sms / 2 ? total : sms / 2);
  p.list = tok_tiles;
  // as the other decode kernels (gemm_pair_decode.cu): the next kernel's weights come under this one's tail
  p.decode = M <= 256;
  p.early = early;
  return run_swap(p, A, M, K, lda, W, 1, ldw, silu, silu ? 2 * N : N, K, 32 * ((p.units + tok_tiles - 1) / tok_tiles), dtype, pairs, stream);
}

}  // namespace spd

using namespace spd;

extern "C" {

int spd_gemm_grouped_rows(void* C, const void* A, const void* W, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldw,
                          int64_t ldc, int num_groups, const int32_t* group_rows, int64_t w_group_col_stride, int dtype,
                          int epilogue, int sm_budget, spd_stream_t stream) {
  SPD_REQUIRE(C && A && W && group_rows, SPD_E_BADARG, "spd_gemm_grouped_rows: null pointer");
  SPD_REQUIRE(M >= 0 && N > 0 && K > 0 && num_groups > 0, SPD_E_BADARG, "spd_gemm_grouped_rows: bad sizes");
  SPD_REQUIRE(num_groups <= kPsThreads && M / 256 + num_groups <= kPsMaxTiles && M < (1ll << 31), SPD_E_SHAPE,
              "spd_gemm_grouped_rows: at most %d groups, and rows / 256 + groups at most %d", kPsThreads, kPsMaxTiles);
  SPD_REQUIRE(dtype == SPD_BF16 || dtype == SPD_F16, SPD_E_BADARG, "spd_gemm_grouped_rows: bad dtype %d", dtype);
  SPD_REQUIRE(epilogue == SPD_EPI_NONE || epilogue == SPD_EPI_SILU_MUL, SPD_E_BADARG, "spd_gemm_grouped_rows: bad epilogue %d",
              epilogue);
  SPD_REQUIRE(K % 8 == 0 && N % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && ldc % 8 == 0, SPD_E_ALIGN,
              "spd_gemm_grouped_rows: K, N and leading dimensions must be multiples of 8");
  SPD_REQUIRE(aligned16(A) && aligned16(W) && aligned16(C), SPD_E_ALIGN, "spd_gemm_grouped_rows: pointers must be 16-byte aligned");
  SPD_REQUIRE(lda >= K && ldc >= N, SPD_E_BADARG, "spd_gemm_grouped_rows: leading dimension too small");
  SPD_REQUIRE(w_group_col_stride == 0 || (w_group_col_stride >= K && w_group_col_stride % 8 == 0 && K % kPsBK == 0 &&
                                          epilogue == SPD_EPI_NONE && ldw >= num_groups * w_group_col_stride),
              SPD_E_BADARG, "spd_gemm_grouped_rows: bad w_group_col_stride (K-concatenated weights need K %% 64 == 0, no epilogue)");
  SPD_REQUIRE(ldw >= K, SPD_E_BADARG, "spd_gemm_grouped_rows: ldw too small");
  if (M == 0) return 0;
  const int sms = sm_budget > 0 ? sm_budget : device_sm_count_cached();
  SPD_REQUIRE(sms >= 2, SPD_E_BADARG, "spd_gemm_grouped_rows: needs two SMs");
  SwapGemmParams p{};
  const bool silu = epilogue == SPD_EPI_SILU_MUL;
  p.C = C;
  p.ldc = ldc;
  p.n_cols = static_cast<int>(N);
  p.w_tiles = static_cast<int>(silu ? (N + 127) / 128 : (N + 255) / 256);
  p.kblocks = static_cast<int>((K + kPsBK - 1) / kPsBK);
  p.rows = static_cast<int>(M);
  p.group_rows = reinterpret_cast<const int2*>(group_rows);
  p.num_groups = num_groups;
  const bool concat = w_group_col_stride > 0;
  p.w_group_rows = concat ? 0 : N;
  p.w_group_cols = w_group_col_stride;
  p.list = static_cast<int>(M / 256 + num_groups);
  const int64_t most = static_cast<int64_t>(p.w_tiles) * (M / 256 + num_groups);
  const int pairs = static_cast<int>(most < sms / 2 ? most : sms / 2);
  return run_swap(p, A, M, K, lda, W, num_groups, ldw, silu, concat ? N : num_groups * N,
                  concat ? num_groups * w_group_col_stride : K, 256, dtype, pairs, as_stream(stream));
}

}  // extern "C"
