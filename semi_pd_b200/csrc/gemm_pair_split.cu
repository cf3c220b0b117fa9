// GEMM of decode-sized batches on few weight tiles: operands swapped on CTA pairs as in gemm_pair_swap.cu, K cut over the
// pairs of a THREAD-BLOCK CLUSTER and reduced through distributed shared memory.
//
// Why: layers with fewer than 74 tiles of 256 weight rows need several pairs per tile to stream their weights at HBM speed.
// Cut stream-K style (gemm_pair_decode.cu) the partial sums of a tile travel through global memory to one owner, which adds
// them alone: 5 us at 64 tokens, 15 at 256.  Here every pair of the cluster leaves its partial sums in its own (by then idle)
// operand ring, and after one cluster barrier each of them adds all pairs' sums for its share of the tokens, in ascending k,
// so that the sums are read once over all SMs of the tile.  The hardware co-schedules a cluster: nothing spins on another
// CTA.
//
// A cluster of 2 S CTAs has one (weight tile, token tile); pair s the k-blocks [s kb / S, (s + 1) kb / S).  Warp 0: TMA, the
// ring filled with weights before the grid waits for its predecessor; warp 1 of a pair's leader: MMAs; warps 4-7:
// TMEM to shared memory as [token][128 rows] fp32; then all warps add and store, a warp a token, 256 (SiLU: 128) contiguous
// bytes.
#include <cuda.h>
#include <atomic>

#include "common.cuh"
#include "pair.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace spd {

constexpr int kPtThreads = 256;
constexpr int kPtBK = 64;
constexpr int kPtStages = 12;  // at most
constexpr int kPtWBytes = 128 * kPtBK * 2;
constexpr int kPtFixedSmem = 256 + 1024;
constexpr int kPtMaxSmem = 232448;
constexpr int kPtMaxSplit = 4;

struct PairSplitParams {
  void* C;
  int64_t ldc;
  int n_cols, m_rows;  // output columns, tokens
  int tok_tiles, n;    // token tiles, MMA columns of each
  int kblocks, stages, slot;
  int out_f32;
  int early;  // the first weights are fetched before the grid waits for its predecessor
  unsigned* wait_expired;
};

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

template <typename T, bool kSilu>
__global__ void __launch_bounds__(kPtThreads, 1)
gemm_pair_split_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA, const PairSplitParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + p.stages * p.slot);  // [stages]  (the leaders' are the live ones)
  uint64_t* empty = full + kPtStages;
  uint64_t* tfull = empty + kPtStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank(), rank = crank & 1, leader = crank & ~1u;
  const int S = static_cast<int>(cluster_nctarank() >> 1), s = static_cast<int>(crank >> 1);
  const int tile = blockIdx.x / (2 * S), wt = tile / p.tok_tiles, tt = tile - wt * p.tok_tiles;
  const int kb0 = s * p.kblocks / S, kb1 = (s + 1) * p.kblocks / S;
  const int half = p.n >> 1, tmem_cols = p.n <= 32 ? 32 : p.n <= 64 ? 64 : p.n <= 128 ? 128 : 256;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmA);
    *dead = 0;
  }
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(tfull, 1);
    fence_barrier_init();
  }
  if (warp == 2) {
    tmem_alloc_2cta(tmem_slot, tmem_cols);
    tmem_relinquish_2cta();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // the pair's barriers exist before any cross-CTA signal
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  griddep_launch_dependents();

  if (warp == 0) {
    if (elect_one()) {
      const uint32_t lead_full0 = map_to_rank(smem_u32(full), leader);
      const uint32_t bytes = 2 * (kPtWBytes + half * (kPtBK * 2));
      auto load_w = [&](int stage, int kb) {
        if constexpr (kSilu)
          tma_load_5d_2cta(smem + stage * p.slot, &tmW, lead_full0 + stage * 8, kb * kPtBK, 0, 0, wt * 16 + static_cast<int>(rank) * 8,
                           0, kEvictFirst);
        else
          tma_load_2d_2cta(smem + stage * p.slot, &tmW, lead_full0 + stage * 8, kb * kPtBK, wt * 256 + static_cast<int>(rank) * 128,
                           kEvictFirst);
      };
      const int ahead = min(p.stages, kb1 - kb0);
      if (!p.early) griddep_wait();
      for (int i = 0; i < ahead; ++i) {
        if (rank == 0) mbar_expect_tx(&full[i], bytes);
        load_w(i, kb0 + i);
      }
      if (p.early) griddep_wait();
      int stage = 0, phase = 0;
      const int a_row = tt * p.n + static_cast<int>(rank) * half;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (kb - kb0 >= ahead) {
          mbar_wait_bounded(&empty[stage], phase ^ 1, dead);
          if (rank == 0) mbar_expect_tx(&full[stage], bytes);
          load_w(stage, kb);
        }
        tma_load_2d_2cta(smem + stage * p.slot + kPtWBytes, &tmA, lead_full0 + stage * 8, kb * kPtBK, a_row, kEvictLast);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc<T>(256, p.n, 0, 0);
      const uint16_t both = static_cast<uint16_t>(0b11 << leader);
      int stage = 0, phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait_bounded(&full[stage], phase, dead);
        tc_fence_after_sync();
        const uint32_t wa = smem_u32(smem + stage * p.slot), aa = wa + kPtWBytes;
#pragma unroll
        for (int k = 0; k < kPtBK / 16; ++k)
          umma_ss_2cta(tmem, umma_desc_sw128(wa + k * 32, 16, 1024), umma_desc_sw128(aa + k * 32, 16, 1024), idesc,
                       (kb > kb0 || k > 0) ? 1u : 0u);
        umma_commit_2cta_mc(&empty[stage], both);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      umma_commit_2cta_mc(tfull, both);
    }
    __syncwarp();
  } else if (warp >= 4) {
    const int q = warp & 3;
    mbar_wait_bounded(tfull, 0, dead);  // every MMA of the pair is done: both rings are idle
    tc_fence_after_sync();
    const uint32_t taddr = tmem + (static_cast<uint32_t>(q * 32) << 16);
    float* part = reinterpret_cast<float*>(smem) + q * 32 + lane;
    const int used = min(p.n, (p.m_rows - tt * p.n + 31) & ~31);
#pragma unroll 1
    for (int c = 0; c < used; c += 32) {
      uint32_t r[32];
      tmem_ld_32x32b_x32(taddr + c, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) part[(c + j) * 128] = __uint_as_float(r[j]);
    }
    tc_fence_before_sync();
  }
  griddep_wait();      // C is written from here on
  cluster_sync_all();  // all pairs' sums are in place

  const int tok0 = s * p.n / S, tok1 = min((s + 1) * p.n / S, p.m_rows - tt * p.n);
  const uint32_t base = smem_u32(smem);
  uint32_t src[kPtMaxSplit];
#pragma unroll
  for (int i = 0; i < kPtMaxSplit; ++i) src[i] = map_to_rank(base, (i < S ? i : 0) * 2 + rank);
  auto sum = [&](int tok, int row) {
    float4 f[kPtMaxSplit];
#pragma unroll
    for (int i = 0; i < kPtMaxSplit; ++i)
      if (i < S) f[i] = ld_cluster_v4(src[i] + (tok * 128 + row) * 4);
    float4 v = f[0];
#pragma unroll
    for (int i = 1; i < kPtMaxSplit; ++i)
      if (i < S) {
        v.x += f[i].x;
        v.y += f[i].y;
        v.z += f[i].z;
        v.w += f[i].w;
      }
    return v;
  };
  if constexpr (kSilu) {
    const int j = lane & 15, row = (j >> 1) * 16 + (j & 1) * 4, col = wt * 128 + static_cast<int>(rank) * 64 + j * 4;
#pragma unroll 2
    for (int tok = tok0 + warp * 2 + (lane >> 4); tok < tok1; tok += 16) {
      const float4 g = sum(tok, row), u = sum(tok, row + 8);
      auto one = [&](float a, float b) {  // gate_up_proj's output is rounded to T before SiluAndMul reads it
        return silu_f32(to_f32<T>(from_f32<T>(a))) * to_f32<T>(from_f32<T>(b));
      };
      if (col < p.n_cols)
        *reinterpret_cast<uint2*>(reinterpret_cast<T*>(p.C) + static_cast<int64_t>(tt * p.n + tok) * p.ldc + col) =
            make_uint2(pack2<T>(one(g.x, u.x), one(g.y, u.y)), pack2<T>(one(g.z, u.z), one(g.w, u.w)));
    }
  } else {
    const int col = wt * 256 + static_cast<int>(rank) * 128 + lane * 4;
#pragma unroll 4
    for (int tok = tok0 + warp; tok < tok1; tok += 8) {
      const float4 v = sum(tok, lane * 4);
      const int64_t at = static_cast<int64_t>(tt * p.n + tok) * p.ldc + col;
      if (col < p.n_cols) {
        if (p.out_f32)  // (rounded to T first)
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.C) + at) =
              make_float4(f32_result<T>(v.x, p.out_f32), f32_result<T>(v.y, p.out_f32), f32_result<T>(v.z, p.out_f32),
                          f32_result<T>(v.w, p.out_f32));
        else
          *reinterpret_cast<uint2*>(reinterpret_cast<T*>(p.C) + at) = make_uint2(pack2<T>(v.x, v.y), pack2<T>(v.z, v.w));
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*dead) {
    wait_drain();
    if (threadIdx.x == 0) wait_report(p.wait_expired);
  }
  cluster_sync_all();  // nobody leaves while a peer may still read its shared memory
  if (warp == 2) tmem_dealloc_2cta(tmem, tmem_cols);
}

template <typename T, bool kSilu>
static int launch_split(const CUtensorMap& tw, const CUtensorMap& ta, const PairSplitParams& p, int clusters, int split,
                        cudaStream_t stream) {
  auto kern = gemm_pair_split_kernel<T, kSilu>;
  static bool configured = false;
  if (!configured) {
    SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPtMaxSmem));
    configured = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(clusters * 2 * split);
  cfg.blockDim = dim3(kPtThreads);
  cfg.dynamicSmemBytes = p.stages * p.slot + kPtFixedSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  SPD_CUDA(cudaLaunchKernelEx(&cfg, kern, tw, ta, p));
  return 0;
}

int get_gate_up_tmap(CUtensorMap* out, const void* W, uint64_t groups, uint64_t inter, uint64_t cols, uint64_t ldw);

int gemm_pair_split(void* C, const void* A, const void* W, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldw, int64_t ldc,
                    int dtype, int out_f32, int epilogue, int tok_tiles, int split, bool early, cudaStream_t stream) {
  const bool silu = epilogue == SPD_EPI_SILU_MUL;
  PairSplitParams p{};
  p.C = C;
  p.ldc = ldc;
  p.n_cols = static_cast<int>(N);
  p.m_rows = static_cast<int>(M);
  p.tok_tiles = tok_tiles;
  p.n = static_cast<int>(32 * (((M + 31) / 32 + tok_tiles - 1) / tok_tiles));
  p.kblocks = static_cast<int>((K + kPtBK - 1) / kPtBK);
  p.out_f32 = out_f32;
  p.early = early;
  p.slot = kPtWBytes + p.n * kPtBK;
  const int fit = (kPtMaxSmem - kPtFixedSmem) / p.slot, most = (p.kblocks + split - 1) / split;
  const int sums = (p.n * 512 + p.slot - 1) / p.slot;  // slots that the partial sums need
  p.stages = fit < kPtStages ? fit : kPtStages;
  if (p.stages > most) p.stages = most < sums ? sums : most;
  const int w_tiles = static_cast<int>(silu ? (N + 127) / 128 : (N + 255) / 256);
  CUtensorMap tw, ta;
  if (int rc = get_tmap(&ta, A, M, K, lda, p.n / 2)) return rc;
  if (int rc = silu ? get_gate_up_tmap(&tw, W, 1, N, K, ldw) : get_tmap(&tw, W, N, K, ldw, 128)) return rc;
  if (int rc = wait_flag(&p.wait_expired)) return rc;
  if (silu) SPD_DISPATCH_DTYPE(dtype, { return launch_split<T, true>(tw, ta, p, w_tiles * tok_tiles, split, stream); });
  SPD_DISPATCH_DTYPE(dtype, { return launch_split<T, false>(tw, ta, p, w_tiles * tok_tiles, split, stream); });
}

// Clusters of 2 `split` CTAs that the choice below reckons with on `sms` SMs when the driver says that `found` run at once
// (-1: there is no device to ask).  0 is an answer: no cluster of this size fits.
static int split_room(int split, int found, int sms) {
  static const int b200[kPtMaxSplit + 1] = {0, 74, 33, 22, 15};
  if (found < 0) {
    const int whole = device_sm_count_cached();
    found = sms >= whole ? b200[split] : b200[split] * sms / whole;
  }
  const int most = sms / (2 * split);
  return found < most ? found : most;
}

// What the driver says of a stream: a partition holds as many clusters as its SMs' places on the chip allow, which its number
// of SMs does not tell (whole B200: 74, 33, 22, 15 clusters of 2, 4, 6, 8 CTAs; 76 SMs beside 72: 38, 15, 9, 6, the 72: 36, 18, 9, 9;
// 108 beside 40: 54, 23, 13, 10).  Reckoned by number, 4096 x 14336 got 16 clusters of four on the 76 SMs, two waves: 23 us of
// one token became 48.  A query takes 1 us of host time, so the whole device is asked once.
static int split_clusters(int split, int sms, cudaStream_t stream) {
  static std::atomic<int> cached[kPtMaxSplit + 1];  // the whole device's answer + 2
  const bool whole = sms >= device_sm_count_cached();
  int n = whole ? cached[split].load(std::memory_order_relaxed) - 2 : -2;
  if (n > -2) return n;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2 * split);
  cfg.blockDim = dim3(kPtThreads);
  cfg.dynamicSmemBytes = kPtMaxSmem;
  cfg.stream = whole ? nullptr : stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto kern = gemm_pair_split_kernel<__nv_bfloat16, false>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPtMaxSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = -1;  // no device to ask (the choice of kernel can be asked for without one)
  }
  if (whole) cached[split].store(n + 2, std::memory_order_relaxed);
  return n;
}

int gemm_cluster_ctas(int64_t M, int64_t N, int64_t K, int sms);
int split_room_of(int split, int found, int sms) { return split >= 1 && split <= kPtMaxSplit ? split_room(split, found, sms) : 0; }

// The tiles of a GEMM on few weight tiles, 0: the other kernels.  *split = pairs per tile in a cluster (this kernel), 0: tiles
// of gemm_pair_swap.cu that one wave holds.  scratch: the call has the workspace that stream-K wants.
//
// Every form's time is estimated in us from what was measured with weights out of L2 (1 - 1024 tokens, weights of 64 x 2048 to
// 14336 x 1024 and 4096 x 14336; the form chosen took 1.02 times the fastest one's time in the mean): a k-block of a pair 0.175
// and up to 0.1 more for 256 tokens; the weights once at 6.2 GB/ms from HBM and what all pairs fetch, tokens and weights of every
// token tile, at 8 GB/ms; adding the sums 4.6 for 256 tokens.  Stream-K (gemm_pair_decode.cu) or the cluster of single CTAs
// (gemm_cluster.cu) / the form chosen, us: 4096 x 4096, 16 tokens 10.2 / 9.5, 64 12.3 / 10.1, 256 24.4 / 14; 6144 x 4096
// 12.7 / 12.0, 15.0 / 12.9, 26.5 / 17.3; 2048 x 2816 6.2 / 5.9, 9.8 / 6.6, 21.3 / 9.4; 64 x 2048 5.3 / 4.2, 10.0 / 4.4, 24.0 / 5.2.
// Up to 16 tokens a long stream of weights goes to the cluster of single CTAs where that covers more SMs: behind another
// kernel of a decode step each CTA's ring fills early (a Llama-3-8B layer of one token 151.1 us with 4096 x 4096 there,
// 151.4 here; 4096 x 14336 by itself 21.6 / 21.9).  Beyond 256 tokens the tiles of
// gemm_pair_swap.cu / gemm_pair.cu serve unless this kernel is estimated a tenth faster, three tenths beyond 512 tokens
// (4096 x 14336, 448 tokens 51 / 44; 64 x 2048, 1024 9.1 / 7.3; 4096 x 4096, 640 18.5 / 20 and not taken), and unless K is not cut
// (4096 x 14336, 512 tokens on 108 SMs 57 / 77).
int gemm_split_tiles(int64_t M, int64_t N, int64_t K, int epilogue, int out_f32, int sms, bool scratch, cudaStream_t on, int* split) {
  *split = 0;
  // Rows beyond 16384 and unrounded fp32 results keep the finer cuts of the other kernels: an accumulator's error grows with
  // the products it adds up.
  if (sms < 2 || (epilogue != SPD_EPI_NONE && epilogue != SPD_EPI_SILU_MUL) || M > 8192 || K > 16384 || out_f32 == 2) return 0;
  const bool silu = epilogue == SPD_EPI_SILU_MUL;
  const int64_t w_tiles = silu ? (N + 127) / 128 : (N + 255) / 256;
  const int pairs = sms / 2;
  if (w_tiles > pairs) return 0;
  const double bytes = 2.0 * K * (silu ? 2 * N : N), kb = static_cast<double>((K + kPtBK - 1) / kPtBK);
  static const double more[kPtMaxSplit + 1] = {0, 0, 0.36, 0.3, 0.4};
  const int units = static_cast<int>((M + 31) / 32);
  int room[kPtMaxSplit + 1];
  for (int s = 1; s <= kPtMaxSplit; ++s) {
    const bool may = w_tiles * 2 * s <= sms && 8 * (s - 1) <= kb;
    room[s] = !may ? 0 : split_room(s, s == 1 ? pairs : split_clusters(s, sms, on), sms);
  }
  double best = 0, swap = 0;
  int tiles = 0, swap_tiles = 0;
  for (int t = (units + 7) / 8; t <= units && t * w_tiles <= pairs; ++t) {
    const int n = 32 * ((units + t - 1) / t);
    const double stream = 3 + bytes / 6.2e6, fetch = 3 + t * w_tiles * 2.0 * K * (256 + n) / 8e6;
    double us = 3 + kb * (0.175 + 0.18 * (n > 64 ? n - 64 : 0) / 192), weights = 3 + bytes / 5.2e6;
    us = (us > weights ? us > fetch ? us : fetch : weights > fetch ? weights : fetch) + 0.6 * n / 256;
    if (!out_f32 && (swap_tiles == 0 || us < swap)) {
      swap = us;
      swap_tiles = t;
    }
    for (int s = 1; s <= kPtMaxSplit; ++s) {
      if (t * w_tiles > room[s]) continue;
      us = 2.5 + (kb / s) * (0.176 + 0.1 * n / 256) + more[s];
      us = (us > stream ? us > fetch ? us : fetch : stream > fetch ? stream : fetch) + 4.6 * n / 256;
      if (tiles == 0 || us < best) {
        best = us;
        tiles = t;
        *split = s;
      }
    }
  }
  if (M > 256) {
    if (tiles == 0 || swap_tiles == 0 || *split < 2 || best > swap * (M <= 512 ? 0.9 : 0.7)) {
      *split = 0;
      return 0;
    }
    return tiles;
  }
  if (swap_tiles > 0 && (tiles == 0 || swap < best)) {
    tiles = swap_tiles;
    *split = 0;
  }
  if (M <= 16 && bytes > 2.5e7 && !silu) {
    const int ctas = static_cast<int>(w_tiles) * tiles * 2 * (*split > 0 ? *split : 1);
    if (gemm_cluster_ctas(M, N, K, sms) > ctas) {
      *split = 0;
      return 0;
    }
  }
  // A partition that has little more SMs than these tiles have CTAs is better used by the kernels that deal k-blocks evenly over
  // all of them: the cluster of single CTAs and stream-K by single CTAs, or by pairs beyond 32 tokens.  Their time on 40 - 108 SMs,
  // from the same measurements: weights at 113 MB/ms an SM, at most 7.2 GB/ms, a k-block of a pair 0.15 and 0.1 more for 256
  // tokens, fix-up.  Stream-K / these, us: 4096 x 14336 on 40 SMs, one token 32.7 / 43, 64 35.5 / 43.7, on 76 SMs 64 26.1 / 43.5, on 72
  // 1 23.1 / 25.3, 256 46.1 / 42.0; 6144 x 4096 on 72 SMs, one token 13.9 / 15.9; 4096 x 4096 on 40, one token 14.1 / 15.6, 64 16.7 /
  // 15.9.  Of 859 calls on partitions 13 took up to 9 % more than before this kernel then, the form chosen 0.2 % more than the
  // faster one in the mean.
  if (sms < device_sm_count_cached() && scratch && !silu) {
    const double rate = 113e3 * sms < 7.2e6 ? 113e3 * sms : 7.2e6, even = kb * w_tiles / pairs * (0.15 + 0.1 * (M > 64 ? 32 * units - 64 : 0) / 192);
    double old = bytes / rate;
    if (M <= 32) old += M <= 16 ? 6 : 6.6;
    else old = 7 + 10.0 * 32 * units / 256 + (old > even ? old : even);
    if ((*split > 0 ? best : swap) > old) {
      *split = 0;
      return 0;
    }
  }
  return tiles;
}

}  // namespace spd
