// Prefill-regime GEMM on CTA PAIRS: C[M,N] = A[M,K] * W[N,K]^T with tcgen05.mma.cta_group::2.
//
// Two CTAs on the two SMs of one TPC (cluster of 2) own one 256 x BN output tile (BN = 256, see pair_tile_cols for the
// others).  CTA r holds the A rows [r*128, r*128+128) of the tile and HALF of the W tile (128 of its 256 rows); one
// UMMA of shape M=256, N=256, K=16 issued by the leader CTA reads both CTAs' shared memory and
// writes each CTA's 128 x 256 fp32 accumulator into that CTA's own TMEM.  Against the single-CTA
// 128 x 256 tile (gemm.cu) every CTA stages 32 KB instead of 48 KB per k-block and the tensor
// core reads a third fewer operand bytes from shared memory per FLOP — on a power-capped B200
// (measured: ~1 kW, SM clock 1.15-1.45 GHz under sustained GEMM load) the
// joules per FLOP are what sets the sustained rate.
//
// Pipeline (per CTA: 256 threads; warp 0 = TMA producer, warp 1 = MMA issuer (leader CTA only),
// warp 2 = TMEM allocator, warps 4-7 = epilogue):
//   full[s]   leader's barrier: 1 arrive (leader producer, expect_tx of BOTH CTAs' 64 KB) + the
//             transaction bytes of the four TMA loads (two per CTA, .cta_group::2 so the peer's
//             loads may signal the leader's barrier)
//   empty[s]  one per CTA, count 1: tcgen05.commit.cta_group::2 ... multicast to both CTAs
//   tfull[a]  one per CTA, count 1: multicast commit when an accumulator stage is complete
//   tempty[a] leader's barrier, count 8: the four epilogue warps of each CTA (the peer's arrive
//             remotely with release.cluster)
// The fused SiLU*mul epilogue maps naturally: CTA 0 stages the 128 gate rows, CTA 1 the 128 up
// rows of the tile, so accumulator columns [0,128) are gate and [128,256) are up in both CTAs.
#include <cuda.h>
#include <stdlib.h>

#include "common.cuh"
#include "pair.cuh"
#include "ptx.cuh"
#include "row_stage.cuh"
#include "tmap.cuh"

namespace spd {

constexpr int kPgThreads = 256;
constexpr int kPgBM = 128;   // rows per CTA (pair tile = 256)
constexpr int kPgBN = 256;   // the widest tile
constexpr int kPgBK = 64;
constexpr int kPgABytes = kPgBM * kPgBK * 2;  // 16 KB
template <int BN>
struct PairShape {
  static constexpr int kBBytes = (BN / 2) * kPgBK * 2;  // this CTA's half of the W tile
  static constexpr int kStages = BN >= 224 ? 6 : 7;
  static constexpr int kSmem = kStages * (kPgABytes + kBBytes) + 4 * kStageWarp + 1024 + 256;
  static_assert(BN % 32 == 0 && kSmem <= 232448, "tile shape");
};

struct PairGemmParams {
  void* C;
  int64_t ldc;
  int64_t m_rows;    // M
  int64_t n_cols;    // output columns (SILU_MUL: the intermediate size)
  int64_t up_row0;   // SILU_MUL: row of W where the "up" half starts
  int x_tiles, y_tiles, kblocks;
  int panel;         // y tiles per L2 rasterisation panel (see gemm.cu: tile_coords)
  int out_f32;
};

__device__ __forceinline__ void pair_tile_coords(const PairGemmParams& p, int tile, int& xt, int& yt) {
  if (p.panel <= 1) {
    xt = tile % p.x_tiles;
    yt = tile / p.x_tiles;
    return;
  }
  const int per_panel = p.x_tiles * p.panel;
  const int pn = tile / per_panel;
  const int r = tile - pn * per_panel;
  const int y0 = pn * p.panel;
  const int q = min(p.panel, p.y_tiles - y0);
  xt = r / q;
  yt = y0 + r - xt * q;
}

template <typename T, int kEpi, int BN>
__global__ void __launch_bounds__(kPgThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW,
                 const PairGemmParams p) {
  constexpr int kStages = PairShape<BN>::kStages, kBBytes = PairShape<BN>::kBBytes;
  constexpr int kBNOut = (kEpi == SPD_EPI_SILU_MUL) ? BN / 2 : BN;
  constexpr int kTmemStage = 256;
  constexpr int kTmemCols = 2 * kTmemStage;  // two accumulator stages
  static_assert(kBNOut % 32 == 0, "the epilogue goes by 32 columns");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + kStages * kPgABytes;
  uint8_t* sOut = smem + kStages * (kPgABytes + kBBytes);  // kStageWarp per epilogue warp
  uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + 4 * kStageWarp);
  uint64_t* full = bars;                        // [kStages]  (leader's are the live ones)
  uint64_t* empty = bars + kStages;           // [kStages]
  uint64_t* tfull = bars + 2 * kStages;       // [2]
  uint64_t* tempty = bars + 2 * kStages + 2;  // [2]          (leader's are the live ones)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1;
  const int npairs = gridDim.x >> 1;
  const int num_tiles = p.x_tiles * p.y_tiles;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmW);
  }
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < kStages; ++i) {
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
    tmem_alloc_2cta(tmem_slot, kTmemCols);
    tmem_relinquish_2cta();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before any cross-CTA signal
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  griddep_wait();

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0, phase = 0;
      for (int tile = pair; tile < num_tiles; tile += npairs) {
        int xt, yt;
        pair_tile_coords(p, tile, xt, yt);
        const int a_row = xt * (2 * kPgBM) + static_cast<int>(rank) * kPgBM;
        const int w_row = (kEpi == SPD_EPI_SILU_MUL)
                              ? (rank == 0 ? yt * kBNOut : static_cast<int>(p.up_row0) + yt * kBNOut)
                              : yt * BN + static_cast<int>(rank) * (BN / 2);
        for (int kb = 0; kb < p.kblocks; ++kb) {
          mbar_wait(&empty[stage], phase ^ 1);
          if (rank == 0) mbar_expect_tx(&full[stage], 2 * (kPgABytes + kBBytes));
          const uint32_t lead_full = map_to_rank(smem_u32(&full[stage]), 0);
          tma_load_2d_2cta(sA + stage * kPgABytes, &tmA, lead_full, kb * kPgBK, a_row, kEvictNormal);
          tma_load_2d_2cta(sB + stage * kBBytes, &tmW, lead_full, kb * kPgBK, w_row, kEvictNormal);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = umma_idesc<T>(2 * kPgBM, BN, 0, 0);
      int stage = 0, phase = 0, n = 0;
      for (int tile = pair; tile < num_tiles; tile += npairs) {
        const int as = n & 1, aphase = (n >> 1) & 1;
        ++n;
        mbar_wait_cluster_acquire(&tempty[as], aphase ^ 1);  // both CTAs drained this accumulator
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + as * kTmemStage;
        for (int kb = 0; kb < p.kblocks; ++kb) {
          mbar_wait(&full[stage], phase);
          tc_fence_after_sync();
          const uint32_t aa = smem_u32(sA + stage * kPgABytes);
          const uint32_t ba = smem_u32(sB + stage * kBBytes);
#pragma unroll
          for (int k = 0; k < kPgBK / 16; ++k)
            umma_ss_2cta(d_tmem, umma_desc_sw128(aa + k * 32, 16, 1024), umma_desc_sw128(ba + k * 32, 16, 1024),
                         idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit_2cta_mc(&empty[stage], 0b11);  // both CTAs' slots are free once these MMAs are done
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        umma_commit_2cta_mc(&tfull[as], 0b11);
      }
    }
  } else if (warp >= 4) {
    const int q = warp & 3;
    uint8_t* stage = sOut + q * kStageWarp;
    const uint32_t lead_tempty0 = map_to_rank(smem_u32(&tempty[0]), 0);
    int n = 0;
    for (int tile = pair; tile < num_tiles; tile += npairs) {
      int xt, yt;
      pair_tile_coords(p, tile, xt, yt);
      const int as = n & 1, aphase = (n >> 1) & 1;
      ++n;
      mbar_wait(&tfull[as], aphase);
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + as * kTmemStage;
      const int64_t m0 = static_cast<int64_t>(xt) * (2 * kPgBM) + rank * kPgBM + q * 32;
      const int rows = static_cast<int>(min(static_cast<int64_t>(32), p.m_rows - m0));
      auto values = [&](int c, float (&v)[32]) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + c, r);
        if constexpr (kEpi == SPD_EPI_SILU_MUL) {
          uint32_t u[32];
          tmem_ld_32x32b_x32(taddr + kBNOut + c, u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            // gate_up_proj output is rounded to T before SiluAndMul reads it
            const float g = to_f32<T>(from_f32<T>(__uint_as_float(r[j])));
            const float up = to_f32<T>(from_f32<T>(__uint_as_float(u[j])));
            v[j] = silu_f32(g) * up;
          }
        } else {
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j)
            v[j] = kEpi == SPD_EPI_GELU ? gelu_fast_f32(to_f32<T>(from_f32<T>(__uint_as_float(r[j])))) : __uint_as_float(r[j]);
        }
      };
      const int step = p.out_f32 ? 32 : 64;
#pragma unroll 1
      for (int c = 0; c < kBNOut; c += step) {
        const int64_t n0 = static_cast<int64_t>(yt) * kBNOut + c;
        const int cols = static_cast<int>(min(static_cast<int64_t>(min(step, kBNOut - c)), p.n_cols - n0));
        float v[32];
        values(c, v);
        if (p.out_f32) {
          stage_put32<T>(stage, lane, v, p.out_f32);
          stage_out(stage, lane, reinterpret_cast<uint8_t*>(p.C) + (m0 * p.ldc + n0) * 4, p.ldc * 4, rows, cols * 4);
        } else {
          stage_put16<T>(stage, lane, 0, v);
          if (c + 32 < kBNOut) {
            values(c + 32, v);
            stage_put16<T>(stage, lane, 1, v);
          }
          stage_out(stage, lane, reinterpret_cast<uint8_t*>(p.C) + (m0 * p.ldc + n0) * 2, p.ldc * 2, rows, cols * 2);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote_release(lead_tempty0 + as * 8);
    }
  }

  __syncwarp();  // the warps of the elected lanes come together before the barriers, which count whole warps
  griddep_launch_dependents();
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // the peer may still read this CTA's shared memory / signal its barriers
  if (warp == 2) tmem_dealloc_2cta(tmem_base, kTmemCols);
}

template <typename T, int kEpi, int BN>
static int launch_pair_gemm(const CUtensorMap& ta, const CUtensorMap& tw, const PairGemmParams& p, int pairs,
                            cudaStream_t stream) {
  auto kern = gemm_pair_kernel<T, kEpi, BN>;
  static bool configured = false;
  if (!configured) {
    SPD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairShape<BN>::kSmem));
    configured = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2 * pairs);
  cfg.blockDim = dim3(kPgThreads);
  cfg.dynamicSmemBytes = PairShape<BN>::kSmem;
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
  SPD_CUDA(cudaLaunchKernelEx(&cfg, kern, ta, tw, p));
  return 0;
}

// Columns of a pair tile: the width whose waves take least.  A wave of BN columns takes about BN + 100 units (a tile's A rows,
// its beginning and end do not shrink with it), so a narrower tile serves where the widest leaves a last wave nearly empty.
// 256 / the one chosen, us: 4096 x 14336 weights, M = 700 84.9 / 67.3 (192), 1300 147 / 127 (192); 4096 x 4096, 700 31.1 /
// 24.9 (192), 1300 49.7 / 41.0 (192); 3648 x 2048, 4096 54.1 / 48.0 (224).  160 and 128 were never the fastest; SiLU tiles
// (gate and up rows in one) gained nothing from 192.
static int pair_tile_cols(int64_t N, int64_t x_tiles, int epilogue, int pairs, int64_t* cost) {
  int best = 0;
  for (int bn : {256, 224, 192}) {
    const int64_t n_out = epilogue == SPD_EPI_SILU_MUL ? bn / 2 : bn;
    const int64_t waves = (x_tiles * ((N + n_out - 1) / n_out) + pairs - 1) / pairs;
    if (best == 0 || waves * (bn + 100) < *cost) {
      best = bn;
      *cost = waves * (bn + 100);
    }
    if (epilogue != SPD_EPI_NONE) break;
  }
  return best;
}

// Columns of the pair tiles that a GEMM of these sizes takes, 0: single-CTA tiles.  *cost: what either takes, in the units
// of pair_tile_cols.
int gemm_pair_cols(int64_t M, int64_t N, int64_t K, int epilogue, int sms, int64_t* cost_out) {
  if (cost_out) *cost_out = 0;
  static const int enabled = getenv("SPD_GEMM_2CTA") ? atoi(getenv("SPD_GEMM_2CTA")) : 1;
  if (!enabled || M <= 256 || sms < 2) return 0;
  // A wave of 256 x 256 pair tiles takes about 0.9 of the time of a wave of 128 x 256 single tiles, so the pair serves also
  // where its taller tiles pad M more, unless that costs it another wave — or the call is so short (under 48 k-blocks in
  // all waves) that the pair's longer start and end decide.  4096 x 14336 weights: M = 300 87 -> 70 us, 600 87 -> 72,
  // 1300 167 -> 156; 3648 x 2048, M = 600: 15.7 us single, 17.9 pair, 1300: 35 single, 28 pair.
  const int64_t rows_pair = (M + 255) / 256 * 256, rows_single = (M + 127) / 128 * 128;
  int64_t cost;
  const int bn = pair_tile_cols(N, rows_pair / 256, epilogue, sms / 2, &cost);
  if (cost_out) *cost_out = cost;
  if (rows_pair != rows_single && M < 2048) {
    const int n_tile = epilogue == SPD_EPI_SILU_MUL ? kPgBN / 2 : kPgBN;
    const int64_t cols = (N + n_tile - 1) / n_tile, kblocks = (K + kPgBK - 1) / kPgBK;
    const int64_t waves_single = (rows_single / 128 * cols + sms - 1) / sms;
    if (cost * 9 >= waves_single * (kPgBN + 100) * 10 || waves_single * kblocks < 48) {
      if (cost_out) {
        // (few tiles of 256 columns that N does not fill are cut to 128, which the 0.9 does not hold for: see gemm_swap_tiles)
        const bool narrow = epilogue != SPD_EPI_SILU_MUL && N % kPgBN != 0 && rows_single / 128 * cols < sms;
        const int64_t waves128 = (rows_single / 128 * ((N + 127) / 128) + sms - 1) / sms;
        *cost_out = narrow ? waves128 * (128 + 100) : waves_single * (kPgBN + 100) * 10 / 9;
      }
      return 0;
    }
  }
  return bn;
}

// Called by spd_gemm for the prefill regime.  Returns 1 if this path does not apply (the caller
// falls through to the single-CTA kernel), 0 on launch, else an error code.
int gemm_pair_try(void* C, const void* A, const void* W, int64_t M, int64_t N, int64_t K, int64_t lda,
                  int64_t ldw, int64_t ldc, int dtype, int out_f32, int epilogue, int sms, int panel_mb,
                  cudaStream_t stream) {
  const int bn = gemm_pair_cols(M, N, K, epilogue, sms, nullptr);
  if (bn == 0) return 1;
  PairGemmParams p{};
  p.C = C;
  p.ldc = ldc;
  p.m_rows = M;
  p.n_cols = N;
  p.up_row0 = N;
  p.out_f32 = out_f32;
  p.kblocks = static_cast<int>((K + kPgBK - 1) / kPgBK);
  p.x_tiles = static_cast<int>((M + 255) / 256);
  const int n_out = epilogue == SPD_EPI_SILU_MUL ? bn / 2 : bn;
  p.y_tiles = static_cast<int>((N + n_out - 1) / n_out);
  const long long tile_bytes = static_cast<long long>(bn) * K * 2;
  const long long q = (static_cast<long long>(panel_mb) << 20) / tile_bytes;
  p.panel = static_cast<int>(q < 1 ? 1 : q);
  const int total = p.x_tiles * p.y_tiles;
  const int pairs = total < sms / 2 ? total : sms / 2;
  CUtensorMap ta, tw;
  int rc;
  if ((rc = get_tmap(&ta, A, M, K, lda, kPgBM))) return rc;
  if ((rc = get_tmap(&tw, W, epilogue == SPD_EPI_SILU_MUL ? 2 * N : N, K, ldw, bn / 2))) return rc;
#define SPD_PAIR(EPI, BN) \
  if (epilogue == EPI && bn == BN) SPD_DISPATCH_DTYPE(dtype, { return launch_pair_gemm<T, EPI, BN>(ta, tw, p, pairs, stream); })
  SPD_PAIR(SPD_EPI_SILU_MUL, 256);
  SPD_PAIR(SPD_EPI_GELU, 256);
  SPD_PAIR(SPD_EPI_NONE, 256);
  SPD_PAIR(SPD_EPI_NONE, 224);
  SPD_PAIR(SPD_EPI_NONE, 192);
#undef SPD_PAIR
  return 1;
}

}  // namespace spd
