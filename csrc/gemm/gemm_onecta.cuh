// bf16 GEMM on the 5th-generation tensor cores: C[M,N] = A[M,K] * B[N,K]^T with fp32
// accumulation in tensor memory and a fused epilogue.
//
// One persistent CTA per SM walks a static tile schedule (M fastest, so the CTAs that run at
// the same time share one B panel out of L2). Inside the CTA the work is split by warp role:
//
//   warp 0      TMA producer   cp.async.bulk.tensor 2-D tiles, 128-byte swizzle, ring of 4 stages (6 and 8
//                              for tiles of 128 and 64 columns)
//   warp 1      MMA issuer     one elected lane issues tcgen05.mma (128 x BN x 16) and commits
//                              stage releases / accumulator completions to mbarriers
//   warps 2-9   epilogue       tcgen05.ld the 128 x BN fp32 accumulator (one row per thread, two
//                              warps per TMEM lane quarter, each taking half of the columns; tiles of
//                              64 columns have one per quarter, warps 2-5), apply bias / GELU / residual /
//                              GELU' and store
//
// The tile is 128 x BN, BN = 256, 128 or 64. Two accumulators of BN TMEM columns each are used in turn, so the
// epilogue of tile i runs while the tensor cores already work on tile i+1.
//
// Either operand may be K-major (the contraction index is contiguous in global memory) or
// MN-major (the M / N index is contiguous); the second form is what the weight-gradient and
// data-gradient GEMMs of a linear layer need, so no transposed copies are ever made.
//
// Replaces the nn.Linear calls of the reference model (nn/gpt2/modules.py:21-22,49-51,82) and
// their autograd; the reference's own tensor-core kernel is gpu-mojo/problems/p33/p33.mojo:130-245.
#pragma once
#include "../common/launch.cuh"
#include "../common/ptx.cuh"
#include "../common/tma_desc.h"
#include "gemm.h"

#include "../common/trace.cuh"

#include "gemm_epilogue.cuh"

namespace z2h {

namespace {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int A_STAGE_BYTES = BM * BK * 2;  // 16 KiB

// What follows from the tile width: 256 columns (the default), or 128 and 64 for outputs that have too
// few 128x256 tiles to occupy the SMs (pick_bn).
template <int BN>
struct TileCfg {
  static constexpr int STAGES = BN == 256 ? 4 : BN == 128 ? 6 : 8;
  static constexpr int B_STAGE_BYTES = BN * BK * 2;  // 32 KiB at 256
  static constexpr int EPI_WARPS = BN == 64 ? 4 : 8;
  static constexpr int EPI_BLOCKS = BN / 32 / (EPI_WARPS / 4);  // 32-column blocks per epilogue warp
  static constexpr int NUM_THREADS = 64 + 32 * EPI_WARPS;       // TMA warp, MMA warp, epilogue warps
  static constexpr int TMEM_COLS = 2 * BN;
  static constexpr int SMEM_BYTES =
      1024 + STAGES * (A_STAGE_BYTES + B_STAGE_BYTES) + 256 + EPI_WARPS * gemm_detail::kEpiWarpBytes;
  static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KiB a CTA may use");
};

using gemm_detail::KernelParams;


// EXTRA: the instantiation that carries the newer epilogue kinds (see epilogue_tile_streamed).
template <int A_MN, int B_MN, bool EXTRA, int BN>
__global__ void __launch_bounds__(TileCfg<BN>::NUM_THREADS, 1)
gemm_bf16_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA,
                         const __grid_constant__ CUtensorMap tmB, const KernelParams p) {
  using Cfg = TileCfg<BN>;
  constexpr int STAGES = Cfg::STAGES, B_STAGE_BYTES = Cfg::B_STAGE_BYTES, EPI_WARPS = Cfg::EPI_WARPS;
  constexpr int TMEM_COLS = Cfg::TMEM_COLS, EPI_COLS = Cfg::EPI_BLOCKS * 32;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * A_STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sB + STAGES * B_STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* epi_bias = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(full_bar) + 256);  // 4 KiB per epilogue warp: bias slice or transposition buffer

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  pdl_launch_dependents();

  // every role walks the same sequence of work segments
  gemm_detail::TileScheduler sched(p, BM, BN, BK, blockIdx.x, gridDim.x);
  gemm_detail::Segment sg;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], EPI_WARPS);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();  // everything above overlaps the previous kernel's tail; global memory from here on

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      Z2H_TRACE_DECL(0)
      Z2H_TRACE();
      while (ok && sched.next(sg)) {
        const int mt = sg.mt, nt = sg.nt, kb0 = sg.kb0, kb1 = sg.kb1;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_bounded(&empty_bar[stage], phase ^ 1u, abort_flag, p.status,
                                 kTimeoutEmpty)) {
            ok = false;
            break;
          }
          Z2H_TRACE();
          mbar_arrive_expect_tx(&full_bar[stage], A_STAGE_BYTES + B_STAGE_BYTES);
          uint8_t* a_dst = sA + stage * A_STAGE_BYTES;
          uint8_t* b_dst = sB + stage * B_STAGE_BYTES;
          if (A_MN == 0) {
            tma_load_2d(a_dst, &tmA, &full_bar[stage], kb * BK, mt * BM);
          } else {
#pragma unroll
            for (int c = 0; c < BM / 64; ++c)
              tma_load_2d(a_dst + c * (64 * BK * 2), &tmA, &full_bar[stage], mt * BM + c * 64,
                          kb * BK);
          }
          if (B_MN == 0) {
            tma_load_2d(b_dst, &tmB, &full_bar[stage], kb * BK, nt * BN);
          } else {
#pragma unroll
            for (int c = 0; c < BN / 64; ++c)
              tma_load_2d(b_dst + c * (64 * BK * 2), &tmB, &full_bar[stage], nt * BN + c * 64,
                          kb * BK);
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!ok) {
        // give copies that are still in flight a bounded time to land before the CTA exits
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(BM, BN, A_MN, B_MN);
      constexpr uint32_t a_lbo = A_MN ? 64 * BK * 2 : 16;
      constexpr uint32_t b_lbo = B_MN ? 64 * BK * 2 : 16;
      constexpr uint32_t a_kstep = A_MN ? UMMA_K * 128 : UMMA_K * 2;
      constexpr uint32_t b_kstep = B_MN ? UMMA_K * 128 : UMMA_K * 2;
      // Descriptors of stage 0; a stage or a K step further on is an addition to the address field. Built
      // anew for every MMA they were most of what this thread did between two waits: a k-block took about
      // 550 cycles whatever the tile width (64 columns need 300 of the tensor pipe).
      const uint64_t adesc0 = make_smem_desc_sw128(smem_u32(sA), a_lbo, 1024);
      const uint64_t bdesc0 = make_smem_desc_sw128(smem_u32(sB), b_lbo, 1024);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      Z2H_TRACE_DECL(1)
      Z2H_TRACE();
      for (; ok && sched.next(sg); ++it) {
        const int kb0 = sg.kb0, kb1 = sg.kb1;
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        if (!mbar_wait_bounded(&tempty_bar[acc], acc_phase ^ 1u, abort_flag, p.status,
                               kTimeoutTmemEmpty)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_bounded(&full_bar[stage], phase, abort_flag, p.status, kTimeoutFull)) {
            ok = false;
            break;
          }
          tc_fence_after();
          Z2H_TRACE();
          const uint64_t ad = desc_advance(adesc0, stage * A_STAGE_BYTES);
          const uint64_t bd = desc_advance(bdesc0, stage * B_STAGE_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            tc_mma_f16_ss(d_tmem, desc_advance(ad, k * a_kstep), desc_advance(bd, k * b_kstep), idesc,
                          (kb > kb0 || k > 0) ? 1u : 0u);
          tc_commit(&empty_bar[stage]);
          Z2H_TRACE();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) tc_commit(&tfull_bar[acc]);
      }
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    int it = 0;
    bool ok = true;
    Z2H_TRACE_DECL(2)
    for (; ok && sched.next(sg); ++it) {
      const int mt = sg.mt, nt = sg.nt;
      const bool empty_split = sg.kb0 >= sg.kb1;
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      // bias of this warp's columns, staged before the wait for the accumulator
      const int gcol0 = nt * BN + half * EPI_COLS;
      const float* sbias = gemm_detail::stage_bias(p, epi_bias + (warp - 2) * gemm_detail::kEpiBiasFloats, gcol0, lane);
      if (!empty_split) gemm_detail::prefetch_second_operand(p, (long long)mt * BM + quarter * 32 + lane, gcol0);
      if (!mbar_wait_bounded(&tfull_bar[acc], acc_phase, abort_flag, p.status, kTimeoutTmemFull)) {
        ok = false;
        break;
      }
      tc_fence_after();
      if (warp == 2 && lane == 0) Z2H_TRACE();
      const long long row_base = (long long)mt * BM + quarter * 32;
      const uint32_t taddr = tmem_base + (uint32_t(quarter * 32) << 16) + acc * BN;
      // this warp drains its share of the column blocks of its 32 rows
      const int c0 = half * Cfg::EPI_BLOCKS;
      uint64_t* const tempty = &tempty_bar[acc];
      gemm_detail::epilogue_tile_streamed<EXTRA, Cfg::EPI_BLOCKS>(p, taddr + c0 * 32, row_base + lane, gcol0, sbias, lane,
                                          smem_u32(epi_bias + (warp - 2) * gemm_detail::kEpiBiasFloats),
                                          !empty_split, (EXTRA && p.split_k > 1) ? sg.kb0 / sched.kb_per_split : 0,
                                          [tempty] { mbar_arrive(tempty); });
      if (warp == 2 && lane == 0) Z2H_TRACE();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int A_MN, int B_MN, int BN>
int launch(const GemmArgs& g, cudaStream_t stream) {
  CUtensorMap tmA, tmB;
  bool ok;
  if (A_MN == 0)
    ok = make_tma_2d_bf16(&tmA, g.A, g.M, g.K, g.lda, BM, BK, kSwizzle128);
  else
    ok = make_tma_2d_bf16(&tmA, g.A, g.K, g.M, g.lda, BK, 64, kSwizzle128);
  if (!ok) return 2;
  if (B_MN == 0)
    ok = make_tma_2d_bf16(&tmB, g.B, g.N, g.K, g.ldb, BN, BK, kSwizzle128);
  else
    ok = make_tma_2d_bf16(&tmB, g.B, g.K, g.N, g.ldb, BK, 64, kSwizzle128);
  if (!ok) return 2;

  KernelParams p = gemm_detail::make_kernel_params(g);
  p.raster_n = gemm_detail::pick_raster_n(g, BM, BN);

  auto kern = g.epi >= kEpiGeluSaveGrad ? gemm_bf16_tcgen05_kernel<A_MN, B_MN, true, BN>
                                        : gemm_bf16_tcgen05_kernel<A_MN, B_MN, false, BN>;
  constexpr int SMEM_BYTES = TileCfg<BN>::SMEM_BYTES, NUM_THREADS = TileCfg<BN>::NUM_THREADS;
  static std::atomic<unsigned long long> attr_seen{0};
  if (first_use_on_current_device(attr_seen)) {
    cudaFuncSetAttribute(gemm_bf16_tcgen05_kernel<A_MN, B_MN, true, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    cudaFuncSetAttribute(gemm_bf16_tcgen05_kernel<A_MN, B_MN, false, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  }
  const int num_sms = sm_count_current_device();
  const long long tiles = (long long)((g.M + BM - 1) / BM) * ((g.N + BN - 1) / BN) *
                          (p.stream_k ? (g.K + BK - 1) / BK : p.split_k);
  int grid = tiles < num_sms ? (int)tiles : num_sms;
  if (g.max_ctas > 0 && grid > g.max_ctas) grid = g.max_ctas;
  if (grid < 1) return 0;
  return launch_kernel(kern, dim3(grid), dim3(NUM_THREADS), SMEM_BYTES, stream, true, tmA, tmB, p) == cudaSuccess
             ? 0
             : 3;
}

template <int BN>
int launch_onecta(const GemmArgs& g, cudaStream_t stream) {
  if (g.a_mn == 0 && g.b_mn == 0) return launch<0, 0, BN>(g, stream);
  if (g.a_mn == 0 && g.b_mn == 1) return launch<0, 1, BN>(g, stream);
  if (g.a_mn == 1 && g.b_mn == 0) return launch<1, 0, BN>(g, stream);
  return launch<1, 1, BN>(g, stream);
}

}  // namespace
}  // namespace z2h
