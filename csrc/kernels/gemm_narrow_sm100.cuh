// Small-output variant of the bf16 GEMM: one 128 x BN output tile per CTA, no persistent schedule.
//
// Why: a product with few output tiles leaves most of the chip idle on the persistent kernels, and what it then waits for
// is the fixed cost of a CTA (about 4,000 cycles: descriptors, first loads, epilogue) and the serial walk over the reduction
// (512 to 620 cycles per 64-element block of a 256-wide tile). Narrower tiles bring more SMs in. The products of an output
// element are added in the same order as in the persistent kernels, so the result has the same bits: which kernel a product
// takes depends on its number of rows, and a row's result must not.
#pragma once
#include "gemm2_sm100.cuh"

namespace opk {

template <int BN>
struct GemmNarrowCfg {
  static constexpr int BM = 128, BK = 64;
  static constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  // Pipeline depth: `FEW` stages (at most 96 KB) leave room for a second CTA on the SM, `MANY` cover the load latency
  // (about 1,650 cycles) of a CTA that has the SM for itself.
  static constexpr int FEW = BN == 256 ? 4 : BN == 128 ? 3 : 4, MANY = BN == 256 ? 4 : BN == 128 ? 6 : 8;
  static constexpr int smem_bytes(int stages) { return stages * STAGE_BYTES + 1024 + 256; }
  static_assert(8 * kEpiScratch <= FEW * STAGE_BYTES, "the epilogue's scratch reuses the pipeline buffers");
};
constexpr int kNarrowEpiWarps = 8;

template <bool A_MN, bool B_MN, int BN, int EPI>
__global__ void __launch_bounds__(64 + 32 * kNarrowEpiWarps, BN == 256 || EPI == EPI_SWIGLU_BWD ? 1 : 2)
gemm_narrow_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p,
                   const int STAGES) {
  using Cfg = GemmNarrowCfg<BN>;
  constexpr int BM = Cfg::BM, BK = Cfg::BK;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty = full + Cfg::MANY;
  uint64_t* tfull = empty + Cfg::MANY;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();       // after this CTA's TMEM is allocated: a successor that allocates next can only wait for a running grid
  pdl_wait();

  // grid = (row tiles, column tiles, batch): no divisions before the first load (the persistent kernels' tile arithmetic, cold
  // in the instruction cache, costs 1,400 cycles there), and the row tiles of a column follow each other, so that a weight
  // matrix larger than the L2 is read once (the other order read it per row tile: 317 x 28672 x 4096 129 us)
  const int kblocks = (p.K + BK - 1) / BK;
  const int tm = blockIdx.x, tn = blockIdx.y, b = blockIdx.z;
  if (warp == 0) {
    int s = 0;
    uint32_t ph = 0;
    const int bb = b / p.b_batch_div;
    for (int kb = 0; kb < kblocks; ++kb) {
      if (!mbar_wait_warp(&empty[s], ph ^ 1u, abort_flag)) break;
      if (elect_one()) {
        uint8_t* sa = smem + s * Cfg::STAGE_BYTES;
        uint8_t* sb = sa + Cfg::A_BYTES;
        mbar_expect_tx(&full[s], Cfg::STAGE_BYTES);
        if (A_MN) {
#pragma unroll
          for (int j = 0; j < BM / 64; ++j) tma_load_3d(sa + j * (BK * 128), &tmA, &full[s], tm * BM + j * 64, kb * BK, b);
        } else {
          tma_load_3d(sa, &tmA, &full[s], kb * BK, tm * BM, b);
        }
        if (B_MN) {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_3d(sb + j * (BK * 128), &tmB, &full[s], tn * BN + j * 64, kb * BK, bb);
        } else {
          tma_load_3d(sb, &tmB, &full[s], kb * BK, tn * BN, bb);
        }
      }
      __syncwarp();
      if (++s == STAGES) { s = 0; ph ^= 1u; }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(BM, BN, A_MN, B_MN);
    int s = 0;
    uint32_t ph = 0;
    // Two blocks per wait: a barrier probe holds back the products issued after it by 120 to 160 cycles, more than a
    // block of a narrow tile has tensor-core work to cover (128 x 128: 376 cycles per block with a probe for each, 259
    // without).
    for (int kb = 0; kb < kblocks; kb += 2) {
      const bool two = kb + 1 < kblocks;
      const int t = s + 1 == STAGES ? 0 : s + 1;
      const uint32_t pt = t == 0 ? ph ^ 1u : ph;
      const bool r0 = mbar_try_wait(&full[s], ph), r1 = !two || mbar_try_wait(&full[t], pt);
      if (!__all_sync(0xffffffffu, r0 && r1)) {
        if (!mbar_wait_warp(&full[s], ph, abort_flag)) break;
        if (two && !mbar_wait_warp(&full[t], pt, abort_flag)) break;
      }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t sa = smem_u32(smem + s * Cfg::STAGE_BYTES);
        issue_kblock<A_MN, B_MN, false>(tmem_base, sa, sa + Cfg::A_BYTES, idesc, kb == 0);
        umma_commit(&empty[s]);
        if (two) {
          const uint32_t ta = smem_u32(smem + t * Cfg::STAGE_BYTES);
          issue_kblock<A_MN, B_MN, false>(tmem_base, ta, ta + Cfg::A_BYTES, idesc, false);
          umma_commit(&empty[t]);
        }
        if (kb + 2 >= kblocks) umma_commit(tfull);
      }
      __syncwarp();
      s = t + 1 == STAGES ? 0 : t + 1;
      ph = s == 0 ? pt ^ 1u : pt;
    }
  } else {
    const int ew = warp - 2, quad = warp & 3;
    constexpr int CSPLIT = kNarrowEpiWarps / 4;
    const int c_begin = (ew >> 2) * (BN / CSPLIT), c_end = c_begin + BN / CSPLIT;
    int ok = 1;
    if (lane == 0) ok = mbar_wait(tfull, 0, abort_flag) ? 1 : 0;
    __syncwarp();
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (ok) {
      // all loads have landed and all products have read them: the pipeline buffers are free
      tc_fence_after();
      const uint32_t tmem_tile = tmem_base + (uint32_t(quad * 32) << 16);
      EpiState e = epi_begin<EPI>(p, smem + ew * kEpiScratch, tm * BM + quad * 32, b);
      epilogue_tile<BN, EPI>(p, e, tmem_tile, tn * BN, c_begin, c_end, [] {});
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
  if (threadIdx.x == 0 && *abort_flag && p.err) atomicExch(p.err, 1);
}

}  // namespace opk
