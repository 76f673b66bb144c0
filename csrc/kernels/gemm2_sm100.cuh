// Two-CTA (cta_group::2) variant of the bf16 GEMM: a cluster of two CTAs on a pair of SMs computes one 256 x 256 (G2_HALF: 256 x
// 128) output tile per step. Each CTA stages its own 128 rows of A and its own 128 columns of B (32 KB per pipeline stage
// instead of 48 KB for a 128 x 256 tile), the even CTA of the pair issues tcgen05.mma.cta_group::2 instructions that
// read both CTAs' shared memory, and each CTA ends up with the accumulator of its own 128 rows (all 256 columns) in
// its own TMEM. Per tensor-core cycle this halves the shared-memory and TMA traffic of the B operand, which is what
// limits the single-CTA kernel.
//
// Roles per CTA: warp 0 = TMA producer (both CTAs; every load reports its bytes to the EVEN CTA's `full`
// barrier), warp 1 = TMEM allocation (both) and MMA issue (even CTA only), warps 2.. = epilogue (both; they
// release the accumulator buffer by arriving on the even CTA's `tempty` barrier). tcgen05.commit with a CTA mask
// signals the barriers at the same offset in both CTAs. All mbarrier waits are bounded as in the single-CTA kernel;
// the loads are ordinary tile loads that each CTA issues for its own shared memory.
#pragma once
#include "gemm_sm100.cuh"

namespace opk {

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the same variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(rank));
  return out;
}
// Hands a TMEM buffer back to the MMA issuer: no global memory is published through this barrier, and a release would make
// the warp wait until its earlier stores of the tile have drained (1,000 to 2,500 cycles per tile, measured).
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t* smem_out, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_out)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Tile load into this CTA's shared memory whose completion bytes are counted on the barrier at `bar_cluster_addr`
// (a shared::cluster address: the even CTA's barrier).
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int c0,
                                                 int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(bar_cluster_addr), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// Arrives (once all earlier MMAs of this thread have completed) on the barrier at this offset in both CTAs of the pair.
__device__ __forceinline__ void umma2_commit_both(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)),
               "h"(mask)
               : "memory");
}

template <int COLS>
struct Gemm2Cfg {
  static constexpr int BM = 128;            // rows per CTA (256 per pair)
  static constexpr int BN = COLS;           // columns per pair (256 or 128); each CTA stages BN / 2 of them
  static constexpr int BK = 64;
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = (BN / 2) * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;          // 32 KB, 24 KB
  static constexpr int STAGES = BN == 256 ? 6 : 8;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256 + 8 * kEpiScratch + 8 * 8 * 8;
  static constexpr int TMEM_COLS = 2 * BN;                        // two accumulator buffers
};

constexpr int kStageWarps = 8;     // copier warps per CTA of the staged variant
// G2_WIDE: eight epilogue warps (see wide_epilogue); G2_HALF: the same with tiles of 128 columns (see choose_tile); G2_TEAMS: eight
// epilogue warps in two teams of four that take the tiles in turn, so that a warp still covers the whole width of its tile and a
// norm's fp32 partial sums are those of four warps.
enum Gemm2Variant : int { G2_PLAIN = 0, G2_STAGE = 1, G2_WIDE = 2, G2_HALF = 3, G2_TEAMS = 4 };
__host__ __device__ constexpr int gemm2_cols(int variant) { return variant == G2_HALF ? 128 : 256; }
// The staged variant keeps four epilogue warps: with eight next to its copier warps a thread would have 112 registers.
__host__ __device__ constexpr int gemm2_epi_warps(int epi, int variant) {
  return variant == G2_STAGE ? 4 : variant >= G2_WIDE ? 8 : gemm_epi_warps(epi);
}

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <bool A_MN, bool B_MN, int EPI, int VARIANT = G2_PLAIN>
__global__ void __cluster_dims__(2, 1, 1)
__launch_bounds__(64 + 32 * gemm2_epi_warps(EPI, VARIANT) + (VARIANT == G2_STAGE ? 32 * kStageWarps : 0), 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  using Cfg = Gemm2Cfg<gemm2_cols(VARIANT)>;
  constexpr bool STAGE = VARIANT == G2_STAGE;
  constexpr int TEAMS = VARIANT == G2_TEAMS ? 2 : 1;        // each with an accumulator buffer of its own
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);   // used in the even CTA
  uint64_t* empty = full + STAGES;                                                  // one set per CTA
  uint64_t* tfull = empty + STAGES;                                                 // one set per CTA
  uint64_t* tempty = tfull + 2;                                                     // used in the even CTA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  double* sq_slots = reinterpret_cast<double*>(smem + STAGES * Cfg::STAGE_BYTES + 256 + 8 * kEpiScratch);   // EPI_SUMSQ: [warp][kSqSums]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);      // one arm (expect_tx) by the even CTA's producer, bytes from both CTAs
      mbar_init(&empty[s], 1);     // one commit per use
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 2 * gemm2_epi_warps(EPI, VARIANT) / TEAMS);    // the epilogue warps of both CTAs
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  cluster_sync_all();              // barriers of both CTAs are initialised before anyone signals a peer
  if (warp == 1) {
    tmem_alloc2(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish2();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();          // no early trigger, as in the single-CTA kernel

  const int tiles_m = (p.M + 2 * BM - 1) / (2 * BM);
  const int tiles_n = (p.N + BN - 1) / BN;
  const int per_batch = tiles_m * tiles_n;
  const int total = per_batch * p.batch;
  const int kblocks = (p.K + BK - 1) / BK;
  const int n_clusters = gridDim.x >> 1, cluster_id = blockIdx.x >> 1;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    int have_band = -1;
    for (int tile = cluster_id; tile < total && ok; tile += n_clusters) {
      const int b = tile / per_batch;
      const int r = tile - b * per_batch;
      int tm, tn;
      tile_coords(r, tiles_m, tiles_n, tm, tn);
      if (STAGE && tn / kRasterBand > have_band) {
        // the band's rows of B must have been copied into the local scratch by the copier warps of every CTA
        const int band = tn / kRasterBand;
        const int* ready = p.stage_ready + band;
        const long long t0 = clock64();
        while (ld_acquire_gpu(ready) < (int)gridDim.x) {
          if (*abort_flag || clock64() - t0 > kWaitBudgetCycles) { *abort_flag = 1; ok = false; break; }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        asm volatile("fence.proxy.async;" ::: "memory");   // generic-proxy stores -> TMA (async proxy) loads
        have_band = band;
      }
      const int bb = b / p.b_batch_div;
      const int row0 = tm * 2 * BM + (int)rank * BM;          // this CTA's rows of A
      const int col0 = tn * BN + (int)rank * (BN / 2);        // this CTA's columns of B
      for (int kb = 0; kb < kblocks; ++kb) {
        if (!mbar_wait_warp(&empty[s], ph ^ 1u, abort_flag)) { ok = false; break; }
        if (elect_one()) {
          uint8_t* sa = smem + s * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + Cfg::A_BYTES;
          const uint32_t full_leader = mapa_u32(smem_u32(&full[s]), 0);
          if (leader) mbar_expect_tx(&full[s], 2 * Cfg::STAGE_BYTES);
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_3d_pair(sa + j * (BK * 128), &tmA, full_leader, row0 + j * 64, kb * BK, b);
          } else {
            tma_load_3d_pair(sa, &tmA, full_leader, kb * BK, row0, b);
          }
          if (B_MN) {
#pragma unroll
            for (int j = 0; j < BN / 2 / 64; ++j) tma_load_3d_pair(sb + j * (BK * 128), &tmB, full_leader, col0 + j * 64, kb * BK, bb);
          } else {
            tma_load_3d_pair(sb, &tmB, full_leader, kb * BK, col0, bb);
          }
        }
        __syncwarp();
        if (++s == STAGES) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (even CTA only)
    if (leader) {
      constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      int it = 0;
      for (int tile = cluster_id; tile < total && ok; tile += n_clusters, ++it) {
        const int buf = it & 1;
        const uint32_t tph = (it >> 1) & 1;
        if (!mbar_wait_warp(&tempty[buf], tph ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * BN;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait_warp(&full[s], ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
            const uint32_t sa = smem_u32(smem + s * Cfg::STAGE_BYTES);
            issue_kblock<A_MN, B_MN, true>(d_tmem, sa, sa + Cfg::A_BYTES, idesc, kb == 0);
            umma2_commit_both(&empty[s]);       // frees this stage in both CTAs
            if (kb == kblocks - 1) umma2_commit_both(&tfull[buf]);
          }
          __syncwarp();
          if (++s == STAGES) { s = 0; ph ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else if (STAGE && warp >= 2 + gemm2_epi_warps(EPI, VARIANT)) {
    // ------------------------------------------------------------ copiers: remote B -> local scratch, band by band
    const int ctid = (warp - 2 - gemm2_epi_warps(EPI, VARIANT)) * 32 + lane;
    const long long nthreads = (long long)gridDim.x * (32 * kStageWarps);
    const long long gtid = (long long)blockIdx.x * (32 * kStageWarps) + ctid;
    // K-major B ([N][K], a band = 2048 whole rows) or MN-major B ([K][N], a band = 2048 columns of every row)
    const int band_span = kRasterBand * BN;
    const int n_bands = (p.N + band_span - 1) / band_span;
    const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(p.stage_src);
    uint4* dst = reinterpret_cast<uint4*>(p.stage_dst);
    for (int band = 0; band < n_bands; ++band) {
      const int n0 = band * band_span, n1 = min(p.N, n0 + band_span);
      const int vec_per_row = B_MN ? (n1 - n0) >> 3 : p.K >> 3;     // 16-byte vectors per copied row segment
      const int n_rows = B_MN ? p.K : n1 - n0;
      const long long dst_ld = B_MN ? p.N >> 3 : p.K >> 3;           // scratch row pitch in vectors
      const long long nvec = (long long)n_rows * vec_per_row;
      constexpr int U = 8;                                     // remote loads in flight per thread
      for (long long i0 = gtid; i0 < nvec; i0 += U * nthreads) {
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const long long i = i0 + u * nthreads;
          if (i < nvec) {
            const long long rr = i / vec_per_row, cv = i % vec_per_row;
            const long long row = B_MN ? rr : n0 + rr;
            const long long col = B_MN ? n0 + cv * 8 : cv * 8;
            v[u] = __ldcg(reinterpret_cast<const uint4*>(src + row * p.stage_ld + col));
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const long long i = i0 + u * nthreads;
          if (i < nvec) {
            const long long rr = i / vec_per_row, cv = i % vec_per_row;
            const long long row = B_MN ? rr : n0 + rr;
            dst[row * dst_ld + (B_MN ? (n0 >> 3) + cv : cv)] = v[u];
          }
        }
      }
      __threadfence();
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kStageWarps) : "memory");
      if (ctid == 0) atomicAdd(p.stage_ready + band, 1);
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs, own 128 rows each)
    const int quad = warp & 3, quartet = (warp - 2) >> 2;
    constexpr int CSPLIT = gemm2_epi_warps(EPI, VARIANT) / 4 / TEAMS;
    const int c_begin = TEAMS == 1 ? quartet * (BN / CSPLIT) : 0, c_end = c_begin + BN / CSPLIT;
    uint8_t* scratch = smem + STAGES * Cfg::STAGE_BYTES + 256 + (warp - 2) * kEpiScratch;
    int it = 0;
    double* sq = sq_slots + (warp - 2) * kSqSums;
    if (EPI == EPI_SUMSQ) epi_zero_sq(sq);
    for (int tile = cluster_id; tile < total; tile += n_clusters, ++it) {
      const int buf = it & 1;
      if (TEAMS == 2 && buf != quartet) continue;           // the other team's tile
      const int b = tile / per_batch;
      const int r = tile - b * per_batch;
      int tm, tn;
      tile_coords(r, tiles_m, tiles_n, tm, tn);
      const uint32_t tph = (it >> 1) & 1;
      if (EPI == EPI_SWIGLU_BWD) prefetch_swiglu_row<BN>(p, tm * 2 * BM + (int)rank * BM + quad * 32 + lane, tn);
      int ok = 1;
      if (lane == 0) ok = mbar_wait(&tfull[buf], tph, abort_flag) ? 1 : 0;
      __syncwarp();
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      tc_fence_after();
      EpiState e = epi_begin<EPI>(p, scratch, tm * 2 * BM + (int)rank * BM + quad * 32, b);
      epilogue_tile<BN, EPI>(p, e, tmem_base + (uint32_t(quad * 32) << 16) + buf * BN, tn * BN, c_begin, c_end, [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(mapa_u32(smem_u32(&tempty[buf]), 0));
      });
      epi_end<EPI>(p, e, tn * CSPLIT + c_begin / (BN / CSPLIT), tiles_n * CSPLIT);
      if (EPI == EPI_SUMSQ) epi_add_sq(p, e, b, sq);
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();              // neither CTA frees TMEM or exits while its partner may still use its memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc2(tmem_base, Cfg::TMEM_COLS);
  }
  if (EPI == EPI_SUMSQ) epi_flush_sq(p, sq_slots, gemm2_epi_warps(EPI, VARIANT));
  if (threadIdx.x == 0 && *abort_flag && p.err) atomicExch(p.err, 1);
}

}  // namespace opk
