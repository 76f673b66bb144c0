// Persistent, warp-specialised bf16 GEMM for sm_100a built on tcgen05.mma with TMEM accumulators.
//
//   D[b][M][N] = sum_k A[b][m][k] * B[b'][n][k]           (fp32 accumulate in TMEM)
//
// * operands arrive through TMA into 128-byte-swizzled shared-memory tiles (4-6 stage mbarrier ring),
// * one elected thread issues 128 x BN x 16 UMMAs, the accumulator is double-buffered in TMEM so the
//   epilogue of tile i overlaps the main loop of tile i+1,
// * each operand may be K-major (reduction index contiguous in memory) or MN-major (row/column index
//   contiguous), which covers forward (X W^T), data-gradient (dY W) and weight-gradient (dY^T X)
//   products without any transposed copies,
// * the epilogue is a template hook: plain store (+bias, +residual), store + sum of squares (per-example
//   gradient norm), SwiGLU, and the two halves of a fused linear-cross-entropy.
//
// Warp roles (192 threads): warp 0 = TMA producer, warp 1 = TMEM owner + MMA issuer, warps 2..5 = epilogue
// (warp w may touch TMEM lanes 32*(w%4) .. +31).
#pragma once
#include "ptx_sm100.cuh"
#include "pdl.cuh"

namespace opk {

enum GemmEpilogue : int {
  EPI_STORE = 0,    // C = alpha*acc (+bias[n]) (+R[m][n])
  EPI_SUMSQ = 1,    // C = bf16(alpha*acc); *sumsq += sum(C^2); with C == nullptr only the sum is produced
  EPI_SWIGLU = 2,   // columns interleaved (gate, up): C = raw, act[m][n/2] = silu(gate)*up
  EPI_LCE_FWD = 3,  // per-(row, column-tile) max / sum-exp partials and the target logit; no logits stored
  EPI_LCE_BWD = 4,  // C = (exp(z - lse[m]) - [n == label[m]]) * coef[m]
  EPI_SWIGLU_BWD = 5,  // acc = d(act); act = saved (gate, up) pairs [M][2N]; C[m][2n], C[m][2n+1] = d(gate), d(up)
  EPI_LCE_FWD2 = 6,    // EPI_LCE_FWD with two column parts per tile (twice the epilogue warps), chosen by lce_parts == 2
  EPI_LCE_GRAD = 7,    // EPI_LCE_BWD on logits that the forward pass stored (lce_grad_kernel): no product
  // Forms of their own: asking in every chunk whether to store cost the products that store nothing 2 to 3 % (us, before there was
  // anything to store -> asked -> now: 2048 x 50257 x 768 139.5 -> 142.0 -> 139.5, 1520 x 11421 x 128 25.2 -> 26.0 -> 25.2).
  EPI_LCE_KEEP = 8,    // EPI_LCE_FWD that also stores the logits (`z`)
  EPI_LCE_KEEP2 = 9,   // EPI_LCE_FWD2 that does
};

struct GemmParams {
  int M, N, K, batch;
  int b_batch_div;       // B uses batch index b / b_batch_div (shared K/V heads, shared weights)
  long long ldc;         // elements
  long long strideC;     // elements between batches of C / R
  void* C;               // bf16
  const void* R;         // optional residual, same layout as C (may alias C)
  const void* bias;      // optional bf16 [N]
  float alpha;
  int stepwise;          // EPI_STORE: the product is rounded to bf16, scaled and rounded again before R is added
  double* sumsq;         // EPI_SUMSQ: one accumulator per batch entry (sumsq[b])
  void* act;             // EPI_SWIGLU: bf16 [M][ld_act] (written); EPI_SWIGLU_BWD: saved pre-activations (read)
  long long ld_act;
  const int* labels;     // EPI_LCE_*: [M], negative = ignored
  float* pmax;           // EPI_LCE_FWD: [M][parts * tiles_n], parts = 1 (EPI_LCE_FWD) or 2 (EPI_LCE_FWD2)
  float* psum;           // EPI_LCE_FWD: [M][parts * tiles_n], parts = 1 (EPI_LCE_FWD) or 2 (EPI_LCE_FWD2)
  float* tgt;            // EPI_LCE_FWD: [M] target logit (written by the tile that owns the label)
  float* z;              // EPI_LCE_KEEP: fp32 logits for the backward pass in blocks of 32 x 32 (see z_block)
  const float* lse;      // EPI_LCE_BWD: [M]
  const float* coef;     // EPI_LCE_BWD: [M] per-row scale (mask / divisor * upstream grad)
  float softcap;         // EPI_LCE_*: 0 = off, else z = cap * tanh(z / cap)
  float inv_cap, inv_cap_lo;   // 1 / cap as the sum of two floats (see cap_quotient)
  int* err;              // set to 1 when a bounded wait expired
  // Grouped modes (mixture-of-experts), both driven by small device-side tables so that data-dependent group sizes
  // need no host synchronisation and the launch stays capturable in a CUDA graph:
  //  * tile_group[m_tile] (forward / dgrad): A and C are ONE row-grouped matrix, every 128-row tile belongs to one
  //    group; B is batched and the tile uses B[tile_group[m_tile]]; tiles marked -1 are skipped.
  //  * group_k[2*b] / group_k[2*b+1] (wgrad): first reduction element and number of 64-element blocks of batch entry
  //    b inside the un-batched operands, i.e. C[b] = A[:, k0:k0+len]^T-style reduction over that group's rows.
  const int* tile_group;
  const int* group_k;
  int sumsq_stride;      // EPI_SUMSQ accumulator index = b * sumsq_stride (0: all batch entries share sumsq[0])
  // Staged B operand (two-CTA kernel only): B lives in ANOTHER GPU's memory. Extra warps of every CTA copy it, one
  // band of column tiles at a time, into a local scratch matrix [N][K]; the TMA producers read the scratch and wait
  // per band for stage_ready[band] to reach the number of CTAs. Each remote byte crosses NVLink exactly once.
  const void* stage_src;   // remote [N][stage_ld] bf16
  long long stage_ld;
  void* stage_dst;         // local [N][K] bf16
  int* stage_ready;        // [ceil(N / (kRasterBand * BN))] counters, zero at launch
};

// Epilogue warps per CTA: four (one per TMEM lane quadrant) for the epilogues that only store; eight (two per
// quadrant, each taking half of the tile's columns) for the SwiGLU-backward epilogue, which reads and writes four
// times the bytes of a plain store per accumulator column, and for the cross-entropy epilogues that are a long chain of
// dependent instructions per column (one warp per scheduler leaves it idle most of the time): the backward one, and the
// forward one with a soft cap's hyperbolic tangents. The forward SwiGLU epilogue (an exponential and a division per pair)
// takes eight too: with four it set the pace up to K = 4096 (2048 x 16384 x 2048 116 us, 97 with eight; 2048 x 28672 x 4096
// 324 and 319). (With eight warps the store-only kernels measured 3-5 % slower; the
// plain forward cross-entropy hides under its main loop with four.)
__host__ __device__ constexpr bool lce_keeps(int epi) { return epi == EPI_LCE_KEEP || epi == EPI_LCE_KEEP2; }
__host__ __device__ constexpr bool lce_forward(int epi) { return epi == EPI_LCE_FWD || epi == EPI_LCE_FWD2 || lce_keeps(epi); }
__host__ __device__ constexpr int gemm_epi_warps(int epi) {
  return epi == EPI_SWIGLU || epi == EPI_SWIGLU_BWD || epi == EPI_LCE_FWD2 || epi == EPI_LCE_KEEP2 || epi == EPI_LCE_BWD ? 8 : 4;
}
// The single-CTA kernel serves the grouped (mixture-of-experts) modes, whose per-expert reductions are only a few
// k-blocks long while every tile is still written in full: there the epilogue, not the main loop, sets the pace.
__host__ __device__ constexpr int gemm1_epi_warps(int epi) { return epi == EPI_LCE_FWD || epi == EPI_LCE_KEEP ? 4 : 8; }

constexpr int kEpiScratch = 2048;      // bytes of shared memory per epilogue warp (see store_pieces)

template <int BN>
struct GemmCfg {
  static constexpr int BM = 128;
  static constexpr int BK = 64;
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (BN == 256) ? 4 : 6;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/ + 8 * kEpiScratch + 8 * 8 * 8 /*norm sums*/;
  static constexpr int TMEM_COLS = 2 * BN;
};

__device__ __forceinline__ uint4 pack8_bf16(const float* v) {
  return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}
__device__ __forceinline__ void unpack8_bf16(const uint4& q, float* f) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 t = __bfloat1622float2(h[e]);
    f[2 * e] = t.x;
    f[2 * e + 1] = t.y;
  }
}
// The warp's 32 rows x 32 columns at `base` (row 0 of the warp, first column), pieces[q] = columns 8q .. 8q+7 of this
// lane's row. TMEM hands every thread one row, so a direct 16-byte store would touch 32 rows (half a sector each) per
// instruction. The block goes through kEpiScratch bytes of shared memory instead (16-byte slots permuted inside a row so
// that both sides are free of bank conflicts) and leaves with four lanes covering 64 contiguous bytes of a row.
__device__ __forceinline__ uint4* epi_slot(uint8_t* scr, int row, int piece) {
  return reinterpret_cast<uint4*>(scr + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4));
}
__device__ __forceinline__ void store_pieces(uint8_t* scr, __nv_bfloat16* base, long long ld, int rows_left, const uint4 (&pieces)[4]) {
  const int lane = threadIdx.x & 31, r0 = lane >> 2, p = lane & 3;
#pragma unroll
  for (int q = 0; q < 4; ++q) *epi_slot(scr, lane, q) = pieces[q];
  __syncwarp();
  uint4 v[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) v[s] = *epi_slot(scr, 8 * s + r0, p);
  __syncwarp();
  __nv_bfloat16* dst = base + (long long)r0 * ld + p * 8;
#pragma unroll
  for (int s = 0; s < 4; ++s)
    if (8 * s + r0 < rows_left) *reinterpret_cast<uint4*>(dst + 8 * s * ld) = v[s];
}
__device__ __forceinline__ void load_pieces(uint8_t* scr, const __nv_bfloat16* base, long long ld, int rows_left, uint4 (&pieces)[4]) {
  const int lane = threadIdx.x & 31, r0 = lane >> 2, p = lane & 3;
  const __nv_bfloat16* src = base + (long long)r0 * ld + p * 8;
  uint4 v[4];
#pragma unroll
  for (int s = 0; s < 4; ++s)
    v[s] = 8 * s + r0 < rows_left ? *reinterpret_cast<const uint4*>(src + 8 * s * ld) : make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int s = 0; s < 4; ++s) *epi_slot(scr, 8 * s + r0, p) = v[s];
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 4; ++q) pieces[q] = *epi_slot(scr, lane, q);
  __syncwarp();
}

// v / cap with the reciprocal carried in two floats (48 bits): one rounding, as in a division. A division costs the epilogue of
// the soft-capped cross-entropy 0.27 ms of 2.73 (4 x 1024 x 2048 x 50257, both directions), the product with a reciprocal of 24
// bits has a second rounding. Infinities are handed on (their tanh is 1): infinity times the low part would be NaN.
__device__ __forceinline__ float cap_quotient(const GemmParams& p, float v) {
  return fabsf(v) < INFINITY ? __fmaf_rn(v, p.inv_cap, __fmul_rn(v, p.inv_cap_lo)) : v;
}
// Stored logits: [ceil(M / 32)][ceil(N / 32)] blocks of 1,024 floats, element (r, c) of a block at (c / 4) * 128 + r * 4 + c % 4.
// A thread that owns row r of the block moves 16 bytes at a time and the 32 threads of a warp 512 contiguous ones, in the
// epilogue that writes the block as in the kernel that reads it, without a pass through shared memory.
__device__ __forceinline__ float4* z_block(float* z, int N, int row0, int col0) {
  return reinterpret_cast<float4*>(z) + ((long long)(row0 >> 5) * ((N + 31) >> 5) + (col0 >> 5)) * 256 + (threadIdx.x & 31);
}
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16(x)); }

// L2 prefetch of the 2 * BN saved pre-activation values (gate / up pairs) that the SwiGLU-backward epilogue of this
// thread's row will read: issued before the wait for the accumulator, so the loads later hit L2 instead of DRAM.
template <int BN>
__device__ __forceinline__ void prefetch_swiglu_row(const GemmParams& p, int row, int tn) {
  if (row < p.M) {
    const char* g = reinterpret_cast<const char*>(reinterpret_cast<const __nv_bfloat16*>(p.act) + (long long)row * p.ld_act +
                                                  2LL * tn * BN);
    const int cols = min(2 * BN, 2 * (p.N - tn * BN));
#pragma unroll
    for (int b = 0; b < 2 * BN * 2; b += 128)
      if (b < cols * 2) asm volatile("prefetch.global.L2 [%0];" ::"l"(g + b));
  }
}

// Epilogue of one accumulator tile, one row per thread (warp = 32 consecutive rows starting at row0). The columns come
// in chunks of 32; the whole warp takes part in every chunk, rows past M included (their stores are masked).
//
// What bounds it: the issue slots of one warp per scheduler, and the load / store unit, where a 16-byte access per row
// costs a cycle per row touched: 850 cycles per chunk with direct stores, 6,600 for a 128 x 256 tile against 512 cycles per
// 64-element step of the main loop (measured). See store_pieces for the layout used instead.
struct EpiState {
  uint8_t* scr;                // kEpiScratch bytes of shared memory of this warp
  __nv_bfloat16* C;            // row row0 of C (this batch entry)
  const __nv_bfloat16* R;
  int row, rows_left;          // this thread's row; rows from row0 to M
  bool row_ok, vec_ok, act_ok;
  float sq;                    // EPI_SUMSQ: fp32 partial (at most 256 squares per thread), flushed to fp64 by the caller
  float run_max, run_sum;      // EPI_LCE_FWD: running statistics of (row, column part)
  int label;
  float lse, coef;
};

template <int EPI>
__device__ __forceinline__ EpiState epi_begin(const GemmParams& p, uint8_t* scr, int row0, int b) {
  EpiState e;
  e.scr = scr;
  const long long off = b * p.strideC + (long long)row0 * p.ldc;
  e.row = row0 + (threadIdx.x & 31);
  e.rows_left = p.M - row0;
  e.row_ok = e.row < p.M;
  e.C = reinterpret_cast<__nv_bfloat16*>(p.C) + off;
  e.R = p.R ? reinterpret_cast<const __nv_bfloat16*>(p.R) + off : nullptr;
  e.vec_ok = ((p.ldc & 7) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0) && (((b * p.strideC) & 7) == 0) &&
             ((reinterpret_cast<uintptr_t>(p.R) & 15) == 0);
  e.act_ok = ((p.ld_act & 7) == 0) && ((reinterpret_cast<uintptr_t>(p.act) & 15) == 0);
  e.sq = 0.f;
  e.run_max = -INFINITY;
  e.run_sum = 0.f;
  e.label = -1;
  e.lse = e.coef = 0.f;
  if (lce_forward(EPI) || EPI == EPI_LCE_BWD || EPI == EPI_LCE_GRAD) {
    if (e.row_ok) e.label = p.labels[e.row];
    if ((EPI == EPI_LCE_BWD || EPI == EPI_LCE_GRAD) && e.row_ok) { e.lse = p.lse[e.row]; e.coef = p.coef[e.row]; }
  }
  return e;
}

// v: 32 fp32 accumulators of this thread's row, columns col0 .. col0+31 (col0 a multiple of 32, the same in all lanes).
template <int EPI>
__device__ __forceinline__ void epi_chunk(const GemmParams& p, EpiState& e, float (&v)[32], int col0) {
  const int ncols = min(32, p.N - col0);
  if (ncols <= 0 || e.rows_left <= 0) return;      // the same in all lanes
  const bool full = ncols == 32 && e.vec_ok;
  __nv_bfloat16* Crow = e.C + (long long)(threadIdx.x & 31) * p.ldc + col0;
  if (EPI == EPI_LCE_GRAD) {
    // the stored values are scaled already
  } else if (EPI == EPI_STORE && p.stepwise) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = bf16_round(__fmul_rn(bf16_round(v[j]), p.alpha));
  } else if (p.alpha != 1.f) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] *= p.alpha;
  }

  if (EPI == EPI_STORE || EPI == EPI_SUMSQ || EPI == EPI_SWIGLU) {
    if (p.bias) {
      const __nv_bfloat16* bs = reinterpret_cast<const __nv_bfloat16*>(p.bias) + col0;
      if (ncols == 32 && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float f[8];
          unpack8_bf16(reinterpret_cast<const uint4*>(bs)[q], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[8 * q + j] += f[j];
        }
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) if (j < ncols) v[j] += __bfloat162float(bs[j]);
      }
    }
    if (e.R) {
      if (full) {
        uint4 r[4];
        load_pieces(e.scr, e.R + col0, p.ldc, e.rows_left, r);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float f[8];
          unpack8_bf16(r[q], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[8 * q + j] += f[j];
        }
      } else if (e.row_ok) {
        const __nv_bfloat16* Rrow = e.R + (long long)(threadIdx.x & 31) * p.ldc + col0;
#pragma unroll
        for (int j = 0; j < 32; ++j) if (j < ncols) v[j] += __bfloat162float(Rrow[j]);
      }
    }
    if (full) {
      uint4 o[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) o[q] = pack8_bf16(v + 8 * q);
      if (EPI == EPI_SUMSQ && e.row_ok) {     // squares of the stored values, column by column
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float f[8];
          unpack8_bf16(o[q], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) e.sq += f[j] * f[j];
        }
      }
      if (EPI != EPI_SUMSQ || p.C) store_pieces(e.scr, e.C + col0, p.ldc, e.rows_left, o);   // EPI_SUMSQ without C: norm only
    } else if (e.row_ok) {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < ncols) {
          const float q = bf16_round(v[j]);
          if (EPI == EPI_SUMSQ) e.sq += q * q;
          if (EPI != EPI_SUMSQ || p.C) Crow[j] = __float2bfloat16(q);
        }
    }
    if (EPI == EPI_SWIGLU) {
      float a[16];
      // Not for rows past M: their accumulators are zero, and a division of zero leaves the fast path of the whole warp (with
      // four epilogue warps 1021 x 16384 x 2048 took 101 us so and 72 without them, 317 x 16384 x 2048 72 and 42).
      if (e.row_ok) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          // match the stored (bf16-rounded) pre-activations so backward recomputes the same values
          const float g = bf16_round(v[2 * j]), u = bf16_round(v[2 * j + 1]);
          a[j] = g / (1.f + __expf(-g)) * u;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) a[j] = 0.f;
      }
      const int lane = threadIdx.x & 31;
      __nv_bfloat16* act0 = reinterpret_cast<__nv_bfloat16*>(p.act) + (long long)(e.row - lane) * p.ld_act + (col0 >> 1);
      if (ncols == 32 && e.act_ok) {
        // two pieces per row through the same scratch: two lanes cover the 32 contiguous bytes of a row
        auto slot = [&](int row, int piece) { return reinterpret_cast<uint4*>(e.scr + row * 32 + ((piece ^ ((row >> 2) & 1)) << 4)); };
        *slot(lane, 0) = pack8_bf16(a);
        *slot(lane, 1) = pack8_bf16(a + 8);
        __syncwarp();
        const int r0 = lane >> 1, q = lane & 1;
        const uint4 lo = *slot(r0, q), hi = *slot(16 + r0, q);
        __syncwarp();
        __nv_bfloat16* dst = act0 + (long long)r0 * p.ld_act + q * 8;
        if (r0 < e.rows_left) *reinterpret_cast<uint4*>(dst) = lo;
        if (16 + r0 < e.rows_left) *reinterpret_cast<uint4*>(dst + 16 * p.ld_act) = hi;
      } else if (e.row_ok) {
        const int na = ncols >> 1;
        __nv_bfloat16* arow = act0 + (long long)lane * p.ld_act;
#pragma unroll
        for (int j = 0; j < 16; ++j) if (j < na) arow[j] = __float2bfloat16(a[j]);
      }
    }
  } else if (EPI == EPI_SWIGLU_BWD) {
    // 32 accumulator columns = 32 (gate, up) pairs = 64 stored columns, read and written as two halves of 64 bytes per row
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16* g0 = reinterpret_cast<const __nv_bfloat16*>(p.act) + (long long)(e.row - lane) * p.ld_act + 2 * col0;
    if (full && e.act_ok) {
      uint4 gin[2][4];
      load_pieces(e.scr, g0, p.ld_act, e.rows_left, gin[0]);
      load_pieces(e.scr, g0 + 32, p.ld_act, e.rows_left, gin[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float gu[8];
          unpack8_bf16(gin[h][q], gu);
          float o[8];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float d = bf16_round(v[16 * h + 4 * q + t]);
            const float sg = 1.f / (1.f + __expf(-gu[2 * t]));
            o[2 * t] = d * gu[2 * t + 1] * (sg * (1.f + gu[2 * t] * (1.f - sg)));
            o[2 * t + 1] = d * (gu[2 * t] * sg);
          }
          gin[h][q] = pack8_bf16(o);
        }
        store_pieces(e.scr, e.C + 2 * col0 + 32 * h, p.ldc, e.rows_left, gin[h]);
      }
    } else if (e.row_ok) {
      const __nv_bfloat16* grow = g0 + (long long)lane * p.ld_act;
      __nv_bfloat16* drow = Crow + col0;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < ncols) {
          const float g = __bfloat162float(grow[2 * j]), u = __bfloat162float(grow[2 * j + 1]);
          const float d = bf16_round(v[j]);
          const float sg = 1.f / (1.f + __expf(-g));
          drow[2 * j] = __float2bfloat16(d * u * (sg * (1.f + g * (1.f - sg))));
          drow[2 * j + 1] = __float2bfloat16(d * (g * sg));
        }
    }
  } else if (lce_forward(EPI)) {
    if (p.softcap > 0.f) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        v[j] = tanhf(cap_quotient(p, v[j]));
        if (!lce_keeps(EPI)) v[j] *= p.softcap;
      }
    }
    if constexpr (lce_keeps(EPI)) {      // the scaled logit, or the hyperbolic tangent of the soft cap: what EPI_LCE_GRAD starts from
      float4* z = z_block(p.z, p.N, e.row - (int)(threadIdx.x & 31), col0);
#pragma unroll
      for (int q = 0; q < 8; ++q) __stcs(z + 32 * q, make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
      if (p.softcap > 0.f) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] *= p.softcap;
      }
    }
    float cmax = -INFINITY;
#pragma unroll
    for (int j = 0; j < 32; ++j) if (j < ncols) cmax = fmaxf(cmax, v[j]);
    const float nmax = fmaxf(e.run_max, cmax);
    float add = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) if (j < ncols) add += __expf(v[j] - nmax);
    e.run_sum = e.run_sum * __expf(e.run_max - nmax) + add;
    e.run_max = nmax;
    if (e.label >= col0 && e.label < col0 + ncols) {
      float t = 0.f;
#pragma unroll
      for (int j = 0; j < 32; ++j) if (col0 + j == e.label) t = v[j];
      p.tgt[e.row] = t;
    }
  } else {  // EPI_LCE_BWD, EPI_LCE_GRAD
    if (p.softcap > 0.f) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float th = EPI == EPI_LCE_GRAD ? v[j] : tanhf(cap_quotient(p, v[j]));
        const float pr = __expf(p.softcap * th - e.lse);
        v[j] = (pr - ((col0 + j == e.label) ? 1.f : 0.f)) * e.coef * (1.f - th * th);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = (__expf(v[j] - e.lse) - ((col0 + j == e.label) ? 1.f : 0.f)) * e.coef;
    }
    if (full) {
      uint4 o[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) o[q] = pack8_bf16(v + 8 * q);
      store_pieces(e.scr, e.C + col0, p.ldc, e.rows_left, o);
    } else if (e.row_ok) {
#pragma unroll
      for (int j = 0; j < 32; ++j) if (j < ncols) Crow[j] = __float2bfloat16(v[j]);
    }
  }
}

// part: index of this (column tile, column part of the tile); parts: their number per row.
template <int EPI>
__device__ __forceinline__ void epi_end(const GemmParams& p, const EpiState& e, int part, int parts) {
  if (lce_forward(EPI) && e.row_ok) {
    p.pmax[(long long)e.row * parts + part] = e.run_max;
    p.psum[(long long)e.row * parts + part] = e.run_sum;
  }
}

// Squared norm of one finished tile. All tiles of a launch usually add to ONE double, and atomics on one address are served
// one after the other (about 5 ns each: 4,096 of them, one per tile and warp of a 16384 x 2048 gradient, took 20 us, and
// the 65,536 of an OLMoE expert gradient 320 us, longer than the products). So lane 0 of every epilogue warp keeps a
// running double per sum in shared memory (`slots`, kSqSums per warp), and the CTA adds its warps' sums once, when it is done
// (epi_flush_sq). Only launches with more than kSqSums sums (one per batch entry, sumsq_stride != 0) add per tile.
constexpr int kSqSums = 8;
__device__ __forceinline__ int sq_sums(const GemmParams& p) { return p.sumsq_stride == 0 ? 1 : p.batch; }
__device__ __forceinline__ void epi_zero_sq(double* slots) {
  const int lane = threadIdx.x & 31;
  if (lane < kSqSums) slots[lane] = 0.0;
  __syncwarp();
}
__device__ __forceinline__ void epi_add_sq(const GemmParams& p, const EpiState& e, int b, double* slots) {
  float w = e.sq;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  if ((threadIdx.x & 31) == 0) {
    if (sq_sums(p) <= kSqSums) slots[p.sumsq_stride == 0 ? 0 : b] += (double)w;
    else atomicAdd(&p.sumsq[b * p.sumsq_stride], (double)w);
  }
}
// After a CTA barrier behind the warps' last tiles, by the first kSqSums threads: `slots` of all `warps` epilogue warps.
__device__ __forceinline__ void epi_flush_sq(const GemmParams& p, const double* slots, int warps) {
  const int n = sq_sums(p);
  if (n > kSqSums || (int)threadIdx.x >= n) return;
  double t = 0.0;
  for (int i = 0; i < warps; ++i) t += slots[i * kSqSums + threadIdx.x];
  if (t != 0.0) atomicAdd(p.sumsq + threadIdx.x, t);
}

// Columns [c_begin, c_end) of one accumulator tile, read from TMEM (tmem_tile = lane-adjusted address of the tile).
// `release` runs once, in all lanes, as soon as the last column has left TMEM: before the last chunk is processed, so that
// the tensor cores get the buffer back while its values are still being stored.
template <int BN, int EPI, class Release>
__device__ __forceinline__ void epilogue_tile(const GemmParams& p, EpiState& e, uint32_t tmem_tile, int n0, int c_begin, int c_end,
                                              Release release) {
#pragma unroll 1
  for (int c0 = c_begin; c0 < c_end; c0 += 32) {
    uint32_t raw[32];
    __syncwarp();  // tcgen05.ld is warp-collective
    tmem_ld32(tmem_tile + c0, raw);
    tc_wait_ld();
    if (c0 + 32 >= c_end) release();
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(raw[j]);
    epi_chunk<EPI>(p, e, v, n0 + c0);
  }
}

// Tile order of the persistent schedule. Column tiles are walked in bands of kRasterBand; inside a band the column
// index runs fastest, then the row index. The CTAs that run at the same time therefore cover a roughly square patch
// of the output (8 column tiles x as many row tiles as there are CTAs / 8): the band's B tiles and the patch's A tiles
// stay in L2 and each operand is fetched from DRAM about once per band instead of once per column tile.
constexpr int kRasterBand = 8;
__device__ __forceinline__ void tile_coords(int r, int tiles_m, int tiles_n, int& tm, int& tn) {
  const int band_tiles = kRasterBand * tiles_m;
  const int band = r / band_tiles;
  const int rr = r - band * band_tiles;
  const int w = min(kRasterBand, tiles_n - band * kRasterBand);
  tm = rr / w;
  tn = band * kRasterBand + (rr - tm * w);
}

// The four products of one 64-element block of the reduction (operand tiles at the shared addresses sa and sb).
template <bool A_MN, bool B_MN, bool PAIR>
__device__ __forceinline__ void issue_kblock(uint32_t d_tmem, uint32_t sa, uint32_t sb, uint32_t idesc, bool first) {
  // a step of 16 reduction elements: 32 bytes inside a K-major row, 16 rows of 128 bytes of an MN-major tile
  const uint64_t ad = A_MN ? make_smem_desc(sa, 64 * 128, 1024) : make_smem_desc(sa, 16, 1024);
  const uint64_t bd = B_MN ? make_smem_desc(sb, 64 * 128, 1024) : make_smem_desc(sb, 16, 1024);
#pragma unroll
  for (int k4 = 0; k4 < 4; ++k4) {
    const uint64_t ak = ad + k4 * (A_MN ? 2048 / 16 : 32 / 16), bk = bd + k4 * (B_MN ? 2048 / 16 : 32 / 16);
    const uint32_t acc = (k4 != 0 || !first) ? 1u : 0u;
    if (PAIR) umma2_bf16(d_tmem, ak, bk, idesc, acc);
    else umma_bf16(d_tmem, ak, bk, idesc, acc);
  }
}

template <bool A_MN, bool B_MN, int BN, int EPI>
__global__ void __launch_bounds__(64 + 32 * gemm1_epi_warps(EPI), 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const GemmParams p) {
  using Cfg = GemmCfg<BN>;
  constexpr int BM = Cfg::BM, BK = Cfg::BK, STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  double* sq_slots = reinterpret_cast<double*>(smem + STAGES * Cfg::STAGE_BYTES + 256 + 8 * kEpiScratch);   // EPI_SUMSQ: [warp][kSqSums]

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], gemm1_epi_warps(EPI));
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();          // no early trigger: a waiting successor would keep the second stream's kernels off the SMs this grid's last wave leaves idle

  const int tiles_m = (p.M + BM - 1) / BM;
  const int tiles_n = (p.N + BN - 1) / BN;
  const int per_batch = tiles_m * tiles_n;
  const int total = per_batch * p.batch;
  const int kblocks = (p.K + BK - 1) / BK;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
      const int b = tile / per_batch;
      const int r = tile - b * per_batch;
      int tm, tn;
      tile_coords(r, tiles_m, tiles_n, tm, tn);
      int bb = b / p.b_batch_div, ba = b;
      int kb0 = 0, nkb = kblocks;
      if (p.tile_group) {
        bb = p.tile_group[tm];
        if (bb < 0) continue;
      }
      if (p.group_k) { kb0 = p.group_k[2 * b] / BK; nkb = p.group_k[2 * b + 1]; ba = 0; bb = 0; }
      for (int kq = 0; kq < nkb; ++kq) {
        const int kb = kb0 + kq;
        if (!mbar_wait_warp(&empty[s], ph ^ 1u, abort_flag)) { ok = false; break; }
        if (elect_one()) {
          uint8_t* sa = smem + s * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + Cfg::A_BYTES;
          mbar_expect_tx(&full[s], Cfg::STAGE_BYTES);
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_3d(sa + j * (BK * 128), &tmA, &full[s], tm * BM + j * 64, kb * BK, ba);
          } else {
            tma_load_3d(sa, &tmA, &full[s], kb * BK, tm * BM, ba);
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
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    constexpr uint32_t idesc = make_idesc_bf16(BM, BN, A_MN, B_MN);
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    int it = 0;
    for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
      int nkb = kblocks;
      if (p.tile_group || p.group_k) {
        const int b = tile / per_batch;
        const int r = tile - b * per_batch;
        int tm, tn;
        tile_coords(r, tiles_m, tiles_n, tm, tn);
        if (p.tile_group && p.tile_group[tm] < 0) continue;
        if (p.group_k) nkb = p.group_k[2 * b + 1];
      }
      const int buf = it & 1;
      const uint32_t tph = (it >> 1) & 1;
      ++it;
      if (!mbar_wait_warp(&tempty[buf], tph ^ 1u, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + buf * BN;
      for (int kb = 0; kb < nkb; ++kb) {
        if (!mbar_wait_warp(&full[s], ph, abort_flag)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const uint32_t sa = smem_u32(smem + s * Cfg::STAGE_BYTES);
          issue_kblock<A_MN, B_MN, false>(d_tmem, sa, sa + Cfg::A_BYTES, idesc, kb == 0);
          umma_commit(&empty[s]);  // frees the smem stage once these UMMAs have read it
        }
        __syncwarp();
        if (++s == STAGES) { s = 0; ph ^= 1u; }
      }
      if (ok && elect_one()) umma_commit(&tfull[buf]);
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------ epilogue (one TMEM lane quadrant per warp & 3)
    const int quad = warp & 3;
    constexpr int CSPLIT = gemm1_epi_warps(EPI) / 4;
    const int c_begin = ((warp - 2) >> 2) * (BN / CSPLIT), c_end = c_begin + BN / CSPLIT;
    uint8_t* scratch = smem + STAGES * Cfg::STAGE_BYTES + 256 + (warp - 2) * kEpiScratch;
    int it = 0;
    double* sq = sq_slots + (warp - 2) * kSqSums;
    if (EPI == EPI_SUMSQ) epi_zero_sq(sq);
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      const int b = tile / per_batch;
      const int r = tile - b * per_batch;
      int tm, tn;
      tile_coords(r, tiles_m, tiles_n, tm, tn);
      if (p.tile_group && p.tile_group[tm] < 0) continue;
      const int buf = it & 1;
      const uint32_t tph = (it >> 1) & 1;
      ++it;
      if (EPI == EPI_SWIGLU_BWD) prefetch_swiglu_row<BN>(p, tm * BM + quad * 32 + lane, tn);
      int ok = 1;
      if (lane == 0) ok = mbar_wait(&tfull[buf], tph, abort_flag) ? 1 : 0;
      __syncwarp();   // orders the other lanes' accesses after lane 0's acquire (a shuffle is no memory barrier)
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      tc_fence_after();

      EpiState e = epi_begin<EPI>(p, scratch, tm * BM + quad * 32, b);
      epilogue_tile<BN, EPI>(p, e, tmem_base + (uint32_t(quad * 32) << 16) + buf * BN, tn * BN, c_begin, c_end, [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_relaxed(&tempty[buf]);
      });
      epi_end<EPI>(p, e, tn * CSPLIT + c_begin / (BN / CSPLIT), tiles_n * CSPLIT);
      if (EPI == EPI_SUMSQ) epi_add_sq(p, e, b, sq);
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
  if (EPI == EPI_SUMSQ) epi_flush_sq(p, sq_slots, gemm1_epi_warps(EPI));
  if (threadIdx.x == 0 && *abort_flag && p.err) atomicExch(p.err, 1);
}

}  // namespace opk
