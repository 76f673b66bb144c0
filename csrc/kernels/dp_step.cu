// Differential-privacy step kernels for sm_100a:
//   * guarded clip scale from a per-example squared norm (conservative rounding: the stored clipped
//     gradient never exceeds the clipping norm),
//   * clipped accumulation  acc += bf16(g * scale),
//   * counter-based Philox4x32-10 Gaussian noise indexed by the global element offset, so every
//     sharding of the parameter vector draws the same global noise tensor exactly once,
//   * the fused step: reduce-scatter of the clipped-gradient sums over peer memory (plain P2P loads),
//     normalisation, noise (optionally correlated through a buffered-linear-Toeplitz state), DP-AdamW with
//     noise bias correction, and the all-gather of the updated bf16 parameters as P2P stores.
#include "opk_api.h"
#include "philox.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>

namespace {

#define OPK_LAUNCH_CHECK()                                   \
  do {                                                       \
    cudaError_t e__ = cudaGetLastError();                    \
    if (e__ != cudaSuccess) return (int)e__;                 \
  } while (0)

// ------------------------------------------------------------------------------------------- Philox4x32-10
using opk::normal4;

__global__ void philox_normal_kernel(float* __restrict__ out, long long n, uint64_t seed, uint32_t stream_id,
                                     uint32_t step, uint64_t offset, float sigma, int accumulate) {
  // thread handles one aligned quad of the GLOBAL index space; elements outside [offset, offset+n) are skipped
  const uint64_t q0 = offset >> 2;
  const uint64_t q1 = (offset + (uint64_t)n + 3) >> 2;
  for (uint64_t q = q0 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < q1; q += (uint64_t)gridDim.x * blockDim.x) {
    float z[4];
    normal4(q, seed, stream_id, step, z);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t e = q * 4 + j;
      if (e >= offset && e < offset + (uint64_t)n) {
        const long long i = (long long)(e - offset);
        out[i] = accumulate ? out[i] + sigma * z[j] : sigma * z[j];
      }
    }
  }
}

// ------------------------------------------------------------------------------------------- clip scale
// Conservative clip factor (fixed clipping): the factor is shrunk by the worst-case rounding of the norm
// accumulation, of the fp32 multiply and of the bf16 store, so that the norm of the *stored* clipped gradient
// is <= clip. AUTO-S (mode_auto): R / (norm + gamma) with the same guard and no clamp to one.
__global__ void clip_scale_kernel(double* sumsq, float clip, int mode_auto, float gamma, int n_leaves,
                                  long long widest_leaf, float* scale_out, float* norm_out, int* counters, int reset,
                                  const float* loss, float* loss_sum) {
  const int j = threadIdx.x;             // one example per thread
  if (loss_sum && j == 0) {              // in the order of the examples, as one by one
    float sum = *loss_sum;
    for (int k = 0; k < (int)blockDim.x; ++k) sum += loss[k];
    *loss_sum = sum;
  }
  const double sq = sumsq[j];
  if (reset) sumsq[j] = 0.0;
  const double norm = sqrt(sq > 0.0 ? sq : 0.0);
  if (norm_out) norm_out[j] = (float)norm;
  const double c = clip > 0.f ? (double)clip : 0.0;
  double ratio;
  if (mode_auto) ratio = c / (norm + (double)gamma);
  else ratio = norm > 0.0 ? c / norm : INFINITY;
  if (counters && !mode_auto && norm > c) atomicAdd(counters, 1);
  // unit roundoffs
  const double u_acc = 1.1920928955078125e-07 / 2.0;   // fp32
  const double u_sq = 2.220446049250313e-16 / 2.0;     // fp64
  const double n_red = widest_leaf > 4096 ? 2048.0 + ceil((double)widest_leaf / 2048.0) : (double)widest_leaf;
  // the tile epilogues add 256 squares per thread in fp32 plus a 5-level shuffle tree before going to fp64
  const double tile_slack = 264.0 * u_acc;
  const double roundoff = (u_acc + ((double)(n_leaves > 1 ? n_leaves : 1) + n_red) * u_sq + tile_slack) / 2.0;
  const double store_eps = 0.0078125, mult_eps = 1.1920928955078125e-07;  // bf16 store, fp32 multiply
  const double rounding = store_eps / 2.0 + mult_eps;
  double s = ratio * (1.0 - rounding - 2.0 * roundoff) - 1.1754943508222875e-38 * store_eps;
  if (!mode_auto && s > 1.0) s = 1.0;
  if (!isfinite(s)) s = (!mode_auto && ratio > 0) ? 1.0 : 0.0;
  if (s < 0.0) s = 0.0;
  if (clip <= 0.f) s = 0.0;
  // round the fp32 factor toward zero so the cast itself cannot enlarge it
  float sf = (float)s;
  if ((double)sf > s) sf = nextafterf(sf, 0.0f);
  scale_out[j] = sf;
}

struct alignas(16) bf16x8 { __nv_bfloat162 h[4]; };

// a value that rounded *up* into (or within) the subnormal range would break the bound: flush it
__device__ __forceinline__ float flush_rounded_up(float stored, float scaled) {
  return fabsf(stored) <= 1.1754943508222875e-38f && fabsf(stored) > fabsf(scaled) ? 0.f : stored;
}
__device__ __forceinline__ float clip_store(float g, float s) {
  const float scaled = g * s;
  return flush_rounded_up(__bfloat162float(__float2bfloat16(scaled)), scaled);
}

__global__ void __launch_bounds__(256) clip_accumulate_kernel(const bf16x8* __restrict__ g, const float* __restrict__ scale,
                                                              float4* __restrict__ acc, long long nvec, int overwrite) {
  const float s = *scale;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < nvec; i += (long long)gridDim.x * 256) {
    // streaming accesses: this kernel runs next to tensor-core GEMMs whose operand tiles live in L2
    const uint4 raw = __ldcs(reinterpret_cast<const uint4*>(g) + i);
    const bf16x8 v = *reinterpret_cast<const bf16x8*>(&raw);
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 t = __bfloat1622float2(v.h[j]);
      f[2 * j] = t.x;
      f[2 * j + 1] = t.y;
    }
    float4 a0, a1;
    if (overwrite) {
      a0 = make_float4(0.f, 0.f, 0.f, 0.f);
      a1 = a0;
    } else {
      a0 = __ldcs(acc + 2 * i);
      a1 = __ldcs(acc + 2 * i + 1);
    }
    a0.x += clip_store(f[0], s); a0.y += clip_store(f[1], s); a0.z += clip_store(f[2], s); a0.w += clip_store(f[3], s);
    a1.x += clip_store(f[4], s); a1.y += clip_store(f[5], s); a1.z += clip_store(f[6], s); a1.w += clip_store(f[7], s);
    __stcs(acc + 2 * i, a0);
    __stcs(acc + 2 * i + 1, a1);
  }
}
// N examples in one pass over the fp32 sums: acc += sum_j stored(g_j * s_j). Per example this moves 2 + 8 / N bytes per
// parameter; N is bounded by how many whole-model gradient buffers fit next to the optimizer state.
struct AccGroup {
  const bf16x8* g[OPK_ACC_GROUP_MAX];
  const float* scale[OPK_ACC_GROUP_MAX];
};
template <int N>
__global__ void __launch_bounds__(256) clip_accumulate_group_kernel(const AccGroup grp, float4* __restrict__ acc, long long nvec,
                                                                    int overwrite) {
  float s[N];
#pragma unroll
  for (int j = 0; j < N; ++j) s[j] = *grp.scale[j];
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < nvec; i += (long long)gridDim.x * 256) {
    uint4 r[N];
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] = __ldcs(reinterpret_cast<const uint4*>(grp.g[j]) + i);
    float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
    if (!overwrite) {
      a0 = __ldcs(acc + 2 * i);
      a1 = __ldcs(acc + 2 * i + 1);
    }
    float f[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) f[q] = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {       // examples in slot order: the sum does not depend on the launch shape
      const bf16x8 v = *reinterpret_cast<const bf16x8*>(&r[j]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 t = __bfloat1622float2(v.h[q]);
        f[2 * q] += clip_store(t.x, s[j]);
        f[2 * q + 1] += clip_store(t.y, s[j]);
      }
    }
    a0.x += f[0]; a0.y += f[1]; a0.z += f[2]; a0.w += f[3];
    a1.x += f[4]; a1.y += f[5]; a1.z += f[6]; a1.w += f[7];
    __stcs(acc + 2 * i, a0);
    __stcs(acc + 2 * i + 1, a1);
  }
}
__global__ void clip_accumulate_tail_kernel(const __nv_bfloat16* __restrict__ g, const float* __restrict__ scale,
                                            float* __restrict__ acc, long long begin, long long n, int overwrite) {
  const float s = *scale;
  const long long i = begin + blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) acc[i] = (overwrite ? 0.f : acc[i]) + clip_store(__bfloat162float(g[i]), s);
}

// ------------------------------------------------------------------------------------------- fused DP step
struct StepParams {
  OpkDpStepArgs a;
};

constexpr int MAX_PEERS = 16;
struct PeerTable {
  const float* grad[MAX_PEERS];
  __nv_bfloat16* param[MAX_PEERS];
};

// Two lanes of fp32 arithmetic per instruction: same rounding as the scalar forms, half the issue slots.
__device__ __forceinline__ float2 pair(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// Two parameter updates given the averaged, noised gradients. Returns the new parameter values.
template <bool ADAM>
__device__ __forceinline__ float2 dp_update(const OpkDpStepArgs& a, float inv_bc1, float inv_bc2, float2 grad, float2 p_old,
                                            float2& m, float2& v) {
  float2 upd;
  if (!ADAM) {
    upd = fma2(pair(a.weight_decay), p_old, grad);
  } else {
    m = fma2(pair(a.beta1), m, mul2(pair(1.f - a.beta1), grad));
    v = fma2(pair(a.beta2), v, mul2(mul2(pair(1.f - a.beta2), grad), grad));
    const float2 mh = mul2(m, pair(inv_bc1)), vh = mul2(v, pair(inv_bc2));
    const float2 d = add2(vh, pair(-a.phi_hat));            // noise bias correction: subtract the noise's share of v-hat
    const float2 den = add2(make_float2(sqrtf(d.x > 0.f ? d.x : vh.x), sqrtf(d.y > 0.f ? d.y : vh.y)), pair(a.eps));
    upd = fma2(pair(a.weight_decay), p_old, make_float2(__fdividef(mh.x, den.x), __fdividef(mh.y, den.y)));
  }
  return fma2(pair(-a.lr), upd, p_old);
}

// Correlated-noise transforms of the iid draw z (DP-FTRL), applied element-wise on the shard:
//   CORR_BLT       buffered linear Toeplitz C^{-1}: zhat = z - <scale, state>; state_k = decay_k * state_k + zhat
//   CORR_TOEPLITZ  banded Toeplitz C^{-1} (band-MF, banded square root): zhat = (z - sum_{k>=1} c_k zhat_{t-k}) / c_0
//                  with the last nlag outputs kept in a ring; lag k lives in ring slot (pos + k - 1) mod nlag and the
//                  new output overwrites the oldest slot, (pos + nlag - 1) mod nlag, which the host makes the next pos
enum { CORR_NONE = 0, CORR_BLT = 1, CORR_TOEPLITZ = 2 };

// VEC consecutive elements of a streamed array: one 32-byte access (8 floats), or 16 bytes where the alignment allows no more.
// Everything is touched once: streaming loads and stores.
template <int VEC>
__device__ __forceinline__ void ld_stream(const float* p, float (&o)[VEC]) {
  static_assert(VEC == 4 || VEC == 8);
  if constexpr (VEC == 8)
    asm volatile("ld.global.cs.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4]), "=f"(o[5]), "=f"(o[6]), "=f"(o[7])
                 : "l"(p));
  else
    asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]) : "l"(p));
}
template <int VEC>
__device__ __forceinline__ void st_stream(float* p, const float (&o)[VEC]) {
  if constexpr (VEC == 8)
    asm volatile("st.global.cs.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(o[0]), "f"(o[1]), "f"(o[2]), "f"(o[3]),
                 "f"(o[4]), "f"(o[5]), "f"(o[6]), "f"(o[7]));
  else
    asm volatile("st.global.cs.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(o[0]), "f"(o[1]), "f"(o[2]), "f"(o[3]));
}
template <int VEC>
__device__ __forceinline__ void ld_stream(const __nv_bfloat16* p, uint32_t (&o)[VEC / 2]) {
  if constexpr (VEC == 8)
    asm volatile("ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3]) : "l"(p));
  else
    asm volatile("ld.global.cs.v2.u32 {%0, %1}, [%2];" : "=r"(o[0]), "=r"(o[1]) : "l"(p));
}
__device__ __forceinline__ float2 unpack2(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w)); }

// The rows of correlation state that a vector needs first are loaded with everything else (four rows: BLT with up to four buffers
// needs no other access before its stores; two in vectors of eight next to eight gradient buffers, which leave no registers for more).
template <int CORR, int VEC, int ROWS>
struct CorrIn {
  float row[ROWS][VEC];
};
template <int VEC, int ROWS>
struct CorrIn<CORR_NONE, VEC, ROWS> {};

__device__ __forceinline__ int toep_slot(const OpkDpStepArgs& a, int k) {      // ring slot of lag k + 1
  const int slot = a.toep_pos + k;
  return slot >= a.toep_nlag ? slot - a.toep_nlag : slot;
}
template <int CORR, int VEC, int ROWS>
__device__ __forceinline__ void load_corr(const OpkDpStepArgs& a, long long i0, int first, CorrIn<CORR, VEC, ROWS>& in) {
  if constexpr (CORR == CORR_BLT) {
#pragma unroll
    for (int k = 0; k < ROWS; ++k)
      if (first + k < a.blt_nbuf) ld_stream<VEC>(a.blt_state + (long long)(first + k) * a.shard_len + i0, in.row[k]);
  } else if constexpr (CORR == CORR_TOEPLITZ) {
#pragma unroll
    for (int k = 0; k < ROWS; ++k)
      if (first + k < a.toep_nlag) ld_stream<VEC>(a.toep_state + (long long)toep_slot(a, first + k) * a.shard_len + i0, in.row[k]);
  }
}
template <int CORR, int VEC, int ROWS>
__device__ __forceinline__ void correlate(const OpkDpStepArgs& a, long long i0, CorrIn<CORR, VEC, ROWS>& in, float (&z)[VEC]) {
  if constexpr (CORR != CORR_NONE) {
    const int rows = CORR == CORR_BLT ? a.blt_nbuf : a.toep_nlag;
    float rd[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) rd[j] = 0.f;
    for (int first = 0; first < rows; first += ROWS) {
      if (first) load_corr<CORR, VEC, ROWS>(a, i0, first, in);
#pragma unroll
      for (int k = 0; k < ROWS; ++k)
        if (first + k < rows) {
          const float c = CORR == CORR_BLT ? a.blt_scale[first + k] : a.toep_coef[first + k + 1];
#pragma unroll
          for (int j = 0; j < VEC; ++j) rd[j] += c * in.row[k][j];
        }
    }
    if constexpr (CORR == CORR_BLT) {
#pragma unroll
      for (int j = 0; j < VEC; ++j) z[j] -= rd[j];
      for (int first = 0; first < rows; first += ROWS) {
        if (rows > ROWS) load_corr<CORR, VEC, ROWS>(a, i0, first, in);
#pragma unroll
        for (int k = 0; k < ROWS; ++k)
          if (first + k < rows) {
            const float dc = a.blt_decay[first + k];
            float st[VEC];
#pragma unroll
            for (int j = 0; j < VEC; ++j) st[j] = dc * in.row[k][j] + z[j];
            st_stream<VEC>(a.blt_state + (long long)(first + k) * a.shard_len + i0, st);
          }
      }
    } else {
      const float inv_c0 = 1.f / a.toep_coef[0];
#pragma unroll
      for (int j = 0; j < VEC; ++j) z[j] = (z[j] - rd[j]) * inv_c0;
      if (rows > 0) st_stream<VEC>(a.toep_state + (long long)(a.toep_pos == 0 ? rows - 1 : a.toep_pos - 1) * a.shard_len + i0, z);
    }
  }
}
template <int CORR>
__device__ __forceinline__ float correlate_one(const OpkDpStepArgs& a, long long i, float z) {
  if (CORR == CORR_BLT) {
    float rd = 0.f;
    for (int k = 0; k < a.blt_nbuf; ++k) rd += a.blt_scale[k] * a.blt_state[(long long)k * a.shard_len + i];
    z -= rd;
    for (int k = 0; k < a.blt_nbuf; ++k) {
      float* sp = &a.blt_state[(long long)k * a.shard_len + i];
      *sp = a.blt_decay[k] * (*sp) + z;
    }
  } else if (CORR == CORR_TOEPLITZ) {
    float rd = 0.f;
    int slot = a.toep_pos;
    for (int k = 1; k <= a.toep_nlag; ++k) {
      rd += a.toep_coef[k] * a.toep_state[(long long)slot * a.shard_len + i];
      if (++slot == a.toep_nlag) slot = 0;
    }
    z = (z - rd) / a.toep_coef[0];
    if (a.toep_nlag > 0) a.toep_state[(long long)(a.toep_pos == 0 ? a.toep_nlag - 1 : a.toep_pos - 1) * a.shard_len + i] = z;
  }
  return z;
}

// Everything a vector of elements needs from memory, fetched before any arithmetic.
template <int NG, int CORR, int VEC>
struct VecIn {
  float g[VEC], m[VEC], v[VEC], mw[VEC];
  uint32_t pw[VEC / 2], gr[NG > 0 ? NG : 1][VEC / 2];
  CorrIn<CORR, VEC, (NG > 2 && CORR == CORR_BLT && VEC == 8 ? 2 : 4)> corr;
};
// NG > 0 (the most buffers the variant takes: 2, or all 8): the last group of per-example gradients is clipped and added here
// instead of in a pass of its own. A separate pass reads and writes the fp32 sums once more and the step reads them again: 12 bytes
// per parameter (with the zeroing of the sums, which a first group that overwrites them makes unnecessary), 2.8 ms of a 58 ms step
// at 1.49e9 parameters.
struct StepGroup {
  const __nv_bfloat16* g[OPK_ACC_GROUP_MAX];
  const float* scale[OPK_ACC_GROUP_MAX];
  int n, skip_sum;
  long long len;
};
template <int NG, int CORR, int VEC>
__device__ __forceinline__ void add_group(const StepGroup& grp, const float (&s)[NG > 0 ? NG : 1], const VecIn<NG, CORR, VEC>& q,
                                          float (&gr)[VEC]) {
  float2 f[VEC / 2];
#pragma unroll
  for (int k = 0; k < VEC / 2; ++k) f[k] = pair(0.f);
#pragma unroll
  for (int j = 0; j < NG; ++j)
    if (j < grp.n) {                    // examples in slot order, as in the separate pass
      float2 scaled[VEC / 2], stored[VEC / 2];
      float least = INFINITY;
#pragma unroll
      for (int k = 0; k < VEC / 2; ++k) {
        scaled[k] = mul2(unpack2(q.gr[j][k]), pair(s[j]));
        stored[k] = __bfloat1622float2(__floats2bfloat162_rn(scaled[k].x, scaled[k].y));
        least = fminf(least, fminf(fabsf(scaled[k].x), fabsf(scaled[k].y)));
      }
      if (least < 1.1754943508222875e-38f) {      // clip_store: only a subnormal product may have to be flushed
#pragma unroll
        for (int k = 0; k < VEC / 2; ++k) {
          stored[k].x = flush_rounded_up(stored[k].x, scaled[k].x);
          stored[k].y = flush_rounded_up(stored[k].y, scaled[k].y);
        }
      }
#pragma unroll
      for (int k = 0; k < VEC / 2; ++k) f[k] = add2(f[k], stored[k]);
    }
#pragma unroll
  for (int k = 0; k < VEC / 2; ++k) {
    gr[2 * k] += f[k].x;
    gr[2 * k + 1] += f[k].y;
  }
}
template <bool ADAM, bool MASTER, int CORR, int NG, int VEC>
__device__ __forceinline__ void load_vec(const OpkDpStepArgs& a, const PeerTable& pt, const StepGroup& grp, long long i0, long long e0,
                                         VecIn<NG, CORR, VEC>& q) {
  // reduce-scatter: sum the owned elements over every rank's buffer (peer reads travel over NVLink)
  if (NG == 0 || !grp.skip_sum || e0 >= grp.len) {
    ld_stream<VEC>(pt.grad[0] + e0, q.g);
  } else {
#pragma unroll
    for (int j = 0; j < VEC; ++j) q.g[j] = 0.f;
  }
  for (int r = 1; r < a.n_src; ++r) {
    float t[VEC];
    ld_stream<VEC>(pt.grad[r] + e0, t);
#pragma unroll
    for (int j = 0; j < VEC; ++j) q.g[j] += t[j];
  }
  if (NG > 0 && e0 < grp.len) {
#pragma unroll
    for (int j = 0; j < NG; ++j)
      if (j < grp.n) ld_stream<VEC>(grp.g[j] + e0, q.gr[j]);
  }
  if (MASTER) ld_stream<VEC>(a.master + i0, q.mw);
  else ld_stream<VEC>(reinterpret_cast<const __nv_bfloat16*>(a.param_src) + e0, q.pw);
  if (ADAM) {
    ld_stream<VEC>(a.m + i0, q.m);
    ld_stream<VEC>(a.v + i0, q.v);
  } else {
#pragma unroll
    for (int j = 0; j < VEC; ++j) q.m[j] = q.v[j] = 0.f;
  }
  load_corr(a, i0, 0, q.corr);
}
template <bool ADAM, bool MASTER, int CORR, int NG, int VEC>
__device__ __forceinline__ void finish_vec(const OpkDpStepArgs& a, const opk::PhiloxKeys& key, const PeerTable& pt, const StepGroup& grp,
                                           const float (&gs)[NG > 0 ? NG : 1], float inv_bc1, float inv_bc2, long long i0, long long e0,
                                           VecIn<NG, CORR, VEC>& q) {
  float z[VEC];
#pragma unroll
  for (int h = 0; h < VEC; h += 4) {
    float n[4] = {0.f, 0.f, 0.f, 0.f};
    if (a.sigma != 0.f) normal4((uint64_t)(e0 + h) >> 2, key, a.stream_id, a.step, n);
#pragma unroll
    for (int j = 0; j < 4; ++j) z[h + j] = n[j];
  }
  correlate(a, i0, q.corr, z);
  if (NG > 0 && e0 < grp.len) add_group<NG, CORR, VEC>(grp, gs, q, q.g);
  float pn[VEC];
#pragma unroll
  for (int j = 0; j < VEC; j += 2) {
    const float2 po = MASTER ? make_float2(q.mw[j], q.mw[j + 1]) : unpack2(q.pw[j / 2]);
    const float2 grad = fma2(make_float2(q.g[j], q.g[j + 1]), pair(a.inv_batch), mul2(pair(a.sigma), make_float2(z[j], z[j + 1])));
    float2 m = make_float2(q.m[j], q.m[j + 1]), v = make_float2(q.v[j], q.v[j + 1]);
    const float2 p = dp_update<ADAM>(a, inv_bc1, inv_bc2, grad, po, m, v);
    q.m[j] = m.x; q.m[j + 1] = m.y;
    q.v[j] = v.x; q.v[j + 1] = v.y;
    pn[j] = p.x; pn[j + 1] = p.y;
  }
  if (ADAM) {
    st_stream<VEC>(a.m + i0, q.m);
    st_stream<VEC>(a.v + i0, q.v);
  }
  if (MASTER) st_stream<VEC>(a.master + i0, pn);
  // all-gather: write the updated bf16 values into every destination parameter buffer
  uint32_t o[VEC / 2];
#pragma unroll
  for (int j = 0; j < VEC / 2; ++j) {
    const __nv_bfloat162 both = __floats2bfloat162_rn(pn[2 * j], pn[2 * j + 1]);
    o[j] = *reinterpret_cast<const uint32_t*>(&both);
  }
  for (int r = 0; r < a.n_dst; ++r) {
    if constexpr (VEC == 8) *reinterpret_cast<uint4*>(pt.param[r] + e0) = make_uint4(o[0], o[1], o[2], o[3]);
    else *reinterpret_cast<uint2*>(pt.param[r] + e0) = make_uint2(o[0], o[1]);
  }
  if (a.zero_grad) {
    float none[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) none[j] = 0.f;
    st_stream<VEC>(const_cast<float*>(pt.grad[0]) + e0, none);
  }
}

// Whether a thread holds two vectors of four at a time. With a group to add and much state next to it there are no registers for two,
// and four rows of BLT state take those of the second; the loads of more CTAs are in flight instead. (us at 2^26 elements off a 32-byte
// boundary: quads of the kernel before -> two vectors -> one: SGD with five buffers 290 -> 320 -> 260; AdamW with master weights and two
// 364 -> 382 -> 352; four BLT rows, AdamW with five 809 -> 979 -> 732, SGD with eight 713 -> 853 -> 628, AdamW alone 692 -> 668 -> 644.
// Two is the better one for SGD alone, 146 -> 121 -> 130 to 194, and for AdamW with eight and Toeplitz rows, 891 -> 613 -> 624 to 673.)
__host__ __device__ constexpr bool step_two(bool adam, bool master, int corr, int ng) {
  return corr == CORR_TOEPLITZ || (corr == CORR_NONE && ng <= 2 && !(adam && master && ng > 0));
}
// CTAs per SM that the registers must allow: what the variant fits with a few bytes of spills at most.
constexpr int step_min_ctas(bool adam, bool master, int corr, int ng, int vec) {
  if (vec == 8 || corr == CORR_TOEPLITZ) return 2;
  if (corr == CORR_BLT) return 3;
  return adam && (step_two(adam, master, corr, ng) || (master && ng > 2)) ? 3 : 4;
}
template <bool ADAM, bool MASTER, int CORR, int NG, int VEC>
__global__ void __launch_bounds__(256, step_min_ctas(ADAM, MASTER, CORR, NG, VEC))
dp_step_kernel(const OpkDpStepArgs a, const opk::PhiloxKeys key, const PeerTable pt, const StepGroup grp) {
  // Each thread owns aligned vectors of the shard: eight elements an iteration, or four, or two times four (step_two); a ragged end
  // takes the scalar path.
  //
  // What bounds it: memory, 28 bytes per parameter with two gradient buffers, and next to it the issue slots: 118 instructions per
  // parameter kept 72 % of them busy at full clock, and a step under the power cap runs at two thirds of that. Eight elements per
  // thread halve the accesses and their addresses, the round keys come from the constant bank, fp32 arithmetic goes two lanes an
  // instruction and only subnormal products are looked at for the flush. AdamW with two buffers, 1.49e9 parameters, right after
  // large products: 8.56 -> 7.41 ms (5.6 TB/s); without buffers 6.77 -> 5.88. Correlation state is read with everything else, not
  // row by row behind the noise: 2^28 elements, three Toeplitz rows 2.61 -> 1.83 ms (6.4 TB/s), four BLT buffers 3.00 -> 2.75.
  // Loading the next vector before this one is finished changed nothing without state (7.2 ms) and spills with it.
  const long long nfull = a.shard_len / VEC;
  const float inv_bc1 = 1.f / a.bc1, inv_bc2 = 1.f / a.bc2;
  float gs[NG > 0 ? NG : 1];
#pragma unroll
  for (int j = 0; j < NG; ++j) gs[j] = j < grp.n ? *grp.scale[j] : 0.f;
  const long long stride = (long long)gridDim.x * 256;
  long long q = blockIdx.x * 256ll + threadIdx.x;
  if constexpr (VEC == 4 && step_two(ADAM, MASTER, CORR, NG)) {
#pragma unroll 1
    for (; q + stride < nfull; q += 2 * stride) {
      const long long q2 = q + stride;
      VecIn<NG, CORR, VEC> in, in2;
      load_vec<ADAM, MASTER, CORR, NG, VEC>(a, pt, grp, q * VEC, a.shard_begin + q * VEC, in);
      load_vec<ADAM, MASTER, CORR, NG, VEC>(a, pt, grp, q2 * VEC, a.shard_begin + q2 * VEC, in2);
      finish_vec<ADAM, MASTER, CORR, NG, VEC>(a, key, pt, grp, gs, inv_bc1, inv_bc2, q * VEC, a.shard_begin + q * VEC, in);
      finish_vec<ADAM, MASTER, CORR, NG, VEC>(a, key, pt, grp, gs, inv_bc1, inv_bc2, q2 * VEC, a.shard_begin + q2 * VEC, in2);
    }
  }
#pragma unroll 1
  for (; q < nfull; q += stride) {
    VecIn<NG, CORR, VEC> in;
    load_vec<ADAM, MASTER, CORR, NG, VEC>(a, pt, grp, q * VEC, a.shard_begin + q * VEC, in);
    finish_vec<ADAM, MASTER, CORR, NG, VEC>(a, key, pt, grp, gs, inv_bc1, inv_bc2, q * VEC, a.shard_begin + q * VEC, in);
  }
  // ragged end: one thread per element
  const long long i = nfull * VEC + threadIdx.x;
  if (blockIdx.x == 0 && i < a.shard_len) {
    const long long e = a.shard_begin + i;
    float z4[4] = {0.f, 0.f, 0.f, 0.f};
    if (a.sigma != 0.f) normal4((uint64_t)e >> 2, key, a.stream_id, a.step, z4);
    const int lane = (int)(e & 3);
    const float z = lane == 0 ? z4[0] : lane == 1 ? z4[1] : lane == 2 ? z4[2] : z4[3];
    float g = 0.f;
    const bool in_group = NG > 0 && e < grp.len;
    for (int r = 0; r < a.n_src; ++r)
      if (!(in_group && grp.skip_sum)) g += pt.grad[r][e];
    if (in_group) {
      float f = 0.f;
      for (int k = 0; k < grp.n; ++k) f += clip_store(__bfloat162float(grp.g[k][e]), *grp.scale[k]);
      g += f;
    }
    const float noise = correlate_one<CORR>(a, i, z);
    const float p_old = MASTER ? a.master[i] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.param_src)[e]);
    float2 m = pair(ADAM ? a.m[i] : 0.f), v = pair(ADAM ? a.v[i] : 0.f);
    const float grad = fmaf(g, a.inv_batch, a.sigma * noise);
    const float p_new = dp_update<ADAM>(a, inv_bc1, inv_bc2, pair(grad), pair(p_old), m, v).x;
    if (ADAM) { a.m[i] = m.x; a.v[i] = v.x; }
    if (MASTER) a.master[i] = p_new;
    for (int r = 0; r < a.n_dst; ++r) pt.param[r][e] = __float2bfloat16(p_new);
    if (a.zero_grad) const_cast<float*>(pt.grad[0])[e] = 0.f;
  }
}

// ------------------------------------------------------------------------------------------- sharded sums (push)
// The fp32 sums are sharded: rank o owns elements [begin[o], begin[o+1]) of the flat parameter vector and keeps them in
// a peer-addressable buffer. A group of clipped per-example gradients is added with reductions sent to the owner
// (red.add over NVLink for remote owners), so no rank ever holds a full-size fp32 sum. Peers add into the same shard
// concurrently, hence reductions for the local part as well.
struct ShardTable {
  float* acc[MAX_PEERS];
  long long begin[MAX_PEERS + 1];
  int n;
};
__device__ __forceinline__ void red_add_f32x4(float* dst, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
template <int N>
__global__ void __launch_bounds__(256) clip_accumulate_group_push_kernel(const AccGroup grp, const ShardTable sh, long long nvec,
                                                                         long long rot) {
  float s[N];
#pragma unroll
  for (int j = 0; j < N; ++j) s[j] = *grp.scale[j];
  for (long long t = blockIdx.x * 256ll + threadIdx.x; t < nvec; t += (long long)gridDim.x * 256) {
    // every rank starts at its own shard and walks the owners in rank order: at any moment the ranks push to
    // different owners
    long long i = t + rot;
    if (i >= nvec) i -= nvec;
    uint4 r[N];
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] = __ldcs(reinterpret_cast<const uint4*>(grp.g[j]) + i);
    float f[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) f[q] = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const bf16x8 v = *reinterpret_cast<const bf16x8*>(&r[j]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 u = __bfloat1622float2(v.h[q]);
        f[2 * q] += clip_store(u.x, s[j]);
        f[2 * q + 1] += clip_store(u.y, s[j]);
      }
    }
    const long long e = i << 3;
    int o = 0;
    while (o + 1 < sh.n && e >= sh.begin[o + 1]) ++o;
    float* dst = sh.acc[o] + (e - sh.begin[o]);
    red_add_f32x4(dst, f[0], f[1], f[2], f[3]);
    red_add_f32x4(dst + 4, f[4], f[5], f[6], f[7]);
  }
}
template <int N>
void launch_acc_group_push(const AccGroup& grp, const ShardTable& sh, long long nvec, long long rot, cudaStream_t st) {
  long long g = (nvec + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  clip_accumulate_group_push_kernel<N><<<(int)g, 256, 0, st>>>(grp, sh, nvec, rot);
}

// Plain copy between two device buffers that may live on different GPUs (peer-mapped memory): 16-byte vectors, eight
// loads in flight per thread. Used to refresh the parts of a parameter replica that no GEMM stages for itself.
__global__ void __launch_bounds__(256) copy_vec_kernel(uint4* __restrict__ dst, const uint4* __restrict__ src, long long nvec) {
  constexpr int U = 8;
  const long long stride = (long long)gridDim.x * 256;
  for (long long i0 = blockIdx.x * 256ll + threadIdx.x; i0 < nvec; i0 += U * stride) {
    uint4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + u * stride;
      if (i < nvec) v[u] = __ldcg(src + i);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + u * stride;
      if (i < nvec) dst[i] = v[u];
    }
  }
}

inline int grid_for(long long n, int block, int cap_blocks) {
  long long g = (n + block - 1) / block;
  if (g > cap_blocks) g = cap_blocks;
  if (g < 1) g = 1;
  return (int)g;
}

// ragged tail (fewer than 8 elements) of the group pass, same association as the vector body
__global__ void clip_accumulate_group_tail_kernel(const AccGroup grp, int n_group, float* __restrict__ acc, long long begin,
                                                  long long n, int overwrite) {
  const long long i = begin + threadIdx.x;
  if (i >= n) return;
  float f = 0.f;
  for (int j = 0; j < n_group; ++j)
    f += clip_store(__bfloat162float(reinterpret_cast<const __nv_bfloat16*>(grp.g[j])[i]), *grp.scale[j]);
  acc[i] = (overwrite ? 0.f : acc[i]) + f;
}
template <int N>
void launch_acc_group(const AccGroup& grp, float* acc, long long nvec, int overwrite, cudaStream_t st) {
  clip_accumulate_group_kernel<N><<<grid_for(nvec, 256, 148 * 16), 256, 0, st>>>(grp, reinterpret_cast<float4*>(acc), nvec, overwrite);
}

}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)

extern "C" int opk_philox_normal(float* out, int64_t n, uint64_t seed, uint32_t stream_id, uint32_t step,
                                 uint64_t offset, float sigma, int accumulate, void* stream) {
  if (n <= 0) return 0;
  philox_normal_kernel<<<grid_for((n + 3) / 4 + 1, 256, 148 * 8), 256, 0, ST(stream)>>>(out, n, seed, stream_id, step,
                                                                                      offset, sigma, accumulate);
  OPK_LAUNCH_CHECK();
  return 0;
}

extern "C" int opk_clip_scale(double* sumsq, float clip, int mode_auto, float gamma, int n_leaves, int64_t widest_leaf,
                              float* scale_out, float* norm_out, int32_t* counters, int reset, int batch, const float* loss,
                              float* loss_sum, void* stream) {
  if (batch < 1 || batch > 32 || (loss_sum && !loss)) return -1;
  clip_scale_kernel<<<1, batch, 0, ST(stream)>>>(sumsq, clip, mode_auto, gamma, n_leaves, widest_leaf, scale_out, norm_out,
                                            counters, reset, loss, loss_sum);
  OPK_LAUNCH_CHECK();
  return 0;
}

extern "C" int opk_clip_accumulate(const void* g, const float* scale, float* acc, int64_t n, void* stream);
extern "C" int opk_clip_accumulate2(const void* g, const float* scale, float* acc, int64_t n, int overwrite,
                                    void* stream) {
  if (n <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(g) & 15) || (reinterpret_cast<uintptr_t>(acc) & 15)) return -1;
  const long long nvec = n >> 3;
  static int cap_ctas = -1;
  if (cap_ctas < 0) {
    // Same shared-memory carve-out as the GEMM kernels, so that CTAs of this kernel can be co-resident with them
    // on an SM (an SM does not mix carve-out configurations).
    cudaFuncSetAttribute(clip_accumulate_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cap_ctas = 148 * 16;
  }
  if (nvec > 0)
    clip_accumulate_kernel<<<grid_for(nvec, 256, cap_ctas), 256, 0, ST(stream)>>>(
        reinterpret_cast<const bf16x8*>(g), scale, reinterpret_cast<float4*>(acc), nvec, overwrite);
  const long long tail = n - (nvec << 3);
  if (tail > 0)
    clip_accumulate_tail_kernel<<<1, 32, 0, ST(stream)>>>(reinterpret_cast<const __nv_bfloat16*>(g), scale, acc,
                                                         nvec << 3, n, overwrite);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_clip_accumulate_group(const void* const* g, const float* const* scale, int n_group, float* acc, int64_t n,
                                         int overwrite, void* stream) {
  if (n <= 0 || n_group <= 0) return 0;
  if (n_group > OPK_ACC_GROUP_MAX || (reinterpret_cast<uintptr_t>(acc) & 15)) return -1;
  AccGroup grp;
  for (int j = 0; j < OPK_ACC_GROUP_MAX; ++j) {
    grp.g[j] = j < n_group ? reinterpret_cast<const bf16x8*>(g[j]) : nullptr;
    grp.scale[j] = j < n_group ? scale[j] : nullptr;
    if (j < n_group && (reinterpret_cast<uintptr_t>(g[j]) & 15)) return -1;
  }
  const long long nvec = n >> 3;
  cudaStream_t st = ST(stream);
  if (nvec > 0) {
    switch (n_group) {
      case 1: launch_acc_group<1>(grp, acc, nvec, overwrite, st); break;
      case 2: launch_acc_group<2>(grp, acc, nvec, overwrite, st); break;
      case 3: launch_acc_group<3>(grp, acc, nvec, overwrite, st); break;
      case 4: launch_acc_group<4>(grp, acc, nvec, overwrite, st); break;
      case 5: launch_acc_group<5>(grp, acc, nvec, overwrite, st); break;
      case 6: launch_acc_group<6>(grp, acc, nvec, overwrite, st); break;
      case 7: launch_acc_group<7>(grp, acc, nvec, overwrite, st); break;
      default: launch_acc_group<8>(grp, acc, nvec, overwrite, st); break;
    }
  }
  const long long tail = n - (nvec << 3);
  if (tail > 0) clip_accumulate_group_tail_kernel<<<1, 32, 0, st>>>(grp, n_group, acc, nvec << 3, n, overwrite);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_clip_accumulate(const void* g, const float* scale, float* acc, int64_t n, void* stream) {
  return opk_clip_accumulate2(g, scale, acc, n, 0, stream);
}

// Up to 2^23 elements one round of resident CTAs walks the shard, so that every CTA gets the same share (2^20 elements, one round ->
// eight CTAs per SM: SGD 3.3 -> 3.6 us, AdamW 4.8 -> 5.1, with two buffers 6.1 -> 6.6). On larger shards eight per SM, which start
// and end at different times, except for AdamW that adds a group without correlated noise (2^26 elements: AdamW 275 -> 249 us, with
// master weights 336 -> 312, four BLT rows 608 -> 584, three Toeplitz rows 437 -> 412, SGD 106 -> 102; with two buffers 286 -> 289).
template <bool ADAM, bool MASTER, int CORR, int NG, int VEC>
void launch_dp_step(cudaStream_t st, const OpkDpStepArgs& args, const PeerTable& pt, const StepGroup& grp) {
  auto kernel = dp_step_kernel<ADAM, MASTER, CORR, NG, VEC>;
  int per_sm = 8, dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const bool eight = args.shard_len > (1ll << 23) && (!ADAM || NG == 0 || CORR != CORR_NONE);
  if (!eight && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0) != cudaSuccess || per_sm < 1)) per_sm = 2;
  kernel<<<grid_for((args.shard_len + VEC - 1) / VEC, 256, sms * per_sm), 256, 0, st>>>(args, opk::philox_keys(args.seed), pt, grp);
}
// Whether every array of the step can be read eight elements at a time: 32-byte fp32 and 16-byte bf16 vectors that start with the
// shard, whole vectors in the group's buffers and in every row of correlation state.
bool eight_at_a_time(const OpkDpStepArgs& a, const PeerTable& pt, const StepGroup& grp) {
  auto off = [](const void* p) { return reinterpret_cast<uintptr_t>(p) & 31; };
  if ((a.shard_begin & 7) || (grp.len & 7)) return false;
  for (int r = 0; r < a.n_src; ++r)
    if (off(pt.grad[r])) return false;
  for (int r = 0; r < a.n_dst; ++r)
    if (off(pt.param[r]) & 15) return false;
  for (int j = 0; j < grp.n; ++j)
    if (off(grp.g[j]) & 15) return false;
  if ((off(a.param_src) & 15) || off(a.m) || off(a.v) || off(a.master)) return false;
  if (a.blt_nbuf > 0 && (off(a.blt_state) || (a.blt_nbuf > 1 && (a.shard_len & 7)))) return false;
  if (a.toep_nlag > 0 && (off(a.toep_state) || (a.toep_nlag > 1 && (a.shard_len & 7)))) return false;
  return true;
}

// grad_src / param_dst are HOST arrays of device pointers here (copied into the kernel's parameter space).
extern "C" int opk_dp_step(const OpkDpStepArgs* args, void* stream) {
  if (!args || args->shard_len <= 0) return 0;
  if (args->n_src < 1 || args->n_src > MAX_PEERS || args->n_dst < 0 || args->n_dst > MAX_PEERS) return -1;
  if (args->shard_begin & 3) return -2;
  PeerTable pt;
  for (int r = 0; r < MAX_PEERS; ++r) {
    pt.grad[r] = r < args->n_src ? args->grad_src[r] : nullptr;
    pt.param[r] = r < args->n_dst ? reinterpret_cast<__nv_bfloat16*>(args->param_dst[r]) : nullptr;
  }
  if (args->blt_nbuf > 0 && args->toep_nlag > 0) return -3;       // one correlation transform per step
  // rows of the [buffers][shard_len] state are read as 16-byte vectors: every row must start on a 16-byte boundary
  if ((args->blt_nbuf > 1 || args->toep_nlag > 1) && (args->shard_len & 3)) return -2;
  if ((args->blt_nbuf > 0 && (reinterpret_cast<uintptr_t>(args->blt_state) & 15)) ||
      (args->toep_nlag > 0 && (reinterpret_cast<uintptr_t>(args->toep_state) & 15)) ||
      (reinterpret_cast<uintptr_t>(args->m) & 15) || (reinterpret_cast<uintptr_t>(args->v) & 15) ||
      (reinterpret_cast<uintptr_t>(args->master) & 15))
    return -2;
  if (args->toep_nlag > 0 && (!args->toep_state || !args->toep_coef || args->toep_pos < 0 || args->toep_pos >= args->toep_nlag)) return -3;
  cudaStream_t st = ST(stream);
  const int corr = args->blt_nbuf > 0 ? CORR_BLT : (args->toep_coef ? CORR_TOEPLITZ : CORR_NONE);
  const bool adam = !args->sgd_mode, master = args->master != nullptr;
  StepGroup grp = {};
  const bool group = args->n_group > 0 || args->skip_sum != 0;
  if (group) {
    // quads must not straddle the end of the group's buffers, which are read 8 bytes at a time
    if (args->n_group < 0 || args->n_group > OPK_ACC_GROUP_MAX || args->group_len < 0 || (args->group_len & 3)) return -4;
    if (args->skip_sum && args->n_src != 1) return -4;
    if (args->n_group > 0 && (!args->group_g || !args->group_scale)) return -4;
    for (int j = 0; j < args->n_group; ++j) {
      grp.g[j] = reinterpret_cast<const __nv_bfloat16*>(args->group_g[j]);
      grp.scale[j] = args->group_scale[j];
      if (!grp.g[j] || !grp.scale[j] || (reinterpret_cast<uintptr_t>(grp.g[j]) & 7)) return -4;
    }
    grp.n = args->n_group;
    grp.skip_sum = args->skip_sum;
    grp.len = args->group_len;
  }
  // One variant for groups of at most two and one for all others, because registers set how many CTAs an SM holds: with two
  // buffers 287 us against 300 on the variant for eight (2^26 elements, AdamW), with one 270 against 284. From three buffers on
  // only the wide one fits: 316 us for three, 404 for eight (6.6 TB/s).
  const bool wide = eight_at_a_time(*args, pt, grp);
#define OPK_DP_STEP_VEC(A, M, C, N)                                                  \
  do {                                                                               \
    if (wide) launch_dp_step<A, M, C, N, 8>(st, *args, pt, grp);                     \
    else launch_dp_step<A, M, C, N, 4>(st, *args, pt, grp);                          \
  } while (0)
#define OPK_DP_STEP_LAUNCH(A, M, C)                                                  \
  do {                                                                               \
    if (!group) OPK_DP_STEP_VEC(A, M, C, 0);                                         \
    else if (grp.n <= 2) OPK_DP_STEP_VEC(A, M, C, 2);                                \
    else OPK_DP_STEP_VEC(A, M, C, OPK_ACC_GROUP_MAX);                                \
  } while (0)
#define OPK_DP_STEP_CORR(A, M)                                      \
  do {                                                              \
    if (corr == CORR_BLT) OPK_DP_STEP_LAUNCH(A, M, CORR_BLT);       \
    else if (corr == CORR_TOEPLITZ) OPK_DP_STEP_LAUNCH(A, M, CORR_TOEPLITZ); \
    else OPK_DP_STEP_LAUNCH(A, M, CORR_NONE);                       \
  } while (0)
  if (adam && master) OPK_DP_STEP_CORR(true, true);
  else if (adam) OPK_DP_STEP_CORR(true, false);
  else if (master) OPK_DP_STEP_CORR(false, true);
  else OPK_DP_STEP_CORR(false, false);
#undef OPK_DP_STEP_CORR
#undef OPK_DP_STEP_LAUNCH
#undef OPK_DP_STEP_VEC
  OPK_LAUNCH_CHECK();
  return 0;
}

// Sharded fp32 sums: acc_shards[o] is the base of owner o's shard (a peer-mapped address for o != this rank), which
// holds the elements [bounds[o], bounds[o+1]) of the flat vector; bounds are multiples of 8. rank selects where this
// rank starts walking (its own shard first).
extern "C" int opk_clip_accumulate_group_push(const void* const* g, const float* const* scale, int n_group,
                                              float* const* acc_shards, const int64_t* bounds, int n_shards, int rank,
                                              int64_t n, void* stream) {
  if (n <= 0 || n_group <= 0) return 0;
  if (n_group > OPK_ACC_GROUP_MAX || n_shards < 1 || n_shards > MAX_PEERS || rank < 0 || rank >= n_shards || (n & 7)) return -1;
  AccGroup grp;
  for (int j = 0; j < OPK_ACC_GROUP_MAX; ++j) {
    grp.g[j] = j < n_group ? reinterpret_cast<const bf16x8*>(g[j]) : nullptr;
    grp.scale[j] = j < n_group ? scale[j] : nullptr;
    if (j < n_group && (reinterpret_cast<uintptr_t>(g[j]) & 15)) return -1;
  }
  ShardTable sh;
  sh.n = n_shards;
  for (int o = 0; o < MAX_PEERS; ++o) sh.acc[o] = o < n_shards ? acc_shards[o] : nullptr;
  for (int o = 0; o <= MAX_PEERS; ++o) sh.begin[o] = o <= n_shards ? bounds[o] : bounds[n_shards];
  for (int o = 0; o < n_shards; ++o) {
    if ((bounds[o] & 7) || bounds[o + 1] < bounds[o] || (reinterpret_cast<uintptr_t>(acc_shards[o]) & 15)) return -1;
  }
  if (bounds[0] != 0 || bounds[n_shards] < n) return -1;
  const long long nvec = n >> 3;
  long long rot = bounds[rank] >> 3;
  if (rot >= nvec) rot = 0;
  cudaStream_t st = ST(stream);
  switch (n_group) {
    case 1: launch_acc_group_push<1>(grp, sh, nvec, rot, st); break;
    case 2: launch_acc_group_push<2>(grp, sh, nvec, rot, st); break;
    case 3: launch_acc_group_push<3>(grp, sh, nvec, rot, st); break;
    case 4: launch_acc_group_push<4>(grp, sh, nvec, rot, st); break;
    case 5: launch_acc_group_push<5>(grp, sh, nvec, rot, st); break;
    case 6: launch_acc_group_push<6>(grp, sh, nvec, rot, st); break;
    case 7: launch_acc_group_push<7>(grp, sh, nvec, rot, st); break;
    default: launch_acc_group_push<8>(grp, sh, nvec, rot, st); break;
  }
  OPK_LAUNCH_CHECK();
  return 0;
}

extern "C" int opk_copy_bytes(void* dst, const void* src, int64_t nbytes, void* stream) {
  if (nbytes <= 0) return 0;
  if ((nbytes & 15) || (reinterpret_cast<uintptr_t>(dst) & 15) || (reinterpret_cast<uintptr_t>(src) & 15)) return -1;
  const long long nvec = nbytes >> 4;
  copy_vec_kernel<<<grid_for((nvec + 7) / 8, 256, 148 * 8), 256, 0, ST(stream)>>>(reinterpret_cast<uint4*>(dst),
                                                                                  reinterpret_cast<const uint4*>(src), nvec);
  OPK_LAUNCH_CHECK();
  return 0;
}
