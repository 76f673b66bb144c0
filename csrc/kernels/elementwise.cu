// Bandwidth-bound model kernels for sm_100a: RMSNorm / LayerNorm, rotary embedding, SwiGLU / GEGLU / GELU,
// embedding gather and per-example compact embedding gradient, cross-entropy helpers.
// All activations are bf16 in memory with fp32 arithmetic; rows are processed with 16-byte vector accesses.
#include "opk_api.h"
#include "pdl.cuh"
#include "debug_bounds.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>
#include <stdio.h>

namespace {

#define OPK_LAUNCH_CHECK()                                   \
  do {                                                       \
    cudaError_t e__ = cudaGetLastError();                    \
    if (e__ != cudaSuccess) return (int)e__;                 \
  } while (0)

struct alignas(16) bf16x8 {
  __nv_bfloat162 h[4];
};

__device__ __forceinline__ void unpack8(const bf16x8& v, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(v.h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ bf16x8 pack8(const float (&f)[8]) {
  bf16x8 v;
#pragma unroll
  for (int i = 0; i < 4; ++i) v.h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return v;
}

template <int NT>
__device__ __forceinline__ float block_sum(float v, float* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float r = (threadIdx.x < NT / 32) ? sh[threadIdx.x] : 0.f;
  if (w == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if (l == 0) sh[0] = r;
  }
  __syncthreads();
  return sh[0];
}

constexpr int NT = 256;

// ------------------------------------------------------------------------------------------- RMSNorm
// COPY: sum_out receives x.
template <bool ADD, bool COPY>
__global__ void __launch_bounds__(NT) rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                         const __nv_bfloat16* __restrict__ r,
                                                         const __nv_bfloat16* __restrict__ w,
                                                         __nv_bfloat16* __restrict__ sum_out,
                                                         __nv_bfloat16* __restrict__ y, float* __restrict__ rstd,
                                                         int D, float eps, float w_off, long long ldx, long long ldy,
                                                         long long ld_sum) {
  opk::pdl_trigger();
  __shared__ float sh[32];
  const long long row = blockIdx.x;
  const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * ldx);
  const bf16x8* rr = ADD ? reinterpret_cast<const bf16x8*>(r + row * D) : nullptr;
  bf16x8* sr = ADD || COPY ? reinterpret_cast<bf16x8*>(sum_out + row * (COPY ? ld_sum : D)) : nullptr;
  const int nv = D >> 3;
  float ss = 0.f;
  for (int i = threadIdx.x; i < nv; i += NT) {
    float f[8];
    const bf16x8 in = xr[i];
    unpack8(in, f);
    if (COPY) sr[i] = in;
    if (ADD) {
      float g[8];
      unpack8(rr[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += g[j];
      bf16x8 s = pack8(f);
      sr[i] = s;
      unpack8(s, f);  // normalise the stored (rounded) residual stream
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  const float tot = block_sum<NT>(ss, sh);
  const float rs = rsqrtf(tot / (float)D + eps);
  if (threadIdx.x == 0 && rstd) rstd[row] = rs;
  const bf16x8* src = ADD ? reinterpret_cast<const bf16x8*>(sum_out + row * D) : xr;
  const bf16x8* wr = reinterpret_cast<const bf16x8*>(w);
  bf16x8* yr = reinterpret_cast<bf16x8*>(y + row * ldy);
  for (int i = threadIdx.x; i < nv; i += NT) {
    float f[8], g[8];
    unpack8(src[i], f);
    unpack8(wr[i], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * rs * (g[j] + w_off);
    yr[i] = pack8(f);
  }
}

// One warp per row, the row held in registers (VPL vectors of 8 per lane): one pass over memory, no block barrier.
// (Without the opaque barrier below the compiler keeps the row UNPACKED across the reduction, 255 registers per thread at
// 16 vectors per lane: one CTA per SM and 12 % of the warp slots in use. Packed, the row is 64 registers.)
//
// `copy` (optional) receives the row as it was read, for a norm in place whose input the backward pass needs (query and key columns
// of a fused projection: 4096 x 4096 values took 107 us in a strided copy of their own, 428 us of a 22.6 ms OLMoE step).
template <int VPL, bool COPY>
__global__ void __launch_bounds__(256, VPL >= 16 ? 2 : 4) rmsnorm_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x,
                                                               const __nv_bfloat16* __restrict__ w,
                                                               __nv_bfloat16* __restrict__ y, float* __restrict__ rstd, int T,
                                                               float eps, float w_off, long long ldx, long long ldy,
                                                               __nv_bfloat16* __restrict__ copy, long long ld_copy) {
  opk::pdl_trigger();
  constexpr int D = VPL * 32 * 8;
  const int lane = threadIdx.x & 31;
  const long long row = blockIdx.x * 8ll + (threadIdx.x >> 5);
  if (row >= T) return;
  const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * ldx);
  bf16x8 v[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) v[i] = xr[lane + 32 * i];
  if constexpr (COPY) {
    bf16x8* cr = reinterpret_cast<bf16x8*>(copy + row * ld_copy);
#pragma unroll
    for (int i = 0; i < VPL; ++i) cr[lane + 32 * i] = v[i];
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    float f[8];
    unpack8(v[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float rs = rsqrtf(ss / (float)D + eps);
  if (lane == 0 && rstd) rstd[row] = rs;
  const bf16x8* wr = reinterpret_cast<const bf16x8*>(w);
  bf16x8* yr = reinterpret_cast<bf16x8*>(y + row * ldy);
  // the packed words pass through an empty asm: the floats computed for the reduction cannot be reused below
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
#pragma unroll
    for (int q = 0; q < 4; ++q) asm volatile("" : "+r"(*reinterpret_cast<uint32_t*>(&v[i].h[q])));
  }
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    float f[8], g[8];
    unpack8(v[i], f);
    unpack8(wr[lane + 32 * i], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * rs * (g[j] + w_off);
    yr[lane + 32 * i] = pack8(f);
  }
}

// Residual add + RMSNorm, one CTA per row with the row held packed in registers: one pass over memory (the general kernel
// writes the sum, then reads it back). ITERS vectors of 8 per thread, D <= ITERS * 2048.
template <int ITERS>
__global__ void __launch_bounds__(NT) add_rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ r,
                                                             const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ sum_out,
                                                             __nv_bfloat16* __restrict__ y, float* __restrict__ rstd, int D, float eps,
                                                             float w_off) {
  opk::pdl_trigger();
  __shared__ float sh[32];
  const long long row = blockIdx.x;
  const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * D);
  const bf16x8* rr = reinterpret_cast<const bf16x8*>(r + row * D);
  bf16x8* sr = reinterpret_cast<bf16x8*>(sum_out + row * D);
  const int nv = D >> 3;
  bf16x8 v[ITERS], q[ITERS];
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int i = threadIdx.x + it * NT;
    if (i < nv) { v[it] = xr[i]; q[it] = rr[i]; }
  }
  float ss = 0.f;
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int i = threadIdx.x + it * NT;
    if (i < nv) {
      float f[8], g[8];
      unpack8(v[it], f);
      unpack8(q[it], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += g[j];
      v[it] = pack8(f);
      sr[i] = v[it];
      unpack8(v[it], f);  // normalise the stored (rounded) residual stream
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    }
  }
  const float rs = rsqrtf(block_sum<NT>(ss, sh) / (float)D + eps);
  if (threadIdx.x == 0 && rstd) rstd[row] = rs;
  const bf16x8* wr = reinterpret_cast<const bf16x8*>(w);
  bf16x8* yr = reinterpret_cast<bf16x8*>(y + row * D);
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int i = threadIdx.x + it * NT;
    if (i < nv) {
      float f[8], g[8];
      unpack8(v[it], f);
      unpack8(wr[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = f[j] * rs * (g[j] + w_off);
      yr[i] = pack8(f);
    }
  }
}

// RMSNorm backward. A CTA of 512 threads walks rows with a grid stride; every thread owns the same columns for
// all rows (ITERS vectors of 8), so the weight gradient accumulates in registers without atomics and is written once
// per CTA to partial[CTA][D]. A second kernel adds the column sums of `partial` into dw. gridDim.y examples of T rows each:
// an example's rows meet the same CTAs in the same order as in a launch of its own, so its weight gradient has the same bits.
constexpr int MAX_COL_ITERS = 8;  // layernorm backward: D <= 8 * 2048
constexpr int RMS_BWD_NT = 512;
// (MANY: more than one; a single example keeps the shorter addresses.)
template <int ITERS, bool MANY>
__global__ void __launch_bounds__(RMS_BWD_NT) rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy,
                                                                 const __nv_bfloat16* __restrict__ x,
                                                                 const __nv_bfloat16* __restrict__ w,
                                                                 const float* __restrict__ rstd,
                                                                 const __nv_bfloat16* __restrict__ dres,
                                                                 __nv_bfloat16* __restrict__ dx,
                                                                 float* __restrict__ partial, int T, int D,
                                                                 float w_off, long long ld_dy, long long ldx,
                                                                 long long ld_dx) {
  __shared__ float sh[32];
  const int nv = D >> 3;
  const long long first = MANY ? (long long)blockIdx.y * T : 0;
  float wv[ITERS][8], acc[ITERS][8];
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int v = threadIdx.x + it * RMS_BWD_NT;
#pragma unroll
    for (int j = 0; j < 8; ++j) { acc[it][j] = 0.f; wv[it][j] = 0.f; }
    if (v < nv) {
      unpack8(reinterpret_cast<const bf16x8*>(w)[v], wv[it]);
#pragma unroll
      for (int j = 0; j < 8; ++j) wv[it][j] += w_off;
    }
  }
  int par = 0;
  for (long long row = first + blockIdx.x; row < first + T; row += gridDim.x) {
    const bf16x8* dyr = reinterpret_cast<const bf16x8*>(dy + row * ld_dy);
    const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * ldx);
    const float rs = rstd[row];
    float g[ITERS][8], xv[ITERS][8];
    float dot = 0.f;
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
      const int v = threadIdx.x + it * RMS_BWD_NT;
      if (v < nv) {
        unpack8(dyr[v], g[it]);
        unpack8(xr[v], xv[it]);
#pragma unroll
        for (int j = 0; j < 8; ++j) dot += g[it][j] * wv[it][j] * xv[it][j];
      }
    }
    // one barrier per row: warp sums go to one of two alternating sets of slots and every thread adds the sixteen
    // partials itself (a set is rewritten two rows later, after the barrier of the row in between)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    float* slots = sh + par * (RMS_BWD_NT / 32);
    par ^= 1;
    if ((threadIdx.x & 31) == 0) slots[threadIdx.x >> 5] = dot;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int wq = 0; wq < RMS_BWD_NT / 32; ++wq) tot += slots[wq];
    const float mean_dot = tot * rs / (float)D;
    const bf16x8* drr = dres ? reinterpret_cast<const bf16x8*>(dres + row * ld_dx) : nullptr;
    bf16x8* dxr = reinterpret_cast<bf16x8*>(dx + row * ld_dx);
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
      const int v = threadIdx.x + it * RMS_BWD_NT;
      if (v < nv) {
        float o[8];
        if (drr) unpack8(drr[v], o);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = xv[it][j] * rs;
          const float d = rs * (g[it][j] * wv[it][j] - xh * mean_dot);
          o[j] = drr ? o[j] + d : d;
          acc[it][j] += g[it][j] * xh;
        }
        dxr[v] = pack8(o);
      }
    }
  }
  if (partial) {
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
      const int v = threadIdx.x + it * RMS_BWD_NT;
      if (v < nv) {
        float4* dst = reinterpret_cast<float4*>(partial + ((MANY ? (long long)blockIdx.y * gridDim.x : 0ll) + blockIdx.x) * D + v * 8);
        dst[0] = make_float4(acc[it][0], acc[it][1], acc[it][2], acc[it][3]);
        dst[1] = make_float4(acc[it][4], acc[it][5], acc[it][6], acc[it][7]);
      }
    }
  }
}

// dst[b][c] += sum_r partial[b][r][c] (b = blockIdx.y); CTA = 32 columns x 8 row groups.
template <bool MANY>
__global__ void __launch_bounds__(256) colsum_add_kernel(const float* __restrict__ partial, float* __restrict__ dst,
                                                         int rows, int D, long long dst_stride) {
  opk::pdl_trigger();
  __shared__ float sh[8][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (c < D) {
    if constexpr (!MANY) {
      for (int r = ry; r < rows; r += 8) s += partial[(long long)r * D + c];
    } else {
      // with one more term in the address the compiler has fewer loads in flight: eight are asked for ahead (1.0 us less for 296 rows)
      const float* src = partial + ((long long)blockIdx.y * rows + ry) * D + c;
      int r = ry;
      for (; r + 56 < rows; r += 64, src += 64ll * D) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v[u]) : "l"(src + 8ll * u * D));
#pragma unroll
        for (int u = 0; u < 8; ++u) s += v[u];
      }
      for (; r < rows; r += 8, src += 8ll * D) s += *src;
    }
  }
  sh[ry][cx] = s;
  __syncthreads();
  if (ry == 0 && c < D) {
#pragma unroll
    for (int k = 1; k < 8; ++k) s += sh[k][cx];
    dst[(MANY ? blockIdx.y * dst_stride : 0) + c] += s;
  }
}

// ------------------------------------------------------------------------------------------- LayerNorm
__global__ void __launch_bounds__(NT) layernorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                           const __nv_bfloat16* __restrict__ w,
                                                           const __nv_bfloat16* __restrict__ b,
                                                           __nv_bfloat16* __restrict__ y, float* __restrict__ mean,
                                                           float* __restrict__ rstd, int D, float eps) {
  opk::pdl_trigger();
  __shared__ float sh[32];
  const long long row = blockIdx.x;
  const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * D);
  const int nv = D >> 3;
  float s = 0.f;
  for (int i = threadIdx.x; i < nv; i += NT) {
    float f[8];
    unpack8(xr[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += f[j];
  }
  const float mu = block_sum<NT>(s, sh) / (float)D;
  float ss = 0.f;
  for (int i = threadIdx.x; i < nv; i += NT) {
    float f[8];
    unpack8(xr[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += (f[j] - mu) * (f[j] - mu);
  }
  const float rs = rsqrtf(block_sum<NT>(ss, sh) / (float)D + eps);
  if (threadIdx.x == 0) {
    if (mean) mean[row] = mu;
    if (rstd) rstd[row] = rs;
  }
  const bf16x8* wr = reinterpret_cast<const bf16x8*>(w);
  const bf16x8* br = b ? reinterpret_cast<const bf16x8*>(b) : nullptr;
  bf16x8* yr = reinterpret_cast<bf16x8*>(y + row * D);
  for (int i = threadIdx.x; i < nv; i += NT) {
    float f[8], g[8], bb[8];
    unpack8(xr[i], f);
    unpack8(wr[i], g);
    if (br) unpack8(br[i], bb);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = (f[j] - mu) * rs * g[j] + (br ? bb[j] : 0.f);
    yr[i] = pack8(f);
  }
}

template <bool MANY>
__global__ void __launch_bounds__(NT) layernorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy,
                                                           const __nv_bfloat16* __restrict__ x,
                                                           const __nv_bfloat16* __restrict__ w,
                                                           const float* __restrict__ mean,
                                                           const float* __restrict__ rstd,
                                                           const __nv_bfloat16* __restrict__ dres,
                                                           __nv_bfloat16* __restrict__ dx, float* __restrict__ dw,
                                                           float* __restrict__ db, int T, int D, long long stride) {
  __shared__ float sh[32];
  const int nv = D >> 3;
  const long long first = MANY ? (long long)blockIdx.y * T : 0;       // gridDim.y examples of T rows, gradients `stride` floats apart
  float dwp[MAX_COL_ITERS][8], dbp[MAX_COL_ITERS][8];
#pragma unroll
  for (int c = 0; c < MAX_COL_ITERS; ++c)
#pragma unroll
    for (int j = 0; j < 8; ++j) { dwp[c][j] = 0.f; dbp[c][j] = 0.f; }
  const bf16x8* wr = reinterpret_cast<const bf16x8*>(w);
  for (long long row = first + blockIdx.x; row < first + T; row += gridDim.x) {
    const bf16x8* dyr = reinterpret_cast<const bf16x8*>(dy + row * D);
    const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * D);
    const float rs = rstd[row], mu = mean[row];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int c = 0; c < MAX_COL_ITERS; ++c) {
      const int i = threadIdx.x + c * NT;
      if (i < nv) {
        float g[8], xv[8], wv[8];
        unpack8(dyr[i], g);
        unpack8(xr[i], xv);
        unpack8(wr[i], wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = (xv[j] - mu) * rs;
          dwp[c][j] += g[j] * xh;
          dbp[c][j] += g[j];
          const float gw = g[j] * wv[j];
          s1 += gw;
          s2 += gw * xh;
        }
      }
    }
    const float m1 = block_sum<NT>(s1, sh) / (float)D;
    const float m2 = block_sum<NT>(s2, sh) / (float)D;
    const bf16x8* drr = dres ? reinterpret_cast<const bf16x8*>(dres + row * D) : nullptr;
    bf16x8* dxr = reinterpret_cast<bf16x8*>(dx + row * D);
#pragma unroll
    for (int c = 0; c < MAX_COL_ITERS; ++c) {
      const int i = threadIdx.x + c * NT;
      if (i < nv) {
        float g[8], xv[8], wv[8], o[8];
        unpack8(dyr[i], g);
        unpack8(xr[i], xv);
        unpack8(wr[i], wv);
        if (drr) unpack8(drr[i], o);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = (xv[j] - mu) * rs;
          const float d = rs * (g[j] * wv[j] - m1 - xh * m2);
          o[j] = drr ? o[j] + d : d;
        }
        dxr[i] = pack8(o);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < MAX_COL_ITERS; ++c) {
    const int i = threadIdx.x + c * NT;
    if (i < nv) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (dw) atomicAdd(&dw[(MANY ? blockIdx.y * stride : 0) + i * 8 + j], dwp[c][j]);
        if (db) atomicAdd(&db[(MANY ? blockIdx.y * stride : 0) + i * 8 + j], dbp[c][j]);
      }
    }
  }
}

// LayerNorm backward for D <= 1024, one warp per row, the row in registers (VPL vectors of 8 per lane): no block barrier
// inside the row loop. The weight and bias gradients are kept per lane over the warp's rows, added over the CTA's warps in
// shared memory and leave as one vector reduction per four columns and CTA. (The general kernel above reserves registers
// for 16,384 columns, synchronises four times per row and issues one scalar atomic per column, thread and CTA:
// 30.6 us at 1024 x 768.)
__device__ __forceinline__ void red_add_v4(float* dst, const float* v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
}
template <int VPL, bool MANY>
__global__ void __launch_bounds__(256) layernorm_bwd_warp_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                                 const __nv_bfloat16* __restrict__ w, const float* __restrict__ mean,
                                                                 const float* __restrict__ rstd, const __nv_bfloat16* __restrict__ dres,
                                                                 __nv_bfloat16* __restrict__ dx, float* __restrict__ dw,
                                                                 float* __restrict__ db, int T, int D, long long stride) {
  opk::pdl_trigger();
  const long long first = MANY ? (long long)blockIdx.y * T : 0;       // gridDim.y examples of T rows, gradients `stride` floats apart
  constexpr int W = VPL * 256;
  __shared__ float sh[8 * W];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nv = D >> 3;
  float gw[VPL][8], gb[VPL][8];
#pragma unroll
  for (int i = 0; i < VPL; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) { gw[i][j] = 0.f; gb[i][j] = 0.f; }
  for (long long row = first + blockIdx.x * 8ll + warp; row < first + T; row += gridDim.x * 8ll) {
    const bf16x8* dyr = reinterpret_cast<const bf16x8*>(dy + row * D);
    const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * D);
    const bf16x8* drr = dres ? reinterpret_cast<const bf16x8*>(dres + row * D) : nullptr;
    const bf16x8* wr = reinterpret_cast<const bf16x8*>(w);
    const float rs = rstd[row], mu = mean[row];
    float g[VPL][8], xh[VPL][8], wv[VPL][8];
    float p1[4] = {0.f, 0.f, 0.f, 0.f}, p2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = lane + 32 * i;
      if (v < nv) {
        float xv[8];
        unpack8(dyr[v], g[i]);
        unpack8(xr[v], xv);
        unpack8(wr[v], wv[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[i][j] = (xv[j] - mu) * rs;
          gw[i][j] += g[i][j] * xh[i][j];
          gb[i][j] += g[i][j];
          const float t = g[i][j] * wv[i][j];
          p1[i] += t;
          p2[i] += t * xh[i][j];
        }
      }
    }
    // every 256 columns are summed by themselves and then together in the order of the general kernel's block reduction:
    // the input gradient does not depend on which of the two kernels a width takes
#pragma unroll
    for (int i = 0; i < VPL; ++i)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        p1[i] += __shfl_xor_sync(0xffffffffu, p1[i], o);
        p2[i] += __shfl_xor_sync(0xffffffffu, p2[i], o);
      }
    const float m1 = ((p1[0] + p1[2]) + (p1[1] + p1[3])) / (float)D, m2 = ((p2[0] + p2[2]) + (p2[1] + p2[3])) / (float)D;
    bf16x8* dxr = reinterpret_cast<bf16x8*>(dx + row * D);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = lane + 32 * i;
      if (v < nv) {
        float o[8];
        if (drr) unpack8(drr[v], o);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float d = rs * (g[i][j] * wv[i][j] - m1 - xh[i][j] * m2);
          o[j] = drr ? o[j] + d : d;
        }
        dxr[v] = pack8(o);
      }
    }
  }
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    float* out = which ? db : dw;
    if (!out) continue;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < VPL; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {      // columns past D hold zeros and are not read below
        const float* g = which ? gb[i] : gw[i];
        *reinterpret_cast<float4*>(&sh[warp * W + (lane + 32 * i) * 8 + 4 * h]) = make_float4(g[4 * h], g[4 * h + 1], g[4 * h + 2], g[4 * h + 3]);
      }
    __syncthreads();
    const int c = threadIdx.x * 4;         // D <= 1024: one group of four columns per thread
    if (c < D) {
      float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) a[j] += sh[k * W + c + j];
      red_add_v4(out + (MANY ? blockIdx.y * stride : 0) + c, a);
    }
  }
}

// ------------------------------------------------------------------------------------------- RoPE
__global__ void rope_kernel(__nv_bfloat16* __restrict__ qk, const float* __restrict__ cs,
                            const int* __restrict__ pos, int period, long long T, int n_heads, int hd, long long ld, float sign) {
  const int half = hd >> 1;
  const long long total = T * n_heads * half;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int i = idx % half;
    const long long th = idx / half;
    const int h = th % n_heads;
    const long long t = th / n_heads;
    const long long p = pos ? pos[t] : (period ? t % period : t);
    const float c = cs[(p * half + i) * 2], s = cs[(p * half + i) * 2 + 1] * sign;
    __nv_bfloat16* base = qk + t * ld + (long long)h * hd;
    const float x1 = __bfloat162float(base[i]), x2 = __bfloat162float(base[i + half]);
    base[i] = __float2bfloat16(x1 * c - x2 * s);
    base[i + half] = __float2bfloat16(x2 * c + x1 * s);
  }
}

// Vector form: a thread rotates 8 consecutive pairs (x[i..i+7], x[i+half..i+half+7]) with 16-byte accesses.
__global__ void __launch_bounds__(256) rope_vec8_kernel(__nv_bfloat16* __restrict__ qk, const float* __restrict__ cs,
                                                        const int* __restrict__ pos, int period, long long T, int n_heads, int hd,
                                                        long long ld, float sign) {
  opk::pdl_trigger();
  const int half = hd >> 1, hv = half >> 3;
  const long long total = T * n_heads * hv;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int iv = (int)(idx % hv);
    const long long th = idx / hv;
    const int h = (int)(th % n_heads);
    const long long t = th / n_heads;
    const long long p = pos ? pos[t] : (period ? t % period : t);
    const float4* c4 = reinterpret_cast<const float4*>(cs + (p * half + iv * 8) * 2);
    bf16x8* lo = reinterpret_cast<bf16x8*>(qk + t * ld + (long long)h * hd + iv * 8);
    bf16x8* hi = reinterpret_cast<bf16x8*>(qk + t * ld + (long long)h * hd + half + iv * 8);
    float a[8], b[8];
    unpack8(*lo, a);
    unpack8(*hi, b);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 v = c4[q];            // (cos, sin) of pairs 2q and 2q + 1
      const float s0 = v.y * sign, s1 = v.w * sign;
      const float x1 = a[2 * q], x2 = b[2 * q], y1 = a[2 * q + 1], y2 = b[2 * q + 1];
      a[2 * q] = x1 * v.x - x2 * s0;
      b[2 * q] = x2 * v.x + x1 * s0;
      a[2 * q + 1] = y1 * v.z - y2 * s1;
      b[2 * q + 1] = y2 * v.z + y1 * s1;
    }
    *lo = pack8(a);
    *hi = pack8(b);
  }
}

// ------------------------------------------------------------------------------------------- gated activations
__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ float gelu_tanh(float x) {
  const float k = 0.7978845608028654f;
  return 0.5f * x * (1.f + tanhf(k * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ float gelu_tanh_grad(float x) {
  const float k = 0.7978845608028654f;
  const float u = k * (x + 0.044715f * x * x * x);
  const float t = tanhf(u);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k * (1.f + 3.f * 0.044715f * x * x);
}
__device__ __forceinline__ float gelu_erf(float x) { return 0.5f * x * (1.f + erff(x * 0.7071067811865476f)); }
__device__ __forceinline__ float gelu_erf_grad(float x) {
  return 0.5f * (1.f + erff(x * 0.7071067811865476f)) + x * 0.3989422804014327f * __expf(-0.5f * x * x);
}

// MODE 0 = SwiGLU, 1 = GEGLU exact, 2 = GEGLU tanh
template <int MODE>
__device__ __forceinline__ float gate_fn(float g) {
  return MODE == 0 ? g * sigmoidf_(g) : (MODE == 1 ? gelu_erf(g) : gelu_tanh(g));
}
template <int MODE>
__device__ __forceinline__ float gate_grad(float g) {
  if (MODE == 0) {
    const float s = sigmoidf_(g);
    return s * (1.f + g * (1.f - s));
  }
  return MODE == 1 ? gelu_erf_grad(g) : gelu_tanh_grad(g);
}

// MODE 3 = SwiGLU, 4 = GEGLU tanh with the library's exponential and every operation rounded by itself, in the order of the
// formulas that they stand for in the LoRA operators: the result does not depend on whether a call reaches the kernel.
template <int MODE>
__device__ __forceinline__ float glu_value(float g, float u) {
  if (MODE == 3) return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.f, expf(-g))), u);
  return MODE == 4 ? __fmul_rn(gelu_tanh(g), u) : gate_fn<MODE>(g) * u;
}
template <int MODE>
__device__ __forceinline__ void glu_grads(float d, float g, float u, float& dg, float& du) {
  if (MODE < 3) {
    dg = d * u * gate_grad<MODE>(g);
    du = d * gate_fn<MODE>(g);
    return;
  }
  float a, da;
  if (MODE == 3) {
    const float s = __fdiv_rn(1.f, __fadd_rn(1.f, expf(-g)));
    a = __fmul_rn(g, s);
    da = __fmul_rn(s, __fadd_rn(1.f, __fmul_rn(g, __fadd_rn(1.f, -s))));
  } else {
    const float k = 0.7978845608028654f, h = __fmul_rn(0.5f, g);
    const float t = tanhf(__fmul_rn(k, __fadd_rn(g, __fmul_rn(0.044715f, __fmul_rn(__fmul_rn(g, g), g)))));
    const float t1 = __fadd_rn(1.f, t);
    a = __fmul_rn(h, t1);
    const float slope = __fadd_rn(1.f, __fmul_rn(__fmul_rn((float)(3 * 0.044715), g), g));
    da = __fadd_rn(__fmul_rn(0.5f, t1), __fmul_rn(__fmul_rn(__fmul_rn(h, __fadd_rn(1.f, -__fmul_rn(t, t))), k), slope));
  }
  dg = __fmul_rn(__fmul_rn(d, u), da);
  du = __fmul_rn(d, a);
}

// Gate and up either interleaved pairwise in one buffer (SPLIT = false: gate[2i], gate[2i+1] = gate, up of element i) or
// in two buffers. A thread handles 8 elements with 16-byte accesses; n is a multiple of 8 in the vector kernels (rows are
// multiples of 8 elements for every caller), the scalar kernel takes the rest. Bound by memory: 3 (forward) or 5
// (backward) bf16 values per element.
template <int MODE, bool SPLIT>
__global__ void __launch_bounds__(256) glu_fwd_kernel(const __nv_bfloat16* __restrict__ gate, const __nv_bfloat16* __restrict__ up,
                                                      __nv_bfloat16* __restrict__ act, long long nvec) {
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < nvec; i += (long long)gridDim.x * 256) {
    float a[8], b[8], o[8];
    if (SPLIT) {
      unpack8(reinterpret_cast<const bf16x8*>(gate)[i], a);
      unpack8(reinterpret_cast<const bf16x8*>(up)[i], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = glu_value<MODE>(a[j], b[j]);
    } else {
      unpack8(reinterpret_cast<const bf16x8*>(gate)[2 * i], a);
      unpack8(reinterpret_cast<const bf16x8*>(gate)[2 * i + 1], b);
#pragma unroll
      for (int j = 0; j < 4; ++j) { o[j] = gate_fn<MODE>(a[2 * j]) * a[2 * j + 1]; o[4 + j] = gate_fn<MODE>(b[2 * j]) * b[2 * j + 1]; }
    }
    reinterpret_cast<bf16x8*>(act)[i] = pack8(o);
  }
}
template <int MODE, bool SPLIT>
__global__ void __launch_bounds__(256) glu_bwd_kernel(const __nv_bfloat16* __restrict__ dact, const __nv_bfloat16* __restrict__ gate,
                                                      const __nv_bfloat16* __restrict__ up, __nv_bfloat16* __restrict__ dgate,
                                                      __nv_bfloat16* __restrict__ dup, long long nvec) {
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < nvec; i += (long long)gridDim.x * 256) {
    float d[8], a[8], b[8], oa[8], ob[8];
    unpack8(reinterpret_cast<const bf16x8*>(dact)[i], d);
    if (SPLIT) {
      unpack8(reinterpret_cast<const bf16x8*>(gate)[i], a);
      unpack8(reinterpret_cast<const bf16x8*>(up)[i], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) glu_grads<MODE>(d[j], a[j], b[j], oa[j], ob[j]);
      reinterpret_cast<bf16x8*>(dgate)[i] = pack8(oa);
      reinterpret_cast<bf16x8*>(dup)[i] = pack8(ob);
    } else {
      unpack8(reinterpret_cast<const bf16x8*>(gate)[2 * i], a);
      unpack8(reinterpret_cast<const bf16x8*>(gate)[2 * i + 1], b);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        glu_grads<MODE>(d[j], a[2 * j], a[2 * j + 1], oa[2 * j], oa[2 * j + 1]);
        glu_grads<MODE>(d[4 + j], b[2 * j], b[2 * j + 1], ob[2 * j], ob[2 * j + 1]);
      }
      reinterpret_cast<bf16x8*>(dgate)[2 * i] = pack8(oa);
      reinterpret_cast<bf16x8*>(dgate)[2 * i + 1] = pack8(ob);
    }
  }
}
// interleaved form, one element per thread from `begin` on; WORD: a pair is read and written as one 32-bit word
template <int MODE, bool WORD>
__global__ void __launch_bounds__(256) glu_fwd_pair_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act, long long begin,
                                                           long long n) {
  for (long long i = begin + blockIdx.x * 256ll + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    const float2 p = WORD ? __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(gu)[i])
                          : make_float2(__bfloat162float(gu[2 * i]), __bfloat162float(gu[2 * i + 1]));
    act[i] = __float2bfloat16(gate_fn<MODE>(p.x) * p.y);
  }
}
template <int MODE, bool WORD>
__global__ void __launch_bounds__(256) glu_bwd_pair_kernel(const __nv_bfloat16* __restrict__ dact, const __nv_bfloat16* __restrict__ gu,
                                                           __nv_bfloat16* __restrict__ dgu, long long begin, long long n) {
  for (long long i = begin + blockIdx.x * 256ll + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    const float2 p = WORD ? __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(gu)[i])
                          : make_float2(__bfloat162float(gu[2 * i]), __bfloat162float(gu[2 * i + 1]));
    float dg, du;
    glu_grads<MODE>(__bfloat162float(dact[i]), p.x, p.y, dg, du);
    const __nv_bfloat162 o = __floats2bfloat162_rn(dg, du);
    if (WORD) {
      reinterpret_cast<__nv_bfloat162*>(dgu)[i] = o;
    } else {
      dgu[2 * i] = o.x;
      dgu[2 * i + 1] = o.y;
    }
  }
}
__global__ void __launch_bounds__(256) gelu_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, long long nvec,
                                                       long long n) {
  opk::pdl_trigger();
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < nvec; i += (long long)gridDim.x * 256) {
    float a[8];
    unpack8(reinterpret_cast<const bf16x8*>(x)[i], a);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = gelu_tanh(a[j]);
    reinterpret_cast<bf16x8*>(y)[i] = pack8(a);
  }
  for (long long i = nvec * 8 + blockIdx.x * 256ll + threadIdx.x; i < n; i += (long long)gridDim.x * 256)
    y[i] = __float2bfloat16(gelu_tanh(__bfloat162float(x[i])));
}
__global__ void __launch_bounds__(256) gelu_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                       __nv_bfloat16* __restrict__ dx, long long nvec, long long n) {
  opk::pdl_trigger();
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < nvec; i += (long long)gridDim.x * 256) {
    float a[8], d[8];
    unpack8(reinterpret_cast<const bf16x8*>(x)[i], a);
    unpack8(reinterpret_cast<const bf16x8*>(dy)[i], d);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = d[j] * gelu_tanh_grad(a[j]);
    reinterpret_cast<bf16x8*>(dx)[i] = pack8(a);
  }
  for (long long i = nvec * 8 + blockIdx.x * 256ll + threadIdx.x; i < n; i += (long long)gridDim.x * 256)
    dx[i] = __float2bfloat16(__bfloat162float(dy[i]) * gelu_tanh_grad(__bfloat162float(x[i])));
}

// ------------------------------------------------------------------------------------------- embedding
template <bool PERIODIC>
__global__ void embedding_fwd_kernel(const int* __restrict__ tok, const __nv_bfloat16* __restrict__ table,
                                     const __nv_bfloat16* __restrict__ pos_table, __nv_bfloat16* __restrict__ out,
                                     int D, int vocab, int period) {
  const long long t = blockIdx.x;
  // an id outside the table yields a zero embedding row: never an address outside the table
  const bool in_table = tok[t] >= 0 && tok[t] < vocab;
  (void)OPK_IDX_OK(tok[t], vocab);
  const bf16x8* src = reinterpret_cast<const bf16x8*>(table + (long long)(in_table ? tok[t] : 0) * D);
  const bf16x8* ps = pos_table ? reinterpret_cast<const bf16x8*>(pos_table + (PERIODIC ? t % period : t) * D) : nullptr;
  bf16x8* dst = reinterpret_cast<bf16x8*>(out + t * D);
  for (int i = threadIdx.x; i < (D >> 3); i += blockDim.x) {
    if (ps || !in_table) {
      float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, b[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (in_table) unpack8(src[i], a);
      if (ps) unpack8(ps[i], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += b[j];
      dst[i] = pack8(a);
    } else {
      dst[i] = src[i];
    }
  }
}
// Token ids outside [0, vocab) are skipped by all three table kernels (their rep[] entry becomes -1, which the
// accumulate / add-rows kernels treat as "not a representative row"), so a bad id can never index past the table.
__device__ __forceinline__ bool emb_tok_ok(int tok, int vocab) {
  (void)OPK_IDX_OK(tok, vocab);
  return (unsigned)tok < (unsigned)vocab;
}
OPK_DEBUG_BOUNDS_UNIT();
// gridDim.y examples of T tokens each, with a first-occurrence table, representatives and rows of their own.
__global__ void emb_first_pos_kernel(const int* __restrict__ tok, int* __restrict__ first_pos, int T, int vocab) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  tok += (long long)blockIdx.y * T;
  first_pos += (long long)blockIdx.y * vocab;
  if (t < T && emb_tok_ok(tok[t], vocab)) atomicMin(&first_pos[tok[t]], t);
}
__global__ void emb_scatter_kernel(const int* __restrict__ tok, const __nv_bfloat16* __restrict__ dx,
                                   const int* __restrict__ first_pos, int* __restrict__ rep, float* __restrict__ gc,
                                   int T, int D, int vocab) {
  const long long t = blockIdx.x, first = (long long)blockIdx.y * T;
  tok += first;
  rep += first;
  dx += first * D;
  gc += first * D;
  first_pos += (long long)blockIdx.y * vocab;
  if (!emb_tok_ok(tok[t], vocab)) {
    if (threadIdx.x == 0) rep[t] = -1;
    return;
  }
  const int r = first_pos[tok[t]];
  if (threadIdx.x == 0) rep[t] = r;
  const __nv_bfloat16* src = dx + t * D;
  float* dst = gc + (long long)r * D;
  for (int d = threadIdx.x; d < D; d += blockDim.x) atomicAdd(&dst[d], __bfloat162float(src[d]));
}
__global__ void emb_reset_kernel(const int* __restrict__ tok, int* __restrict__ first_pos, int T, int vocab) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  tok += (long long)blockIdx.y * T;
  first_pos += (long long)blockIdx.y * vocab;
  if (t < T && emb_tok_ok(tok[t], vocab)) first_pos[tok[t]] = INT_MAX;
}
// ATOMIC: the rows of acc are shared with other GPUs' kernels (sharded sums, acc may be peer-mapped), so the add is a
// reduction instead of a read-modify-write.
template <bool ATOMIC>
__global__ void emb_accumulate_kernel(const int* __restrict__ tok, const int* __restrict__ rep,
                                      const float* __restrict__ gc, const float* __restrict__ scale,
                                      float* __restrict__ acc, int D) {
  const long long t = blockIdx.x;
  if (rep[t] != (int)t) return;
  const float s = *scale;
  const float* src = gc + t * D;
  float* dst = acc + (long long)tok[t] * D;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    const float g = __bfloat162float(__float2bfloat16(src[d]));            // the stored per-example gradient
    const float c = __bfloat162float(__float2bfloat16(g * s));             // clipped in storage precision
    if (ATOMIC) atomicAdd(&dst[d], c);
    else dst[d] += c;
  }
}

// ------------------------------------------------------------------------------------------- reductions
template <bool FP32> constexpr int kVec16 = FP32 ? 4 : 8;
template <bool FP32>
__device__ __forceinline__ void load_vec16(const void* p, long long i, float (&f)[8]) {
  if (FP32) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + i));
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
  } else {
    const uint4 raw = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p) + i));
    unpack8(*reinterpret_cast<const bf16x8*>(&raw), f);
  }
}
// MANY: gridDim.y buffers with one sum each, on one 16-byte boundary. One buffer has no offset in its addresses: with it 8192 x 8192
// values take 23 us instead of 21.
template <bool FP32, bool ROUND, bool MANY>
__global__ void __launch_bounds__(NT) sumsq_kernel(const void* __restrict__ x, long long n, double* out, long long stride) {
  double acc = 0.0;
  const long long first = MANY ? blockIdx.y * stride : 0;
  float part = 0.f;
  int cnt = 0;
  // 16-byte loads, four vectors in flight, when the base allows it; fp32 partials of at most 64 squares as below
  constexpr int VW = FP32 ? 4 : 8;
  const long long nvec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? n / VW : 0;
#pragma unroll 4
  for (long long i = blockIdx.x * (long long)NT + threadIdx.x; i < nvec; i += (long long)gridDim.x * NT) {
    float f[8];
    load_vec16<FP32>(x, first + i * VW, f);
    float p8 = 0.f;
#pragma unroll
    for (int j = 0; j < VW; ++j) {
      const float v = ROUND ? __bfloat162float(__float2bfloat16(f[j])) : f[j];
      p8 += v * v;
    }
    acc += (double)p8;
  }
  for (long long i = nvec * VW + blockIdx.x * (long long)NT + threadIdx.x; i < n; i += (long long)gridDim.x * NT) {
    float v = FP32 ? reinterpret_cast<const float*>(x)[first + i] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(x)[first + i]);
    if (ROUND) v = __bfloat162float(__float2bfloat16(v));
    part += v * v;
    if (++cnt == 64) { acc += (double)part; part = 0.f; cnt = 0; }
  }
  acc += (double)part;
  // fp64 block reduction through two fp32 words would lose bits; reduce doubles with shuffles directly
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __shared__ double shd[NT / 32];
  if ((threadIdx.x & 31) == 0) shd[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < NT / 32; ++w) t += shd[w];
    atomicAdd(MANY ? out + blockIdx.y : out, t);
  }
}

// ------------------------------------------------------------------------------------------- cross entropy
__global__ void lce_finalize_kernel(const float* __restrict__ pmax, const float* __restrict__ psum,
                                    const float* __restrict__ tgt, const int* __restrict__ labels,
                                    float* __restrict__ lse, float* __restrict__ nll, int T, int tiles) {
  opk::pdl_trigger();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= T) return;
  const float* pm = pmax + (long long)row * tiles;
  const float* ps = psum + (long long)row * tiles;
  float m = -INFINITY;
  for (int i = lane; i < tiles; i += 32) m = fmaxf(m, pm[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  float s = 0.f;
  for (int i = lane; i < tiles; i += 32) s += ps[i] * __expf(pm[i] - m);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    const float l = m + logf(s);
    lse[row] = l;
    if (nll) nll[row] = labels[row] >= 0 ? l - tgt[row] : 0.f;
  }
}

// Per-example RMSNorm weight gradient: dw[b][c] += sum over the rows of example b of dy * x * rstd (the normalised
// input). One thread per column, grid.y = example, grid.z = row chunk; fp32 atomics combine the row chunks.
__global__ void __launch_bounds__(256) rmsnorm_dw_per_example_kernel(const __nv_bfloat16* __restrict__ dy,
                                                                     const __nv_bfloat16* __restrict__ x,
                                                                     const float* __restrict__ rstd, float* __restrict__ dw,
                                                                     int rows, int D) {
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= D) return;
  const long long b = blockIdx.y;
  const int chunk = (rows + gridDim.z - 1) / gridDim.z;
  const int r0 = blockIdx.z * chunk, r1 = min(rows, r0 + chunk);
  float acc = 0.f;
  for (int r = r0; r < r1; ++r) {
    const long long row = b * rows + r;
    acc += __bfloat162float(dy[row * D + c]) * __bfloat162float(x[row * D + c]) * rstd[row];
  }
  if (r1 > r0) atomicAdd(&dw[b * D + c], acc);
}

// Per-example loss bookkeeping in one CTA: ntok = max(1, #labels >= 0); coef[t] = [label >= 0] / ntok (* *weight);
// loss = sum_t nll[t] * coef[t]. Two block reductions; T is a sequence length.
__global__ void __launch_bounds__(1024) loss_coef_kernel(const int* __restrict__ labels, const float* __restrict__ nll,
                                                         const float* __restrict__ weight, float* __restrict__ coef,
                                                         float* __restrict__ loss, float* __restrict__ ntok, int T) {
  opk::pdl_trigger();
  labels += (long long)blockIdx.x * T;         // one CTA per example
  nll += (long long)blockIdx.x * T;
  coef += (long long)blockIdx.x * T;
  __shared__ float red[32];
  __shared__ float bcast;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float cnt = 0.f;
  for (int t = threadIdx.x; t < T; t += blockDim.x) cnt += labels[t] >= 0 ? 1.f : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if (lane == 0) red[warp] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    bcast = fmaxf(s, 1.f);
  }
  __syncthreads();
  const float n = bcast;
  const float w = weight ? *weight : 1.f;
  float acc = 0.f;
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    const float c = labels[t] >= 0 ? w / n : 0.f;
    coef[t] = c;
    acc += nll[t] * c;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __syncthreads();
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int wi = 0; wi < (int)(blockDim.x >> 5); ++wi) s += red[wi];
    loss[blockIdx.x] = s;
    if (ntok) ntok[blockIdx.x] = n;
  }
}

template <bool FP32>
__device__ __forceinline__ float load_logit(const void* p, long long i) {
  return FP32 ? reinterpret_cast<const float*>(p)[i] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
}
__device__ __forceinline__ float cap(float z, float scale, float softcap) {
  z *= scale;
  return softcap > 0.f ? softcap * tanhf(z / softcap) : z;
}

// Rows start anywhere (V need not be a multiple of the vector width): up to VW - 1 elements before the first 16-byte
// boundary and after the last one are handled one by one, everything between with 16-byte accesses.
// first element of the row that lies on a 16-byte boundary (at most n)
template <bool FP32>
__device__ __forceinline__ int ce_head(const void* p, long long base, int n) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p) + (uintptr_t)base * (FP32 ? 4 : 2);
  const int h = (int)(((16 - (a & 15)) & 15) / (FP32 ? 4 : 2));
  return h < n ? h : n;
}

// What bounds the row kernels when there are fewer rows than SMs is the chain of load latencies of one CTA: the 16-byte loads of
// kRowLoads vectors are issued before the first is used (with the loads one after the other behind the streaming stores, 40 rows
// of 50,257 fp32 logits took 25 us backward, 11.5 now; forward 14.5, 9.3 now). Rows of at most kNarrowRow columns go
// element by element: a vector gives one thread the work of eight (16,384 rows of 130 bf16 logits with a soft cap: forward 35 us,
// 22.7 now).
template <bool FP32> constexpr int kRowLoads = FP32 ? 4 : 2;
constexpr int kNarrowRow = 2 * NT;

// One CTA per row, online (max, sum) per thread: one exponential per element plus one per vector. Entries of -inf that come
// before any other value are passed over (the sum stays 0); a NaN is not, although fmaxf ignores it: the row's loss is NaN.
template <bool FP32, bool NARROW>
__global__ void __launch_bounds__(NT) ce_fwd_kernel(const void* __restrict__ logits, const int* __restrict__ labels,
                                                    float* __restrict__ nll, float* __restrict__ lse, int V,
                                                    long long ld, float scale, float softcap) {
  constexpr int VW = kVec16<FP32>;
  __shared__ float sh[32];
  const long long row = blockIdx.x;
  const long long base = row * ld;
  float m = -INFINITY, s = 0.f;
  auto one = [&](float raw) {
    const float z = cap(raw, scale, softcap);
    const float nm = fmaxf(m, z);
    if (nm == -INFINITY && z == -INFINITY) return;
    s = s * __expf(m - nm) + __expf(z - nm);
    m = nm;
  };
  auto eight = [&](float (&z)[8]) {
    float nm = m;
#pragma unroll
    for (int j = 0; j < VW; ++j) { z[j] = cap(z[j], scale, softcap); nm = fmaxf(nm, z[j]); }
    if (nm == -INFINITY) {
      float t = z[0];
#pragma unroll
      for (int j = 1; j < VW; ++j) t += z[j];
      if (t == -INFINITY) return;         // all of them -inf, no NaN among them
    }
    float add = 0.f;
#pragma unroll
    for (int j = 0; j < VW; ++j) add += __expf(z[j] - nm);
    s = s * __expf(m - nm) + add;
    m = nm;
  };
  if (NARROW) {
    for (int i = threadIdx.x; i < V; i += NT) one(load_logit<FP32>(logits, base + i));
  } else {
    constexpr int U = kRowLoads<FP32>;
    const int head = ce_head<FP32>(logits, base, V);
    const int nvec = (V - head) / VW, tail = head + nvec * VW;
    if ((int)threadIdx.x < head) one(load_logit<FP32>(logits, base + threadIdx.x));
    if (tail + (int)threadIdx.x < V) one(load_logit<FP32>(logits, base + tail + threadIdx.x));
    int i = threadIdx.x;
    for (; i + (U - 1) * NT < nvec; i += U * NT) {
      float z[U][8];
#pragma unroll
      for (int u = 0; u < U; ++u) load_vec16<FP32>(logits, base + head + (long long)(i + u * NT) * VW, z[u]);
#pragma unroll
      for (int u = 0; u < U; ++u) eight(z[u]);
    }
    for (; i < nvec; i += NT) {
      float z[8];
      load_vec16<FP32>(logits, base + head + (long long)i * VW, z);
      eight(z);
    }
  }
  // combine (m, s) pairs: first the max, then rescaled sums
  float gm = m;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = gm;
  __syncthreads();
  float bm = sh[0];
  for (int w = 1; w < NT / 32; ++w) bm = fmaxf(bm, sh[w]);
  const float tot = block_sum<NT>(m == -INFINITY ? s : s * __expf(m - bm), sh);   // m = -inf: s is 0, or NaN
  if (threadIdx.x == 0) {
    const float l = bm + logf(tot);
    if (lse) lse[row] = l;
    const int lab = labels[row];
    if (lab >= 0) (void)OPK_IDX_OK(lab, V);
    nll[row] = (lab >= 0 && lab < V) ? l - cap(load_logit<FP32>(logits, base + lab), scale, softcap) : 0.f;
  }
}

template <bool FP32, bool NARROW>
__global__ void __launch_bounds__(NT) ce_bwd_kernel(const void* __restrict__ logits, const int* __restrict__ labels,
                                                    const float* __restrict__ lse, const float* __restrict__ coef,
                                                    void* __restrict__ dlogits, int V, long long ld, float scale,
                                                    float softcap) {
  constexpr int VW = kVec16<FP32>;
  const long long row = blockIdx.x;
  const long long base = row * ld;
  const int lab = labels[row];
  const float l = lse[row], c = lab < 0 ? 0.f : coef[row];
  auto grad = [&](float logit, int i) {
    const float raw = logit * scale;
    float z = raw, dz = scale;
    if (softcap > 0.f) {
      const float th = tanhf(raw / softcap);
      z = softcap * th;
      dz = scale * (1.f - th * th);
    }
    return (__expf(z - l) - (i == lab ? 1.f : 0.f)) * c * dz;
  };
  auto put = [&](int i) {
    const float g = grad(load_logit<FP32>(logits, base + i), i);
    if (FP32) reinterpret_cast<float*>(dlogits)[base + i] = g;
    else reinterpret_cast<__nv_bfloat16*>(dlogits)[base + i] = __float2bfloat16(g);
  };
  const int head = ce_head<FP32>(logits, base, V);
  // vectors need both rows on the same 16-byte phase
  const bool vec = ((reinterpret_cast<uintptr_t>(logits) ^ reinterpret_cast<uintptr_t>(dlogits)) & 15) == 0;
  if (NARROW || !vec) {
    for (int i = threadIdx.x; i < V; i += NT) put(i);
    return;
  }
  const int nvec = (V - head) / VW, tail = head + nvec * VW;
  if ((int)threadIdx.x < head) put(threadIdx.x);
  if (tail + (int)threadIdx.x < V) put(tail + threadIdx.x);
  auto store = [&](float (&z)[8], int i) {
#pragma unroll
    for (int j = 0; j < VW; ++j) z[j] = grad(z[j], i + j);
    if (FP32) {
      __stcs(reinterpret_cast<float4*>(reinterpret_cast<float*>(dlogits) + base + i), make_float4(z[0], z[1], z[2], z[3]));
    } else {
      const bf16x8 o = pack8(z);
      __stcs(reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(dlogits) + base + i), *reinterpret_cast<const uint4*>(&o));
    }
  };
  constexpr int U = kRowLoads<FP32>;
  int v = threadIdx.x;
  for (; v + (U - 1) * NT < nvec; v += U * NT) {
    float z[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u) load_vec16<FP32>(logits, base + head + (long long)(v + u * NT) * VW, z[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) store(z[u], head + (v + u * NT) * VW);
  }
  for (; v < nvec; v += NT) {
    float z[8];
    load_vec16<FP32>(logits, base + head + (long long)v * VW, z);
    store(z, head + v * VW);
  }
}

// rows of an fp32 [R][D] matrix (the first widths[r] columns of each, all D without widths) -> bf16 at dst_base +
// offsets[r]; sumsq += sum(bf16(v)^2)
__global__ void __launch_bounds__(NT) scatter_rows_cast_sumsq_kernel(const float* __restrict__ src,
                                                                     __nv_bfloat16* __restrict__ dst_base,
                                                                     const long long* __restrict__ offsets,
                                                                     const int* __restrict__ widths, int D, double* sumsq,
                                                                     long long dst_stride) {
  __shared__ float sh[32];
  const long long r = blockIdx.x;
  const float* s = src + ((long long)blockIdx.y * gridDim.x + r) * D;         // gridDim.y examples
  __nv_bfloat16* d = dst_base + blockIdx.y * dst_stride + offsets[r];
  const int n = widths ? widths[r] : D;
  float part = 0.f;
  for (int i = threadIdx.x; i < n; i += NT) {
    const __nv_bfloat16 b = __float2bfloat16(s[i]);
    d[i] = b;
    const float f = __bfloat162float(b);
    part += f * f;
  }
  const float tot = block_sum<NT>(part, sh);
  if (threadIdx.x == 0 && sumsq) atomicAdd(sumsq + blockIdx.y, (double)tot);
}

// out[n] (+)= sum_t dy[t][n]  (bias gradient)
__global__ void colsum_kernel(const __nv_bfloat16* __restrict__ dy, float* __restrict__ out, int T, int N, long long ld,
                              long long out_stride) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const long long first = (long long)blockIdx.z * T;        // gridDim.z examples of T rows
  float a = 0.f;
  for (int t = blockIdx.y; t < T; t += gridDim.y) a += __bfloat162float(dy[(first + t) * ld + n]);
  atomicAdd(&out[blockIdx.z * out_stride + n], a);
}

// The same for a 16-byte aligned matrix whose width is a multiple of 8: a warp reads 256 columns of a row at a time, the
// eight warps of a CTA take every eighth row of the CTA's row chunk and meet in shared memory, one vector reduction per
// four columns and CTA. (2-byte loads and one atomic per column and row chunk measured 9.2 us on average over the
// GPT-2-small bias gradients, 1024 x 768 .. 3072.)
//
// What bounds it: the loads in flight of one CTA per SM. The compiler spread four unrolled loads over 32 registers, and fewer were in
// flight as soon as the address had one more term; eight are asked for before the first is added (us, with one example: four unrolled
// without that term -> with it -> eight ahead: 4007 x 6712 28.6 -> 37.3 -> 12.8, 2048 x 4096 9.7 -> 12.6 -> 5.8, 1024 x 3072 3.2 -> 3.5 -> 2.6,
// 1024 x 768 2.2 each).
__device__ __forceinline__ bf16x8 ld_vec(const bf16x8* p) {
  uint4 q;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w) : "l"(p));
  return *reinterpret_cast<const bf16x8*>(&q);
}
__global__ void __launch_bounds__(256, 4) colsum_vec_kernel(const __nv_bfloat16* __restrict__ dy, float* __restrict__ out, int T, int N,
                                                            long long ld, int rows_per_cta, long long out_stride) {
  opk::pdl_trigger();
  const long long first = (long long)blockIdx.z * T;
  __shared__ float sh[8][256 + 4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = blockIdx.x * 256, c = c0 + lane * 8;
  const int t0 = blockIdx.y * rows_per_cta, t1 = min(T, t0 + rows_per_cta);
  float a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = 0.f;
  if (c < N) {
    const bf16x8* src = reinterpret_cast<const bf16x8*>(dy + (first + t0 + warp) * ld + c);        // `ld` vectors are eight rows
    int t = t0 + warp;
    for (; t + 56 < t1; t += 64, src += 8 * ld) {
      bf16x8 r[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) r[u] = ld_vec(src + u * ld);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        float f[8];
        unpack8(r[u], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] += f[j];
      }
    }
    for (; t < t1; t += 8, src += ld) {
      float f[8];
      unpack8(*src, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += f[j];
    }
  }
  *reinterpret_cast<float4*>(&sh[warp][lane * 8]) = make_float4(a[0], a[1], a[2], a[3]);
  *reinterpret_cast<float4*>(&sh[warp][lane * 8 + 4]) = make_float4(a[4], a[5], a[6], a[7]);
  __syncthreads();
  if (threadIdx.x < 64 && c0 + (int)threadIdx.x * 4 < N) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] += sh[k][threadIdx.x * 4 + j];
    red_add_v4(out + blockIdx.z * out_stride + c0 + threadIdx.x * 4, v);
  }
}

// tied embeddings: dense[tok[t]] += gc[t] for representative rows (no two representatives share a row)
__global__ void emb_add_rows_kernel(const int* __restrict__ tok, const int* __restrict__ rep,
                                    const float* __restrict__ gc, __nv_bfloat16* __restrict__ dense, int T, int D,
                                    long long dense_stride) {
  const long long t = blockIdx.x, first = (long long)blockIdx.y * T;
  if (rep[first + t] != (int)t) return;
  const float* src = gc + (first + t) * D;
  __nv_bfloat16* dst = dense + blockIdx.y * dense_stride + (long long)tok[first + t] * D;
  for (int d = threadIdx.x; d < D; d += blockDim.x) dst[d] = __float2bfloat16(__bfloat162float(dst[d]) + src[d]);
}

inline int grid_for(long long n, int block, int cap_blocks = 148 * 16) {
  long long g = (n + block - 1) / block;
  if (g > cap_blocks) g = cap_blocks;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)
#define BF(p) reinterpret_cast<const __nv_bfloat16*>(p)
#define BFM(p) reinterpret_cast<__nv_bfloat16*>(p)

template <bool FP32, bool ROUND>
void launch_sumsq(int ctas, int batch, cudaStream_t st, const void* x, long long n, double* sums, long long stride) {
  if (batch == 1) sumsq_kernel<FP32, ROUND, false><<<ctas, NT, 0, st>>>(x, n, sums, 0);
  else sumsq_kernel<FP32, ROUND, true><<<dim3(ctas, batch), NT, 0, st>>>(x, n, sums, stride);
}

template <bool COPY>
void launch_rmsnorm_fwd(cudaStream_t st, const __nv_bfloat16* x, const __nv_bfloat16* w, __nv_bfloat16* y, float* rstd, int T, int D, float eps,
                        float w_offset, long long ldx, long long ldy, __nv_bfloat16* copy, long long ld_copy) {
  const int warp_grid = (T + 7) / 8;
  if (D == 4096) rmsnorm_fwd_warp_kernel<16, COPY><<<warp_grid, 256, 0, st>>>(x, w, y, rstd, T, eps, w_offset, ldx, ldy, copy, ld_copy);
  else if (D == 2048) rmsnorm_fwd_warp_kernel<8, COPY><<<warp_grid, 256, 0, st>>>(x, w, y, rstd, T, eps, w_offset, ldx, ldy, copy, ld_copy);
  else if (D == 1024) rmsnorm_fwd_warp_kernel<4, COPY><<<warp_grid, 256, 0, st>>>(x, w, y, rstd, T, eps, w_offset, ldx, ldy, copy, ld_copy);
  else rmsnorm_fwd_kernel<false, COPY><<<T, NT, 0, st>>>(x, nullptr, w, copy, y, rstd, D, eps, w_offset, ldx, ldy, ld_copy);
}
extern "C" int opk_rmsnorm_fwd_ld(const void* x, int64_t ldx, const void* w, void* y, int64_t ldy, float* rstd, int T, int D,
                                  float eps, float w_offset, void* copy, int64_t ld_copy, void* stream) {
  if (T <= 0) return 0;
  if (D % 8 || ldx % 8 || ldy % 8 || ldx < D || ldy < D) return -1;
  if (copy && (ld_copy % 8 || ld_copy < D || (reinterpret_cast<uintptr_t>(copy) & 15))) return -1;
  if (copy) launch_rmsnorm_fwd<true>(ST(stream), BF(x), BF(w), BFM(y), rstd, T, D, eps, w_offset, ldx, ldy, BFM(copy), ld_copy);
  else launch_rmsnorm_fwd<false>(ST(stream), BF(x), BF(w), BFM(y), rstd, T, D, eps, w_offset, ldx, ldy, nullptr, 0);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int T, int D, float eps,
                               float w_offset, void* stream) {
  return opk_rmsnorm_fwd_ld(x, D, w, y, D, rstd, T, D, eps, w_offset, nullptr, 0, stream);
}
extern "C" int opk_add_rmsnorm_fwd(const void* x, const void* r, const void* w, void* sum_out, void* y, float* rstd,
                                   int T, int D, float eps, float w_offset, void* stream) {
  if (T <= 0) return 0;
  if (D % 8) return -1;
  if (D <= 2048)
    add_rmsnorm_fwd_kernel<1><<<T, NT, 0, ST(stream)>>>(BF(x), BF(r), BF(w), BFM(sum_out), BFM(y), rstd, D, eps, w_offset);
  else if (D <= 4096)
    add_rmsnorm_fwd_kernel<2><<<T, NT, 0, ST(stream)>>>(BF(x), BF(r), BF(w), BFM(sum_out), BFM(y), rstd, D, eps, w_offset);
  else if (D <= 8192)
    add_rmsnorm_fwd_kernel<4><<<T, NT, 0, ST(stream)>>>(BF(x), BF(r), BF(w), BFM(sum_out), BFM(y), rstd, D, eps, w_offset);
  else
    rmsnorm_fwd_kernel<true, false><<<T, NT, 0, ST(stream)>>>(BF(x), BF(r), BF(w), BFM(sum_out), BFM(y), rstd, D, eps, w_offset, D, D, D);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_rmsnorm_bwd_ld(const void* dy, int64_t ld_dy, const void* x, int64_t ldx, const void* w, const float* rstd,
                                  const void* dres, void* dx_out, int64_t ld_dx, float* dw, float* workspace, int ws_rows,
                                  int T, int D, float w_offset, int batch, int64_t dw_stride, void* stream) {
  if (T <= 0 || batch <= 0) return 0;
  if (batch > 65535) return -1;
  if (D % 8 || D > 3 * RMS_BWD_NT * 8) return -1;
  if (ld_dy % 8 || ldx % 8 || ld_dx % 8 || ld_dy < D || ldx < D || ld_dx < D) return -1;
  if (dw && (!workspace || ws_rows < batch)) return -1;
  int ctas = T < 148 * 2 ? T : 148 * 2;
  if (dw && ctas > ws_rows / batch) ctas = ws_rows / batch;
  const dim3 grid((unsigned)ctas, (unsigned)batch);
  float* part = dw ? workspace : nullptr;
  const int iters = (D / 8 + RMS_BWD_NT - 1) / RMS_BWD_NT;
#define OPK_RMS_BWD(I)                                                                                                                 \
  do {                                                                                                                                 \
    if (batch == 1)                                                                                                                    \
      rmsnorm_bwd_kernel<I, false><<<grid, RMS_BWD_NT, 0, ST(stream)>>>(BF(dy), BF(x), BF(w), rstd, BF(dres), BFM(dx_out), part, T, D, \
                                                                        w_offset, ld_dy, ldx, ld_dx);                                  \
    else                                                                                                                               \
      rmsnorm_bwd_kernel<I, true><<<grid, RMS_BWD_NT, 0, ST(stream)>>>(BF(dy), BF(x), BF(w), rstd, BF(dres), BFM(dx_out), part, T, D,  \
                                                                       w_offset, ld_dy, ldx, ld_dx);                                   \
  } while (0)
  if (iters == 1)
    OPK_RMS_BWD(1);
  else if (iters == 2)
    OPK_RMS_BWD(2);
  else
    OPK_RMS_BWD(3);
#undef OPK_RMS_BWD
  OPK_LAUNCH_CHECK();
  if (dw) {
    if (batch == 1) colsum_add_kernel<false><<<(D + 31) / 32, 256, 0, ST(stream)>>>(part, dw, ctas, D, 0);
    else colsum_add_kernel<true><<<dim3((D + 31) / 32, batch), 256, 0, ST(stream)>>>(part, dw, ctas, D, dw_stride);
    OPK_LAUNCH_CHECK();
  }
  return 0;
}
extern "C" int opk_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                               void* dx_out, float* dw, float* workspace, int ws_rows, int T, int D, float w_offset,
                               void* stream) {
  return opk_rmsnorm_bwd_ld(dy, D, x, D, w, rstd, dres, dx_out, D, dw, workspace, ws_rows, T, D, w_offset, 1, 0, stream);
}
extern "C" int opk_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, int T,
                                 int D, float eps, void* stream) {
  if (T <= 0) return 0;
  if (D % 8) return -1;
  layernorm_fwd_kernel<<<T, NT, 0, ST(stream)>>>(BF(x), BF(w), BF(b), BFM(y), mean, rstd, D, eps);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_layernorm_bwd(const void* dy, const void* x, const void* w, const float* mean, const float* rstd,
                                 const void* dres, void* dx_out, float* dw, float* db, int T, int D, int batch, int64_t stride,
                                 void* stream) {
  if (T <= 0 || batch <= 0) return 0;
  if (D % 8 || D > MAX_COL_ITERS * NT * 8 || batch > 65535) return -1;
  if (D <= 1024 && (batch == 1 || stride % 4 == 0) && (reinterpret_cast<uintptr_t>(dw) & 15) == 0 && (reinterpret_cast<uintptr_t>(db) & 15) == 0) {
    const int g = (T + 7) / 8 < 148 ? (T + 7) / 8 : 148;
#define OPK_LN_BWD(V)                                                                                                                  \
  do {                                                                                                                                 \
    if (batch == 1)                                                                                                                    \
      layernorm_bwd_warp_kernel<V, false><<<g, 256, 0, ST(stream)>>>(BF(dy), BF(x), BF(w), mean, rstd, BF(dres), BFM(dx_out), dw, db,  \
                                                                     T, D, 0);                                                         \
    else                                                                                                                               \
      layernorm_bwd_warp_kernel<V, true><<<dim3(g, batch), 256, 0, ST(stream)>>>(BF(dy), BF(x), BF(w), mean, rstd, BF(dres),           \
                                                                                 BFM(dx_out), dw, db, T, D, stride);                   \
  } while (0)
    if (D <= 256) OPK_LN_BWD(1);
    else if (D <= 512) OPK_LN_BWD(2);
    else if (D <= 768) OPK_LN_BWD(3);
    else OPK_LN_BWD(4);
#undef OPK_LN_BWD
    OPK_LAUNCH_CHECK();
    return 0;
  }
  const dim3 grid(T < 148 * 2 ? T : 148 * 2, batch);
  if (batch == 1) layernorm_bwd_kernel<false><<<grid, NT, 0, ST(stream)>>>(BF(dy), BF(x), BF(w), mean, rstd, BF(dres), BFM(dx_out), dw, db, T, D, 0);
  else layernorm_bwd_kernel<true><<<grid, NT, 0, ST(stream)>>>(BF(dy), BF(x), BF(w), mean, rstd, BF(dres), BFM(dx_out), dw, db, T, D, stride);
  OPK_LAUNCH_CHECK();
  return 0;
}
// period > 0: row t sits at position t % period (sequences of `period` rows one after the other).
extern "C" int opk_rope(void* qk, const float* cs, const int32_t* pos, int period, int64_t T, int n_rot_heads, int head_dim,
                              int64_t ld, float sign, void* stream) {
  const long long n = (long long)T * n_rot_heads * (head_dim / 2);
  if (n <= 0) return 0;
  if (period < 0) return -1;
  if ((head_dim % 16) == 0 && (ld % 8) == 0 && (reinterpret_cast<uintptr_t>(qk) & 15) == 0 &&
      (reinterpret_cast<uintptr_t>(cs) & 15) == 0)
    rope_vec8_kernel<<<grid_for(n / 8, 256), 256, 0, ST(stream)>>>(BFM(qk), cs, pos, period, T, n_rot_heads, head_dim, ld, sign);
  else
    rope_kernel<<<grid_for(n, 256), 256, 0, ST(stream)>>>(BFM(qk), cs, pos, period, T, n_rot_heads, head_dim, ld, sign);
  OPK_LAUNCH_CHECK();
  return 0;
}
namespace {
bool aligned16(const void* a, const void* b, const void* c = nullptr, const void* d = nullptr, const void* e = nullptr) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(d) |
           reinterpret_cast<uintptr_t>(e)) & 15) == 0;
}
bool aligned4(const void* a, const void* b) { return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 3) == 0; }
// Interleaved pairs: eight elements per thread where that is the faster form, one otherwise. Forward, small calls are bound by the
// latency of one thread's eight activations (40 x 1024 pairs: 2.3 us in vectors, 1.7 one by one; 2048 x 256 2.7 and 3.5).
// Backward, vectors pay only where the call is bound by HBM and the activation is cheap: SwiGLU 2048 x 2048 13.7 us in vectors and
// 9.4 one by one, 16384 x 2048 80 and 87; GEGLU 16384 x 8192 401 and 274.
constexpr long long kGluFwdVec = 1ll << 17, kGluBwdVec = 12ll << 20;
template <int MODE>
int glu_fwd(const void* gu, void* act, long long n, cudaStream_t st) {
  if (n <= 0) return 0;
  const long long nvec = n > kGluFwdVec && aligned16(gu, act) ? n >> 3 : 0, rest = n - nvec * 8;
  if (nvec) glu_fwd_kernel<MODE, false><<<grid_for(nvec, 256), 256, 0, st>>>(BF(gu), nullptr, BFM(act), nvec);
  if (rest && aligned4(gu, nullptr)) glu_fwd_pair_kernel<MODE, true><<<grid_for(rest, 256), 256, 0, st>>>(BF(gu), BFM(act), nvec * 8, n);
  else if (rest) glu_fwd_pair_kernel<MODE, false><<<grid_for(rest, 256), 256, 0, st>>>(BF(gu), BFM(act), nvec * 8, n);
  OPK_LAUNCH_CHECK();
  return 0;
}
template <int MODE>
int glu_bwd(const void* dact, const void* gu, void* dgu, long long n, cudaStream_t st) {
  if (n <= 0) return 0;
  long long nvec = 0;
  if constexpr (MODE == 0) {
    nvec = n > kGluBwdVec && aligned16(dact, gu, dgu) ? n >> 3 : 0;
    if (nvec) glu_bwd_kernel<0, false><<<grid_for(nvec, 256), 256, 0, st>>>(BF(dact), BF(gu), nullptr, BFM(dgu), nullptr, nvec);
  }
  const long long rest = n - nvec * 8;
  if (rest && aligned4(gu, dgu)) glu_bwd_pair_kernel<MODE, true><<<grid_for(rest, 256), 256, 0, st>>>(BF(dact), BF(gu), BFM(dgu), nvec * 8, n);
  else if (rest) glu_bwd_pair_kernel<MODE, false><<<grid_for(rest, 256), 256, 0, st>>>(BF(dact), BF(gu), BFM(dgu), nvec * 8, n);
  OPK_LAUNCH_CHECK();
  return 0;
}
}  // namespace
extern "C" int opk_swiglu_fwd(const void* gu, void* act, int T, int F, void* stream) {
  return glu_fwd<0>(gu, act, (long long)T * F, ST(stream));
}
extern "C" int opk_swiglu_bwd(const void* dact, const void* gu, void* dgu, int T, int F, void* stream) {
  return glu_bwd<0>(dact, gu, dgu, (long long)T * F, ST(stream));
}
extern "C" int opk_geglu_fwd(const void* gu, void* act, int T, int F, int approx, void* stream) {
  return approx ? glu_fwd<2>(gu, act, (long long)T * F, ST(stream)) : glu_fwd<1>(gu, act, (long long)T * F, ST(stream));
}
extern "C" int opk_geglu_bwd(const void* dact, const void* gu, void* dgu, int T, int F, int approx, void* stream) {
  return approx ? glu_bwd<2>(dact, gu, dgu, (long long)T * F, ST(stream)) : glu_bwd<1>(dact, gu, dgu, (long long)T * F, ST(stream));
}
// Gate and up in separate buffers of n elements; kind 0 = SwiGLU, 1 = GEGLU (erf), 2 = GEGLU (tanh), 3 and 4 = 0 and 2 rounded
// operation by operation. n a multiple of 8, every buffer 16-byte aligned.
extern "C" int opk_glu_split_fwd(const void* gate, const void* up, void* act, int64_t n, int kind, void* stream) {
  if (n <= 0) return 0;
  if (n % 8 || kind < 0 || kind > 4 || !aligned16(gate, up, act)) return -1;
  const int g = grid_for(n >> 3, 256);
  if (kind == 0) glu_fwd_kernel<0, true><<<g, 256, 0, ST(stream)>>>(BF(gate), BF(up), BFM(act), n >> 3);
  else if (kind == 1) glu_fwd_kernel<1, true><<<g, 256, 0, ST(stream)>>>(BF(gate), BF(up), BFM(act), n >> 3);
  else if (kind == 3) glu_fwd_kernel<3, true><<<g, 256, 0, ST(stream)>>>(BF(gate), BF(up), BFM(act), n >> 3);
  else if (kind == 4) glu_fwd_kernel<4, true><<<g, 256, 0, ST(stream)>>>(BF(gate), BF(up), BFM(act), n >> 3);
  else glu_fwd_kernel<2, true><<<g, 256, 0, ST(stream)>>>(BF(gate), BF(up), BFM(act), n >> 3);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_glu_split_bwd(const void* dact, const void* gate, const void* up, void* dgate, void* dup, int64_t n, int kind,
                                 void* stream) {
  if (n <= 0) return 0;
  if (n % 8 || kind < 0 || kind > 4 || !aligned16(dact, gate, up, dgate, dup)) return -1;
  const int g = grid_for(n >> 3, 256);
  if (kind == 0) glu_bwd_kernel<0, true><<<g, 256, 0, ST(stream)>>>(BF(dact), BF(gate), BF(up), BFM(dgate), BFM(dup), n >> 3);
  else if (kind == 1) glu_bwd_kernel<1, true><<<g, 256, 0, ST(stream)>>>(BF(dact), BF(gate), BF(up), BFM(dgate), BFM(dup), n >> 3);
  else if (kind == 3) glu_bwd_kernel<3, true><<<g, 256, 0, ST(stream)>>>(BF(dact), BF(gate), BF(up), BFM(dgate), BFM(dup), n >> 3);
  else if (kind == 4) glu_bwd_kernel<4, true><<<g, 256, 0, ST(stream)>>>(BF(dact), BF(gate), BF(up), BFM(dgate), BFM(dup), n >> 3);
  else glu_bwd_kernel<2, true><<<g, 256, 0, ST(stream)>>>(BF(dact), BF(gate), BF(up), BFM(dgate), BFM(dup), n >> 3);
  OPK_LAUNCH_CHECK();
  return 0;
}
// Smaller calls go element by element (40 x 1024 backward: 2.1 us in vectors, 1.7 one by one; 2048 x 64: 2.1 and 2.2).
constexpr long long kGeluVec = 1ll << 17;
extern "C" int opk_gelu_fwd(const void* x, void* y, int64_t n, void* stream) {
  if (n <= 0) return 0;
  const long long nvec = n >= kGeluVec && aligned16(x, y) ? n >> 3 : 0;
  gelu_fwd_kernel<<<grid_for(nvec ? nvec : n, 256), 256, 0, ST(stream)>>>(BF(x), BFM(y), nvec, n);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_gelu_bwd(const void* dy, const void* x, void* dx, int64_t n, void* stream) {
  if (n <= 0) return 0;
  const long long nvec = n >= kGeluVec && aligned16(dy, x, dx) ? n >> 3 : 0;
  gelu_bwd_kernel<<<grid_for(nvec ? nvec : n, 256), 256, 0, ST(stream)>>>(BF(dy), BF(x), BFM(dx), nvec, n);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_embedding_fwd(const int32_t* tok, const void* table, const void* pos_table, void* out, int T, int D,
                                 int vocab, int period, void* stream) {
  if (T <= 0) return 0;
  if (D % 8 || vocab <= 0) return -1;
  if (period > 0 && pos_table) embedding_fwd_kernel<true><<<T, 128, 0, ST(stream)>>>(tok, BF(table), BF(pos_table), BFM(out), D, vocab, period);
  else embedding_fwd_kernel<false><<<T, 128, 0, ST(stream)>>>(tok, BF(table), BF(pos_table), BFM(out), D, vocab, 0);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_embedding_bwd_compact(const int32_t* tok, const void* dx, int32_t* first_pos, int32_t* rep,
                                         float* gc, double* sumsq, int T, int D, int vocab, int batch, void* stream) {
  if (T <= 0 || batch <= 0) return 0;
  if (vocab <= 0 || batch > 65535) return -1;
  cudaStream_t st = ST(stream);
  cudaError_t e = cudaMemsetAsync(gc, 0, sizeof(float) * (size_t)batch * T * D, st);
  if (e != cudaSuccess) return (int)e;
  const dim3 by_token((T + 255) / 256, batch);
  emb_first_pos_kernel<<<by_token, 256, 0, st>>>(tok, first_pos, T, vocab);
  emb_scatter_kernel<<<dim3(T, batch), 256, 0, st>>>(tok, BF(dx), first_pos, rep, gc, T, D, vocab);
  emb_reset_kernel<<<by_token, 256, 0, st>>>(tok, first_pos, T, vocab);
  const long long n = (long long)T * D;
  if (sumsq) launch_sumsq<true, true>(grid_for(n, NT, 148 * 4), batch, st, gc, n, sumsq, n);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_embedding_accumulate(const int32_t* tok, const int32_t* rep, const float* gc, const float* scale,
                                        float* acc, int T, int D, void* stream) {
  if (T <= 0) return 0;
  emb_accumulate_kernel<false><<<T, 256, 0, ST(stream)>>>(tok, rep, gc, scale, acc, D);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_embedding_accumulate_shared(const int32_t* tok, const int32_t* rep, const float* gc, const float* scale,
                                               float* acc, int T, int D, void* stream) {
  if (T <= 0) return 0;
  emb_accumulate_kernel<true><<<T, 256, 0, ST(stream)>>>(tok, rep, gc, scale, acc, D);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_lce_finalize(const float* pmax, const float* psum, const float* tgt, const int32_t* labels,
                                float* lse, float* nll, int T, int tiles, void* stream) {
  if (T <= 0) return 0;
  lce_finalize_kernel<<<(T + 7) / 8, 256, 0, ST(stream)>>>(pmax, psum, tgt, labels, lse, nll, T, tiles);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_rmsnorm_dw_per_example(const void* dy, const void* x, const float* rstd, float* dw, int B, int rows, int D,
                                          void* stream) {
  if (B <= 0 || rows <= 0 || D <= 0) return 0;
  if (B > 65535) return -1;
  int z = (rows + 63) / 64;
  if (z > 32) z = 32;
  dim3 grid((D + 255) / 256, B, z);
  rmsnorm_dw_per_example_kernel<<<grid, 256, 0, ST(stream)>>>(BF(dy), BF(x), rstd, dw, rows, D);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_loss_coef(const int32_t* labels, const float* nll, const float* weight, float* coef, float* loss, float* ntok,
                             int T, int batch, void* stream) {
  if (T <= 0 || batch <= 0 || !labels || !nll || !coef || !loss) return -1;
  loss_coef_kernel<<<batch, 1024, 0, ST(stream)>>>(labels, nll, weight, coef, loss, ntok, T);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_cross_entropy_fwd(const void* logits, int is_fp32, const int32_t* labels, float* nll, float* lse,
                                     int T, int V, int64_t ld, float scale, float softcap, void* stream) {
  if (T <= 0) return 0;
#define OPK_CE_FWD(F, N) ce_fwd_kernel<F, N><<<T, NT, 0, ST(stream)>>>(logits, labels, nll, lse, V, ld, scale, softcap)
  if (V <= kNarrowRow) { if (is_fp32) OPK_CE_FWD(true, true); else OPK_CE_FWD(false, true); }
  else { if (is_fp32) OPK_CE_FWD(true, false); else OPK_CE_FWD(false, false); }
#undef OPK_CE_FWD
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_cross_entropy_bwd(const void* logits, int is_fp32, const int32_t* labels, const float* lse,
                                     const float* coef, void* dlogits, int T, int V, int64_t ld, float scale,
                                     float softcap, void* stream) {
  if (T <= 0) return 0;
#define OPK_CE_BWD(F, N) ce_bwd_kernel<F, N><<<T, NT, 0, ST(stream)>>>(logits, labels, lse, coef, dlogits, V, ld, scale, softcap)
  if (V <= kNarrowRow) { if (is_fp32) OPK_CE_BWD(true, true); else OPK_CE_BWD(false, true); }
  else { if (is_fp32) OPK_CE_BWD(true, false); else OPK_CE_BWD(false, false); }
#undef OPK_CE_BWD
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_sumsq(const void* x, int is_fp32, int round_bf16, int64_t n, double* sumsq, int batch, int64_t stride, void* stream) {
  if (n <= 0 || batch <= 0) return 0;
  // the 16-byte form is chosen by the base, so every buffer of a batch has to lie on the same boundary
  if (batch > 65535 || (batch > 1 && stride % 8)) return -1;
  const int g = grid_for(n, NT, 148 * 8);
  if (is_fp32) {
    if (round_bf16) launch_sumsq<true, true>(g, batch, ST(stream), x, n, sumsq, stride);
    else launch_sumsq<true, false>(g, batch, ST(stream), x, n, sumsq, stride);
  } else {
    launch_sumsq<false, false>(g, batch, ST(stream), x, n, sumsq, stride);
  }
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_scatter_rows_cast_sumsq(const float* src, void* dst_base, const int64_t* offsets, const int32_t* widths, int R,
                                                  int D, double* sumsq, int batch, int64_t dst_stride, void* stream) {
  if (R <= 0 || batch <= 0) return 0;
  if (batch > 65535) return -1;
  scatter_rows_cast_sumsq_kernel<<<dim3(R, batch), NT, 0, ST(stream)>>>(src, BFM(dst_base), reinterpret_cast<const long long*>(offsets), widths, D, sumsq, dst_stride);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_colsum(const void* dy, float* out, int T, int N, int64_t ld, int batch, int64_t out_stride, void* stream) {
  if (T <= 0 || N <= 0 || batch <= 0) return 0;
  if (batch > 65535) return -1;
  if (N % 8 == 0 && ld % 8 == 0 && aligned16(dy, out) && (batch == 1 || out_stride % 4 == 0)) {
    // about one CTA per SM over all column blocks, at least 8 rows (one per warp) each
    const int cols = (N + 255) / 256;
    int rows = (int)(((long long)T * cols + 147) / 148);
    rows = rows < 8 ? 8 : (rows + 7) / 8 * 8;
    colsum_vec_kernel<<<dim3(cols, (T + rows - 1) / rows, batch), 256, 0, ST(stream)>>>(BF(dy), out, T, N, ld, rows, out_stride);
    OPK_LAUNCH_CHECK();
    return 0;
  }
  dim3 grid((N + 127) / 128, T < 32 ? T : 32, batch);
  colsum_kernel<<<grid, 128, 0, ST(stream)>>>(BF(dy), out, T, N, ld, out_stride);
  OPK_LAUNCH_CHECK();
  return 0;
}
extern "C" int opk_embedding_add_rows(const int32_t* tok, const int32_t* rep, const float* gc, void* dense, int T, int D,
                                      int batch, int64_t dense_stride, void* stream) {
  if (T <= 0 || batch <= 0) return 0;
  if (batch > 65535) return -1;
  emb_add_rows_kernel<<<dim3(T, batch), 256, 0, ST(stream)>>>(tok, rep, gc, BFM(dense), T, D, dense_stride);
  OPK_LAUNCH_CHECK();
  return 0;
}

// ---------------------------------------------------------------------------------------------------------------------
// Allocation-free variant of the compact embedding gradient (declared in opk_noalloc.h).
// The scratch table is a file-scope device array; host code must not pass its name to a kernel (on the host the name
// is only a stand-in), so the device address is resolved once per device with cudaGetSymbolAddress.
#include "opk_noalloc.h"

namespace {
static __device__ __align__(256) int g_noalloc_first_pos[OPK_NOALLOC_MAX_VOCAB];

__global__ void noalloc_fill_kernel(int* __restrict__ p, int n, int value) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = value;
}

constexpr int kMaxDevices = 64;
int* g_noalloc_ptr[kMaxDevices] = {nullptr};
}  // namespace

extern "C" int opk_embedding_bwd_compact_noalloc(const int32_t* tok, const void* dx, int32_t* rep, float* gc,
                                                 double* sumsq, int T, int D, int vocab, void* stream) {
  if (T < 0 || D <= 0 || vocab <= 0 || !tok || !dx || !rep || !gc) return -1;
  if (vocab > OPK_NOALLOC_MAX_VOCAB) return -2;
  if (T == 0) return 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return -1;
  cudaStream_t st = ST(stream);
  if (g_noalloc_ptr[dev] == nullptr) {
    // one-time set-up for this device: resolve the device address and put every entry into the idle state
    int* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_first_pos);
    if (e != cudaSuccess) return (int)e;
    noalloc_fill_kernel<<<256, 256, 0, st>>>(p, OPK_NOALLOC_MAX_VOCAB, INT_MAX);
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    g_noalloc_ptr[dev] = p;
  }
  int* first_pos = g_noalloc_ptr[dev];
  e = cudaMemsetAsync(gc, 0, sizeof(float) * (size_t)T * D, st);
  if (e != cudaSuccess) return (int)e;
  // entries touched by this call are forced to the idle value first: the table keeps whatever the previous call
  // (possibly one that was interrupted) left behind
  emb_reset_kernel<<<(T + 255) / 256, 256, 0, st>>>(tok, first_pos, T, vocab);
  emb_first_pos_kernel<<<(T + 255) / 256, 256, 0, st>>>(tok, first_pos, T, vocab);
  emb_scatter_kernel<<<T, 256, 0, st>>>(tok, BF(dx), first_pos, rep, gc, T, D, vocab);
  emb_reset_kernel<<<(T + 255) / 256, 256, 0, st>>>(tok, first_pos, T, vocab);
  if (sumsq) launch_sumsq<true, true>(grid_for((long long)T * D, NT, 148 * 4), 1, st, gc, (long long)T * D, sumsq, 0);
  OPK_LAUNCH_CHECK();
  return 0;
}
