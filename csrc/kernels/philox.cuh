// Counter-based Gaussian noise: Philox4x32-10 and the Box-Muller transform, shared by the fused optimizer step and the
// multi-tensor kernels of the functional API. Element e of the flattened parameters uses counter e / 4.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace opk {

struct U4 { uint32_t x, y, z, w; };
// The keys of the ten rounds. A kernel that draws in its inner loop takes them as an argument: as operands from the constant bank
// they cost nothing, computed from the seed two additions per round.
struct PhiloxKeys { uint32_t k0[10], k1[10]; };
__host__ __device__ __forceinline__ PhiloxKeys philox_keys(uint64_t seed) {
  PhiloxKeys k;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    k.k0[r] = (uint32_t)seed + (uint32_t)r * 0x9E3779B9u;
    k.k1[r] = (uint32_t)(seed >> 32) + (uint32_t)r * 0xBB67AE85u;
  }
  return k;
}
__host__ __device__ __forceinline__ U4 philox4x32_10(U4 c, const PhiloxKeys& key) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = (uint64_t)M0 * c.x, p1 = (uint64_t)M1 * c.z;
    U4 n;
    n.x = (uint32_t)(p1 >> 32) ^ c.y ^ key.k0[r];
    n.y = (uint32_t)p1;
    n.z = (uint32_t)(p0 >> 32) ^ c.w ^ key.k1[r];
    n.w = (uint32_t)p0;
    c = n;
  }
  return c;
}
// log2 of a normal number (no code for subnormal ones)
__device__ __forceinline__ float lg2_normal(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Four standard normals for the aligned group of four elements with index q = element / 4.
__device__ __forceinline__ void normal4(uint64_t q, const PhiloxKeys& key, uint32_t stream_id, uint32_t step, float (&z)[4]) {
  const U4 r = philox4x32_10(U4{(uint32_t)q, (uint32_t)(q >> 32), step, stream_id}, key);
  const float k = 2.3283064365386963e-10f;  // 2^-32: scaling by it is exact, so each line below rounds once, as written
  const float u1 = fmaf((float)r.x, k, k), u3 = fmaf((float)r.z, k, k);             // (r + 1) * 2^-32, in (0, 1]
  // hardware lg2 / sin / cos (absolute error about 1e-6 here); the angle is taken in [-pi, pi), where the fast
  // sine and cosine are most accurate, and the half-turn is undone by the sign: sin(t + pi) = -sin t, cos likewise
  const float ra = sqrtf(-1.3862943611198906f * lg2_normal(u1)), rb = sqrtf(-1.3862943611198906f * lg2_normal(u3));   // -2 ln u
  const float two_pi = 6.283185307179586f;
  const float ta = two_pi * fmaf((float)r.y, k, -0.5f), tb = two_pi * fmaf((float)r.w, k, -0.5f);
  z[0] = -ra * __cosf(ta);
  z[1] = -ra * __sinf(ta);
  z[2] = -rb * __cosf(tb);
  z[3] = -rb * __sinf(tb);
}

__device__ __forceinline__ void normal4(uint64_t q, uint64_t seed, uint32_t stream_id, uint32_t step, float (&z)[4]) {
  normal4(q, philox_keys(seed), stream_id, step, z);
}

}  // namespace opk
