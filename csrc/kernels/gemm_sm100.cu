// Host side of the tcgen05 GEMM: builds the TMA tensor maps and launches the persistent kernel.
#include "gemm_narrow_sm100.cuh"
#include "lce_grad.cuh"
#include "opk_api.h"
#include "debug_bounds.cuh"

#include <cudaTypedefs.h>
#include <mutex>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

namespace {

thread_local char g_err[512] = "";
void set_err(const char* msg) { snprintf(g_err, sizeof(g_err), "%s", msg); }

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn get_encode() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(p);
  });
  return fn;
}

// 3-D bf16 map {inner, rows, batch} with a {64, box_rows, 1} box and 128-byte swizzle.
bool make_map(CUtensorMap* m, const void* base, uint64_t inner, uint64_t rows, uint64_t batch, uint64_t ld,
              uint64_t batch_stride, uint32_t box_rows) {
  EncodeFn enc = get_encode();
  if (!enc) { set_err("cuTensorMapEncodeTiled not available"); return false; }
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) { set_err("TMA operand base must be 16-byte aligned"); return false; }
  if ((ld * 2) % 16 != 0) { set_err("TMA operand row pitch must be a multiple of 8 elements"); return false; }
  if (batch > 1 && (batch_stride * 2) % 16 != 0) { set_err("TMA batch stride must be a multiple of 8 elements"); return false; }
  cuuint64_t dims[3] = {inner, rows, batch};
  cuuint64_t bs = batch > 1 ? batch_stride * 2 : rows * ld * 2;
  cuuint64_t strides[2] = {ld * 2, bs};
  cuuint32_t box[3] = {64, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[160];
    snprintf(buf, sizeof(buf), "cuTensorMapEncodeTiled failed (%d): inner=%llu rows=%llu batch=%llu ld=%llu", (int)r,
             (unsigned long long)inner, (unsigned long long)rows, (unsigned long long)batch, (unsigned long long)ld);
    set_err(buf);
    return false;
  }
  return true;
}

int g_num_sms = 0;
int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

template <bool A_MN, bool B_MN, int BN, int EPI>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const opk::GemmParams& p, int max_ctas, cudaStream_t st) {
  using Cfg = opk::GemmCfg<BN>;
  auto kern = opk::gemm_bf16_kernel<A_MN, B_MN, BN, EPI>;
  static bool attr_done = false;
  if (!attr_done) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e != cudaSuccess) { set_err(cudaGetErrorString(e)); return (int)e; }
    attr_done = true;
  }
  const int tiles = ((p.M + 127) / 128) * ((p.N + BN - 1) / BN) * p.batch;
  int grid = max_ctas > 0 ? max_ctas : num_sms();
  if (grid > tiles) grid = tiles;
  cudaError_t e = opk::launch(kern, grid, 64 + 32 * opk::gemm1_epi_warps(EPI), Cfg::SMEM_BYTES, st, ta, tb, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) { set_err(cudaGetErrorString(e)); return (int)e; }
  return 0;
}

// Pair mode: eligible products (256-wide column tiles, no grouped tables, at least 256 rows) run on the two-CTA
// kernel. On by default; opk_gemm_set_pair_mode selects the single-CTA kernel (the tests run both).
int g_pair_mode = 1;
bool pair_mode() { return g_pair_mode == 1; }

template <bool A_MN, bool B_MN, int EPI, int VARIANT = opk::G2_PLAIN>
int launch2(const CUtensorMap& ta, const CUtensorMap& tb, const opk::GemmParams& p, int max_ctas, cudaStream_t st) {
  using Cfg = opk::Gemm2Cfg<opk::gemm2_cols(VARIANT)>;
  auto kern = opk::gemm2_bf16_kernel<A_MN, B_MN, EPI, VARIANT>;
  constexpr int kThreads = 64 + 32 * opk::gemm2_epi_warps(EPI, VARIANT) + (VARIANT == opk::G2_STAGE ? 32 * opk::kStageWarps : 0);
  static bool attr_done = false;
  if (!attr_done) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e != cudaSuccess) { set_err(cudaGetErrorString(e)); return (int)e; }
    attr_done = true;
  }
  const int tiles = ((p.M + 255) / 256) * ((p.N + Cfg::BN - 1) / Cfg::BN) * p.batch;
  int grid = (max_ctas > 0 ? max_ctas : num_sms()) & ~1;   // whole CTA pairs
  if (grid < 2) grid = 2;
  if (grid > 2 * tiles) grid = 2 * tiles;
  cudaError_t e = opk::launch(kern, grid, kThreads, Cfg::SMEM_BYTES, st, ta, tb, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) { set_err(cudaGetErrorString(e)); return (int)e; }
  return 0;
}

template <bool A_MN, bool B_MN, int BN, int EPI>
int launch_narrow(const CUtensorMap& ta, const CUtensorMap& tb, const opk::GemmParams& p, cudaStream_t st) {
  using Cfg = opk::GemmNarrowCfg<BN>;
  auto kern = opk::gemm_narrow_kernel<A_MN, B_MN, BN, EPI>;
  static bool attr_done = false;
  if (!attr_done) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::smem_bytes(Cfg::MANY));
    if (e != cudaSuccess) { set_err(cudaGetErrorString(e)); return (int)e; }
    attr_done = true;
  }
  const dim3 grid((unsigned)((p.M + 127) / 128), (unsigned)((p.N + BN - 1) / BN), (unsigned)p.batch);
  const int stages = (long long)grid.x * grid.y * grid.z > num_sms() ? Cfg::FEW : Cfg::MANY;
  cudaError_t e = opk::launch(kern, grid, 64 + 32 * opk::kNarrowEpiWarps, Cfg::smem_bytes(stages), st, ta, tb, p, stages);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) { set_err(cudaGetErrorString(e)); return (int)e; }
  return 0;
}

constexpr int kHalfPair = 1;      // choose_tile: pairs of CTAs on tiles of 256 x 128

// Tile width of the narrow kernel for this product, kHalfPair, or 0: one of the persistent kernels. Never EPI_SUMSQ: a norm's fp32 partial
// sums follow the tiles, and the clip factor of an example must not depend on which kernel its length favours.
int choose_tile(const OpkGemmArgs* a, int bn, bool pair) {
  if (!pair_mode() || a->tile_group || a->group_k || a->stage_dst || a->max_ctas > 0) return 0;
  const int key = (a->a_mn ? 1 : 0) | (a->b_mn ? 2 : 0);
  const bool ok = a->epilogue == opk::EPI_STORE ? key != 1
                  : a->epilogue == opk::EPI_SWIGLU ? key == 0
                  : a->epilogue == opk::EPI_SWIGLU_BWD ? key == 2 : false;
  if (!ok) return 0;
  auto ceil_div = [](long long x, long long y) { return (x + y - 1) / y; };
  const long long kb = ceil_div(a->K, 64), sms = num_sms();
  // Estimated nanoseconds, fitted to graph replays on B200 over 36 shapes (rows 40 .. 4096, columns 16 .. 16384, reductions
  // 16 .. 128256): a fixed part and a slope per 64-element block of the reduction and round of tiles.
  //   tile            fixed   slope   measured at M x N x K (persistent kernel -> narrow kernel, us)
  //   256 x 256 pair   6600     280
  //   256 x 128 pair   6600     205
  //   128 x 256        5200     315   2048 x 2048 x 2048: 16.9 -> 16.3; 1024 x 3072 x 768: 10.3 -> 9.5
  //   128 x 128        4200     235   1024 x 2304 x 768: 10.2 -> 7.6
  //   128 x 64         3500     225   1024 x 768 x 768: 10.0 -> 6.3
  // Below the line the persistent kernel is the better one: 1021 x 4096 x 4096 26.7 against 27.2 us.
  long long cost = pair ? ceil_div(ceil_div(a->M, 256) * ceil_div(a->N, 256) * a->batch, sms / 2) * kb * 280 + 6600
                        : ceil_div(ceil_div(a->M, 128) * ceil_div(a->N, bn) * a->batch, sms) * kb * 320 + 5300;
  int best = 0;
  for (int w = 64; w <= 256; w *= 2) {
    const long long per = ceil_div(ceil_div(a->M, 128) * ceil_div(a->N, w) * a->batch, sms);
    // Fewer than 32 rows: many CTAs that ask for the same few lines of A at once wait for them. 8 x 6144 x 4096 took 28.4 us on
    // 96 tiles, 18.5 on 48, 22.6 on the persistent kernel; 8 x 8192 x 2048 16.5 on 128, 13.7 persistent (32 rows: 9.5).
    if (per > 4 || (a->M < 32 && ceil_div(a->N, w) > 48)) continue;
    const long long fixed = w == 256 ? 5200 : w == 128 ? 4200 : 3500, slope = w == 256 ? 315 : w == 128 ? 235 : 225;
    const long long round = w == 256 ? 4500 : w == 128 ? 1500 : 800;          // epilogue of every further round
    const long long c = fixed + per * kb * slope + (per - 1) * round;
    if (c < cost) { cost = c; best = w; }
  }
  // Pairs on tiles of 256 x 128: 24 KB per block and SM for the work of a 128 x 128 tile (32 KB) where 256-wide tiles leave pairs
  // idle. From long reductions on, for the layouts of forward products and input gradients (us, before -> with it): 634 x 2048 over
  // 8192 34.2 -> 31.4, over 16384 64.4 -> 56.6, over 128256 477 -> 396; 1021 x 2048 x 50304 197 -> 180; 2048 x 768 x 50257 (two
  // examples' logit gradients) 230 -> 187; 3000 x 768 x 3072 20 -> 17. Short reductions stay with one CTA (2048 x 2048 over 634 rows
  // 11.3, in pairs 12.3) and so does what 64-wide tiles finish in one round (256 x 768 x 50257 175, in pairs 177).
  if (pair && a->epilogue == opk::EPI_STORE && key != 3 && best != 64) {
    const long long per = ceil_div(ceil_div(a->M, 256) * ceil_div(a->N, 128) * a->batch, sms / 2);
    if (6600 + per * kb * 205 + (per - 1) * 1200 < cost) best = kHalfPair;
  }
  return best;
}

// Whether the pair kernel takes eight epilogue warps for a plain store. Where the main loop covers the epilogue of the tile before,
// four are as good and draw less power; eight pay where the epilogue sets the pace (us, four -> eight):
//   weight gradients over few rows   16384 x 2048 over 317: 28.8 -> 24.3; over 64 25.4 -> 20.4; over 1024 51.0 -> 50.4; 128256 x 2048
//                                    over 317 189 -> 164 (its 525 MB take 170 us in a copy)
//   a residual to read               4096 x 768 x 3072 40 -> 33; 2048 x 16384 x 2048 111 -> 103; 1021 x 4096 x 4096 37 -> 33
//   one round of tiles               the only epilogue is exposed: 2304 x 768 over 1024 16.6 -> 13.1
// Not for norms: halves of a tile's columns would be halves of their fp32 partial sums (see teams_epilogue).
bool wide_epilogue(const OpkGemmArgs* a) {
  const long long tiles = (long long)((a->M + 255) / 256) * ((a->N + 255) / 256);
  return a->R || (a->a_mn && a->K <= 512) || tiles <= num_sms() / 2;
}

// Whether the pair kernel takes two teams of epilogue warps for a weight gradient with its norm: where the epilogue sets the pace, that
// is over few rows, and a pair has more than one tile. The bits are those of the four warps: how long an example is, and how many
// share a launch, chooses the faster form and nothing else. (us, four warps -> teams: 16384 x 2048 over 317 rows 35.1 -> 28.1, two examples
// 65.7 -> 49.7, over 64 rows 33.4 -> 27.8; 128256 x 2048 over 317, two examples 487 -> 381; 3072 x 2048 over 317, two examples 17.4 -> 15.6.)
bool teams_epilogue(const OpkGemmArgs* a) {
  const long long tiles = (long long)((a->M + 255) / 256) * ((a->N + 255) / 256) * a->batch;
  return a->K <= 512 && tiles > num_sms() / 2;
}

int pick_bn(int N, int epilogue) {
  if (epilogue == opk::EPI_LCE_FWD || epilogue == opk::EPI_LCE_FWD2 || epilogue == opk::EPI_LCE_BWD || epilogue == opk::EPI_SWIGLU ||
      epilogue == opk::EPI_SWIGLU_BWD)
    return 256;
  return N <= 128 ? 128 : 256;
}

}  // namespace

extern "C" const char* opk_last_error(void) { return g_err; }

// ---- debug-build index checks: registry of the translation units' records (see debug_bounds.cuh)
#ifdef OPK_DEBUG_BOUNDS
namespace opk { namespace dbg {
struct Unit { ReadFn fn; const char* file; };
static Unit* units() { static Unit u[16]; return u; }       // function-local: usable from other units' static initialisers
static int& n_units() { static int n = 0; return n; }
void register_unit(ReadFn fn, const char* file) {
  if (n_units() < 16) units()[n_units()++] = Unit{fn, file};
}
}}  // namespace opk::dbg
#endif

extern "C" int opk_debug_bounds_read(int64_t* out4, char* file_out, int file_cap, int reset) {
#ifdef OPK_DEBUG_BOUNDS
  using namespace opk::dbg;
  out4[0] = out4[1] = out4[2] = out4[3] = 0;
  if (file_out && file_cap > 0) file_out[0] = 0;
  for (int i = 0; i < n_units(); ++i) {
    unsigned long long rec[4] = {0, 0, 0, 0};
    const int e = units()[i].fn(rec, reset);
    if (e != 0) { set_err(cudaGetErrorString((cudaError_t)e)); return e; }
    if (rec[0] && !out4[0]) {
      out4[1] = (int64_t)rec[1]; out4[2] = (int64_t)rec[2]; out4[3] = (int64_t)rec[3];
      if (file_out && file_cap > 0) snprintf(file_out, (size_t)file_cap, "%s", units()[i].file);
    }
    out4[0] += (int64_t)rec[0];
  }
  return 0;
#else
  (void)out4; (void)file_out; (void)file_cap; (void)reset;
  set_err("this library was built without OPK_DEBUG_BOUNDS");
  return -3;
#endif
}
extern "C" int opk_num_sms(void) { return num_sms(); }
extern "C" void opk_gemm_set_pair_mode(int on) { g_pair_mode = on ? 1 : 0; }
extern "C" int opk_gemm_get_pair_mode(void) { return pair_mode() ? 1 : 0; }
extern "C" int opk_gemm_tiles_n(int N, int epilogue) {
  const int bn = pick_bn(N, epilogue);
  return (N + bn - 1) / bn * (epilogue == opk::EPI_LCE_FWD2 ? 2 : 1);
}

extern "C" int opk_gemm(const OpkGemmArgs* a, void* stream) {
  if (!a || a->M <= 0 || a->N <= 0 || a->K <= 0 || a->batch <= 0) { set_err("opk_gemm: bad sizes"); return -1; }
  const int bn = pick_bn(a->N, a->epilogue);
  const bool pair = bn == 256 && !a->tile_group && !a->group_k && a->M >= 256 && pair_mode();
  const int tile = choose_tile(a, bn, pair);
  const bool half = tile == kHalfPair;
  const int narrow = half ? 0 : tile;
  CUtensorMap ta, tb;
  // A: K-major -> {K, M, batch} box {64, 128}; MN-major -> {M, K, batch} box {64, 64}
  if (a->tile_group && (a->batch != 1 || a->n_groups <= 0)) { set_err("opk_gemm: tile_group needs batch == 1 and n_groups"); return -1; }
  if (a->tile_group && a->group_k) { set_err("opk_gemm: tile_group and group_k are exclusive"); return -1; }
  const int abatch = a->group_k ? 1 : a->batch;
  if (a->a_mn) {
    if (!make_map(&ta, a->A, a->M, a->K, abatch, a->lda, a->strideA, 64)) return -2;
  } else {
    if (!make_map(&ta, a->A, a->K, a->M, abatch, a->lda, a->strideA, 128)) return -2;
  }
  const int bdiv = a->b_batch_div > 0 ? a->b_batch_div : 1;
  const int bbatch = a->tile_group ? a->n_groups : (a->group_k ? 1 : (a->batch + bdiv - 1) / bdiv);
  const bool stage = a->stage_dst != nullptr;
  if (stage) {
    // B is read once over NVLink by the kernel's copier warps into stage_dst; the tensor map covers the scratch
    if (!pair || a->a_mn || (a->epilogue != opk::EPI_STORE && !(a->epilogue == opk::EPI_SWIGLU && !a->b_mn && a->act && !(a->N & 1))) ||
        a->batch != 1 || !a->stage_ready || (a->K % 8) || (a->N % 8) ||
        (a->ldb % 8) || (reinterpret_cast<uintptr_t>(a->B) & 15) || (reinterpret_cast<uintptr_t>(a->stage_dst) & 15)) {
      set_err("opk_gemm: staged B needs a plain or SwiGLU product with at least 256 rows, 256-wide tiles and 16-byte aligned rows");
      return -1;
    }
    if (a->b_mn) {
      if (!make_map(&tb, a->stage_dst, a->N, a->K, 1, a->N, 0, 64)) return -2;
    } else {
      if (!make_map(&tb, a->stage_dst, a->K, a->N, 1, a->K, 0, 128)) return -2;
    }
  } else if (a->b_mn) {
    if (!make_map(&tb, a->B, a->N, a->K, bbatch, a->ldb, a->strideB, 64)) return -2;
  } else {
    if (!make_map(&tb, a->B, a->K, a->N, bbatch, a->ldb, a->strideB, narrow ? narrow : half ? 64 : pair ? 128 : bn)) return -2;
  }
  if (a->stepwise && (a->epilogue != opk::EPI_STORE || a->bias)) { set_err("opk_gemm: stepwise rounding takes a plain store without a bias"); return -1; }
  opk::GemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = a->M; p.N = a->N; p.K = a->K; p.batch = a->batch; p.b_batch_div = bdiv;
  p.ldc = a->ldc; p.strideC = a->strideC; p.C = a->C; p.R = a->R; p.bias = a->bias;
  p.alpha = a->alpha; p.stepwise = a->stepwise; p.sumsq = a->sumsq; p.act = a->act; p.ld_act = a->ld_act; p.labels = a->labels;
  p.pmax = a->pmax; p.psum = a->psum; p.tgt = a->tgt; p.lse = a->lse; p.coef = a->coef; p.softcap = a->softcap;
  p.z = a->z;
  if (a->softcap > 0.f) {
    const double inv = 1.0 / (double)a->softcap;
    p.inv_cap = (float)inv;
    p.inv_cap_lo = p.inv_cap <= 3.4028234e38f ? (float)(inv - (double)p.inv_cap) : 0.f;      // 1 / cap beyond fp32: no low part
  }
  p.err = a->err;
  p.tile_group = a->tile_group; p.group_k = a->group_k; p.sumsq_stride = a->sumsq_shared ? 0 : 1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int key = (a->a_mn ? 1 : 0) | (a->b_mn ? 2 : 0);
  const int mc = a->max_ctas;
  if (stage) {
    const int n_bands = (a->N + opk::kRasterBand * 256 - 1) / (opk::kRasterBand * 256);
    cudaError_t e = cudaMemsetAsync(a->stage_ready, 0, sizeof(int32_t) * n_bands, st);
    if (e != cudaSuccess) { set_err(cudaGetErrorString(e)); return (int)e; }
    p.stage_src = a->B; p.stage_ld = a->ldb; p.stage_dst = a->stage_dst; p.stage_ready = a->stage_ready;
    if (a->epilogue == opk::EPI_SWIGLU) return launch2<false, false, opk::EPI_SWIGLU, opk::G2_STAGE>(ta, tb, p, mc, st);
    return a->b_mn ? launch2<false, true, opk::EPI_STORE, opk::G2_STAGE>(ta, tb, p, mc, st)
                   : launch2<false, false, opk::EPI_STORE, opk::G2_STAGE>(ta, tb, p, mc, st);
  }
  if (narrow) {
    if (a->epilogue == opk::EPI_SWIGLU && (!a->act || (a->N & 1))) { set_err("opk_gemm: swiglu needs act and even N"); return -1; }
    if (a->epilogue == opk::EPI_SWIGLU_BWD && (!a->act || a->R || a->bias)) {
      set_err("opk_gemm: swiglu backward needs the saved pre-activations and takes no bias / residual");
      return -1;
    }
#define OPK_NARROW(AM, BM_, E) \
  (narrow == 256   ? launch_narrow<AM, BM_, 256, E>(ta, tb, p, st)          \
   : narrow == 128 ? launch_narrow<AM, BM_, 128, E>(ta, tb, p, st)          \
                   : launch_narrow<AM, BM_, 64, E>(ta, tb, p, st))
    if (a->epilogue == opk::EPI_SWIGLU) return OPK_NARROW(false, false, opk::EPI_SWIGLU);
    if (a->epilogue == opk::EPI_SWIGLU_BWD) return OPK_NARROW(false, true, opk::EPI_SWIGLU_BWD);
    if (key == 0) return OPK_NARROW(false, false, opk::EPI_STORE);
    if (key == 2) return OPK_NARROW(false, true, opk::EPI_STORE);
    return OPK_NARROW(true, true, opk::EPI_STORE);
#undef OPK_NARROW
  }
  if (pair) {
    switch (a->epilogue) {
      case opk::EPI_STORE:
        if (half)
          return key == 0 ? launch2<false, false, opk::EPI_STORE, opk::G2_HALF>(ta, tb, p, mc, st)
                          : launch2<false, true, opk::EPI_STORE, opk::G2_HALF>(ta, tb, p, mc, st);
        if (wide_epilogue(a)) {
          if (key == 0) return launch2<false, false, opk::EPI_STORE, opk::G2_WIDE>(ta, tb, p, mc, st);
          if (key == 2) return launch2<false, true, opk::EPI_STORE, opk::G2_WIDE>(ta, tb, p, mc, st);
          if (key == 3) return launch2<true, true, opk::EPI_STORE, opk::G2_WIDE>(ta, tb, p, mc, st);
          break;
        }
        if (key == 0) return launch2<false, false, opk::EPI_STORE>(ta, tb, p, mc, st);
        if (key == 2) return launch2<false, true, opk::EPI_STORE>(ta, tb, p, mc, st);
        if (key == 3) return launch2<true, true, opk::EPI_STORE>(ta, tb, p, mc, st);
        break;
      case opk::EPI_SUMSQ:
        if (!a->sumsq) { set_err("opk_gemm: sumsq pointer required"); return -1; }
        if (key == 3 && teams_epilogue(a)) return launch2<true, true, opk::EPI_SUMSQ, opk::G2_TEAMS>(ta, tb, p, mc, st);
        if (key == 3) return launch2<true, true, opk::EPI_SUMSQ>(ta, tb, p, mc, st);
        break;
      case opk::EPI_SWIGLU:
        if (!a->act || (a->N & 1)) { set_err("opk_gemm: swiglu needs act and even N"); return -1; }
        if (key == 0) return launch2<false, false, opk::EPI_SWIGLU>(ta, tb, p, mc, st);
        break;
      case opk::EPI_SWIGLU_BWD:
        if (!a->act || a->R || a->bias) { set_err("opk_gemm: swiglu backward needs the saved pre-activations and takes no bias / residual"); return -1; }
        if (key == 2) return launch2<false, true, opk::EPI_SWIGLU_BWD>(ta, tb, p, mc, st);
        break;
      case opk::EPI_LCE_FWD:
        if (!a->labels || !a->pmax || !a->psum || !a->tgt) { set_err("opk_gemm: lce fwd buffers required"); return -1; }
        if (key == 0)
          return a->z ? a->lce_parts == 2 ? launch2<false, false, opk::EPI_LCE_KEEP2>(ta, tb, p, mc, st)
                                          : launch2<false, false, opk::EPI_LCE_KEEP>(ta, tb, p, mc, st)
                 : a->lce_parts == 2 ? launch2<false, false, opk::EPI_LCE_FWD2>(ta, tb, p, mc, st)
                                     : launch2<false, false, opk::EPI_LCE_FWD>(ta, tb, p, mc, st);
        break;
      case opk::EPI_LCE_BWD:
        if (!a->labels || !a->lse || !a->coef) { set_err("opk_gemm: lce bwd buffers required"); return -1; }
        if (key == 0) return launch2<false, false, opk::EPI_LCE_BWD>(ta, tb, p, mc, st);
        break;
      default: break;
    }
    set_err("opk_gemm: unsupported (layout, epilogue) combination");
    return -3;
  }
  switch (a->epilogue) {
    case opk::EPI_STORE:
      if (key == 0) return bn == 256 ? launch<false, false, 256, opk::EPI_STORE>(ta, tb, p, mc, st)
                                     : launch<false, false, 128, opk::EPI_STORE>(ta, tb, p, mc, st);
      if (key == 2) return bn == 256 ? launch<false, true, 256, opk::EPI_STORE>(ta, tb, p, mc, st)
                                     : launch<false, true, 128, opk::EPI_STORE>(ta, tb, p, mc, st);
      if (key == 3) return bn == 256 ? launch<true, true, 256, opk::EPI_STORE>(ta, tb, p, mc, st)
                                     : launch<true, true, 128, opk::EPI_STORE>(ta, tb, p, mc, st);
      break;
    case opk::EPI_SUMSQ:
      if (!a->sumsq) { set_err("opk_gemm: sumsq pointer required"); return -1; }
      if (key == 3) return bn == 256 ? launch<true, true, 256, opk::EPI_SUMSQ>(ta, tb, p, mc, st)
                                     : launch<true, true, 128, opk::EPI_SUMSQ>(ta, tb, p, mc, st);
      break;
    case opk::EPI_SWIGLU:
      if (!a->act || (a->N & 1)) { set_err("opk_gemm: swiglu needs act and even N"); return -1; }
      if (key == 0) return launch<false, false, 256, opk::EPI_SWIGLU>(ta, tb, p, mc, st);
      break;
    case opk::EPI_SWIGLU_BWD:
      if (!a->act || a->R || a->bias) { set_err("opk_gemm: swiglu backward needs the saved pre-activations and takes no bias / residual"); return -1; }
      if (key == 2) return launch<false, true, 256, opk::EPI_SWIGLU_BWD>(ta, tb, p, mc, st);
      break;
    case opk::EPI_LCE_FWD:
      if (!a->labels || !a->pmax || !a->psum || !a->tgt) { set_err("opk_gemm: lce fwd buffers required"); return -1; }
      if (key == 0)
        return a->z ? a->lce_parts == 2 ? launch<false, false, 256, opk::EPI_LCE_KEEP2>(ta, tb, p, mc, st)
                                        : launch<false, false, 256, opk::EPI_LCE_KEEP>(ta, tb, p, mc, st)
               : a->lce_parts == 2 ? launch<false, false, 256, opk::EPI_LCE_FWD2>(ta, tb, p, mc, st)
                                   : launch<false, false, 256, opk::EPI_LCE_FWD>(ta, tb, p, mc, st);
      break;
    case opk::EPI_LCE_BWD:
      if (!a->labels || !a->lse || !a->coef) { set_err("opk_gemm: lce bwd buffers required"); return -1; }
      if (key == 0) return launch<false, false, 256, opk::EPI_LCE_BWD>(ta, tb, p, mc, st);
      break;
    default: break;
  }
  set_err("opk_gemm: unsupported (layout, epilogue) combination");
  return -3;
}

extern "C" int64_t opk_lce_logits_floats(int M, int N) {
  return M > 0 && N > 0 ? (int64_t)((M + 31) / 32) * ((N + 31) / 32) * 1024 : 0;
}

extern "C" int opk_lce_grad(const float* z, const int32_t* labels, const float* lse, const float* coef, void* out, int64_t ld, int M,
                            int N, float softcap, void* stream) {
  if (M <= 0 || N <= 0 || ld < N || !z || !labels || !lse || !coef || !out || (reinterpret_cast<uintptr_t>(z) & 15)) {
    set_err("opk_lce_grad: bad arguments");
    return -1;
  }
  opk::GemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.batch = 1; p.alpha = 1.f; p.C = out; p.ldc = ld;
  p.z = const_cast<float*>(z); p.labels = labels; p.lse = lse; p.coef = coef; p.softcap = softcap;
  const long long groups = ((N + 31) / 32 + opk::kLceGradChunks - 1) / opk::kLceGradChunks;
  const long long items = groups * ((M + 31) / 32);
  opk::lce_grad_kernel<<<(unsigned)((items + 7) / 8), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_err(cudaGetErrorString(e)); return (int)e; }
  return 0;
}

// ------------------------------------------------------------------------------------------------ wait self-test
// One CTA waits on an mbarrier that nothing ever completes, with a short cycle budget. The wait gives up, the abort
// flag is raised and the error word is set: the same unwinding path every pipeline role of the real kernels takes
// when a producer or peer never shows up. The kernel returns normally and the context stays usable.
namespace {
__global__ void wait_selftest_kernel(int* err, long long budget_cycles, long long* waited_cycles) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    opk::mbar_init(&bar, 1);
    abort_flag = 0;
    opk::fence_barrier_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const long long t0 = clock64();
    const bool ok = opk::mbar_wait(&bar, 0, &abort_flag, budget_cycles);
    if (waited_cycles) *waited_cycles = clock64() - t0;
    if (!ok && err) atomicExch(err, 1);
  }
  __syncthreads();
  // every other thread sees the flag the waiting role raised
  if (threadIdx.x == 1 && abort_flag && err) atomicOr(err, 2);
}
}  // namespace

extern "C" int opk_wait_selftest(int32_t* err, int64_t budget_cycles, int64_t* waited_cycles, void* stream) {
  if (budget_cycles <= 0 || budget_cycles > 4000000000LL) return -1;
  wait_selftest_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(err, budget_cycles,
                                                                           reinterpret_cast<long long*>(waited_cycles));
  return (int)cudaGetLastError();
}
