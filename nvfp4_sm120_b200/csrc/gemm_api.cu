// nvfp4_gemm: argument checks, tensor maps, kernel choice (C ABI; declared in include/nvfp4_b200.h).
#include "gemm_common.cuh"

namespace nvfp4 { namespace gemm3 {
int launch_pair(int tile_n, const CUtensorMap& map_d, const uint8_t* a_q, const uint8_t* b_q, const gemm::Params& p,
                cudaStream_t stream);
}}
namespace nvfp4 { namespace gemm {
int launch_1cta(int tile_n, const CUtensorMap& map_d, const uint8_t* a_q, const uint8_t* b_q, const Params& p,
                cudaStream_t stream);
}}

#include <atomic>

static std::atomic<int> g_gemm_mode{0};
// test hooks (nvfp4_test_hooks): the wait limit of the next launches and the dropped arrival
static std::atomic<unsigned long long> g_gemm_wait_ns{0};
static std::atomic<int> g_gemm_drop_arrival{0};
namespace nvfp4 { namespace gemm {
void set_test_hooks(unsigned long long wait_ns, int drop_arrival) {
  g_gemm_wait_ns.store(wait_ns, std::memory_order_relaxed);
  g_gemm_drop_arrival.store(drop_arrival, std::memory_order_relaxed);
}
}}
extern "C" int nvfp4_gemm_set_mode(int mode) {
  if (mode < 0 || mode > 2) return NVFP4_E_MODE;
  g_gemm_mode.store(mode, std::memory_order_relaxed);
  return NVFP4_OK;
}

namespace nvfp4 { namespace gemm {
__global__ void pts_from_amax_kernel(const float* __restrict__ amax, float* __restrict__ pts) {
  *pts = __fdiv_rn(fmaxf(*amax, kAmaxFloor), kGlobalDiv);
}
int launch_pts_from_amax(const float* amax, float* pts, cudaStream_t stream) {
  pts_from_amax_kernel<<<1, 1, 0, stream>>>(amax, pts);
  return cudaGetLastError() == cudaSuccess ? NVFP4_OK : NVFP4_E_LAUNCH;
}
}}

// Kernel, tile width and CTAs per tile.
struct Choice { bool pair; int tile_n, splits; };

// The rule: the candidate with the smallest estimate of its time in us,
//   fixed part + waves * K slices per CTA * time per slice + drain of the waves before the last (+ sum over the cluster),
// with constants measured on a B200 (CUDA graph of 24 launches, operands in L2) over 1 .. 16384 x 300 .. 14336 x 512 ..
// 16384: launch, pipeline fill and epilogue 3.8 us for a 128 x 64 tile, 5.75 us for a 256 x 256 pair; a slice is bound by
// the fill of shared memory from L2 (about 64 bytes per SM and clock) in the one-CTA kernel, by the shared-memory data
// stage in the pair kernel.  The estimate orders the candidates right where they differ by more than about 5 %.  Where
// the lines fall (us, best candidate against the 256 x 256 pair tiles): 512 x 768 x 768 4.9 / 6.8 (128 x 64), 5328 x 768 x
// 768 6.7 / 7.2 (128 x 256), 2048 x 768 x 3072 8.6 / 9.8 (pair 256 x 128), 1000 x 2584 x 7136 17.0 / 18.6 (pair 256 x 192),
// 256 x 1024 x 8192 8.9 / 14.9 (128 x 64, four CTAs per tile), 64 x 4096 x 14336 12.6 / 22.9 (128 x 128, four),
// 768 x 768 x 16384 15.7 / 24.7 (128 x 256, four), 8 x 14336 x 4096 11.9 / 12.6 (128 x 256, two).
static Choice choose(int64_t M, int64_t N, int64_t K, int forced) {
  struct Kind { bool pair; int tile_n; float fixed, slice, drain, sum; };
  static const Kind kinds[] = {{true, 256, 5.75f, 0.315f, 1.3f, 0.0f}, {true, 192, 5.35f, 0.31f, 0.85f, 0.0f},
                               {true, 128, 4.75f, 0.29f, 0.6f, 0.0f},  {false, 256, 5.35f, 0.39f, 4.3f, 2.6f},
                               {false, 128, 4.25f, 0.345f, 3.8f, 1.6f}, {false, 64, 3.8f, 0.32f, 2.4f, 1.2f}};
  // CTAs that the device holds at once as clusters of 1, 2, 4, 8 (clusters of 8: 16 of them did not fit)
  static const int caps[] = {148, 148, 128, 112};
  const int64_t slices = (K + 255) / 256;
  Choice best{true, 256, 1};
  float best_us = 3.0e38f;
  for (const Kind& k : kinds) {
    if (forced != 0 && k.pair != (forced == 2)) continue;
    const int64_t rows = k.pair ? 256 : 128, tiles = ((M + rows - 1) / rows) * ((N + k.tile_n - 1) / k.tile_n);
    for (int log_s = 0; log_s < (k.pair ? 1 : 4); ++log_s) {
      const int s = 1 << log_s;
      const int64_t per = (slices + s - 1) / s, cap = k.pair ? 74 : caps[log_s];
      if (s > 1 && (tiles * s > cap || per * (s - 1) >= slices)) break;      // one wave, and work for every CTA
      const int64_t waves = (tiles * s + cap - 1) / cap;
      float us = k.fixed + (float)waves * (float)per * k.slice + (float)(waves - 1) * k.drain;
      if (s > 1) us += 0.3f + 0.15f * (float)s + k.sum * (float)(M < 128 ? M : 128) / 128.0f;
      if (us < best_us) { best_us = us; best = Choice{k.pair, k.tile_n, s}; }
    }
  }
  return best;
}

extern "C" int nvfp4_gemm_choice(int64_t M, int64_t N, int64_t K, int32_t* choice3) {
  if (choice3 == nullptr) return NVFP4_E_NULL;
  if (M <= 0 || N <= 0 || K <= 0) return NVFP4_E_SHAPE;
  const Choice c = choose(M, N, K, g_gemm_mode.load(std::memory_order_relaxed));
  choice3[0] = c.pair ? 2 : 1;
  choice3[1] = c.tile_n;
  choice3[2] = c.splits;
  return NVFP4_OK;
}

static int gemm_any(const uint8_t* a_q, const uint8_t* a_sf, const float* a_pts, const uint8_t* b_q,
                    const uint8_t* b_sf, const float* b_pts, void* d, int out_dtype, int64_t M, int64_t N,
                    int64_t K, int64_t ldd, uint8_t* d_sf, const float* d_amax, float* d_amax_out, int32_t* status,
                    void* stream_, int round_bf16 = 0) {
  using namespace nvfp4::gemm;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const bool fp4_out = d_sf != nullptr;
  if (!a_q || !a_sf || !a_pts || !b_q || !b_sf || !b_pts || !d) return NVFP4_E_NULL;
  if (M <= 0 || N <= 0 || K <= 0 || (K & 31) != 0 || ldd < N) return NVFP4_E_SHAPE;
  if (M > 0x7fffffffLL || N > 0x7fffffffLL || K > 0x7fffffffLL) return NVFP4_E_SHAPE;
  if (out_dtype != NVFP4_OUT_BF16 && out_dtype != NVFP4_OUT_F32) return NVFP4_E_MODE;
  auto mis = [](const void* p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) != 0; };
  if (mis(a_q, 16) || mis(b_q, 16) || mis(a_sf, 16) || mis(b_sf, 16) || mis(d, 16)) return NVFP4_E_ALIGN;
  if (d_amax_out != nullptr) {
    if (fp4_out) return NVFP4_E_MODE;
    if (cudaMemsetAsync(d_amax_out, 0, sizeof(float), stream) != cudaSuccess) return NVFP4_E_LAUNCH;
  }
  const int forced = g_gemm_mode.load(std::memory_order_relaxed);
  // One choice for every form of output, so that all of them hold the same sums.  (A quantized output wants whole blocks
  // of 16 columns in a CTA's share: 64 columns over eight CTAs become 128, the same shares of K.)
  Choice pick = choose(M, N, K, forced);
  if (fp4_out && pick.tile_n < 16 * pick.splits) pick.tile_n = 128;
  Params p{a_sf, b_sf, a_pts, b_pts, d, M, N, K, ldd, out_dtype == NVFP4_OUT_F32 ? 1 : 0, status, pick.splits, 0,
           g_gemm_wait_ns.load(std::memory_order_relaxed), g_gemm_drop_arrival.load(std::memory_order_relaxed),
           d_sf, d_amax, fp4_out ? 1 : 0, round_bf16, d_amax_out};
  // The epilogue stores through TMA when the row pitch allows a tensor map (a multiple of 16 bytes).
  CUtensorMap map_d{};                                         // unused otherwise
  if (p.splits == 1 && !fp4_out && (ldd * (p.out_f32 ? 4 : 2)) % 16 == 0) {
    if (!make_output_map(&map_d, d, M, N, ldd, p.out_f32 != 0)) return NVFP4_E_DRIVER;
    p.tma_store = 1;
  }
  return pick.pair ? nvfp4::gemm3::launch_pair(pick.tile_n, map_d, a_q, b_q, p, stream)
              : launch_1cta(pick.tile_n, map_d, a_q, b_q, p, stream);
}

extern "C" int nvfp4_gemm(const uint8_t* a_q, const uint8_t* a_sf, const float* a_pts, const uint8_t* b_q,
                          const uint8_t* b_sf, const float* b_pts, void* d, int out_dtype, int64_t M, int64_t N,
                          int64_t K, int64_t ldd, int32_t* status, void* stream_) {
  return gemm_any(a_q, a_sf, a_pts, b_q, b_sf, b_pts, d, out_dtype, M, N, K, ldd, nullptr, nullptr, nullptr, status,
                  stream_);
}

extern "C" int nvfp4_gemm_bf16_as_f32(const uint8_t* a_q, const uint8_t* a_sf, const float* a_pts, const uint8_t* b_q,
                                      const uint8_t* b_sf, const float* b_pts, float* d, int64_t M, int64_t N, int64_t K,
                                      int64_t ldd, int32_t* status, void* stream_) {
  return gemm_any(a_q, a_sf, a_pts, b_q, b_sf, b_pts, d, NVFP4_OUT_F32, M, N, K, ldd, nullptr, nullptr, nullptr, status,
                  stream_, 1);
}

extern "C" int nvfp4_gemm_amax(const uint8_t* a_q, const uint8_t* a_sf, const float* a_pts, const uint8_t* b_q,
                               const uint8_t* b_sf, const float* b_pts, void* d, int out_dtype, int64_t M, int64_t N,
                               int64_t K, int64_t ldd, float* d_amax_out, int32_t* status, void* stream_) {
  if (!d_amax_out) return NVFP4_E_NULL;
  return gemm_any(a_q, a_sf, a_pts, b_q, b_sf, b_pts, d, out_dtype, M, N, K, ldd, nullptr, nullptr, d_amax_out, status,
                  stream_);
}

extern "C" int nvfp4_gemm_fp4out(const uint8_t* a_q, const uint8_t* a_sf, const float* a_pts, const uint8_t* b_q,
                                 const uint8_t* b_sf, const float* b_pts, int64_t M, int64_t N, int64_t K,
                                 const float* d_amax, uint8_t* d_q, uint8_t* d_sf, float* d_pts, int32_t* status,
                                 void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!d_amax || !d_q || !d_sf || !d_pts) return NVFP4_E_NULL;
  if ((N & 15) != 0) return NVFP4_E_SHAPE;
  if ((reinterpret_cast<uintptr_t>(d_sf) & 15u) != 0) return NVFP4_E_ALIGN;
  // padding of the tiled scale buffer reads as zero; the per-tensor scale is the given maximum / 2688
  const int64_t sm = (M + 127) / 128 * 128, sk = (N / 16 + 3) / 4 * 4;
  if ((sm != M || sk != N / 16) && cudaMemsetAsync(d_sf, 0, (size_t)(sm * sk), stream) != cudaSuccess) return NVFP4_E_LAUNCH;
  const int rc = gemm_any(a_q, a_sf, a_pts, b_q, b_sf, b_pts, d_q, NVFP4_OUT_BF16, M, N, K, N, d_sf, d_amax, nullptr, status,
                          stream_);
  if (rc != NVFP4_OK) return rc;
  return nvfp4::gemm::launch_pts_from_amax(d_amax, d_pts, stream);
}
