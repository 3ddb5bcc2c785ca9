// Rotary position embedding of the query and key projections and its backward, one launch each (sm_100a).
//
// The models rotate the two halves (a, b) of every head against each other by the tables of their position,
// a' = a cos - b sin, b' = b cos + a sin, in fp32 and hand bf16 to the attention kernel (nvfp4_train.py:91-98).  As
// torch operations that is, for q and k, forward and backward, about fifty element-wise launches and fp32 copies of
// both tensors: 0.75 ms of a decoder block's 2.29 ms of kernels (d 768, 16 x 1024 tokens), and as much host time.
// Here a thread takes eight elements of each half with one 16-byte access per half and direction, and both tensors go
// in one launch: 19 us for forward or backward of that block (100 MB, 5.3 TB/s).  HBM-bound.
// The roundings are those of the torch operations, so the result has the same bits.  Forward: products and sum rounded
// separately in fp32, the result once to bf16.  Backward (the transposed rotation): autograd rounds the gradient
// of every product to bf16, the type of its input, and adds the two in bf16.
#include "common.cuh"
#include "nvfp4_b200.h"

namespace nvfp4 {
namespace rotary {

struct Side {
  const uint16_t* x;       // [rows, heads * head_dim], contiguous
  uint16_t* out;
  int heads;
};

__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

template <bool BACKWARD>
__global__ void __launch_bounds__(256) rotary_kernel(Side q, Side k, int64_t rows, int seq, int head_dim,
                                                     const float* __restrict__ cosine, const float* __restrict__ sine) {
  const Side s = blockIdx.y == 0 ? q : k;
  const int half = head_dim >> 1, chunks = half >> 3;                 // 16-byte chunks of a half
  const int64_t items = rows * s.heads * chunks;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < items; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t head_row = i / chunks;                              // row * heads + head
    const int c = (int)(i - head_row * chunks) * 8;
    const int t = (int)((head_row / s.heads) % seq);
    const int64_t at = head_row * head_dim + c;
    const uint4 a4 = __ldg(reinterpret_cast<const uint4*>(s.x + at)), b4 = __ldg(reinterpret_cast<const uint4*>(s.x + at + half));
    const uint32_t aw[4] = {a4.x, a4.y, a4.z, a4.w}, bw[4] = {b4.x, b4.y, b4.z, b4.w};
    float cs[8], sn[8];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float4 u = __ldg(reinterpret_cast<const float4*>(cosine + (int64_t)t * half + c) + j);
      const float4 v = __ldg(reinterpret_cast<const float4*>(sine + (int64_t)t * half + c) + j);
      cs[4 * j] = u.x; cs[4 * j + 1] = u.y; cs[4 * j + 2] = u.z; cs[4 * j + 3] = u.w;
      sn[4 * j] = v.x; sn[4 * j + 1] = v.y; sn[4 * j + 2] = v.z; sn[4 * j + 3] = v.w;
    }
    uint32_t oa[4], ob[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float ra[2], rb[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float a = h ? bf16_hi(aw[j]) : bf16_lo(aw[j]), b = h ? bf16_hi(bw[j]) : bf16_lo(bw[j]);
        const float cc = cs[2 * j + h], ss = sn[2 * j + h];
        if (BACKWARD) {
          ra[h] = round_bf16(__fmul_rn(a, cc)) + round_bf16(__fmul_rn(b, ss));
          rb[h] = round_bf16(__fmul_rn(b, cc)) - round_bf16(__fmul_rn(a, ss));
        } else {
          ra[h] = __fsub_rn(__fmul_rn(a, cc), __fmul_rn(b, ss));
          rb[h] = __fadd_rn(__fmul_rn(b, cc), __fmul_rn(a, ss));
        }
      }
      const __nv_bfloat162 pa = __floats2bfloat162_rn(ra[0], ra[1]), pb = __floats2bfloat162_rn(rb[0], rb[1]);
      oa[j] = *reinterpret_cast<const uint32_t*>(&pa);
      ob[j] = *reinterpret_cast<const uint32_t*>(&pb);
    }
    *reinterpret_cast<uint4*>(s.out + at) = make_uint4(oa[0], oa[1], oa[2], oa[3]);
    *reinterpret_cast<uint4*>(s.out + at + half) = make_uint4(ob[0], ob[1], ob[2], ob[3]);
  }
}

}  // namespace rotary
}  // namespace nvfp4

extern "C" int nvfp4_rotary_bf16(const void* q, void* q_out, int q_heads, const void* k, void* k_out, int k_heads,
                                 int64_t rows, int64_t seq, int head_dim, const float* cosine, const float* sine,
                                 int backward, void* stream_) {
  if (!q || !q_out || !k || !k_out || !cosine || !sine) return NVFP4_E_NULL;
  if (rows <= 0 || seq <= 0 || seq > 0x7fffffffLL || rows % seq != 0 || q_heads <= 0 || k_heads <= 0 || head_dim <= 0 ||
      (head_dim & 15) != 0)
    return NVFP4_E_SHAPE;
  auto mis = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) != 0; };
  if (mis(q) || mis(q_out) || mis(k) || mis(k_out) || mis(cosine) || mis(sine)) return NVFP4_E_ALIGN;
  const int64_t items = rows * (q_heads > k_heads ? q_heads : k_heads) * (head_dim / 16);
  const int64_t blocks = (items + 255) / 256;
  const dim3 grid((unsigned)(blocks < 148 * 32 ? blocks : 148 * 32), 2);
  const nvfp4::rotary::Side a{static_cast<const uint16_t*>(q), static_cast<uint16_t*>(q_out), q_heads};
  const nvfp4::rotary::Side b{static_cast<const uint16_t*>(k), static_cast<uint16_t*>(k_out), k_heads};
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (backward) nvfp4::rotary::rotary_kernel<true><<<grid, 256, 0, stream>>>(a, b, rows, (int)seq, head_dim, cosine, sine);
  else nvfp4::rotary::rotary_kernel<false><<<grid, 256, 0, stream>>>(a, b, rows, (int)seq, head_dim, cosine, sine);
  return cudaGetLastError() == cudaSuccess ? NVFP4_OK : NVFP4_E_LAUNCH;
}
