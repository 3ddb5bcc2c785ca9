// Per-tensor amax and the fused NVFP4 quantizer for B200 (sm_100a).
//
// One pass computes, per 16-element block: [random-sign Hadamard] -> block amax -> E4M3 block
// scale -> E2M1 codes (round-to-nearest-even, or hardware stochastic rounding fed by a Philox
// stream) -> packed nibbles, and writes the scale byte straight to its place in the 128x4-tiled
// layout the tcgen05 block-scaled MMA reads.  The arithmetic follows the reference's pure-torch
// quantizer operation by operation (nvfp4_gemm.py:36-45): true fp32 divisions, no fast-math.
#include "quantize_common.cuh"

namespace nvfp4 {

using fused::PhiloxKeys;

// ---------------------------------------------------------------------------------------
// shared per-block arithmetic: that of the single-launch kernels (quantize_common.cuh) -- the block
// scale byte by the checked one-multiply shortcut, (1 / pts) / scale from a 128-entry table made with
// true divisions, Philox with host-made round keys -- so the bytes are the same and a block costs
// about 80 instructions less than with three true divisions and in-kernel key updates.
// ---------------------------------------------------------------------------------------
struct GlobalScale {
  fused::Scale sc;          // pts = amax / 2688, 1 / pts, 1 / (6 pts)
  const float* recip;       // shared memory: recip[b] = (1 / pts) / e4m3(b)
  float pts;
};

// Every thread of the CTA calls this (it holds a barrier); `tab` is 128 floats of shared memory.
__device__ __forceinline__ GlobalScale global_scale(const float* __restrict__ amax, float* tab) {
  GlobalScale g;
  g.sc.pts = __fdiv_rn(fmaxf(__ldg(amax), kAmaxFloor), kGlobalDiv);
  g.sc.inv_pts = __fdiv_rn(1.0f, g.sc.pts);
  g.sc.c = __fdiv_rn(1.0f, kF4Max * g.sc.pts);
  g.pts = g.sc.pts;
  g.recip = tab;
  if (threadIdx.x < 128) tab[threadIdx.x] = __fdiv_rn(g.sc.inv_pts, e4m3_to_f32(threadIdx.x));
  __syncthreads();
  return g;
}

inline PhiloxKeys make_philox_keys(uint64_t seed) {
  PhiloxKeys keys;
  for (int r = 0; r < 10; ++r) {
    keys.k[r][0] = (uint32_t)seed + (uint32_t)r * 0x9E3779B9u;
    keys.k[r][1] = (uint32_t)(seed >> 32) + (uint32_t)r * 0xBB67AE85u;
  }
  return keys;
}

// v[16] (already Hadamard-transformed if wanted) -> 8 bytes of codes (lo, hi) and the E4M3 byte.
__device__ __forceinline__ float block_amax16(const float (&v)[16]) {
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
  return amax;
}

// amax: the maximum the block scale is derived from -- the block's own (1 x 16 scaling), or that of
// the 16 x 16 tile around it (2-D weight scaling, nvfp4_validate.py:68-82)
template <bool SR>
__device__ __forceinline__ void encode_block_scaled(const float (&v)[16], float amax, const GlobalScale& g,
                                                    uint64_t blk_index, const PhiloxKeys& keys, uint64_t offset,
                                                    uint32_t& lo, uint32_t& hi, uint32_t& sf_byte) {
  sf_byte = fused::block_scale_byte(amax, g.sc);                   // nvfp4_gemm.py:39-40
  const float recip = g.recip[sf_byte];                            // :41
  // the clamp to +-6 of :42 is the saturation of the conversions below
  if (SR) {
    const Philox4 r = fused::philox_rounds((uint32_t)blk_index, (uint32_t)(blk_index >> 32),
                                           (uint32_t)offset, (uint32_t)(offset >> 32), keys);
    const uint32_t q0 = e2m1x4_rs(v[0] * recip, v[1] * recip, v[2] * recip, v[3] * recip, r.x);
    const uint32_t q1 = e2m1x4_rs(v[4] * recip, v[5] * recip, v[6] * recip, v[7] * recip, r.y);
    const uint32_t q2 = e2m1x4_rs(v[8] * recip, v[9] * recip, v[10] * recip, v[11] * recip, r.z);
    const uint32_t q3 = e2m1x4_rs(v[12] * recip, v[13] * recip, v[14] * recip, v[15] * recip, r.w);
    lo = q0 | (q1 << 16);
    hi = q2 | (q3 << 16);
  } else {
    float d[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) d[j] = v[j] * recip;
    lo = fused::e2m1x8_rn(d);
    hi = fused::e2m1x8_rn(d + 8);
  }
}

template <bool SR>
__device__ __forceinline__ void encode_block(const float (&v)[16], const GlobalScale& g,
                                             uint64_t blk_index, const PhiloxKeys& keys, uint64_t offset,
                                             uint32_t& lo, uint32_t& hi, uint32_t& sf_byte) {
  encode_block_scaled<SR>(v, block_amax16(v), g, blk_index, keys, offset, lo, hi, sf_byte);
}

__device__ __forceinline__ void load_signs(const float* __restrict__ signs16, float (&sg)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 s = __ldg(reinterpret_cast<const float4*>(signs16) + i);
    sg[4 * i] = s.x; sg[4 * i + 1] = s.y; sg[4 * i + 2] = s.z; sg[4 * i + 3] = s.w;
  }
}

__device__ __forceinline__ void atomic_max_nonneg(float* addr, float v) {
  // non-negative floats order like their bit patterns
  atomicMax(reinterpret_cast<unsigned int*>(addr), __float_as_uint(v));
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Maximum of a non-negative per-thread value over the CTA, then ONE atomic per CTA: same-address atomics
// from every warp serialise in the L2 (19 000 of them cost 25 us, more than reading 64 MiB does).
// Every thread of the CTA calls this; `slot` selects one of two independent reductions.
__device__ __forceinline__ void cta_max_to(float* addr, float v, int slot = 0) {
  __shared__ float part[2][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  if (lane == 0) part[slot][warp] = v;
  __syncthreads();
  if (warp == 0) {
    float m = lane < nwarps ? part[slot][lane] : 0.0f;
    m = warp_max(m);
    if (lane == 0 && !(m == 0.0f)) atomic_max_nonneg(addr, m);
  }
}

// ---------------------------------------------------------------------------------------
// amax kernels
// ---------------------------------------------------------------------------------------
// plain |x| maximum: 16-byte loads, max of packed bf16 magnitudes
__global__ void __launch_bounds__(512) amax_plain_kernel(const uint16_t* __restrict__ x, int64_t rows,
                                                         int vec_per_row, int64_t ld,
                                                         float* __restrict__ amax) {
  const int64_t total = rows * vec_per_row;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  uint32_t m = 0;
  auto fold = [&](const uint4& q) { m = fused::max_abs_word(m, q); };   // both halves of m carry a running maximum
  const bool flat = ld == (int64_t)vec_per_row * 8;      // contiguous rows: no division per load
  auto load = [&](int64_t i) {
    if (flat) return __ldg(reinterpret_cast<const uint4*>(x) + i);
    const int64_t r = i / vec_per_row;
    const int cv = (int)(i - r * vec_per_row);
    return __ldg(reinterpret_cast<const uint4*>(x + r * ld) + cv);
  };
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // Eight 16-byte loads per thread in flight and one wave of four CTAs per SM: 8192 x 4096 out of HBM 21.4 -> 17.1 us with
  // the clearing of the word, 4096 x 14336 25.2 -> 22.9 (four loads and up to eight CTAs per SM in turn before).
  for (; i + 7 * stride < total; i += 8 * stride) {
    uint4 q[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) q[u] = load(i + u * stride);
#pragma unroll
    for (int u = 0; u < 8; ++u) fold(q[u]);
  }
  for (; i + 3 * stride < total; i += 4 * stride) {
    const uint4 q0 = load(i), q1 = load(i + stride), q2 = load(i + 2 * stride), q3 = load(i + 3 * stride);
    fold(q0); fold(q1); fold(q2); fold(q3);
  }
  for (; i < total; i += stride) fold(load(i));
  cta_max_to(amax, fused::max_abs_value(m));
}

// eight fp32 values -> eight packed bf16, round to nearest even
__device__ __forceinline__ uint4 round8(const float4& a, const float4& b) {
  auto pack = [](float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  };
  return make_uint4(pack(a.x, a.y), pack(a.z, a.w), pack(b.x, b.y), pack(b.z, b.w));
}

// fp32 -> bf16 copy (contiguous rows) and the plain maximum of the copy in one pass of 6 bytes per element, where a
// cast and amax_plain_kernel move 8.  HBM-bound; two 32-byte reads per thread in flight.
__global__ void __launch_bounds__(512) round_amax_kernel(const float* __restrict__ x, int64_t rows, int vec_per_row,
                                                         int64_t ld, uint16_t* __restrict__ out,
                                                         float* __restrict__ amax) {
  const int64_t total = rows * vec_per_row, stride = (int64_t)gridDim.x * blockDim.x;
  const bool flat = ld == (int64_t)vec_per_row * 8;
  uint32_t m = 0;
  auto src = [&](int64_t i) {
    if (flat) return reinterpret_cast<const float4*>(x) + 2 * i;
    const int64_t r = i / vec_per_row;
    return reinterpret_cast<const float4*>(x + r * ld) + 2 * (i - r * vec_per_row);
  };
  auto fold = [&](int64_t i, const float4& a, const float4& b) {
    const uint4 q = round8(a, b);
    reinterpret_cast<uint4*>(out)[i] = q;
    m = fused::max_abs_word(m, q);
  };
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + stride < total; i += 2 * stride) {
    const float4 *p = src(i), *q = src(i + stride);
    const float4 a0 = __ldg(p), b0 = __ldg(p + 1), a1 = __ldg(q), b1 = __ldg(q + 1);
    fold(i, a0, b0);
    fold(i + stride, a1, b1);
  }
  if (i < total) {
    const float4* p = src(i);
    fold(i, __ldg(p), __ldg(p + 1));
  }
  cta_max_to(amax, fused::max_abs_value(m));
}

// maximum after the Hadamard transform, blocks along the columns: one thread per block
__global__ void __launch_bounds__(256) amax_rht_rows_kernel(const uint16_t* __restrict__ x,
                                                            int64_t rows, int blk_per_row, int64_t ld,
                                                            const float* __restrict__ signs16,
                                                            float* __restrict__ amax) {
  float sg[16];
  load_signs(signs16, sg);
  const int64_t total = rows * blk_per_row;
  float m = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / blk_per_row;
    const int kb = (int)(i - r * blk_per_row);
    const uint4* p = reinterpret_cast<const uint4*>(x + r * ld + (int64_t)kb * 16);
    const uint4 a = __ldg(p), b = __ldg(p + 1);
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    float v[16];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[2 * j] = bf16_lo(w[j]) * sg[2 * j];
      v[2 * j + 1] = bf16_hi(w[j]) * sg[2 * j + 1];
    }
    hadamard16_inplace(v);
#pragma unroll
    for (int j = 0; j < 16; ++j) m = fmaxf(m, fabsf(v[j]));
  }
  cta_max_to(amax, m);
}

// ---------------------------------------------------------------------------------------
// quantizer, blocks along the columns (output describes x itself)
// ---------------------------------------------------------------------------------------
template <bool SR, bool RHT>
__global__ void __launch_bounds__(256) quant_rows_kernel(const uint16_t* __restrict__ x, int64_t rows,
                                                         int blk_per_row, int64_t ld,
                                                         const float* __restrict__ signs16,
                                                         const float* __restrict__ amax,
                                                         const PhiloxKeys keys, uint64_t offset,
                                                         uint8_t* __restrict__ qdata,
                                                         uint8_t* __restrict__ scales,
                                                         float* __restrict__ pts_out,
                                                         uint64_t ctr_pitch, uint64_t ctr_base) {
  // Philox counter of block (row, kb) = row * ctr_pitch + ctr_base + kb: the block's index in the
  // whole tensor when x is a column shard of it (pitch = blocks per row of the whole tensor)
  __shared__ float recip_tab[128];
  const GlobalScale g = global_scale(amax, recip_tab);
  if (blockIdx.x == 0 && threadIdx.x == 0 && pts_out != nullptr) *pts_out = g.pts;
  float sg[16];
  if (RHT) load_signs(signs16, sg);
  const int64_t total = rows * blk_per_row;
  const int64_t col_tiles = (blk_per_row + 3) >> 2;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / blk_per_row;
    const int kb = (int)(i - r * blk_per_row);
    const uint4* p = reinterpret_cast<const uint4*>(x + r * ld + (int64_t)kb * 16);
    const uint4 a = __ldg(p), b = __ldg(p + 1);
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    float v[16];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[2 * j] = bf16_lo(w[j]);
      v[2 * j + 1] = bf16_hi(w[j]);
    }
    if (RHT) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] *= sg[j];
      hadamard16_inplace(v);
    }
    uint32_t lo, hi, sf;
    encode_block<SR>(v, g, (uint64_t)r * ctr_pitch + ctr_base + (uint64_t)kb, keys, offset, lo, hi, sf);
    *reinterpret_cast<uint2*>(qdata + i * 8) = make_uint2(lo, hi);
    scales[sf_offset(r, kb, col_tiles)] = (uint8_t)sf;
  }
}

// The 16-point butterfly of two adjacent columns at once: (v0[i], v1[i]) ride in the two lanes of the
// packed fp32 add / sub / fma, half the instructions of two scalar butterflies and the same bits
// (same operations in the same order as hadamard16_inplace, exact zeros made +0).
__device__ __forceinline__ void hadamard16_pair(float (&v0)[16], float (&v1)[16]) {
#pragma unroll
  for (int s = 1; s < 16; s <<= 1) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if ((i & s) == 0) fused::addsub2(v0[i], v1[i], v0[i | s], v1[i | s]);
    }
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) fused::mul2_poszero(v0[i], v1[i], 0.25f, v0[i], v1[i]);
}

// sign-bit masks of the 16 rows for a packed bf16 pair (both halves of a word belong to one row)
__device__ __forceinline__ void sign_masks(const float (&sg)[16], uint32_t (&sm)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) sm[i] = sg[i] < 0.0f ? 0x80008000u : 0u;
}

// ---------------------------------------------------------------------------------------
// Both maxima of an fp32 matrix's bf16 rounding, which goes to memory on the way (16-byte rows, cols % 8 == 0).  A CTA
// takes tiles of 16 rows x 512 columns the way the activation kernels do (csrc/swiglu.cu): thread t and step k load the
// eight columns 8 * (t % 64) of row 4k + t / 64, the rounded tile goes to padded shared memory, and thread t then
// reads its two columns of all 16 rows from there (consecutive lanes, consecutive banks), with the next tile's loads in
// flight.  bf16 matrices: quantize_dual.cu.
// ---------------------------------------------------------------------------------------
constexpr int kWideCols = 512;
constexpr int kWidePitch = kWideCols / 2 + 4;            // 32-bit words per tile row, padded

struct WideTile {
  int64_t c0, r_base, c;        // first column of the CTA, first row of its 64, this thread's column pair
  int cc, lr;                   // load role: eight columns at cc, row 4k + lr of a tile
  bool col_in, mine;
};
__device__ __forceinline__ WideTile wide_tile(int64_t cols) {
  WideTile t;
  t.c0 = (int64_t)blockIdx.x * kWideCols;
  t.r_base = (int64_t)blockIdx.y * 64;
  t.cc = (threadIdx.x & 63) * 8;
  t.lr = threadIdx.x >> 6;
  t.col_in = t.c0 + t.cc < cols;
  t.c = t.c0 + 2 * (int64_t)threadIdx.x;
  t.mine = t.c < cols;
  return t;
}
__device__ __forceinline__ void wide_stage(uint32_t* tile, const WideTile& t, const uint4 (&d)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(&tile[(4 * k + t.lr) * kWidePitch + (t.cc >> 1)]) = d[k];
}

// The same tile out of an fp32 matrix, rounded to bf16 on the way (and written to `out`, contiguous rows).
__device__ __forceinline__ void wide_fetch_round(const float* __restrict__ x, int64_t rows, int64_t cols, int64_t ld,
                                                 const WideTile& t, int j, uint16_t* __restrict__ out, uint4 (&d)[4]) {
  float4 a[4], b[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t r = t.r_base + 16 * j + 4 * k + t.lr;
    const bool in = t.col_in && r < rows;
    const float4* p = reinterpret_cast<const float4*>(x + r * ld + t.c0 + t.cc);
    a[k] = in ? __ldg(p) : make_float4(0.f, 0.f, 0.f, 0.f);
    b[k] = in ? __ldg(p + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t r = t.r_base + 16 * j + 4 * k + t.lr;
    d[k] = round8(a[k], b[k]);
    if (t.col_in && r < rows) *reinterpret_cast<uint4*>(out + r * cols + t.c0 + t.cc) = d[k];
  }
}

// out[0] = plain maximum, out[1] = maximum after the transform
__global__ void __launch_bounds__(256) round_amax_both_kernel(const float* __restrict__ x, int64_t rows, int64_t cols,
                                                              int64_t ld, const float* __restrict__ signs16,
                                                              float* __restrict__ out, uint16_t* __restrict__ rounded) {
  __shared__ __align__(16) uint32_t tile[16 * kWidePitch];
  float sg[16];
  load_signs(signs16, sg);
  uint32_t sm[16];
  sign_masks(sg, sm);
  const WideTile t = wide_tile(cols);
  float m = 0.0f;
  uint32_t mp = 0u;
  uint4 nxt[4];
  wide_fetch_round(x, rows, cols, ld, t, 0, rounded, nxt);
#pragma unroll 1
  for (int j = 0; j < 4; ++j) {
    if (t.r_base + 16 * j >= rows) break;                  // uniform over the CTA
    wide_stage(tile, t, nxt);
#pragma unroll
    for (int k = 0; k < 4; ++k) mp = fused::max_abs_word(mp, nxt[k]);
    if (j + 1 < 4) wide_fetch_round(x, rows, cols, ld, t, j + 1, rounded, nxt);
    __syncthreads();
    if (t.mine) {
      float v0[16], v1[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint32_t u = tile[i * kWidePitch + threadIdx.x] ^ sm[i];
        v0[i] = bf16_lo(u);
        v1[i] = bf16_hi(u);
      }
      hadamard16_pair(v0, v1);
#pragma unroll
      for (int i = 0; i < 16; ++i) m = fmaxf(m, fmaxf(fabsf(v0[i]), fabsf(v1[i])));
    }
    __syncthreads();
  }
  cta_max_to(out, fused::max_abs_value(mp), 0);
  cta_max_to(out + 1, m, 1);
}

// ---------------------------------------------------------------------------------------
// weights under 16 x 16 scaling: both layouts from one read.  A CTA takes a 64 x 64 tile of w [rows, cols]; thread
// (row t / 4, segment t % 4) loads the 16 elements of row-wise block (row, segment) and leaves them in
// a padded shared tile, from which thread (column t % 64, row block t / 64) reads the 16 elements of
// column-wise block (column, row block).  Round to nearest.  One scale per 16 x 16 tile is shared by the row-wise and
// the column-wise blocks that cross it, so that both quantized layouts hold the same values (the reference
// simulator's weight scaling, nvfp4_validate.py:68-82).  1 x 16 scaling is quantize_dual.cu.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) quant_weight_2d_kernel(const uint16_t* __restrict__ w, int64_t rows, int64_t cols,
                                                              int64_t ld, const float* __restrict__ amax,
                                                              uint8_t* __restrict__ q_rows, uint8_t* __restrict__ sf_rows,
                                                              uint8_t* __restrict__ q_cols, uint8_t* __restrict__ sf_cols,
                                                              float* __restrict__ pts_out) {
  __shared__ uint16_t tile[64][66];          // 33 words per row: a column walk touches 16 different banks
  __shared__ float bmax[64][4];              // row-wise block maxima of the tile
  __shared__ float tmax[4][4];               // 16 x 16 tile maxima
  __shared__ float recip_tab[128];
  const GlobalScale g = global_scale(amax, recip_tab);
  const PhiloxKeys keys{};                   // round to nearest: unused
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && pts_out != nullptr) *pts_out = g.pts;
  const int t = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.y * 64, c0 = (int64_t)blockIdx.x * 64;
  // ---- load: row-wise block (r, seg) ----
  const int r = t >> 2, seg = t & 3;
  const int64_t gr = r0 + r, gc = c0 + seg * 16;
  const bool have = gr < rows && gc < cols;          // rows and cols are multiples of 16: a block is whole or absent
  uint32_t wv[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  if (have) {
    const uint4* p = reinterpret_cast<const uint4*>(w + gr * ld + gc);
    const uint4 a = __ldg(p), b = __ldg(p + 1);
    wv[0] = a.x; wv[1] = a.y; wv[2] = a.z; wv[3] = a.w; wv[4] = b.x; wv[5] = b.y; wv[6] = b.z; wv[7] = b.w;
  }
  float v[16];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[2 * j] = bf16_lo(wv[j]);
    v[2 * j + 1] = bf16_hi(wv[j]);
    *reinterpret_cast<uint32_t*>(&tile[r][seg * 16 + 2 * j]) = wv[j];
  }
  bmax[r][seg] = block_amax16(v);
  __syncthreads();
  if (t < 16) {
    const int rb = t >> 2, cb = t & 3;
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) m = fmaxf(m, bmax[rb * 16 + i][cb]);
    tmax[rb][cb] = m;
  }
  __syncthreads();
  // ---- row-wise output ----
  if (have) {
    uint32_t lo, hi, sf;
    encode_block_scaled<false>(v, tmax[r >> 4][seg], g, 0, keys, 0, lo, hi, sf);
    const int64_t kb = gc >> 4;
    *reinterpret_cast<uint2*>(q_rows + gr * (cols >> 1) + kb * 8) = make_uint2(lo, hi);
    sf_rows[sf_offset(gr, kb, ((cols >> 4) + 3) >> 2)] = (uint8_t)sf;
  }
  // ---- column-wise output: block (column c, row block rb) ----
  const int c = t & 63, rb = t >> 6;
  const int64_t oc = c0 + c, orow0 = r0 + rb * 16;
  if (oc < cols && orow0 < rows) {
    float u[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) u[i] = __uint_as_float((uint32_t)tile[rb * 16 + i][c] << 16);
    uint32_t lo, hi, sf;
    encode_block_scaled<false>(u, tmax[rb][c >> 4], g, 0, keys, 0, lo, hi, sf);
    const int64_t kb = orow0 >> 4;
    *reinterpret_cast<uint2*>(q_cols + oc * (rows >> 1) + kb * 8) = make_uint2(lo, hi);
    sf_cols[sf_offset(oc, kb, ((rows >> 4) + 3) >> 2)] = (uint8_t)sf;
  }
}


static inline int grid_for(int64_t work_items, int threads, int max_blocks) {
  int64_t b = (work_items + threads - 1) / threads;
  if (b > max_blocks) b = max_blocks;
  if (b < 1) b = 1;
  return (int)b;
}

}  // namespace nvfp4

using namespace nvfp4;

static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

namespace nvfp4 { namespace dual {
int launch_amax(const void* x, int64_t rows, int64_t cols, int64_t ld, const float* signs16, bool both, float* out,
                cudaStream_t stream);
int launch(const void* x, int64_t rows, int64_t cols, int64_t ld, int rows_mode, bool sr_c, const float* signs16,
           const float* amax_r, const float* amax_c, uint64_t seed_r, uint64_t seed_c, uint64_t offset,
           const uint64_t* counters4, uint8_t* q_r, uint8_t* sf_r, float* pts_r, uint8_t* q_c, uint8_t* sf_c, float* pts_c,
           cudaStream_t stream);
}}
extern "C" int nvfp4_amax_bf16(const void* x, int64_t rows, int64_t cols, int64_t ld, int rht,
                               int transpose, const float* signs16, float* amax, int zero_first,
                               void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (x == nullptr || amax == nullptr || (rht && signs16 == nullptr)) return NVFP4_E_NULL;
  if (rows <= 0 || cols <= 0 || ld < cols) return NVFP4_E_SHAPE;
  if (!aligned16(x) || (ld & 7) != 0 || (rht && !aligned16(signs16))) return NVFP4_E_ALIGN;
  if (zero_first && cudaMemsetAsync(amax, 0, sizeof(float), stream) != cudaSuccess) return NVFP4_E_LAUNCH;
  const uint16_t* xp = static_cast<const uint16_t*>(x);
  if (!rht) {
    if ((cols & 7) != 0) return NVFP4_E_SHAPE;
    const int vpr = (int)(cols >> 3);
    amax_plain_kernel<<<grid_for(rows * vpr, 512 * 8, 148 * 4), 512, 0, stream>>>(xp, rows, vpr, ld, amax);
  } else if (!transpose) {
    if ((cols & 15) != 0) return NVFP4_E_SHAPE;
    const int bpr = (int)(cols >> 4);
    amax_rht_rows_kernel<<<grid_for(rows * bpr, 256 * 2, 148 * 16), 256, 0, stream>>>(xp, rows, bpr, ld, signs16, amax);
  } else {
    if ((rows & 15) != 0 || (cols & 1) != 0) return NVFP4_E_SHAPE;
    if ((rows + 63) / 64 > 65535) return NVFP4_E_SHAPE;
    return nvfp4::dual::launch_amax(x, rows, cols, ld, signs16, false, amax, stream);
  }
  return cudaGetLastError() == cudaSuccess ? NVFP4_OK : NVFP4_E_LAUNCH;
}

namespace nvfp4 { namespace fused {
int quantize_rows_known_amax(const void* x, int64_t rows, int64_t cols, int64_t ld, int mode, int rht,
                             const float* signs16, const float* amax, uint64_t seed, uint64_t offset,
                             uint64_t counter_pitch, uint64_t counter_base,
                             uint8_t* qdata, uint8_t* scales, float* pts_out, cudaStream_t stream);
}}

extern "C" int nvfp4_quantize_shard_bf16(const void* x, int64_t rows, int64_t cols, int64_t ld, int transpose,
                                         int mode, int rht, const float* signs16, const float* amax,
                                         uint64_t seed, uint64_t offset, uint64_t counter_pitch, uint64_t counter_base,
                                         uint8_t* qdata, uint8_t* scales, float* pts_out, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (x == nullptr || amax == nullptr || qdata == nullptr || scales == nullptr || (rht && signs16 == nullptr))
    return NVFP4_E_NULL;
  if (rows <= 0 || cols <= 0 || ld < cols) return NVFP4_E_SHAPE;
  if (mode != NVFP4_ROUND_NEAREST && mode != NVFP4_ROUND_STOCHASTIC) return NVFP4_E_MODE;
  if (!aligned16(x) || (ld & 7) != 0 || (reinterpret_cast<uintptr_t>(qdata) & 15u) != 0 ||
      (reinterpret_cast<uintptr_t>(scales) & 15u) != 0 || (rht && !aligned16(signs16)))
    return NVFP4_E_ALIGN;
  if (((transpose ? rows : cols) & 15) != 0) return NVFP4_E_SHAPE;
  if (transpose && (cols & 1) != 0) return NVFP4_E_SHAPE;
  const bool sr = mode == NVFP4_ROUND_STOCHASTIC;
  if (transpose) {
    if ((rows + 63) / 64 > 65535) return NVFP4_E_SHAPE;
    const uint64_t ctr[4] = {0, 0, counter_pitch, counter_base};
    return nvfp4::dual::launch(x, rows, cols, ld, 0, sr, rht ? signs16 : nullptr, nullptr, amax, 0, seed, offset, ctr,
                               nullptr, nullptr, nullptr, qdata, scales, pts_out, stream);
  }
  // row-wise output with the maximum given: one streaming pass of the single-launch kernel's
  // quantize phase (it declines only tensors of 2^31 blocks or more, which the plain kernel takes)
  const int rc = nvfp4::fused::quantize_rows_known_amax(x, rows, cols, ld, mode, rht, signs16, amax, seed, offset,
                                                        counter_pitch, counter_base, qdata, scales, pts_out, stream);
  if (rc != NVFP4_E_LIMIT) return rc;
  // padding of the tiled scale buffer must read as zero (the reference pads with zeros)
  const int64_t sm = (rows + 127) / 128 * 128, sk = (cols / 16 + 3) / 4 * 4;
  if (sm != rows || sk != cols / 16) {
    if (cudaMemsetAsync(scales, 0, (size_t)(sm * sk), stream) != cudaSuccess) return NVFP4_E_LAUNCH;
  }
  const uint16_t* xp = static_cast<const uint16_t*>(x);
  const PhiloxKeys keys = make_philox_keys(seed);
  const int bpr = (int)(cols >> 4);
  const int grid = grid_for(rows * bpr, 256, 1 << 30);
#define NVFP4_LAUNCH_ROWS(SR_, RHT_) \
  quant_rows_kernel<SR_, RHT_><<<grid, 256, 0, stream>>>(xp, rows, bpr, ld, signs16, amax, keys, offset, qdata, scales, pts_out, counter_pitch, counter_base)
  if (sr && rht) NVFP4_LAUNCH_ROWS(true, true);
  else if (sr) NVFP4_LAUNCH_ROWS(true, false);
  else if (rht) NVFP4_LAUNCH_ROWS(false, true);
  else NVFP4_LAUNCH_ROWS(false, false);
#undef NVFP4_LAUNCH_ROWS
  return cudaGetLastError() == cudaSuccess ? NVFP4_OK : NVFP4_E_LAUNCH;
}


extern "C" int nvfp4_quantize_weight_bf16(const void* w, int64_t rows, int64_t cols, int64_t ld, int two_d,
                                          const float* amax, uint8_t* qdata_rows, uint8_t* scales_rows,
                                          uint8_t* qdata_cols, uint8_t* scales_cols, float* pts_out, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!w || !amax || !qdata_rows || !scales_rows || !qdata_cols || !scales_cols) return NVFP4_E_NULL;
  if (rows <= 0 || cols <= 0 || ld < cols || (rows & 15) != 0 || (cols & 15) != 0) return NVFP4_E_SHAPE;
  if (!aligned16(w) || (ld & 7) != 0 || !aligned16(qdata_rows) || !aligned16(qdata_cols) || !aligned16(scales_rows) ||
      !aligned16(scales_cols))
    return NVFP4_E_ALIGN;
  if ((rows + 63) / 64 > 65535) return NVFP4_E_LIMIT;
  if (!two_d) {
    const uint64_t ctr[4] = {0, 0, 0, 0};                       // round to nearest: unused
    return nvfp4::dual::launch(w, rows, cols, ld, 1, false, nullptr, amax, amax, 0, 0, 0, ctr, qdata_rows, scales_rows,
                               pts_out, qdata_cols, scales_cols, nullptr, stream);
  }
  // padding of the tiled scale buffers must read as zero
  auto clear_if_padded = [&](uint8_t* sf, int64_t m, int64_t k) {
    const int64_t sm = (m + 127) / 128 * 128, sk = (k / 16 + 3) / 4 * 4;
    if (sm == m && sk == k / 16) return true;
    return cudaMemsetAsync(sf, 0, (size_t)(sm * sk), stream) == cudaSuccess;
  };
  if (!clear_if_padded(scales_rows, rows, cols) || !clear_if_padded(scales_cols, cols, rows)) return NVFP4_E_LAUNCH;
  const dim3 grid((unsigned)((cols + 63) / 64), (unsigned)((rows + 63) / 64));
  quant_weight_2d_kernel<<<grid, 256, 0, stream>>>(static_cast<const uint16_t*>(w), rows, cols, ld, amax, qdata_rows,
                                                   scales_rows, qdata_cols, scales_cols, pts_out);
  return cudaGetLastError() == cudaSuccess ? NVFP4_OK : NVFP4_E_LAUNCH;
}


extern "C" int nvfp4_amax_both_bf16(const void* x, int64_t rows, int64_t cols, int64_t ld, const float* signs16,
                                    float* maxima2, int zero_first, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!x || !signs16 || !maxima2) return NVFP4_E_NULL;
  if (rows <= 0 || cols <= 0 || ld < cols || (rows & 15) != 0 || (cols & 1) != 0) return NVFP4_E_SHAPE;
  if (!aligned16(x) || (ld & 7) != 0 || !aligned16(signs16)) return NVFP4_E_ALIGN;
  if (zero_first && cudaMemsetAsync(maxima2, 0, 2 * sizeof(float), stream) != cudaSuccess) return NVFP4_E_LAUNCH;
  if ((rows + 63) / 64 > 65535) return NVFP4_E_LIMIT;
  return nvfp4::dual::launch_amax(x, rows, cols, ld, signs16, true, maxima2, stream);
}

extern "C" int nvfp4_round_amax_f32(const float* x, int64_t rows, int64_t cols, int64_t ld, void* out_bf16,
                                    const float* signs16, float* maxima, int zero_first, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!x || !out_bf16 || !maxima) return NVFP4_E_NULL;
  if (rows <= 0 || cols <= 0 || ld < cols || (cols & 7) != 0 || (signs16 != nullptr && (rows & 15) != 0)) return NVFP4_E_SHAPE;
  if (!aligned16(x) || (ld & 3) != 0 || !aligned16(out_bf16) || (signs16 != nullptr && !aligned16(signs16)))
    return NVFP4_E_ALIGN;
  if ((rows + 63) / 64 > 65535 || cols / 8 > 0x7fffffffLL) return NVFP4_E_LIMIT;
  const size_t words = signs16 != nullptr ? 2 : 1;
  if (zero_first && cudaMemsetAsync(maxima, 0, words * sizeof(float), stream) != cudaSuccess) return NVFP4_E_LAUNCH;
  uint16_t* out = static_cast<uint16_t*>(out_bf16);
  if (signs16 != nullptr) {
    const dim3 grid((unsigned)((cols + kWideCols - 1) / kWideCols), (unsigned)((rows + 63) / 64));
    round_amax_both_kernel<<<grid, 256, 0, stream>>>(x, rows, cols, ld, signs16, maxima, out);
  } else {
    const int vpr = (int)(cols >> 3);
    round_amax_kernel<<<grid_for(rows * vpr, 512 * 2, 148 * 4), 512, 0, stream>>>(x, rows, vpr, ld, out, maxima);
  }
  return cudaGetLastError() == cudaSuccess ? NVFP4_OK : NVFP4_E_LAUNCH;
}

extern "C" int nvfp4_quantize_dual_bf16(const void* x, int64_t rows, int64_t cols, int64_t ld, int mode_rows,
                                        int mode_cols, const float* signs16, const float* amax_rows,
                                        const float* amax_cols, uint64_t seed_rows, uint64_t seed_cols, uint64_t offset,
                                        const uint64_t* counters4, uint8_t* qdata_rows, uint8_t* scales_rows,
                                        float* pts_rows, uint8_t* qdata_cols, uint8_t* scales_cols, float* pts_cols,
                                        void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!x || !signs16 || !amax_rows || !amax_cols || !qdata_rows || !scales_rows || !qdata_cols || !scales_cols)
    return NVFP4_E_NULL;
  if (rows <= 0 || cols <= 0 || ld < cols || (rows & 15) != 0 || (cols & 15) != 0) return NVFP4_E_SHAPE;
  auto bad_mode = [](int m) { return m != NVFP4_ROUND_NEAREST && m != NVFP4_ROUND_STOCHASTIC; };
  if (bad_mode(mode_rows) || bad_mode(mode_cols)) return NVFP4_E_MODE;
  if (!aligned16(x) || (ld & 7) != 0 || !aligned16(qdata_rows) || !aligned16(qdata_cols) || !aligned16(scales_rows) ||
      !aligned16(scales_cols) || !aligned16(signs16))
    return NVFP4_E_ALIGN;
  uint64_t ctr[4] = {(uint64_t)(cols >> 4), 0, (uint64_t)(rows >> 4), 0};      // pitch, base of rows / cols: a whole tensor
  if (counters4 != nullptr)
    for (int i = 0; i < 4; ++i) ctr[i] = counters4[i];
  // the hardware draws from a 32-bit counter word pair; keep both layouts' counters inside 2^64 trivially,
  // and inside the documented 2^32 blocks per tensor
  if ((uint64_t)rows * ctr[0] + ctr[1] >= (1ull << 32) || (uint64_t)cols * ctr[2] + ctr[3] >= (1ull << 32))
    return NVFP4_E_LIMIT;
  if ((rows + 63) / 64 > 65535) return NVFP4_E_LIMIT;
  return nvfp4::dual::launch(x, rows, cols, ld, mode_rows == NVFP4_ROUND_STOCHASTIC ? 2 : 1,
                             mode_cols == NVFP4_ROUND_STOCHASTIC, signs16, amax_rows, amax_cols, seed_rows, seed_cols,
                             offset, ctr, qdata_rows, scales_rows, pts_rows, qdata_cols, scales_cols, pts_cols, stream);
}

extern "C" int nvfp4_quantize_bf16(const void* x, int64_t rows, int64_t cols, int64_t ld, int transpose,
                                   int mode, int rht, const float* signs16, const float* amax,
                                   uint64_t seed, uint64_t offset, uint8_t* qdata, uint8_t* scales,
                                   float* pts_out, void* stream_) {
  // the tensor is whole: a block's counter is its index in x (or in x^T): out_row * (K / 16) + k / 16
  const uint64_t pitch = (uint64_t)((transpose ? rows : cols) / 16);
  return nvfp4_quantize_shard_bf16(x, rows, cols, ld, transpose, mode, rht, signs16, amax, seed, offset, pitch, 0,
                                   qdata, scales, pts_out, stream_);
}
