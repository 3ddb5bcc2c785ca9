// Quantizers whose output describes x^T (blocks along the ROWS of x), alone or together with the row-wise output
// of the same tensor, maxima given (sm_100a).
//
// What they serve: the transposed operands W^T, dY^T, X^T of FP4Linear (nvfp4_train.py:36-55) and every tensor that
// is wanted in both layouts at once.  One persistent kernel walks over tiles of 128 rows x 128 columns of x.  A tile
// arrives as two TMA tensor copies (128 x 64 elements, 128-byte swizzle, out-of-range elements read as zero) in one
// of two 32 KiB slots; the next tile's copies are in flight while this one is encoded.
//   row-wise     a lane takes a 16-element block: a warp covers rows {2w, 2w+1} + 32 g of a 128 x 64 half, so its 32
//                scale bytes are one sector of the tiled layout and its codes eight full sectors
//   transposed   a lane takes the 16 rows of two adjacent columns (a warp reads one 128-byte row of the half per
//                instruction, no bank conflicts); the Hadamard butterflies of the two columns ride in the two lanes
//                of packed fp32 instructions.  Codes and scales are collected in shared memory and leave as 64
//                contiguous bytes per output row (two full sectors) and 1024 contiguous scale bytes.
// A tensor of fewer tiles than the chip holds CTAs is cut finer: one CTA takes a tile's row-wise output, another its
// transposed one (512 x 768, both stochastic: 6.0 -> 4.7 us when this was decided; the whole tile per CTA wins once the
// grid is full).
// What bounds it: instruction issue and the barrier per tile, not memory: 255 warp instructions per 32 blocks with Philox
// and the butterfly, issue slots 64 % busy, ALU pipe 47 %, heavy FMA pipe 47 %, DRAM 34 % (4096 x 14336 transposed).
// Measured, maxima given, HBM-cold, us (before = one 64 x 64 tile per 256-thread CTA, and for the transposed output alone
// two columns x 64 rows per thread straight from global memory):
//   4096 x 28672   transposed nearest 68.2 -> 49.6, RHT 74.6 -> 59.0, RHT + stochastic 87.9 -> 78.3; both layouts
//                  nearest 169.6 -> 95.7, stochastic 192.5 -> 137.5; a weight in both layouts 123.7 -> 82.9
//   16384 x 768    transposed RHT + stochastic 17.2 -> 13.2, both layouts stochastic 24.4 -> 20.5
//   512 x 768      transposed RHT + stochastic 6.6 -> 3.9, both layouts stochastic 4.0 -> 4.1, a weight 3.1 -> 3.4
// Rows and columns outside the matrix get zero scale bytes, so the padding of the scale buffers needs no clearing.
#include <mutex>

#include "quantize_common.cuh"
#include "gemm_common.cuh"      // encode_fn(): the driver's tensor-map encoder, looked up once

namespace nvfp4 {
namespace dual {

using fused::PhiloxKeys;

constexpr int kTile = 128;                        // rows and columns of x per tile
constexpr int kThreads = 512;
constexpr int kHalfBytes = kTile * 128;           // 128 rows x 64 columns
constexpr int kSlotBytes = 2 * kHalfBytes;
constexpr int kSlots = 2;
constexpr int kOutPitch = 72;                     // 64 bytes of codes per output row, padded: 4 wavefronts per store
constexpr int kOutBytes = kTile * kOutPitch + 1024;   // codes and scales of one tile's transposed output
constexpr int kMiscOff = kSlots * kSlotBytes + 2 * kOutBytes;
constexpr int kSmemBytes = kMiscOff + 1280 /* tables, signs, barriers */ + 1024 /* alignment slack */;

struct Params {
  int64_t rows, cols;
  uint32_t ntc, nunits;          // column tiles per row of tiles; units of work in all
  uint32_t split;                // 0: a unit is a tile; 1: units 2t and 2t + 1 are tile t's transposed and row-wise output
  const float* signs16;
  const float* amax_r;
  const float* amax_c;
  PhiloxKeys keys_r, keys_c;
  uint64_t offset;
  uint64_t pitch_r, base_r, pitch_c, base_c;      // Philox counter of a block = out_row * pitch + base + k_block
  uint8_t* q_r;
  uint8_t* sf_r;
  float* pts_r;
  uint8_t* q_c;
  uint8_t* sf_c;
  float* pts_c;
  unsigned long long wait_limit_ns;
  uint32_t extra_arrivals;       // test hook (normally 0): what the barriers of the copies expect beside the copies
};

__device__ __forceinline__ void tma_half_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}

__device__ __forceinline__ fused::Scale global_scale(float amax) {
  fused::Scale s;
  s.pts = __fdiv_rn(fmaxf(amax, kAmaxFloor), kGlobalDiv);
  s.inv_pts = __fdiv_rn(1.0f, s.pts);
  s.c = __fdiv_rn(1.0f, kF4Max * s.pts);
  return s;
}

// d[16] = the scaled values of a block -> codes
template <bool SR>
__device__ __forceinline__ void encode(const float (&d)[16], uint64_t counter, const PhiloxKeys& keys, uint64_t offset,
                                       uint32_t& lo, uint32_t& hi) {
  if (SR) {
    const Philox4 r = fused::philox_rounds((uint32_t)counter, (uint32_t)(counter >> 32), (uint32_t)offset,
                                           (uint32_t)(offset >> 32), keys);
    lo = e2m1x4_rs(d[0], d[1], d[2], d[3], r.x) | (e2m1x4_rs(d[4], d[5], d[6], d[7], r.y) << 16);
    hi = e2m1x4_rs(d[8], d[9], d[10], d[11], r.z) | (e2m1x4_rs(d[12], d[13], d[14], d[15], r.w) << 16);
  } else {
    lo = fused::e2m1x8_rn(d);
    hi = fused::e2m1x8_rn(d + 8);
  }
}

// ROWS: 0 no row-wise output, 1 round to nearest, 2 stochastic.  SR_C, RHT: rounding and random-sign Hadamard (along
// the rows of x) of the transposed output.
template <int ROWS, bool SR_C, bool RHT>
__global__ void __launch_bounds__(kThreads, 2)
quant_dual_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = fused::smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);          // the swizzle wants 1024-byte alignment
  float* recip_r = reinterpret_cast<float*>(smem + kMiscOff);            // 128 floats each
  float* recip_c = recip_r + 128;
  uint32_t* sgn = reinterpret_cast<uint32_t*>(recip_c + 128);            // 16 sign-flip masks
  const uint32_t bars = fused::smem_u32(sgn + 16);
  volatile int* gave_up = reinterpret_cast<volatile int*>(sgn + 16 + 2 * kSlots);

  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t my_tiles = blockIdx.x < p.nunits ? (p.nunits - blockIdx.x + gridDim.x - 1u) / gridDim.x : 0u;
  auto locate = [&](uint32_t i, int64_t& r0, int64_t& c0) {
    const uint32_t tile = (blockIdx.x + i * gridDim.x) >> p.split, rt = tile / p.ntc;
    r0 = (int64_t)rt * kTile;
    c0 = (int64_t)(tile - rt * p.ntc) * kTile;
  };
  auto fetch = [&](uint32_t i) {                  // one thread: both halves of this CTA's tile i into slot i % kSlots
    int64_t r0, c0;
    locate(i, r0, c0);
    const uint32_t s = i % kSlots, bar = bars + 8u * s, dst = fused::smem_u32(smem) + s * kSlotBytes;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)kSlotBytes) : "memory");
    tma_half_load(dst, &map_x, (int)c0, (int)r0, bar);
    tma_half_load(dst + kHalfBytes, &map_x, (int)(c0 + 64), (int)r0, bar);
  };
  if (tid == 0) {
    for (int s = 0; s < kSlots; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bars + 8u * s), "r"(1u + p.extra_arrivals));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *gave_up = 0;
    for (uint32_t i = 0; i < (uint32_t)kSlots && i < my_tiles; ++i) fetch(i);
  }
  // scales and tables while the first tiles arrive
  const fused::Scale sc_c = global_scale(__ldg(p.amax_c));
  fused::Scale sc_r = sc_c;
  if (ROWS) sc_r = global_scale(__ldg(p.amax_r));
  // The transform is butterfly / 4.  The quarter is folded into the reciprocals (an exact scaling) unless that could
  // make one a denormal: then (maxima above 1e38) the values take it.
  const bool fold = !RHT || sc_c.inv_pts >= 4.0f * kE4M3Max * 1.17549435e-38f;
  const float rht_scale = RHT && fold ? 0.25f : 1.0f;
  if (tid < 128) recip_c[tid] = __fdiv_rn(sc_c.inv_pts, e4m3_to_f32(tid)) * rht_scale;
  else if (ROWS && tid < 256) recip_r[tid - 128] = __fdiv_rn(sc_r.inv_pts, e4m3_to_f32(tid - 128));
  else if (RHT && tid >= 256 && tid < 272) sgn[tid - 256] = __ldg(p.signs16 + (tid - 256)) < 0.0f ? 0x80000000u : 0u;
  if (blockIdx.x == 0 && tid == 0) {
    if (p.pts_c != nullptr) *p.pts_c = sc_c.pts;
    if (ROWS && p.pts_r != nullptr) *p.pts_r = sc_r.pts;
  }
  __syncthreads();

  const int64_t blk_r = p.cols >> 4, blk_c = p.rows >> 4;               // blocks per output row of the two layouts
  const int64_t ct_r = (blk_r + 3) >> 2, ct_c = (blk_c + 3) >> 2;       // scale tiles per 128 output rows
  for (uint32_t i = 0; i < my_tiles; ++i) {
    int64_t r0, c0;
    locate(i, r0, c0);
    const uint32_t slot_off = (i % kSlots) * kSlotBytes, bar = bars + 8u * (i % kSlots);
    if (!fused::wait_copy(bar, (i / kSlots) & 1u, p.wait_limit_ns)) { *gave_up = 1; atomicCAS(&fused::g_wait_error, 0, 2); }
    const uint8_t* slot = smem + slot_off;
    uint8_t* out = smem + kSlots * kSlotBytes + (i & 1u) * kOutBytes;
    uint8_t* out_sf = out + kTile * kOutPitch;

    const uint32_t part = (blockIdx.x + i * gridDim.x) & p.split;
    const bool do_cols = ROWS == 0 || part == 0, do_rows = p.split == 0 || part != 0;
    // ---- transposed: this warp's half and 16-row block, two columns per lane
    if (do_cols) {
      const uint32_t half = warp & 1u, rb = warp >> 1;
      // 128-byte swizzle: 16-byte chunk c of row k sits at c ^ (k & 7)
      const uint32_t addr = fused::smem_u32(slot) + half * kHalfBytes + rb * 2048u + lane * 4u;
      float v0[16], v1[16];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 m4 = make_uint4(0u, 0u, 0u, 0u);
        if (RHT) m4 = reinterpret_cast<const uint4*>(sgn)[q];
        const uint32_t m[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int k = 4 * q + e;
          uint32_t w;
          asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"((addr ^ ((uint32_t)(k & 7) << 4)) + 128 * k));
          v0[k] = __uint_as_float((w << 16) + m[e]);                     // adding the top bit flips the sign: one
          v1[k] = __uint_as_float((w & 0xffff0000u) ^ m[e]);             // instruction each with the unpacking
        }
      }
      if (RHT) {
#pragma unroll
        for (int s = 1; s < 16; s <<= 1) {
#pragma unroll
          for (int k = 0; k < 16; ++k)
            if ((k & s) == 0) fused::addsub2(v0[k], v1[k], v0[k | s], v1[k | s]);
        }
        if (!fold) {
#pragma unroll
          for (int k = 0; k < 16; ++k) fused::mul2(v0[k], v1[k], 0.25f, v0[k], v1[k]);
        }
      }
      const int64_t kb = (r0 >> 4) + rb;
      const uint32_t c = half * 64u + 2u * lane;                         // column inside the tile
      const uint64_t ctr = (uint64_t)(c0 + c) * p.pitch_c + p.base_c + (uint64_t)kb;
      // both columns' values stay paired up to the conversion
      const uint32_t sf0 = fused::block_scale_byte(fused::max_abs16(v0) * rht_scale, sc_c);
      const uint32_t sf1 = fused::block_scale_byte(fused::max_abs16(v1) * rht_scale, sc_c);
      const float rc0 = recip_c[sf0], rc1 = recip_c[sf1];
#pragma unroll
      for (int k = 0; k < 16; ++k) {                                     // an exact zero that left the butterfly as -0: +0
        if (RHT) fused::mul2_pair_poszero(v0[k], v1[k], rc0, rc1, v0[k], v1[k]);
        else fused::mul2_pair(v0[k], v1[k], rc0, rc1, v0[k], v1[k]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t lo, hi;
        encode<SR_C>(h ? v1 : v0, ctr + (h ? p.pitch_c : 0ull), p.keys_c, p.offset, lo, hi);
        *reinterpret_cast<uint2*>(out + (c + h) * kOutPitch + rb * 8u) = make_uint2(lo, hi);
        const bool inside = c0 + c + h < p.cols && kb < blk_c;
        out_sf[(rb >> 2) * 512u + ((c + h) & 31u) * 16u + ((c + h) >> 5) * 4u + (rb & 3u)] =
            inside ? (uint8_t)(h ? sf1 : sf0) : (uint8_t)0;
      }
    }
    // ---- row-wise: blocks (row_t, kb) of the two halves
    if (ROWS && do_rows) {
      const uint32_t kb4 = lane & 3u, hrow = (lane >> 2) & 1u, grp = lane >> 3;
      const uint32_t row_t = 2u * warp + hrow + 32u * grp;
      const uint32_t off0 = row_t * 128u + (((2u * kb4) ^ (row_t & 7u)) << 4);
      const uint32_t off1 = row_t * 128u + (((2u * kb4 + 1u) ^ (row_t & 7u)) << 4);
      const int64_t r = r0 + row_t;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (c0 + 64 * half >= p.cols) break;                             // no such scale tile (uniform)
        const int64_t kb = (c0 >> 4) + 4 * half + kb4;
        const uint4 a = *reinterpret_cast<const uint4*>(slot + half * kHalfBytes + off0);
        const uint4 b = *reinterpret_cast<const uint4*>(slot + half * kHalfBytes + off1);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        float v[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) { v[2 * j] = bf16_lo(w[j]); v[2 * j + 1] = bf16_hi(w[j]); }
        uint32_t lo, hi;
        const uint32_t sf = fused::block_scale_byte(fused::amax_packed8(w), sc_r);
        const float recip = recip_r[sf];
#pragma unroll
        for (int j = 0; j < 8; ++j) fused::mul2(v[2 * j], v[2 * j + 1], recip, v[2 * j], v[2 * j + 1]);
        encode<ROWS == 2>(v, (uint64_t)r * p.pitch_r + p.base_r + (uint64_t)kb, p.keys_r, p.offset, lo, hi);
        const bool inside = r < p.rows && kb < blk_r;
        if (inside) *reinterpret_cast<uint2*>(p.q_r + r * (p.cols >> 1) + kb * 8) = make_uint2(lo, hi);
        p.sf_r[((r0 >> 7) * ct_r + (c0 >> 6) + half) * 512 + (2u * warp + hrow) * 16u + grp * 4u + kb4] =
            inside ? (uint8_t)sf : (uint8_t)0;
      }
    }
    __syncthreads();                                                     // the slot is read, the output collected
    // (every copy in flight was issued before the wait that gave up began, so it has had the limit to land)
    if (*gave_up != 0) return;
    if (tid == 0 && i + kSlots < my_tiles) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // generic reads before the async write
      fetch(i + kSlots);
    }
    // ---- transposed output: thread t writes 16 of the 64 bytes of output row t / 4; 64 threads write the scales
    if (do_cols) {
      const uint32_t row = tid >> 2, b16 = (tid & 3u) * 16u;
      const int64_t oc = c0 + row, k_byte = (r0 >> 1) + b16, out_ld = p.rows >> 1;
      if (oc < p.cols && k_byte < out_ld) {
        const uint2 a = *reinterpret_cast<const uint2*>(out + row * kOutPitch + b16);
        const uint2 b = *reinterpret_cast<const uint2*>(out + row * kOutPitch + b16 + 8);
        uint8_t* dst = p.q_c + oc * out_ld + k_byte;
        if ((out_ld & 15) == 0) {
          *reinterpret_cast<uint4*>(dst) = make_uint4(a.x, a.y, b.x, b.y);
        } else {                                                         // rows of 8-byte multiples
          *reinterpret_cast<uint2*>(dst) = a;
          if (k_byte + 8 < out_ld) *reinterpret_cast<uint2*>(dst + 8) = b;
        }
      }
      if (tid < 64 && (r0 >> 6) + (tid >> 5) < ct_c)
        *reinterpret_cast<uint4*>(p.sf_c + ((c0 >> 7) * ct_c + (r0 >> 6)) * 512 + tid * 16u) =
            *reinterpret_cast<const uint4*>(out_sf + tid * 16u);
    }
  }
}

// ---------------------------------------------------------------------------------------
// The maxima of the same tiles: after the Hadamard transform along the rows, and with BOTH the plain one too
// (out[0] = plain, out[1] = transformed; without BOTH out[0] = transformed).  Three slots of 32 KiB per CTA, two CTAs per
// SM: 192 KiB in flight or in work per SM, one atomic per CTA and maximum.  HBM-bound, us with the clearing of the words,
// both maxima: 4096 x 28672 51.5 -> 41.2 (5.7 TB/s), 4096 x 14336 30.8 -> 24.6, 4096 x 4096 14.7 -> 12.4, 16384 x 768
// 14.7 -> 10.8, 512 x 768 7.3 -> 6.0 (before: a CTA per 64 rows x 512 columns, staged through registers, thousands of CTAs).
// ---------------------------------------------------------------------------------------
constexpr int kMaxSlots = 3;
constexpr int kMaxMiscOff = kMaxSlots * kSlotBytes;
constexpr int kMaxSmemBytes = kMaxMiscOff + 512 /* signs, barriers, partial maxima */ + 1024 /* alignment slack */;

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <bool BOTH>
__global__ void __launch_bounds__(kThreads, 2)
amax_tiles_kernel(const __grid_constant__ CUtensorMap map_x, uint32_t ntc, uint32_t ntiles,
                  const float* __restrict__ signs16, float* __restrict__ out, unsigned long long wait_limit_ns,
                  uint32_t extra_arrivals) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = fused::smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint32_t* sgn = reinterpret_cast<uint32_t*>(smem + kMaxMiscOff);       // 16 sign-flip masks
  float* part = reinterpret_cast<float*>(sgn + 16);                       // 2 x 16 warp maxima
  const uint32_t bars = fused::smem_u32(part + 32);
  volatile int* gave_up = reinterpret_cast<volatile int*>(part + 32 + 2 * kMaxSlots);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t my_tiles = blockIdx.x < ntiles ? (ntiles - blockIdx.x + gridDim.x - 1u) / gridDim.x : 0u;
  auto fetch = [&](uint32_t i) {
    const uint32_t tile = blockIdx.x + i * gridDim.x, rt = tile / ntc, ct = tile - rt * ntc;
    const uint32_t s = i % kMaxSlots, bar = bars + 8u * s, dst = fused::smem_u32(smem) + s * kSlotBytes;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)kSlotBytes) : "memory");
    tma_half_load(dst, &map_x, (int)(ct * kTile), (int)(rt * kTile), bar);
    tma_half_load(dst + kHalfBytes, &map_x, (int)(ct * kTile + 64), (int)(rt * kTile), bar);
  };
  if (tid == 0) {
    for (int s = 0; s < kMaxSlots; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bars + 8u * s), "r"(1u + extra_arrivals));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *gave_up = 0;
    for (uint32_t i = 0; i < (uint32_t)kMaxSlots && i < my_tiles; ++i) fetch(i);
  }
  if (tid >= 32 && tid < 48) sgn[tid - 32] = __ldg(signs16 + (tid - 32)) < 0.0f ? 0x80000000u : 0u;
  __syncthreads();
  float m = 0.0f;
  uint32_t mp = 0u;                                // both 16-bit halves carry a running maximum of bf16 magnitudes
  const uint32_t half = warp & 1u, rb = warp >> 1;
  for (uint32_t i = 0; i < my_tiles; ++i) {
    const uint32_t slot = (i % kMaxSlots) * kSlotBytes, bar = bars + 8u * (i % kMaxSlots);
    if (!fused::wait_copy(bar, (i / kMaxSlots) & 1u, wait_limit_ns)) { *gave_up = 1; atomicCAS(&fused::g_wait_error, 0, 2); }
    const uint32_t addr = fused::smem_u32(smem) + slot + half * kHalfBytes + rb * 2048u + lane * 4u;
    float v0[16], v1[16];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 m4 = reinterpret_cast<const uint4*>(sgn)[q];
      const uint32_t sm[4] = {m4.x, m4.y, m4.z, m4.w};
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = 4 * q + e;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[e]) : "r"((addr ^ ((uint32_t)(k & 7) << 4)) + 128 * k));
        v0[k] = __uint_as_float((w[e] << 16) + sm[e]);
        v1[k] = __uint_as_float((w[e] & 0xffff0000u) ^ sm[e]);
      }
      if (BOTH) mp = fused::max_abs_word(mp, make_uint4(w[0], w[1], w[2], w[3]));
    }
#pragma unroll
    for (int s = 1; s < 16; s <<= 1) {
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if ((k & s) == 0) fused::addsub2(v0[k], v1[k], v0[k | s], v1[k | s]);
    }
    m = fmaxf(m, fmaxf(fused::max_abs16(v0), fused::max_abs16(v1)));
    __syncthreads();                                                      // the slot is read
    if (*gave_up != 0) return;                                            // no maximum of a part of the tensor
    if (tid == 0 && i + kMaxSlots < my_tiles) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");        // generic reads before the async write
      fetch(i + kMaxSlots);
    }
  }
  // neither maximum can be a NaN (NaNs do not count), so they order like their bits
  const uint32_t plain_bits = __reduce_max_sync(0xffffffffu, __float_as_uint(fused::max_abs_value(mp)));
  m = warp_max(m * 0.25f);                                                // the transform is butterfly / 4
  if (lane == 0) { part[warp] = m; part[16 + warp] = __uint_as_float(plain_bits); }
  __syncthreads();
  if (warp == 0) {
    const float r = warp_max(lane < 16 ? part[lane] : 0.0f);
    const uint32_t pb = __reduce_max_sync(0xffffffffu, lane < 16 ? __float_as_uint(part[16 + lane]) : 0u);
    if (lane == 0) {
      unsigned int* o = reinterpret_cast<unsigned int*>(out);             // non-negative floats order like their bits
      if (BOTH && pb != 0u) atomicMax(o, pb);
      if (r > 0.0f) atomicMax(o + (BOTH ? 1 : 0), __float_as_uint(r));
    }
  }
}

namespace {
std::mutex g_mutex;
int g_sms[64];

const void* kernel_fn(int rows_mode, bool sr_c, bool rht) {
#define NVFP4_DUAL_FN(R_) \
  (sr_c ? (rht ? (const void*)quant_dual_kernel<R_, true, true> : (const void*)quant_dual_kernel<R_, true, false>) \
        : (rht ? (const void*)quant_dual_kernel<R_, false, true> : (const void*)quant_dual_kernel<R_, false, false>))
  return rows_mode == 0 ? NVFP4_DUAL_FN(0) : (rows_mode == 1 ? NVFP4_DUAL_FN(1) : NVFP4_DUAL_FN(2));
#undef NVFP4_DUAL_FN
}

int sm_count(int& out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NVFP4_E_LAUNCH;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (g_sms[dev] == 0) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) return NVFP4_E_LAUNCH;
    for (int v = 0; v < 12; ++v)
      if (cudaFuncSetAttribute(kernel_fn(v >> 2, (v & 2) != 0, (v & 1) != 0), cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kSmemBytes) != cudaSuccess) {
        cudaGetLastError();
        return NVFP4_E_LAUNCH;
      }
    if (cudaFuncSetAttribute(amax_tiles_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmemBytes) != cudaSuccess ||
        cudaFuncSetAttribute(amax_tiles_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmemBytes) != cudaSuccess) {
      cudaGetLastError();
      return NVFP4_E_LAUNCH;
    }
    g_sms[dev] = sms;
  }
  out = g_sms[dev];
  return NVFP4_OK;
}
}  // namespace

static PhiloxKeys make_keys(uint64_t seed) {
  PhiloxKeys keys;
  for (int r = 0; r < 10; ++r) {
    keys.k[r][0] = (uint32_t)seed + (uint32_t)r * 0x9E3779B9u;
    keys.k[r][1] = (uint32_t)(seed >> 32) + (uint32_t)r * 0xBB67AE85u;
  }
  return keys;
}

// tiles of 128 rows x 64 columns of x [rows, cols] bf16, row pitch ld
static bool make_tile_map(CUtensorMap* map, const void* x, int64_t rows, int64_t cols, int64_t ld) {
  gemm::EncodeTiledFn enc = gemm::encode_fn();
  if (enc == nullptr) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2u};
  cuuint32_t box[2] = {64u, (cuuint32_t)kTile};
  cuuint32_t estr[2] = {1u, 1u};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The maxima of x, into words that are zero: the transformed one, or (both) the plain one and the transformed one.
int launch_amax(const void* x, int64_t rows, int64_t cols, int64_t ld, const float* signs16, bool both, float* out,
                cudaStream_t stream) {
  int sms = 0;
  const int rc = sm_count(sms);
  if (rc != NVFP4_OK) return rc;
  CUtensorMap map;
  if (!make_tile_map(&map, x, rows, cols, ld)) return NVFP4_E_DRIVER;
  const int64_t ntc = (cols + kTile - 1) / kTile, ntiles = ntc * ((rows + kTile - 1) / kTile);
  if (ntiles >= (1ll << 31)) return NVFP4_E_LIMIT;
  const uint32_t grid = ntiles < 2 * sms ? (uint32_t)ntiles : 2u * (uint32_t)sms;
  const unsigned long long limit = fused::hook_wait_limit_ns();
  const uint32_t extra = fused::hook_extra_arrivals(), nc = (uint32_t)ntc, nt = (uint32_t)ntiles;
  if (both) amax_tiles_kernel<true><<<grid, kThreads, kMaxSmemBytes, stream>>>(map, nc, nt, signs16, out, limit, extra);
  else amax_tiles_kernel<false><<<grid, kThreads, kMaxSmemBytes, stream>>>(map, nc, nt, signs16, out, limit, extra);
  return cudaGetLastError() == cudaSuccess ? NVFP4_OK : NVFP4_E_LAUNCH;
}

// x [rows, cols] bf16, row pitch ld elements; rows_mode 0 / 1 / 2 = no row-wise output / nearest / stochastic; signs16
// null = no Hadamard on the transposed output.  counters4 = pitch_r, base_r, pitch_c, base_c.  Arguments have been
// validated by the caller (quantize.cu): 16-byte aligned pointers, ld % 8 == 0, rows % 16 == 0, and cols % 16 == 0 when
// there is a row-wise output.
int launch(const void* x, int64_t rows, int64_t cols, int64_t ld, int rows_mode, bool sr_c, const float* signs16,
           const float* amax_r, const float* amax_c, uint64_t seed_r, uint64_t seed_c, uint64_t offset,
           const uint64_t* counters4, uint8_t* q_r, uint8_t* sf_r, float* pts_r, uint8_t* q_c, uint8_t* sf_c, float* pts_c,
           cudaStream_t stream) {
  int sms = 0;
  const int rc = sm_count(sms);
  if (rc != NVFP4_OK) return rc;
  CUtensorMap map;
  if (!make_tile_map(&map, x, rows, cols, ld)) return NVFP4_E_DRIVER;
  Params p;
  p.rows = rows;
  p.cols = cols;
  const int64_t ntc = (cols + kTile - 1) / kTile, ntiles = ntc * ((rows + kTile - 1) / kTile);
  if (ntiles >= (1ll << 30)) return NVFP4_E_LIMIT;
  p.ntc = (uint32_t)ntc;
  // (three half units of work per SM at most are better balanced than two whole ones)
  p.split = rows_mode != 0 && ntiles <= 2 * sms ? 1u : 0u;
  p.nunits = (uint32_t)ntiles << p.split;
  p.signs16 = signs16;
  p.amax_r = amax_r;
  p.amax_c = amax_c;
  p.keys_r = make_keys(seed_r);
  p.keys_c = make_keys(seed_c);
  p.offset = offset;
  p.pitch_r = counters4[0]; p.base_r = counters4[1]; p.pitch_c = counters4[2]; p.base_c = counters4[3];
  p.q_r = q_r; p.sf_r = sf_r; p.pts_r = pts_r;
  p.q_c = q_c; p.sf_c = sf_c; p.pts_c = pts_c;
  p.wait_limit_ns = fused::hook_wait_limit_ns();
  p.extra_arrivals = fused::hook_extra_arrivals();
  const uint32_t grid = p.nunits < 2u * (uint32_t)sms ? p.nunits : 2u * (uint32_t)sms;      // two resident CTAs per SM
  void* args[] = {&map, &p};
  if (cudaLaunchKernel(kernel_fn(rows_mode, sr_c, signs16 != nullptr), dim3(grid), dim3(kThreads), args, kSmemBytes,
                       stream) != cudaSuccess) {
    cudaGetLastError();          // a refused launch must not show up as the next call's error
    return NVFP4_E_LAUNCH;
  }
  return NVFP4_OK;
}

}  // namespace dual
}  // namespace nvfp4

namespace nvfp4 { namespace tiled { int wait_error_address(void** out); }}

extern "C" int nvfp4_quantize_wait_status(int32_t* host_out, int clear, void* stream_) {
  if (host_out == nullptr) return NVFP4_E_NULL;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  void* word[2] = {nullptr, nullptr};
  int32_t got[2] = {0, 0};
  bool ok = cudaGetSymbolAddress(&word[0], nvfp4::fused::g_wait_error) == cudaSuccess &&
            nvfp4::tiled::wait_error_address(&word[1]) == NVFP4_OK;
  for (int i = 0; i < 2 && ok; ++i) {
    ok = cudaMemcpyAsync(&got[i], word[i], sizeof(int32_t), cudaMemcpyDeviceToHost, stream) == cudaSuccess;
    if (ok && clear) ok = cudaMemsetAsync(word[i], 0, sizeof(int32_t), stream) == cudaSuccess;
  }
  if (!ok || cudaStreamSynchronize(stream) != cudaSuccess) {
    cudaGetLastError();
    return NVFP4_E_LAUNCH;
  }
  *host_out = got[0] != 0 ? got[0] : got[1];
  return NVFP4_OK;
}
