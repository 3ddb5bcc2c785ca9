// Block-scaled NVFP4 GEMM for B200 (sm_100a): D[M,N] = (A.sfA)(B.sfB)^T * ptsA * ptsB.
//
// tcgen05.mma kind::mxf4nvf4 with 1x16 E4M3 block scales (scale_vec::4X), fp32 accumulators in
// tensor memory.  Per CTA: one 128 x TN output tile (TN 64, 128 or 256); K is walked in slices of 256 elements
// (= one 128-byte swizzled row per operand row).  Warp roles:
//   warp 0      TMA producer: A and B slices by tensor-map copies into 128B-swizzled shared
//               memory, the matching scale-factor tiles by tensor-map copies too (the 128x4-tiled
//               scale layout makes the scales of one slice contiguous per 128 rows)
//   warp 1      allocates tensor memory; per slice one elected lane copies the scale tiles to tensor memory
//               (tcgen05.cp) and issues the MMAs
//   warps 2..5  the epilogue: tcgen05.ld the accumulators, multiply by ptsA*ptsB, store bf16/fp32
// It serves the products that do not fill the chip with the 256 x 256 tiles of the pair kernel: few rows (decode), small
// layers, weight gradients with few output tiles and a long contraction.  Where even its tiles leave SMs idle, a cluster
// of p.splits CTAs shares a tile: each takes a part of the K slices, leaves its fp32 accumulator in its shared memory,
// and sums its share of the columns over the cluster in rank order -- no zeroed output, no atomics, the same bits on
// every run.
// All waits are bounded: a wait that gives up writes a code to *status, raises a CTA-wide abort
// flag, and the kernel drains and frees its tensor memory before returning.
// gemm_pair.cu holds the persistent cta_group::2 kernel (256 rows per CTA pair), gemm_api.cu the C entry point and
// the rule that chooses.
#include <atomic>

#include "gemm_common.cuh"

namespace nvfp4 {
namespace gemm {

constexpr int kTileM = 128;
constexpr int kThreads = 192;

// What follows from the tile width TN (128 rows by TN columns per CTA)
template <int TN> struct Tile {
  static constexpr int kSfGroups = TN == 256 ? 2 : 1;           // 128-row groups of B scales per tile
  static constexpr int kStages = TN == 256 ? 4 : (TN == 128 ? 6 : 7);   // all of shared memory: latency counts here
  static constexpr int kPartPitch = TN + 4;                     // floats per row of a partial sum, no bank conflicts
  static constexpr int kABytes = kTileM * 128;                  // 16 KiB
  static constexpr int kBBytes = TN * 128;
  static constexpr int kSfaBytes = 4 * 512;                     // 128 rows x 16 scales
  static constexpr int kSfbBytes = kSfGroups * 4 * 512;
  static constexpr int kStageBytes = kABytes + kBBytes + kSfaBytes + kSfbBytes;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment slack*/ + 256 /*barriers*/;
  static constexpr int kSfCols = 16 + 16 * kSfGroups;           // tensor-memory columns of one K slice's scales
  static constexpr int kSfRing = 4;                             // slices of scale factors in tensor memory
  static constexpr int kCols = TN == 256 ? 512 : 256;           // tensor-memory columns allocated
  static_assert(TN + kSfRing * kSfCols <= kCols, "tensor memory");
  static_assert(kSmemBytes <= 232448 && 128 * kPartPitch * 4 <= kStages * kStageBytes, "shared memory");
  static_assert(4 * 128 * TN <= kStages * kStageBytes, "the epilogue stages its output in the operand buffers");
};

__device__ __forceinline__ void tc_copy_scales(uint32_t tmem, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(tmem), "l"(desc) : "memory");
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 load_cluster(uint32_t addr, uint32_t rank) {
  float4 v;
  asm volatile(
      "{\n.reg .b32 a;\nmapa.shared::cluster.u32 a, %4, %5;\nld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n}"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"(rank) : "memory");
  return v;
}
// This CTA's share of the tile's columns (TN / S of them), summed over the cluster in rank order.  Eight remote loads per
// thread are in flight: one at a time the sum took 7 us for a 128 x 256 tile.
template <int TN, int S>
__device__ __forceinline__ void sum_partials(const Params& p, uint32_t smem_base, uint32_t rank, int64_t m0, int64_t n0) {
  constexpr int kVecs = TN / S / 4, kBatch = 8 / S;
  const int rows = (int)min((int64_t)kTileM, p.M - m0), items = rows * kVecs;
  const float alpha = __ldg(p.a_pts) * __ldg(p.b_pts);
  float m = 0.0f;                                               // max|D| of what this thread stores
  for (int i0 = threadIdx.x; i0 < items; i0 += kThreads * kBatch) {
    float4 v[kBatch][S];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int i = min(i0 + b * kThreads, items - 1), r = i / kVecs, c = ((int)rank * kVecs + (i - r * kVecs)) * 4;
      const uint32_t at = smem_base + 4u * (uint32_t)(r * Tile<TN>::kPartPitch + c);
#pragma unroll
      for (int k = 0; k < S; ++k) v[b][k] = load_cluster(at, (uint32_t)k);
    }
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int i = i0 + b * kThreads;
      if (i >= items) break;
      const int r = i / kVecs, c = ((int)rank * kVecs + (i - r * kVecs)) * 4;
      const int64_t col = n0 + c;
      if (col >= p.N) continue;
      float4 s = v[b][0];
#pragma unroll
      for (int k = 1; k < S; ++k) { s.x += v[b][k].x; s.y += v[b][k].y; s.z += v[b][k].z; s.w += v[b][k].w; }
      float o[4] = {s.x * alpha, s.y * alpha, s.z * alpha, s.w * alpha};
      if (p.round_bf16)
        for (int j = 0; j < 4; ++j) o[j] = __bfloat162float(__float2bfloat16_rn(o[j]));
      if (p.d_amax_out != nullptr)                              // (columns outside hold zeros)
        for (int j = 0; j < 4; ++j) m = fmaxf(m, fabsf(p.out_f32 ? o[j] : __bfloat162float(__float2bfloat16_rn(o[j]))));
      const int64_t d = (m0 + r) * p.ldd + col;
      const bool vec = col + 4 <= p.N && (p.ldd & 3) == 0;
      if (p.out_f32) {
        float* out = static_cast<float*>(p.d) + d;
        if (vec) *reinterpret_cast<float4*>(out) = make_float4(o[0], o[1], o[2], o[3]);
        else
          for (int j = 0; j < 4; ++j)
            if (col + j < p.N) out[j] = o[j];
      } else {
        __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.d) + d;
        if (vec) {
          const __nv_bfloat162 lo = __floats2bfloat162_rn(o[0], o[1]), hi = __floats2bfloat162_rn(o[2], o[3]);
          *reinterpret_cast<uint2*>(out) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        } else {
          for (int j = 0; j < 4; ++j)
            if (col + j < p.N) out[j] = __float2bfloat16_rn(o[j]);
        }
      }
    }
  }
  flush_amax(p, __float_as_uint(m), threadIdx.x & 31);
}
// The same share as NVFP4: a thread takes one block of 16 columns.  The sums are those of sum_partials, in its order, so
// the bytes are what quantizing its bf16 result gives.
template <int TN, int S>
__device__ __forceinline__ void quantize_partials(const Params& p, uint32_t smem_base, uint32_t rank, int64_t m0, int64_t n0) {
  constexpr int kBlocks = TN / S / 16, kDiv = kBlocks > 0 ? kBlocks : 1;   // none for TN 64, S 8: not launched with this output
  const float alpha = __ldg(p.a_pts) * __ldg(p.b_pts);
  const float pts = __fdiv_rn(fmaxf(__ldg(p.d_amax), kAmaxFloor), kGlobalDiv), inv_pts = __fdiv_rn(1.0f, pts);
  const int64_t col_tiles = ((p.N >> 4) + 3) >> 2;
  const int items = (int)min((int64_t)kTileM, p.M - m0) * kBlocks;
  for (int i = threadIdx.x; i < items; i += kThreads) {
    const int r = i / kDiv, c = ((int)rank * kBlocks + (i - r * kBlocks)) * 16;
    const int64_t row = m0 + r, col = n0 + c;
    if (col >= p.N) continue;                                   // N is a multiple of 16: a block is whole or absent
    const uint32_t at = smem_base + 4u * (uint32_t)(r * Tile<TN>::kPartPitch + c);
    float4 v[4][S];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int k = 0; k < S; ++k) v[q][k] = load_cluster(at + 16u * q, (uint32_t)k);
    uint32_t acc[16];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float4 s = v[q][0];
#pragma unroll
      for (int k = 1; k < S; ++k) { s.x += v[q][k].x; s.y += v[q][k].y; s.z += v[q][k].z; s.w += v[q][k].w; }
      acc[4 * q] = __float_as_uint(s.x); acc[4 * q + 1] = __float_as_uint(s.y);
      acc[4 * q + 2] = __float_as_uint(s.z); acc[4 * q + 3] = __float_as_uint(s.w);
    }
    uint32_t lo, hi, sf;
    quantize_out_block(acc, alpha, pts, inv_pts, lo, hi, sf);
    *reinterpret_cast<uint2*>(static_cast<uint8_t*>(p.d) + row * (p.N >> 1) + (col >> 1)) = make_uint2(lo, hi);
    p.d_sf[sf_offset(row, col >> 4, col_tiles)] = (uint8_t)sf;
  }
}
template <int TN, int S>
__device__ __forceinline__ void finish_shared_tile(const Params& p, uint32_t smem_base, uint32_t rank, int64_t m0, int64_t n0) {
  if (p.out_fp4) quantize_partials<TN, S>(p, smem_base, rank, m0, n0);
  else sum_partials<TN, S>(p, smem_base, rank, m0, n0);
}

template <int TN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
            const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_sfa,
            const __grid_constant__ CUtensorMap map_sfb, const Params p) {
  using T = Tile<TN>;
  constexpr int kStages = T::kStages, kStageBytes = T::kStageBytes, kABytes = T::kABytes, kBBytes = T::kBBytes;
  constexpr int kSfaBytes = T::kSfaBytes, kTileN = TN;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;                 // 1024-byte alignment for the swizzle
  uint8_t* smem = smem_raw + (base - raw);
  // layout: [stage][A | B | SFA | SFB] ... then barriers
  const uint32_t bar_base = base + kStages * kStageBytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };                  // TMA landed
  auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };      // MMAs have read the stage
  const uint32_t acc_bar = bar_base + 8u * (2 * kStages);
  const uint32_t never_bar = bar_base + 8u * (2 * kStages + 1);               // test hook: nothing arrives here
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + kStages * kStageBytes + 8 * (2 * kStages + 2));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kStages * kStageBytes + 8 * (2 * kStages + 2) + 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // grouped rasterization: consecutive CTAs walk kGroupM row tiles before the next column tile, so
  // that one wave of CTAs touches a near-square patch of A and B (both stay L2 resident)
  const uint32_t tiles_n = (uint32_t)((p.N + kTileN - 1) / kTileN), tiles_m = (uint32_t)((p.M + kTileM - 1) / kTileM);
  const uint32_t per_group = kGroupM * tiles_n;
  const uint32_t tile_id = blockIdx.x / (uint32_t)p.splits, split = blockIdx.x % (uint32_t)p.splits;
  const uint32_t group = tile_id / per_group, first_m = group * kGroupM;
  const uint32_t gsize = min((uint32_t)kGroupM, tiles_m - first_m);
  const uint32_t in_group = tile_id - group * per_group;
  const int64_t m0 = (int64_t)(first_m + in_group % gsize) * kTileM, n0 = (int64_t)(in_group / gsize) * kTileN;
  // this CTA's share of the K slices (all of them unless K is split)
  const int total_kt = (int)((p.K + kTileK - 1) / kTileK);
  const int per_split = (total_kt + p.splits - 1) / p.splits;
  const int kt0 = (int)split * per_split;
  const int num_kt = min(total_kt, kt0 + per_split) - kt0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(acc_bar, 1);
    mbar_init(never_bar, 1);
    *abort_flag = 0;
    set_wait_limit(abort_flag, p.wait_limit_ns);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32((const void*)tmem_slot)), "r"(T::kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_sf0 = tmem_base + kTileN;                  // scale factors behind the accumulator

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    if (lane == 0) {
      int issued = 0;
      for (int kt = 0; kt < num_kt; ++kt) {
        const int s = kt % kStages;
        if (kt >= kStages && !mbar_wait(empty_bar(s), ((kt / kStages) - 1) & 1, abort_flag)) {
          raise(abort_flag, p.status, kErrProducerWait);
          break;
        }
        const uint32_t stage = base + s * kStageBytes;
        // whole boxes always: rows and columns outside the operands arrive as zeros
        mbar_expect_tx(full_bar(s), kStageBytes);
        tma_load_2d(stage, &map_a, (kt0 + kt) * 128, (int)m0, full_bar(s));
        tma_load_2d(stage + kABytes, &map_b, (kt0 + kt) * 128, (int)n0, full_bar(s));
        tma_load_2d(stage + kABytes + kBBytes, &map_sfa, (kt0 + kt) * 256, (int)(m0 >> 7), full_bar(s));
        tma_load_2d(stage + kABytes + kBBytes + kSfaBytes, &map_sfb, (kt0 + kt) * 256, (int)(n0 >> 7), full_bar(s));
        ++issued;
      }
      if (*abort_flag != 0) {
        // give copies already in flight a bounded chance to land before shared memory goes away
        const int first = issued > kStages ? issued - kStages : 0;
        for (int kt = first; kt < issued; ++kt)
          for (uint32_t i = 0; i < (1u << 16) && !mbar_try_wait(full_bar(kt % kStages), (kt / kStages) & 1); ++i) {}
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    // the warp stays converged and one elected lane issues (see elect_one)
    constexpr uint32_t idesc = make_idesc(kTileM, kTileN);
    // K slices that hold all four K=64 blocks (every one except possibly the last of the matrix)
    const int whole_kt = (int)min((int64_t)num_kt, max((int64_t)0, p.K / kTileK - kt0));
    // B scales: a 64-wide tile that starts in the middle of a 128-row group uses columns 2 and 3 of its scale tile
    const uint32_t sfb_shift = TN == 64 ? (uint32_t)(n0 & 127) >> 5 : 0u;
    int s = 0;
    uint32_t parity = 0, sf = 0;
    for (int kt = 0; kt < num_kt; ++kt) {
      if (!__all_sync(0xffffffffu, mbar_wait(p.drop_first_scale_arrival ? never_bar : full_bar(s), parity, abort_flag))) {
        raise(abort_flag, p.status, kErrMmaWait);
        break;
      }
      tc_fence_after();
      const uint32_t stage = base + s * kStageBytes;
      const uint32_t t_sfa = tmem_sf0 + sf * T::kSfCols, t_sfb = t_sfa + 16;
      const uint64_t da = make_desc_sw128(stage), db = make_desc_sw128(stage + kABytes);
      const uint64_t dsa = make_desc_scales(stage + kABytes + kBBytes), dsb = dsa + (kSfaBytes >> 4);
      const int nkb = kt < whole_kt ? 4 : (int)((p.K - (int64_t)(kt0 + kt) * kTileK + 63) / 64);
      if (elect_one()) {
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
          tc_copy_scales(t_sfa + 4 * kb, dsa + 32u * kb);
          tc_copy_scales(t_sfb + 4 * T::kSfGroups * kb, dsb + 32u * kb);
          if (T::kSfGroups == 2) tc_copy_scales(t_sfb + 8 * kb + 4, dsb + 128u + 32u * kb);
        }
        // 64 elements = 32 bytes further along K inside the swizzled row: +2 in 16-byte units
#pragma unroll
        for (int kb = 0; kb < 4; ++kb)
          if (kb < nkb)
            tc_mma_nvf4(tmem_base, da + 2u * kb, db + 2u * kb, idesc, t_sfa + 4 * kb,
                        t_sfb + 4 * T::kSfGroups * kb + sfb_shift, (kt > 0 || kb > 0) ? 1u : 0u);
        tc_commit(empty_bar(s));                                 // frees the stage once these have read it
        if (kt == num_kt - 1) tc_commit(acc_bar);                // accumulator complete
      }
      __syncwarp();
      if (++s == kStages) { s = 0; parity ^= 1u; }
      if (++sf == T::kSfRing) sf = 0;
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    const int quad = warp & 3;                                   // TMEM lanes 32*quad .. +31
    bool ok = true;
    if (ok && lane == 0) {
      ok = mbar_wait(acc_bar, 0, abort_flag);
      if (!ok) raise(abort_flag, p.status, kErrEpilogueWait);
    }
    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    uint32_t mbits = 0u;
    if (ok) {
      tc_fence_after();
      const float alpha = __ldg(p.a_pts) * __ldg(p.b_pts);
      const int64_t row = m0 + quad * 32 + lane;
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
      if (p.splits > 1) {
        // the partial sum, unscaled, in the operand buffers (every MMA has finished and every TMA load has landed)
        float* part = reinterpret_cast<float*>(smem) + (quad * 32 + lane) * T::kPartPitch;
#pragma unroll 1
        for (int c0 = 0; c0 < kTileN; c0 += 32) {
          if (m0 + quad * 32 >= p.M || n0 + c0 >= p.N) break;    // uniform across the warp: nobody reads these
          uint32_t r[32];
          tc_ld_32x32b_x32(taddr + c0, r);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<uint4*>(part + c0 + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
        }
      } else if (p.tma_store) {
        // every MMA has finished and every TMA load has landed, so the stages are free: 128 * TN bytes per warp
        drain_through_tma(p, &map_d, taddr, smem + (warp - 2) * (128 * TN), m0 + quad * 32, n0, 0, kTileN, alpha, lane,
                          mbits);
      } else {
#pragma unroll 1
        for (int c0 = 0; c0 < kTileN; c0 += 32) {
          if (n0 + c0 >= p.N) break;                             // uniform across the warp
          uint32_t r[32];
          tc_ld_32x32b_x32(taddr + c0, r);
          tc_wait_ld();
          if (p.d_amax_out != nullptr) track_amax(p, r, alpha, row, n0 + c0, mbits);
          if (row < p.M) store_row_chunk(p, row, n0 + c0, r, alpha);
        }
      }
    }
    flush_amax(p, mbits, lane);
  }
  tc_fence_before();
  __syncthreads();
  if (p.splits > 1) {
    cluster_sync_all();                                          // every partial sum of the tile is in place
    if (p.splits == 2) finish_shared_tile<TN, 2>(p, base, split, m0, n0);
    else if (p.splits == 4) finish_shared_tile<TN, 4>(p, base, split, m0, n0);
    else finish_shared_tile<TN, 8>(p, base, split, m0, n0);
    cluster_sync_all();                                          // nobody reads this CTA's shared memory any more
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(T::kCols) : "memory");
  }
}

}  // namespace gemm
}  // namespace nvfp4

namespace nvfp4 { namespace gemm {
template <int TN>
static int launch_tile(const CUtensorMap& map_d, const uint8_t* a_q, const uint8_t* b_q, const Params& p, cudaStream_t stream) {
  CUtensorMap map_a, map_b, map_sfa, map_sfb;
  if (!make_operand_map(&map_a, a_q, p.M, p.K, kTileM) || !make_operand_map(&map_b, b_q, p.N, p.K, TN) ||
      !make_scale_map(&map_sfa, p.a_sf, p.M, p.K, 1) || !make_scale_map(&map_sfb, p.b_sf, p.N, p.K, Tile<TN>::kSfGroups))
    return NVFP4_E_DRIVER;
  const int64_t n_tiles = ((p.N + TN - 1) / TN) * ((p.M + kTileM - 1) / kTileM);
  if (n_tiles * p.splits > 0x7fffffffLL) return NVFP4_E_SHAPE;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(n_tiles * p.splits));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = Tile<TN>::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;               // the CTAs that share a tile
  attr.val.clusterDim.x = (unsigned)p.splits;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = p.splits > 1 ? 1 : 0;
  if (cudaLaunchKernelEx(&cfg, gemm_kernel<TN>, map_a, map_b, map_d, map_sfa, map_sfb, p) != cudaSuccess) {
    cudaGetLastError();          // a refused launch must not show up as the next call's error
    return NVFP4_E_LAUNCH;
  }
  return NVFP4_OK;
}

template <int TN> static bool allow_smem() {
  return cudaFuncSetAttribute(gemm_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<TN>::kSmemBytes) ==
         cudaSuccess;
}

// launch of the one-CTA kernel (arguments already validated)
int launch_1cta(int tile_n, const CUtensorMap& map_d, const uint8_t* a_q, const uint8_t* b_q, const Params& p,
                cudaStream_t stream) {
  static std::atomic<bool> attr_set[64];        // setting the attribute twice is harmless; the flag is atomic
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NVFP4_E_LAUNCH;
  if (!attr_set[dev].load(std::memory_order_acquire)) {
    if (!allow_smem<64>() || !allow_smem<128>() || !allow_smem<256>()) return NVFP4_E_LAUNCH;
    attr_set[dev].store(true, std::memory_order_release);
  }
  if (tile_n == 64) return launch_tile<64>(map_d, a_q, b_q, p, stream);
  if (tile_n == 128) return launch_tile<128>(map_d, a_q, b_q, p, stream);
  return launch_tile<256>(map_d, a_q, b_q, p, stream);
}
}}  // namespace nvfp4::gemm
