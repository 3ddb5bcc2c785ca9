// Persistent two-CTA block-scaled NVFP4 GEMM for B200 (sm_100a).
//
// One cluster of two CTAs per pair of SMs stays resident and walks over 256 x 256 output tiles
// (tile = cluster index + i * number of clusters, grouped rasterization).  The roles of a CTA:
//   warp 0      producer: TMA tensor copies of its 128 A rows, its 128 of the 256 B rows and the scale tiles
//               of both (cta_group::2 form, all completing on the leader's barrier; no multicast), into a
//               ring of five stages (four with 192-wide tiles) that runs on across tiles;
//   warp 1      (leader CTA only) per K slice one barrier wait, then twelve tcgen05.cp (the scale tiles of both CTAs,
//               shared -> tensor memory) and four tcgen05.mma cta_group::2, M 256 = 128 per CTA, N 256, K 64;
//   warps 2-9   epilogue: tensor memory -> registers -> swizzled shared memory -> TMA store.
// What bounds it: the shared-memory data stage (per CTA and slice 304 wavefronts of 128 bytes written by TMA, 256
// read by the MMAs, 48 by the scale copies, against 512 cycles of tensor work).  The scale copies used to go through
// registers (four warps each reading all 6 KiB of a slice: 192 wavefronts); tcgen05.cp reads them once.  It pays
// only when the issuing lane is picked by elect.sync (elect_one): behind `lane == 0` the compiler cannot tell that
// one lane runs the tcgen05 instructions, every copy then cost about 40 cycles and the kernel 312 us at 8192^3.
// Measured at 8192^3, bf16 output, one launch after an L2 flush: 223 us through registers, 184 us (5.96 PFLOP/s)
// this way; 16384 x 4096 x 14336 378 -> 324 us, 4096^3 45 -> 39 us, 4096 x 28672 x 4096 with fp32 output 254 -> 219.
// Spreading the copies between the MMAs of the slice measured the same.
// Because the ring never drains, the loads of the next tile are in flight while the epilogue warps
// empty the accumulator; the MMA issuer only waits for "accumulator read" before the next tile, so
// the launch, barrier set-up, tensor-memory allocation and pipeline fill are paid once per SM pair,
// not once per tile.  All waits are bounded (they raise the status word and every role leaves its
// loops); the kernel ends with a cluster barrier before the paired tensor-memory free.
#include <atomic>

#include "gemm_common.cuh"

namespace nvfp4 {
namespace gemm3 {

using namespace nvfp4::gemm;

constexpr int kEpiWarp0 = 2;                // first epilogue warp
constexpr int kThreads = (kEpiWarp0 + 8) * 32;

// What follows from the tile width TN (256 rows by TN columns per pair)
template <int TN> struct Shape {
  static constexpr int kSfGroups = TN > 128 ? 2 : 1;            // 128-row groups of B scales a tile can touch
  static constexpr int kABytes = 128 * 128;                     // this CTA's 128 A rows
  static constexpr int kBBytes = TN / 2 * 128;                  // this CTA's half of the B rows
  static constexpr int kSfaBytes = 4 * 512;
  static constexpr int kSfbBytes = kSfGroups * 4 * 512;
  static constexpr int kStageBytes = kABytes + kBBytes + kSfaBytes + kSfbBytes;
  static constexpr int kBoxes = TN == 256 ? 1 : 2;              // output boxes of 4 KiB per epilogue warp
  static constexpr int kStages = TN == 192 ? 4 : 5;
  static constexpr int kOutBytes = 8 * kBoxes * 4096;
  static constexpr int kSmemBytes = kStages * kStageBytes + kOutBytes + 1024 + 256;
  static constexpr int kAcc = TN == 256 ? 1 : 2;                // accumulators in tensor memory
  static constexpr int kSfCols = 16 + 16 * kSfGroups;           // tensor-memory columns of one K slice's scales
  static constexpr int kSfRing = TN == 192 ? 2 : 4;             // slices of scale factors in tensor memory
  static constexpr int kSplitCol = TN > 128 ? 128 : 64;         // first column of the second warp of a quarter
  static_assert(kAcc * TN + kSfRing * kSfCols <= kTmemCols, "tensor memory");
  static_assert(kSmemBytes <= 232448, "shared memory");
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Remote arrive, relaxed: what it announces (tcgen05.st / tcgen05.ld) has already completed
// (tcgen05.wait precedes it); a release at cluster scope costs about 1100 cycles here.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y,
                                                 uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar_cluster_addr) : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// one 512-byte scale tile of each CTA -> four columns of its tensor memory, in all four 32-lane quarters
__device__ __forceinline__ void tc_copy_scales_pair(uint32_t tmem, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem), "l"(desc) : "memory");
}
__device__ __forceinline__ void tc_mma_nvf4_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                 uint32_t tmem_sfa, uint32_t tmem_sfb, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%5], [%6], p;\n}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
      : "memory");
}

// tile index -> first row of the pair and first column (grouped rasterization over pairs of row tiles)
template <int TN> struct TileMap {
  uint32_t tiles_n, pairs_m, per_group;
  __device__ TileMap(const Params& p)
      : tiles_n((uint32_t)((p.N + TN - 1) / TN)), pairs_m((uint32_t)((p.M + 255) / 256)),
        per_group((kGroupM / 2) * tiles_n) {}
  __device__ uint32_t total() const { return tiles_n * pairs_m; }
  __device__ void locate(uint32_t tile, int64_t& pair_m0, int64_t& n0) const {
    const uint32_t group = tile / per_group, first = group * (kGroupM / 2);
    const uint32_t gsize = min((uint32_t)(kGroupM / 2), pairs_m - first);
    const uint32_t in_group = tile - group * per_group;
    pair_m0 = (int64_t)(first + in_group % gsize) * 256;
    n0 = (int64_t)(in_group / gsize) * TN;
  }
};

template <int TN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm3_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
             const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_sfa,
             const __grid_constant__ CUtensorMap map_sfb, const Params p) {
  using S = Shape<TN>;
  constexpr int kStages = S::kStages, kStageBytes = S::kStageBytes, kOutBytes = S::kOutBytes;
  constexpr int kABytes = S::kABytes, kBBytes = S::kBBytes, kSfaBytes = S::kSfaBytes;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;                 // same offset in both CTAs of the pair
  uint8_t* smem = smem_raw + (base - raw);
  uint8_t* out_stage = smem + kStages * kStageBytes;            // epilogue boxes (1024-byte aligned)
  const uint32_t bar_base = base + kStages * kStageBytes + kOutBytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };                    // leader: A/B of both CTAs landed
  auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };        // MMAs have read the stage
  auto acc_full = [&](int a) { return bar_base + 8u * (2 * kStages + a); };     // accumulator complete (both CTAs)
  auto acc_empty = [&](int a) { return bar_base + 8u * (2 * kStages + 2 + a); };  // leader: accumulator read, both CTAs
  const uint32_t never_bar = bar_base + 8u * (2 * kStages + 4);                 // test hook: nothing arrives here
  const int misc = kStages * kStageBytes + kOutBytes + 8 * (2 * kStages + 5);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + misc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + misc + 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const TileMap<TN> tm(p);
  const uint32_t cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1, total = tm.total();
  const int my_tiles = cluster_id < total ? (int)((total - cluster_id + n_clusters - 1) / n_clusters) : 0;
  const int num_kt = (int)((p.K + kTileK - 1) / kTileK);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < S::kAcc; ++a) { mbar_init(acc_full(a), 1); mbar_init(acc_empty(a), 16); }
    mbar_init(never_bar, 1);
    *abort_flag = 0;
    set_wait_limit(abort_flag, p.wait_limit_ns);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32((const void*)tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // barriers of both CTAs are initialised before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_sf0 = tmem_base + S::kAcc * TN;           // scale factors behind the accumulators

  if (warp == 0) {
    // ------------------------------ producer (one per CTA) ------------------------------
    if (lane == 0) {
      int s = 0, issued = 0;
      uint32_t pass = 0;                                          // parity of the current pass over the ring
      bool ok = true;
      for (int i = 0; i < my_tiles && ok; ++i) {
        int64_t pair_m0, n0;
        tm.locate(cluster_id + (uint32_t)i * n_clusters, pair_m0, n0);
        const int64_t m0 = pair_m0 + (int64_t)rank * 128;
        for (int kt = 0; kt < num_kt; ++kt) {
          if (issued >= kStages && !mbar_wait(empty_bar(s), pass ^ 1u, abort_flag)) {
            raise(abort_flag, p.status, kErrProducerWait);
            ok = false;
            break;
          }
          const uint32_t stage = base + s * kStageBytes;
          const uint32_t leader_full = map_to_cta(full_bar(s), 0);
          if (leader)   // whole boxes always: rows and columns outside the operands arrive as zeros
            mbar_expect_tx(full_bar(s), 2u * kStageBytes);
          tma_load_2d_pair(stage, &map_a, kt * 128, (int)m0, leader_full);
          tma_load_2d_pair(stage + kABytes, &map_b, kt * 128, (int)(n0 + rank * (TN / 2)), leader_full);
          tma_load_2d_pair(stage + kABytes + kBBytes, &map_sfa, kt * 256, (int)(m0 >> 7), leader_full);
          tma_load_2d_pair(stage + kABytes + kBBytes + kSfaBytes, &map_sfb, kt * 256, (int)(n0 >> 7), leader_full);
          ++issued;
          if (++s == kStages) { s = 0; pass ^= 1u; }
        }
      }
      if (*abort_flag != 0) {
        // give copies already in flight a bounded chance to land before shared memory goes away
        // (the leader's barriers count the copies of both CTAs)
        const int first_g = issued > kStages ? issued - kStages : 0;
        for (int g = first_g; leader && g < issued; ++g)
          for (uint32_t n = 0; n < (1u << 16) && !mbar_try_wait(full_bar(g % kStages), (g / kStages) & 1); ++n) {}
        if (!leader) __nanosleep(50000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA only) ------------------------------
    if (leader) {
      constexpr uint32_t idesc = make_idesc(256, TN);
      const int whole_kt = (int)min((int64_t)num_kt, p.K / kTileK);     // K slices with all four K=64 blocks
      int s = 0;
      uint32_t par = 0, sf = 0;
      bool ok = true;
      for (int i = 0; i < my_tiles && ok; ++i) {
        const int a = i % S::kAcc;
        const uint32_t tmem_d = tmem_base + a * TN;
        if (i >= S::kAcc) {                                     // the epilogue warps have read the accumulator
          ok = __all_sync(0xffffffffu, mbar_wait(acc_empty(a), (uint32_t)(i / S::kAcc - 1) & 1u, abort_flag));
          if (!ok) { raise(abort_flag, p.status, kErrMmaWait); break; }
          tc_fence_after();
        }
        // B scales: column 32-row group of the tile's first row inside its 128-row group (0, or 2 for a 192-wide tile
        // that starts in the middle of one)
        int64_t pair_m0, n0;
        tm.locate(cluster_id + (uint32_t)i * n_clusters, pair_m0, n0);
        const uint32_t sfb_shift = TN == 192 ? (uint32_t)(n0 & 127) >> 5 : 0u;
        for (int kt = 0; kt < num_kt; ++kt) {
          ok = __all_sync(0xffffffffu, mbar_wait(p.drop_first_scale_arrival ? never_bar : full_bar(s), par, abort_flag));
          if (!ok) { raise(abort_flag, p.status, kErrMmaWait); break; }
          tc_fence_after();
          const uint32_t stage = base + s * kStageBytes;
          const uint32_t t_sfa = tmem_sf0 + sf * S::kSfCols, t_sfb = t_sfa + 16;
          const uint64_t da = make_desc_sw128(stage), db = make_desc_sw128(stage + kABytes);
          const uint64_t dsa = make_desc_scales(stage + kABytes + kBBytes), dsb = dsa + (kSfaBytes >> 4);
          const int nkb = kt < whole_kt ? 4 : (int)((p.K - (int64_t)kt * kTileK + 63) / 64);
          if (elect_one()) {
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
              tc_copy_scales_pair(t_sfa + 4 * kb, dsa + 32u * kb);
              tc_copy_scales_pair(t_sfb + 4 * S::kSfGroups * kb, dsb + 32u * kb);
              if (S::kSfGroups == 2) tc_copy_scales_pair(t_sfb + 8 * kb + 4, dsb + 128u + 32u * kb);
            }
#pragma unroll
            for (int kb = 0; kb < 4; ++kb)
              if (kb < nkb)
                tc_mma_nvf4_pair(tmem_d, da + 2u * kb, db + 2u * kb, idesc, t_sfa + 4 * kb,
                                 t_sfb + 4 * S::kSfGroups * kb + sfb_shift, (kt > 0 || kb > 0) ? 1u : 0u);
            tc_commit_pair(empty_bar(s));
            if (kt == num_kt - 1) tc_commit_pair(acc_full(a));
          }
          __syncwarp();
          if (++s == kStages) { s = 0; par ^= 1u; }
          if (++sf == S::kSfRing) sf = 0;
        }
      }
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    // Two warps per 32-lane quarter of tensor memory, 128 accumulator columns each (the second one 64 of a 192-wide
    // tile, both 64 of a 128-wide one).  A warp pulls its whole slab into registers with loads that are all under way at
    // once, signals "accumulator read" -- the MMA issuer goes on with the next tile -- and only then converts and writes
    // the slab out at leisure, under the next tile's main loop: swizzled 32 x 128-byte box in shared memory -> TMA store,
    // which writes whole lines and clips at the matrix edge.  Signalling behind the conversion (bf16) or behind the third
    // box (fp32) and polling for the accumulator with sleeps cost, us: 4096 x 28672 x 4096 fp32 222 -> 212, 4096 x 14336 x
    // 4096 fp32 119.7 -> 113.6, bf16 96.7 -> 94.2, 4096^3 bf16 31.4 -> 30.4.  A second box per warp at the price of the fifth
    // stage made 256-wide tiles 6-9 % slower.
    const int quad = warp & 3, second = (warp - kEpiWarp0) >> 2;
    const int c_base = S::kSplitCol * second, n_cols = second ? TN - S::kSplitCol : S::kSplitCol;
    uint8_t* boxes = out_stage + (warp - kEpiWarp0) * (S::kBoxes * 4096);
    int which = 0;                                                // box to write next
    const float alpha = __ldg(p.a_pts) * __ldg(p.b_pts);
    const uint32_t sw = (uint32_t)lane & 7u;
    bool ok = true;
    uint32_t mbits = 0u;                                          // running max|D| (see track_amax)
    auto release_accumulator = [&](int a) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { if (leader) mbar_arrive(acc_empty(a)); else mbar_arrive_cluster(map_to_cta(acc_empty(a), 0)); }
    };
    auto send_box = [&](int64_t x, int64_t y) {                   // the box is written: hand it to the TMA unit
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> TMA reads
      __syncwarp();
      if (lane == 0) tma_store_2d(&map_d, smem_u32(boxes + which * 4096), (int)x, (int)y);
      which = which + 1 == S::kBoxes ? 0 : which + 1;
    };
    auto box_free = [&]() {                                       // the last store out of this box has read it
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(S::kBoxes - 1) : "memory");
      __syncwarp();
    };
    for (int i = 0; i < my_tiles; ++i) {
      int64_t pair_m0, n0;
      tm.locate(cluster_id + (uint32_t)i * n_clusters, pair_m0, n0);
      const int64_t row0 = pair_m0 + (int64_t)rank * 128 + quad * 32;
      const int64_t col0 = n0 + c_base;
      const int a = i % S::kAcc;
      const uint32_t taddr = tmem_base + a * TN + ((uint32_t)(quad * 32) << 16) + c_base;
      if (lane == 0) ok = mbar_wait(acc_full(a), (uint32_t)(i / S::kAcc) & 1u, abort_flag);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) { if (lane == 0) raise(abort_flag, p.status, kErrEpilogueWait); break; }
      tc_fence_after();
      if (row0 >= p.M || col0 >= p.N) {                           // padding only: nothing to read
        release_accumulator(a);
        continue;
      }
      if (p.tma_store) {
        uint32_t acc[S::kSplitCol / 32][32];
#pragma unroll
        for (int ch = 0; ch < S::kSplitCol / 32; ++ch)
          if (32 * ch < n_cols) tc_ld_32x32b_x32(taddr + 32 * ch, acc[ch]);
        tc_wait_ld();
        release_accumulator(a);
        if (p.d_amax_out != nullptr) {
#pragma unroll
          for (int ch = 0; ch < S::kSplitCol / 32; ++ch)
            if (32 * ch < n_cols) track_amax(p, acc[ch], alpha, row0 + lane, col0 + 32 * ch, mbits);
        }
        if (!p.out_f32) {
#pragma unroll
          for (int b = 0; b < S::kSplitCol / 64; ++b) {
            if (64 * b >= n_cols || col0 + 64 * b >= p.N) break;  // uniform across the warp
            uint32_t packed[32];
#pragma unroll
            for (int q = 0; q < 32; ++q) {
              const uint32_t* r = &acc[2 * b + (q >> 4)][2 * (q & 15)];
              __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[0]) * alpha, __uint_as_float(r[1]) * alpha);
              packed[q] = *reinterpret_cast<uint32_t*>(&h);
            }
            box_free();
            uint8_t* rowp = boxes + which * 4096 + lane * 128;
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<uint4*>(rowp + (((uint32_t)j ^ sw) << 4)) =
                  make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
            send_box(col0 + 64 * b, row0);
          }
        } else {
#pragma unroll
          for (int ch = 0; ch < S::kSplitCol / 32; ++ch) {        // fp32: a box is 32 columns
            if (32 * ch >= n_cols || col0 + 32 * ch >= p.N) break;
            box_free();
            uint8_t* rowp = boxes + which * 4096 + lane * 128;
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<float4*>(rowp + (((uint32_t)j ^ sw) << 4)) =
                  make_float4(out_f32(p, acc[ch][4 * j], alpha), out_f32(p, acc[ch][4 * j + 1], alpha),
                              out_f32(p, acc[ch][4 * j + 2], alpha), out_f32(p, acc[ch][4 * j + 3], alpha));
            send_box(col0 + 32 * ch, row0);
          }
        }
      } else {                                                    // rows that no tensor map covers, quantized output
        const int64_t n_left = p.N - col0;
        const int chunks = n_left >= n_cols ? n_cols / 32 : (int)((n_left + 31) / 32);
#pragma unroll 1
        for (int ch = 0; ch < chunks; ++ch) {
          uint32_t r[32];
          tc_ld_32x32b_x32(taddr + 32 * ch, r);
          tc_wait_ld();
          if (ch == chunks - 1) release_accumulator(a);
          if (p.d_amax_out != nullptr) track_amax(p, r, alpha, row0 + lane, col0 + 32 * ch, mbits);
          if (row0 + lane < p.M) store_row_chunk(p, row0 + lane, col0 + 32 * ch, r, alpha);
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // before shared memory goes away
    __syncwarp();
    flush_amax(p, mbits, lane);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // neither CTA frees tensor memory while the partner may still use the pair
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

template <int TN>
static int launch_shape(const CUtensorMap& map_d, const uint8_t* a_q, const uint8_t* b_q, const Params& p, int sms,
                        cudaStream_t stream) {
  CUtensorMap map_a, map_b, map_sfa, map_sfb;
  if (!make_operand_map(&map_a, a_q, p.M, p.K, 128) || !make_operand_map(&map_b, b_q, p.N, p.K, TN / 2) ||
      !make_scale_map(&map_sfa, p.a_sf, p.M, p.K, 1) || !make_scale_map(&map_sfb, p.b_sf, p.N, p.K, Shape<TN>::kSfGroups))
    return NVFP4_E_DRIVER;
  const int64_t tiles = ((p.N + TN - 1) / TN) * ((p.M + 255) / 256);
  if (tiles > 0x3fffffffLL) return NVFP4_E_SHAPE;
  const int64_t clusters = tiles < sms / 2 ? tiles : sms / 2;    // one resident pair per two SMs
  gemm3_kernel<TN><<<dim3((unsigned)(2 * clusters)), kThreads, Shape<TN>::kSmemBytes, stream>>>(map_a, map_b, map_d, map_sfa,
                                                                                             map_sfb, p);
  return cudaGetLastError() == cudaSuccess ? NVFP4_OK : NVFP4_E_LAUNCH;
}

template <int TN> static bool allow_smem() {
  return cudaFuncSetAttribute(gemm3_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<TN>::kSmemBytes) ==
         cudaSuccess;
}

int launch_pair(int tile_n, const CUtensorMap& map_d, const uint8_t* a_q, const uint8_t* b_q, const Params& p,
                cudaStream_t stream) {
  static std::atomic<int> sm_count[64];         // 0 = not looked up yet; a second look-up is harmless
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NVFP4_E_LAUNCH;
  int sms = sm_count[dev].load(std::memory_order_acquire);
  if (sms == 0) {
    if (!allow_smem<128>() || !allow_smem<192>() || !allow_smem<256>()) return NVFP4_E_LAUNCH;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 2)
      return NVFP4_E_LAUNCH;
    sm_count[dev].store(sms, std::memory_order_release);
  }
  if (tile_n == 128) return launch_shape<128>(map_d, a_q, b_q, p, sms, stream);
  if (tile_n == 192) return launch_shape<192>(map_d, a_q, b_q, p, sms, stream);
  return launch_shape<256>(map_d, a_q, b_q, p, sms, stream);
}

}  // namespace gemm3
}  // namespace nvfp4
