// gmm for a handful of row tiles: the contraction of a tile is shared by the CTAs of a cluster.
//
// With few rows (one token routed to four experts; a small layer) there are fewer 128 x 256 output
// tiles than SMs, and the weights, all that matters at this size, are read by those few SMs at about
// 85 GB/s each (128 KB of weights in flight per SM over 1.5 us).  Here S CTAs of a cluster take a
// tile together: CTA r multiplies the r-th part of the contraction into its own accumulator, all
// partial sums meet in shared memory, and every CTA adds up its share of the columns, reading
// the others' sums through distributed shared memory in the order of their ranks (so results do
// not depend on timing) and writing 16-bit results.
// Bound by HBM once enough SMs read, otherwise by the launch, one latency of the ring and the two
// cluster barriers (about 5 us together).  The host picks S (choose_split in rd_api.cu).
//
// Measured, one tile per CTA -> split, cold weights, microseconds of the call (bf16; e4m3): 4 rows of 4096
// into 1536 with 4 live experts 35 -> 23 (23 -> 17); 1 row, k 14336, n 4096 92 -> 35 (53 -> 25); 64 rows, k
// 4096, n 256, 8 experts 33 -> 16; 12 rows into 1536 with 12 experts (72 tiles, two CTAs each) 55 -> 43.
//
// Loads, MMAs (M = 64 for tiles of up to 64 rows), 8-bit operands and waits as in rd_gemm.cuh.  One
// accumulator, and the ring's memory holds the partial sums between tiles: a cluster rarely
// has a second tile.
#pragma once

#include "rd_gemm.cuh"

namespace rd {

constexpr int kSplitBN = 256;
constexpr int kSplitStages = 4;
constexpr int kMaxSplit = 8;
constexpr int kSplitStageBytes = kTileM * kTileK * 2 + kSplitBN * kTileK * 2;  // 48 KB
constexpr int kSplitSmemBytes = kSplitStages * kSplitStageBytes + 1024;
static_assert(kTileM * kSplitBN * 4 <= kSplitStages * kSplitStageBytes, "partial sums fit into the ring");

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t local_addr, uint32_t cta_rank) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(map_to_cta(local_addr, cta_rank))
               : "memory");
  return v;
}

// Partial sums: [row][64 chunks of 4 columns], chunks permuted within a row so that lanes (= rows) that
// write the same chunk hit different banks.
__device__ __forceinline__ uint32_t split_chunk_offset(int row, int chunk) {
  return static_cast<uint32_t>(row * (kSplitBN * 4) + ((chunk ^ (row & 7)) << 4));
}

template <bool kBKMajor, bool kFp8>
__global__ void __launch_bounds__(kGemmThreads, 1)
ragged_gemm_splitk_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                          const GemmArgs p, const int split) {
  static_assert(!kFp8 || kBKMajor, "8-bit inputs: K-major weights");
  constexpr int BN = kSplitBN;
  constexpr int kStages = kSplitStages;
  constexpr uint32_t kABytes = kTileM * kTileK * 2;
  constexpr uint32_t kStageBytes = kSplitStageBytes;

  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t bar_full[kStages];
  __shared__ __align__(8) uint64_t bar_empty[kStages];
  __shared__ __align__(8) uint64_t bar_acc_full;
  __shared__ uint32_t tmem_slot;
  __shared__ WaitCtl wait_ctl;
  __shared__ GroupTable group_table;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_cta_rank());
  const uint32_t stage_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;

  if (threadIdx.x == 0) {
    wait_ctl.abort = 0;
    wait_ctl.limit_us = p.wait_limit_us;
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    mbar_init(smem_u32(&bar_acc_full), 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc<1>(smem_u32(&tmem_slot), BN);
    tmem_relinquish<1>();
  }
  start_inline_groups(p, kTileM, &group_table, warp, lane);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  volatile WaitCtl* abort_ptr = &wait_ctl;

  const int num_tiles = live_row_tiles(p, &group_table) * p.n_tiles;
  const int clusters = static_cast<int>(gridDim.x) / split;
  const int k_blocks = (p.k + kTileK - 1) / kTileK;
  // CTA `rank` takes blocks [kb0, kb1); the host sees to it that every share has some.
  const int kb0 = static_cast<int>(static_cast<long long>(k_blocks) * rank / split);
  const int kb1 = static_cast<int>(static_cast<long long>(k_blocks) * (rank + 1) / split);
  uint16_t* out16 = reinterpret_cast<uint16_t*>(p.out);

  uint32_t it = 0;          // ring position of the loader / the MMA thread
  uint32_t local_tile = 0;
  bool ok = true;           // a wait that expired ends this thread's waiting, not the tile loop:
                            // every CTA of the cluster must reach the same cluster barriers
  for (int tile = static_cast<int>(blockIdx.x) / split; tile < num_tiles; tile += clusters, ++local_tile) {
    const TileCoord t = uniform_coord(decode_gmm_tile<BN, 1>(p, &group_table, tile, 0));
    const bool half = t.rows <= 64;
    if (warp == 0) {
      for (int kb = kb0; kb < kb1 && ok; ++kb, ++it) {
        const uint32_t s = it % kStages;
        const uint32_t ph = (it / kStages) & 1u;
        if (!mbar_wait_warp(smem_u32(&bar_empty[s]), ph ^ 1u, abort_ptr)) {
          ok = false;
          break;
        }
        if (!elect_one()) continue;
        const uint32_t full = smem_u32(&bar_full[s]);
        const uint32_t sa = stage_base + s * kStageBytes;
        const uint32_t sb = sa + kABytes;
        mbar_arrive_expect_tx(full, kStageBytes);
        tma_load_2d(sa, &tmap_a, full, kb * kTileK, t.row0);
        if (kBKMajor) {
          tma_load_3d(sb, &tmap_b, full, kb * kTileK, t.n0, t.weight);
        } else {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j)
            tma_load_3d(sb + j * kBoxBytes, &tmap_b, full, t.n0 + j * 64, kb * kTileK, t.weight);
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      const uint32_t idesc =
          make_idesc_f16(kFp8 ? 0 : p.ab_format, 0, kBKMajor ? 0 : 1, half ? 64 : kTileM, BN);
      constexpr uint32_t kAStep = 32u >> 4;
      constexpr uint32_t kBStep = (kBKMajor ? 32u : 2048u) >> 4;
      const uint64_t adesc0 = make_smem_desc(stage_base, 16, 1024);
      const uint64_t bdesc0 = kBKMajor ? make_smem_desc(stage_base + kABytes, 16, 1024)
                                       : make_smem_desc(stage_base + kABytes, kBoxBytes, 1024);
      const uint32_t desc_hi = static_cast<uint32_t>(adesc0 >> 32);
      for (int kb = kb0; kb < kb1 && ok; ++kb, ++it) {
        const uint32_t s = it % kStages;
        if (!mbar_wait_warp(smem_u32(&bar_full[s]), (it / kStages) & 1u, abort_ptr)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        if (!elect_one()) continue;
        const uint32_t a_lo = static_cast<uint32_t>(adesc0) + s * (kStageBytes >> 4);
        const uint32_t b_lo = static_cast<uint32_t>(bdesc0) + s * (kStageBytes >> 4);
#pragma unroll
        for (int kk = 0; kk < kTileK / kUmmaK; ++kk)
          umma_ab<1, kFp8>(tmem_base, make_desc64(a_lo + kk * kAStep, desc_hi),
                           make_desc64(b_lo + kk * kBStep, desc_hi), idesc, (kb > kb0 || kk > 0) ? 1u : 0u);
        umma_commit(smem_u32(&bar_empty[s]));
      }
      if (ok && elect_one()) umma_commit(smem_u32(&bar_acc_full));
      __syncwarp();
    } else {
      // The accumulator is complete when all MMAs have retired, so the ring is idle and its memory
      // free: the loader does not start on the next tile before the barriers below.
      if (ok && !mbar_wait_warp(smem_u32(&bar_acc_full), local_tile & 1u, abort_ptr)) ok = false;
      __syncwarp();
      tc_fence_after_sync();
      const int quarter = warp & 3;
      const int row = half ? quarter * 16 + lane : quarter * 32 + lane;
      const bool mine = row < t.rows && !(half && lane >= 16);
      const bool warp_has_rows = quarter * (half ? 16 : 32) < t.rows;
      if (warp_has_rows) {
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32(tmem_base + c * 32 + (static_cast<uint32_t>(quarter * 32) << 16), v);
          tmem_ld_wait();
          if (mine) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint32_t a = stage_base + split_chunk_offset(row, c * 8 + j);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v[4 * j]), "r"(v[4 * j + 1]),
                           "r"(v[4 * j + 2]), "r"(v[4 * j + 3])
                           : "memory");
            }
          }
        }
      }
      tc_fence_before_sync();
    }
    __syncwarp();
    cluster_sync();  // every CTA's partial sums are written
    tc_fence_after_sync();
    // Chunk pairs (8 columns) are dealt to the CTAs in turn.
    const float sc = kFp8 && p.weight_scale != nullptr ? p.weight_scale[t.weight] : 1.0f;
    const int pairs = imin(BN, p.n - t.n0) / 8;
    const int my_pairs = (pairs - rank + split - 1) / split;  // may be <= 0
    for (int i = threadIdx.x; i < my_pairs * t.rows; i += kGemmThreads) {
      const int row = i / my_pairs;
      const int pr = (i - row * my_pairs) * split + rank;
      // all parts are fetched before the first is added: one trip through the cluster, not `split`
      float4 a[kMaxSplit], b[kMaxSplit];
#pragma unroll
      for (int r = 0; r < kMaxSplit; ++r) {
        if (r < split) {
          a[r] = ld_cluster_f4(stage_base + split_chunk_offset(row, 2 * pr), r);
          b[r] = ld_cluster_f4(stage_base + split_chunk_offset(row, 2 * pr + 1), r);
        }
      }
      float f[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = 0.0f;
#pragma unroll
      for (int r = 0; r < kMaxSplit; ++r) {
        if (r < split) {
          f[0] += a[r].x; f[1] += a[r].y; f[2] += a[r].z; f[3] += a[r].w;
          f[4] += b[r].x; f[5] += b[r].y; f[6] += b[r].z; f[7] += b[r].w;
        }
      }
      if constexpr (kFp8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] *= sc;
      }
      uint4 o;
      o.x = pack2(f[0], f[1], p.ab_format);
      o.y = pack2(f[2], f[3], p.ab_format);
      o.z = pack2(f[4], f[5], p.ab_format);
      o.w = pack2(f[6], f[7], p.ab_format);
      *reinterpret_cast<uint4*>(out16 + static_cast<size_t>(t.row0 + row) * p.n + t.n0 + pr * 8) = o;
    }
    __syncwarp();
    cluster_sync();  // nobody reads this CTA's partial sums any more
    // the generic accesses above come before the next tile's TMA writes to the same memory
    fence_proxy_async_smem();
  }

  if (p.zero_tail) {
    const int first = first_dead_row(p, &group_table);
    const size_t chunks_per_row = static_cast<size_t>(p.n) / 8;
    const size_t total = static_cast<size_t>(p.m - first) * chunks_per_row;
    const size_t stride = static_cast<size_t>(gridDim.x) * kGemmThreads;
    uint4* dst = reinterpret_cast<uint4*>(out16 + static_cast<size_t>(first) * p.n);
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    for (size_t i = static_cast<size_t>(blockIdx.x) * kGemmThreads + threadIdx.x; i < total; i += stride) dst[i] = z;
  }

  // ------------------------------------------------------------ tear-down
  __syncthreads();
  if (wait_ctl.abort) {
    if (threadIdx.x == 0) atomicMax(p.status, static_cast<int32_t>(kStatusWaitExpired));
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, BN);
  }
}

}  // namespace rd
