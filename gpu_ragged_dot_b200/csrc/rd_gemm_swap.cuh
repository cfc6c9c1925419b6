// gmm with the roles of the operands swapped: the weights' columns are the M side of the MMAs and the
// ragged rows the N side, on CTA pairs.
//
// Two things bound the 256 x 256 tiles of rd_gemm2.cuh on long groups.  Shared memory: a 64-deep
// stage takes 64 KB of TMA writes and 96 KB of operand reads per 1024 clocks of MMAs, 156 bytes per
// clock where a shared memory gives 128, so the tensor cores cannot pass 82 % (and every byte
// costs power, of which a long run of these GEMMs uses all there is).  And rows: M comes in steps of
// 128, so a group pays for 64 rows on average that are not there.
// Here a pair of CTAs owns 512 columns x up to 256 rows.  CTA c holds the accumulators of columns [256 c,
// 256 c + 256) as two 128-lane halves; each half is ONE tcgen05.mma.cta_group::2 with M = 256 (128
// columns of either CTA) and N = the tile's rows in steps of 16 (e4m3 32).  Each CTA loads its own columns of
// the weights (32 KB a stage) and half of the rows (16 KB); shared memory moves 48 KB in and 64 KB
// out per 1024 clocks.  A group's rows are dealt evenly to ceil(rows / 256) tiles, in steps of 16.
//
// Measured against the 256 x 256 one-CTA tiles: m 8192, k 4096, n 14336, 8 unequal groups 694 -> 687 us
// and trans_rhs 687 -> 669 us alone; as part of a training step at the power limit, where less
// traffic and fewer empty rows mean a higher clock, 2.58 -> 2.48 ms for the step.  64 groups of about 512
// rows, k 4096, n 1536, fp16: 402 -> 384 us, in a loop 487 -> 449 us.  e4m3 (m 8192, k 4096, n 14336) 466 -> 447 us
// in a row.
// Rows in steps of 16, heights in order and loops run by whole warps (see SwapGroupTable and rd_tgmm.cuh) against
// steps of 32, groups as they come and loops of one thread, microseconds in a row: m 8192, k 14336, n 4096, 8
// groups, trans_rhs 739 -> 732, 986 -> 925 thousand clocks; k 4096, n 14336 759 -> 732, trans_rhs 757 -> 744, e4m3 413 ->
// 396; 64 groups of 512, k 1536, n 4096, fp16, trans_rhs 393 -> 353.  The faster loops alone lost 8 % at k 14336:
// one thread's MMAs had held short tiles to the pace of full ones.
// What bounds it now: power; alone, the exposed drain of the accumulators, which fill
// tensor memory, and the last round of tiles.
//
// Accumulator lanes are output columns, so a warp's 32 x 32 block is transposed on its way through
// shared memory (two-byte stores, 64 contiguous bytes per row) and leaves by TMA, as 32 rows or 16; the last
// rows of a group, fewer than 16, are stored from registers, 64 bytes per row.
//
// Roles, barriers and waits as in rd_gemm2.cuh (kPair); loads are plain, nothing is broadcast.
// kFp8: e4m3 operands, K-major weights, tiles byte for byte those of a 16-bit problem.
// kF32: one TF32 pass, stages 32 deep, [k, n] weights in the 32-byte-atom swizzle (rd_gemm_f32.cuh), the same sums in
// the same order as there.  One CTA per 128 x 256 tile moves 187 bytes of shared memory per clock of MMAs and stops at 70 %
// of the tensor pipe; microseconds in a row, m 8192, k 4096, n 14336, 8 groups 1500 -> 1390, trans_rhs with k 14336, n
// 4096 1529 -> 1420; 16384, 1024, 4096, 32 268 -> 249.
#pragma once

#include "rd_gemm2.cuh"
#include "rd_gemm_f32_pair.cuh"

namespace rd {

constexpr int kSwapStages = 4;
constexpr int kSwapCols = 512;      // output columns of a pair's tile
constexpr int kSwapCtaCols = 256;   // of one CTA
constexpr int kSwapRows = 256;      // most rows of a tile
constexpr uint32_t kSwapABytes = kSwapCtaCols * kTileK * 2;      // 32 KB: weights
constexpr uint32_t kSwapBBytes = (kSwapRows / 2) * kTileK * 2;   // 16 KB: rows
constexpr uint32_t kSwapStageBytes = kSwapABytes + kSwapBBytes;  // 48 KB
constexpr int kSwapEpilogueWarps = 8;
constexpr int kSwapThreads = 64 + 32 * kSwapEpilogueWarps;
constexpr uint32_t kSwapBoxBytes = 32 * 64;  // [32 rows][32 columns] of the output
constexpr int kSwapSmemBytes = kSwapStages * kSwapStageBytes + kSwapEpilogueWarps * 2 * kSwapBoxBytes + 1024;

// The tile's rows [row0, row0 + rows) of its group and the pair's first column.
struct SwapTile {
  int weight, row0, rows, n0;
  int halves;  // 128-lane halves of each CTA: 2, or 1 for a half tile of 256 columns, or where no more are left
  int mma_n;  // rows in steps of kStep (16; e4m3 32): the N of the MMAs
};

// Groups in the order of their tiles' height, tallest first: `tiles` counts by position in that order.
// A tile's time is its rows, and pairs that share panels of x or of the weights should run side by side: with
// groups as they come, pairs go into a group after tiles of different heights, far apart, and fetch its x once
// more (m 8192, k 14336, n 4096, 8 groups: 2.4 GB from HBM instead of 1.3, at the power limit 8 % of the time).
// The launch always has the table (GemmArgs::inline_groups).
struct SwapGroupTable : GroupTable {
  uint8_t order[kMaxInlineGroups];
};

// One warp.  Counting sort on the possible heights in steps of 16 (0: no rows); equal ones keep their order.
__device__ __forceinline__ void build_group_table(const GemmArgs& p, int tile_rows, SwapGroupTable* tab, int lane) {
  constexpr int kPer = kMaxInlineGroups / 32;
  int rows[kPer], sum = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int i = lane * kPer + j;
    rows[j] = i < p.g ? imax(p.group_sizes[i], 0) : 0;
  }
#pragma unroll
  for (int j = 0; j < kPer; ++j) sum += rows[j];
  int off = warp_inclusive_scan(sum, lane) - sum;
  int tiles[kPer], height[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int i = lane * kPer + j;
    if (i <= p.g) tab->offset[i] = off;
    const int live = imin(rows[j], imax(p.m - off, 0));
    tiles[j] = (live + tile_rows - 1) / tile_rows;
    height[j] = i >= p.g ? -1 : live > 0 ? ((live + 15) / 16 + tiles[j] - 1) / tiles[j] : 0;
    off += rows[j];
  }
  if (lane == 31 && p.g == kMaxInlineGroups) tab->offset[p.g] = off;
  int pos = 0, before = 0;
  for (int h = kSwapRows / 16; h >= 0; --h) {
    int count = 0;  // groups of this height << 20 | their tiles
#pragma unroll
    for (int j = 0; j < kPer; ++j) count += height[j] == h ? (1 << 20) + tiles[j] : 0;
    if (!__any_sync(0xffffffffu, count != 0)) continue;
    const int incl = warp_inclusive_scan(count, lane);
    int at = pos + ((incl - count) >> 20), tile = before + ((incl - count) & 0xfffff);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (height[j] != h) continue;
      tab->order[at] = static_cast<uint8_t>(lane * kPer + j);
      tab->tiles[at++] = static_cast<uint16_t>(tile);
      tile += tiles[j];
    }
    const int all = __shfl_sync(0xffffffffu, incl, 31);
    pos += all >> 20;
    before += all & 0xfffff;
  }
  if (lane == 0) tab->tiles[p.g] = static_cast<uint16_t>(before);
}

__device__ __forceinline__ RowTile find_row_tile(const GemmArgs& p, const SwapGroupTable* tab, int mt) {
  int lo = 0, hi = p.g;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (tab->tiles[mid + 1] > mt) hi = mid; else lo = mid + 1;
  }
  RowTile r;
  r.group = tab->order[lo];
  r.weight = p.group_to_weight != nullptr ? p.group_to_weight[r.group] : r.group;
  r.group_offset = tab->offset[r.group];
  r.group_size = imin(tab->offset[r.group + 1] - r.group_offset, p.m - r.group_offset);
  r.tile_base = tab->tiles[lo];
  r.tiles = tab->tiles[lo + 1] - r.tile_base;
  return r;
}

// What the pairs walk: whole tiles for whole rounds, and what is left too; where that is half a round or less it is
// cut into half tiles of 256 columns, one for a pair at most.  (A last tile of a row with 256 columns or less is
// a half tile anyway.)  Microseconds, alone: m 8192, k 4096, n 5120, 8 groups,
// trans_rhs 271 -> 233; 8192, 2048, 4096, 8 139 -> 106 (in a row, at the power limit, equal: 264 and 266, 114 and 114);
// in a row float32 8192, 4096, 14336, 8 1285 -> 1254, bf16 727 -> 707.
struct SwapWork {
  int whole, items;
  __device__ __forceinline__ SwapWork(int tiles, int pairs) {
    const int left = tiles % pairs;
    const bool cut = 2 * left <= pairs;
    whole = cut ? tiles - left : tiles;
    items = cut ? tiles + left : tiles;
  }
};

template <int kStep>
__device__ __forceinline__ SwapTile decode_swap_tile(const GemmArgs& p, const SwapGroupTable* tab, const SwapWork& work,
                                                     int item) {
  const int past = item - work.whole;
  const int tile = past < 0 ? item : work.whole + (past >> 1);
  const RowTile r = find_row_tile(p, tab, tile / p.n_tiles);
  const int local = tile - r.tile_base * p.n_tiles;
  const int nt = local / r.tiles;
  const int mi = local - nt * r.tiles;
  // The group's rows in blocks of kStep, dealt evenly: a tile's time is its rows, and tiles side by side that
  // take equally long keep sharing panels.  No tile is empty or above 256 rows.
  const int blocks = (r.group_size + kStep - 1) / kStep;
  const int per = blocks / r.tiles, more = blocks - per * r.tiles;  // the first `more` tiles have one more
  const int first = (mi * per + imin(mi, more)) * kStep;
  SwapTile t;
  t.weight = r.weight;
  t.row0 = r.group_offset + first;
  t.mma_n = imax((per + (mi < more ? 1 : 0)) * kStep, kStep);
  t.rows = imax(imin(t.mma_n, r.group_size - first), 0);
  t.halves = past < 0 && p.n - nt * kSwapCols > kSwapCtaCols ? 2 : 1;
  t.n0 = nt * kSwapCols + (past < 0 ? 0 : (past & 1) * kSwapCtaCols);
  return t;
}

template <bool kBKMajor, bool kFp8, bool kF32 = false>
__global__ void __launch_bounds__(kSwapThreads, 1)
ragged_gemm_swap_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                        const __grid_constant__ CUtensorMap tmap_out, const __grid_constant__ CUtensorMap tmap_out16,
                        const GemmArgs p) {
  static_assert(!kFp8 || (kBKMajor && !kF32), "8-bit inputs: K-major weights");
  constexpr int kStages = kSwapStages;
  constexpr uint32_t kStageBytes = kSwapStageBytes;
  constexpr int kStep = kFp8 ? 32 : 16;  // what N comes in, M = 256 on a pair
  constexpr int kDeep = kF32 ? kF32TileK : kTileK;  // elements in a stage's 128 bytes of the contraction

  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t bar_full[kStages];   // leader's is used
  __shared__ __align__(8) uint64_t bar_empty[kStages];
  __shared__ __align__(8) uint64_t bar_acc_full[2];     // per half
  __shared__ __align__(8) uint64_t bar_acc_empty[2];    // per half, leader's is used
  __shared__ uint32_t tmem_slot;
  __shared__ WaitCtl wait_ctl;
  __shared__ SwapGroupTable group_table;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int cta_rank = static_cast<int>(cluster_cta_rank());
  const bool leader = cta_rank == 0;
  const uint32_t stage_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;

  if (threadIdx.x == 0) {
    wait_ctl.abort = 0;
    wait_ctl.limit_us = p.wait_limit_us;
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    tma_prefetch_desc(&tmap_out);
    tma_prefetch_desc(&tmap_out16);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(smem_u32(&bar_acc_full[h]), 1);
      mbar_init(smem_u32(&bar_acc_empty[h]), 8);  // four epilogue warps of either CTA
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc<2>(smem_u32(&tmem_slot), 512);
    tmem_relinquish<2>();
  }
  start_inline_groups(p, kSwapRows, &group_table, warp, lane);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();  // the peer's barriers exist before anything arrives on them
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  volatile WaitCtl* abort_ptr = &wait_ctl;

  const SwapWork work(live_row_tiles(p, &group_table) * p.n_tiles, static_cast<int>(gridDim.x >> 1));
  const int num_tiles = work.items;
  const int tile_start = static_cast<int>(blockIdx.x >> 1);
  const int tile_step = static_cast<int>(gridDim.x >> 1);
  const int k_blocks = (p.k + kDeep - 1) / kDeep;

  // The producer and the MMA warp run their loops as whole warps on values that the compiler knows to be uniform
  // and elect a lane for the TMA and tcgen05 instructions alone (rd_tgmm.cuh).
  auto uniform_tile = [&](int tile) {
    SwapTile t = decode_swap_tile<kStep>(p, &group_table, work, tile);
    t.weight = __shfl_sync(0xffffffffu, t.weight, 0);
    t.row0 = __shfl_sync(0xffffffffu, t.row0, 0);
    t.n0 = __shfl_sync(0xffffffffu, t.n0, 0);
    t.halves = __shfl_sync(0xffffffffu, t.halves, 0);
    t.mma_n = __shfl_sync(0xffffffffu, t.mma_n, 0);
    return t;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    uint32_t it = 0;
    bool ok = true;
    for (int tile = tile_start; tile < num_tiles && ok; tile += tile_step) {
      const SwapTile t = uniform_tile(tile);
      const int col = t.n0 + cta_rank * t.halves * kTileM;
      const uint32_t bytes = t.halves * (kSwapABytes / 2) + kSwapBBytes;  // of one CTA
      const int row = t.row0 + cta_rank * (t.mma_n >> 1);
      for (int kb = 0; kb < k_blocks; ++kb, ++it) {
        const uint32_t s = it % kStages;
        const uint32_t ph = (it / kStages) & 1u;
        if (!mbar_wait_warp(smem_u32(&bar_empty[s]), ph ^ 1u, abort_ptr)) {
          ok = false;
          break;
        }
        const uint32_t sa = stage_base + s * kStageBytes;
        const uint32_t sb = sa + kSwapABytes;
        if (elect_one()) {
          uint32_t full = smem_u32(&bar_full[s]);
          if (leader) {
            mbar_arrive_expect_tx(full, 2 * bytes);
            tma_load_2d(sb, &tmap_x, full, kb * kDeep, row);
            if constexpr (kBKMajor) {
              tma_load_3d(sa, &tmap_w, full, kb * kDeep, col, t.weight);
              if (t.halves == 2) tma_load_3d(sa + kSwapABytes / 2, &tmap_w, full, kb * kDeep, col + kTileM, t.weight);
            } else {
              tma_load_4d(sa, &tmap_w, full, 0, kb * kDeep, col / kDeep, t.weight);
              if (t.halves == 2)
                tma_load_4d(sa + kSwapABytes / 2, &tmap_w, full, 0, kb * kDeep, (col + kTileM) / kDeep, t.weight);
            }
          } else {
            full = map_to_cta(full, 0);
            tma_load_2d_pair(sb, &tmap_x, full, kb * kDeep, row);
            if constexpr (kBKMajor) {
              tma_load_3d_pair(sa, &tmap_w, full, kb * kDeep, col, t.weight);
              if (t.halves == 2) tma_load_3d_pair(sa + kSwapABytes / 2, &tmap_w, full, kb * kDeep, col + kTileM, t.weight);
            } else {
              tma_load_4d_pair(sa, &tmap_w, full, 0, kb * kDeep, col / kDeep, t.weight);
              if (t.halves == 2)
                tma_load_4d_pair(sa + kSwapABytes / 2, &tmap_w, full, 0, kb * kDeep, (col + kTileM) / kDeep, t.weight);
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (of the leader)
    if (leader) {
      constexpr uint32_t kAStep = (kBKMajor ? 32u : kF32 ? 1024u : 2048u) >> 4;
      constexpr uint32_t kBStep = 32u >> 4;
      constexpr uint32_t kHalfA = (kBKMajor ? 128u * 128u : 2u * kBoxBytes) >> 4;  // the next 128 columns
      const uint64_t adesc0 = kBKMajor ? make_smem_desc(stage_base, 16, 1024)
                              : kF32   ? make_smem_desc(stage_base, kF32BoxBytes, 512, 1)
                                       : make_smem_desc(stage_base, kBoxBytes, 1024);
      const uint64_t bdesc0 = make_smem_desc(stage_base + kSwapABytes, 16, 1024);
      const uint32_t adesc0_lo = static_cast<uint32_t>(adesc0);
      const uint32_t bdesc0_lo = static_cast<uint32_t>(bdesc0);
      const uint32_t a_hi = static_cast<uint32_t>(adesc0 >> 32);
      const uint32_t b_hi = static_cast<uint32_t>(bdesc0 >> 32);
      uint32_t it = 0;
      uint32_t uses[2] = {0u, 0u};  // of either half's accumulator
      bool ok = true;
      for (int tile = tile_start; tile < num_tiles && ok; tile += tile_step) {
        const SwapTile t = uniform_tile(tile);
        const uint32_t idesc =
            kF32 ? make_idesc_tf32(kBKMajor ? 0 : 1, 0, 2 * kTileM, t.mma_n)
                 : make_idesc_f16(kFp8 ? 0 : p.ab_format, kBKMajor ? 0 : 1, 0, 2 * kTileM, t.mma_n);
        uint32_t s = it % kStages;
        uint32_t ph = (it / kStages) & 1u;
        for (int kb = 0; kb < k_blocks; ++kb, ++it, s = (s + 1 == kStages ? 0 : s + 1), ph ^= (s == 0)) {
          if (!mbar_wait_warp(smem_u32(&bar_full[s]), ph, abort_ptr)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t b_lo = bdesc0_lo + s * (kStageBytes >> 4);
          auto issue = [&](int h, uint32_t more) {
            const uint32_t a_lo = adesc0_lo + s * (kStageBytes >> 4) + h * kHalfA;
            const uint32_t tmem_d = tmem_base + h * kSwapRows;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {  // 32 bytes of the contraction each
              const uint64_t a = make_desc64(a_lo + kk * kAStep, a_hi), b = make_desc64(b_lo + kk * kBStep, b_hi);
              if constexpr (kF32) {
                umma_tf32_pair(tmem_d, a, b, idesc, kk > 0 ? 1u : more);
              } else {
                umma_ab<2, kFp8>(tmem_d, a, b, idesc, kk > 0 ? 1u : more);
              }
            }
            if (kb == k_blocks - 1) umma_commit_pair(smem_u32(&bar_acc_full[h]), 0x3);
          };
          if (kb == 0) {  // a half's accumulator must have been drained by both CTAs
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (h >= t.halves) break;
              if (!mbar_wait_warp<true>(smem_u32(&bar_acc_empty[h]), (uses[h] & 1u) ^ 1u, abort_ptr)) {
                ok = false;
                break;
              }
              ++uses[h];
              tc_fence_after_sync();
              if (elect_one()) issue(h, 0u);
            }
            if (!ok) break;
            if (elect_one()) umma_commit_pair(smem_u32(&bar_empty[s]), 0x3);
          } else if (elect_one()) {
            issue(0, 1u);
            if (t.halves == 2) issue(1, 1u);
            umma_commit_pair(smem_u32(&bar_empty[s]), 0x3);
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9)
    const int half = (warp - 2) >> 2;
    const int quarter = warp & 3;
    const uint32_t staging = stage_base + kStages * kStageBytes + (warp - 2) * 2 * kSwapBoxBytes;
    uint32_t uses = 0;
    uint32_t boxes_stored = 0;
    bool ok = true;
    uint16_t* out16 = reinterpret_cast<uint16_t*>(p.out);
    for (int tile = tile_start; tile < num_tiles && ok; tile += tile_step) {
      const SwapTile t = decode_swap_tile<kStep>(p, &group_table, work, tile);
      if (half >= t.halves) continue;
      const int col0 = t.n0 + (cta_rank * t.halves + half) * kTileM + quarter * 32;  // this warp's first output column; lane = column
      if (!mbar_wait_warp<true>(smem_u32(&bar_acc_full[half]), uses & 1u, abort_ptr)) {
        ok = false;
        break;
      }
      ++uses;
      tc_fence_after_sync();
      const int chunks = col0 < p.n ? (t.rows + 31) >> 5 : 0;
      const float sc = kFp8 && p.weight_scale != nullptr ? p.weight_scale[t.weight] : 1.0f;
      if constexpr (kF32) {
        // 32 rows at a time as they are; the last four of these leave tensor memory together, then the accumulator
        // is handed back.  A row of 32 columns is 128 bytes: stores of a warp meet no bank twice.
        float* out32 = reinterpret_cast<float*>(p.out);
        auto store = [&](int c, const uint32_t (&v)[32]) {
          const int row0 = t.row0 + c * 32;
          const int rows = t.rows - c * 32;
#pragma unroll
          for (int h = 0; h < 2; ++h) {  // boxes of 16 rows
            if (rows < 16 * h + 16) break;
            const uint32_t buf = staging + (boxes_stored & 1u) * kSwapBoxBytes;
            if (lane == 0) bulk_wait_group_read<1>();
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 16; ++j)
              asm volatile("st.shared.b32 [%0], %1;" ::"r"(buf + j * 128 + lane * 4), "r"(v[16 * h + j]) : "memory");
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&tmap_out16, buf, col0, row0 + 16 * h);
              bulk_commit_group();
            }
            ++boxes_stored;
          }
          if (rows < 32 && (rows & 15) != 0 && col0 + lane < p.n) {  // the group's last rows
            float* dst = out32 + static_cast<size_t>(row0) * p.n + col0 + lane;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (j >= (rows & 16) && j < rows) dst[static_cast<size_t>(j) * p.n] = __uint_as_float(v[j]);
            }
          }
        };
        const uint32_t tmem = tmem_base + half * kSwapRows + (static_cast<uint32_t>(quarter * 32) << 16);
        const int early = imax(chunks - 4, 0);
#pragma unroll 1
        for (int c = 0; c < early; ++c) {
          uint32_t v[32];
          tmem_ld_32x32(tmem + c * 32, v);
          tmem_ld_wait();
          store(c, v);
        }
        uint32_t v[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (early + c < chunks) tmem_ld_32x32(tmem + (early + c) * 32, v[c]);
        }
        tmem_ld_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(smem_u32(&bar_acc_empty[half]), 0);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (early + c < chunks) store(early + c, v[c]);
        }
        continue;
      }
      // All rows leave tensor memory first (packed to 16 bits, 16 registers per 32 rows), so that the
      // next tile's MMAs wait for nothing but the loads below.
      uint32_t o[kSwapRows / 32][16];
#pragma unroll
      for (int c = 0; c < kSwapRows / 32; ++c) {
        if (c < chunks) {
          uint32_t v[32];
          tmem_ld_32x32(tmem_base + half * kSwapRows + c * 32 + (static_cast<uint32_t>(quarter * 32) << 16), v);
          tmem_ld_wait();
          if constexpr (kFp8) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * sc);
          }
#pragma unroll
          for (int j = 0; j < 16; ++j)
            o[c][j] = pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]), p.ab_format);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(smem_u32(&bar_acc_empty[half]), 0);
#pragma unroll
      for (int c = 0; c < kSwapRows / 32; ++c) {
        if (c >= chunks) continue;
        const int row0 = t.row0 + c * 32;
        const int rows = t.rows - c * 32;
        const int by_tma = rows >= 32 ? 32 : rows & 16;  // rows stored as one box of 32 or 16
        if (by_tma > 0) {
          const uint32_t buf = staging + (boxes_stored & 1u) * kSwapBoxBytes;
          if (lane == 0) bulk_wait_group_read<1>();  // the box stored two boxes ago has been read out
          __syncwarp();
          const uint32_t a = buf + lane * 2;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            asm volatile(
                "{\n\t"
                ".reg .b16 lo, hi;\n\t"
                "mov.b32 {lo, hi}, %1;\n\t"
                "st.shared.b16 [%0], lo;\n\t"
                "st.shared.b16 [%0 + 64], hi;\n\t"
                "}\n" ::"r"(a + j * 128),
                "r"(o[c][j])
                : "memory");
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(by_tma == 32 ? &tmap_out : &tmap_out16, buf, col0, row0);
            bulk_commit_group();
          }
          ++boxes_stored;
        }
        if (by_tma < imin(rows, 32) && col0 + lane < p.n) {  // the group's last rows
          uint16_t* dst = out16 + static_cast<size_t>(row0) * p.n + col0 + lane;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (j >= by_tma && j < rows) dst[static_cast<size_t>(j) * p.n] = static_cast<uint16_t>(o[c][j >> 1] >> (16 * (j & 1)));
          }
        }
      }
    }
    if (lane == 0) bulk_wait_group<0>();
    __syncwarp();

    if (p.zero_tail) {
      constexpr int kEpiThreads = 32 * kSwapEpilogueWarps;
      const int first = first_dead_row(p, &group_table);
      const size_t chunks_per_row = static_cast<size_t>(p.n) / (kF32 ? 4 : 8);
      const size_t total = static_cast<size_t>(p.m - first) * chunks_per_row;
      const size_t tid = static_cast<size_t>(blockIdx.x) * kEpiThreads + (threadIdx.x - 64);
      const size_t stride = static_cast<size_t>(gridDim.x) * kEpiThreads;
      uint4* dst = reinterpret_cast<uint4*>(p.out) + static_cast<size_t>(first) * chunks_per_row;
      const uint4 z = make_uint4(0u, 0u, 0u, 0u);
      for (size_t i = tid; i < total; i += stride) dst[i] = z;
    }
  }

  // ------------------------------------------------------------ tear-down
  __syncthreads();
  if (wait_ctl.abort) {
    if (threadIdx.x == 0) atomicMax(p.status, static_cast<int32_t>(kStatusWaitExpired));
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync();  // neither CTA may leave while the other can still reach its barriers or smem
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<2>(tmem_base, 512);
  }
}

}  // namespace rd
