// tgmm, out[i] = x[rows of group i]^T @ dout[rows of group i], with two accumulators per CTA.
//
// A tile contracts over the rows of one group only, often a few 64-row stages, so what bounds it is as
// much the way from one tile to the next as the MMAs.  A CTA owns 128 x 256 tiles (kCtas 2: a pair
// 256 x 256, each CTA its own 128 rows of x^T and half of dout's columns) and has two of them in tensor
// memory: while the MMAs fill one, four of eight epilogue warps (all eight on one CTA) drain the other.  The 256 x 256 tiles per CTA
// that stood here before moved less per flop but left the drain exposed, 5000 clocks per tile.
//
// What made the smaller tiles fast enough is the issue path.  A 64-row stage takes 512 clocks of MMAs here.
// With producer and MMA loops run by one thread (lane == 0) a stage's four MMAs and commit take 420 clocks to issue, and
// its two boxes of loads 395, beside the waits (clock64 around them).  Run by a whole warp on values that the compiler knows to
// be the same in every lane, with a lane elected for the instructions alone, they take 240 and 290 (the same kernel: m 8192,
// k 4096, n 14336, 8 groups 938 -> 722 us).
// The order of tiles is walked without divisions (TgmmWalk), which had taken 650 clocks a tile.
//
// Rows past a group's end in its last stage are cleared by a fixer warp as soon as the stage has landed,
// ahead of the MMAs: such a stage is counted on a barrier of its own (bar_land), and "full" is raised by the
// fixer.
//
// Microseconds in a row, the 256 x 256 (or 512 x 256 pair) tiles before against this: m 8192, k 4096, n 14336, 8
// unequal groups 862 -> 722; 64 groups of 512, k 4096, n 1536 442 -> 391; 128 heavy-tailed groups of 128, k 7168, n
// 2048 989 -> 851; 30 groups of 100, k 2048, n 2048 75 -> 69.
// What bounds it now: long groups the power limit (1.3 GHz); short ones the output: an SM
// sends 128 bytes in five clocks at best, 2560 clocks a tile, and takes 2830 with loads of two stages in between
// (7.5 GB of output at 5.0 TB/s and 1.5 GHz, again at the power limit).
#pragma once

#include "rd_gemm2.cuh"

namespace rd {

constexpr int kTgEpilogueWarps = 8;
constexpr int kTgFixerWarp = 2 + kTgEpilogueWarps;
constexpr int kTgThreads = 64 + 32 * kTgEpilogueWarps + 32;
constexpr int kTgTileN = 256;

template <int kCtas>
__host__ __device__ constexpr uint32_t tg_stage_bytes() {
  return kTileM * kTileK * 2 + kTgTileN / kCtas * kTileK * 2;  // 48 KB on one CTA, 32 KB of each CTA of a pair
}
template <int kCtas>
__host__ __device__ constexpr int tg_stages() {
  return kCtas == 2 ? 5 : 3;
}
template <int kCtas>
__host__ __device__ constexpr int tg_smem_bytes() {
  return tg_stages<kCtas>() * tg_stage_bytes<kCtas>() + kTgEpilogueWarps * 2 * kOutBoxBytes + 1024;
}

// n / d for n * d < 2^32 by one multiplication: mul = floor(2^32 / d) + 1 (0: d is 1).
struct FastDiv {
  uint32_t d, mul;
  __device__ __forceinline__ explicit FastDiv(int d_) : d(d_), mul(d_ > 1 ? 0xffffffffu / static_cast<uint32_t>(d_) + 1u : 0u) {}
  __device__ __forceinline__ int div(int n) const { return mul == 0 ? n : static_cast<int>(__umulhi(n, mul)); }
};

struct TgmmTile : TileCoord {
  int blocks;  // columns of the tile in blocks of 64, 1 to 4
};

// The columns of the output are dealt to its n_tiles tiles evenly in blocks of 64: every tile has its way through the
// pipeline, so a narrow last one takes nearly as long as a wide one, and CTAs that write neighbouring columns stay side
// by side.  128 heavy-tailed groups of 42, k 4096, n 1392, microseconds in a row: 380 -> 261, n 1400 569 -> 428.
// The tiles of one CTA (or pair), first, first + step, ..., in the order of decode_tgmm_tile256: bands of
// kG2TgmmBand column tiles, in a band all k tiles.  No division per tile.
template <int kRows>
struct TgmmWalk {
  int tile, step, group, rem, step_groups, step_rem, per_group, last_width, last_band, per_tile, wide_tiles;
  FastDiv by_band, by_last;
  bool exact;
  __device__ __forceinline__ TgmmWalk(const GemmArgs& p, int first, int step_)
      : tile(first), step(step_), per_group(p.k_tiles * p.n_tiles),
        last_width((p.n_tiles - 1) % kG2TgmmBand + 1), last_band((p.n_tiles - 1) / kG2TgmmBand),
        by_band(p.k_tiles * kG2TgmmBand), by_last(last_width) {
    group = first / per_group;
    rem = first - group * per_group;
    const int blocks = (p.n + 63) >> 6;
    per_tile = blocks / p.n_tiles;
    wide_tiles = blocks - per_tile * p.n_tiles;  // this many tiles have one block more
    step_groups = step / per_group;
    step_rem = step - step_groups * per_group;
    exact = static_cast<unsigned long long>(per_group) * by_band.d < (1ull << 32);
  }
  __device__ __forceinline__ void next() {
    tile += step;
    group += step_groups;
    rem += step_rem;
    if (rem >= per_group) {
      rem -= per_group;
      ++group;
    }
  }
  __device__ __forceinline__ TgmmTile coord(const GemmArgs& p, const GroupTable* tab) const {
    const int band = exact ? by_band.div(rem) : rem / static_cast<int>(by_band.d);
    const int in_band = rem - band * static_cast<int>(by_band.d);
    const bool last = band == last_band;
    const int kt = !last ? in_band / kG2TgmmBand : exact ? by_last.div(in_band) : in_band / last_width;
    TgmmTile t;
    t.group = group;
    t.weight = group;
    group_rows(p, tab, group, t.row0, t.rows);
    const int width = last ? last_width : kG2TgmmBand;
    // A CTA's next tile lies `step` further on: where that shares a factor with the tiles of a row, it would meet the
    // same columns again and again, wide ones or narrow ones.  Turned by a place per row, it meets them all.
    const int turn = p.turn_columns ? kt + group : 0;
    int nt = in_band - kt * width + turn - (!last ? turn & ~(kG2TgmmBand - 1) : (exact ? by_last.div(turn) : turn / last_width) * last_width);
    nt = band * kG2TgmmBand + (nt < width ? nt : nt - width);
    t.n0 = (nt * per_tile + imin(nt, wide_tiles)) * 64;
    t.blocks = per_tile + (nt < wide_tiles ? 1 : 0);
    t.k0 = kt * kRows;
    return t;
  }
};

template <int kCtas>
__global__ void __launch_bounds__(kTgThreads, 1)
ragged_tgmm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_a2,
                   const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ CUtensorMap tmap_b2,
                   const __grid_constant__ CUtensorMap tmap_out, const GemmArgs p) {
  constexpr bool kPair = kCtas == 2;
  constexpr int kStages = tg_stages<kCtas>();
  constexpr uint32_t kABytes = kTileM * kTileK * 2;
  constexpr uint32_t kStageBytes = tg_stage_bytes<kCtas>();
  constexpr int BN = kTgTileN;

  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t bar_full[kStages];   // a stage is ready for the MMAs (pair: the leader's is used)
  __shared__ __align__(8) uint64_t bar_empty[kStages];  // its MMAs have retired
  __shared__ __align__(8) uint64_t bar_land[kStages];   // a stage whose tail rows must be cleared has landed in this CTA
  __shared__ __align__(8) uint64_t bar_acc_full[2];
  __shared__ __align__(8) uint64_t bar_acc_empty[2];    // pair: the leader's is used
  __shared__ uint32_t tmem_slot;
  __shared__ WaitCtl wait_ctl;
  __shared__ GroupTable group_table;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int cta_rank = kPair ? static_cast<int>(cluster_cta_rank()) : 0;
  const bool leader = cta_rank == 0;
  const uint32_t stage_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;

  if (threadIdx.x == 0) {
    wait_ctl.abort = 0;
    wait_ctl.limit_us = p.wait_limit_us;
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_a2);
    tma_prefetch_desc(&tmap_b2);
    tma_prefetch_desc(&tmap_out);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), kCtas);  // two arrivals of the leader's producer, or one of either fixer warp
      mbar_init(smem_u32(&bar_empty[s]), 1);
      mbar_init(smem_u32(&bar_land[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bar_acc_full[a]), 1);
      mbar_init(smem_u32(&bar_acc_empty[a]), kPair ? 8 : kTgEpilogueWarps);
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc<kCtas>(smem_u32(&tmem_slot), 2 * BN);
    tmem_relinquish<kCtas>();
  }
  start_inline_groups(p, kTileM, &group_table, warp, lane);
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (kPair) cluster_sync();  // the peer's barriers exist before anything arrives on them
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  volatile WaitCtl* abort_ptr = &wait_ctl;

  const int num_tiles = p.g * p.k_tiles * p.n_tiles;
  const int tile_start = static_cast<int>(blockIdx.x) / kCtas;
  const int tile_step = static_cast<int>(gridDim.x) / kCtas;
  using Walk = TgmmWalk<kTileM * kCtas>;
  // The producer and the MMA warp run their loops as whole warps whose values the compiler knows to be
  // uniform, and elect a lane for each stage's instructions alone (see above).
  auto uniform_coord = [&](const Walk& w) {
    TgmmTile t = w.coord(p, &group_table);
    t.row0 = __shfl_sync(0xffffffffu, t.row0, 0);
    t.rows = __shfl_sync(0xffffffffu, t.rows, 0);
    return t;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    uint32_t it = 0;
    bool ok = true;
    const uint64_t keep = l2_policy_evict_last();
    for (Walk w(p, tile_start, tile_step); w.tile < num_tiles && ok; w.next()) {
      const TgmmTile t = uniform_coord(w);
      const int kb_count = (t.rows + kTileK - 1) / kTileK;
      const bool tail = tail_needs_clearing(t.rows);
      const int cols = t.blocks * 64 / kCtas;         // of this CTA
      const int boxes = (t.blocks + kCtas - 1) / kCtas;  // what they take in boxes of 64
      const int ka = t.k0 + cta_rank * kTileM;
      const int nb = t.n0 + cta_rank * cols;
      // One box of whole 64-column blocks per operand; at the edge of rows that are not made of
      // such blocks, or for fewer columns, one box per 64 columns.
      const bool a_blocks = (p.k & 63) == 0 || ka + kTileM <= p.k;
      const bool b_blocks = t.blocks == BN / 64 && ((p.n & 63) == 0 || nb + cols <= p.n);
      const uint32_t bytes = kABytes + boxes * kBoxBytes;
      for (int kb = 0; kb < kb_count; ++kb, ++it) {
        const uint32_t s = it % kStages;
        const uint32_t ph = (it / kStages) & 1u;
        if (!mbar_wait_warp(smem_u32(&bar_empty[s]), ph ^ 1u, abort_ptr)) {
          ok = false;
          break;
        }
        const uint32_t sa = stage_base + s * kStageBytes;
        const uint32_t sb = sa + kABytes;
        const int r = t.row0 + kb * kTileK;
        // A stage whose tail rows must be cleared is counted where it lands: that CTA's fixer warp
        // clears it and then reports to the leader's "full" barrier.
        const bool own = tail && kb == kb_count - 1;
        if (elect_one()) {
          uint32_t bar = smem_u32(own ? &bar_land[s] : &bar_full[s]);
          if (own || leader) {
            mbar_arrive_expect_tx(bar, own ? bytes : kCtas * bytes);
            if (kPair && !own) mbar_arrive(bar);
            if (a_blocks) {
              tma_load_3d_hint(sa, &tmap_a, bar, 0, r, ka >> 6, keep);
            } else {
              tma_load_2d_hint(sa, &tmap_a2, bar, ka, r, keep);
              tma_load_2d_hint(sa + kBoxBytes, &tmap_a2, bar, ka + 64, r, keep);
            }
            if (b_blocks) {
              tma_load_3d_hint(sb, &tmap_b, bar, 0, r, nb >> 6, keep);
            } else {
              for (int j = 0; j < boxes; ++j) tma_load_2d_hint(sb + j * kBoxBytes, &tmap_b2, bar, nb + j * 64, r, keep);
            }
          } else {
            bar = map_to_cta(bar, 0);
            if (a_blocks) {
              tma_load_3d_pair_hint(sa, &tmap_a, bar, 0, r, ka >> 6, keep);
            } else {
              tma_load_2d_pair_hint(sa, &tmap_a2, bar, ka, r, keep);
              tma_load_2d_pair_hint(sa + kBoxBytes, &tmap_a2, bar, ka + 64, r, keep);
            }
            if (b_blocks) {
              tma_load_3d_pair_hint(sb, &tmap_b, bar, 0, r, nb >> 6, keep);
            } else {
              for (int j = 0; j < boxes; ++j)
                tma_load_2d_pair_hint(sb + j * kBoxBytes, &tmap_b2, bar, nb + j * 64, r, keep);
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (of the leader)
    if (leader) {
      constexpr uint32_t kStep = 2048u >> 4;  // both operands MN-major: 16 rows of the contraction
      const uint64_t adesc0 = make_smem_desc(stage_base, kBoxBytes, 1024);
      const uint64_t bdesc0 = make_smem_desc(stage_base + kABytes, kBoxBytes, 1024);
      const uint32_t adesc0_lo = static_cast<uint32_t>(adesc0);
      const uint32_t bdesc0_lo = static_cast<uint32_t>(bdesc0);
      const uint32_t desc_hi = static_cast<uint32_t>(adesc0 >> 32);
      uint32_t it = 0;
      uint32_t local_tile = 0;
      bool ok = true;
      for (Walk w(p, tile_start, tile_step); w.tile < num_tiles && ok; w.next(), ++local_tile) {
        const TgmmTile t = uniform_coord(w);
        const int kb_count = (t.rows + kTileK - 1) / kTileK;
        const bool tail = tail_needs_clearing(t.rows);
        const uint32_t idesc = make_idesc_f16(p.ab_format, 1, 1, kTileM * kCtas, t.blocks * 64);
        const uint32_t acc = local_tile & 1u;
        if (!mbar_wait_warp<kPair>(smem_u32(&bar_acc_empty[acc]), ((local_tile >> 1) & 1u) ^ 1u, abort_ptr)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + acc * BN;
        uint32_t s = it % kStages;
        uint32_t ph = (it / kStages) & 1u;
        for (int kb = 0; kb < kb_count; ++kb, ++it, s = (s + 1 == kStages ? 0 : s + 1), ph ^= (s == 0)) {
          const bool last = kb == kb_count - 1;
          const bool cleared = kPair && tail && last;  // reported by both fixer warps: see the peer's, too
          if (!(cleared ? mbar_wait_warp<kPair>(smem_u32(&bar_full[s]), ph, abort_ptr)
                        : mbar_wait_warp(smem_u32(&bar_full[s]), ph, abort_ptr))) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t a_lo = adesc0_lo + s * (kStageBytes >> 4);
          const uint32_t b_lo = bdesc0_lo + s * (kStageBytes >> 4);
          const int live = t.rows - kb * kTileK;
          if (elect_one()) {
            if (live <= kTileK - kUmmaK) {
              const int n_mma = (live + kUmmaK - 1) / kUmmaK;
              for (int kk = 0; kk < n_mma; ++kk)
                umma_ab<kCtas, false>(tmem_d, make_desc64(a_lo + kk * kStep, desc_hi),
                                      make_desc64(b_lo + kk * kStep, desc_hi), idesc, (kb > 0 || kk > 0) ? 1u : 0u);
            } else {
#pragma unroll
              for (int kk = 0; kk < kTileK / kUmmaK; ++kk)
                umma_ab<kCtas, false>(tmem_d, make_desc64(a_lo + kk * kStep, desc_hi),
                                      make_desc64(b_lo + kk * kStep, desc_hi), idesc, (kb > 0 || kk > 0) ? 1u : 0u);
            }
            if constexpr (kPair) {
              umma_commit_pair(smem_u32(&bar_empty[s]), 0x3);
            } else {
              umma_commit(smem_u32(&bar_empty[s]));
            }
          }
        }
        if (!ok) break;
        const uint32_t bar = smem_u32(&bar_acc_full[acc]);
        if (elect_one()) {
          if (kb_count == 0) {  // empty group: the epilogue writes zeros
            mbar_arrive(bar);
            if constexpr (kPair) mbar_arrive_cluster(bar, 1);
          } else if constexpr (kPair) {
            umma_commit_pair(bar, 0x3);
          } else {
            umma_commit(bar);
          }
        }
      }
    }
  } else if (warp == kTgFixerWarp) {
    // ------------------------------------------------------------ tail fixer
    uint32_t it = 0;
    uint32_t parity = 0;  // bit s: parity of the next landing on bar_land[s]
    for (Walk w(p, tile_start, tile_step); w.tile < num_tiles; w.next()) {
      const TgmmTile t = w.coord(p, &group_table);
      const int kb_count = (t.rows + kTileK - 1) / kTileK;
      it += kb_count;
      if (kb_count == 0 || !tail_needs_clearing(t.rows)) continue;
      const uint32_t s = (it - 1) % kStages;
      if (!mbar_wait_warp(smem_u32(&bar_land[s]), (parity >> s) & 1u, abort_ptr)) break;
      parity ^= 1u << s;
      clear_tail_rows<kStageBytes / kBoxBytes>(stage_base + s * kStageBytes, t.rows - (kb_count - 1) * kTileK, lane);
      __syncwarp();
      if (lane == 0) {
        if constexpr (kPair) {
          mbar_arrive_cluster(smem_u32(&bar_full[s]), 0);
        } else {
          mbar_arrive(smem_u32(&bar_full[s]));
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // Of a pair: warps 2..5 drain accumulator 0, 6..9 accumulator 1.  On one CTA: 2..5 the first 128 columns of
    // every tile, 6..9 the others, so that neighbouring columns are written at nearly the same time.
    const int side = (warp - 2) >> 2;
    const int quarter = warp & 3;
    const uint32_t buf = stage_base + kStages * kStageBytes + (warp - 2) * 2 * kOutBoxBytes;
    const uint64_t stream_out = l2_policy_evict_first();
    const int skip = kPair ? side : 0, every = kPair ? 2 : 1;
    uint32_t uses = 0;
    for (Walk w(p, tile_start + skip * tile_step, every * tile_step); w.tile < num_tiles; w.next(), ++uses) {
      const TgmmTile t = w.coord(p, &group_table);
      const uint32_t acc = kPair ? side : uses & 1u;
      const uint32_t phase = (kPair ? uses : uses >> 1) & 1u;
      const int out_row0 = t.k0 + cta_rank * kTileM + quarter * 32;
      const int first = kPair ? 0 : 2 * side;  // 64-column blocks [first, chunks) are this warp's
      const int chunks = out_row0 < p.k ? imin(t.blocks, kPair ? 4 : first + 2) : 0;
      const bool zero_only = t.rows <= 0;
      if (!mbar_wait_warp<kPair>(smem_u32(&bar_acc_full[acc]), phase, abort_ptr)) break;
      tc_fence_after_sync();
      auto hand_back = [&]() {  // everything this warp needs of the accumulator is in registers
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          if constexpr (kPair) {
            mbar_arrive_cluster(smem_u32(&bar_acc_empty[acc]), 0);
          } else {
            mbar_arrive(smem_u32(&bar_acc_empty[acc]));
          }
        }
      };
#pragma unroll 1
      for (int c = first; c < chunks; c += 2) {  // 128 columns at a time
        uint4 o[4][4];
#pragma unroll
        for (int b = 0; b < 4; b += 2) {
          uint32_t v[64];
          if (!zero_only) {
            const uint32_t taddr = tmem_base + acc * BN + c * 64 + b * 32 + (static_cast<uint32_t>(quarter * 32) << 16);
            tmem_ld_32x32(taddr, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
            tmem_ld_32x32(taddr + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int j = 0; j < 64; ++j) v[j] = 0u;
          }
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            o[b + (q >> 2)][q & 3].x = pack2(__uint_as_float(v[q * 8 + 0]), __uint_as_float(v[q * 8 + 1]), p.ab_format);
            o[b + (q >> 2)][q & 3].y = pack2(__uint_as_float(v[q * 8 + 2]), __uint_as_float(v[q * 8 + 3]), p.ab_format);
            o[b + (q >> 2)][q & 3].z = pack2(__uint_as_float(v[q * 8 + 4]), __uint_as_float(v[q * 8 + 5]), p.ab_format);
            o[b + (q >> 2)][q & 3].w = pack2(__uint_as_float(v[q * 8 + 6]), __uint_as_float(v[q * 8 + 7]), p.ab_format);
          }
        }
        if (c + 2 >= chunks) hand_back();
        if (lane == 0) bulk_wait_group_read<0>();  // the boxes stored before have left the buffers
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t row_addr = buf + h * kOutBoxBytes + lane * 128;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint4 v = o[2 * h + (q >> 2)][q & 3];
            const uint32_t a = row_addr + (((q ^ (lane & 7)) & 7) << 4);  // 128-byte swizzle
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                         : "memory");
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_3d_hint(&tmap_out, buf, t.n0 + c * 64, out_row0, t.group, stream_out);
          if (c + 1 < chunks)
            tma_store_3d_hint(&tmap_out, buf + kOutBoxBytes, t.n0 + (c + 1) * 64, out_row0, t.group, stream_out);
          bulk_commit_group();
        }
      }
      if (chunks <= first) hand_back();
    }
    if (lane == 0) bulk_wait_group<0>();
    __syncwarp();
  }

  // ------------------------------------------------------------ tear-down
  __syncthreads();
  if (wait_ctl.abort) {
    if (threadIdx.x == 0) atomicMax(p.status, static_cast<int32_t>(kStatusWaitExpired));
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if constexpr (kPair) cluster_sync();  // neither CTA may leave while the other can still reach its barriers or smem
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<kCtas>(tmem_base, 2 * BN);
  }
}

}  // namespace rd
