// float32 grouped GEMM kernels on CTA pairs, float32 output: three-pass gmm / gmm trans_rhs / tgmm, one-pass tgmm.
//
//   kSplit == false  one TF32 pass (the same arithmetic as ragged_gemm_f32_kernel), tgmm only
//   kSplit == true   nearly float32 accuracy: every operand is split into a TF32 head and a
//                    remainder, t = hi + lo, and a.b ~ lo.hi + hi.lo + hi.hi (the dropped lo.lo
//                    term is 2^-22 relative).  The two small products have an accumulator of
//                    their own, so that the order of their additions does not disturb the sum of
//                    the large one; the epilogue adds the two in fp32.
//
// Two CTAs of a cluster own a 256 x 256 tile (tcgen05.mma.cta_group::2, M = N = 256): CTA c loads
// rows [128 c, 128 c + 128) of the A operand and columns [128 c, 128 c + 128) of the B operand,
// 32 KB per 32-deep stage for the MMAs of 128 x 256 outputs per SM, where one CTA per tile loads
// 48 KB; nothing is broadcast.
//
// kSplit works on operands as they lie in HBM: eight converter warps read a landed stage, write
// the heads back in place and the remainders into a second 32 KB (the split is element by
// element, so the swizzled layout does not matter), and the MMA thread issues the three products
// of a stage from the two.  Per stage of 3 x 512 tensor-core clocks shared memory moves 32 KB by
// TMA, 96 KB by the converters and 96 KB to the tensor cores: about 1800 clocks at 128 bytes per
// clock, so this kernel is bound by shared memory, close to the tensor pipe.  A single CTA per tile
// would move 336 KB, half as much again; splitting in a kernel of its own would add a read of every operand
// and a write of twice its size to HBM.
//
// Measured (m 4096, k 4096, n 1536, 8 groups, three products): 0.25 / 0.25 / 0.24 ms for gmm / trans_rhs
// / tgmm = 610 to 640 TFLOP/s of TF32 MMAs, where splitting in torch and three launches took 0.99 /
// 0.92 / 0.85 ms; forward + backward 2.78 -> 0.87 ms.  The [32][32] boxes of an MN-major operand come as ONE
// box of a column-blocked view where its rows are multiples of 32; other rows, four 4 KB boxes per operand,
// only reach the three-product form.  One product, measured on both sides: choose_f32_pair in rd_api.cu.
//
// Roles: warp 0 = TMA producer, warp 1 = MMA issuer (of the leader CTA), warps 2..5 =
// epilogue, warps 6.. = converters (kSplit, eight) or the tail fixer (one, tgmm).  tgmm rows past
// a group's end are cleared by the converters as they pass, or by the fixer as in rd_gemm.cuh.
// Operand layouts are those of rd_gemm_f32.cuh; waits are bounded as everywhere.
// The producer and the MMA warp run their loops as whole warps and elect a lane per stage (rd_tgmm.cuh): one-product tgmm,
// m 8192, k 4096, n 1536, 8 groups 201 -> 182 us, three products forward + backward, m 4096, 872 -> 863.
#pragma once

#include "rd_gemm_f32.cuh"

namespace rd {

constexpr int kF32PairBN = 256;
constexpr int kF32ConvWarps = 8;
constexpr int kF32ConvWarp0 = 6;
constexpr uint32_t kF32PairABytes = kTileM * 128;               // this CTA's 128 rows
constexpr uint32_t kF32PairBBytes = (kF32PairBN / 2) * 128;     // this CTA's 128 columns
constexpr uint32_t kF32PairRawBytes = kF32PairABytes + kF32PairBBytes;  // 32 KB

template <bool kSplit>
__host__ __device__ constexpr int f32_pair_threads() { return 32 * (kF32ConvWarp0 + (kSplit ? kF32ConvWarps : 1)); }
template <bool kSplit>
__host__ __device__ constexpr int f32_pair_stages() { return kSplit ? 3 : 6; }
template <bool kSplit>
__host__ __device__ constexpr uint32_t f32_pair_stage_bytes() { return kSplit ? 2 * kF32PairRawBytes : kF32PairRawBytes; }
template <bool kSplit>
__host__ __device__ constexpr int f32_pair_smem_bytes() {
  return f32_pair_stages<kSplit>() * f32_pair_stage_bytes<kSplit>() + kOutStagingBytes + 1024;
}

__device__ __forceinline__ void umma_tf32_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                               uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// t = hi + lo exactly: hi keeps the top 10 explicit mantissa bits, rounded to nearest (the tensor
// cores read it without loss).  Where that rounds up to infinity, and for values that are not
// finite, hi = t.
__device__ __forceinline__ void split_tf32(uint32_t bits, uint32_t& hi, uint32_t& lo) {
  uint32_t h = (bits + 0x1000u) & ~0x1fffu;
  if ((h & 0x7f800000u) == 0x7f800000u) h = bits;
  hi = h;
  lo = __float_as_uint(__uint_as_float(bits) - __uint_as_float(h));
}

template <bool kBKMajor, bool kTgmm, bool kSplit>
__global__ void __launch_bounds__(f32_pair_threads<kSplit>(), 1)
ragged_gemm_f32_pair_kernel(const __grid_constant__ CUtensorMap tmap_a,
                            const __grid_constant__ CUtensorMap tmap_b,
                            const __grid_constant__ CUtensorMap tmap_out, const GemmArgs p) {
  static_assert(!(kTgmm && kBKMajor), "tgmm reads both operands MN-major");
  static_assert(kSplit || kTgmm, "one-pass gmm runs on one CTA per tile");
  constexpr int BN = kF32PairBN;
  constexpr int kBCols = BN / 2;
  constexpr int kStages = f32_pair_stages<kSplit>();
  constexpr uint32_t kStageBytes = f32_pair_stage_bytes<kSplit>();
  constexpr int kChunkCols = 32;  // fp32 columns per 128-byte output row

  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t bar_full[kStages];   // TMA data landed
  __shared__ __align__(8) uint64_t bar_conv[kStages];   // kSplit: both CTAs' converters are done (leader's is used)
  __shared__ __align__(8) uint64_t bar_empty[kStages];  // MMAs reading the stage retired
  __shared__ __align__(8) uint64_t bar_tail_go;
  __shared__ __align__(8) uint64_t bar_tail_done;  // leader's is used
  __shared__ __align__(8) uint64_t bar_acc_full[2];
  __shared__ __align__(8) uint64_t bar_acc_empty[2];  // leader's is used
  __shared__ uint32_t tmem_slot;
  __shared__ WaitCtl wait_ctl;
  __shared__ GroupTable group_table;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int cta_rank = static_cast<int>(cluster_cta_rank());
  const bool leader = cta_rank == 0;
  const uint32_t stage_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;

  if (threadIdx.x == 0) {
    wait_ctl.abort = 0;
    wait_ctl.limit_us = p.wait_limit_us;
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_out);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_conv[s]), 2 * kF32ConvWarps);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    mbar_init(smem_u32(&bar_tail_go), 1);
    mbar_init(smem_u32(&bar_tail_done), 2);
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bar_acc_full[a]), 1);
      mbar_init(smem_u32(&bar_acc_empty[a]), 8);  // four epilogue warps of either CTA
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc<2>(smem_u32(&tmem_slot), 2 * BN);
    tmem_relinquish<2>();
  }
  start_inline_groups(p, 2 * kTileM, &group_table, warp, lane);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();  // the peer's barriers exist before anything arrives on them
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  volatile WaitCtl* abort_ptr = &wait_ctl;

  const int num_tiles =
      kTgmm ? p.g * p.k_tiles * p.n_tiles : live_row_tiles(p, &group_table) * p.n_tiles;
  const int tile_start = static_cast<int>(blockIdx.x >> 1);
  const int tile_step = static_cast<int>(gridDim.x >> 1);
  const int k_blocks_gmm = (p.k + kF32TileK - 1) / kF32TileK;
  auto decode = [&](int tile) -> TileCoord {
    return kTgmm ? decode_tgmm_tile<BN, 2>(p, &group_table, tile, cta_rank) : decode_gmm_tile<BN, 2>(p, &group_table, tile, cta_rank);
  };
  auto blocks_of = [&](const TileCoord& t) -> int {
    return kTgmm ? (t.rows + kF32TileK - 1) / kF32TileK : k_blocks_gmm;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    uint32_t it = 0;
    bool ok = true;
    for (int tile = tile_start; tile < num_tiles && ok; tile += tile_step) {
      const TileCoord t = uniform_coord(decode(tile));
      const int nb = t.n0 + cta_rank * kBCols;  // first B column this CTA loads
      const int kb_count = blocks_of(t);
      for (int kb = 0; kb < kb_count; ++kb, ++it) {
        const uint32_t s = it % kStages;
        const uint32_t ph = (it / kStages) & 1u;
        if (!mbar_wait_warp(smem_u32(&bar_empty[s]), ph ^ 1u, abort_ptr)) {
          ok = false;
          break;
        }
        if (!elect_one()) continue;
        uint32_t full = smem_u32(&bar_full[s]);
        const uint32_t sa = stage_base + s * kStageBytes;
        const uint32_t sb = sa + kF32PairABytes;
        // kSplit: each CTA's converters wait for that CTA's own data.  Otherwise the peer's bytes
        // are counted on the leader's barrier, except for a stage whose tail rows it clears first.
        const bool local_stage = kSplit || (kTgmm && kb == kb_count - 1 && tail_needs_clearing_f32(t.rows));
        bool remote_bar = false;
        if (leader) {
          mbar_arrive_expect_tx(full, local_stage ? kF32PairRawBytes : 2 * kF32PairRawBytes);
        } else if (local_stage) {
          mbar_arrive_expect_tx(full, kF32PairRawBytes);
        } else {
          full = map_to_cta(full, 0);
          remote_bar = true;
        }
        if (kTgmm) {
          const int r = t.row0 + kb * kF32TileK;
          if (!kSplit || p.blocked_maps) {  // one box per operand: (32 columns, 32 rows, 4 blocks of 32 columns)
            load_3d(remote_bar, sa, &tmap_a, full, 0, r, t.k0 >> 5);
            load_3d(remote_bar, sb, &tmap_b, full, 0, r, nb >> 5);
          } else {
#pragma unroll
            for (int j = 0; j < kTileM / 32; ++j)
              load_2d(remote_bar, sa + j * kF32BoxBytes, &tmap_a, full, t.k0 + j * 32, r);
#pragma unroll
            for (int j = 0; j < kBCols / 32; ++j)
              load_2d(remote_bar, sb + j * kF32BoxBytes, &tmap_b, full, nb + j * 32, r);
          }
        } else {
          load_2d(remote_bar, sa, &tmap_a, full, kb * kF32TileK, t.row0);
          if (kBKMajor) {
            load_3d(remote_bar, sb, &tmap_b, full, kb * kF32TileK, nb, t.weight);
          } else if (p.blocked_maps) {  // (32 columns, 32 rows of k, 4 blocks of 32 columns, weight)
            if (remote_bar) {
              tma_load_4d_pair(sb, &tmap_b, full, 0, kb * kF32TileK, nb >> 5, t.weight);
            } else {
              tma_load_4d(sb, &tmap_b, full, 0, kb * kF32TileK, nb >> 5, t.weight);
            }
          } else {
#pragma unroll
            for (int j = 0; j < kBCols / 32; ++j)
              load_3d(remote_bar, sb + j * kF32BoxBytes, &tmap_b, full, nb + j * 32, kb * kF32TileK, t.weight);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (of the leader)
    if (leader) {
      const uint32_t idesc = make_idesc_tf32(kTgmm ? 1 : 0, kBKMajor ? 0 : 1, 2 * kTileM, BN);
      constexpr uint32_t kAStep = (kTgmm ? 1024u : 32u) >> 4;  // 8 k-rows of 128 B, or 8 k-elements
      constexpr uint32_t kBStep = (kBKMajor ? 32u : 1024u) >> 4;
      const uint64_t adesc0 = kTgmm ? make_smem_desc(stage_base, kF32BoxBytes, 512, 1)
                                    : make_smem_desc(stage_base, 16, 1024, 2);
      const uint64_t bdesc0 = kBKMajor ? make_smem_desc(stage_base + kF32PairABytes, 16, 1024, 2)
                                       : make_smem_desc(stage_base + kF32PairABytes, kF32BoxBytes, 512, 1);
      const uint32_t adesc0_lo = static_cast<uint32_t>(adesc0);
      const uint32_t bdesc0_lo = static_cast<uint32_t>(bdesc0);
      const uint32_t a_hi = static_cast<uint32_t>(adesc0 >> 32);
      const uint32_t b_hi = static_cast<uint32_t>(bdesc0 >> 32);
      constexpr uint32_t kLo = kF32PairRawBytes >> 4;  // remainders lie 32 KB behind the heads
      uint32_t it = 0;
      uint32_t local_tile = 0;
      uint32_t tail_events = 0;
      bool ok = true;
      for (int tile = tile_start; tile < num_tiles && ok; tile += tile_step, ++local_tile) {
        const TileCoord t = uniform_coord(decode(tile));
        const int kb_count = blocks_of(t);
        const bool tail_stage = !kSplit && kTgmm && kb_count > 0 && tail_needs_clearing_f32(t.rows);
        // kSplit: one tile at a time, large products in columns [0, BN), small ones in [BN, 2 BN).
        const uint32_t acc = kSplit ? 0u : (local_tile & 1u);
        const uint32_t acc_ph = kSplit ? (local_tile & 1u) : ((local_tile >> 1) & 1u);
        if (!mbar_wait_warp<true>(smem_u32(&bar_acc_empty[acc]), acc_ph ^ 1u, abort_ptr)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + acc * BN;
        uint32_t s = it % kStages;
        uint32_t ph = (it / kStages) & 1u;
        for (int kb = 0; kb < kb_count; ++kb, ++it, s = (s + 1 == kStages ? 0 : s + 1), ph ^= (s == 0)) {
          const uint32_t landed = kSplit ? smem_u32(&bar_conv[s]) : smem_u32(&bar_full[s]);
          if (!mbar_wait_warp<kSplit>(landed, ph, abort_ptr)) {
            ok = false;
            break;
          }
          if (!kSplit && kTgmm && tail_stage && kb == kb_count - 1) {
            if (elect_one()) {
              mbar_arrive(smem_u32(&bar_tail_go));
              mbar_arrive_cluster(smem_u32(&bar_tail_go), 1);
            }
            if (!mbar_wait_warp<true>(smem_u32(&bar_tail_done), tail_events & 1u, abort_ptr)) {
              ok = false;
              break;
            }
            ++tail_events;
          }
          tc_fence_after_sync();
          const uint32_t a_lo = adesc0_lo + s * (kStageBytes >> 4);
          const uint32_t b_lo = bdesc0_lo + s * (kStageBytes >> 4);
          const uint32_t more = kb > 0 ? 1u : 0u;
          if (!elect_one()) continue;
          if constexpr (kSplit) {
#pragma unroll
            for (int kk = 0; kk < kF32TileK / kF32UmmaK; ++kk)  // lo . hi
              umma_tf32_pair(tmem_d + BN, make_desc64(a_lo + kLo + kk * kAStep, a_hi),
                             make_desc64(b_lo + kk * kBStep, b_hi), idesc, kk > 0 ? 1u : more);
#pragma unroll
            for (int kk = 0; kk < kF32TileK / kF32UmmaK; ++kk)  // hi . lo
              umma_tf32_pair(tmem_d + BN, make_desc64(a_lo + kk * kAStep, a_hi),
                             make_desc64(b_lo + kLo + kk * kBStep, b_hi), idesc, 1u);
          }
          const int live = kTgmm ? t.rows - kb * kF32TileK : kF32TileK;
          if (!kSplit && kTgmm && live <= kF32TileK - kF32UmmaK) {  // whole 8-deep MMAs past the group's end
            const int n_mma = (live + kF32UmmaK - 1) / kF32UmmaK;
            for (int kk = 0; kk < n_mma; ++kk)
              umma_tf32_pair(tmem_d, make_desc64(a_lo + kk * kAStep, a_hi),
                             make_desc64(b_lo + kk * kBStep, b_hi), idesc, kk > 0 ? 1u : more);
          } else {
#pragma unroll
            for (int kk = 0; kk < kF32TileK / kF32UmmaK; ++kk)
              umma_tf32_pair(tmem_d, make_desc64(a_lo + kk * kAStep, a_hi),
                             make_desc64(b_lo + kk * kBStep, b_hi), idesc, kk > 0 ? 1u : more);
          }
          umma_commit_pair(smem_u32(&bar_empty[s]), 0x3);
        }
        if (!ok) break;
        const uint32_t bar = smem_u32(&bar_acc_full[acc]);
        if (elect_one()) {
          if (kb_count > 0) {
            umma_commit_pair(bar, 0x3);
          } else {  // empty group: nothing to wait for
            mbar_arrive(bar);
            mbar_arrive_cluster(bar, 1);
          }
        }
      }
    }
  } else if (warp >= kF32ConvWarp0) {
    if constexpr (kSplit) {
      // ------------------------------------------------------------ converters
      const int ct = threadIdx.x - 32 * kF32ConvWarp0;
      uint32_t it = 0;
      bool ok = true;
      for (int tile = tile_start; tile < num_tiles && ok; tile += tile_step) {
        const TileCoord t = decode(tile);
        const int kb_count = blocks_of(t);
        for (int kb = 0; kb < kb_count; ++kb, ++it) {
          const uint32_t s = it % kStages;
          const uint32_t ph = (it / kStages) & 1u;
          if (!mbar_wait_warp(smem_u32(&bar_full[s]), ph, abort_ptr)) {
            ok = false;
            break;
          }
          // tgmm boxes are [32 rows][128 B]: rows from `live` on belong to the next group.
          const int live = kTgmm ? t.rows - kb * kF32TileK : kF32TileK;
          const uint32_t base = stage_base + s * kStageBytes + ct * 16;
          constexpr int kPer = kF32PairRawBytes / 16 / (32 * kF32ConvWarps);
          constexpr int kBatch = 4;  // loads in flight per thread
#pragma unroll
          for (int i0 = 0; i0 < kPer; i0 += kBatch) {
            uint32_t v[kBatch][4];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
              const uint32_t a = base + (i0 + i) * (32 * kF32ConvWarps * 16);
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(v[i][0]), "=r"(v[i][1]), "=r"(v[i][2]), "=r"(v[i][3])
                           : "r"(a)
                           : "memory");
            }
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
              const uint32_t a = base + (i0 + i) * (32 * kF32ConvWarps * 16);
              // 256 threads cover one 4 KB box per step, so a thread's row is the same in every box
              if (kTgmm && (ct >> 3) >= live) v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0u;
              uint32_t hi[4], lo[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) split_tf32(v[i][j], hi[j], lo[j]);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(hi[0]), "r"(hi[1]),
                           "r"(hi[2]), "r"(hi[3])
                           : "memory");
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a + kF32PairRawBytes), "r"(lo[0]),
                           "r"(lo[1]), "r"(lo[2]), "r"(lo[3])
                           : "memory");
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (leader) {
              mbar_arrive(smem_u32(&bar_conv[s]));
            } else {
              mbar_arrive_cluster(smem_u32(&bar_conv[s]), 0);
            }
          }
        }
      }
    } else if constexpr (kTgmm) {
      // ------------------------------------------------------------ tail fixer
      uint32_t it = 0;
      uint32_t events = 0;
      uint32_t own_parity = 0;  // peer, bit s: parity of the next landing on its own barrier of slot s
      bool ok = true;
      for (int tile = tile_start; tile < num_tiles && ok; tile += tile_step) {
        const TileCoord t = decode(tile);
        const int kb_count = blocks_of(t);
        it += kb_count;
        if (kb_count == 0 || !tail_needs_clearing_f32(t.rows)) continue;
        const uint32_t s = (it - 1) % kStages;
        if (!mbar_wait_warp<true>(smem_u32(&bar_tail_go), events & 1u, abort_ptr)) {
          ok = false;
          break;
        }
        if (!leader) {  // the peer's bytes of such a stage are counted on its own barrier
          const uint32_t par = (own_parity >> s) & 1u;
          own_parity ^= 1u << s;
          if (!mbar_wait_warp(smem_u32(&bar_full[s]), par, abort_ptr)) {
            ok = false;
            break;
          }
        }
        ++events;
        clear_tail_rows_f32<kF32PairRawBytes / kF32BoxBytes>(stage_base + s * kStageBytes,
                                                             t.rows - (kb_count - 1) * kF32TileK, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(smem_u32(&bar_tail_done), 0);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5)
    const int quarter = warp & 3;
    const int r_in_tile = quarter * 32 + lane;
    const uint32_t staging = stage_base + kStages * kStageBytes + (warp - 2) * 2 * kOutBoxBytes;
    uint32_t local_tile = 0;
    uint32_t boxes_stored = 0;
    bool ok = true;
    float* out32 = reinterpret_cast<float*>(p.out);
    for (int tile = tile_start; tile < num_tiles && ok; tile += tile_step, ++local_tile) {
      const TileCoord t = decode(tile);
      const int n0 = t.n0;
      const uint32_t acc = kSplit ? 0u : (local_tile & 1u);
      const uint32_t acc_ph = kSplit ? (local_tile & 1u) : ((local_tile >> 1) & 1u);
      if (!mbar_wait_warp<true>(smem_u32(&bar_acc_full[acc]), acc_ph, abort_ptr)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();

      bool row_ok, warp_has_rows, slab_by_tma, zero_only = false;
      size_t row_off;
      int out_row0;
      if (kTgmm) {
        const int kr = t.k0 + r_in_tile;
        out_row0 = t.k0 + quarter * 32;
        row_ok = kr < p.k;
        warp_has_rows = out_row0 < p.k;
        slab_by_tma = true;  // rows >= k are outside the map and dropped by the store
        row_off = (static_cast<size_t>(t.group) * p.k + kr) * static_cast<size_t>(p.n);
        zero_only = t.rows <= 0;
      } else {
        out_row0 = t.row0 + quarter * 32;
        row_ok = r_in_tile < t.rows;
        warp_has_rows = quarter * 32 < t.rows;
        slab_by_tma = quarter * 32 + 32 <= t.rows;  // else the box would overwrite the next group
        row_off = static_cast<size_t>(t.row0 + r_in_tile) * static_cast<size_t>(p.n);
      }

      const int n_chunks =
          warp_has_rows ? imin(BN / kChunkCols, (p.n - n0 + kChunkCols - 1) / kChunkCols) : 0;
      const uint32_t acc_empty_bar = smem_u32(&bar_acc_empty[acc]);
#pragma unroll 1
      for (int c = 0; c < n_chunks; ++c) {
        const int col = n0 + c * kChunkCols;
        uint32_t v[32];
        if (!zero_only) {
          const uint32_t taddr =
              tmem_base + acc * BN + c * kChunkCols + (static_cast<uint32_t>(quarter * 32) << 16);
          tmem_ld_32x32(taddr, v);
          if constexpr (kSplit) {
            uint32_t small[32];
            tmem_ld_32x32(taddr + BN, small);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j)
              v[j] = __float_as_uint(__uint_as_float(small[j]) + __uint_as_float(v[j]));
          } else {
            tmem_ld_wait();
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0u;
        }
        if (c == n_chunks - 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(acc_empty_bar, 0);
        }
        if (slab_by_tma) {
          const uint32_t buf = staging + (boxes_stored & 1u) * kOutBoxBytes;
          if (lane == 0) bulk_wait_group_read<1>();
          __syncwarp();
          const uint32_t row_addr = buf + lane * 128;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint32_t a = row_addr + (((q ^ (lane & 7)) & 7) << 4);  // 128-byte swizzle
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v[q * 4 + 0]),
                         "r"(v[q * 4 + 1]), "r"(v[q * 4 + 2]), "r"(v[q * 4 + 3])
                         : "memory");
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (kTgmm) {
              tma_store_3d(&tmap_out, buf, col, out_row0, t.group);
            } else {
              tma_store_2d(&tmap_out, buf, col, out_row0);
            }
            bulk_commit_group();
          }
          ++boxes_stored;
        } else if (row_ok) {
          float* dst = out32 + row_off + col;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            if (col + q * 4 < p.n) {  // n is a multiple of 4: a chunk is all in or all out
              *reinterpret_cast<uint4*>(dst + q * 4) =
                  make_uint4(v[q * 4 + 0], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
            }
          }
        }
      }
      if (n_chunks == 0) {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc_empty_bar, 0);
      }
    }
    if (lane == 0) bulk_wait_group<0>();
    __syncwarp();

    if (!kTgmm && p.zero_tail) {
      const int first = first_dead_row(p, &group_table);
      const size_t chunks_per_row = static_cast<size_t>(p.n) / 4;
      const size_t total = static_cast<size_t>(p.m - first) * chunks_per_row;
      const size_t tid = static_cast<size_t>(blockIdx.x) * 128 + (threadIdx.x - 64);
      const size_t stride = static_cast<size_t>(gridDim.x) * 128;
      uint4* dst = reinterpret_cast<uint4*>(out32 + static_cast<size_t>(first) * p.n);
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
    tmem_dealloc<2>(tmem_base, 2 * BN);
  }
}

}  // namespace rd
