// C ABI of the ragged-dot library (declared in include/ragged_dot_b200.h): argument checks,
// TMA descriptor encoding, tile selection and kernel launches.  No torch / XLA types here;
// the XLA-FFI and Python layers sit on top of these entry points.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include <atomic>
#include <mutex>
#include <numeric>

#include "../../include/ragged_dot_b200.h"
#include "rd_gemm.cuh"
#include "rd_dispatch.cuh"
#include "rd_gemm2.cuh"
#include "rd_gemm_f32.cuh"
#include "rd_gemm_f32_pair.cuh"
#include "rd_gemm_perm.cuh"
#include "rd_gemm_splitk.cuh"
#include "rd_gemm_swap.cuh"
#include "rd_metadata.cuh"
#include "rd_rows.cuh"
#include "rd_tgmm.cuh"

namespace {

using rd::GemmArgs;
using rd::WorkspaceLayout;

// ------------------------------------------------------------------ driver entry point
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
  });
  return fn;
}

// The tensor-map encoder needs a context on the calling thread.  A runtime launch binds the device's
// primary context, but threads such as torch's autograd workers arrive here without one.
int ensure_context() {
  typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
  static CtxGetCurrentFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<CtxGetCurrentFn>(sym);
  });
  CUcontext ctx = nullptr;
  if (fn != nullptr && fn(&ctx) == CUDA_SUCCESS && ctx != nullptr) return RD_OK;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return RD_ERR_LAUNCH;
  }
  return RD_OK;
}

// rank-2 or rank-3 tiled map over a dense row-major 16-bit or 32-bit float tensor, 128-byte swizzle (or none),
// zero fill outside the bounds.  dims / box are innermost first.
int encode_map(CUtensorMap* map, const void* base, int dtype, int rank, const uint64_t* dims,
               const uint32_t* box, bool atom32 = false, bool swizzled = true) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return RD_ERR_DRIVER;
  cuuint64_t gdims[3];
  cuuint64_t gstrides[2];
  cuuint32_t gbox[3];
  cuuint32_t estr[3] = {1, 1, 1};
  uint64_t stride = dtype == RD_DTYPE_F32 ? 4 : 2;
  for (int i = 0; i < rank; ++i) {
    gdims[i] = dims[i];
    gbox[i] = box[i];
    stride *= dims[i];
    if (i + 1 < rank) gstrides[i] = stride;
  }
  const CUtensorMapDataType dt = dtype == RD_DTYPE_BF16  ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                 : dtype == RD_DTYPE_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                                         : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUresult r = fn(map, dt, static_cast<cuuint32_t>(rank), const_cast<void*>(base), gdims, gstrides,
                  gbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  !swizzled ? CU_TENSOR_MAP_SWIZZLE_NONE
                  : atom32  ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B
                            : CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    fprintf(stderr,
            "ragged_dot_b200: cuTensorMapEncodeTiled failed (CUresult %d): base=%p rank=%d "
            "dims={%llu,%llu,%llu} box={%u,%u,%u}\n",
            static_cast<int>(r), base, rank, (unsigned long long)gdims[0],
            (unsigned long long)gdims[1], (unsigned long long)(rank > 2 ? gdims[2] : 0), gbox[0],
            gbox[1], rank > 2 ? gbox[2] : 0u);
    return RD_ERR_TENSOR_MAP;
  }
  return RD_OK;
}

// "Column-blocked" view of a dense row-major [rows, cols] tensor, cols a multiple of c = 64 (16-bit) or
// 32 (float32, in the 32-byte-atom swizzle): (c columns, rows, cols / c blocks).  A box of (c,
// box_rows, box_blocks) lands in shared memory as box_blocks slabs of [box_rows][128 B], block after
// block -- what box_blocks separate 2-D boxes of c columns would write -- in ONE TMA instruction.
// `mats` > 0 adds a fourth dimension: that many such tensors one after the other.
int encode_blocked_map(CUtensorMap* map, const void* base, int dtype, int cols, int rows, int box_rows,
                       int box_blocks, int mats = 0) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return RD_ERR_DRIVER;
  const bool f32 = dtype == RD_DTYPE_F32;
  const int c = f32 ? 32 : 64;
  const cuuint64_t row_bytes = static_cast<cuuint64_t>(cols) * (f32 ? 4 : 2);
  cuuint64_t gdims[4] = {static_cast<cuuint64_t>(c), static_cast<cuuint64_t>(rows),
                         static_cast<cuuint64_t>(cols / c), static_cast<cuuint64_t>(mats)};
  cuuint64_t gstrides[3] = {row_bytes, 128, row_bytes * static_cast<cuuint64_t>(rows)};
  cuuint32_t gbox[4] = {static_cast<cuuint32_t>(c), static_cast<cuuint32_t>(box_rows),
                        static_cast<cuuint32_t>(box_blocks), 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUtensorMapDataType dt = dtype == RD_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                 : f32                  ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                                        : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUresult r = fn(map, dt, mats > 0 ? 4 : 3, const_cast<void*>(base), gdims, gstrides, gbox, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE,
                  f32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    fprintf(stderr, "ragged_dot_b200: cuTensorMapEncodeTiled failed (CUresult %d): blocked map base=%p "
            "rows=%d cols=%d box=(%d,%d,%d)\n", static_cast<int>(r), base, rows, cols, c, box_rows, box_blocks);
    return RD_ERR_TENSOR_MAP;
  }
  return RD_OK;
}

// ------------------------------------------------------------------ device properties
int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

bool aligned16(const void* p) { return p != nullptr && (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int max_row_tiles(int m, int g) { return (m + rd::kTileM - 1) / rd::kTileM + g; }

struct Workspace {
  WorkspaceLayout layout;
  int32_t* base;
  int32_t* status() const { return base + layout.off_status(); }
  int32_t* totals() const { return base + layout.off_totals(); }
  int32_t* group_offsets() const { return base + layout.off_group_offsets(); }
  int32_t* tile_prefix() const { return base + layout.off_tile_prefix(); }
  int32_t* tile2group() const { return base + layout.off_tile2group(); }
  int32_t* tile2idx() const { return base + layout.off_tile2idx(); }
  rd::TileRecord* tile_rec() const {
    return reinterpret_cast<rd::TileRecord*>(base + layout.off_tile_rec());
  }
};

int bind_workspace(void* ws, size_t ws_bytes, int m, int g, Workspace* out) {
  if (!aligned16(ws)) return RD_ERR_BAD_POINTER;
  out->layout.g = g;
  out->layout.max_tiles = max_row_tiles(m, g);
  if (ws_bytes < static_cast<size_t>(out->layout.total_words()) * sizeof(int32_t))
    return RD_ERR_WORKSPACE;
  out->base = static_cast<int32_t*>(ws);
  return RD_OK;
}

void launch_internal_metadata(const int32_t* group_sizes, const int32_t* group_to_weight, int g,
                              int m, int tile_m, const Workspace& w, cudaStream_t stream,
                              bool by_weight = false) {
  if (by_weight && group_to_weight != nullptr && m > 0) {
    // the two reference-shaped arrays are not needed by the kernels: their space (U >= g + 1
    // words each) serves as the scratch of the visiting order
    rd::group_metadata_kernel<<<1, rd::kMetaThreads, 0, stream>>>(
        group_sizes, g, m, tile_m, w.layout.max_tiles, w.group_offsets(), nullptr, nullptr, w.totals(),
        w.tile_prefix(), w.totals() + 1, w.status(), w.tile_rec(), group_to_weight, w.tile2group(),
        w.tile2idx());
    return;
  }
  rd::group_metadata_kernel<<<1, rd::kMetaThreads, 0, stream>>>(
      group_sizes, g, m, tile_m, w.layout.max_tiles, w.group_offsets(), w.tile2group(),
      w.tile2idx(), w.totals(), w.tile_prefix(), w.totals() + 1, w.status(), w.tile_rec(),
      group_to_weight);
}

// Do the CTAs make their own group table (rd_gemm.cuh), so that no metadata launch is needed?  Not for
// more groups or row tiles than the table holds.
bool inline_groups(int m, int g) {
  return g <= rd::kMaxInlineGroups && max_row_tiles(m, g) <= rd::kMaxInlineRowTiles;
}

// ------------------------------------------------------------------ tile selection
// The committed replacement for the reference's run-time tune-jax search.  Measured on B200:
// the 256-wide tile wins at every benchmark shape, compute-bound or bandwidth-bound (decode m=256: 93 % of copy bandwidth at 256, 67 % at 128, 39 % at 64), so
// narrower tiles are only used when n itself is narrow.
int choose_tile_n(long long /*row_tiles*/, int n, int /*sms*/) {
  if (n <= 64) return 64;
  if (n <= 128) return 128;
  return 256;
}

// One launch on clusters of `cluster` CTAs (1: none).  `early`: the kernel waits for its predecessor itself
// (start_inline_groups, repitch_rows_kernel) and may be started before that has finished.
template <typename... Params, typename... Args>
int launch_kernel(void (*kernel)(Params...), int ctas, int threads, size_t smem_bytes, int cluster, bool early,
                  cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(ctas, 1, 1);
  lc.blockDim = dim3(threads, 1, 1);
  lc.dynamicSmemBytes = smem_bytes;
  lc.stream = stream;
  cudaLaunchAttribute attr[2];
  lc.attrs = attr;
  if (cluster > 1) {
    cudaLaunchAttribute& a = attr[lc.numAttrs++];
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = cluster;
    a.val.clusterDim.y = 1;
    a.val.clusterDim.z = 1;
  }
  if (early) {
    cudaLaunchAttribute& a = attr[lc.numAttrs++];
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
  }
  if (cudaLaunchKernelEx(&lc, kernel, Params(args)...) != cudaSuccess) {
    (void)cudaGetLastError();
    return RD_ERR_LAUNCH;
  }
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

// Start a kernel while the one before it still runs?  Only kernels that wait for it themselves, and
// where no CTA has more than one tile: there the launch is a good part of the time (4 rows through
// 4 of 64 experts, k 4096, n 1536: 17.9 -> 15.7 us a call back to back).  With more tiles it costs: CTAs
// then land on SMs in the order in which the kernel before leaves them, and neighbours in the tile
// order, which share operand panels, no longer lie side by side (Mixtral-shaped training step 2.57 ->
// 2.70 ms, 64 groups 1.41 -> 1.54 ms, 256 groups 5.1 -> 5.5 ms).
// Groups of 64 rows and less read (or write) weights that no neighbour shares, so there it gains its 2 us too, up to 256
// million weights, 80 us and more (counted for the groups that can have rows, in elements of any type, e4m3 in pairs): 256
// rows, k 4096, n 1536, 64 groups of e4m3 67.7 -> 65.4; 4000, 1024, 1024, 64 30.9 -> 29.5, tgmm 37.0 -> 34.9; 300, 1000,
// 2000, 100 tgmm 72.5 -> 69.1; float32 2000, 1024, 2048, 64 (537 MB) 99 -> 98, tgmm 114 -> 107; tgmm of 64 rows in 256 groups,
// k 1536, n 1536, float32 (2.4 GB) 422 -> 410.  Above, nothing or less: the first in bf16 119.0 -> 119.3; 512, 7168, 2048, 256
// 755 -> 770.  Weights with rows along the contraction lose sooner, where it is long, so of these 75 million: bf16 3383, 8936,
// 384, 64 109 -> 115; 2000, 3000, 1024, 64 (393 MB) 82 -> 86.  (Short contractions would gain: float32 2000, 1024, 1024, 64 54 ->
// 52.)  On pairs, which take such weights for three float32 products only, it does no harm: 2000, 768, 1024, 64 121 -> 119,
// 1536, 2048 429 -> 427.
// tgmm on 256 columns, whose tiles are a few stages each: up to two tiles per CTA (`rounds`).  82 sizes of one to two rounds: 1.25
// times as fast below 256 rows per group, 1.15 below 768, 1.05 above.
bool launch_early(const GemmArgs& args, int ctas_per_tile = 1, bool wide_k_major = false, int rounds = 1) {
  if (!args.inline_groups) return false;
  const long long row_tiles = args.k_tiles > 0 ? static_cast<long long>(args.g) * args.k_tiles
                                               : static_cast<long long>(args.m < args.g ? args.m : args.g) + args.m / rd::kTileM;
  if (row_tiles * args.n_tiles * ctas_per_tile <= static_cast<long long>(rounds) * sm_count()) return true;
  const double weights = 1.0 * (args.m < args.g ? args.m : args.g) * args.k * args.n;
  return args.m <= 64LL * args.g && weights <= (wide_k_major ? 75e6 : 256e6);
}

// How many clusters of two CTAs can be resident at once (0: the query failed).
template <typename Kernel>
int resident_pairs(Kernel kernel, int threads, size_t smem_bytes) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(2, 1, 1);
  lc.blockDim = dim3(threads, 1, 1);
  lc.dynamicSmemBytes = smem_bytes;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &lc) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return clusters;
}

// The same, asked once for a kernel and device (the query takes longer than the launch).  A template argument, so that
// every kernel has its own answers.
template <auto kKernel>
int resident_pairs_once(int threads, size_t smem_bytes) {
  static std::atomic<int> known[64];  // pairs + 1; 0 = not asked yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return resident_pairs(kKernel, threads, smem_bytes);
  int n = known[dev].load(std::memory_order_relaxed) - 1;
  if (n <= 0) {
    n = resident_pairs(kKernel, threads, smem_bytes);
    known[dev].store(n + 1, std::memory_order_relaxed);
  }
  return n;
}

// A persistent grid of pairs must be fully co-resident.
template <auto kKernel, int kEarlyRounds = 1, typename... Maps>
int launch_pairs(int threads, int smem_bytes, const GemmArgs& args, int ctas, cudaStream_t stream,
                 const Maps&... maps) {
  if (cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess)
    return RD_ERR_LAUNCH;
  const int clusters = resident_pairs_once<kKernel>(threads, smem_bytes);
  if (clusters <= 0) return RD_ERR_LAUNCH;
  int pairs = ctas / 2;
  if (pairs > clusters) pairs = clusters;
  if (pairs < 1) pairs = 1;
  return launch_kernel(kKernel, 2 * pairs, threads, smem_bytes, 2, launch_early(args, 2, false, kEarlyRounds), stream,
                       maps..., args);
}

template <int BN, bool kBKMajor, bool kTgmm, int kCtas, bool kSeg = false, bool kFp8 = false, bool kOneThread = false>
int launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tout,
                const GemmArgs& args, int ctas, cudaStream_t stream) {
  constexpr int kStageBytes = rd::stage_bytes<BN, kCtas>();
  constexpr int kStages = (196608 / kStageBytes) > 8 ? 8 : (196608 / kStageBytes);
  constexpr int kSmem = kStages * kStageBytes + rd::kOutStagingBytes + 1024;
  constexpr auto kernel = rd::ragged_gemm_kernel<BN, kBKMajor, kStages, kTgmm, kCtas, kSeg, kFp8, false, kOneThread>;
  if constexpr (kCtas == 2) return launch_pairs<kernel>(rd::kGemmFixerThreads, kSmem, args, ctas, stream, ta, tb, tout);
  // The attribute is per device; setting it again is cheap, so do it on every call rather
  // than track which devices have seen it.
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) !=
      cudaSuccess)
    return RD_ERR_LAUNCH;
  return launch_kernel(kernel, ctas, rd::kGemmFixerThreads, kSmem, 1,
                       launch_early(args, 1, kBKMajor && !kFp8, kTgmm && BN == 256 ? 2 : 1), stream, ta, tb, tout, args);
}

// Rows that are not multiples of 16 bytes (see kUnaligned in rd_gemm.cuh).
template <int BN, bool kBKMajor, bool kTgmm>
int launch_gemm_unaligned(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& args, int ctas,
                          cudaStream_t stream) {
  constexpr int kStageBytes = rd::stage_bytes<BN, 1>();
  constexpr int kStages = (196608 / kStageBytes) > 8 ? 8 : (196608 / kStageBytes);
  constexpr int kSmem = kStages * kStageBytes + rd::kOutStagingBytes + 1024;
  auto kernel = rd::ragged_gemm_kernel<BN, kBKMajor, kStages, kTgmm, 1, false, false, true>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess)
    return RD_ERR_LAUNCH;
  return launch_kernel(kernel, ctas, rd::kGemmFixerThreads, kSmem, 1, launch_early(args, 1, kBKMajor), stream, ta, tb, ta, args);
}

template <int BN, bool kBKMajor, bool kTgmm>
int launch_gemm_f32(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tout,
                    const GemmArgs& args, int ctas, cudaStream_t stream) {
  constexpr int kStageBytes = rd::f32_stage_bytes<BN>();
  constexpr int kStages = (196608 / kStageBytes) > 8 ? 8 : (196608 / kStageBytes);
  constexpr int kSmem = kStages * kStageBytes + rd::kOutStagingBytes + 1024;
  auto kernel = rd::ragged_gemm_f32_kernel<BN, kBKMajor, kStages, kTgmm>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) !=
      cudaSuccess)
    return RD_ERR_LAUNCH;
  return launch_kernel(kernel, ctas, rd::kGemmThreads, kSmem, 1, launch_early(args, 1, kBKMajor), stream, ta, tb, tout, args);
}

template <int BN, bool kBKMajor, bool kTgmm>
int launch_gemm_perm(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tout,
                     const GemmArgs& args, const rd::PermArgs& perm, int ctas, cudaStream_t stream) {
  constexpr int kStageBytes = rd::stage_bytes<BN, 1>();
  constexpr int kStages = (196608 / kStageBytes) > 8 ? 8 : (196608 / kStageBytes);
  constexpr int kSmem = kStages * kStageBytes + rd::kOutStagingBytes + 1024;
  auto kernel = rd::ragged_gemm_perm_kernel<BN, kBKMajor, kStages, kTgmm>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) !=
      cudaSuccess)
    return RD_ERR_LAUNCH;
  kernel<<<ctas, rd::kPermThreads, kSmem, stream>>>(ta, tb, tout, args, perm);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

// Tile-load map over a [rows, cols] 16-bit tensor with boxes of [box_rows][64 columns].  The
// permuted kernels use it for an operand without a row index; with one they read the tensor
// through its base pointer and the map is only prefetched.
int encode_rows_map(CUtensorMap* map, const void* base, int dtype, int cols, int rows, int box_rows) {
  const uint64_t dims[2] = {static_cast<uint64_t>(cols), static_cast<uint64_t>(rows)};
  const uint32_t box[2] = {64, static_cast<uint32_t>(box_rows)};
  return encode_map(map, base, dtype, 2, dims, box);
}

template <bool kBKMajor, bool kTgmm, bool kVariant = false>
int launch_gemm2(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tout,
                 const GemmArgs& args, int ctas, cudaStream_t stream) {
  if constexpr (!kTgmm && !kVariant) {
    // ready flags / sender CTAs live in a separate instantiation (see rd_gemm2.cuh)
    if (args.ready_flags != nullptr || args.send.world > 0)
      return launch_gemm2<kBKMajor, false, true>(ta, tb, tout, args, ctas, stream);
  }
  auto kernel = rd::ragged_gemm2_kernel<kBKMajor, kTgmm, kVariant>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, rd::kG2SmemBytes) !=
      cudaSuccess)
    return RD_ERR_LAUNCH;
  return launch_kernel(kernel, ctas, rd::kG2Threads, rd::kG2SmemBytes, 1, launch_early(args, 1, kBKMajor), stream, ta, tb, tout,
                       args);
}

// e4m3 on 256-row tiles (rd_gemm2.cuh, kFp8).
int launch_gemm2_fp8(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tout, const GemmArgs& args,
                     int ctas, cudaStream_t stream) {
  auto kernel = rd::ragged_gemm2_kernel<true, false, false, true>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, rd::kG2SmemBytes) !=
      cudaSuccess)
    return RD_ERR_LAUNCH;
  return launch_kernel(kernel, ctas, rd::kG2Threads, rd::kG2SmemBytes, 1, launch_early(args), stream, ta, tb, tout,
                       args);
}

// float32 on CTA pairs (rd_gemm_f32_pair.cuh).
template <bool kBKMajor, bool kTgmm, bool kSplit>
int launch_gemm_f32_pair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tout, const GemmArgs& args,
                         int ctas, cudaStream_t stream) {
  return launch_pairs<rd::ragged_gemm_f32_pair_kernel<kBKMajor, kTgmm, kSplit>>(rd::f32_pair_threads<kSplit>(),
                      rd::f32_pair_smem_bytes<kSplit>(), args, ctas, stream, ta, tb, tout);
}

// Cluster size for a gmm whose tiles are too few for the SMs (rd_gemm_splitk.cuh), 1 = no split.
// `tiles` bounds the live tiles, `rows` is what a large tile may hold.  All clusters must be resident at
// once and every CTA gets at least four 64-deep blocks.  Split where the contraction of a tile on one CTA
// (0.3 us per block) takes longer than 3 us and 15 us more for 128 rows: adding the partial sums up costs
// about 1 us and 10 us more for 128 rows, the rest is a margin (1024 rows in 2 groups, k 1024, n 1024,
// 16 blocks: 17 us whole, 25 us split; 300 rows in 4 groups, k 8192, n 256, 128 blocks: 55 and 27).
template <bool kBKMajor, bool kFp8>
int choose_split(long long tiles, int rows, int k_blocks) {
  const int sms = sm_count();
  if (tiles <= 0 || tiles * 2 > sms || k_blocks < 8) return 1;
  if (0.3 * k_blocks < 3.0 + 15.0 * rows / rd::kTileM) return 1;
  static std::mutex mu;
  static int fit[64][rd::kMaxSplit + 1];  // clusters of each size that fit, + 1; 0 = not asked yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
  auto kernel = rd::ragged_gemm_splitk_kernel<kBKMajor, kFp8>;
  std::lock_guard<std::mutex> lock(mu);
  for (int s = rd::kMaxSplit; s >= 2; --s) {
    if (tiles * s > sms || k_blocks < 4 * s) continue;
    if (fit[dev][s] == 0) {
      cudaLaunchConfig_t lc = {};
      lc.blockDim = dim3(rd::kGemmThreads, 1, 1);
      lc.gridDim = dim3(s, 1, 1);
      lc.dynamicSmemBytes = rd::kSplitSmemBytes;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = s;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      lc.attrs = attr;
      lc.numAttrs = 1;
      int clusters = 0;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, rd::kSplitSmemBytes) !=
              cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&clusters, kernel, &lc) != cudaSuccess) {
        (void)cudaGetLastError();
        clusters = 0;
      }
      fit[dev][s] = clusters + 1;
    }
    if (tiles <= fit[dev][s] - 1) return s;
  }
  return 1;
}

template <bool kBKMajor, bool kFp8>
int launch_gemm_splitk(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& args, int split, int tiles,
                       cudaStream_t stream) {
  auto kernel = rd::ragged_gemm_splitk_kernel<kBKMajor, kFp8>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, rd::kSplitSmemBytes) !=
      cudaSuccess)
    return RD_ERR_LAUNCH;
  return launch_kernel(kernel, split * tiles, rd::kGemmThreads, rd::kSplitSmemBytes, split, true, stream, ta, tb, args,
                       split);
}

// Fewer rounds than choose_swap asks for: the clocks of both kernels, from their rounds of tiles.  A pair takes 4 clocks per
// row and block of the contraction and 5000 to drain a tile, a last half round costs 0.55 of one (SwapWork), one CTA 560
// per block of a 128 x 256 tile; a group's last tile is half full on average.  A last tile of a row that is a half tile counts
// whole: pairs do not share such tiles evenly (counted half, 704 columns were up to 29 % slower).  The tiles of a single
// group are counted: 590 rows, k 10912, n 12640, float32, are 75 tiles for 74 pairs (293 -> 372 us where an average of 70
// had said one round).  Under half a round, and for groups shorter than `least`, it is wrong too often.
// Timed on both sides on 477 sizes that this takes and the rules below do not (1 to 256 groups, equal to heavy-tailed): 16 bits
// 1.17 times as fast on average, slower by more than 5 % in 7 of 191; e4m3 1.17, 22 of 189; float32 1.14, 2 of 97.  Most of the slower
// ones are heavy-tailed, which the host cannot know: worst, e4m3 4842, 3840, 584, 28 groups 28 -> 43, 16 bits 4567, 3216, 3192, 7
// 95 -> 114.  e4m3 within a twentieth of one whole round is as often slower as faster (11257, 5632, 432, 62 55 -> 74; 2595, 5200,
// 2296, 9 67 -> 46).
bool swap_takes_less(long long m, int k_blocks, int n, int g, int least, double margin) {
  if (m / g < least) return false;
  const long long sms = sm_count(), pairs = sms / 2;
  const long long cols = (n + rd::kSwapCols - 1) / rd::kSwapCols, cols128 = (n + 255) / 256;
  double rounds, height, rounds128;
  if (g == 1) {
    const long long per = (m + rd::kSwapRows - 1) / rd::kSwapRows, tiles = per * cols, left = tiles % pairs;
    if (2 * tiles < pairs) return false;
    rounds = static_cast<double>(tiles / pairs) + (left == 0 ? 0.0 : 2 * left <= pairs ? 0.55 : 1.0);
    height = static_cast<double>((m + 16 * per - 1) / (16 * per) * 16);
    rounds128 = static_cast<double>(((m + rd::kTileM - 1) / rd::kTileM * cols128 + sms - 1) / sms);
    margin = 1.0;
  } else {
    const double rows = static_cast<double>(m) / g, per = rows > 128.0 ? rows / rd::kSwapRows + 0.5 : 1.0;
    const double exact = g * per * cols / pairs;
    if (exact < 0.5) return false;
    if (exact < 1.0) margin = 1.25;
    const double whole = static_cast<double>(static_cast<long long>(exact)), left = exact - whole;
    rounds = whole + (left < 0.03 ? 0.0 : left <= 0.5 ? 0.55 : 1.0);
    height = rows / per + 8.0;
    const double per128 = rows > 64.0 ? rows / rd::kTileM + 0.5 : 1.0;
    rounds128 = static_cast<double>(static_cast<long long>(g * per128 * cols128 / sms + 0.97));
  }
  if (height > rd::kSwapRows) height = rd::kSwapRows;
  return rounds * (4.0 * height * k_blocks + 5000.0) * margin < (rounds128 > 1.0 ? rounds128 : 1.0) * 560.0 * k_blocks;
}

// Should a gmm put its rows on the N side of the MMAs (rd_gemm_swap.cuh)?  Where swap_takes_less says so; and when groups are
// long, there are at least three rounds of tiles for the pairs and the last 512-column tile is nearly full.
// Microseconds in a row, one-CTA tiles (better of the two heights) against swapped: m 8192, k 4096, n 14336, 8
// groups 726 -> 659, trans_rhs with k 14336, n 4096 723 -> 703; 13304, 2824, 11264, 16 685 -> 627; 28320, 5656, 1536, 32
// 430 -> 410; 64 groups of 512, k 4096, n 1536, fp16 339 -> 333; e4m3 8192, 4096, 14336, 8 397 -> 370.  Not there: 4096, 4096, 4096, 8 (1.7
// rounds) 107 -> 109 with equal groups, 120 -> 126 with unequal ones; 8192, 4096, 2304, 8 (last tile half full, equal groups) 107 -> 134.
// A short contraction (fewer than nine 64-deep blocks) leaves the drain of both accumulators exposed once per
// tile: 4928, 264, 7232, 4 29 -> 33, 22000, 512, 4032, 12 90 -> 86 with equal groups, 95 -> 97 with unequal ones; 16 bits win again
// from twenty rounds on (17184, 456, 13568, 32 272 -> 247), e4m3 does not (25960, 448, 4928, 24 96 -> 97, unequal 105 -> 111).
// e4m3 (128-row tiles otherwise) with few rounds: they are compared, a swapped tile taking 1.7 times as long
// as a 128-row one.  (That was fitted to a slower swapped kernel: 8192, 14336, 4096, 16, five rounds against eight, is refused and would
// take 357 instead of 392, with unequal groups 422 instead of 437.)
bool choose_swap(long long m, int k_blocks, int n, int g, bool trans_rhs, bool fp8) {
  if (g <= 0 || (!trans_rhs && n % 64 != 0)) return false;
  if (swap_takes_less(m, k_blocks, n, g, fp8 ? 128 : 384, fp8 ? 1.2 : 1.0)) return true;
  if (m / g < 512) return false;
  const long long pairs = sm_count() / 2;
  const long long col_tiles = (static_cast<long long>(n) + rd::kSwapCols - 1) / rd::kSwapCols;
  if ((col_tiles * rd::kSwapCols - n) * 16 > n || m / rd::kSwapRows * col_tiles < 3 * pairs) return false;
  const long long tiles = (m / rd::kSwapRows + g / 2) * col_tiles;  // half a tile more per group
  if (k_blocks < 9 && (fp8 || tiles < 20 * pairs)) return false;
  if (!fp8 || tiles >= 6 * pairs) return true;
  const long long tiles128 = ((m + 127) / 128 + g / 2) * ((static_cast<long long>(n) + 255) / 256);
  return 1.7 * static_cast<double>((tiles + pairs - 1) / pairs) <
         static_cast<double>((tiles128 + 2 * pairs - 1) / (2 * pairs));
}

// The same for float32 in one pass (128-row tiles on one CTA otherwise), k_blocks of 32.  70 sizes that it takes and
// swap_takes_less does not, timed on both sides: 1.10 times as fast on average (m 32768, k 2624, n 928, 26 groups 282 -> 237 us; 15103,
// 584, 8480, 16 402 -> 316), slower by more than 5 % in four (worst 8835, 384, 4192, 2, 12 blocks and a narrow last tile, 67 -> 75).
// Below three rounds either side wins by up to 1.6, by how rounds fall.
bool choose_swap_f32(long long m, int k_blocks, int n, int g, bool trans_rhs) {
  if (g <= 0 || (!trans_rhs && n % 32 != 0)) return false;
  if (swap_takes_less(m, k_blocks, n, g, 384, 1.0)) return true;
  if (m / g < 256 || k_blocks < 12) return false;
  const long long col_tiles = (static_cast<long long>(n) + rd::kSwapCols - 1) / rd::kSwapCols;
  return (col_tiles * rd::kSwapCols - n) * 10 <= n && (m / rd::kSwapRows + g / 2) * col_tiles >= 3 * (sm_count() / 2);
}

// Tensor maps and launch of the swapped kernel; k in 2-byte units for 8-bit and 16-bit types (kFp8: half of the elements).
template <bool kBKMajor, bool kFp8, bool kF32 = false>
int launch_gemm_swap(const void* x, const void* A, void* y, int dtype, int num_weights, GemmArgs args,
                     cudaStream_t stream) {
  constexpr int kDeep = kF32 ? rd::kF32TileK : rd::kTileK;  // elements in 128 bytes
  CUtensorMap tw, tx, tout, tout16;
  int rc;
  {
    const uint64_t dims[2] = {static_cast<uint64_t>(args.k), static_cast<uint64_t>(args.m)};
    const uint32_t box[2] = {kDeep, rd::kSwapRows / 2};
    rc = encode_map(&tx, x, dtype, 2, dims, box);
    if (rc != RD_OK) return rc;
  }
  if (kBKMajor) {
    const uint64_t dims[3] = {static_cast<uint64_t>(args.k), static_cast<uint64_t>(args.n),
                              static_cast<uint64_t>(num_weights)};
    const uint32_t box[3] = {kDeep, rd::kTileM, 1};  // one half of a CTA's columns
    rc = encode_map(&tw, A, dtype, 3, dims, box);
  } else {
    rc = encode_blocked_map(&tw, A, dtype, args.n, args.k, kDeep, rd::kTileM / kDeep, num_weights);
  }
  if (rc != RD_OK) return rc;
  {
    const uint64_t dims[2] = {static_cast<uint64_t>(args.n), static_cast<uint64_t>(args.m)};
    const uint32_t box[2] = {32, 32}, box16[2] = {32, 16};
    rc = encode_map(&tout, y, dtype, 2, dims, box, false, /*swizzled=*/false);
    if (rc != RD_OK) return rc;
    rc = encode_map(&tout16, y, dtype, 2, dims, box16, false, /*swizzled=*/false);
    if (rc != RD_OK) return rc;
  }
  args.n_tiles = (args.n + rd::kSwapCols - 1) / rd::kSwapCols;
  return launch_pairs<rd::ragged_gemm_swap_kernel<kBKMajor, kFp8, kF32>>(rd::kSwapThreads, rd::kSwapSmemBytes, args,
                      sm_count(), stream, tw, tx, tout, tout16);
}

// Tensor maps and launch of tgmm with two accumulators per CTA (rd_tgmm.cuh); args.k_tiles and n_tiles are set.
template <int kCtas>
int launch_tgmm(const void* x, const void* dout, const CUtensorMap& tout, int dtype, const GemmArgs& args, int ctas,
                cudaStream_t stream) {
  CUtensorMap ta, ta2, tb, tb2;
  int rc = encode_rows_map(&ta2, x, dtype, args.k, args.m, rd::kTileK);
  if (rc != RD_OK) return rc;
  rc = encode_rows_map(&tb2, dout, dtype, args.n, args.m, rd::kTileK);
  if (rc != RD_OK) return rc;
  // Whole blocks of 64 columns only; the kernel reads what is left through the plain maps.
  ta = ta2;
  tb = tb2;
  if (args.k >= 64) rc = encode_blocked_map(&ta, x, dtype, args.k, args.m, rd::kTileK, rd::kTileM / 64);
  if (rc == RD_OK && args.n >= 64)
    rc = encode_blocked_map(&tb, dout, dtype, args.n, args.m, rd::kTileK, rd::kTgTileN / 64 / kCtas);
  if (rc != RD_OK) return rc;
  constexpr auto kernel = rd::ragged_tgmm_kernel<kCtas>;
  constexpr int kSmem = rd::tg_smem_bytes<kCtas>();
  if constexpr (kCtas == 2)
    return launch_pairs<kernel, 2>(rd::kTgThreads, kSmem, args, ctas, stream, ta, ta2, tb, tb2, tout);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess)
    return RD_ERR_LAUNCH;
  return launch_kernel(kernel, ctas, rd::kTgThreads, kSmem, 1, launch_early(args, 1, false, 2), stream, ta, ta2, tb, tb2, tout,
                       args);
}

// Upper bound on the live 128 x 256 tiles of a gmm: a group has at least one row, and only whole
// 128-row steps of m add tiles to that.
long long split_tiles_bound(int m, int g, int n) {
  const long long row_tiles = (m < g ? m : g) + m / rd::kTileM;
  return row_tiles * ((n + rd::kSplitBN - 1) / rd::kSplitBN);
}

// Rows of a large tile: twice the mean of the groups that can have rows.
int split_tile_rows(int m, int g) {
  const long long mean2 = 2LL * m / (m < g ? m : g);
  return mean2 < rd::kTileM ? static_cast<int>(mean2) : rd::kTileM;
}

// Only calls that leave the tile and the grid to the library are split.
bool split_allowed(const rd_tile_cfg* cfg) {
  return cfg == nullptr || (cfg->tile_n == 0 && cfg->max_ctas == 0 && cfg->cta_group == 0 && cfg->tile_m == 0);
}

// 256-row tiles on one CTA (rd_gemm2.cuh) move a third less data per flop than 128-row tiles.
// They pay off when a tile's second half usually exists: tgmm with k >= 256, and gmm when the
// groups are long (a half without rows is skipped, so the cost of a wrong guess is only a
// shallower smem ring) -- unless the larger tiles fill the SMs badly.
// 512 rows per group and more: always from three rounds of 256-row tiles on (128 rows against 256, microseconds in a row, m,
// k, n, groups: 6120, 6528, 3304, 8 279 -> 237; 8304, 1768, 5112, 16 229 -> 182; equal on narrow outputs, 28448, 952, 576, 16 43 -> 45;
// 24104, 304, 2560, 6 50 -> 51).  Below, the rounds are compared, a 256-row tile taking 1.5 times as long as a 128-row one: 4096,
// 4096, 4096, 8 (4 rounds against 3, unequal groups) 120 -> 152; 512, 4096, 4096, 1 (1 against 1) 24 -> 42; but 6000, 4096, 1024, 8
// (2 against 1) 57 -> 50; 4352, 2928, 2232, 2 (3 against 2) 78 -> 70; 7184, 448, 2296, 8 (4 against 2) 24.7 -> 20.5.
// 256 to 511 rows: only where 256-row tiles need fewer rounds even with a tile more per group than m asks for and
// no tile more for 128 rows; 2048, 7168, 2048, 8 would take 2 rounds against 1 with unequal groups (90 -> 80) but
// 1 against 1 with equal ones (59 -> 92), and 6352, 968, 896, 24 loses (20 -> 30).
// e4m3, whose MMAs take half as long: 1.7 times, always from six rounds on, never with fewer than nine blocks of
// the contraction (m 8192, k 4096, n 14336, 8 groups 390 -> 378; but 8192, 14336, 4096, 16, five rounds against
// eight, 422 -> 472; 31480, 640, 1088, 32, five blocks, 46 -> 48).
bool choose_two_half(bool tgmm, long long m, int k, int n, int g, int bn, bool fp8 = false) {
  if (bn != 256 || g <= 0) return false;
  if (tgmm) return k >= 256;
  const long long rows = m / g, sms = sm_count();
  const long long n_tiles = (static_cast<long long>(n) + 255) / 256;
  auto rounds = [&](long long row_tiles) { return (row_tiles * n_tiles + sms - 1) / sms; };
  const long long m128 = (m + 127) / 128, m256 = (m + 255) / 256;
  if (rows < 512) return !fp8 && rows >= 256 && 1.84 * rounds(m256 + g) < static_cast<double>(rounds(m128));
  // a group's last tile is half full on average
  const long long tiles256 = (m256 + g / 2) * n_tiles, r128 = rounds(m128 + g / 2);
  if (fp8)
    return (k + 127) / 128 >= 9 && (tiles256 >= 6 * sms || 1.7 * rounds(m256 + g / 2) < static_cast<double>(r128));
  if (tiles256 >= 3 * sms) return true;
  // a twentieth of a round is no round: the tiles of a group are an estimate
  const long long r256 = (tiles256 - sms / 20 + sms - 1) / sms;
  return 1.5 * (r256 > 0 ? r256 : 1) <= static_cast<double>(r128);
}

// float32 tiles on CTA pairs (rd_gemm_f32_pair.cuh).  A caller who asks for three TF32 passes always
// gets them: only that kernel splits its operands.  One pass: tgmm with rows that are multiples of 32, where pairs take no
// more than a tenth more rounds of tiles; groups of 256 rows from two rounds on one CTA per tile on, of 100 from seven.
// Of 350 sizes timed on both sides that takes 109, one of them 7 % slower than on one CTA, the others 2 % at most.  One CTA
// against a pair, microseconds: m 4096, k 1536, n 4096, 32 unequal groups 201 -> 188; 16384, 2048, 2048, 128 506 -> 471; one
// round: 888, 1184, 2656, 1 15.5 -> 16.4; groups of 245 in five rounds: 14210, 1376, 160, 58 49 -> 57; without the
// column-blocked boxes (n 12976, 17 groups of 399) 457 -> 650.
// gmm on long groups takes the swapped kernel instead (choose_swap_f32).
bool choose_f32_pair(bool tgmm, long long m, int k, int n, int g, int bn, const rd_tile_cfg* cfg) {
  if (cfg && (cfg->flags & RD_CFG_F32_THREE_PASS)) return true;
  if (!tgmm || bn != 256 || g <= 0 || (cfg && (cfg->cta_group == 1 || cfg->tile_m == 128))) return false;
  if (k % 32 != 0 || n % 32 != 0) return false;
  const long long sms = sm_count(), cols = (static_cast<long long>(n) + 255) / 256 * g;
  const long long r1 = ((k + 127) / 128 * cols + sms - 1) / sms;
  const long long r2 = ((k + 255) / 256 * cols + sms / 2 - 1) / (sms / 2);
  return 10 * r2 <= 11 * r1 && r1 > 1 && (m / g >= 256 || (m / g >= 100 && r1 > 6));
}

// tgmm with 256-column tiles: which kernel?  By rounds of tiles (128 x 256 on one CTA, 256 x 256 on a pair) and the mean rows of
// a group.  Timed all five ways on 640 sizes (16 to 32768 rows per call, 1 to 256 groups, equal to heavy-tailed) the choice takes
// 1.1 % longer than the best of them on average.  Microseconds in a row, sizes m, k, n, groups:
// - One round: the plain 128-row kernel (rd_gemm.cuh), which starts sooner and has a stage more (171, 1880, 768, 3 6.3 against 7.5 on two
//   accumulators; 260, 1056, 3432, 1 7.7 against 9.2); from 768 rows per group on the MMAs count, and a pair moves a third less
//   data (2077, 344, 880, 1 19.8 -> 17.6; 9424, 640, 360, 2 37 -> 27; just above equal: 884, 4408, 536, 1 13.4 -> 12.8).
// - Groups of 512 rows and more: pairs, up to a quarter more rounds (m 8192, k 4096, n 14336, 8 groups 908 -> 722); of 256 rows up to
//   three rounds only with no more of them (2683, 472, 2600, 6 26.6 -> 23.1; three against two, 4150, 544, 1152, 10 16.4 -> 18.4).
// - Groups of 64 to 255 rows: pairs likewise, but from seven rounds on (9101, 4496, 1944, 37 307 -> 248; 672, 7288, 11816, 4 257 ->
//   232); up to six the plain kernel (7474, 376, 1280, 44 27.1 against 28.6; 579, 320, 8192, 3 10.7 against 14.3).  Up to 100 rows, more
//   than 36 rounds and rows that begin inside a sector: as below 64 rows (16612, 4216, 1576, 174 715 plain, pair 897; 4108, 11704, 424,
//   52 turned 160, 211).
// - Groups of less than 64 rows: up to three rounds the plain kernel, then by the output's rows.  Whole 256 bytes: two accumulators
//   (1085, 520, 2048, 67 33.2 plain, 29.2).  Other rows: a column tile's edge falls inside 256 bytes (or a sector) of every other
//   row, and what counts is that the CTAs that write either side of it stay side by side.  Whole sectors: two accumulators with the
//   order of columns turned by a place per row, so that no CTA meets the same columns again and again (115, 2248, 912, 93 73 plain,
//   68, turned 61); but the plain kernel with fewer rows than groups, tiles of which no CTA meets the same columns anyway and more than
//   63 rounds, nearly all of them zeros (18, 5912, 3680, 42 288 plain, turned 349; 25 such sizes 0.90, up to 63 rounds 1.08 times as
//   fast turned).  Rows that begin inside a sector (n % 16 == 8): the same where a CTA's step, `ctas`
//   tiles, shares a factor with the tiles of a row and the plain kernel's last tile, less to write than the others, always falls to the
//   same CTAs: where it pads a thirty-second of the row (128 groups of 42, k 4096, n 776 290 plain, 323, 195; 1288 551, 485, 362; 1104,
//   14168, 984, 92 one thread 831, 692), or a block of 64 with up to five tiles of rows (527, 280, 8984, 31 47 plain, 42) or from 160
//   rounds on (585, 3416, 9048, 65 one thread 1315, 1238; but in fewer rounds 280, 2688, 9320, 20 223, 268).  Otherwise the plain
//   kernel, whose CTAs write one tile at a time, its loops issued by one thread from 37 rounds on (kOneThread, rd_gemm.cuh; no padding:
//   396, 4928, 2504, 66 turned 467, 324).  On 775 sizes the better of the two within 1 % on average.
// - Few columns (n 296: 512 are multiplied by the plain kernel, 320 here, dealt evenly): two accumulators or pairs from four rounds on,
//   with less than 64 rows from three (90, 11464, 312, 2 9.9 plain, 8.5; two rounds equal), whatever the output's rows up to 36 rounds
//   (1796, 5480, 304, 10 24.6 plain, 20.6; groups below 64 rows 1.07 to 1.4 times as fast; but with 140 rounds 67, 11464, 520, 77 one
//   thread 205, turned 241).
enum class TgmmWay { kPair, kPlain, kOneThread, kTwoAcc, kTurned };
TgmmWay tgmm_way(long long m, int k, int n, int g, int ctas, int cta_group) {
  const long long rows = m / g, tiles = (static_cast<long long>(n) + 255) / 256, blocks = (static_cast<long long>(n) + 63) / 64;
  const long long r1 = ((k + 127) / 128 * tiles * g + ctas - 1) / ctas;
  const bool narrow = 40 * tiles >= 13 * blocks;  // tiles of 256 columns are 1.3 times the columns there are
  const bool split = n % 16 != 0 && rows <= 100 && r1 > 36;  // sectors in two parts, more output than L2 holds
  if (cta_group == 2) return TgmmWay::kPair;
  if (cta_group == 0) {
    const long long pairs = sm_count() / 2, r2 = ((k + 255) / 256 * tiles * g + pairs - 1) / pairs;
    if (r1 <= 1) {
      if (rows >= 768 && r2 <= 1) return TgmmWay::kPair;
    } else if (rows >= 512 || (rows >= 256 && r1 > 3) || (rows >= 64 && r1 > (narrow ? 3 : 6) && !split)) {
      if (4 * r2 <= 5 * r1) return TgmmWay::kPair;
    } else if (rows >= 256) {
      if (r2 <= r1) return TgmmWay::kPair;
    }
  }
  if (r1 <= (narrow && rows < 64 ? 2 : 3) || (rows >= 64 && !narrow && !split)) return TgmmWay::kPlain;
  if (n % 128 == 0 || tiles == 1) return TgmmWay::kTwoAcc;
  const bool shared = std::gcd(tiles, static_cast<long long>(ctas)) > 1;
  if (n % 16 == 0 && rows == 0 && r1 > 63 && !shared && !narrow) return TgmmWay::kPlain;
  if (n % 16 == 0 || (narrow && r1 <= 36)) return TgmmWay::kTurned;
  const long long padding = 256 * tiles - n;
  if (shared && (padding >= 8 * tiles || (padding >= 64 && (r1 >= 160 || k <= 640)))) return TgmmWay::kTurned;
  return r1 > 36 ? TgmmWay::kOneThread : TgmmWay::kPlain;
}

// Limit of every bounded wait inside a kernel, in microseconds: rd_tile_cfg.wait_limit_ms if
// set, else the environment variable RD_WAIT_LIMIT_MS (read once), else two seconds.
uint32_t wait_limit_us(const rd_tile_cfg* cfg) {
  static const long env_ms = [] {
    const char* v = getenv("RD_WAIT_LIMIT_MS");
    const long ms = v ? strtol(v, nullptr, 10) : 0;
    return ms > 0 ? ms : 0;
  }();
  long ms = (cfg && cfg->wait_limit_ms > 0) ? cfg->wait_limit_ms : env_ms;
  if (ms <= 0) return rd::kDefaultWaitLimitUs;
  if (ms > 4000000) ms = 4000000;
  return static_cast<uint32_t>(ms) * 1000u;
}

int pick_ctas(const rd_tile_cfg* cfg) {
  int ctas = sm_count();
  if (cfg && cfg->max_ctas > 0 && cfg->max_ctas < ctas) ctas = cfg->max_ctas;
  return ctas;
}

}  // namespace

extern "C" {

int rd_version(void) { return RD_VERSION; }

const char* rd_status_string(int code) {
  switch (code) {
    case RD_OK: return "ok";
    case RD_ERR_BAD_SHAPE: return "bad shape: sizes must be >= 0 and rows of k, n elements multiples of 16 bytes";
    case RD_ERR_BAD_DTYPE: return "unsupported dtype: f16, bf16 or f32";
    case RD_ERR_BAD_POINTER: return "null or misaligned pointer (16-byte alignment required)";
    case RD_ERR_WORKSPACE: return "workspace too small (see rd_workspace_bytes)";
    case RD_ERR_BAD_CONFIG: return "unsupported tile configuration";
    case RD_ERR_TENSOR_MAP: return "driver rejected a TMA tensor map";
    case RD_ERR_LAUNCH: return "kernel launch failed";
    case RD_ERR_DRIVER: return "cuTensorMapEncodeTiled entry point not available";
    case RD_ERR_DEVICE_WAIT: return "a bounded wait inside a kernel expired";
    case RD_ERR_TOO_LARGE:
      return "problem too large for the built-in scratch of rd_gmm_static_scratch "
             "(needs 12*g + 10*ceil(m/128) + 16 <= 16384 words); use rd_gmm with a workspace";
    case RD_ERR_SCRATCH_SETUP: return "could not resolve the address of the built-in scratch array";
    default: return "unknown status";
  }
}

int rd_workspace_bytes(int m, int g, size_t* bytes) {
  if (m < 0 || g < 0 || bytes == nullptr) return RD_ERR_BAD_SHAPE;
  WorkspaceLayout l;
  l.g = g;
  l.max_tiles = max_row_tiles(m, g);
  size_t b = static_cast<size_t>(l.total_words()) * sizeof(int32_t);
  *bytes = (b + 255) & ~static_cast<size_t>(255);
  return RD_OK;
}

int rd_metadata(const int32_t* group_sizes, int g, int m, int chunk_m, int32_t* group_offsets,
                int32_t* row_it2group, int32_t* row_it2it_in_group, int32_t* total_row_its,
                void* stream) {
  if (g < 0 || m < 0 || chunk_m <= 0) return RD_ERR_BAD_SHAPE;
  if (g == 0) {
    // U = ceil(m / chunk_m) rows of zeros and a zero total.
    const int u = (m + chunk_m - 1) / chunk_m;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (row_it2group && u) cudaMemsetAsync(row_it2group, 0, sizeof(int32_t) * u, s);
    if (row_it2it_in_group && u) cudaMemsetAsync(row_it2it_in_group, 0, sizeof(int32_t) * u, s);
    if (total_row_its) cudaMemsetAsync(total_row_its, 0, sizeof(int32_t), s);
    return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
  }
  if (group_sizes == nullptr) return RD_ERR_BAD_POINTER;
  const int u = (m + chunk_m - 1) / chunk_m + g;
  rd::group_metadata_kernel<<<1, rd::kMetaThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      group_sizes, g, m, chunk_m, u, group_offsets, row_it2group, row_it2it_in_group,
      total_row_its, nullptr, nullptr, nullptr, nullptr, nullptr);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

// Shared body of rd_gmm / rd_gmm_indexed.  `num_weights` is A's leading dimension;
// `group_to_weight` (device, [g]) is null when group i uses A[i].
struct ReadyFlags {
  const int32_t* flags;  // null: no waiting
  int groups_per_flag;
  int epoch;
};

static int gmm_impl(const void* x, const void* A, const int32_t* group_sizes,
                    const int32_t* group_to_weight, int num_weights, void* y, void* workspace,
                    size_t workspace_bytes, int m, int k, int n, int g, int trans_rhs, int dtype,
                    const rd_tile_cfg* cfg, void* stream_v, ReadyFlags ready = {nullptr, 1, 0},
                    const rd::EpSendArgs* send = nullptr) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (dtype != RD_DTYPE_F16 && dtype != RD_DTYPE_BF16 && dtype != RD_DTYPE_F32) return RD_ERR_BAD_DTYPE;
  const bool f32 = dtype == RD_DTYPE_F32;
  const int esize = f32 ? 4 : 2;            // bytes per element
  const int amask = f32 ? 3 : 7;            // rows must be multiples of 16 bytes
  const int row_elems = 128 / esize;        // elements per 128-byte swizzle row
  if (m < 0 || k < 0 || n < 0 || g < 0 || num_weights < 0 || (k & amask) || (n & amask))
    return RD_ERR_BAD_SHAPE;
  if (m == 0 || n == 0) return RD_OK;
  if (!aligned16(y)) return RD_ERR_BAD_POINTER;
  if (g == 0 || k == 0 || num_weights == 0) {  // nothing contributes: every row is a zero row
    cudaMemsetAsync(y, 0, static_cast<size_t>(m) * n * esize, stream);
    return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
  }
  if (!aligned16(x) || !aligned16(A) || group_sizes == nullptr) return RD_ERR_BAD_POINTER;
  Workspace w;
  int rc = bind_workspace(workspace, workspace_bytes, m, g, &w);
  if (rc != RD_OK) return rc;

  const int sms = sm_count();
  int bn = cfg && cfg->tile_n ? cfg->tile_n : choose_tile_n((m + rd::kTileM - 1) / rd::kTileM, n, sms);
  if (bn != 64 && bn != 128 && bn != 256) return RD_ERR_BAD_CONFIG;
  int cta_group = cfg ? cfg->cta_group : 0;
  if (cta_group < 0 || cta_group > 2 || (cta_group == 2 && bn != 256)) return RD_ERR_BAD_CONFIG;
  // 256-row tiles on pairs waste more of a group's last rows than the pair saves: only on request.
  if (cta_group == 0) cta_group = 1;
  int tile_m = cfg ? cfg->tile_m : 0;
  if (tile_m != 0 && tile_m != 128 && tile_m != 256) return RD_ERR_BAD_CONFIG;
  if (tile_m == 256 && (bn != 256 || cta_group != 1)) return RD_ERR_BAD_CONFIG;
  const bool three_pass = cfg && (cfg->flags & RD_CFG_F32_THREE_PASS);
  if (three_pass && !f32) return RD_ERR_BAD_CONFIG;
  if (f32) {  // the float32 kernels choose between one CTA and a pair themselves
    if ((cfg && cfg->cta_group == 2) || tile_m == 256) return RD_ERR_BAD_CONFIG;
    const bool pair = choose_f32_pair(false, m, k, n, g, bn, cfg);
    if (pair) bn = rd::kF32PairBN;
    cta_group = pair ? 2 : 1;
    tile_m = 128;
  }
  if (tile_m == 0) tile_m = (cta_group == 1 && choose_two_half(false, m, k, n, g, bn)) ? 256 : 128;
  const bool two_half = tile_m == 256;

  // The expert-parallel forms (flags, senders, groups visited by weight) keep the metadata launch.
  const bool by_weight = cfg != nullptr && (cfg->flags & RD_CFG_GROUP_BY_WEIGHT) != 0;
  const bool in_kernel = inline_groups(m, g) && ready.flags == nullptr && send == nullptr &&
                         !(by_weight && group_to_weight != nullptr);
  const long long split_tiles = split_tiles_bound(m, g, n);
  int split = 1;
  if (in_kernel && !f32 && !two_half && cta_group == 1 && split_allowed(cfg)) {
    const int k_blocks = (k + rd::kTileK - 1) / rd::kTileK;
    split = trans_rhs ? choose_split<true, false>(split_tiles, split_tile_rows(m, g), k_blocks)
                      : choose_split<false, false>(split_tiles, split_tile_rows(m, g), k_blocks);
    if (split > 1) bn = rd::kSplitBN;
  }
  if (in_kernel) {
    rc = ensure_context();
    if (rc != RD_OK) return rc;
  } else {
    launch_internal_metadata(group_sizes, group_to_weight, g, m,
                             two_half ? rd::kG2TileRows : rd::kTileM * cta_group, w, stream, by_weight);
    if (cudaGetLastError() != cudaSuccess) return RD_ERR_LAUNCH;
  }
  if (in_kernel && split == 1 && split_allowed(cfg) &&
      (f32 ? !three_pass && choose_swap_f32(m, (k + rd::kF32TileK - 1) / rd::kF32TileK, n, g, trans_rhs != 0)
           : choose_swap(m, (k + rd::kTileK - 1) / rd::kTileK, n, g, trans_rhs != 0, false))) {
    GemmArgs args = {};
    args.m = m; args.k = k; args.n = n; args.g = g;
    args.max_m_tiles = w.layout.max_tiles;
    args.ab_format = dtype;
    args.wait_limit_us = wait_limit_us(cfg);
    args.zero_tail = (cfg && (cfg->flags & RD_CFG_NO_ZERO_TAIL)) ? 0 : 1;
    args.inline_groups = 1;
    args.group_to_weight = group_to_weight;
    args.group_sizes = group_sizes;
    args.status = w.status();
    args.out = y;
    if (f32)
      return trans_rhs ? launch_gemm_swap<true, false, true>(x, A, y, dtype, num_weights, args, stream)
                       : launch_gemm_swap<false, false, true>(x, A, y, dtype, num_weights, args, stream);
    return trans_rhs ? launch_gemm_swap<true, false>(x, A, y, dtype, num_weights, args, stream)
                     : launch_gemm_swap<false, false>(x, A, y, dtype, num_weights, args, stream);
  }

  // float32 weights [k, n] with rows that are multiples of 32: one box per stage instead of one per 32 columns.
  const bool blocked = f32 && !trans_rhs && n % 32 == 0;
  CUtensorMap ta, tb;
  {
    const uint64_t dims[2] = {static_cast<uint64_t>(k), static_cast<uint64_t>(m)};
    const uint32_t box[2] = {static_cast<uint32_t>(row_elems), rd::kTileM};
    rc = encode_map(&ta, x, dtype, 2, dims, box);
    if (rc != RD_OK) return rc;
  }
  if (trans_rhs) {  // A[g, n, k]: rows of k, K-major operand, one [BN][128 B] box per stage
    const uint64_t dims[3] = {static_cast<uint64_t>(k), static_cast<uint64_t>(n),
                              static_cast<uint64_t>(num_weights)};
    const uint32_t box[3] = {static_cast<uint32_t>(row_elems), static_cast<uint32_t>(bn / cta_group), 1};
    rc = encode_map(&tb, A, dtype, 3, dims, box);
  } else if (blocked) {
    rc = encode_blocked_map(&tb, A, dtype, n, k, row_elems, bn / cta_group / 32, num_weights);
  } else {  // A[g, k, n]: rows of n, MN-major operand, [stage-depth k][128 B of n] boxes
    const uint64_t dims[3] = {static_cast<uint64_t>(n), static_cast<uint64_t>(k),
                              static_cast<uint64_t>(num_weights)};
    const uint32_t box[3] = {static_cast<uint32_t>(row_elems), static_cast<uint32_t>(row_elems), 1};
    rc = encode_map(&tb, A, dtype, 3, dims, box, /*atom32=*/f32);  // MN-major fp32: 32-byte atoms
  }
  if (rc != RD_OK) return rc;
  CUtensorMap tout;
  {  // y[m, n] written as [32 rows][128 B] boxes
    const uint64_t dims[2] = {static_cast<uint64_t>(n), static_cast<uint64_t>(m)};
    const uint32_t box[2] = {static_cast<uint32_t>(row_elems), 32};
    rc = encode_map(&tout, y, dtype, 2, dims, box);
    if (rc != RD_OK) return rc;
  }

  GemmArgs args = {};
  args.m = m; args.k = k; args.n = n; args.g = g;
  args.n_tiles = (n + bn - 1) / bn;
  args.k_tiles = 0;
  args.blocked_maps = blocked ? 1 : 0;
  args.max_m_tiles = w.layout.max_tiles;
  args.ab_format = dtype;
  args.wait_limit_us = wait_limit_us(cfg);
  args.zero_tail = (cfg && (cfg->flags & RD_CFG_NO_ZERO_TAIL)) ? 0 : 1;
  args.group_sizes = group_sizes;
  args.group_offsets = w.group_offsets();
  args.tile_rec = w.tile_rec();
  args.totals = w.totals();
  args.status = w.status();
  args.out = y;
  args.inline_groups = in_kernel ? 1 : 0;
  args.group_to_weight = group_to_weight;
  args.ready_flags = ready.flags;
  args.groups_per_flag = ready.groups_per_flag > 0 ? ready.groups_per_flag : 1;
  args.ready_epoch = ready.epoch;
  if (send != nullptr) {
    if (f32 || cta_group == 2) return RD_ERR_BAD_CONFIG;  // the sender role lives in the 16-bit 1-CTA kernels
    args.send = *send;
  }

  const int ctas = pick_ctas(cfg);
  if (send != nullptr && send->sender_ctas >= ctas) return RD_ERR_BAD_CONFIG;
  if (f32) {
    if (ready.flags != nullptr) return RD_ERR_BAD_DTYPE;  // the float32 kernels do not wait on flags
    if (cta_group == 2)  // three passes
      return trans_rhs ? launch_gemm_f32_pair<true, false, true>(ta, tb, tout, args, ctas, stream)
                       : launch_gemm_f32_pair<false, false, true>(ta, tb, tout, args, ctas, stream);
    if (trans_rhs) {
      if (bn == 256) return launch_gemm_f32<256, true, false>(ta, tb, tout, args, ctas, stream);
      if (bn == 128) return launch_gemm_f32<128, true, false>(ta, tb, tout, args, ctas, stream);
      return launch_gemm_f32<64, true, false>(ta, tb, tout, args, ctas, stream);
    }
    if (bn == 256) return launch_gemm_f32<256, false, false>(ta, tb, tout, args, ctas, stream);
    if (bn == 128) return launch_gemm_f32<128, false, false>(ta, tb, tout, args, ctas, stream);
    return launch_gemm_f32<64, false, false>(ta, tb, tout, args, ctas, stream);
  }
  if (split > 1)
    return trans_rhs ? launch_gemm_splitk<true, false>(ta, tb, args, split, static_cast<int>(split_tiles), stream)
                     : launch_gemm_splitk<false, false>(ta, tb, args, split, static_cast<int>(split_tiles), stream);
  if (two_half) {
    return trans_rhs ? launch_gemm2<true, false>(ta, tb, tout, args, ctas, stream)
                     : launch_gemm2<false, false>(ta, tb, tout, args, ctas, stream);
  }
  if (trans_rhs) {
    if (cta_group == 2) return launch_gemm<256, true, false, 2>(ta, tb, tout, args, ctas, stream);
    if (bn == 256) return launch_gemm<256, true, false, 1>(ta, tb, tout, args, ctas, stream);
    if (bn == 128) return launch_gemm<128, true, false, 1>(ta, tb, tout, args, ctas, stream);
    return launch_gemm<64, true, false, 1>(ta, tb, tout, args, ctas, stream);
  }
  if (cta_group == 2) return launch_gemm<256, false, false, 2>(ta, tb, tout, args, ctas, stream);
  if (bn == 256) return launch_gemm<256, false, false, 1>(ta, tb, tout, args, ctas, stream);
  if (bn == 128) return launch_gemm<128, false, false, 1>(ta, tb, tout, args, ctas, stream);
  return launch_gemm<64, false, false, 1>(ta, tb, tout, args, ctas, stream);
}

int rd_gmm(const void* x, const void* A, const int32_t* group_sizes, void* y, void* workspace,
           size_t workspace_bytes, int m, int k, int n, int g, int trans_rhs, int dtype,
           const rd_tile_cfg* cfg, void* stream) {
  return gmm_impl(x, A, group_sizes, nullptr, g, y, workspace, workspace_bytes, m, k, n, g, trans_rhs,
                  dtype, cfg, stream);
}

int rd_gmm_indexed(const void* x, const void* A, int num_weights, const int32_t* group_sizes,
                   const int32_t* group_to_weight, void* y, void* workspace, size_t workspace_bytes,
                   int m, int k, int n, int g, int trans_rhs, int dtype, const rd_tile_cfg* cfg,
                   void* stream) {
  if (g > 0 && group_to_weight == nullptr) return RD_ERR_BAD_POINTER;
  return gmm_impl(x, A, group_sizes, group_to_weight, num_weights, y, workspace, workspace_bytes, m, k,
                  n, g, trans_rhs, dtype, cfg, stream);
}

static int gather_rows_impl(const void* src, const int32_t* row_index, void* dst, int rows_out, int rows_in,
                            int row_bytes, bool clamp, void* stream) {
  if (rows_out < 0 || rows_in < 0 || row_bytes < 0 || (row_bytes & 15)) return RD_ERR_BAD_SHAPE;
  if (rows_out == 0 || row_bytes == 0) return RD_OK;
  if (!aligned16(src) || !aligned16(dst) || row_index == nullptr) return RD_ERR_BAD_POINTER;
  const int warps_per_block = rd::kGatherThreads / 32;
  int blocks = (rows_out + warps_per_block - 1) / warps_per_block;
  const int cap = sm_count() * 8;
  if (blocks > cap) blocks = cap;
  rd::gather_rows_kernel<<<blocks, rd::kGatherThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(src), row_index, static_cast<uint4*>(dst), rows_out, rows_in,
      row_bytes / 16, clamp);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_gather_rows(const void* src, const int32_t* row_index, void* dst, int rows_out, int rows_in,
                   int row_bytes, void* stream) {
  return gather_rows_impl(src, row_index, dst, rows_out, rows_in, row_bytes, false, stream);
}

int rd_gather_rows_clamped(const void* src, const int32_t* row_index, void* dst, int rows_out, int rows_in,
                           int row_bytes, void* stream) {
  return gather_rows_impl(src, row_index, dst, rows_out, rows_in, row_bytes, true, stream);
}

size_t rd_sum_rows_scratch_bytes(int rows_in, int rows_out) {
  if (rows_in < 0 || rows_out < 0) return 0;
  return (2 * static_cast<size_t>(rows_out) + 1 + 2 * static_cast<size_t>(rows_in)) * sizeof(int32_t);
}

int rd_sum_rows(const void* src, const int32_t* row_index, const int32_t* group_sizes, int g, void* dst,
                int rows_in, int rows_out, int cols, int dtype, void* scratch, size_t scratch_bytes,
                void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (dtype != RD_DTYPE_F16 && dtype != RD_DTYPE_BF16 && dtype != RD_DTYPE_F32) return RD_ERR_BAD_DTYPE;
  if (rows_in < 0 || rows_out < 0 || cols < 0 || g < 0) return RD_ERR_BAD_SHAPE;
  if (rows_out == 0 || cols == 0) return RD_OK;
  if (dst == nullptr) return RD_ERR_BAD_POINTER;
  const size_t row_bytes = static_cast<size_t>(cols) * (dtype == RD_DTYPE_F32 ? 4 : 2);
  if (rows_in == 0 || g == 0) {
    cudaMemsetAsync(dst, 0, row_bytes * rows_out, stream);
    return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
  }
  if (src == nullptr || row_index == nullptr || group_sizes == nullptr) return RD_ERR_BAD_POINTER;
  if (scratch == nullptr || (reinterpret_cast<uintptr_t>(scratch) & 3u)) return RD_ERR_BAD_POINTER;
  if (scratch_bytes < rd_sum_rows_scratch_bytes(rows_in, rows_out)) return RD_ERR_WORKSPACE;
  int32_t* count = static_cast<int32_t*>(scratch);
  int32_t* cursor = count + rows_out;
  int32_t* start = cursor + 1;
  int32_t* rank = start + rows_out;
  int32_t* list = rank + rows_in;
  if (cudaMemsetAsync(count, 0, sizeof(int32_t) * (static_cast<size_t>(rows_out) + 1), stream) != cudaSuccess)
    return RD_ERR_LAUNCH;
  constexpr int kT = rd::kGatherThreads;
  rd::sum_rows_count_kernel<<<(rows_in + kT - 1) / kT, kT, 0, stream>>>(row_index, rows_in, rows_out, group_sizes,
                                                                      g, count, rank);
  rd::sum_rows_start_kernel<<<(rows_out + kT - 1) / kT, kT, 0, stream>>>(count, rows_out, start, cursor);
  rd::sum_rows_fill_kernel<<<(rows_in + kT - 1) / kT, kT, 0, stream>>>(row_index, rows_in, rows_out, start, rank,
                                                                     list);
  const bool wide = row_bytes % 16 == 0 && aligned16(src) && aligned16(dst);
  const int vec = wide ? (dtype == RD_DTYPE_F32 ? 4 : 8) : 1;
  const int vecs = cols / vec;
  const int chunks = (vecs + 127) / 128;
  const long long warps = static_cast<long long>(rows_out) * chunks;
  long long blocks = (warps + kT / 32 - 1) / (kT / 32);
  const long long cap = static_cast<long long>(sm_count()) * 64;
  if (blocks > cap) blocks = cap;
#define RD_SUM_ROWS(TY, V)                                                                              \
  rd::sum_rows_kernel<TY, V><<<static_cast<int>(blocks), kT, 0, stream>>>(                                \
      static_cast<const uint8_t*>(src), list, start, count, static_cast<uint8_t*>(dst), rows_out, vecs, chunks)
  if (dtype == RD_DTYPE_F32) { if (wide) RD_SUM_ROWS(2, 4); else RD_SUM_ROWS(2, 1); }
  else if (dtype == RD_DTYPE_BF16) { if (wide) RD_SUM_ROWS(1, 8); else RD_SUM_ROWS(1, 1); }
  else { if (wide) RD_SUM_ROWS(0, 8); else RD_SUM_ROWS(0, 1); }
#undef RD_SUM_ROWS
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_zero_unwritten_rows(void* y, int y_rows, int row_bytes, const int32_t* out_rows, int m,
                           const int32_t* group_sizes, int g, int32_t* scratch, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (y_rows < 0 || m < 0 || g < 0 || row_bytes < 0 || (row_bytes & 15)) return RD_ERR_BAD_SHAPE;
  if (y_rows == 0 || row_bytes == 0) return RD_OK;
  if (!aligned16(y) || scratch == nullptr) return RD_ERR_BAD_POINTER;
  if (m > 0 && g > 0 && (out_rows == nullptr || group_sizes == nullptr)) return RD_ERR_BAD_POINTER;
  if (cudaMemsetAsync(scratch, 0, sizeof(int32_t) * y_rows, stream) != cudaSuccess) return RD_ERR_LAUNCH;
  constexpr int kT = rd::kGatherThreads;
  if (m > 0 && g > 0)
    rd::mark_rows_kernel<<<(m + kT - 1) / kT, kT, 0, stream>>>(out_rows, m, y_rows, group_sizes, g, scratch);
  int blocks = (y_rows + kT / 32 - 1) / (kT / 32);
  const int cap = sm_count() * 8;
  if (blocks > cap) blocks = cap;
  rd::zero_unwritten_rows_kernel<<<blocks, kT, 0, stream>>>(scratch, static_cast<uint4*>(y), y_rows,
                                                            row_bytes / 16);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_ep_count(const int32_t* routing, int entries, int num_experts, int32_t* counts, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (entries < 0 || num_experts <= 0 || num_experts > 8192) return RD_ERR_BAD_SHAPE;
  if (counts == nullptr || (entries > 0 && routing == nullptr)) return RD_ERR_BAD_POINTER;
  if (cudaMemsetAsync(counts, 0, sizeof(int32_t) * num_experts, stream) != cudaSuccess)
    return RD_ERR_LAUNCH;
  if (entries == 0) return RD_OK;
  int blocks = (entries + rd::kEpThreads - 1) / rd::kEpThreads;
  if (blocks > sm_count()) blocks = sm_count();
  rd::ep_count_kernel<<<blocks, rd::kEpThreads, sizeof(int32_t) * num_experts, stream>>>(
      routing, entries, num_experts, counts);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_ep_plan(const int32_t* counts_all, int world, int num_experts, int rank, int32_t* dest_offset,
               int32_t* segment_sizes, int32_t* fill, int32_t* totals, void* stream) {
  if (world <= 0 || num_experts <= 0 || num_experts % world != 0 || rank < 0 || rank >= world)
    return RD_ERR_BAD_SHAPE;
  if (!counts_all || !dest_offset || !segment_sizes || !fill || !totals) return RD_ERR_BAD_POINTER;
  rd::ep_plan_kernel<<<1, rd::kEpThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      counts_all, world, num_experts, rank, dest_offset, segment_sizes, fill, totals, 0, nullptr, nullptr,
      nullptr, nullptr, 0, 0u, nullptr);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_ep_plan_ring(const int32_t* counts_all, int world, int num_experts, int rank,
                    int32_t* dest_offset, int32_t* segment_sizes, int32_t* fill, int32_t* totals,
                    int32_t* phase_done, int32_t* send_start, int32_t* list_fill, void* stream) {
  if (world <= 0 || num_experts <= 0 || num_experts % world != 0 || rank < 0 || rank >= world)
    return RD_ERR_BAD_SHAPE;
  if (!counts_all || !dest_offset || !segment_sizes || !fill || !totals || !phase_done)
    return RD_ERR_BAD_POINTER;
  if ((send_start == nullptr) != (list_fill == nullptr)) return RD_ERR_BAD_POINTER;
  rd::ep_plan_kernel<<<1, rd::kEpThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      counts_all, world, num_experts, rank, dest_offset, segment_sizes, fill, totals, 1, phase_done,
      send_start, list_fill, nullptr, 0, 0u, nullptr);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_ep_count_share(const int32_t* routing, int entries, int num_experts, int32_t* counts_scratch,
                      int32_t* ticket, int world, int rank, const uint64_t* peer_counts,
                      const uint64_t* peer_flags, int epoch, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (entries < 0 || num_experts <= 0 || num_experts > 8192 || world <= 0 || world > rd::kEpThreads ||
      rank < 0 || rank >= world)
    return RD_ERR_BAD_SHAPE;
  if (!counts_scratch || !ticket || !peer_counts || !peer_flags || (entries > 0 && routing == nullptr))
    return RD_ERR_BAD_POINTER;
  int blocks = (entries + rd::kEpThreads - 1) / rd::kEpThreads;
  if (blocks > sm_count()) blocks = sm_count();
  if (blocks < 1) blocks = 1;  // the counts (zeros) and the flag go out even without entries
  rd::ep_count_share_kernel<<<blocks, rd::kEpThreads, sizeof(int32_t) * num_experts, stream>>>(
      routing, entries, num_experts, counts_scratch, ticket, world, rank, peer_counts, peer_flags, epoch);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_ep_plan_ring_when_counted(const int32_t* counts_all, const int32_t* count_flags, int epoch,
                                 int world, int num_experts, int rank, int32_t* dest_offset,
                                 int32_t* segment_sizes, int32_t* fill, int32_t* totals,
                                 int32_t* phase_done, int32_t* send_start, int32_t* list_fill,
                                 int32_t* status, int wait_limit_ms, void* stream) {
  if (world <= 0 || world > rd::kEpThreads || num_experts <= 0 || num_experts % world != 0 || rank < 0 ||
      rank >= world)
    return RD_ERR_BAD_SHAPE;
  if (!counts_all || !count_flags || !dest_offset || !segment_sizes || !fill || !totals || !phase_done)
    return RD_ERR_BAD_POINTER;
  if ((send_start == nullptr) != (list_fill == nullptr)) return RD_ERR_BAD_POINTER;
  rd_tile_cfg cfg = {};
  cfg.wait_limit_ms = wait_limit_ms;
  rd::ep_plan_kernel<<<1, rd::kEpThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      counts_all, world, num_experts, rank, dest_offset, segment_sizes, fill, totals, 1, phase_done,
      send_start, list_fill, count_flags, epoch, wait_limit_us(&cfg), status);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_ep_assign(const int32_t* routing, int entries, int num_experts, int world, int rank,
                 const int32_t* dest_offset, int32_t* fill, int capacity_rows, int32_t* dest_pos,
                 const int32_t* send_start, int32_t* list_fill, int32_t* send_index, void* stream) {
  if (entries < 0 || world <= 0 || num_experts <= 0 || num_experts % world != 0 || rank < 0 ||
      rank >= world || capacity_rows < 0)
    return RD_ERR_BAD_SHAPE;
  if (entries == 0) return RD_OK;
  if (!routing || !dest_offset || !fill || !dest_pos || !send_start || !list_fill || !send_index)
    return RD_ERR_BAD_POINTER;
  if (num_experts + world > 5000) return RD_ERR_BAD_SHAPE;  // shared-memory counters of the kernel
  const int blocks = (entries + rd::kEpThreads - 1) / rd::kEpThreads;
  const size_t smem = 2 * static_cast<size_t>(num_experts + world) * sizeof(int32_t);
  rd::ep_assign_kernel<<<blocks, rd::kEpThreads, smem, static_cast<cudaStream_t>(stream)>>>(
      routing, entries, num_experts, num_experts / world, world, rank, dest_offset, fill, capacity_rows,
      dest_pos, send_start, list_fill, send_index);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_ep_send_list(const void* x, int top_k, int row_bytes, const int32_t* send_index,
                    const int32_t* send_start, int phase, int world, int max_rows,
                    const int32_t* dest_pos, void* dest_base, int capacity_rows, int32_t* phase_done,
                    int32_t* dest_ready_flag, int epoch, void* stream) {
  if (top_k <= 0 || row_bytes <= 0 || (row_bytes & 15) || world <= 0 || phase < 0 || phase >= world ||
      max_rows < 0 || capacity_rows < 0)
    return RD_ERR_BAD_SHAPE;
  if (!aligned16(dest_base) || !send_index || !send_start || !dest_pos || !phase_done ||
      !dest_ready_flag || (max_rows > 0 && !aligned16(x)))
    return RD_ERR_BAD_POINTER;
  const int warps_per_block = rd::kEpThreads / 32;
  int blocks = (max_rows + warps_per_block - 1) / warps_per_block;
  const int cap = sm_count() * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;  // the flag is raised even when the list is empty
  rd::ep_send_list_kernel<<<blocks, rd::kEpThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(x), top_k, row_bytes / 16, send_index, send_start, phase, dest_pos,
      static_cast<uint4*>(dest_base), capacity_rows, phase_done, dest_ready_flag, epoch);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_ep_combine_pull(const int32_t* routing, const int32_t* dest_pos, int tokens, int top_k,
                       int row_bytes, int num_experts, int world, const uint64_t* peer_base,
                       int capacity_rows, int dtype, void* out, int max_blocks, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (dtype != RD_DTYPE_F16 && dtype != RD_DTYPE_BF16) return RD_ERR_BAD_DTYPE;
  if (tokens < 0 || top_k <= 0 || top_k > 8 || row_bytes <= 0 || (row_bytes & 15) || world <= 0 ||
      num_experts <= 0 || num_experts % world != 0 || capacity_rows < 0)
    return RD_ERR_BAD_SHAPE;
  if (tokens == 0) return RD_OK;
  if (!routing || !dest_pos || !peer_base || !aligned16(out)) return RD_ERR_BAD_POINTER;
  const int warps_per_block = rd::kEpThreads / 32;
  int blocks = (tokens + warps_per_block - 1) / warps_per_block;
  const int cap = max_blocks > 0 ? max_blocks : sm_count() * 8;
  if (blocks > cap) blocks = cap;
  const int vecs = row_bytes / 16, local = num_experts / world;
  uint4* o = static_cast<uint4*>(out);
#define RD_COMBINE(BF, TK)                                                                          \
  rd::ep_combine_pull_kernel<BF, TK><<<blocks, rd::kEpThreads, 0, stream>>>(                        \
      routing, dest_pos, tokens, top_k, vecs, num_experts, local, peer_base, capacity_rows, o)
  const bool bf = dtype == RD_DTYPE_BF16;
  if (top_k <= 2) { if (bf) RD_COMBINE(true, 2); else RD_COMBINE(false, 2); }
  else if (top_k <= 4) { if (bf) RD_COMBINE(true, 4); else RD_COMBINE(false, 4); }
  else { if (bf) RD_COMBINE(true, 8); else RD_COMBINE(false, 8); }
#undef RD_COMBINE
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

int rd_gmm_indexed_when_ready(const void* x, const void* A, int num_weights, const int32_t* group_sizes,
                              const int32_t* group_to_weight, void* y, void* workspace,
                              size_t workspace_bytes, int m, int k, int n, int g, int trans_rhs,
                              int dtype, const rd_tile_cfg* cfg, const int32_t* ready_flags,
                              int groups_per_flag, int epoch, void* stream) {
  if (g > 0 && group_to_weight == nullptr) return RD_ERR_BAD_POINTER;
  if (ready_flags == nullptr) return RD_ERR_BAD_POINTER;
  if (groups_per_flag <= 0) return RD_ERR_BAD_SHAPE;
  if (cfg && cfg->cta_group == 2) return RD_ERR_BAD_CONFIG;  // CTA pairs do not wait on flags
  return gmm_impl(x, A, group_sizes, group_to_weight, num_weights, y, workspace, workspace_bytes, m, k,
                  n, g, trans_rhs, dtype, cfg, stream, ReadyFlags{ready_flags, groups_per_flag, epoch});
}

int rd_ep_dispatch(const void* x, const int32_t* routing, int tokens, int top_k, int row_bytes,
                   int num_experts, int world, const int32_t* dest_offset, int32_t* fill,
                   const uint64_t* peer_base, int capacity_rows, int32_t* dest_pos, void* stream) {
  if (tokens < 0 || top_k <= 0 || row_bytes <= 0 || (row_bytes & 15) || world <= 0 ||
      num_experts <= 0 || num_experts % world != 0 || capacity_rows < 0)
    return RD_ERR_BAD_SHAPE;
  if (tokens == 0) return RD_OK;
  if (!aligned16(x) || !routing || !dest_offset || !fill || !peer_base || !dest_pos)
    return RD_ERR_BAD_POINTER;
  const long long entries = static_cast<long long>(tokens) * top_k;
  const int warps_per_block = rd::kEpThreads / 32;
  long long blocks = (entries + warps_per_block - 1) / warps_per_block;
  const int cap = sm_count() * 8;
  if (blocks > cap) blocks = cap;
  rd::ep_dispatch_kernel<<<static_cast<int>(blocks), rd::kEpThreads, 0,
                           static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(x), routing, tokens, top_k, row_bytes / 16, num_experts,
      num_experts / world, dest_offset, fill, peer_base, capacity_rows, dest_pos);
  return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
}

// Shared body of rd_tgmm / rd_tgmm_strided: `g` output blocks, block i contracting over the rows
// of groups i, i + g, ..., i + (seg_count - 1) * g of group_sizes (seg_count * g entries).
static int tgmm_impl(const void* x, const void* dout, const int32_t* group_sizes, void* out,
                     void* workspace, size_t workspace_bytes, int m, int k, int n, int g, int seg_count,
                     int dtype, const rd_tile_cfg* cfg, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (seg_count < 1 || (seg_count > 1 && g > 0 && seg_count > 0x7fffffff / g)) return RD_ERR_BAD_SHAPE;
  const int g_fine = g * seg_count;
  if (dtype != RD_DTYPE_F16 && dtype != RD_DTYPE_BF16 && dtype != RD_DTYPE_F32) return RD_ERR_BAD_DTYPE;
  const bool f32 = dtype == RD_DTYPE_F32;
  const int esize = f32 ? 4 : 2;
  const int amask = f32 ? 3 : 7;
  const int row_elems = 128 / esize;
  if (m < 0 || k < 0 || n < 0 || g < 0 || (k & amask) || (n & amask)) return RD_ERR_BAD_SHAPE;
  if (g == 0 || k == 0 || n == 0) return RD_OK;
  if (!aligned16(out)) return RD_ERR_BAD_POINTER;
  if (m == 0) {  // every group is empty
    cudaMemsetAsync(out, 0, static_cast<size_t>(g) * k * n * esize, stream);
    return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
  }
  if (!aligned16(x) || !aligned16(dout) || group_sizes == nullptr) return RD_ERR_BAD_POINTER;
  Workspace w;
  int rc = bind_workspace(workspace, workspace_bytes, m, g_fine, &w);
  if (rc != RD_OK) return rc;

  const int sms = sm_count();
  int bn = cfg && cfg->tile_n
               ? cfg->tile_n
               : choose_tile_n(static_cast<long long>((k + rd::kTileM - 1) / rd::kTileM) * g, n, sms);
  if (bn != 64 && bn != 128 && bn != 256) return RD_ERR_BAD_CONFIG;
  int cta_group = cfg ? cfg->cta_group : 0;
  int tile_m = cfg ? cfg->tile_m : 0;
  if (cta_group < 0 || cta_group > 2 || (cta_group == 2 && bn != 256)) return RD_ERR_BAD_CONFIG;
  if (tile_m != 0 && tile_m != 128 && tile_m != 256) return RD_ERR_BAD_CONFIG;
  if (tile_m == 256 && bn != 256) return RD_ERR_BAD_CONFIG;
  const bool three_pass = cfg && (cfg->flags & RD_CFG_F32_THREE_PASS);
  if (three_pass && !f32) return RD_ERR_BAD_CONFIG;
  if (f32) {  // the float32 kernels choose between one CTA and a pair themselves
    if (cta_group == 2 || tile_m == 256 || seg_count > 1) return RD_ERR_BAD_CONFIG;
    const bool pair = choose_f32_pair(true, m, k, n, g, bn, cfg);
    if (pair) bn = rd::kF32PairBN;
    cta_group = pair ? 2 : 1;
    tile_m = 128;
  }
  if (seg_count > 1) {  // strided segments: one CTA per tile
    if (cta_group == 2) return RD_ERR_BAD_CONFIG;
    cta_group = 1;
  }
  // 256 columns, plain: 128 rows per CTA, whatever tile height the caller names.
  const bool two_acc = !f32 && bn == 256 && seg_count == 1;
  const int ctas = pick_ctas(cfg);
  TgmmWay way = TgmmWay::kPlain;
  if (two_acc) {
    tile_m = 128;
    way = tgmm_way(m, k, n, g, ctas, cta_group);
    cta_group = way == TgmmWay::kPair ? 2 : 1;
  }
  if (cta_group == 0) cta_group = 1;
  if (tile_m == 0) tile_m = choose_two_half(true, m, k, n, g, bn) ? 256 : 128;
  const bool two_half = tile_m == 256;
  const int tile_rows = two_half ? rd::kG2TileRows : rd::kTileM * cta_group;
  const long long k_tiles = (k + tile_rows - 1) / tile_rows;

  const bool in_kernel = seg_count == 1 && inline_groups(m, g);
  if (in_kernel) {
    rc = ensure_context();
    if (rc != RD_OK) return rc;
  } else {
    launch_internal_metadata(group_sizes, nullptr, g_fine, m, rd::kTileM, w, stream);
    if (cudaGetLastError() != cudaSuccess) return RD_ERR_LAUNCH;
  }

  // 256-row tiles fetch each operand of a stage with one box when the 64-column blocks tile the
  // rows exactly (see rd_gemm2.cuh); otherwise one 2-D box per 64 columns.
  // The float32 kernels likewise, with blocks of 32 columns.
  const bool f32_pair = f32 && cta_group == 2;
  const bool blocked = f32 ? (k % 32 == 0 && n % 32 == 0)
                           : (two_half && k % 64 == 0 && n % 64 == 0);
  if (f32_pair && !three_pass && !blocked) return RD_ERR_BAD_CONFIG;  // choose_f32_pair does not ask for it
  CUtensorMap ta, tb;
  if (blocked && f32) {
    rc = encode_blocked_map(&ta, x, dtype, k, m, rd::kF32TileK, rd::kTileM / 32);
    if (rc != RD_OK) return rc;
    rc = encode_blocked_map(&tb, dout, dtype, n, m, rd::kF32TileK, bn / cta_group / 32);
    if (rc != RD_OK) return rc;
  } else if (blocked) {
    rc = encode_blocked_map(&ta, x, dtype, k, m, rd::kTileK, rd::kG2TileRows / 64);
    if (rc != RD_OK) return rc;
    rc = encode_blocked_map(&tb, dout, dtype, n, m, rd::kTileK, rd::kG2TileN / 64);
    if (rc != RD_OK) return rc;
  } else {
    {
      const uint64_t dims[2] = {static_cast<uint64_t>(k), static_cast<uint64_t>(m)};
      const uint32_t box[2] = {static_cast<uint32_t>(row_elems), static_cast<uint32_t>(row_elems)};
      rc = encode_map(&ta, x, dtype, 2, dims, box, /*atom32=*/f32);
      if (rc != RD_OK) return rc;
    }
    {
      const uint64_t dims[2] = {static_cast<uint64_t>(n), static_cast<uint64_t>(m)};
      const uint32_t box[2] = {static_cast<uint32_t>(row_elems), static_cast<uint32_t>(row_elems)};
      rc = encode_map(&tb, dout, dtype, 2, dims, box, /*atom32=*/f32);
      if (rc != RD_OK) return rc;
    }
  }

  CUtensorMap tout;
  {  // out[g, k, n] written as [32 rows][128 B] boxes of one group
    const uint64_t dims[3] = {static_cast<uint64_t>(n), static_cast<uint64_t>(k),
                              static_cast<uint64_t>(g)};
    const uint32_t box[3] = {static_cast<uint32_t>(row_elems), 32, 1};
    rc = encode_map(&tout, out, dtype, 3, dims, box);
    if (rc != RD_OK) return rc;
  }

  GemmArgs args = {};
  args.m = m; args.k = k; args.n = n; args.g = g;
  args.n_tiles = (n + bn - 1) / bn;
  args.k_tiles = static_cast<int>(k_tiles);
  args.seg_count = seg_count;
  args.seg_stride = g;
  args.blocked_maps = blocked ? 1 : 0;
  args.max_m_tiles = w.layout.max_tiles;
  args.ab_format = dtype;
  args.wait_limit_us = wait_limit_us(cfg);
  args.zero_tail = 0;
  args.inline_groups = in_kernel ? 1 : 0;
  args.group_sizes = group_sizes;
  args.group_offsets = w.group_offsets();
  args.tile_rec = w.tile_rec();
  args.totals = w.totals();
  args.status = w.status();
  args.out = out;

  if (f32_pair)
    return three_pass ? launch_gemm_f32_pair<false, true, true>(ta, tb, tout, args, ctas, stream)
                      : launch_gemm_f32_pair<false, true, false>(ta, tb, tout, args, ctas, stream);
  if (f32) {
    if (bn == 256) return launch_gemm_f32<256, false, true>(ta, tb, tout, args, ctas, stream);
    if (bn == 128) return launch_gemm_f32<128, false, true>(ta, tb, tout, args, ctas, stream);
    return launch_gemm_f32<64, false, true>(ta, tb, tout, args, ctas, stream);
  }
  if (two_half) return launch_gemm2<false, true, true>(ta, tb, tout, args, ctas, stream);  // strided segments
  if (seg_count > 1) {
    if (bn == 256) return launch_gemm<256, false, true, 1, true>(ta, tb, tout, args, ctas, stream);
    if (bn == 128) return launch_gemm<128, false, true, 1, true>(ta, tb, tout, args, ctas, stream);
    return launch_gemm<64, false, true, 1, true>(ta, tb, tout, args, ctas, stream);
  }
  if (two_acc) {
    args.turn_columns = way == TgmmWay::kTurned ? 1 : 0;
    switch (way) {
      case TgmmWay::kPair: return launch_tgmm<2>(x, dout, tout, dtype, args, ctas, stream);
      case TgmmWay::kPlain: return launch_gemm<256, false, true, 1>(ta, tb, tout, args, ctas, stream);
      case TgmmWay::kOneThread: return launch_gemm<256, false, true, 1, false, false, true>(ta, tb, tout, args, ctas, stream);
      default: return launch_tgmm<1>(x, dout, tout, dtype, args, ctas, stream);
    }
  }
  if (bn == 128) return launch_gemm<128, false, true, 1>(ta, tb, tout, args, ctas, stream);
  return launch_gemm<64, false, true, 1>(ta, tb, tout, args, ctas, stream);
}

int rd_tgmm(const void* x, const void* dout, const int32_t* group_sizes, void* out,
            void* workspace, size_t workspace_bytes, int m, int k, int n, int g, int dtype,
            const rd_tile_cfg* cfg, void* stream) {
  return tgmm_impl(x, dout, group_sizes, out, workspace, workspace_bytes, m, k, n, g, 1, dtype, cfg, stream);
}

int rd_tgmm_strided(const void* x, const void* dout, const int32_t* group_sizes, void* out,
                    void* workspace, size_t workspace_bytes, int m, int k, int n, int g, int seg_count,
                    int dtype, const rd_tile_cfg* cfg, void* stream) {
  return tgmm_impl(x, dout, group_sizes, out, workspace, workspace_bytes, m, k, n, g, seg_count, dtype, cfg,
                   stream);
}

// ------------------------------------------------------------------ rows that are not multiples of 16 bytes
namespace {

// Tiled map, 128-byte swizzle, over `mats` row-major 16-bit matrices [rows, cols] whose rows are
// `pitch` elements apart (a multiple of 8); zero fill outside.
int encode_pitched_map(CUtensorMap* map, const void* base, int dtype, int cols, int rows, int mats, int pitch,
                       uint32_t box_cols, uint32_t box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return RD_ERR_DRIVER;
  const cuuint64_t row_bytes = static_cast<cuuint64_t>(pitch) * 2;
  cuuint64_t gdims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(mats)};
  cuuint64_t gstrides[2] = {row_bytes, row_bytes * static_cast<cuuint64_t>(rows)};
  cuuint32_t gbox[3] = {box_cols, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r =
      fn(map, dtype == RD_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
         mats > 0 ? 3 : 2, const_cast<void*>(base), gdims, gstrides, gbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? RD_OK : RD_ERR_TENSOR_MAP;
}

bool tma_rows(const void* p, int cols) { return (cols & 7) == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
int padded_cols(int cols) { return (cols + 7) & ~7; }

// Copies whichever of the two matrices TMA cannot read into scratch, in one launch; the pointers
// returned are what the tensor maps start at.
int repitch_operands(const void** a, long long a_rows, int a_cols, const void** b, long long b_rows, int b_cols,
                     void* scratch, size_t scratch_bytes, cudaStream_t stream) {
  rd::Repitch ra = {}, rb = {};
  uint8_t* next = static_cast<uint8_t*>(scratch);
  size_t used = 0;
  auto plan = [&](rd::Repitch& r, const void** p, long long rows, int cols) {
    if (tma_rows(*p, cols)) return;
    r.src = static_cast<const uint16_t*>(*p);
    r.dst = reinterpret_cast<uint4*>(next + used);
    r.cols = cols;
    r.vecs_per_row = padded_cols(cols) / 8;
    r.vecs = rows * r.vecs_per_row;
    *p = r.dst;
    used += static_cast<size_t>(r.vecs) * 16;
  };
  plan(ra, a, a_rows, a_cols);
  plan(rb, b, b_rows, b_cols);
  if (used == 0) return RD_OK;
  if (!aligned16(scratch)) return RD_ERR_BAD_POINTER;
  if (used > scratch_bytes) return RD_ERR_WORKSPACE;
  const long long vecs = ra.vecs + rb.vecs;
  long long blocks = (vecs + rd::kGatherThreads - 1) / rd::kGatherThreads;
  const long long cap = static_cast<long long>(sm_count()) * 8;
  if (blocks > cap) blocks = cap;
  return launch_kernel(&rd::repitch_rows_kernel, static_cast<int>(blocks), rd::kGatherThreads, 0, 1, true, stream, ra,
                       rb);
}

bool aligned2(const void* p) { return p != nullptr && (reinterpret_cast<uintptr_t>(p) & 1u) == 0; }

}  // namespace

size_t rd_unaligned_scratch_bytes(long long a_rows, int a_cols, long long b_rows, int b_cols) {
  if (a_rows < 0 || a_cols < 0 || b_rows < 0 || b_cols < 0) return 0;
  return 2 * (static_cast<size_t>(a_rows) * padded_cols(a_cols) + static_cast<size_t>(b_rows) * padded_cols(b_cols));
}

int rd_gmm_unaligned(const void* x, const void* A, const int32_t* group_sizes, void* y, void* workspace,
                     size_t workspace_bytes, void* scratch, size_t scratch_bytes, int m, int k, int n, int g,
                     int trans_rhs, int dtype, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (dtype != RD_DTYPE_F16 && dtype != RD_DTYPE_BF16) return RD_ERR_BAD_DTYPE;
  if (m < 0 || k < 0 || n < 0 || g < 0) return RD_ERR_BAD_SHAPE;
  if (m == 0 || n == 0) return RD_OK;
  if (!aligned2(y)) return RD_ERR_BAD_POINTER;
  if (g == 0 || k == 0) {
    cudaMemsetAsync(y, 0, static_cast<size_t>(m) * n * 2, stream);
    return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
  }
  if (!inline_groups(m, g)) return RD_ERR_BAD_SHAPE;
  if (!aligned2(x) || !aligned2(A) || group_sizes == nullptr) return RD_ERR_BAD_POINTER;
  Workspace w;
  int rc = bind_workspace(workspace, workspace_bytes, m, g, &w);
  if (rc != RD_OK) return rc;
  rc = ensure_context();
  if (rc != RD_OK) return rc;
  const int a_cols = trans_rhs ? k : n, a_rows = trans_rhs ? n : k;
  rc = repitch_operands(&x, m, k, &A, static_cast<long long>(g) * a_rows, a_cols, scratch, scratch_bytes, stream);
  if (rc != RD_OK) return rc;
  const int bn = n <= 64 ? 64 : 128;
  CUtensorMap ta, tb;
  rc = encode_pitched_map(&ta, x, dtype, k, m, 0, padded_cols(k), 64, rd::kTileM);
  if (rc != RD_OK) return rc;
  rc = encode_pitched_map(&tb, A, dtype, a_cols, a_rows, g, padded_cols(a_cols), 64, trans_rhs ? bn : 64);
  if (rc != RD_OK) return rc;
  GemmArgs args = {};
  args.m = m; args.k = k; args.n = n; args.g = g;
  args.n_tiles = (n + bn - 1) / bn;
  args.max_m_tiles = w.layout.max_tiles;
  args.ab_format = dtype;
  args.wait_limit_us = wait_limit_us(nullptr);
  args.zero_tail = 1;
  args.inline_groups = 1;
  args.group_sizes = group_sizes;
  args.status = w.status();
  args.out = y;
  args.groups_per_flag = 1;
  const int ctas = sm_count();
  if (trans_rhs)
    return bn == 64 ? launch_gemm_unaligned<64, true, false>(ta, tb, args, ctas, stream)
                    : launch_gemm_unaligned<128, true, false>(ta, tb, args, ctas, stream);
  return bn == 64 ? launch_gemm_unaligned<64, false, false>(ta, tb, args, ctas, stream)
                  : launch_gemm_unaligned<128, false, false>(ta, tb, args, ctas, stream);
}

int rd_tgmm_unaligned(const void* x, const void* dout, const int32_t* group_sizes, void* out, void* workspace,
                      size_t workspace_bytes, void* scratch, size_t scratch_bytes, int m, int k, int n, int g,
                      int dtype, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (dtype != RD_DTYPE_F16 && dtype != RD_DTYPE_BF16) return RD_ERR_BAD_DTYPE;
  if (m < 0 || k < 0 || n < 0 || g < 0) return RD_ERR_BAD_SHAPE;
  if (g == 0 || k == 0 || n == 0) return RD_OK;
  if (!aligned2(out)) return RD_ERR_BAD_POINTER;
  if (m == 0) {
    cudaMemsetAsync(out, 0, static_cast<size_t>(g) * k * n * 2, stream);
    return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
  }
  if (!inline_groups(m, g)) return RD_ERR_BAD_SHAPE;
  if (!aligned2(x) || !aligned2(dout) || group_sizes == nullptr) return RD_ERR_BAD_POINTER;
  Workspace w;
  int rc = bind_workspace(workspace, workspace_bytes, m, g, &w);
  if (rc != RD_OK) return rc;
  rc = ensure_context();
  if (rc != RD_OK) return rc;
  rc = repitch_operands(&x, m, k, &dout, m, n, scratch, scratch_bytes, stream);
  if (rc != RD_OK) return rc;
  const int bn = n <= 64 ? 64 : 128;
  CUtensorMap ta, tb;
  rc = encode_pitched_map(&ta, x, dtype, k, m, 0, padded_cols(k), 64, rd::kTileK);
  if (rc != RD_OK) return rc;
  rc = encode_pitched_map(&tb, dout, dtype, n, m, 0, padded_cols(n), 64, rd::kTileK);
  if (rc != RD_OK) return rc;
  GemmArgs args = {};
  args.m = m; args.k = k; args.n = n; args.g = g;
  args.n_tiles = (n + bn - 1) / bn;
  args.k_tiles = (k + rd::kTileM - 1) / rd::kTileM;
  args.seg_count = 1;
  args.seg_stride = g;
  args.max_m_tiles = w.layout.max_tiles;
  args.ab_format = dtype;
  args.wait_limit_us = wait_limit_us(nullptr);
  args.inline_groups = 1;
  args.group_sizes = group_sizes;
  args.status = w.status();
  args.out = out;
  const int ctas = sm_count();
  return bn == 64 ? launch_gemm_unaligned<64, false, true>(ta, tb, args, ctas, stream)
                  : launch_gemm_unaligned<128, false, true>(ta, tb, args, ctas, stream);
}

int rd_gmm_permuted(const void* x, int x_rows, const int32_t* in_rows, const void* A, int num_weights,
                    const int32_t* group_sizes, const int32_t* group_to_weight, void* y, int y_rows,
                    const int32_t* out_rows, void* workspace, size_t workspace_bytes, int m, int k,
                    int n, int g, int trans_rhs, int dtype, const rd_tile_cfg* cfg, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (dtype != RD_DTYPE_F16 && dtype != RD_DTYPE_BF16) return RD_ERR_BAD_DTYPE;
  if (m < 0 || k < 0 || n < 0 || g < 0 || num_weights < 0 || x_rows < 0 || y_rows < 0 || (k & 7) ||
      (n & 7))
    return RD_ERR_BAD_SHAPE;
  if (in_rows == nullptr && x_rows < m) return RD_ERR_BAD_SHAPE;
  if (out_rows == nullptr && y_rows != m) return RD_ERR_BAD_SHAPE;
  if (m == 0 || n == 0 || y_rows == 0) return RD_OK;
  if (!aligned16(y)) return RD_ERR_BAD_POINTER;
  if (g == 0 || k == 0 || num_weights == 0 || x_rows == 0) {
    // Nothing contributes.  Without out_rows every row of y is a zero row; with out_rows the
    // rows that would have been written are not known without reading the indices, and the
    // call leaves y alone only if there is no group at all.
    if (out_rows == nullptr || g == 0) {
      if (out_rows == nullptr) cudaMemsetAsync(y, 0, static_cast<size_t>(m) * n * 2, stream);
      return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
    }
    return RD_ERR_BAD_SHAPE;
  }
  if (!aligned16(x) || !aligned16(A) || group_sizes == nullptr) return RD_ERR_BAD_POINTER;
  if (group_to_weight == nullptr && num_weights != g) return RD_ERR_BAD_SHAPE;
  Workspace w;
  int rc = bind_workspace(workspace, workspace_bytes, m, g, &w);
  if (rc != RD_OK) return rc;
  int bn = cfg && cfg->tile_n ? cfg->tile_n : choose_tile_n(0, n, 0);
  if (bn != 64 && bn != 128 && bn != 256) return RD_ERR_BAD_CONFIG;
  if (cfg && (cfg->cta_group == 2 || cfg->tile_m == 256 || (cfg->flags & RD_CFG_F32_THREE_PASS)))
    return RD_ERR_BAD_CONFIG;

  launch_internal_metadata(group_sizes, group_to_weight, g, m, rd::kTileM, w, stream);
  if (cudaGetLastError() != cudaSuccess) return RD_ERR_LAUNCH;

  CUtensorMap ta, tb, tout;
  rc = encode_rows_map(&ta, x, dtype, k, x_rows, rd::kTileM);
  if (rc != RD_OK) return rc;
  if (trans_rhs) {
    const uint64_t dims[3] = {static_cast<uint64_t>(k), static_cast<uint64_t>(n),
                              static_cast<uint64_t>(num_weights)};
    const uint32_t box[3] = {64, static_cast<uint32_t>(bn), 1};
    rc = encode_map(&tb, A, dtype, 3, dims, box);
  } else {
    const uint64_t dims[3] = {static_cast<uint64_t>(n), static_cast<uint64_t>(k),
                              static_cast<uint64_t>(num_weights)};
    const uint32_t box[3] = {64, 64, 1};
    rc = encode_map(&tb, A, dtype, 3, dims, box);
  }
  if (rc != RD_OK) return rc;
  {
    const uint64_t dims[2] = {static_cast<uint64_t>(n), static_cast<uint64_t>(y_rows)};
    const uint32_t box[2] = {64, 32};
    rc = encode_map(&tout, y, dtype, 2, dims, box);
    if (rc != RD_OK) return rc;
  }

  GemmArgs args = {};
  args.m = m; args.k = k; args.n = n; args.g = g;
  args.n_tiles = (n + bn - 1) / bn;
  args.k_tiles = 0;
  args.max_m_tiles = w.layout.max_tiles;
  args.ab_format = dtype;
  args.wait_limit_us = wait_limit_us(cfg);
  args.zero_tail = (cfg && (cfg->flags & RD_CFG_NO_ZERO_TAIL)) ? 0 : 1;
  args.group_sizes = group_sizes;
  args.group_offsets = w.group_offsets();
  args.tile_rec = w.tile_rec();
  args.totals = w.totals();
  args.status = w.status();
  args.out = y;
  rd::PermArgs perm;
  perm.a_rows = in_rows;
  perm.a_base = x;
  perm.a_rows_in = x_rows;
  perm.b_rows = nullptr;
  perm.b_base = nullptr;
  perm.b_rows_in = 0;
  perm.out_rows = out_rows;
  perm.out_rows_n = y_rows;

  const int ctas = pick_ctas(cfg);
  if (trans_rhs) {
    if (bn == 256) return launch_gemm_perm<256, true, false>(ta, tb, tout, args, perm, ctas, stream);
    if (bn == 128) return launch_gemm_perm<128, true, false>(ta, tb, tout, args, perm, ctas, stream);
    return launch_gemm_perm<64, true, false>(ta, tb, tout, args, perm, ctas, stream);
  }
  if (bn == 256) return launch_gemm_perm<256, false, false>(ta, tb, tout, args, perm, ctas, stream);
  if (bn == 128) return launch_gemm_perm<128, false, false>(ta, tb, tout, args, perm, ctas, stream);
  return launch_gemm_perm<64, false, false>(ta, tb, tout, args, perm, ctas, stream);
}

int rd_tgmm_permuted(const void* x, int x_rows, const int32_t* x_row_index, const void* dout,
                     int dout_rows, const int32_t* dout_row_index, const int32_t* group_sizes,
                     void* out, void* workspace, size_t workspace_bytes, int m, int k, int n, int g,
                     int dtype, const rd_tile_cfg* cfg, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (dtype != RD_DTYPE_F16 && dtype != RD_DTYPE_BF16) return RD_ERR_BAD_DTYPE;
  if (m < 0 || k < 0 || n < 0 || g < 0 || x_rows < 0 || dout_rows < 0 || (k & 7) || (n & 7))
    return RD_ERR_BAD_SHAPE;
  if ((x_row_index == nullptr && x_rows < m) || (dout_row_index == nullptr && dout_rows < m))
    return RD_ERR_BAD_SHAPE;
  if (g == 0 || k == 0 || n == 0) return RD_OK;
  if (!aligned16(out)) return RD_ERR_BAD_POINTER;
  if (m == 0 || x_rows == 0 || dout_rows == 0) {
    cudaMemsetAsync(out, 0, static_cast<size_t>(g) * k * n * 2, stream);
    return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
  }
  if (!aligned16(x) || !aligned16(dout) || group_sizes == nullptr) return RD_ERR_BAD_POINTER;
  Workspace w;
  int rc = bind_workspace(workspace, workspace_bytes, m, g, &w);
  if (rc != RD_OK) return rc;
  int bn = cfg && cfg->tile_n ? cfg->tile_n : choose_tile_n(0, n, 0);
  if (bn != 64 && bn != 128 && bn != 256) return RD_ERR_BAD_CONFIG;
  if (cfg && (cfg->cta_group == 2 || cfg->tile_m == 256 || (cfg->flags & RD_CFG_F32_THREE_PASS)))
    return RD_ERR_BAD_CONFIG;

  launch_internal_metadata(group_sizes, nullptr, g, m, rd::kTileM, w, stream);
  if (cudaGetLastError() != cudaSuccess) return RD_ERR_LAUNCH;

  CUtensorMap ta, tb, tout;
  rc = encode_rows_map(&ta, x, dtype, k, x_rows, 64);
  if (rc != RD_OK) return rc;
  rc = encode_rows_map(&tb, dout, dtype, n, dout_rows, 64);
  if (rc != RD_OK) return rc;
  {
    const uint64_t dims[3] = {static_cast<uint64_t>(n), static_cast<uint64_t>(k),
                              static_cast<uint64_t>(g)};
    const uint32_t box[3] = {64, 32, 1};
    rc = encode_map(&tout, out, dtype, 3, dims, box);
    if (rc != RD_OK) return rc;
  }

  GemmArgs args = {};
  args.m = m; args.k = k; args.n = n; args.g = g;
  args.n_tiles = (n + bn - 1) / bn;
  args.k_tiles = (k + rd::kTileM - 1) / rd::kTileM;
  args.max_m_tiles = w.layout.max_tiles;
  args.ab_format = dtype;
  args.wait_limit_us = wait_limit_us(cfg);
  args.zero_tail = 0;
  args.group_sizes = group_sizes;
  args.group_offsets = w.group_offsets();
  args.tile_rec = w.tile_rec();
  args.totals = w.totals();
  args.status = w.status();
  args.out = out;
  rd::PermArgs perm;
  perm.a_rows = x_row_index;
  perm.a_base = x;
  perm.a_rows_in = x_rows;
  perm.b_rows = dout_row_index;
  perm.b_base = dout;
  perm.b_rows_in = dout_rows;
  perm.out_rows = nullptr;
  perm.out_rows_n = 0;

  const int ctas = pick_ctas(cfg);
  if (bn == 256) return launch_gemm_perm<256, false, true>(ta, tb, tout, args, perm, ctas, stream);
  if (bn == 128) return launch_gemm_perm<128, false, true>(ta, tb, tout, args, perm, ctas, stream);
  return launch_gemm_perm<64, false, true>(ta, tb, tout, args, perm, ctas, stream);
}

int rd_gmm_ep_fused(const void* x, const void* A, int num_weights, const int32_t* group_sizes,
                    const int32_t* group_to_weight, void* y, void* workspace, size_t workspace_bytes,
                    int m, int k, int n, int g, int trans_rhs, int dtype, const rd_tile_cfg* cfg,
                    const int32_t* ready_flags, int groups_per_flag, int epoch, const rd_ep_send* send,
                    void* stream) {
  if (g > 0 && group_to_weight == nullptr) return RD_ERR_BAD_POINTER;
  if (ready_flags == nullptr || send == nullptr) return RD_ERR_BAD_POINTER;
  if (groups_per_flag <= 0 || send->world <= 0 || send->rank < 0 ||
      send->rank >= send->world || send->row_bytes <= 0 || (send->row_bytes & 15) || send->top_k <= 0 ||
      send->sender_ctas <= 0 || send->capacity_rows < 0)
    return RD_ERR_BAD_SHAPE;
  if (m == 0 || n == 0 || g == 0 || k == 0) return RD_ERR_BAD_SHAPE;  // the sender role needs a launch
  if (!aligned16(send->x_tokens) || !send->send_index || !send->send_start || !send->dest_pos ||
      !send->phase_done || !send->peer_base || !send->peer_flags)
    return RD_ERR_BAD_POINTER;
  rd::EpSendArgs a = {};
  a.x = static_cast<const uint8_t*>(send->x_tokens);
  a.send_index = send->send_index;
  a.send_start = send->send_start;
  a.dest_pos = send->dest_pos;
  a.phase_done = send->phase_done;
  a.peer_base = send->peer_base;
  a.peer_flags = send->peer_flags;
  a.row_bytes = send->row_bytes;
  a.top_k = send->top_k;
  a.world = send->world;
  a.rank = send->rank;
  a.capacity_rows = send->capacity_rows;
  a.sender_ctas = send->sender_ctas;
  return gmm_impl(x, A, group_sizes, group_to_weight, num_weights, y, workspace, workspace_bytes, m, k,
                  n, g, trans_rhs, dtype, cfg, stream, ReadyFlags{ready_flags, groups_per_flag, epoch}, &a);
}

int rd_ep_fused_forward(const rd_ep_step* st, const void* recv, const void* A, int num_weights,
                        const int32_t* group_to_weight, void* y, void* workspace, size_t workspace_bytes,
                        int capacity_rows, int k, int n, int dtype, const rd_tile_cfg* cfg,
                        const int32_t* ready_flags, const rd_ep_send* send, void* stream) {
  if (st == nullptr || send == nullptr) return RD_ERR_BAD_POINTER;
  const int world = send->world, rank = send->rank;
  if (world < 2 || st->tokens < 0 || st->top_k <= 0 || st->num_experts <= 0 || st->num_experts % world != 0)
    return RD_ERR_BAD_SHAPE;
  const int entries = st->tokens * st->top_k;
  const int local = st->num_experts / world;
  int rc = rd_ep_count_share(st->routing, entries, st->num_experts, st->counts_scratch, st->ticket, world,
                             rank, st->peer_counts, st->peer_count_flags, st->epoch, stream);
  if (rc != RD_OK) return rc;
  rc = rd_ep_plan_ring_when_counted(st->counts_all, st->count_flags, st->epoch, world, st->num_experts, rank,
                                    st->dest_offset, st->segment_sizes, st->fill, st->totals,
                                    send->phase_done, st->send_start, st->list_fill, st->plan_status,
                                    st->wait_limit_ms, stream);
  if (rc != RD_OK) return rc;
  rc = rd_ep_assign(st->routing, entries, st->num_experts, world, rank, st->dest_offset, st->fill,
                    capacity_rows, st->dest_pos, st->send_start, st->list_fill, st->send_index, stream);
  if (rc != RD_OK) return rc;
  rc = rd_ep_send_list(send->x_tokens, st->top_k, send->row_bytes, st->send_index, st->send_start, 0, world,
                       entries, st->dest_pos, st->own_buffer, capacity_rows, send->phase_done,
                       st->own_ready_flag, st->epoch, stream);
  if (rc != RD_OK) return rc;
  return rd_gmm_ep_fused(recv, A, num_weights, st->segment_sizes, group_to_weight, y, workspace,
                         workspace_bytes, capacity_rows, k, n, world * local, 0, dtype, cfg, ready_flags, local,
                         st->epoch, send, stream);
}

int rd_gmm_fp8(const void* x, const void* A, int num_weights, const int32_t* group_sizes,
               const int32_t* group_to_weight, const float* weight_scale, void* y, void* workspace,
               size_t workspace_bytes, int m, int k, int n, int g, const rd_tile_cfg* cfg, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  // rows of k one-byte elements and of n two-byte results must be multiples of 16 bytes
  if (m < 0 || k < 0 || n < 0 || g < 0 || num_weights < 0 || (k & 15) || (n & 7)) return RD_ERR_BAD_SHAPE;
  if (group_to_weight == nullptr && num_weights != g) return RD_ERR_BAD_SHAPE;
  if (m == 0 || n == 0) return RD_OK;
  if (!aligned16(y)) return RD_ERR_BAD_POINTER;
  if (g == 0 || k == 0 || num_weights == 0) {
    cudaMemsetAsync(y, 0, static_cast<size_t>(m) * n * 2, stream);
    return cudaGetLastError() == cudaSuccess ? RD_OK : RD_ERR_LAUNCH;
  }
  if (!aligned16(x) || !aligned16(A) || group_sizes == nullptr) return RD_ERR_BAD_POINTER;
  Workspace w;
  int rc = bind_workspace(workspace, workspace_bytes, m, g, &w);
  if (rc != RD_OK) return rc;
  int bn = cfg && cfg->tile_n ? cfg->tile_n : choose_tile_n(0, n, 0);
  if (bn != 64 && bn != 128 && bn != 256) return RD_ERR_BAD_CONFIG;
  if (cfg && (cfg->cta_group == 2 || cfg->tile_m == 256)) return RD_ERR_BAD_CONFIG;  // the library chooses
  if (cfg && (cfg->flags & RD_CFG_F32_THREE_PASS)) return RD_ERR_BAD_CONFIG;
  const bool two_half = !(cfg && cfg->tile_m == 128) && choose_two_half(false, m, k, n, g, bn, true);

  const bool by_weight = cfg != nullptr && (cfg->flags & RD_CFG_GROUP_BY_WEIGHT) != 0;
  const bool in_kernel = inline_groups(m, g) && !(by_weight && group_to_weight != nullptr);
  const long long split_tiles = split_tiles_bound(m, g, n);
  const int split = in_kernel && !two_half && split_allowed(cfg)
                        ? choose_split<true, true>(split_tiles, split_tile_rows(m, g), (k / 2 + rd::kTileK - 1) / rd::kTileK)
                        : 1;
  if (split > 1) bn = rd::kSplitBN;
  if (in_kernel) {
    rc = ensure_context();
    if (rc != RD_OK) return rc;
  } else {
    launch_internal_metadata(group_sizes, group_to_weight, g, m, two_half ? rd::kG2TileRows : rd::kTileM, w, stream,
                             by_weight);
    if (cudaGetLastError() != cudaSuccess) return RD_ERR_LAUNCH;
  }

  if (in_kernel && split == 1 && split_allowed(cfg) &&
      choose_swap(m, (k / 2 + rd::kTileK - 1) / rd::kTileK, n, g, true, true)) {
    GemmArgs args = {};
    args.m = m; args.k = k / 2; args.n = n; args.g = g;
    args.max_m_tiles = w.layout.max_tiles;
    args.ab_format = RD_DTYPE_BF16;
    args.wait_limit_us = wait_limit_us(cfg);
    args.weight_scale = weight_scale;
    args.zero_tail = (cfg && (cfg->flags & RD_CFG_NO_ZERO_TAIL)) ? 0 : 1;
    args.inline_groups = 1;
    args.group_to_weight = group_to_weight;
    args.group_sizes = group_sizes;
    args.status = w.status();
    args.out = y;
    return launch_gemm_swap<true, true>(x, A, y, RD_DTYPE_BF16, num_weights, args, stream);
  }

  // Both operands are K-major, so a row of k one-byte elements is described to TMA as k/2
  // two-byte elements: the bytes that land in shared memory are the same.
  const int k2 = k / 2;
  CUtensorMap ta, tb, tout;
  {
    const uint64_t dims[2] = {static_cast<uint64_t>(k2), static_cast<uint64_t>(m)};
    const uint32_t box[2] = {64, rd::kTileM};
    rc = encode_map(&ta, x, RD_DTYPE_BF16, 2, dims, box);
    if (rc != RD_OK) return rc;
  }
  {
    const uint64_t dims[3] = {static_cast<uint64_t>(k2), static_cast<uint64_t>(n),
                              static_cast<uint64_t>(num_weights)};
    const uint32_t box[3] = {64, static_cast<uint32_t>(bn), 1};
    rc = encode_map(&tb, A, RD_DTYPE_BF16, 3, dims, box);
    if (rc != RD_OK) return rc;
  }
  {
    const uint64_t dims[2] = {static_cast<uint64_t>(n), static_cast<uint64_t>(m)};
    const uint32_t box[2] = {64, 32};
    rc = encode_map(&tout, y, RD_DTYPE_BF16, 2, dims, box);
    if (rc != RD_OK) return rc;
  }
  GemmArgs args = {};
  args.m = m; args.k = k2; args.n = n; args.g = g;
  args.n_tiles = (n + bn - 1) / bn;
  args.max_m_tiles = w.layout.max_tiles;
  args.ab_format = RD_DTYPE_BF16;  // type of the output
  args.wait_limit_us = wait_limit_us(cfg);
  args.weight_scale = weight_scale;
  args.zero_tail = (cfg && (cfg->flags & RD_CFG_NO_ZERO_TAIL)) ? 0 : 1;
  args.group_sizes = group_sizes;
  args.group_offsets = w.group_offsets();
  args.tile_rec = w.tile_rec();
  args.totals = w.totals();
  args.status = w.status();
  args.out = y;
  args.groups_per_flag = 1;
  args.inline_groups = in_kernel ? 1 : 0;
  args.group_to_weight = group_to_weight;
  const int ctas = pick_ctas(cfg);
  if (split > 1) return launch_gemm_splitk<true, true>(ta, tb, args, split, static_cast<int>(split_tiles), stream);
  if (two_half) return launch_gemm2_fp8(ta, tb, tout, args, ctas, stream);
  if (bn == 256) return launch_gemm<256, true, false, 1, false, true>(ta, tb, tout, args, ctas, stream);
  if (bn == 128) return launch_gemm<128, true, false, 1, false, true>(ta, tb, tout, args, ctas, stream);
  return launch_gemm<64, true, false, 1, false, true>(ta, tb, tout, args, ctas, stream);
}

int rd_device_status(const void* workspace, void* stream) {
  if (workspace == nullptr) return RD_ERR_BAD_POINTER;
  int32_t word = 0;
  cudaError_t e = cudaMemcpyAsync(&word, workspace, sizeof(word), cudaMemcpyDeviceToHost,
                                  static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return RD_ERR_LAUNCH;
  e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return RD_ERR_LAUNCH;
  return word == 0 ? RD_OK : RD_ERR_DEVICE_WAIT;
}

}  // extern "C"

// ------------------------------------------------------------------ entry point that allocates nothing
//
// Some hosts of this library can neither hand over a workspace nor create one: an operator slot
// whose argument list is frozen to "inputs and outputs" (a legacy custom-call interface, a
// plugin ABI defined by someone else), running inside a framework that has reserved the whole
// device for its own allocator -- there a cudaMalloc from inside the call may fail, and where it
// succeeds it synchronises the device and stalls every stream.  For them rd_gmm_static_scratch
// keeps the group-metadata scratch in a fixed array inside this library's device image.
//
// The array costs kStaticScratchBytes (64 KiB) on every GPU that loads the library, until the
// process exits.  It is one array per device, shared by every call: it still holds whatever the
// previous call left there, so the header words the kernels accumulate into are cleared at the
// start of each call, and two calls that overlap on the GPU (different streams, no ordering
// between them) race on it -- serialise them, or use rd_gmm with separate workspaces.
namespace {

constexpr size_t kStaticScratchWords = 16384;
constexpr size_t kStaticScratchBytes = kStaticScratchWords * sizeof(int32_t);

static __device__ __align__(256) int32_t g_static_scratch[kStaticScratchWords];

// In host code `g_static_scratch` is only a handle for the runtime, not a device address; the
// address a kernel can use has to be asked for, per device, with that device current.
int static_scratch_address(int32_t** out) {
  static std::mutex mu;
  static int32_t* per_device[64] = {nullptr};
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return RD_ERR_SCRATCH_SETUP;
  std::lock_guard<std::mutex> lock(mu);
  if (per_device[dev] == nullptr) {
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (e != cudaSuccess || ptr == nullptr) {
      fprintf(stderr, "ragged_dot_b200: cudaGetSymbolAddress(scratch) failed on device %d: %s\n", dev,
              cudaGetErrorString(e));
      return RD_ERR_SCRATCH_SETUP;
    }
    per_device[dev] = static_cast<int32_t*>(ptr);
  }
  *out = per_device[dev];
  return RD_OK;
}

}  // namespace

extern "C" int rd_gmm_static_scratch(const void* x, const void* A, const int32_t* group_sizes,
                                     void* y, int m, int k, int n, int g, int trans_rhs, int dtype,
                                     const rd_tile_cfg* cfg, void* stream) {
  if (m < 0 || g < 0) return RD_ERR_BAD_SHAPE;
  WorkspaceLayout layout;
  layout.g = g;
  layout.max_tiles = max_row_tiles(m, g);
  if (static_cast<size_t>(layout.total_words()) > kStaticScratchWords) return RD_ERR_TOO_LARGE;
  int32_t* scratch = nullptr;
  int rc = static_scratch_address(&scratch);
  if (rc != RD_OK) return rc;
  // The array keeps the last call's contents: start this call's status and totals from zero.
  if (cudaMemsetAsync(scratch, 0, 8 * sizeof(int32_t), static_cast<cudaStream_t>(stream)) !=
      cudaSuccess)
    return RD_ERR_LAUNCH;
  return rd_gmm(x, A, group_sizes, y, scratch, kStaticScratchBytes, m, k, n, g, trans_rhs, dtype, cfg,
                stream);
}
