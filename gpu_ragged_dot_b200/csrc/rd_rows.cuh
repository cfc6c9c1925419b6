// Row movement on either side of the grouped GEMMs in an MoE layer, all of it HBM traffic:
//   gather_rows_kernel          dst[i, :] = src[index[i], :] (tokens replicated per routed expert and
//                               sorted by expert).  One warp per output row, 16-byte vectors, four
//                               loads in flight per lane.
//   sum_rows_kernel             dst[t, :] = sum of the src rows whose index is t (the gradient of that
//                               gather), from per-row lists built by three small kernels
//   zero_unwritten_rows_kernel  clears the rows of a scatter's result that no source row names
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "rd_ptx.cuh"

namespace rd {

constexpr int kGatherThreads = 256;

__global__ void __launch_bounds__(kGatherThreads)
gather_rows_kernel(const uint4* __restrict__ src, const int32_t* __restrict__ index,
                   uint4* __restrict__ dst, int rows_out, int rows_in, int vecs_per_row, bool clamp) {
  const int lane = threadIdx.x & 31;
  const int warps_per_block = kGatherThreads / 32;
  const int warp_global = blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const int warp_stride = gridDim.x * warps_per_block;
  for (int r = warp_global; r < rows_out; r += warp_stride) {
    int s = index[r];
    if (clamp) s = s < 0 ? 0 : (s < rows_in ? s : rows_in - 1);
    uint4* d = dst + static_cast<size_t>(r) * vecs_per_row;
    if (s < 0 || s >= rows_in) {  // an index outside the source gives a zero row
      for (int v = lane; v < vecs_per_row; v += 32) d[v] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    const uint4* p = src + static_cast<size_t>(s) * vecs_per_row;
    int v = lane;
    for (; v + 96 < vecs_per_row; v += 128) {
      const uint4 a = p[v], b = p[v + 32], c = p[v + 64], e = p[v + 96];
      d[v] = a;
      d[v + 32] = b;
      d[v + 64] = c;
      d[v + 96] = e;
    }
    for (; v < vecs_per_row; v += 32) d[v] = p[v];
  }
}

// ------------------------------------------------------------------ rows with another pitch
// Two 16-bit matrices, rows packed, copied to rows of `pitch` elements (a multiple of 8) so that TMA can
// read them: both operands of a product in one launch.  What lies past `cols` in a row is written
// as zeros and never read (the maps end at cols).  `vecs` = 16-byte vectors in all rows; a matrix
// that needs no copy has none.  2.5 us at the sizes below a few MB, where torch's pad of two operands
// took four launches and 6 us of device time (20 us of the host's); larger ones are bound by the
// 2-byte loads (neighbours share lines in L1).
struct Repitch {
  const uint16_t* src;
  uint4* dst;
  int cols;
  int vecs_per_row;
  long long vecs;
};

__global__ void __launch_bounds__(kGatherThreads)
repitch_rows_kernel(const Repitch a, const Repitch b) {
  pdl_wait();  // launched early, as the product that follows it
  pdl_release();
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < a.vecs + b.vecs; i += stride) {
    const bool second = i >= a.vecs;
    const Repitch& m = second ? b : a;
    const long long v = second ? i - a.vecs : i;
    const long long row = v / m.vecs_per_row;
    const int c = static_cast<int>(v - row * m.vecs_per_row) * 8;
    const uint16_t* src = m.src + row * m.cols + c;
    uint16_t h[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) h[j] = c + j < m.cols ? src[j] : 0;
    m.dst[v] = *reinterpret_cast<const uint4*>(h);
  }
}

// ------------------------------------------------------------------ sum of rows by index
// The sum reads every source row once and writes every output row once, in order, where adding
// each source row into a float32 buffer with atomics moved about six times as much (the buffer is
// cleared, added to, read, and the rows are converted to float32 first).
// The lists: rank[i] = how many rows of the same index were counted before row i, start[t] = where
// t's list begins (the lists lie in whatever order the warps reach the cursor), list[start[t] +
// rank[i]] = i.  Only the first `live` = min(sum of group_sizes, rows_in) rows are counted; the
// others are zero rows.

__device__ __forceinline__ int clamp_index(int i, int rows) { return i < 0 ? 0 : (i < rows ? i : rows - 1); }

// min(sum of the non-negative group sizes, m), the same in every thread of the block.
__device__ __forceinline__ int live_rows(const int32_t* __restrict__ group_sizes, int g, int m) {
  __shared__ int total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  int sum = 0;
  for (int i = threadIdx.x; i < g; i += blockDim.x) sum += group_sizes[i] > 0 ? group_sizes[i] : 0;
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d);
  if ((threadIdx.x & 31) == 0 && sum != 0) atomicAdd(&total, sum);
  __syncthreads();
  return total < m ? total : m;
}

__global__ void __launch_bounds__(kGatherThreads)
sum_rows_count_kernel(const int32_t* __restrict__ index, int rows_in, int rows_out,
                      const int32_t* __restrict__ group_sizes, int g, int32_t* __restrict__ count,
                      int32_t* __restrict__ rank) {
  const int live = live_rows(group_sizes, g, rows_in);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < rows_in) rank[i] = i < live ? atomicAdd(&count[clamp_index(index[i], rows_out)], 1) : -1;
}

__global__ void __launch_bounds__(kGatherThreads)
sum_rows_start_kernel(const int32_t* __restrict__ count, int rows_out, int32_t* __restrict__ start,
                      int32_t* __restrict__ cursor) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = t < rows_out ? count[t] : 0;
  int inc = c;
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += v;
  }
  int base = 0;
  if (lane == 31) base = atomicAdd(cursor, inc);
  base = __shfl_sync(0xffffffffu, base, 31);
  if (t < rows_out) start[t] = base + inc - c;
}

__global__ void __launch_bounds__(kGatherThreads)
sum_rows_fill_kernel(const int32_t* __restrict__ index, int rows_in, int rows_out,
                     const int32_t* __restrict__ start, const int32_t* __restrict__ rank,
                     int32_t* __restrict__ list) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < rows_in && rank[i] >= 0) list[start[clamp_index(index[i], rows_out)] + rank[i]] = i;
}

// Element codes of the C ABI: 0 = fp16, 1 = bf16, 2 = float32.  V elements per access: 16 bytes, or
// one element where rows are not multiples of 16 bytes.
template <int kType, int V>
struct RowVec {
  static constexpr int kBytes = (kType == 2 ? 4 : 2) * V;
  static __device__ __forceinline__ void add(float (&acc)[V], const uint8_t* src) {
    if constexpr (kType == 2) {
      float f[V];
      if constexpr (V == 4) {
        const float4 q = *reinterpret_cast<const float4*>(src);
        f[0] = q.x; f[1] = q.y; f[2] = q.z; f[3] = q.w;
      } else {
        f[0] = *reinterpret_cast<const float*>(src);
      }
#pragma unroll
      for (int j = 0; j < V; ++j) acc[j] += f[j];
    } else {
      uint16_t h[V];
      if constexpr (V == 8) {
        *reinterpret_cast<uint4*>(h) = *reinterpret_cast<const uint4*>(src);
      } else {
        h[0] = *reinterpret_cast<const uint16_t*>(src);
      }
#pragma unroll
      for (int j = 0; j < V; ++j)
        acc[j] += kType == 1 ? __uint_as_float(static_cast<uint32_t>(h[j]) << 16)
                             : __half2float(__ushort_as_half(h[j]));
    }
  }
  static __device__ __forceinline__ void store(const float (&acc)[V], uint8_t* dst) {
    if constexpr (kType == 2) {
      if constexpr (V == 4) {
        *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1], acc[2], acc[3]);
      } else {
        *reinterpret_cast<float*>(dst) = acc[0];
      }
    } else {
      uint16_t h[V];
#pragma unroll
      for (int j = 0; j < V; ++j)
        h[j] = kType == 1 ? __bfloat16_as_ushort(__float2bfloat16_rn(acc[j])) : __half_as_ushort(__float2half_rn(acc[j]));
      if constexpr (V == 8) {
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(h);
      } else {
        *reinterpret_cast<uint16_t*>(dst) = h[0];
      }
    }
  }
};

// One warp per (output row, 128 vectors of it).  Source rows are added in ascending order of their index, so
// that results do not depend on the order the lists were built in: up to 32 are ranked in registers,
// a longer list is gone through in windows of 4096 indices, marked in a bitmap and read off in order (each
// window reads the list once more; a list spans rows_in / 4096 windows at most).
// Bound by HBM: bf16, 8192 rows of 4096 into 4096 in 30 us (100 MB), 41 us with the three list kernels,
// where zeroing, converting, index_add and converting back took 350 us.
constexpr int kSumWindow = 4096;

template <int kType, int V>
__global__ void __launch_bounds__(kGatherThreads)
sum_rows_kernel(const uint8_t* __restrict__ src, const int32_t* __restrict__ list,
                const int32_t* __restrict__ start, const int32_t* __restrict__ count,
                uint8_t* __restrict__ dst, int rows_out, int vecs_per_row, int chunks) {
  using R = RowVec<kType, V>;
  constexpr int kPer = 4;  // vectors per lane
  __shared__ uint32_t window[kGatherThreads / 32][kSumWindow / 32];
  const int lane = threadIdx.x & 31;
  uint32_t* marks = window[threadIdx.x >> 5];
  const long long warp = (static_cast<long long>(blockIdx.x) * kGatherThreads + threadIdx.x) >> 5;
  const long long warps = static_cast<long long>(gridDim.x) * (kGatherThreads / 32);
  const size_t row_bytes = static_cast<size_t>(vecs_per_row) * R::kBytes;
  for (long long w = warp; w < static_cast<long long>(rows_out) * chunks; w += warps) {
    const int t = static_cast<int>(w / chunks);
    const int v0 = static_cast<int>(w - static_cast<long long>(t) * chunks) * 32 * kPer + lane;
    const int n = count[t];
    const int32_t* my = list + start[t];
    float acc[kPer][V];
#pragma unroll
    for (int i = 0; i < kPer; ++i)
#pragma unroll
      for (int j = 0; j < V; ++j) acc[i][j] = 0.0f;
    auto add_row = [&](int row) {
      const uint8_t* p = src + static_cast<size_t>(row) * row_bytes;
#pragma unroll
      for (int i = 0; i < kPer; ++i)
        if (v0 + 32 * i < vecs_per_row) R::add(acc[i], p + static_cast<size_t>(v0 + 32 * i) * R::kBytes);
    };
    if (n <= 32) {
      const int mine = lane < n ? my[lane] : 0x7fffffff;
      int rank = 0;
      for (int j = 0; j < n; ++j) rank += __shfl_sync(0xffffffffu, mine, j) < mine ? 1 : 0;
      if (lane >= n) rank = -1;
#pragma unroll 2
      for (int j = 0; j < n; ++j) {
        const int from = __ffs(__ballot_sync(0xffffffffu, rank == j)) - 1;
        add_row(__shfl_sync(0xffffffffu, mine, from));
      }
    } else {
      int lo = 0x7fffffff, hi = 0;
      for (int i = lane; i < n; i += 32) {
        lo = min(lo, my[i]);
        hi = max(hi, my[i]);
      }
      const int last = __reduce_max_sync(0xffffffffu, hi) / kSumWindow;
      for (int win = __reduce_min_sync(0xffffffffu, lo) / kSumWindow; win <= last; ++win) {
        const int first = win * kSumWindow;
        for (int i = lane; i < kSumWindow / 32; i += 32) marks[i] = 0u;
        __syncwarp();
        for (int i = lane; i < n; i += 32) {
          const unsigned e = static_cast<unsigned>(my[i] - first);
          if (e < kSumWindow) atomicOr(&marks[e >> 5], 1u << (e & 31));
        }
        __syncwarp();
        for (int b = 0; b < kSumWindow / 32; b += 32) {
          const uint32_t word = marks[b + lane];
          for (uint32_t some = __ballot_sync(0xffffffffu, word != 0u); some != 0u; some &= some - 1) {
            const int from = __ffs(some) - 1;
            const int row0 = first + (b + from) * 32;
            uint32_t bits = __shfl_sync(0xffffffffu, word, from);
            for (; (bits & (bits - 1)) != 0u;) {  // two rows' loads in flight
              const int r0 = row0 + __ffs(bits) - 1;
              bits &= bits - 1;
              const int r1 = row0 + __ffs(bits) - 1;
              bits &= bits - 1;
              add_row(r0);
              add_row(r1);
            }
            if (bits != 0u) add_row(row0 + __ffs(bits) - 1);
          }
        }
        __syncwarp();
      }
    }
    uint8_t* d = dst + static_cast<size_t>(t) * row_bytes;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      if (v0 + 32 * i < vecs_per_row) R::store(acc[i], d + static_cast<size_t>(v0 + 32 * i) * R::kBytes);
  }
}

// ------------------------------------------------------------------ rows a scatter leaves unwritten
// Marking the rows that are written and clearing the others: 19 us with its launches, in a row, at 8192 rows of
// 14336 (235 MB, none left over), where clearing all of y first takes 68 us; below 48 MB that is the cheaper way.
__global__ void __launch_bounds__(kGatherThreads)
mark_rows_kernel(const int32_t* __restrict__ out_rows, int m, int y_rows,
                 const int32_t* __restrict__ group_sizes, int g, int32_t* __restrict__ marked) {
  const int live = live_rows(group_sizes, g, m);
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= live) return;
  const int t = out_rows[r];
  if (t >= 0 && t < y_rows) marked[t] = 1;
}

__global__ void __launch_bounds__(kGatherThreads)
zero_unwritten_rows_kernel(const int32_t* __restrict__ marked, uint4* __restrict__ y, int y_rows,
                           int vecs_per_row) {
  const int lane = threadIdx.x & 31;
  const int warps_per_block = kGatherThreads / 32;
  for (int r = blockIdx.x * warps_per_block + (threadIdx.x >> 5); r < y_rows; r += gridDim.x * warps_per_block) {
    if (marked[r]) continue;
    uint4* d = y + static_cast<size_t>(r) * vecs_per_row;
    for (int v = lane; v < vecs_per_row; v += 32) d[v] = make_uint4(0u, 0u, 0u, 0u);
  }
}

}  // namespace rd
