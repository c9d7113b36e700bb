// Stable LSD radix sort of point rows by grid cell.
//
// The J^T J column gather needs, for every cell, the point rows that fall in
// it in ascending row order (the reference accumulates each J^T J entry in
// ascending row order, src/solvers/lm_solver.cpp:113-172). Rows arrive in
// row order, so a stable sort on the cell key alone gives that order.
// Digits of up to 9 bits, as few passes as they allow; per pass: a per-tile
// digit histogram, an exclusive scan of each digit's row of it (KDigitScan), and a
// stable scatter that adds the digits' starts and ranks equal digits inside a
// warp with __match_any_sync and across warps with shared counters. The first
// pass reads the rows' cells, so no keys are written beforehand.
#include <cuda_runtime.h>

#include "device.cuh"

namespace sdfgpu {

constexpr int kSortThreads = 256;
constexpr int kSortMaxBins = 512;
/// Keys per thread of a pass: 8 once such tiles fill the 148 SMs, else 2 (the
/// keys of a thread are ranked one after the other: a pass over 10,000 rows
/// took 6 us with 8).
constexpr int kSortItems = 8;
constexpr int kSortFewItems = 2;
/// Bits of the keys (the cells and the sentinel), passes over them.
int CellSortBits(int64_t num_cells) {
  int bits = 1;
  while ((int64_t{1} << bits) <= num_cells) {
    ++bits;
  }
  return bits;
}
int CellSortPasses(int64_t num_cells) { return (CellSortBits(num_cells) + 8) / 9; }
int SortItems(int64_t n) { return n >= int64_t{148} * kSortThreads * kSortItems ? kSortItems : kSortFewItems; }

/// Key i of a pass: a row's cell (rows outside the grid get the sentinel) in
/// the first one.
template <bool kFirst>
__device__ __forceinline__ int32_t SortKey(const int32_t* keys, int64_t i, int32_t sentinel) {
  const int32_t c = keys[i];
  return kFirst && c < 0 ? sentinel : c;
}

template <bool kFirst, int kItems>
__global__ void KRadixHist(const int32_t* keys, int64_t n, int32_t sentinel, int shift, int bins, int32_t* hist,
                           int num_tiles) {
  __shared__ int32_t h[kSortMaxBins];
  for (int d = threadIdx.x; d < bins; d += kSortThreads) {
    h[d] = 0;
  }
  __syncthreads();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * (kSortThreads * kItems);
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int64_t idx = base + q * kSortThreads + threadIdx.x;
    if (idx < n) {
      atomicAdd(&h[(static_cast<uint32_t>(SortKey<kFirst>(keys, idx, sentinel)) >> shift) & (bins - 1u)], 1);
    }
  }
  __syncthreads();
  for (int d = threadIdx.x; d < bins; d += kSortThreads) {
    hist[static_cast<int64_t>(d) * num_tiles + blockIdx.x] = h[d];
  }
}

/// Exclusive scan, in place, of each digit's row hist[digit * tiles ..] over
/// the tiles, a warp per digit, four loads in flight; the rows' totals behind
/// the table. (One block for the whole table took 44 us a pass for the 1.1
/// million rows of a 910-pose office, 67 for 32 instances.)
__global__ void __launch_bounds__(256) KDigitScan(int32_t* hist, int bins, int tiles) {
  constexpr int kLoads = 4;
  const int lane = threadIdx.x & 31;
  const int digit = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (digit >= bins) {
    return;
  }
  int32_t* row = hist + static_cast<int64_t>(digit) * tiles;
  int32_t carry = 0;
  for (int c0 = 0; c0 < tiles; c0 += 32 * kLoads) {
    int32_t v[kLoads];
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int t = c0 + 32 * i + lane;
      v[i] = t < tiles ? row[t] : 0;
    }
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int t = c0 + 32 * i + lane;
      int32_t x = v[i];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) {
          x += y;
        }
      }
      if (t < tiles) {
        row[t] = carry + x - v[i];
      }
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
  }
  if (lane == 0) {
    hist[static_cast<int64_t>(bins) * tiles + digit] = carry;
  }
}

template <bool kFirst, int kItems>
__global__ void __launch_bounds__(kSortThreads) KRadixScatter(const int32_t* keys_in, const int32_t* vals_in,
                                                              int64_t n, int32_t sentinel, int shift, int bins,
                                                              const int32_t* offsets, int num_tiles,
                                                              int32_t* keys_out, int32_t* vals_out) {
  constexpr int kWarps = kSortThreads / 32;
  constexpr int kOwn = kSortMaxBins / kSortThreads;
  __shared__ int32_t wcount[kWarps][kSortMaxBins];
  __shared__ int32_t warp_sum[kWarps];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  for (int d = lane; d < bins; d += 32) {
    wcount[warp][d] = 0;
  }
  // where each digit's keys of this tile start: thread t owns the digits
  // kOwn t ..
  int32_t own[kOwn];
  int32_t at[kOwn];
  int32_t sum = 0;
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    const int d = kOwn * threadIdx.x + i;
    own[i] = d < bins ? offsets[static_cast<int64_t>(bins) * num_tiles + d] : 0;
    at[i] = d < bins ? offsets[static_cast<int64_t>(d) * num_tiles + blockIdx.x] : 0;
    sum += own[i];
  }
  int32_t before_me = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, before_me, d);
    if (lane >= d) {
      before_me += y;
    }
  }
  if (lane == 31) {
    warp_sum[warp] = before_me;
  }
  before_me -= sum;
  __syncwarp();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * (kSortThreads * kItems) + static_cast<int64_t>(warp) * (32 * kItems);
  int rank[kItems];
  int digit[kItems];
  int32_t key[kItems];
  int32_t val[kItems];
  const unsigned lt_mask = (1u << lane) - 1u;
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int64_t idx = base + q * 32 + lane;
    const bool ok = idx < n;
    key[q] = ok ? SortKey<kFirst>(keys_in, idx, sentinel) : 0;
    val[q] = !ok ? 0 : kFirst ? static_cast<int32_t>(idx) : vals_in[idx];
    const int d = ok ? static_cast<int>((static_cast<uint32_t>(key[q]) >> shift) & (bins - 1u)) : kSortMaxBins + lane;
    digit[q] = d;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const int leader = __ffs(peers) - 1;
    int before = 0;
    if (ok) {
      before = wcount[warp][d];
    }
    __syncwarp();
    rank[q] = before + __popc(peers & lt_mask);
    if (ok && lane == leader) {
      wcount[warp][d] = before + __popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();
  for (int w = 0; w < warp; ++w) {
    before_me += warp_sum[w];
  }
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    const int d = kOwn * threadIdx.x + i;
    int running = before_me + at[i];
    before_me += own[i];
    if (d < bins) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const int c = wcount[w][d];
        wcount[w][d] = running;
        running += c;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int64_t idx = base + q * 32 + lane;
    if (idx < n) {
      const int d = digit[q];
      const int pos = wcount[warp][d] + rank[q];
      keys_out[pos] = key[q];
      vals_out[pos] = val[q];
    }
  }
}

namespace {

template <int kItems>
int CellSort(const int32_t* pt_cell, int64_t n, int64_t num_cells, int32_t* keys_a, int32_t* vals_a, int32_t* keys_b,
             int32_t* vals_b, int32_t* hist, cudaStream_t stream) {
  const int tiles = static_cast<int>((n + kSortThreads * kItems - 1) / (kSortThreads * kItems));
  const auto sentinel = static_cast<int32_t>(num_cells);
  const int passes = CellSortPasses(num_cells);
  const int digit_bits = (CellSortBits(num_cells) + passes - 1) / passes;
  const int bins = 1 << digit_bits;
  const int32_t* kin = pt_cell;
  const int32_t* vin = nullptr;
  for (int p = 0; p < passes; ++p) {
    int32_t* kout = (p & 1) == 0 ? keys_a : keys_b;
    int32_t* vout = (p & 1) == 0 ? vals_a : vals_b;
    const int shift = p * digit_bits;
    if (p == 0) {
      KRadixHist<true, kItems><<<tiles, kSortThreads, 0, stream>>>(kin, n, sentinel, shift, bins, hist, tiles);
    } else {
      KRadixHist<false, kItems><<<tiles, kSortThreads, 0, stream>>>(kin, n, sentinel, shift, bins, hist, tiles);
    }
    KDigitScan<<<(bins + 7) / 8, 256, 0, stream>>>(hist, bins, tiles);
    if (p == 0) {
      KRadixScatter<true, kItems><<<tiles, kSortThreads, 0, stream>>>(kin, vin, n, sentinel, shift, bins, hist, tiles,
                                                                     kout, vout);
    } else {
      KRadixScatter<false, kItems><<<tiles, kSortThreads, 0, stream>>>(kin, vin, n, sentinel, shift, bins, hist,
                                                                      tiles, kout, vout);
    }
    kin = kout;
    vin = vout;
  }
  return passes;
}

}  // namespace

/// 32-bit words of the sort's histogram: the digits' rows and their totals.
size_t CellSortWords(int64_t n) {
  const int64_t tile = static_cast<int64_t>(kSortThreads) * SortItems(n);
  return static_cast<size_t>(kSortMaxBins) * static_cast<size_t>((n + tile - 1) / tile + 1);
}

/// Host launcher: sorts (pt_cell, row) pairs; result rows in vals_a / keys_a
/// (ping-pong buffers of n entries each; hist of CellSortWords(n) words).
/// Returns the number of kernels launched.
int LaunchCellSort(const int32_t* pt_cell, int64_t n, int64_t num_cells, int32_t* keys_a, int32_t* vals_a,
                   int32_t* keys_b, int32_t* vals_b, int32_t* hist, cudaStream_t stream, bool* result_in_a) {
  const int passes = SortItems(n) == kSortItems
                         ? CellSort<kSortItems>(pt_cell, n, num_cells, keys_a, vals_a, keys_b, vals_b, hist, stream)
                         : CellSort<kSortFewItems>(pt_cell, n, num_cells, keys_a, vals_a, keys_b, vals_b, hist, stream);
  *result_in_a = (passes & 1) == 1;
  return 3 * passes;
}

}  // namespace sdfgpu
