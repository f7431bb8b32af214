// rpd_scan.cuh -- warp and block prefix sums shared by the kernels that
// scan per-thread counts (scans, compactions, polygon offsets), for 32- and
// 64-bit values, and the device-wide exclusive scan of 32-bit counts built on
// them.
#pragma once

#include <cuda_runtime.h>

namespace rpd {

// inclusive prefix sum of v over the lanes of a full warp
template <class T>
__device__ __forceinline__ T warp_incl_scan(T v, int lane) {
  for (int o = 1; o < 32; o <<= 1) {
    const T t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// block-wide exclusive prefix sum of one value per thread (every thread of
// the block calls it; blockDim.x a multiple of 32, at most 1024); returns
// the thread's exclusive prefix and writes the block total to *total
template <class T>
__device__ __forceinline__ T block_excl_scan(T v, T* total) {
  __shared__ T wsum[32];
  __shared__ T wtot;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const T incl = warp_incl_scan<T>(v, lane);
  if (lane == 31) wsum[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    const T x = lane < nw ? wsum[lane] : T(0);
    const T xi = warp_incl_scan<T>(x, lane);
    if (lane < nw) wsum[lane] = xi - x;
    if (lane == 31) wtot = xi;
  }
  __syncthreads();
  const T res = incl - v + wsum[wid];
  if (total) *total = wtot;
  __syncthreads();
  return res;
}

// ------------------------------------------------------------------------
// exclusive scan of n int32 counts into out[0..n] (out[n] the total; T is
// int32_t or long long; out may be in itself where T is int32_t)
// ------------------------------------------------------------------------
// A block scans tiles of 4,096.  Up to four tiles take one launch of one
// block; more take two: tile sums, then every block adds up the sums before
// its own (1,000 blocks read 2 MB of L2 between them: less than the launch
// of a scan of the sums, which only more than 4,096 tiles get).  Small meshes
// are launch-bound: a pass on 5k tets had ten scans of three launches each.
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int kScanOneBlock = 4 * kScanTile;
constexpr int kScanAddUp = 4096;

// the tile at `base`: out = carry + prefix; returns the tile's total
template <class T>
__device__ __forceinline__ T scan_tile(const int32_t* in, long long n, long long base, T carry,
                                       T* out) {
  const long long i0 = base + (long long)threadIdx.x * kScanItems;
  T v[kScanItems], sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = i0 + k < n ? (T)in[i0 + k] : T(0);
    sum += v[k];
  }
  T total;
  T run = carry + block_excl_scan<T>(sum, &total);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (i0 + k < n) out[i0 + k] = run;
    run += v[k];
  }
  return total;
}

template <class T>
__global__ void __launch_bounds__(kScanThreads) scan_one_block_kernel(const int32_t* in,
                                                                      long long n, T* out) {
  T carry = 0;
  for (long long base = 0; base < n; base += kScanTile)
    carry += scan_tile<T>(in, n, base, carry, out);
  if (threadIdx.x == 0) out[n] = carry;
}

template <class T>
__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(const int32_t* in, long long n,
                                                                 T* sums) {
  const long long base = (long long)blockIdx.x * kScanTile;
  T v = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const long long i = base + threadIdx.x + (long long)k * kScanThreads;
    if (i < n) v += in[i];
  }
  T total;
  block_excl_scan<T>(v, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// the tile sums in place, by one block
template <class T>
__global__ void __launch_bounds__(kScanThreads) scan_of_sums_kernel(T* sums, int nb) {
  T carry = 0;
  for (int base = 0; base < nb; base += kScanThreads) {
    const int i = base + threadIdx.x;
    T total;
    const T ex = block_excl_scan<T>(i < nb ? sums[i] : T(0), &total);
    if (i < nb) sums[i] = ex + carry;
    carry += total;
  }
}

// the sum of the values before this block's (scanned: they are prefixes)
template <class T>
__device__ __forceinline__ T scan_before(const T* sums, bool scanned) {
  if (scanned) return sums[blockIdx.x];
  T v = 0;
  for (int i = threadIdx.x; i < (int)blockIdx.x; i += blockDim.x) v += sums[i];
  T total;
  block_excl_scan<T>(v, &total);
  return total;
}

template <class T>
__global__ void __launch_bounds__(kScanThreads) scan_tiles_kernel(const int32_t* in, long long n,
                                                                  const T* sums, bool scanned,
                                                                  T* out) {
  const T carry = scan_before<T>(sums, scanned);
  const T total = scan_tile<T>(in, n, (long long)blockIdx.x * kScanTile, carry, out);
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = carry + total;
}

void note_launches(int n);

// temp: one T per tile
template <class T>
cudaError_t scan_counts(const int32_t* in, T* out, long long n, T* temp, cudaStream_t st) {
  if (n <= 0) return cudaMemsetAsync(out, 0, sizeof(T), st);
  if (n <= kScanOneBlock) {
    scan_one_block_kernel<T><<<1, kScanThreads, 0, st>>>(in, n, out);
    note_launches(1);
    return cudaGetLastError();
  }
  const int nb = (int)((n + kScanTile - 1) / kScanTile);
  const bool scanned = nb > kScanAddUp;
  scan_sums_kernel<T><<<nb, kScanThreads, 0, st>>>(in, n, temp);
  if (scanned) scan_of_sums_kernel<T><<<1, kScanThreads, 0, st>>>(temp, nb);
  scan_tiles_kernel<T><<<nb, kScanThreads, 0, st>>>(in, n, temp, scanned, out);
  note_launches(scanned ? 3 : 2);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// compaction: the indices q in [0, n) with keep(q), in order
// ------------------------------------------------------------------------
// Two launches: counts per block (count(q) may do more on the way), then
// every block adds up the counts before its own and hands its kept indices
// to put(q, position).  No flag and position arrays in between.
constexpr int kKeepThreads = 256;
constexpr int kKeepTile = 1024;    // least indices of a block
constexpr int kKeepBlocks = 1024;  // blocks that the tile grows for: the sums
                                   // that each adds up stay few

template <class Count>
__global__ void __launch_bounds__(kKeepThreads) keep_count_kernel(Count count, long long n,
                                                                  int tile, int32_t* sums) {
  count.begin();
  const long long base = (long long)blockIdx.x * tile;
  int v = 0;
  for (int k = threadIdx.x; k < tile; k += kKeepThreads)
    if (base + k < n) v += count(base + k) ? 1 : 0;
  int total;
  block_excl_scan<int>(v, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
  count.end();
}

template <class Keep, class Put, class Total>
__global__ void __launch_bounds__(kKeepThreads) keep_put_kernel(Keep keep, Put put, long long n,
                                                                int tile, const int32_t* sums,
                                                                Total* total_out) {
  __shared__ int wsum[kKeepThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long base = (long long)blockIdx.x * tile;
  int at = scan_before<int32_t>(sums, false);
  for (int k = 0; k < tile; k += kKeepThreads) {
    const long long q = base + k + threadIdx.x;
    const bool in = q < n && keep(q);
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (lane == 0) wsum[wid] = __popc(m);
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < kKeepThreads / 32; ++w) {
      before += w < wid ? wsum[w] : 0;
      all += wsum[w];
    }
    if (in) put(q, (long long)at + before + __popc(m & ((1u << lane) - 1u)));
    at += all;
    __syncthreads();
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total_out = (Total)at;
}

// sums: one int32 per kKeepTile indices
template <class Count, class Keep, class Put, class Total>
cudaError_t keep_indices(Count count, Keep keep, Put put, long long n, int32_t* sums,
                         Total* total_out, cudaStream_t st) {
  if (n <= 0) return cudaMemsetAsync(total_out, 0, sizeof(Total), st);
  long long per = (n + kKeepBlocks - 1) / kKeepBlocks;
  if (per < kKeepTile) per = kKeepTile;
  const int tile = (int)((per + kKeepThreads - 1) / kKeepThreads * kKeepThreads);
  const int nb = (int)((n + tile - 1) / tile);
  keep_count_kernel<<<nb, kKeepThreads, 0, st>>>(count, n, tile, sums);
  keep_put_kernel<<<nb, kKeepThreads, 0, st>>>(keep, put, n, tile, sums, total_out);
  note_launches(2);
  return cudaGetLastError();
}

}  // namespace rpd
