// rpd_sort.cu -- stable radix sort of 64-bit keys with 32-bit values.
//
// Used to group per-cell records (power cells: by site, then by neighbour or
// face).  Least-significant-digit first, 8 bits per pass, each pass stable.  A
// block takes 1,024 consecutive keys, its warp w the 128 from 128 w on, 32 at
// a time: a key's rank is the digit's running count in its warp plus the
// equal digits in lower lanes (__match_any_sync), and the digit-major exclusive
// scan of all blocks' counts, followed within a block by a scan over its
// warps, gives each warp its base for every digit.  (256 keys a block made as
// many counts as keys; power cells of the 200k-tet workload, 18 passes and
// fewer over 1.7M keys: 2.40 ms with 16 keys a thread, 2.24 with 8, 2.22 with
// 4, 2.28 with 2, 2.48 with one.)
//
// Keys of two 32-bit fields, of which the lower one holds small numbers, skip
// the passes over its zero digits (low_bits).

#include <cuda_runtime.h>

#include "rpd_kernels.cuh"

namespace rpd {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 4;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kRadix = 256;

// the lanes whose digit equals this one's (lanes without a key have digit -1)
__device__ __forceinline__ unsigned same_digit(int digit) {
  return __match_any_sync(0xffffffffu, digit);
}

__global__ void __launch_bounds__(kSortThreads)
    radix_count_kernel(const unsigned long long* keys, long long n, int shift, int n_blocks,
                       int32_t* hist /* [kRadix][n_blocks] */) {
  __shared__ int counts[kRadix];
  const int lane = threadIdx.x & 31;
  for (int d = threadIdx.x; d < kRadix; d += kSortThreads) counts[d] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * kSortTile;
#pragma unroll 4
  for (int r = 0; r < kSortItems; ++r) {
    const long long i = base + r * kSortThreads + threadIdx.x;
    const int digit = i < n ? (int)((keys[i] >> shift) & 0xffull) : -1;
    const unsigned peers = same_digit(digit);
    if (digit >= 0 && lane == __ffs(peers) - 1) atomicAdd(counts + digit, __popc(peers));
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kRadix; d += kSortThreads)
    hist[(long long)d * n_blocks + blockIdx.x] = counts[d];
}

__global__ void __launch_bounds__(kSortThreads)
    radix_scatter_kernel(const unsigned long long* keys, const uint32_t* vals, long long n,
                         int shift, int n_blocks, const int32_t* base /* scanned hist */,
                         unsigned long long* keys_out, uint32_t* vals_out) {
  __shared__ int next[kSortWarps][kRadix];  // counts, then the next place, of each digit
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < kSortWarps * kRadix; i += kSortThreads) (&next[0][0])[i] = 0;
  __syncthreads();
  const long long first = (long long)blockIdx.x * kSortTile + wid * (32 * kSortItems) + lane;
  unsigned long long k[kSortItems];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r)
    k[r] = first + 32 * r < n ? keys[first + 32 * r] : 0ull;
  auto digit_of = [&](int r) {
    return first + 32 * r < n ? (int)((k[r] >> shift) & 0xffull) : -1;
  };
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int digit = digit_of(r);
    const unsigned peers = same_digit(digit);
    if (digit >= 0 && lane == __ffs(peers) - 1) next[wid][digit] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kRadix; d += kSortThreads) {
    int at = base[(long long)d * n_blocks + blockIdx.x];
    for (int w = 0; w < kSortWarps; ++w) {
      const int c = next[w][d];
      next[w][d] = at;
      at += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int digit = digit_of(r);
    const unsigned peers = same_digit(digit);
    const int leader = __ffs(peers) - 1;
    int at = 0;
    if (digit >= 0 && lane == leader) {
      at = next[wid][digit];
      next[wid][digit] = at + __popc(peers);
    }
    at = __shfl_sync(0xffffffffu, at, leader) + __popc(peers & ((1u << lane) - 1u));
    if (digit >= 0) {
      keys_out[at] = k[r];
      vals_out[at] = vals[first + 32 * r];
    }
    __syncwarp();
  }
}

}  // namespace

size_t radix_hist_ints(long long n) {
  const long long nb = (n + kSortTile - 1) / kSortTile;
  return (size_t)(nb * kRadix + 1);
}

// Sorts (keys, vals) by the low `bits` bits of the keys, stably, bits
// low_bits..31 being zero in all of them (32: none known); the result
// is in keys / vals (the *_tmp buffers are scratch of n entries; hist and
// scan_tmp hold radix_hist_ints(n) and scan_temp_ints(of that) ints).
cudaError_t radix_sort_pairs(unsigned long long* keys, uint32_t* vals, long long n, int bits,
                             unsigned long long* keys_tmp, uint32_t* vals_tmp, int32_t* hist,
                             int32_t* scan_tmp, cudaStream_t st, int low_bits) {
  if (n <= 1 || bits <= 0) return cudaSuccess;
  if (n > 0x7fffffffll) return cudaErrorInvalidValue;  // positions are int32
  const int nb = (int)((n + kSortTile - 1) / kSortTile);
  const long long nh = (long long)nb * kRadix;
  unsigned long long *ka = keys, *kb = keys_tmp;
  uint32_t *va = vals, *vb = vals_tmp;
  int passes = 0;
  for (int shift = 0; shift < bits; shift += 8) {
    if (shift >= low_bits && shift < 32) continue;
    radix_count_kernel<<<nb, kSortThreads, 0, st>>>(ka, n, shift, nb, hist);
    cudaError_t e = scan_exclusive(hist, hist, nh, scan_tmp, st);
    if (e != cudaSuccess) return e;
    radix_scatter_kernel<<<nb, kSortThreads, 0, st>>>(ka, va, n, shift, nb, hist, kb, vb);
    note_launches(2);
    unsigned long long* tk = ka;
    ka = kb;
    kb = tk;
    uint32_t* tv = va;
    va = vb;
    vb = tv;
    ++passes;
  }
  if (passes & 1) {  // result in the scratch buffers: copy back
    cudaError_t e = cudaMemcpyAsync(keys, ka, sizeof(unsigned long long) * (size_t)n,
                                    cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(vals, va, sizeof(uint32_t) * (size_t)n, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

}  // namespace rpd
