// rpd_pairs.cu -- everything around the clip kernel: uniform grids, the
// k-nearest-power-neighbour build, candidate (tet, site) pairs, scans and
// compaction.
//
// Reference counterparts:
//   * neighbour lists: libmat takes each site's regular-triangulation
//     neighbours from CGAL on the CPU (src/rpd3d_base/triangulation.cxx:
//     62-144, :442-558); here the lists are the k smallest power-bisector
//     distances, found by a ring search over a uniform grid of sites.
//   * candidate pairs: libmat tests every (tet, site) with the rule of
//     tet_sphere_relations_dev (src/rpd3d/voronoi.cu:154-193) -- tet t is a
//     candidate of flagged site i iff for every listed neighbour m some tet
//     vertex v has pd_m(v) > pd_i(v), power distances computed as in
//     src/rpd3d/kNN-CUDA/knncuda.cu:21-94 + :130-160 -- on dense n_site x
//     n_vert and n_site x n_tet matrices, then gathers them on the host
//     (:265-317).  Here the same rule is applied only to tets whose centroid
//     lies in a per-site box that provably contains every tet passing it
//     (see site_box_kernel), and the pairs are written as a per-tet CSR with
//     sites ascending, the reference's tet_knn order.
// Compiled with -fmad=false: the power distances and bisector keys are the
// reference's / oracle's float expressions evaluated without contraction.

#include <cuda_runtime.h>

#include <cstdint>

#include "rpd_common.cuh"
#include "rpd_kernels.cuh"
#include "rpd_scan.cuh"

namespace rpd {

static thread_local int tl_launches = 0;
void note_launches(int n) { tl_launches += n; }
int take_launches() {
  int n = tl_launches;
  tl_launches = 0;
  return n;
}

// ------------------------------------------------------------------------
// scan
// ------------------------------------------------------------------------
size_t scan_temp_ints(long long n) { return (size_t)((n + kKeepTile - 1) / kKeepTile) + 1; }

cudaError_t scan_exclusive(const int32_t* in, int32_t* out, long long n, int32_t* temp,
                           cudaStream_t st) {
  return scan_counts<int32_t>(in, out, n, temp, st);
}

// ------------------------------------------------------------------------
// uniform grids
// ------------------------------------------------------------------------
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ int cell_index(const Grid& g, float x, float y, float z) {
  int ix = clampi((int)floorf((x - g.lo.x) * g.inv_cell), 0, g.nx - 1);
  int iy = clampi((int)floorf((y - g.lo.y) * g.inv_cell), 0, g.ny - 1);
  int iz = clampi((int)floorf((z - g.lo.z) * g.inv_cell), 0, g.nz - 1);
  return ix + g.nx * (iy + g.ny * iz);
}

__global__ void bin_points_kernel(const float4* pts, int n, Grid g, int32_t* cell_of,
                                  int32_t* cell_count, const uint8_t* cls, int want,
                                  float* cell_rmax) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (cls && cls[i] != want) {
    cell_of[i] = -1;
    return;
  }
  float4 p = pts[i];
  int c = cell_index(g, p.x, p.y, p.z);
  cell_of[i] = c;
  atomicAdd(cell_count + c, 1);
  // radii are >= 0: their bit patterns order as the floats do
  if (cell_rmax) atomicMax(reinterpret_cast<unsigned int*>(cell_rmax) + c, __float_as_uint(p.w));
}

// the cells' items; their order within a cell is not kept (the pair list is
// sorted per tet, the neighbour lists by key and id)
__global__ void fill_cells_kernel(int n, const int32_t* cell_of, const int32_t* cell_start,
                                  int32_t* cell_fill, int32_t* cell_items, const float4* cent,
                                  const float4* xyz, float4* cent_out, float4* xyz_out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int c = cell_of[i];
  if (c < 0) return;
  const int slot = cell_start[c] + atomicAdd(cell_fill + c, 1);
  cell_items[slot] = i;
  if (cent_out) {
    cent_out[slot] = cent[i];
    for (int k = 0; k < 3; ++k) xyz_out[3ll * slot + k] = xyz[3ll * i + k];
  }
}

static cudaError_t grid_finish(int n, const Grid& g, const int32_t* cell_of, int32_t* cell_count,
                               int32_t* cell_start, int32_t* cell_fill, int32_t* cell_items,
                               int32_t* scan_tmp, cudaStream_t st, const float4* cent = nullptr,
                               const float4* xyz = nullptr, float4* cent_out = nullptr,
                               float4* xyz_out = nullptr) {
  long long n_cells = (long long)g.nx * g.ny * g.nz;
  cudaError_t err = scan_exclusive(cell_count, cell_start, n_cells, scan_tmp, st);
  if (err != cudaSuccess) return err;
  cudaMemsetAsync(cell_fill, 0, sizeof(int32_t) * n_cells, st);
  fill_cells_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, cell_of, cell_start, cell_fill, cell_items,
                                                    cent, xyz, cent_out, xyz_out);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t grid_build_sites(const float4* pts, int n, const Grid& g, int32_t* cell_of,
                             int32_t* cell_count, int32_t* cell_start, int32_t* cell_fill,
                             int32_t* cell_items, int32_t* scan_tmp, cudaStream_t st) {
  long long n_cells = (long long)g.nx * g.ny * g.nz;
  cudaMemsetAsync(cell_count, 0, sizeof(int32_t) * n_cells, st);
  if (n > 0) {
    bin_points_kernel<<<(n + 255) / 256, 256, 0, st>>>(pts, n, g, cell_of, cell_count, nullptr, 0,
                                                      nullptr);
    note_launches(1);
  }
  return grid_finish(n, g, cell_of, cell_count, cell_start, cell_fill, cell_items, scan_tmp, st);
}

// centroid and radius (largest vertex distance) of every tet
__global__ void tet_centroid_kernel(const float* v, const int4* tets, int n_tet, float4* out,
                                    float4* xyz, const int32_t* v_adjs, uchar4* vadj) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tet) return;
  int4 q = tets[t];
  int id[4] = {q.x, q.y, q.z, q.w};
  float cx = 0.f, cy = 0.f, cz = 0.f;
  for (int k = 0; k < 4; ++k) {
    cx += v[3 * id[k]];
    cy += v[3 * id[k] + 1];
    cz += v[3 * id[k] + 2];
  }
  cx *= 0.25f;
  cy *= 0.25f;
  cz *= 0.25f;
  float r2 = 0.f;
  for (int k = 0; k < 4; ++k) {
    float dx = v[3 * id[k]] - cx, dy = v[3 * id[k] + 1] - cy, dz = v[3 * id[k] + 2] - cz;
    r2 = fmaxf(r2, dx * dx + dy * dy + dz * dz);
  }
  out[t] = make_float4(cx, cy, cz, sqrtf(r2));
  if (xyz) {  // the four vertices, packed: (v0, v1.x) (v1.yz, v2.xy) (v2.z, v3)
    float f[12];
    for (int k = 0; k < 4; ++k)
      for (int a = 0; a < 3; ++a) f[3 * k + a] = v[3 * id[k] + a];
    xyz[3ll * t] = make_float4(f[0], f[1], f[2], f[3]);
    xyz[3ll * t + 1] = make_float4(f[4], f[5], f[6], f[7]);
    xyz[3ll * t + 2] = make_float4(f[8], f[9], f[10], f[11]);
  }
  if (vadj)
    vadj[t] = make_uchar4((uint8_t)v_adjs[id[0]], (uint8_t)v_adjs[id[1]], (uint8_t)v_adjs[id[2]],
                          (uint8_t)v_adjs[id[3]]);
}

cudaError_t tet_centroids(const float* vert3f, const int4* tets, int n_tet, float4* centroid,
                          cudaStream_t st, float4* tet_xyz, const int32_t* v_adjs,
                          uchar4* tet_vadj) {
  if (n_tet > 0) {
    tet_centroid_kernel<<<(n_tet + 255) / 256, 256, 0, st>>>(vert3f, tets, n_tet, centroid,
                                                              tet_xyz, v_adjs, tet_vadj);
    note_launches(1);
  }
  return cudaGetLastError();
}

cudaError_t grid_build_tets(const float4* centroid, int n_tet, const uint8_t* cls, int want,
                            const Grid& g, int32_t* cell_of, int32_t* cell_count,
                            int32_t* cell_start, int32_t* cell_fill, int32_t* cell_items,
                            int32_t* scan_tmp, cudaStream_t st, float* cell_rmax,
                            const float4* tet_xyz, float4* cent_out, float4* xyz_out) {
  long long n_cells = (long long)g.nx * g.ny * g.nz;
  cudaMemsetAsync(cell_count, 0, sizeof(int32_t) * n_cells, st);
  if (cell_rmax) cudaMemsetAsync(cell_rmax, 0, sizeof(float) * n_cells, st);
  if (n_tet > 0) {
    bin_points_kernel<<<(n_tet + 255) / 256, 256, 0, st>>>(centroid, n_tet, g, cell_of, cell_count,
                                                          cls, want, cell_rmax);
    note_launches(1);
  }
  return grid_finish(n_tet, g, cell_of, cell_count, cell_start, cell_fill, cell_items, scan_tmp,
                     st, centroid, tet_xyz, cent_out, xyz_out);
}

// ------------------------------------------------------------------------
// warp helper: iterate the items of a set of grid cells, 32 at a time
// ------------------------------------------------------------------------
// cells are enumerated by `cell_at(idx)` for idx in [0, n_cells_iter), which
// returns a cell id or -1; fn(at, valid) is called warp-uniformly for batches
// of 32 positions in the item list (valid = false for padding lanes).  With
// LAST one more call follows, without positions (its third argument is true):
// the caller's code for what is left over is then in one place.
template <bool LAST, class CellAt, class Fn>
__device__ void for_items(int n_cells_iter, CellAt cell_at, const int32_t* cell_start, int lane,
                          Fn fn) {
  for (int cb = 0; cb < n_cells_iter + (LAST ? 32 : 0); cb += 32) {
    const bool last = LAST && cb >= n_cells_iter;
    int ci = cb + lane;
    int cell = ci < n_cells_iter ? cell_at(ci) : -1;
    int b = 0, cnt = 0;
    if (cell >= 0) {
      b = cell_start[cell];
      cnt = cell_start[cell + 1] - b;
    }
    int incl = warp_incl_scan<int>(cnt, lane);
    int total = __shfl_sync(0xffffffffu, incl, 31);
    int excl = incl - cnt;
    for (int ib = 0; ib < total || (last && ib == 0); ib += 32) {
      int g = ib + lane;
      // owner lane: the last lane whose exclusive prefix is <= g
      int owner = 0;
      for (int o = 16; o > 0; o >>= 1) {
        int cand = owner + o;
        int ex = __shfl_sync(0xffffffffu, excl, cand);
        if (ex <= g) owner = cand;
      }
      int ob = __shfl_sync(0xffffffffu, b, owner);
      int oe = __shfl_sync(0xffffffffu, excl, owner);
      bool valid = g < total;
      fn(ob + (g - oe), valid, last);
    }
  }
}

// ------------------------------------------------------------------------
// k nearest power neighbours
// ------------------------------------------------------------------------
constexpr int kKnnBuf = 1024;
constexpr int kKnnWarps = 4;
constexpr int kKnnLongBuf = 8192;  // long lists (k > kKnnBuf - 64): 64 KB, one warp per block
// base lists (k <= kKnnSmallBuf - 64): half the buffer, twice the warps in
// the same shared memory (more warps to hide the search's latency; 1M-tet
// workload, k = 128: 2.64 -> 1.82 ms; a quarter of the buffer with four
// times the warps measured the same)
constexpr int kKnnSmallBuf = 512;
constexpr int kKnnSmallWarps = 8;
// blocks that must fit an SM: 64 registers (the sort of 512 entries holds 32);
// 2 / 3 / 4 / 5 blocks take 1.49 / 1.12 / 1.05 / 1.16 ms there
constexpr int kKnnSmallBlocks = 4;

__device__ __forceinline__ uint32_t order_key(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// power-bisector distance of site j from site i (same expression as the
// oracle): ((|cj - ci|^2 - wj) + wi) / (2 |cj - ci|)
__device__ __forceinline__ float bisector_key(float4 si, float4 sj) {
  float dx = sj.x - si.x, dy = sj.y - si.y, dz = sj.z - si.z;
  float d2 = dx * dx + dy * dy + dz * dz;
  if (d2 == 0.0f) return sj.w > si.w ? -INFINITY : INFINITY;
  float num = (d2 - sj.w) + si.w;
  float den = 2.0f * sqrtf(d2);
  return num / den;
}

// bitonic sort of buf[0..n) (n power of two) by one warp, ascending
__device__ void warp_bitonic_sort(unsigned long long* buf, int n, int lane) {
  for (int k = 2; k <= n; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = lane; i < n; i += 32) {
        int l = i ^ j;
        if (l > i) {
          unsigned long long a = buf[i], b = buf[l];
          bool up = (i & k) == 0;
          if ((a > b) == up) {
            buf[i] = b;
            buf[l] = a;
          }
        }
      }
      __syncwarp();
    }
  }
}

// the same for 32 PER entries in registers, of which the first `keep` come
// back: lane l holds elements PER l .. PER l + PER - 1 of the network, so its
// strides below PER need no exchange between lanes.  (Every exchange of the
// sort above goes through shared memory: 512 entries take about 6,700 warp
// instructions there and 3,400 here.)  The entries are read as they lie (a
// sort may start from any order) and only the kept ones are written back.
template <int PER>
__device__ __forceinline__ void warp_register_sort(unsigned long long* buf, int lane, int keep) {
  unsigned long long v[PER];
#pragma unroll
  for (int r = 0; r < PER; ++r) v[r] = buf[32 * r + lane];
  auto exchange = [&](int r, int j, bool up) {
    const unsigned long long a = v[r], b = v[r + j];
    const bool swap = (a > b) == up;
    v[r] = swap ? b : a;
    v[r + j] = swap ? a : b;
  };
  // levels within a lane
#pragma unroll
  for (int k = 2; k < PER; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int r = 0; r < PER; ++r)
        if ((r & j) == 0) exchange(r, j, (r & k) == 0);
  // levels across lanes
  for (int k = PER > 1 ? PER : 2; k <= 32 * PER; k <<= 1) {
    const bool up = ((lane * PER) & k) == 0;
    for (int j = k >> 1; j >= PER; j >>= 1) {
      const int lj = j / PER;
      const bool take_max = ((lane & lj) != 0) == up;
#pragma unroll
      for (int r = 0; r < PER; ++r) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, v[r], lj);
        v[r] = (o > v[r]) == take_max ? o : v[r];
      }
    }
#pragma unroll
    for (int j = PER >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int r = 0; r < PER; ++r)
        if ((r & j) == 0) exchange(r, j, up);
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < PER; ++r)
    if (PER * lane + r < keep) buf[PER * lane + r] = v[r];
  __syncwarp();
}

// buf[0..n) sorted, n a power of two and at least 32; only the first `keep`
// entries are kept.  MAX: the largest n
template <int MAX>
__device__ __forceinline__ void warp_sort(unsigned long long* buf, int n, int lane, int keep) {
  if (n <= 64) {
    if (n < 64) buf[32 + lane] = ~0ull;
    __syncwarp();
    warp_register_sort<2>(buf, lane, keep);
  } else if (n == 128) {
    warp_register_sort<4>(buf, lane, keep);
  } else if (n == 256) {
    warp_register_sort<8>(buf, lane, keep);
  } else if (n == 512) {
    warp_register_sort<16>(buf, lane, keep);
  } else if (MAX >= 1024 && n == 1024) {
    warp_register_sort<32>(buf, lane, keep);
  } else {
    warp_bitonic_sort(buf, n, lane);
  }
}

__device__ __forceinline__ int next_pow2(int x) {
  int p = 32;
  while (p < x) p <<= 1;
  return p;
}

// One warp per row: the k smallest (key, id) of site i = subset[row] (or
// i = row), optionally only keys <= B (B = R_i * bound_scale + bound_abs,
// R_i the float in radius[i]).  Rings of grid cells around the site are
// searched until every site outside has a key above the k-th kept one (or
// above B): keys of sites at distance >= D are >= (D^2 + w_i - w_max)/(2D).
// Candidates collect in a per-warp buffer of BUF entries (key bits | id,
// 64-bit) that is sorted and cut to k when it fills, and at the end of a ring
// only where the k-th key may end the search.  Sorting bounds it: with a sort
// after every ring, through shared memory, base lists of 128 for 50k sites took
// 1.61 ms and the longer lists of 2.7k of them 0.51 ms; with the sorts that are
// needed, in registers, and rings enumerated as shells 1.05 and 0.25 ms (200k
// tets: 0.31 and 0.36 -> 0.18 and 0.10 ms).
template <int BUF, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == kKnnSmallWarps ? kKnnSmallBlocks : 1)
    knn_kernel(KnnArgs a) {
  extern __shared__ __align__(16) unsigned long long knn_smem[];
  __shared__ int scnt[WARPS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long* buf = knn_smem + (size_t)wid * BUF;
  const int row = blockIdx.x * WARPS + wid;
  if (row >= a.n_rows) return;
  const int i = a.subset ? a.subset[row] : row;
  const int k = a.k;
  const Grid& g = a.g;
  const float4 si = a.site4f[i];
  const int2 rng = a.site_range ? a.site_range[i] : make_int2(0, 0x7fffffff);
  float B = INFINITY;
  if (a.radius) {
    const float R = __uint_as_float(a.radius[i]);
    B = R * a.bound_scale + a.bound_abs;
    if (!(B < INFINITY)) B = INFINITY;  // inf or nan radius: no bound
  }
  const float4 gp = a.grid_pos ? a.grid_pos[i] : si;
  const int cx = clampi((int)floorf((gp.x - g.lo.x) * g.inv_cell), 0, g.nx - 1);
  const int cy = clampi((int)floorf((gp.y - g.lo.y) * g.inv_cell), 0, g.ny - 1);
  const int cz = clampi((int)floorf((gp.z - g.lo.z) * g.inv_cell), 0, g.nz - 1);
  const int rmax = max(max(max(cx, g.nx - 1 - cx), max(cy, g.ny - 1 - cy)), max(cz, g.nz - 1 - cz));
  if (lane == 0) scnt[wid] = 0;
  __syncwarp();
  unsigned long long kth = ~0ull;  // packed k-th best so far (after a sort)
  bool done = false;
  bool sorted = true;  // the buffer holds the best of what was seen, in order
  // sorts the cnt entries and keeps the best k
  auto sort_cut = [&](int cnt) {
    const int n = next_pow2(max(cnt, 1));
    for (int q = cnt + lane; q < n; q += 32) buf[q] = ~0ull;
    __syncwarp();
    warp_sort<BUF>(buf, n, lane, k);
    sorted = true;
    if (cnt >= k) kth = buf[k - 1];
    return min(cnt, k);
  };
  for (int r = 0; r <= rmax && !done; ++r) {
    // the cells at distance r (in cells): the two faces z = -r, r, then the
    // four sides of each layer between them, 2 r cells a side
    const int side = 2 * r + 1;
    const int n_face = side * side;
    const int n_shell = r == 0 ? 1 : 2 * n_face + (side - 2) * 8 * r;
    auto cell_at = [&](int idx) -> int {
      int dx, dy, dz;
      if (idx < 2 * n_face) {
        dz = idx < n_face ? -r : r;
        const int q = idx < n_face ? idx : idx - n_face;
        dy = q / side - r;
        dx = q % side - r;
      } else {
        const int q = idx - 2 * n_face;
        dz = q / (8 * r) - r + 1;
        const int e = q % (8 * r);
        const int t = e % (2 * r) - r;  // -r .. r - 1
        const int edge = e / (2 * r);
        dx = edge == 0 ? t : (edge == 1 ? r : (edge == 2 ? -t : -r));
        dy = edge == 0 ? -r : (edge == 1 ? t : (edge == 2 ? r : -t));
      }
      const int x = cx + dx, y = cy + dy, z = cz + dz;
      if (x < 0 || y < 0 || z < 0 || x >= g.nx || y >= g.ny || z >= g.nz) return -1;
      return x + g.nx * (y + g.ny * z);
    };
    for_items<false>(n_shell, cell_at, a.cell_start, lane, [&](int at, bool valid, bool) {
      const int j = valid ? a.cell_items[at] : -1;
      bool take = false;
      unsigned long long packed = 0;
      if (valid && j != i && j >= rng.x && j < rng.y) {
        float key = bisector_key(si, a.site4f[j]);
        packed = ((unsigned long long)order_key(key) << 32) | (uint32_t)j;
        take = packed < kth && key <= B;
      }
      uint32_t m = __ballot_sync(0xffffffffu, take);
      int base = scnt[wid];
      if (take) buf[base + __popc(m & ((1u << lane) - 1u))] = packed;
      __syncwarp();
      int cnt = base + __popc(m);
      if (m) sorted = false;
      if (cnt > BUF - 32) cnt = sort_cut(cnt);
      if (lane == 0) scnt[wid] = cnt;
      __syncwarp();
    });
    // done once no site outside the searched block can have a key of T or
    // less: keys there are >= f(D) with D >= r * cell, f(D) = (D^2 + wi -
    // wmax) / (2D) increasing in D
    auto reached = [&](float T) {
      const float D = (float)r * g.cell;
      if (!(D > 0.f && T < INFINITY)) return false;
      const float lb = (D * D + si.w - a.w_max) / (2.f * D);
      return T < lb - 1e-4f * (fabsf(lb) + D);
    };
    // fewer than k so far: every key up to B is still wanted.  Else the k-th
    // key of the last sort bounds the wanted ones, and only a search that it
    // does not end sorts again for a smaller one
    int cnt = scnt[wid];
    if (cnt < k) {
      done = reached(B);
    } else {
      done = kth != ~0ull && reached(fminf(B, key_value((uint32_t)(kth >> 32))));
      if (!done && !sorted) {
        cnt = sort_cut(cnt);
        if (lane == 0) scnt[wid] = cnt;
        done = reached(fminf(B, key_value((uint32_t)(kth >> 32))));
      }
    }
    __syncwarp();
  }
  if (!sorted) {
    const int c = sort_cut(scnt[wid]);
    __syncwarp();
    if (lane == 0) scnt[wid] = c;
    __syncwarp();
  }
  int cnt = scnt[wid];
  if (a.status && lane == 0) a.status[row] = done ? 0 : 1;  // 1: exhausted grid
  if (lane == 0) {
    if (a.len_out) a.len_out[row] = cnt;
    // every site not listed has a key >= this: the k-th key when the list
    // is full, else the bound (or none: all sites were seen)
    if (a.bound_out) a.bound_out[row] = cnt >= k ? key_value((uint32_t)(buf[k - 1] >> 32)) : B;
  }
  const long long rb = (long long)row * k;
  // outputs in distance order
  for (int q = lane; q < k; q += 32) {
    int32_t id = q < cnt ? (int32_t)(uint32_t)buf[q] + a.id_offset : -1;
    if (a.keys) a.keys[rb + q] = q < cnt ? key_value((uint32_t)(buf[q] >> 32)) : INFINITY;
    if (!a.order_by_id) a.nbr[rb + q] = id;
    if (a.nbr_dist) a.nbr_dist[rb + q] = id;
  }
  if (a.order_by_id) {
    __syncwarp();
    int n = next_pow2(max(k, 1));
    // reuse the buffer: ids as 64-bit values, padding at the end
    for (int q = lane; q < n; q += 32) {
      unsigned long long v = ~0ull;
      if (q < cnt) v = (unsigned long long)(uint32_t)buf[q];
      __syncwarp();
      buf[q] = v;
    }
    __syncwarp();
    warp_sort<BUF>(buf, n, lane, k);
    for (int q = lane; q < k; q += 32)
      a.nbr[rb + q] = q < cnt ? (int32_t)buf[q] + a.id_offset : -1;
  }
}

int knn_max_k() { return kKnnLongBuf - 64; }

cudaError_t launch_knn(const KnnArgs& a, cudaStream_t st) {
  if (a.n_rows <= 0) return cudaSuccess;
  if (a.k < 1 || a.k > knn_max_k()) return cudaErrorInvalidValue;
  if (a.k <= kKnnSmallBuf - 64) {
    const size_t smem = (size_t)kKnnSmallWarps * kKnnSmallBuf * sizeof(unsigned long long);
    int blocks = (a.n_rows + kKnnSmallWarps - 1) / kKnnSmallWarps;
    knn_kernel<kKnnSmallBuf, kKnnSmallWarps><<<blocks, kKnnSmallWarps * 32, smem, st>>>(a);
  } else if (a.k <= kKnnBuf - 64) {
    const size_t smem = (size_t)kKnnWarps * kKnnBuf * sizeof(unsigned long long);
    int blocks = (a.n_rows + kKnnWarps - 1) / kKnnWarps;
    knn_kernel<kKnnBuf, kKnnWarps><<<blocks, kKnnWarps * 32, smem, st>>>(a);
  } else {
    // long lists: one warp per block, kKnnLongBuf entries of shared memory
    const size_t smem = (size_t)kKnnLongBuf * sizeof(unsigned long long);
    // (set on every such launch: the attribute belongs to the current device)
    cudaError_t e = cudaFuncSetAttribute(knn_kernel<kKnnLongBuf, 1>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    knn_kernel<kKnnLongBuf, 1><<<a.n_rows, 32, smem, st>>>(a);
  }
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_knn(const float4* site4f, int n_site, const Grid& g, const int32_t* cell_start,
                       const int32_t* cell_items, int k, float w_max, int order_by_id,
                       int32_t* nbr, float* keys, int32_t* nbr_dist, int32_t* status,
                       cudaStream_t st, int id_offset, float* bound_out) {
  KnnArgs a = {};
  a.site4f = site4f;
  a.n_rows = n_site;
  a.g = g;
  a.cell_start = cell_start;
  a.cell_items = cell_items;
  a.k = k;
  a.w_max = w_max;
  a.order_by_id = order_by_id;
  a.nbr = nbr;
  a.keys = keys;
  a.nbr_dist = nbr_dist;
  a.status = status;
  a.id_offset = id_offset;
  a.bound_out = bound_out;
  return launch_knn(a, st);
}

// ------------------------------------------------------------------------
// candidate pairs
// ------------------------------------------------------------------------
// power distance of a mesh vertex to a site, the reference's float order
__device__ __forceinline__ float pow_dist(float4 s, float3 v) {
  float t0 = s.x - v.x, t1 = s.y - v.y, t2 = s.z - v.z;
  float ssd = t0 * t0;
  ssd = ssd + t1 * t1;
  ssd = ssd + t2 * t2;
  return ssd - s.w;
}

constexpr int kPairWarps = 4;
// blocks that must fit an SM (72 registers); pair stage of the 1M-tet workload
// with 5 / 6 / 7 / 8 / 9: 4.46 / 4.29 / 4.13 / 4.11 / 4.23 ms, of 5k tets 163 / 172 /
// 169 / 170 / 178 us
constexpr int kPairBlocks = 7;
constexpr int kPairMaxK = 128;  // longest neighbour list (rpd_config.knn_k <= 128)
// a tet goes through three stages, each on full warps: the centroid test
// (one tet per lane); the tets that pass wait in a per-warp queue and try
// the rule's first kRuleFirst neighbours 32 at a time; the tets that survive
// those wait in a second queue and are finished 32 at a time against the rest
// of the list (queues of kRuleQueue entries).  kRuleFirst: 4 to 16 were
// measured, 8 the fastest; it and the acceptance checkpoints go by eights
constexpr int kRuleFirst = 8;
static_assert(kRuleFirst % 8 == 0, "groups of eight");
constexpr int kRuleQueue = 64;

// cell range of the site's box in the tet grid (empty range for no box)
struct CellRange {
  int x0, y0, z0, sx, sy, sz;
};

__device__ __forceinline__ CellRange site_cells(const PairParams& p, int i) {
  CellRange r = {0, 0, 0, 0, 0, 0};
  if (p.flags[p.site_base + i] != 1u) return r;
  const float4 blo = p.site_box[2 * i], bhi = p.site_box[2 * i + 1];
  if (!(blo.x <= bhi.x && blo.y <= bhi.y && blo.z <= bhi.z)) return r;
  const Grid& g = p.tg;
  r.x0 = clampi((int)floorf((blo.x - g.lo.x) * g.inv_cell), 0, g.nx - 1);
  r.y0 = clampi((int)floorf((blo.y - g.lo.y) * g.inv_cell), 0, g.ny - 1);
  r.z0 = clampi((int)floorf((blo.z - g.lo.z) * g.inv_cell), 0, g.nz - 1);
  int x1 = clampi((int)floorf((bhi.x - g.lo.x) * g.inv_cell), 0, g.nx - 1);
  int y1 = clampi((int)floorf((bhi.y - g.lo.y) * g.inv_cell), 0, g.ny - 1);
  int z1 = clampi((int)floorf((bhi.z - g.lo.z) * g.inv_cell), 0, g.nz - 1);
  r.sx = x1 - r.x0 + 1;
  r.sy = y1 - r.y0 + 1;
  r.sz = z1 - r.z0 + 1;
  return r;
}

// grid cells of a task: a warp works through a task alone, so few sites need
// short tasks for the other warps to help; every task stages its site's planes
// and list, so many sites want long ones.  Pair stage (ms) with 16 / 32 / 64 /
// 128 / 256 cells: 92 sites 0.17 / 0.17 / 0.19 / 0.21 / 0.22, 10k sites 1.23 /
// 1.05 / 1.04 / 1.12 / 1.29, 50k sites 5.81 / 4.69 / 4.29 / 4.12 / 4.18.
int pair_task_cells(int n_site) {
  return n_site <= 512 ? 16 : (n_site <= 4096 ? 32 : (n_site <= 16384 ? 64 : 128));
}

// tasks per site: its box's grid cells in chunks of task_cells
__global__ void pair_tasks_kernel(PairParams p, int32_t* n_tasks) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n_site) return;
  CellRange r = site_cells(p, i);
  long long n = (long long)r.sx * r.sy * r.sz;
  n_tasks[i] = (int)((n + p.task_cells - 1) / p.task_cells);
}

// The tets' centroids and vertices are read in the order of the grid's items
// (copied there when the grid is filled), so the tets of a cell come in one
// or two lines.  The larger class's tets are searched with the smaller
// class's planes pushed out further and its scaled regions (site_box_kernel):
// 44 bisectors where its own clip took 12, so fewer tets reach the rule.  Pair
// stage of the 1M-tet workload 5.90 -> 5.16 ms with both, 4.6 with tasks by the
// number of sites, 4.12 with the rule's centroid test, the list staged on
// demand and the rule's code in one place (inlined at each of its calls it
// took 6.1: instruction fetches).
// Persistent warps take (site, chunk of its box's cells) tasks from a work
// counter, so a site with a large box is spread over many warps.
__global__ void __launch_bounds__(kPairWarps * 32, kPairBlocks) pairs_kernel(PairParams p,
                                                                const int32_t* task_off,
                                                                unsigned long long* work) {
  __shared__ float4 spl[kPairWarps][kBoxPlanes];
  __shared__ float spn[kPairWarps][kBoxPlanes];  // |normal| of each plane, rounded down
  // the site's neighbours (rule order), and their bisectors about the site
  __shared__ float4 snb[kPairWarps][kPairMaxK];
  __shared__ float4 sbi[kPairWarps][kPairMaxK];
  // places in the item list: tets whose centroid passed, waiting for the
  // rule's first part, and those that passed it, waiting for the rest
  __shared__ int sa_t[kPairWarps][kRuleQueue];
  __shared__ int sq_t[kPairWarps][kRuleQueue];
  // every 8th neighbour r: its key and the smallest site distance |c_m - c_i|
  // (rounded down) of the neighbours from r on
  __shared__ float schk_key[kPairWarps][kPairMaxK / 8];
  __shared__ float schk_d[kPairWarps][kPairMaxK / 8];
  const int lane = threadIdx.x & 31;
  const int wid = threadIdx.x >> 5;
  const long long n_tasks = task_off[p.n_site];
  unsigned int n_cells_seen = 0, n_keep = 0, n_items = 0, n_in = 0;
  for (;;) {
    long long task = 0;
    if (lane == 0) task = (long long)atomicAdd(work, 1ull);
    task = __shfl_sync(0xffffffffu, task, 0);
    if (task >= n_tasks) break;
    // owning site: last i with task_off[i] <= task, 32 places at a time
    int lo = 0, hi = p.n_site - 1;
    while (lo < hi) {
      const int step = (hi - lo + 31) >> 5;
      const int at = lo + (lane + 1) * step;
      const bool below = at <= hi && __ldg(task_off + at) <= task;
      lo += __popc(__ballot_sync(0xffffffffu, below)) * step;
      hi = min(hi, lo + step - 1);
    }
    const int i = lo;
    const int chunk = (int)(task - task_off[i]);
    const CellRange cr = site_cells(p, i);
    const int n_all = cr.sx * cr.sy * cr.sz;
    const int c_begin = chunk * p.task_cells;
    const int n_iter = min(p.task_cells, n_all - c_begin);
    const float4 blo = p.site_box[2 * i], bhi = p.site_box[2 * i + 1];
    // planes of the site's grown cell, each loosened by its own float
    // evaluation error so that the tests below never reject a centroid the
    // exact planes accept
    const int npl = p.site_nplanes[i];
    const float grow = blo.w == 1.f ? 0.f : p.plane_grow;
    float4* pl = spl[wid];
    float* pn = spn[wid];
    __syncwarp();
    for (int q = lane; q < npl; q += 32) {
      float4 e = p.site_planes[(long long)i * kBoxPlanes + q];
      float tol = 4e-6f * ((fabsf(e.x) + fabsf(e.y) + fabsf(e.z)) * p.coord_scale + fabsf(e.w));
      const float nrm = sqrtf(e.x * e.x + e.y * e.y + e.z * e.z);
      // (the region's own planes are pushed out as well, which only accepts
      // more)
      pl[q] = make_float4(e.x, e.y, e.z, e.w + tol + grow * nrm * (1.0f + 1e-5f));
      // bisectors only: the region's box planes (axis-aligned, the mesh box
      // and its margin) were not pushed out (an axis-aligned bisector is
      // left as it is too, which only accepts more)
      const int n_zero = (e.x == 0.f) + (e.y == 0.f) + (e.z == 0.f);
      pn[q] = n_zero >= 2 ? 0.f : nrm * (1.0f - 1e-5f);
    }
    // the tests take the planes two at a time: an odd count gets a plane
    // that every point passes (kBoxPlanes is even, so the slot exists)
    static_assert(kBoxPlanes % 2 == 0, "plane pairs");
    if (lane == 0 && (npl & 1)) {
      pl[npl] = make_float4(0.f, 0.f, 0.f, 1.f);
      pn[npl] = 0.f;
    }
    __syncwarp();
    const float4 si = p.site4f[p.site_base + i];
    const Grid& g = p.tg;
    // the rule is over the whole list; in ascending bisector distance (when
    // the GPU built it) the neighbour that dominates a far tet comes first
    const int32_t* L = (p.rule_nbr ? p.rule_nbr : p.nbr) + (long long)i * p.k;
    float4 *nb = snb[wid], *bi = sbi[wid];
    const int k_staged = min(p.k, kPairMaxK);
    const bool acc_ok = p.rule_keys != nullptr && k_staged == p.k;
    // the list is staged for the first tet that needs it (many tasks' cells
    // hold none)
    bool staged = false;
    auto stage = [&]() {
      staged = true;
      __syncwarp();  // the task before no longer reads its list
      // The rule needs a vertex v with pd_m(v) > pd_i(v).  That difference is
      // 2 (n . (v - c_i) + g), n = c_i - c_m, g = (|n|^2 + w_i - w_m) / 2:
      // linear, so it suffices that the tet's centroid has it above the float
      // error of the rule's own evaluation (accept_err) and of this one -- one
      // plane test instead of four vertices.  What fails it goes through the
      // rule itself.  g is lowered by both errors; a hole (-1) never rejects.
      for (int r = lane; r < ((k_staged + 7) & ~7); r += 32) {
        const int m = r < k_staged ? __ldg(L + r) : -1;
        float4 e = make_float4(0.f, 0.f, 0.f, 1.f), sm = make_float4(0.f, 0.f, 0.f, -INFINITY);
        if (m >= 0) {
          sm = __ldg(p.site4f + m);
          e.x = si.x - sm.x;
          e.y = si.y - sm.y;
          e.z = si.z - sm.z;
          const float n2 = e.x * e.x + e.y * e.y + e.z * e.z;
          const float err = 0.51f * p.accept_err + 3.0f * p.accept_margin * sqrtf(n2) +
                            5e-7f * (n2 + fabsf(si.w) + fabsf(sm.w));
          e.w = 0.5f * ((n2 + si.w) - sm.w) - err;
        }
        bi[r] = e;
        nb[r] = sm;
      }
      __syncwarp();
      // the acceptance checkpoints (distance-ordered lists with keys only)
      if (acc_ok) {
        float carry = INFINITY;
        for (int w = (k_staged - 1) >> 5; w >= 0; --w) {
          const int r = lane + 32 * w;
          float d = INFINITY;  // a hole never rejects
          if (r < k_staged) {
            const float4 e = bi[r];
            if (nb[r].w != -INFINITY)
              d = sqrtf(e.x * e.x + e.y * e.y + e.z * e.z) * (1.0f - 1e-6f);
          }
          // suffix minimum: lane l gets the minimum over lanes >= l
          for (int o = 1; o < 32; o <<= 1) {
            const float t = __shfl_down_sync(0xffffffffu, d, o);
            if (lane + o < 32) d = fminf(d, t);
          }
          d = fminf(d, carry);
          carry = __shfl_sync(0xffffffffu, d, 0);
          if (r < k_staged && (r & 7) == 0) {
            schk_d[wid][r >> 3] = d;
            schk_key[wid][r >> 3] = __ldg(p.rule_keys + (long long)i * p.k + r);
          }
        }
        __syncwarp();
      }
    };
    auto centroid_passes = [&](int r, float3 y) {
      const float4 e = bi[r];
      return __fmaf_rn(e.x, y.x, __fmaf_rn(e.y, y.y, __fmaf_rn(e.z, y.z, e.w))) > 0.f;
    };
    // the rule for neighbour r: a vertex nearer to the site (in power distance)
    auto rule = [&](const float4& sm, const float3* v, const float* pdi) {
      bool hit = false;
      for (int a = 0; a < 4; ++a) hit |= pow_dist(sm, v[a]) > pdi[a];
      return hit;
    };
    auto rule_site = [&](int r) -> float4 {
      if (r < k_staged) return nb[r];
      const int m = __ldg(L + r);
      return m < 0 ? make_float4(0.f, 0.f, 0.f, -INFINITY) : __ldg(p.site4f + m);
    };
    // centroid about the site
    auto middle = [&](const float3* v) {
      return make_float3(0.25f * (v[0].x + v[1].x + v[2].x + v[3].x) - si.x,
                         0.25f * (v[0].y + v[1].y + v[2].y + v[3].y) - si.y,
                         0.25f * (v[0].z + v[1].z + v[2].z + v[3].z) - si.z);
    };
    n_cells_seen += n_iter;
    // half extent of a grid cell, grown for the rounding of the binning
    const float hc = 0.5f * g.cell * (1.0f + 1e-3f) + 1e-6f * p.coord_scale;
    auto cell_at = [&](int idx) -> int {
      idx += c_begin;
      int x = cr.x0 + idx % cr.sx, y = cr.y0 + (idx / cr.sx) % cr.sy, z = cr.z0 + idx / (cr.sx * cr.sy);
      // reject cells lying entirely outside one plane of the grown cell
      float cxm = g.lo.x + ((float)x + 0.5f) * g.cell;
      float cym = g.lo.y + ((float)y + 0.5f) * g.cell;
      float czm = g.lo.z + ((float)z + 0.5f) * g.cell;
      // (the culling tests use FMA: one rounding per term, well inside the
      // planes' loosening; the rule itself keeps the reference's order)
      auto box_max = [&](float4 e, float off) {
        return __fmaf_rn(e.x, cxm, __fmaf_rn(e.y, cym, __fmaf_rn(e.z, czm,
               __fmaf_rn(hc, fabsf(e.x) + fabsf(e.y) + fabsf(e.z), e.w - off))));
      };
      for (int q = 0; q < npl; q += 2)
        if ((box_max(pl[q], 0.f) < 0.f) | (box_max(pl[q + 1], 0.f) < 0.f)) return -1;
      const int cell = x + g.nx * (y + g.ny * z);
      // again with the cell's largest tet radius in place of the class's
      // (the centroid test below, applied to the best centroid in the cell)
      if (p.tcell_rmax) {
        const float shrink =
            fmaxf(p.offset_r - (__ldg(p.tcell_rmax + cell) * (1.0f + 1e-5f) + 1e-6f * p.coord_scale),
                  0.f);
        if (shrink > 0.f) {
          for (int q = 0; q < npl; q += 2)
            if ((box_max(pl[q], shrink * pn[q]) < 0.f) | (box_max(pl[q + 1], shrink * pn[q + 1]) < 0.f))
              return -1;
        }
      }
      ++n_keep;
      return cell;
    };
    // a tet that passed the rule (its place in the item list) becomes a pair
    auto emit = [&](bool pass, int at) {
      uint32_t msk = __ballot_sync(0xffffffffu, pass);
      if (msk) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(p.pair_cursor, (unsigned long long)__popc(msk));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (pass) {
          const int t = __ldg(p.tcell_items + at);
          unsigned long long slot = base + __popc(msk & ((1u << lane) - 1u));
          if ((long long)slot < p.pair_cap)
            p.pair_buf[slot] = make_int2(t + p.tet_base, i + p.site_base);
          atomicAdd(p.tet_count + p.tet_base + t, 1);
        }
      }
    };
    // a queued tet's vertices and their power distances to the site
    auto vertices = [&](int at, float3* v, float* pdi) {
      const float4 q0 = __ldg(p.tcell_xyz + 3ll * at), q1 = __ldg(p.tcell_xyz + 3ll * at + 1),
                   q2 = __ldg(p.tcell_xyz + 3ll * at + 2);
      v[0] = make_float3(q0.x, q0.y, q0.z);
      v[1] = make_float3(q0.w, q1.x, q1.y);
      v[2] = make_float3(q1.z, q1.w, q2.x);
      v[3] = make_float3(q2.y, q2.z, q2.w);
      for (int a = 0; a < 4; ++a) pdi[a] = pow_dist(si, v[a]);
    };
    int* qt = sq_t[wid];
    int qn = 0;  // queued tets (warp-uniform)
    // the first n queued tets, one per lane, against the rest of the list;
    // the others move to the front
    auto drain = [&](int n) {
      bool pass = false;
      int t = -1;
      if (lane < n) {
        float3 v[4];
        float pdi[4];
        t = qt[lane];
        vertices(t, v, pdi);
        pass = true;
        // distance from the site to the tet's nearest vertex, rounded up
        float m2 = INFINITY;
        for (int a = 0; a < 4; ++a) {
          const float dx = v[a].x - si.x, dy = v[a].y - si.y, dz = v[a].z - si.z;
          m2 = fminf(m2, dx * dx + dy * dy + dz * dz);
        }
        const float d_up = sqrtf(m2) * (1.0f + 1e-6f);
        const float3 y = middle(v);
        bool accepted = false;
#pragma unroll 1
        for (int base = kRuleFirst; base < k_staged && pass && !accepted; base += 32) {
          uint32_t fails = 0;
#pragma unroll 1
          for (int o = 0; o < 32 && base + o < k_staged; o += 8) {
            const int r = base + o;
            // pd_m(v) - pd_i(v) = 2 |c_m - c_i| (key_m - (v - c_i).u_m) for
            // the unit direction u_m to m: a vertex within key_m of the site,
            // by more than the float error of the two power distances, has
            // pd_m(v) > pd_i(v) as evaluated; keys ascend along the list
            if (acc_ok) {
              const float g = schk_key[wid][r >> 3] * (1.0f - 64.0f * 5.9604645e-08f) -
                              p.accept_margin - d_up;
              if (g > 0.f && 2.0f * schk_d[wid][r >> 3] * g > p.accept_err) {
                accepted = true;
                break;
              }
            }
#pragma unroll
            for (int x = 0; x < 8; ++x)
              if (!centroid_passes(r + x, y)) fails |= 1u << (o + x);
          }
          while (fails && pass) {
            const int r = base + __ffs(fails) - 1;
            fails &= fails - 1u;
            pass = rule(rule_site(r), v, pdi);
          }
        }
        // (long user lists beyond the staged part)
        for (int r = k_staged; r < p.k && pass; ++r) pass = rule(rule_site(r), v, pdi);
      }
      emit(pass, t);
      __syncwarp();
      const int rest = qn - n;  // < 32: sources n.., targets 0.. do not overlap
      if (lane < rest) qt[lane] = qt[n + lane];
      __syncwarp();
      qn = rest;
    };
    // the first n tets of the centroid queue, one per lane: their vertices,
    // power distances and the rule's first kRuleFirst neighbours; survivors
    // join the drain's queue (qn <= 31 before, so there is room for 32)
    int* qa_t = sa_t[wid];
    int qa = 0;  // tets in the centroid queue (warp-uniform)
    auto first_part = [&](int n) {
      if (!staged) stage();
      bool pass = false, survive = false;
      float3 v[4] = {};
      float pdi[4] = {};
      int t = -1;
      if (lane < n) {
        t = qa_t[lane];
        vertices(t, v, pdi);
        // voronoi.cu:154-193 (holes, -1, never reject: voronoi.cu:171):
        // a candidate iff every neighbour m has a tet vertex where
        // pd_m > pd_i; the order of the neighbours does not matter
        pass = true;
        const float3 y = middle(v);
        uint32_t fails = 0;
#pragma unroll
        for (int x = 0; x < kRuleFirst; ++x)
          if (!centroid_passes(x, y)) fails |= 1u << x;
        while (fails && pass) {
          const int r = __ffs(fails) - 1;
          fails &= fails - 1u;
          pass = rule(rule_site(r), v, pdi);
        }
        if (pass && p.k > kRuleFirst) {
          survive = true;
          pass = false;
        }
      }
      __syncwarp();  // every lane has read its entry
      const int rest = qa - n;  // < 32: sources n.., targets 0.. do not overlap
      if (lane < rest) qa_t[lane] = qa_t[n + lane];
      const uint32_t sv = __ballot_sync(0xffffffffu, survive);
      if (survive) {
        const int pos = qn + __popc(sv & ((1u << lane) - 1u));
        qt[pos] = t;
      }
      qn += __popc(sv);
      emit(pass, t);
      __syncwarp();
      qa = rest;
    };
    for_items<true>(n_iter, cell_at, p.tcell_start, lane, [&](int at, bool valid, bool last) {
      bool in = false;
      if (valid) {
        ++n_items;
        const float4 c = __ldg(p.tcell_cent + at);
        in = c.x >= blo.x && c.x <= bhi.x && c.y >= blo.y && c.y <= bhi.y && c.z >= blo.z &&
             c.z <= bhi.z;
        // A tet passes the rule for neighbour m only if a vertex lies on the
        // site's side of their bisector, so its centroid lies within the
        // tet's own radius of it: the planes were pushed out by the class's
        // largest radius, and each test takes back (R - r_t) |n|, r_t the
        // tet's radius (c.w, a float square root) rounded up and |n| rounded
        // down so that the test only ever accepts more than the exact one
        const float shrink = fmaxf(p.offset_r - (c.w * (1.0f + 1e-5f) + 1e-6f * p.coord_scale), 0.f);
        auto side = [&](int q) {
          const float4 e = pl[q];
          return __fmaf_rn(e.x, c.x, __fmaf_rn(e.y, c.y, __fmaf_rn(e.z, c.z,
                 __fmaf_rn(-shrink, pn[q], e.w))));
        };
        for (int q = 0; q < npl && in; q += 2) in = (side(q) >= 0.f) & (side(q + 1) >= 0.f);
        if (in) ++n_in;
      }
      // (the whole warp from here) the tets that passed join the centroid
      // queue: qa <= 31 before, so there is room for 32 more; the rule then
      // runs on full warps, and in the last call on what is left
      const uint32_t ia = __ballot_sync(0xffffffffu, in);
      if (in) qa_t[qa + __popc(ia & ((1u << lane) - 1u))] = at;
      qa += __popc(ia);
      __syncwarp();
      do {
        if (qa >= 32 || (last && qa > 0)) first_part(min(qa, 32));
        if (qn >= 32 || (last && qa == 0 && qn > 0)) drain(min(qn, 32));
      } while (last && qa + qn > 0);
    });
  }
  if (p.diag) {
    n_keep = __reduce_add_sync(0xffffffffu, n_keep);
    n_items = __reduce_add_sync(0xffffffffu, n_items);
    n_in = __reduce_add_sync(0xffffffffu, n_in);
    if (lane == 0) {
      atomicAdd(p.diag + 0, (unsigned long long)n_cells_seen);
      atomicAdd(p.diag + 1, (unsigned long long)n_keep);
      atomicAdd(p.diag + 2, (unsigned long long)n_items);
      atomicAdd(p.diag + 3, (unsigned long long)n_in);
    }
  }
}

cudaError_t launch_pairs(PairParams p, int32_t* n_tasks, int32_t* task_off,
                         int32_t* scan_tmp, unsigned long long* work, int num_sms,
                         cudaStream_t st) {
  if (p.n_site <= 0) return cudaSuccess;
  p.task_cells = pair_task_cells(p.n_site);
  pair_tasks_kernel<<<(p.n_site + 255) / 256, 256, 0, st>>>(p, n_tasks);
  note_launches(1);
  cudaError_t err = scan_exclusive(n_tasks, task_off, p.n_site, scan_tmp, st);
  if (err != cudaSuccess) return err;
  cudaMemsetAsync(work, 0, sizeof(unsigned long long), st);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pairs_kernel, kPairWarps * 32, 0);
  pairs_kernel<<<num_sms * (per_sm > 0 ? per_sm : 1), kPairWarps * 32, 0, st>>>(p, task_off, work);
  note_launches(1);
  return cudaGetLastError();
}

__global__ void scatter_pairs_kernel(const int2* buf, long long n, const int32_t* offs,
                                     int32_t* fill, int32_t* pair_site) {
  long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  int2 pr = buf[q];
  int slot = atomicAdd(fill + pr.x, 1);
  pair_site[offs[pr.x] + slot] = pr.y;
}

// The sites of each tet in ascending order.  The lists of a warp's 32 tets
// follow one another: it stages them (as many tets at a time as fit) and a lane
// ranks an entry among its tet's, so nothing waits on a chain of stores and the
// lanes stay busy whatever the lists' lengths.  1M tets, 4.05M pairs: 212 us
// with a lane sorting each tet's list in place, 47 here; a list longer than
// the stage is still sorted that way.
constexpr int kCsrWarps = 4;
constexpr int kCsrStage = 1024;
__global__ void __launch_bounds__(kCsrWarps * 32)
    sort_tet_pairs_kernel(int n_tet, const int32_t* offs, int32_t* pair_site, int32_t* pair_tet,
                          int32_t* tet_k) {
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ int32_t stage[kCsrWarps][kCsrStage];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t* const sh = stage[wid];
  const int t0 = (blockIdx.x * kCsrWarps + wid) * 32;
  if (t0 >= n_tet) return;
  const int nt = min(32, n_tet - t0);
  const int b = offs[t0 + min(lane, nt)], e = offs[t0 + min(lane + 1, nt)];
  const int longest = __reduce_max_sync(kAll, e - b);
  if (lane == 0 && longest > __ldcg(tet_k)) atomicMax(tet_k, longest);
  for (int first = 0; first < nt;) {
    const int base = __shfl_sync(kAll, b, first);
    const int fit =
        __popc(__ballot_sync(kAll, lane >= first && lane < nt && e - base <= kCsrStage));
    if (fit == 0) {
      if (lane == first) {
        for (int i = b + 1; i < e; ++i) {
          const int v = pair_site[i];
          int j = i - 1;
          for (; j >= b && pair_site[j] > v; --j) pair_site[j + 1] = pair_site[j];
          pair_site[j + 1] = v;
        }
        for (int i = b; i < e; ++i) pair_tet[i] = t0 + first;
      }
      ++first;
      continue;
    }
    const int n = __shfl_sync(kAll, e, first + fit - 1) - base;
    for (int i = lane; i < n; i += 32) sh[i] = pair_site[base + i];
    __syncwarp();
    for (int i = lane; i - lane < n; i += 32) {
      // the last tet that starts at or before the entry: the one that holds it
      int r = 0;
#pragma unroll
      for (int step = 16; step; step >>= 1) {
        const int at = __shfl_sync(kAll, b, r + step);
        if (at <= base + i) r += step;
      }
      const int lo = __shfl_sync(kAll, b, r) - base, hi = __shfl_sync(kAll, e, r) - base;
      if (i < n) {
        const int v = sh[i];
        int rank = 0;
        for (int j = lo; j < hi; ++j) rank += sh[j] < v || (sh[j] == v && j < i);
        pair_site[base + lo + rank] = v;
        pair_tet[base + i] = t0 + r;
      }
    }
    __syncwarp();
    first += fit;
  }
}

cudaError_t pairs_to_csr(const int2* pair_buf, long long n_pairs, int n_tet,
                         const int32_t* tet_offsets, int32_t* tet_fill, int32_t* pair_site,
                         int32_t* pair_tet, int32_t* tet_k_out, cudaStream_t st) {
  cudaMemsetAsync(tet_fill, 0, sizeof(int32_t) * (size_t)n_tet, st);
  cudaMemsetAsync(tet_k_out, 0, sizeof(int32_t), st);
  if (n_pairs > 0) {
    scatter_pairs_kernel<<<(int)((n_pairs + 255) / 256), 256, 0, st>>>(pair_buf, n_pairs,
                                                                      tet_offsets, tet_fill,
                                                                      pair_site);
    note_launches(1);
  }
  if (n_tet > 0) {
    const int tets = kCsrWarps * 32;
    sort_tet_pairs_kernel<<<(n_tet + tets - 1) / tets, tets, 0, st>>>(n_tet, tet_offsets, pair_site,
                                                                     pair_tet, tet_k_out);
    note_launches(1);
  }
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// compaction
// ------------------------------------------------------------------------
// statuses counted on the way: hist[0..8], 9 other, 10 lost to a full
// payload buffer; uncertified cells
struct CountCells {
  const rpd_cell_header* h;
  unsigned long long* hist;
  unsigned long long* n_uncert;
  static __device__ unsigned int* bins() {
    __shared__ unsigned int sh[12];
    return sh;
  }
  __device__ void begin() const {
    if (threadIdx.x < 12) bins()[threadIdx.x] = 0;
    __syncthreads();
  }
  __device__ bool operator()(long long q) const {
    const int4 v = reinterpret_cast<const int4*>(h + q)[0];
    const int s = v.z;
    atomicAdd(bins() + ((s >= 0 && s <= 8) ? s : (s == kPayloadFull ? 10 : 9)), 1u);
    if (s == kSuccess && (((uint32_t)v.w >> 24) & RPD_CELL_UNCERTIFIED)) atomicAdd(bins() + 11, 1u);
    return s == kSuccess;
  }
  __device__ void end() const {
    __syncthreads();
    const unsigned int* sh = bins();
    if (threadIdx.x < 11 && sh[threadIdx.x])
      atomicAdd(hist + threadIdx.x, (unsigned long long)sh[threadIdx.x]);
    if (threadIdx.x == 11 && n_uncert && sh[11])
      atomicAdd(n_uncert, (unsigned long long)sh[11]);
  }
};

// a test without anything counted on the way
template <class Test>
struct Plain {
  Test test;
  __device__ void begin() const {}
  __device__ bool operator()(long long q) const { return test(q); }
  __device__ void end() const {}
};

struct HasStatus {
  const rpd_cell_header* h;
  int status;
  __device__ bool operator()(long long q) const { return h[q].status == status; }
};
struct IsUncertified {
  const rpd_cell_header* h;
  __device__ bool operator()(long long q) const {
    const int4 v = reinterpret_cast<const int4*>(h + q)[0];
    return v.z == kSuccess && (((uint32_t)v.w >> 24) & RPD_CELL_UNCERTIFIED);
  }
};
struct IsNeeded {
  const unsigned int* need;
  __device__ bool operator()(long long q) const { return need[q] != 0u; }
};

struct PutHeader {
  const rpd_cell_header* h;
  rpd_cell_header* out;
  __device__ void operator()(long long q, long long at) const {
    const int4* a = reinterpret_cast<const int4*>(h + q);
    int4* b = reinterpret_cast<int4*>(out + at);
    b[0] = a[0];
    b[1] = a[1];
  }
};
struct PutIndex {
  int32_t* idx;
  __device__ void operator()(long long q, long long at) const { idx[at] = (int32_t)q; }
};

cudaError_t compact_cells(const rpd_cell_header* pair_headers, long long n_pairs,
                          int32_t* scan_tmp, rpd_cell_header* out, long long* n_out_dev,
                          unsigned long long* status_hist, cudaStream_t st,
                          unsigned long long* n_uncert) {
  return keep_indices(CountCells{pair_headers, status_hist, n_uncert},
                      HasStatus{pair_headers, kSuccess}, PutHeader{pair_headers, out}, n_pairs,
                      scan_tmp, n_out_dev, st);
}

cudaError_t select_pairs(const rpd_cell_header* h, long long n, int status, int32_t* scan_tmp,
                         int32_t* idx_out, int32_t* count_out, cudaStream_t st) {
  const HasStatus t{h, status};
  return keep_indices(Plain<HasStatus>{t}, t, PutIndex{idx_out}, n, scan_tmp, count_out, st);
}

cudaError_t select_uncertified(const rpd_cell_header* h, long long n, int32_t* scan_tmp,
                               int32_t* idx_out, int32_t* count_out, cudaStream_t st) {
  const IsUncertified t{h};
  return keep_indices(Plain<IsUncertified>{t}, t, PutIndex{idx_out}, n, scan_tmp, count_out, st);
}

cudaError_t select_sites(const unsigned int* site_need, int n, int32_t* scan_tmp,
                         int32_t* idx_out, int32_t* count_out, cudaStream_t st) {
  const IsNeeded t{site_need};
  return keep_indices(Plain<IsNeeded>{t}, t, PutIndex{idx_out}, (long long)n, scan_tmp, count_out,
                      st);
}

__global__ void assign_rows_kernel(const int32_t* sites, int n, int row0, long long off0,
                                   int stride, int32_t* site_row, long long* ext_off) {
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f < n) {
    site_row[sites[f]] = row0 + f;
    ext_off[row0 + f] = off0 + (long long)f * stride;
  }
}

cudaError_t assign_rows(const int32_t* sites, int n, int row0, long long off0, int stride,
                        int32_t* site_row, long long* ext_off, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  assign_rows_kernel<<<(n + 255) / 256, 256, 0, st>>>(sites, n, row0, off0, stride, site_row,
                                                      ext_off);
  note_launches(1);
  return cudaGetLastError();
}

// complete rows: one shared list of every site (ids 0..n_site-1, the seed
// itself included: its bisector is the zero plane, which clips nothing) at
// ext_nbr[off..off + n_site), and rows row0 + f of the sites sites[f] on it
__global__ void complete_rows_kernel(const int32_t* sites, int n, int row0, long long off,
                                     int n_site, int32_t* site_row, long long* ext_off,
                                     int32_t* ext_len, float* ext_bound, int32_t* ext_nbr,
                                     const int2* site_range) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_site) ext_nbr[off + i] = i;
  if (i < n) {
    const int s = sites[i];
    const int2 r = site_range ? site_range[s] : make_int2(0, n_site);
    site_row[s] = row0 + i;
    ext_off[row0 + i] = off + r.x;
    ext_len[row0 + i] = r.y - r.x;
    ext_bound[row0 + i] = INFINITY;
  }
}

cudaError_t complete_rows(const int32_t* sites, int n, int row0, long long off, int n_site,
                          int32_t* site_row, long long* ext_off, int32_t* ext_len,
                          float* ext_bound, int32_t* ext_nbr, cudaStream_t st,
                          const int2* site_range) {
  const int m = n > n_site ? n : n_site;
  if (m <= 0) return cudaSuccess;
  complete_rows_kernel<<<(m + 255) / 256, 256, 0, st>>>(sites, n, row0, off, n_site, site_row,
                                                        ext_off, ext_len, ext_bound, ext_nbr,
                                                        site_range);
  note_launches(1);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// reference site_knn layout ((k+1) rows x n_site) -> row-major lists
// ------------------------------------------------------------------------
__global__ void ref_lists_kernel(const int32_t* ref, int k, int n_site, int32_t* nbr) {
  long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (long long)n_site * k) return;
  int i = (int)(q / k), r = (int)(q % k);
  nbr[q] = ref[(long long)r * n_site + i];
}

cudaError_t neighbors_from_reference(const int32_t* ref, int k, int n_site, int32_t* nbr,
                                     cudaStream_t st) {
  long long n = (long long)n_site * k;
  if (n > 0) {
    ref_lists_kernel<<<(int)((n + 255) / 256), 256, 0, st>>>(ref, k, n_site, nbr);
    note_launches(1);
  }
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// batches of meshes
// ------------------------------------------------------------------------
// first compacted cell of every mesh: cells are in ascending tet id and the
// meshes' tets are consecutive ranges starting at tet_base[m]
__global__ void mesh_cell_ranges_kernel(const rpd_cell_header* cells, const long long* n_cells,
                                        const int32_t* tet_base, int n_mesh, long long* first) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m > n_mesh) return;
  const long long n = *n_cells;
  if (m == n_mesh) {
    first[m] = n;
    return;
  }
  const int key = tet_base[m];
  long long lo = 0, hi = n;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (cells[mid].tet_id < key) lo = mid + 1;
    else hi = mid;
  }
  first[m] = lo;
}

cudaError_t mesh_cell_ranges(const rpd_cell_header* cells, const long long* n_cells,
                             const int32_t* tet_base, int n_mesh, long long* first,
                             cudaStream_t st) {
  mesh_cell_ranges_kernel<<<(n_mesh + 1 + 127) / 128, 128, 0, st>>>(cells, n_cells, tet_base,
                                                                     n_mesh, first);
  note_launches(1);
  return cudaGetLastError();
}

// records of cells [0, n) copied to consecutive offsets new_off[q] of out,
// with mesh-local ids: tet - tet_base, site - site_base in the headers and
// in the site pairs of the bisector planes (planes 4.. of a record)
__global__ void gather_records_kernel(const rpd_cell_header* cells, long long n,
                                      const unsigned long long* new_off, const uint8_t* payload,
                                      int tet_base, int site_base, rpd_cell_header* hout,
                                      uint8_t* out) {
  const int lane = threadIdx.x & 31;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long q = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < n; q += n_warps) {
    rpd_cell_header h = cells[q];
    const PayloadLayout L(h.nb_v, h.nb_p, h.nb_e);
    const uint4* src = reinterpret_cast<const uint4*>(payload + h.offset);
    uint4* dst = reinterpret_cast<uint4*>(out + new_off[q]);
    for (uint32_t i = lane; i < L.total / 16u; i += 32) dst[i] = src[i];
    __syncwarp();
    int2* id2 = reinterpret_cast<int2*>(out + new_off[q] + L.id2);
    for (int i = 4 + lane; i < h.nb_p; i += 32) {
      int2 v = id2[i];
      id2[i] = make_int2(v.x - site_base, v.y - site_base);
    }
    if (lane == 0) {
      h.tet_id -= tet_base;
      h.site_id -= site_base;
      h.offset = new_off[q];
      hout[q] = h;
    }
  }
}

cudaError_t gather_records(const rpd_cell_header* cells, long long n,
                           const unsigned long long* new_off, const uint8_t* payload,
                           int tet_base, int site_base, rpd_cell_header* hout, uint8_t* out,
                           cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  long long blocks = (n + 7) / 8;
  if (blocks > 65535) blocks = 65535;
  gather_records_kernel<<<(unsigned)blocks, 256, 0, st>>>(cells, n, new_off, payload, tet_base,
                                                          site_base, hout, out);
  note_launches(1);
  return cudaGetLastError();
}

// record sizes of cells [0, n) (for the offsets of a gather)
__global__ void record_sizes_kernel(const rpd_cell_header* cells, long long n,
                                    unsigned long long* size) {
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const rpd_cell_header h = cells[q];
  size[q] = PayloadLayout(h.nb_v, h.nb_p, h.nb_e).total;
}

cudaError_t record_sizes(const rpd_cell_header* cells, long long n, unsigned long long* size,
                         cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  record_sizes_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(cells, n, size);
  note_launches(1);
  return cudaGetLastError();
}

}  // namespace rpd
