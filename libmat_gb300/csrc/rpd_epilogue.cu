// rpd_epilogue.cu -- coordinates, volume and topology hash of the emitted
// cells, from their records (plane ids and dual triangles), and the tets'
// face planes in double-float.
//
// The clip kernels leave these to a pass of their own: it keeps their code
// (and its instruction-cache footprint) to the topology update.  Compiled
// with -fmad=false: the double-float arithmetic and the reference's FP32
// volume expressions are evaluated one rounding at a time, FMA where written.

#include <cuda_runtime.h>

#include <algorithm>

#include "rpd_clip_pred.cuh"
#include "rpd_common.cuh"
#include "rpd_df64.cuh"
#include "rpd_kernels.cuh"

namespace rpd {

// ------------------------------------------------------------------------
// FP64-accurate reconstruction of the emitted cell
// ------------------------------------------------------------------------
// The clip kernels' float planes decide the topology exactly as the reference does.
// The coordinates reported for the surviving vertices are rebuilt from the
// FP64 inputs instead: every plane is recomputed in the frame centred on the
// seed S, from double-float copies of the FP64 mesh vertices and sites
// (hi + lo, about 48 bits), and each vertex -- the intersection of its three
// planes, by Cramer's rule as in compute_vertex_coordinates
// (convex_cell.cu:319-351) -- is solved in double-float arithmetic on the
// FP32 pipe, then translated back by S and rounded to FP64 with one FP64
// add.  The cell volume uses the reference's per-vertex decomposition into
// six tets (convex_cell.cu:986-1069) in FP32, about a point of the cell
// (small coordinates, no cancellation against the scene's extent).

__device__ __forceinline__ float3 f3sub(float3 a, float3 b) {
  return make_float3(a.x - b.x, a.y - b.y, a.z - b.z);
}
__device__ __forceinline__ float f3dot(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 f3cross(float3 a, float3 b) {
  return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float3 f3axpy(float a, float3 x, float3 y) {
  return make_float3(a * x.x + y.x, a * x.y + y.y, a * x.z + y.z);
}
__device__ __forceinline__ float det3f(float3 a, float3 b, float3 c) { return f3dot(a, f3cross(b, c)); }

// foot of the origin O = (0,0,0) on the plane n.x + d = 0
__device__ __forceinline__ float3 face_foot(float3 n, float d) {
  const float n2 = f3dot(n, n);
  const float lam = n2 > 0.f ? __fdividef(d, n2) : 0.f;
  return make_float3(-lam * n.x, -lam * n.y, -lam * n.z);
}

// signed volume of one vertex's six flag tets, origin O = (0,0,0): feet of
// O on the three faces (given) and on the three edge lines through A.  The
// volume is reported in FP32, so the quotients use the fast division.
__device__ float vertex_volume_f(float3 A, const float3* n, const float3* foot) {
  float3 P[6];
  for (int i = 0; i < 3; ++i) P[2 * i] = foot[i];
  for (int i = 0; i < 3; ++i) {
    float3 t = f3cross(n[i], n[(i + 1) % 3]);
    float t2 = f3dot(t, t);
    float lam = t2 > 0.f ? __fdividef(f3dot(t, A), t2) : 0.f;
    P[2 * i + 1] = f3axpy(-lam, t, A);
  }
  float3 mA = make_float3(-A.x, -A.y, -A.z);
  float v = 0.f;
  for (int i = 0; i < 6; ++i) v -= det3f(f3sub(P[i], A), f3sub(P[(i + 1) % 6], A), mA);
  return v * (1.0f / 6.0f);
}

__device__ __forceinline__ df ldf(const float2* p) {
  const float2 v = __ldg(p);
  return df_make(v.x, v.y);
}

// exact float -> double widening with integer operations (IEEE-754 binary32
// to binary64: same sign, exponent re-biased by 1023 - 127, fraction shifted
// by 29 bits); zeros, subnormals, infinities and NaNs take the conversion
// instruction
__device__ __forceinline__ double widen(float f) {
  const uint32_t u = __float_as_uint(f);
  const uint32_t e = (u >> 23) & 0xffu;
  if (e == 0u || e == 0xffu) return (double)f;
  const uint64_t bits = ((uint64_t)(u >> 31) << 63) | ((uint64_t)(e + 896u) << 52) |
                        ((uint64_t)(u & 0x7fffffu) << 29);
  return __longlong_as_double((long long)bits);
}

// S + X (double-float) rounded to double: hi and lo widen exactly, one add
__device__ __forceinline__ double df_translate(df S, df X) {
  const df t = df_add_s(S, X);
  return widen(t.hi) + widen(t.lo);
}

// canonical topology of a cell, independent of the clipping order: the sum
// over its vertices of a hash of the sorted face keys (clip_id2) of the
// vertex's three planes and its #adjacent cells (splitmix64 mixing, Steele,
// Lea and Flood, OOPSLA 2014).  Planes that clipped intermediate vertices and
// no longer bound the cell appear in no vertex, so they do not count.
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ uint64_t face_key(int2 id) {
  return ((uint64_t)(uint32_t)id.x << 32) | (uint32_t)id.y;
}

// the hash of one vertex: its planes' face keys and its #adjacent cells
__device__ __forceinline__ uint64_t vertex_hash(int2 ia, int2 ib, int2 ic, uint8_t adj) {
  uint64_t a = face_key(ia), b = face_key(ib), d = face_key(ic), x;
  if (a > b) { x = a; a = b; b = x; }
  if (b > d) { x = b; b = d; d = x; }
  if (a > b) { x = a; a = b; b = x; }
  uint64_t hv = mix64(a);
  hv = mix64(hv ^ b);
  hv = mix64(hv ^ d);
  return mix64(hv ^ (uint64_t)adj);
}

// ------------------------------------------------------------------------
// the epilogue kernel
// ------------------------------------------------------------------------
// A warp takes 16 pairs and lays their cells' planes, then their vertices,
// out over its 32 lanes, whichever cell each belongs to: a cell has about
// seven of either, so a half-warp per cell kept 14 of 32 lanes busy.  The
// work is issue-bound (FMA pipe: about 100 instructions a plane and 500 a
// vertex in double-float).  1M-tet workload (3.35M cells): 2.85 ms a
// half-warp per cell, 1.43 ms here; 200k tets
// (750k cells, with hashes) 0.72 and 0.40.
constexpr int kEpiWarps = 4;
constexpr int kEpiCells = 16;
constexpr int kEpiP = 128;  // planes and vertices laid out at a time (any cell
constexpr int kEpiV = 128;  // has at most kMaxP and kMaxT of them)
static_assert(kEpiP >= kMaxP && kEpiV >= kMaxT, "a cell fits");

// seed-frame planes (nx, ny | nz, d as double-float), the feet of the volume
// origin on them, their ids, and the vertices' volumes
struct EpiStore {
  float4 xy[kEpiP];
  float4 zd[kEpiP];
  float4 foot[kEpiP];
  int2 id2[kEpiP];
  float vol[kEpiV];
};

struct EpiPlane {
  df x, y, z, d;
};
__device__ __forceinline__ EpiPlane epi_plane(const EpiStore& w, int i) {
  const float4 a = w.xy[i], b = w.zd[i];
  return {df_make(a.x, a.y), df_make(a.z, a.w), df_make(b.x, b.y), df_make(b.z, b.w)};
}

// vertex (X, Y, Z) of three planes
__device__ __forceinline__ void epi_vertex(const EpiPlane& a, const EpiPlane& b, const EpiPlane& c,
                                           df& X, df& Y, df& Z) {
  const df mxy = minor2(b.x, b.y, c.x, c.y), mxz = minor2(b.x, b.z, c.x, c.z),
           mxw = minor2(b.x, b.d, c.x, c.d);
  const df myz = minor2(b.y, b.z, c.y, c.z), myw = minor2(b.y, b.d, c.y, c.d),
           mzw = minor2(b.z, b.d, c.z, c.d);
  const df Dw = df_add_s(df_sub_s(df_mul(a.x, myz), df_mul(a.y, mxz)), df_mul(a.z, mxy));
  const df Dx = df_add_s(df_sub_s(df_mul(a.y, mzw), df_mul(a.z, myw)), df_mul(a.d, myz));
  const df Dy = df_add_s(df_sub_s(df_mul(a.x, mzw), df_mul(a.z, mxw)), df_mul(a.d, mxz));
  const df Dz = df_add_s(df_sub_s(df_mul(a.x, myw), df_mul(a.y, mxw)), df_mul(a.d, mxy));
  const df inv = df_recip(Dw);
  X = df_neg(df_mul(Dx, inv));
  Y = df_mul(Dy, inv);
  Z = df_neg(df_mul(Dz, inv));
}

// float intersection of three planes (Cramer); used only as the origin of
// the volume decomposition, so any point near the cell will do
__device__ __forceinline__ float3 epi_origin(const EpiPlane& a, const EpiPlane& b,
                                             const EpiPlane& c) {
  // n_k . x = -d_k
  const float3 n0 = make_float3(a.x.hi, a.y.hi, a.z.hi);
  const float3 n1 = make_float3(b.x.hi, b.y.hi, b.z.hi);
  const float3 n2 = make_float3(c.x.hi, c.y.hi, c.z.hi);
  const float3 c12 = f3cross(n1, n2), c20 = f3cross(n2, n0), c01 = f3cross(n0, n1);
  const float s = -1.0f / f3dot(n0, c12);
  const float3 x = make_float3(s * (a.d.hi * c12.x + b.d.hi * c20.x + c.d.hi * c01.x),
                               s * (a.d.hi * c12.y + b.d.hi * c20.y + c.d.hi * c01.y),
                               s * (a.d.hi * c12.z + b.d.hi * c20.z + c.d.hi * c01.z));
  if (!(isfinite(x.x) && isfinite(x.y) && isfinite(x.z))) return make_float3(0.f, 0.f, 0.f);
  return x;
}

__global__ void __launch_bounds__(kEpiWarps * 32) cell_epilogue_kernel(EpilogueParams p,
                                                                       int cells) {
  constexpr uint32_t kAll = 0xffffffffu;
  __shared__ EpiStore store[kEpiWarps];
  const int lane = threadIdx.x & 31;
  EpiStore& w = store[threadIdx.x >> 5];
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long base = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * cells;
       base < p.n_pairs; base += cells * n_warps) {
    // lane l < cells (<= 16) holds pair base + l
    const long long q = base + lane;
    int tet = 0, sid = 0, np = 0, nv = 0, ne = 0;
    uint8_t* rec = p.payload;
    bool emitted = false;
    if (lane < cells && q < p.n_pairs) {
      const int4* hd = reinterpret_cast<const int4*>(p.headers + q);
      const int4 h0 = hd[0], h1 = hd[1];
      emitted = h0.z == kSuccess;
      if (emitted) {
        tet = h0.x;
        sid = h0.y;
        nv = h0.w & 255;
        np = (h0.w >> 8) & 255;
        ne = (h0.w >> 16) & 255;
        rec += (unsigned long long)(uint32_t)h1.x | ((unsigned long long)(uint32_t)h1.y << 32);
      } else if (p.topo_hash) {
        p.topo_hash[q] = 0ull;
      }
    }
    if (!p.geometry && emitted) {
      double* xyz = reinterpret_cast<double*>(rec + PayloadLayout(nv, np, ne).xyz);
      for (int i = 0; i < 3 * nv; ++i) xyz[i] = 0.0;
      p.headers[q].volume = 0.0;
    }
    if (!p.geometry && !p.topo_hash) continue;
    // as many of the cells at a time as the store holds
    uint32_t todo = __ballot_sync(kAll, emitted);
    while (todo) {
      const bool mine = (todo >> lane) & 1u;
      const uint32_t need = mine ? (uint32_t)np | ((uint32_t)nv << 16) : 0u;
      uint32_t incl = need;
      for (int o = 1; o < kEpiCells; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kAll, incl, o);
        if (lane >= o) incl += y;
      }
      const bool take = mine && (incl & 0xffffu) <= kEpiP && (incl >> 16) <= kEpiV;
      const uint32_t taken = __ballot_sync(kAll, take);  // a prefix of todo
      todo &= ~taken;
      const uint32_t total = __shfl_sync(kAll, incl, 31 - __clz((int)taken));
      const int n_p = (int)(total & 0xffffu), n_v = (int)(total >> 16);
      // first plane and vertex of each cell (those not taken: past the end)
      const int p0 = take ? (int)((incl - need) & 0xffffu) : (mine ? n_p : min((int)(incl & 0xffffu), n_p));
      const int v0 = take ? (int)((incl - need) >> 16) : (mine ? n_v : min((int)(incl >> 16), n_v));
      // the last cell whose first item is at most `item`
      auto owner = [&](int first, int item) {
        int own = 0;
#pragma unroll
        for (int o = kEpiCells / 2; o > 0; o >>= 1)
          if (__shfl_sync(kAll, first, own + o) <= item) own += o;
        return own;
      };
      const unsigned long long rec_bits = (unsigned long long)rec;
      auto record = [&](int own) {
        const uint32_t lo = __shfl_sync(kAll, (uint32_t)rec_bits, own);
        const uint32_t hi = __shfl_sync(kAll, (uint32_t)(rec_bits >> 32), own);
        return reinterpret_cast<uint8_t*>(((unsigned long long)hi << 32) | lo);
      };

      // ---- planes in the seed frame
      for (int b = 0; b < n_p; b += 32) {
        const int item = b + lane;
        const int own = owner(p0, item);
        const int i = item - __shfl_sync(kAll, p0, own);
        const int os = __shfl_sync(kAll, sid, own), ot = __shfl_sync(kAll, tet, own);
        const int onp = __shfl_sync(kAll, np, own);
        const uint8_t* r = record(own);
        if (item < n_p) {
          const int2 id = reinterpret_cast<const int2*>(r + 16 * onp)[i];
          w.id2[item] = id;
          if (p.geometry) {
            const float2* S2 = p.site2 + 4 * (long long)os;
            const df Sx = ldf(S2), Sy = ldf(S2 + 1), Sz = ldf(S2 + 2);
            df nx, ny, nz, d;
            if (i < 4) {
              // the tet's face plane (FP64, once per mesh), moved to the seed
              // frame: d' = d + n . S
              const float2* f = p.face2 + 16 * (long long)ot + 4 * i;
              nx = ldf(f);
              ny = ldf(f + 1);
              nz = ldf(f + 2);
              d = df_add_s(ldf(f + 3),
                           df_add_s(df_add_s(df_mul(nx, Sx), df_mul(ny, Sy)), df_mul(nz, Sz)));
            } else {
              const df Sw = ldf(S2 + 3);
              const float2* B = p.site2 + 4 * (long long)(id.x == os ? id.y : id.x);
              // bisector in the seed frame: n = S - B, d = (|n|^2 + wS - wB) / 2
              nx = df_sub_s(Sx, ldf(B));
              ny = df_sub_s(Sy, ldf(B + 1));
              nz = df_sub_s(Sz, ldf(B + 2));
              const df n2 = df_add_s(df_add_s(df_mul(nx, nx), df_mul(ny, ny)), df_mul(nz, nz));
              d = df_add_s(n2, df_sub_s(Sw, ldf(B + 3)));
              d = df_make(0.5f * d.hi, 0.5f * d.lo);
            }
            w.xy[item] = make_float4(nx.hi, nx.lo, ny.hi, ny.lo);
            w.zd[item] = make_float4(nz.hi, nz.lo, d.hi, d.lo);
          }
        }
      }
      __syncwarp();
      if (p.geometry) {
        // ---- volume origin O near the cell (its vertex 0, in float): the
        // decomposition's terms then scale with the cell's own size
        float3 O = make_float3(0.f, 0.f, 0.f);
        if (take) {
          const uchar4 tr = *reinterpret_cast<const uchar4*>(rec + 16 * np + al16(8u * np));
          O = epi_origin(epi_plane(w, p0 + tr.x), epi_plane(w, p0 + tr.y), epi_plane(w, p0 + tr.z));
        }
        for (int b = 0; b < n_p; b += 32) {
          const int item = b + lane;
          const int own = owner(p0, item);
          const float ox = __shfl_sync(kAll, O.x, own), oy = __shfl_sync(kAll, O.y, own),
                      oz = __shfl_sync(kAll, O.z, own);
          if (item < n_p) {
            const EpiPlane a = epi_plane(w, item);
            const df dc = df_add_s(a.d, df_add_s(df_add_s(df_mul(a.x, df_make(ox, 0.f)),
                                                          df_mul(a.y, df_make(oy, 0.f))),
                                                 df_mul(a.z, df_make(oz, 0.f))));
            const float3 f = face_foot(make_float3(a.x.hi, a.y.hi, a.z.hi), dc.hi);
            w.foot[item] = make_float4(f.x, f.y, f.z, 0.f);
          }
        }
        __syncwarp();
        // ---- vertices
        for (int b = 0; b < n_v; b += 32) {
          const int item = b + lane;
          const int own = owner(v0, item);
          const int v = item - __shfl_sync(kAll, v0, own);
          const int op = __shfl_sync(kAll, p0, own), os = __shfl_sync(kAll, sid, own);
          const int onp = __shfl_sync(kAll, np, own), onv = __shfl_sync(kAll, nv, own),
                    one = __shfl_sync(kAll, ne, own);
          const float3 oo = make_float3(__shfl_sync(kAll, O.x, own), __shfl_sync(kAll, O.y, own),
                                        __shfl_sync(kAll, O.z, own));
          uint8_t* r = record(own);
          if (item < n_v) {
            const PayloadLayout L(onv, onp, one);
            const uchar4 tr = reinterpret_cast<const uchar4*>(r + L.ver)[v];
            const int pl[3] = {op + tr.x, op + tr.y, op + tr.z};
            df X, Y, Z;
            float3 nn[3], ft[3];
            {
              const EpiPlane a = epi_plane(w, pl[0]), c = epi_plane(w, pl[1]),
                             e = epi_plane(w, pl[2]);
              epi_vertex(a, c, e, X, Y, Z);
              nn[0] = make_float3(a.x.hi, a.y.hi, a.z.hi);
              nn[1] = make_float3(c.x.hi, c.y.hi, c.z.hi);
              nn[2] = make_float3(e.x.hi, e.y.hi, e.z.hi);
            }
            const float2* S2 = p.site2 + 4 * (long long)os;
            double* xyz = reinterpret_cast<double*>(r + L.xyz) + 3 * v;
            xyz[0] = df_translate(ldf(S2), X);
            xyz[1] = df_translate(ldf(S2 + 1), Y);
            xyz[2] = df_translate(ldf(S2 + 2), Z);
            const float3 A = make_float3(df_sub_s(X, df_make(oo.x, 0.f)).hi,
                                         df_sub_s(Y, df_make(oo.y, 0.f)).hi,
                                         df_sub_s(Z, df_make(oo.z, 0.f)).hi);
            for (int k = 0; k < 3; ++k) {
              const float4 f = w.foot[pl[k]];
              ft[k] = make_float3(f.x, f.y, f.z);
            }
            w.vol[item] = vertex_volume_f(A, nn, ft);
          }
        }
        __syncwarp();
        // ---- the cell's volume: 16 partial sums (vertices i, i + 16, ...)
        // added pairwise
        if (take) {
          float s[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) s[i] = i < nv ? 0.f + w.vol[v0 + i] : 0.f;
          for (int b = 16; b < nv; b += 16) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (b + i < nv) s[i] += w.vol[v0 + b + i];
          }
#pragma unroll
          for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < o; ++i) s[i] += s[i + o];
          p.headers[q].volume = (double)s[0];
        }
      }
      if (p.topo_hash) {
        // ---- topology hashes: the vertices' terms over the planes' place
        __syncwarp();
        uint64_t* term = reinterpret_cast<uint64_t*>(w.xy);
        static_assert(sizeof(uint64_t) * kEpiV <= sizeof(w.xy), "hash terms fit");
        for (int b = 0; b < n_v; b += 32) {
          const int item = b + lane;
          const int own = owner(v0, item);
          const int v = item - __shfl_sync(kAll, v0, own);
          const int op = __shfl_sync(kAll, p0, own), onp = __shfl_sync(kAll, np, own);
          const uint8_t* r = record(own);
          if (item < n_v) {
            const uchar4 t = reinterpret_cast<const uchar4*>(r + 16 * onp + al16(8u * onp))[v];
            term[item] = vertex_hash(w.id2[op + t.x], w.id2[op + t.y], w.id2[op + t.z], t.w);
          }
        }
        __syncwarp();
        if (take) {
          uint64_t h = 0;
          for (int v = 0; v < nv; ++v) h += term[v0 + v];
          p.topo_hash[q] = h;
        }
      }
      __syncwarp();
    }
  }
}

cudaError_t launch_cell_epilogue(const EpilogueParams& p, int num_sms, cudaStream_t st) {
  if (p.n_pairs <= 0) return cudaSuccess;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cell_epilogue_kernel, kEpiWarps * 32, 0);
  if (per_sm < 1) per_sm = 1;
  // few pairs: fewer cells a warp, on more warps
  const long long warps = (long long)num_sms * per_sm * kEpiWarps;
  const int cells = (int)std::min<long long>(kEpiCells, (p.n_pairs + warps - 1) / warps);
  const long long want = (p.n_pairs + cells * kEpiWarps - 1) / (cells * kEpiWarps);
  const long long blocks = std::min<long long>((long long)num_sms * per_sm * 4, want);
  cell_epilogue_kernel<<<(unsigned)blocks, kEpiWarps * 32, 0, st>>>(p, cells);
  note_launches(1);
  return cudaGetLastError();
}

// face planes of every tet in FP64 (inward normals as tri2plane,
// common_cuda.h:248-254: n = (b - a) x (e - a), d = -a . n), stored as
// double-float (nx, ny, nz, d) per face
__global__ void tet_face_planes_kernel(const double* vert, const int4* tets, int n_tet, float2* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tet) return;
  const int4 q = tets[t];
  const int id[4] = {q.x, q.y, q.z, q.w};
  for (int i = 0; i < 4; ++i) {
    const double* a = vert + 3 * (long long)id[cFaceLv[i][0]];
    const double* b = vert + 3 * (long long)id[cFaceLv[i][1]];
    const double* e = vert + 3 * (long long)id[cFaceLv[i][2]];
    const double ux = b[0] - a[0], uy = b[1] - a[1], uz = b[2] - a[2];
    const double vx = e[0] - a[0], vy = e[1] - a[1], vz = e[2] - a[2];
    const double nx = uy * vz - uz * vy, ny = uz * vx - ux * vz, nz = ux * vy - uy * vx;
    const double d = -(a[0] * nx + a[1] * ny + a[2] * nz);
    const double v[4] = {nx, ny, nz, d};
    for (int k = 0; k < 4; ++k) {
      const df x = df_from_double(v[k]);
      out[16ll * t + 4 * i + k] = make_float2(x.hi, x.lo);
    }
  }
}

cudaError_t launch_tet_face_planes(const double* vert3d, const int4* tets, int n_tet, float2* out,
                                   cudaStream_t st) {
  if (n_tet <= 0) return cudaSuccess;
  tet_face_planes_kernel<<<(n_tet + 255) / 256, 256, 0, st>>>(vert3d, tets, n_tet, out);
  note_launches(1);
  return cudaGetLastError();
}

}  // namespace rpd
