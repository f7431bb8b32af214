// rpd_clip_thread.cu -- clipping of small cells, one thread per cell.
//
// The cells of a tet mesh finer than the sites are small (1M tets / 50k
// sites: 6.9 planes and 6.9 vertices, 3.0 clips, 27 list entries until the
// certificate holds), so a warp per cell (clip_cells_kernel) leaves most
// lanes idle in most instructions: 3,959 warp instructions a pair.  Here a
// lane owns a cell and runs the reference's sequential update on it; a cell
// that outgrows the lane's storage goes to a list that clip_cells_kernel
// takes up from its tet again.  The records are the reference's, byte for
// byte, as clip_cells_kernel's are (see rpd_clip.cu for the reference's
// lines).
//
// Measured (1M tets, 50k sites, 4.05M pairs, certified lists of 128): 18.2 ms
// a warp per cell, 5.4 ms here with the 1.1 % of the pairs that go back.  What
// bounds it is issue and latency: the phases run with 12 to 20 of 32 lanes, and
// twelve warps an SM hide only part of the shared-memory and list loads.
//
// State: 576 bytes a cell in shared memory, each lane in banks of its own
// (a float4 of slot s lies at 16 (32 s + lane)), so indices that differ from
// lane to lane cost nothing.  Twelve warps fit an SM.
//
// Control: each lane is a state machine -- cull a group of four list entries,
// test a candidate plane against the vertices, clip, emit -- and the warp
// takes a phase when enough lanes wait for it; finished lanes are refilled
// from the queue, so short and long cells share a warp.
//
// Predicates: a vertex keeps its position x' about the tet's centroid c and
// a bound eps of its error (from its cofactors and their permanents, the
// filter's bounds).  With w' = n.c + w, a plane's value at the vertex is
// w' + n.x' to within |n| eps + tol.  If that decides the sign, the sign is
// the reference's determinant's (det4x4 = K_w times the value, K_w < 0
// certain; eps holds 6u of every permanent term where the FP32 evaluation
// takes 5u, far above the FP64 determinant's own error); if not, the
// cofactor filter, and after it FP64 or the exact sign, decides.  A plane
// that leaves the box of the vertices (eps included) on its inner side by
// more than tol conflicts with none of them: most of the list ends there.

#include <cuda_runtime.h>

#include <algorithm>

#include "rpd_clip_box.cuh"
#include "rpd_clip_pred.cuh"
#include "rpd_common.cuh"
#include "rpd_kernels.cuh"

namespace rpd {

namespace {

constexpr int kTP = 14;  // planes, vertices and edges of a lane's cell
constexpr int kTV = 16;
constexpr int kTE = 40;
constexpr int kTWarps = 4;
constexpr int kTBlocks = 3;  // per SM
static_assert(kTP <= 16 && kTV <= 16, "plane ids are 4 bits, conflict masks 16");

struct WarpStore {
  float4 pl[kTP][32];
  float4 vx[kTV][32];  // x', and packed: planes 4 x 3 bits, #adjacent 8, eps 12
  int32_t id[kTP - 4][32];  // the other site of each bisector
  uint32_t ed[kTE / 4][32];  // edges: two plane ids, 4 bits each
  uint32_t next[4][32];      // a cavity's boundary: the plane after each plane
};

// eps as the upper 12 bits of its (non-negative) float, rounded up
constexpr uint32_t kEpsInf = 0xff0u;
__device__ __forceinline__ uint32_t eps_code(float e) {
  const uint32_t u = (__float_as_uint(e) + 0x7ffffu) >> 19;
  return e < 1e30f ? u : kEpsInf;
}
__device__ __forceinline__ float eps_of(float packed) {
  return __uint_as_float((__float_as_uint(packed) >> 20) << 19);
}
__device__ __forceinline__ float sqrt_fast(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// the vertex of planes p1, p2, p3 about c; bits = its packed topology
__device__ __forceinline__ float4 make_vertex(float4 p1, float4 p2, float4 p3, float3 c,
                                              uint32_t bits) {
  float4 K, M;
  vertex_cofactors(p1, p2, p3, K, M);
  const float g = 6.0f * 5.9604645e-08f;
  const float ew = g * M.w, aw = -K.w;
  float x = 0.f, y = 0.f, z = 0.f;
  uint32_t code = kEpsInf;
  // else (or K_w > 0, or too small to divide by with the error taken below)
  // every test of it goes to the filter
  if (aw > __fmaf_rn(2.0f * g, M.w, 1e-36f)) {
    const float nx = __fmaf_rn(aw, c.x, K.x), ny = __fmaf_rn(aw, c.y, K.y),
                nz = __fmaf_rn(aw, c.z, K.z);
    const float e = g * (M.x + M.y + M.z + (fabsf(c.x) + fabsf(c.y) + fabsf(c.z)) * M.w) +
                    2.4e-7f * (fabsf(nx) + fabsf(ny) + fabsf(nz));
    const float inv = __fdividef(1.0f, aw);
    x = -nx * inv;
    y = -ny * inv;
    z = -nz * inv;
    const float a1 = fabsf(x) + fabsf(y) + fabsf(z);
    const float eps = __fdividef(e + ew * a1, aw - ew) * (1.0f + 4e-6f) + 4e-7f * a1;
    code = eps_code(eps);
    if (code == kEpsInf) x = y = z = 0.f;
  }
  return make_float4(x, y, z, __uint_as_float(bits | (code << 20)));
}

// a sign the positions cannot decide (SignBits)
template <int PRED>
__device__ __noinline__ int slow_conflict(float4 p1, float4 p2, float4 p3, float4 e) {
  // on a plane identical to e the vertex is no conflict (its value is zero,
  // which the filters cannot decide: every such test arrives here)
  if (plane_eq(e, p1) || plane_eq(e, p2) || plane_eq(e, p3)) return 0;
  float4 K, M;
  vertex_cofactors(p1, p2, p3, K, M);
  const int s = filter_sign(K, M, e);
  if (s != 0) return s > 0 ? kSignConflict : 0;
  if (PRED == RPD_PRED_EXACT) return kSignEscalated | exact_conflict(p1, p2, p3, e, M);
  return kSignEscalated | (det4x4_ref(p1, p2, p3, e) > 0.0 ? kSignConflict : 0);
}

// the radius bound finish_list tests (rpd_clip.cu): the largest of the
// vertices' bounds about the seed, from the planes
__device__ __noinline__ float fresh_radius(const WarpStore& w, int lane, int nv, float3 S) {
  float r = 0.f;
  for (int v = 0; v < nv; ++v) {
    const uint32_t b = __float_as_uint(w.vx[v][lane].w);
    float4 K, M;
    vertex_cofactors(w.pl[b & 15u][lane], w.pl[(b >> 4) & 15u][lane], w.pl[(b >> 8) & 15u][lane],
                     K, M);
    r = fmaxf(r, vertex_radius(K, M, S));
  }
  return r;
}

enum Outcome { kRun = 0, kBack = 1 };  // kBack: to clip_cells_kernel

}  // namespace

// EXT: the re-clips of the exact-lists rounds: pairs p.pair_index[..], each with
// its site's extended row
template <int PRED, bool CERT, bool EXT>
__global__ void __launch_bounds__(kTWarps * 32, kTBlocks) clip_threads_kernel(ClipParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr uint32_t kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  WarpStore& w = reinterpret_cast<WarpStore*>(smem_raw)[threadIdx.x >> 5];
  uint32_t n_pred = 0, n_esc = 0;
  // the lane's cell's predicates, escalations and exact signs: they count only
  // if it ends here (clip_cells_kernel counts those it takes up again)
  struct {
    uint32_t pred, esc, uncertain, flips;
  } cell = {0u, 0u, 0u, 0u};

  // the lane's cell
  int q = -1, t = 0, sid = 0;
  float4 seed = make_float4(0.f, 0.f, 0.f, 0.f);
  float3 c = make_float3(0.f, 0.f, 0.f);
  float cmag = 0.f;      // |c|
  float span = 0.f;      // largest |x'|
  CullBox box = {c, c, 0.f};  // box of the vertices (about c) and their radius about
                              // the seed, eps and a slack included
  int np = 0, nv = 0, ne = 0, status = kSuccess, pos = 0;
  uint32_t h4 = 0;       // #adjacent of the tet's faces
  int4 jn = make_int4(-1, -1, -1, -1);  // the next group of the list
  float4 kn = make_float4(0.f, 0.f, 0.f, 0.f);
  int4 jc = jn;          // the group at pos - 4
  uint32_t cand = 0;     // entries of the group at pos - 4 left to test
  int last = 0;          // the entry of that group tested last
  int skip = 0;          // entries of the next group already clipped by
  int fin = 0;           // after those: 1 certified, 2 the list ended
  uint32_t hit = 0;      // vertices the pending plane conflicts with
  uint32_t und = 0;      // its vertices whose sign is not decided yet
  uint32_t some = 0;     // and the conflicts among the others
  float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
  int je = -1;
  int want = 0;          // vertices to make: a new cell's, or around the boundary
  uint64_t seq = 0;      // of the planes seq holds, 4 bits each (a new cell: counts)
  bool active = false, done = false;
  Outcome out = kRun;
  bool more = true;      // the queue has pairs left
  const int32_t* list = nullptr;  // the site's row
  const float* keys = nullptr;
  int len = p.k;
  int row = -1;  // (EXT) its extended row

  auto fetch_group = [&]() {
    const int m = len - pos;
    if (m <= 0) {
      jn = make_int4(-1, -1, -1, -1);
    } else if (m >= 4 && (reinterpret_cast<size_t>(list + pos) & 15) == 0) {
      jn = __ldg(reinterpret_cast<const int4*>(list + pos));
      if (CERT) kn = __ldg(reinterpret_cast<const float4*>(keys + pos));
    } else {
      const int32_t* l = list + pos;
      jn = make_int4(__ldg(l), m > 1 ? __ldg(l + 1) : -1, m > 2 ? __ldg(l + 2) : -1,
                     m > 3 ? __ldg(l + 3) : -1);
      if (CERT) {
        const float* f = keys + pos;
        kn = make_float4(__ldg(f), m > 1 ? __ldg(f + 1) : 0.f, m > 2 ? __ldg(f + 2) : 0.f,
                         m > 3 ? __ldg(f + 3) : 0.f);
      }
    }
  };
  // span and box of the vertices.  The box takes a slack of 2^-10 span, so that
  // a clip's new vertices (their eps) stay inside the one the cull of a group
  // used; true if one does not: a clip shrinks the cell, but where signs are
  // ties a vertex of three nearly dependent planes can land outside it
  auto bounds = [&]() {
    const float sx = c.x - seed.x, sy = c.y - seed.y, sz = c.z - seed.z;
    float d2 = 0.f, s2 = 0.f, em = 0.f;
    float3 lo = make_float3(INFINITY, INFINITY, INFINITY);
    float3 hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
#pragma unroll 2
    for (int v = 0; v < nv; ++v) {
      const float4 x = w.vx[v][lane];
      const float eps = eps_of(x.w);
      d2 = fmaxf(d2, __fmaf_rn(x.x, x.x, __fmaf_rn(x.y, x.y, x.z * x.z)));
      const float a = x.x + sx, b = x.y + sy, d = x.z + sz;
      s2 = fmaxf(s2, __fmaf_rn(a, a, __fmaf_rn(b, b, d * d)));
      em = fmaxf(em, eps);
      lo = make_float3(fminf(lo.x, x.x - eps), fminf(lo.y, x.y - eps), fminf(lo.z, x.z - eps));
      hi = make_float3(fmaxf(hi.x, x.x + eps), fmaxf(hi.y, x.y + eps), fmaxf(hi.z, x.z + eps));
    }
    span = sqrt_fast(d2) * (1.0f + 2e-6f);
    const float r = (sqrt_fast(s2) + em) * (1.0f + 2e-6f) +
                    3e-7f * (span + fabsf(sx) + fabsf(sy) + fabsf(sz));
    const bool outside = fit_box(box, lo, hi, r, span * (1.0f / 1024.0f));
    // a sliver's vertex whose place is hardly known would send every test of
    // it to the filter, one lane at a time
    if (!(em < 0.25f * span)) out = kBack;
    return outside;
  };

  for (;;) {
    // ---- emit the finished cells and take new pairs, once a quarter of the
    // lanes (or every one left) waits for it
    const uint32_t idle = __ballot_sync(kAll, !active && lane < p.cell_lanes);
    const uint32_t waiting = __ballot_sync(kAll, done);
    if (__ballot_sync(kAll, active) == 0u || (more && __popc(idle) >= p.refill_lanes)) {
      if (waiting) {
        bool uncert = false;
        if (done && out == kRun && status == kSuccess && fin == 2) {
          // the whole list without the certificate: the sites missing from
          // it have keys >= its bound (finish_list, rpd_clip.cu)
          const float bound = EXT ? __ldg(p.ext_bound + row)
                                  : (p.nbr_bound ? __ldg(p.nbr_bound + sid) : INFINITY);
          if (bound < INFINITY) {
            // finish_list's bound F exactly, unless R tells that it holds:
            // a vertex's terms of F about the seed S exceed those of eps
            // about c by no more than (|S|_1 + 2 R) / |c|_1 times eps.  (In
            // site-id order a flagged cell is clipped again in another
            // order, so the same cells have to be flagged.)
            const float s1 = fabsf(seed.x) + fabsf(seed.y) + fabsf(seed.z);
            const float c1 = fabsf(c.x) + fabsf(c.y) + fabsf(c.z);
            float em = 0.f;
            for (int v = 0; v < nv; ++v) em = fmaxf(em, eps_of(w.vx[v][lane].w));
            const float F = box.R * (1.0f + 1e-6f) +
                            1.1f * em * (1.0f + __fdividef(s1 + 2.0f * box.R, c1));
            if (!cert_holds(bound, F, p.cert_margin))
              uncert = !cert_holds(
                  bound, fresh_radius(w, lane, nv, make_float3(seed.x, seed.y, seed.z)),
                  p.cert_margin);
          }
        }
        const bool emit = done && out == kRun && status == kSuccess;
        const PayloadLayout L(nv, np, ne);
        const uint32_t size = emit ? L.total : 0u;
        uint32_t incl = size;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(kAll, incl, o);
          if (lane >= o) incl += y;
        }
        unsigned long long base = 0;
        if (lane == 31 && incl) base = atomicAdd(p.payload_cursor, (unsigned long long)incl);
        base = __shfl_sync(kAll, base, 31);
        if (done && out == kBack) {
          p.back_idx[atomicAdd(p.back_count, 1ull)] = q;
        } else if (done) {
          n_pred += cell.pred;
          n_esc += cell.esc;
          if (PRED == RPD_PRED_EXACT && p.exact_counters && cell.uncertain) {
            atomicAdd(p.exact_counters, (unsigned long long)cell.uncertain);
            if (cell.flips) atomicAdd(p.exact_counters + 1, (unsigned long long)cell.flips);
          }
          int st = status;
          unsigned long long off = 0;
          if (emit) {
            off = base + (incl - size);
            if (off + size > p.payload_cap) {
              st = kPayloadFull;
              off = 0;
            } else {
              uint8_t* dst = p.payload + off;
              const int4 fid = __ldg(reinterpret_cast<const int4*>(p.f_ids) + t);
#pragma unroll 1
              for (int i = 0; i < np; ++i)
                reinterpret_cast<float4*>(dst)[i] = w.pl[i][lane];
              // id2, two planes at a time (padded with zero)
#pragma unroll 1
              for (int i = 0; i < np; i += 2) {
                int4 v;
                if (i < 4) {
                  v = make_int4(i == 0 ? fid.x : fid.z, -1, i == 0 ? fid.y : fid.w, -1);
                } else {
                  const int a = w.id[i - 4][lane];
                  v = make_int4(min(sid, a), max(sid, a), 0, 0);
                  if (i + 1 < np) {
                    const int b = w.id[i - 3][lane];
                    v.z = min(sid, b);
                    v.w = max(sid, b);
                  }
                }
                *reinterpret_cast<int4*>(dst + L.id2 + 8 * i) = v;
              }
#pragma unroll 1
              for (int i = 0; i < nv; i += 4) {
                uint32_t x[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  x[k] = 0u;
                  if (i + k < nv) {
                    const uint32_t b = __float_as_uint(w.vx[i + k][lane].w);
                    x[k] = (b & 15u) | ((b & 0xf0u) << 4) | ((b & 0xf00u) << 8) |
                           ((b & 0xff000u) << 12);
                  }
                }
                *reinterpret_cast<uint4*>(dst + L.ver + 4 * i) = make_uint4(x[0], x[1], x[2], x[3]);
              }
              // an edge's count: the tet's own for its six, the larger of the
              // two planes' for the others (the new plane's is 1)
#pragma unroll 1
              for (int i = 0; i < ne; i += 4) {
                const uint32_t pack = w.ed[i >> 2][lane];
                uint32_t x[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  x[k] = 0u;
                  if (i + k < ne) {
                    const uint32_t a = (pack >> (8 * k)) & 15u, b = (pack >> (8 * k + 4)) & 15u;
                    uint32_t z = 1u;
                    if (i + k < 6) z = __ldg(p.e_adj6 + 6ll * t + i + k);
                    else if (a < 4u) z = max(1u, (h4 >> (8 * a)) & 255u);
                    x[k] = a | (b << 8) | (z << 16);
                  }
                }
                *reinterpret_cast<uint4*>(dst + L.edge + 4 * i) =
                    make_uint4(x[0], x[1], x[2], x[3]);
              }
              // plane counts: the tet's faces', then 1 (np <= 16: one chunk)
              const uint32_t ones = 0x01010101u;
              auto tail = [&](int first) {
                const int n = min(max(np - first, 0), 4);
                return n == 4 ? ones : ones & ((1u << (8 * n)) - 1u);
              };
              *reinterpret_cast<uint4*>(dst + L.h) = make_uint4(h4, tail(4), tail(8), tail(12));
            }
          }
          int4 ha, hb;
          const bool rec = emit && st == kSuccess;
          ha = make_int4(t, sid, st,
                         (rec ? (nv | (np << 8) | (ne << 16)) : 0) |
                             (uncert ? (RPD_CELL_UNCERTIFIED << 24) : 0));
          hb = make_int4((int)(uint32_t)off, (int)(uint32_t)(off >> 32), 0, 0);
          int4* hd = reinterpret_cast<int4*>(p.headers + q);
          hd[0] = ha;
          hd[1] = hb;
        }
        done = false;
      }
      __syncwarp();
      // ---- new pairs for the idle lanes
      long long base = 0;
      const int n_idle = __popc(idle);
      if (more) {
        if (lane == 0) base = (long long)atomicAdd(p.work, (unsigned long long)n_idle);
        base = __shfl_sync(kAll, base, 0);
        if (base + n_idle >= p.n_work) more = false;
      } else {
        base = p.n_work;
      }
      const long long mine = base + __popc(idle & ((1u << lane) - 1u));
      if (!active && lane < p.cell_lanes && mine < p.n_work) {
        q = EXT ? __ldg(p.pair_index + mine) : (int)mine;
        t = __ldg(p.pair_tet + q);
        sid = __ldg(p.pair_site + q);
        if (EXT) {
          row = __ldg(p.site_row + sid);
          const long long off = __ldg(p.ext_off + row);
          list = p.ext_nbr + off;
          keys = p.ext_keys + off;
          len = __ldg(p.ext_len + row);
        } else {
          list = p.nbr + (long long)sid * p.k;
          keys = p.keys + (long long)sid * p.k;
        }
        pos = 0;
        fetch_group();
        seed = __ldg(p.site4f + sid);
        const float4 q0 = __ldg(p.tet_xyz + 3ll * t), q1 = __ldg(p.tet_xyz + 3ll * t + 1),
                     q2 = __ldg(p.tet_xyz + 3ll * t + 2);
        const float3 t0 = make_float3(q0.x, q0.y, q0.z), t1 = make_float3(q0.w, q1.x, q1.y),
                     t2 = make_float3(q1.z, q1.w, q2.x), t3 = make_float3(q2.y, q2.z, q2.w);
        const float4 ct = __ldg(p.centroid + t);
        c = make_float3(ct.x, ct.y, ct.z);
        cmag = sqrt_fast(__fmaf_rn(c.x, c.x, __fmaf_rn(c.y, c.y, c.z * c.z))) * (1.0f + 1e-6f);
        // cell = tet: faces (2,1,3), (0,2,3), (1,0,3), (0,1,2)
        const float4 f0 = tri2plane_f(t2, t1, t3), f1 = tri2plane_f(t0, t2, t3),
                     f2 = tri2plane_f(t1, t0, t3), f3 = tri2plane_f(t0, t1, t2);
        w.pl[0][lane] = f0;
        w.pl[1][lane] = f1;
        w.pl[2][lane] = f2;
        w.pl[3][lane] = f3;
        const int4 fa = __ldg(reinterpret_cast<const int4*>(p.f_adjs) + t);
        h4 = (uint32_t)(uint8_t)fa.x | ((uint32_t)(uint8_t)fa.y << 8) |
             ((uint32_t)(uint8_t)fa.z << 16) | ((uint32_t)(uint8_t)fa.w << 24);
        const uchar4 va = __ldg(p.tet_vadj + t);
        seq = (uint64_t)((uint32_t)va.x | ((uint32_t)va.y << 8) | ((uint32_t)va.z << 16) |
                         ((uint32_t)va.w << 24));
        // edges (2,3), (1,3), (1,2), (0,3), (0,2), (0,1)
        w.ed[0][lane] = 0x30213132u;
        w.ed[1][lane] = 0x1020u;
        np = 4;
        nv = 0;
        ne = 6;
        want = 4;  // its vertices
        box.mid = make_float3(0.f, 0.f, 0.f);
        box.half = make_float3(INFINITY, INFINITY, INFINITY);
        box.R = INFINITY;
        cell = {0u, 0u, 0u, 0u};
        status = kSuccess;
        out = kRun;
        cand = 0;
        skip = 0;
        fin = 0;
        hit = und = 0;
        active = true;
      }
      if (__ballot_sync(kAll, active) == 0u) break;  // (every lane: queue empty)
    }

    // ---- make the vertices asked for (a new cell's four, a clip's), one a
    // lane whichever cell they belong to
    __syncwarp();
    uint32_t incl = (uint32_t)want;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kAll, incl, o);
      if (lane >= o) incl += y;
    }
    const int total = (int)__shfl_sync(kAll, incl, 31);
    const int excl = (int)incl - want;
    for (int base = 0; base < total; base += 32) {
      const int item = base + lane;
      int own = 0;  // the last lane whose first item is at most this one
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(kAll, excl, own + o) <= item) own += o;
      const int k = item - __shfl_sync(kAll, excl, own);
      const uint32_t slo = __shfl_sync(kAll, (uint32_t)seq, own);
      const uint32_t shi = __shfl_sync(kAll, (uint32_t)(seq >> 32), own);
      // (a new cell's planes are 0..3: np - 1 = 3)
      const uint32_t meta = __shfl_sync(
          kAll, (uint32_t)want | ((uint32_t)nv << 8) | ((uint32_t)(np - 1) << 16) | ((uint32_t)ne << 24), own);
      const float3 co = make_float3(__shfl_sync(kAll, c.x, own), __shfl_sync(kAll, c.y, own),
                                    __shfl_sync(kAll, c.z, own));
      const uint32_t ho = __shfl_sync(kAll, h4, own);
      const int to = __shfl_sync(kAll, t, own);
      bool zero = false;
      if (item < total) {
        const int len = meta & 255u, slot = ((meta >> 8) & 255u) + k, cur = (meta >> 16) & 255u;
        int x, y, z;
        uint32_t adj;
        if (cur == 3) {
          // triangles (1,3,2), (0,2,3), (0,3,1), (0,1,2)
          x = k == 0 ? 1 : 0;
          y = k == 3 ? 1 : (k == 1 ? 2 : 3);
          z = k == 1 ? 3 : (k == 2 ? 1 : 2);
          adj = (slo >> (8 * k)) & 255u;
        } else {
          const uint64_t sq = ((uint64_t)shi << 32) | slo;
          x = cur;
          y = (int)((sq >> (4 * k)) & 15u);
          z = (int)((sq >> (4 * (k + 1 == len ? 0 : k + 1))) & 15u);
          // edge y - cur; the largest count of the vertex's three edges
          // (clip_full, rpd_clip.cu)
          const int en = (int)(meta >> 24) + k;
          reinterpret_cast<uint8_t*>(&w.ed[en >> 2][own])[en & 3] = (uint8_t)(y | (cur << 4));
          adj = 1u;
          if (y < 4) adj = max(adj, (ho >> (8 * y)) & 255u);
          if (z < 4) {
            adj = max(adj, (ho >> (8 * z)) & 255u);
            if (y < 4) adj = max(adj, (uint32_t)__ldg(p.e_adj6 + 6ll * to + cTetEdgeSlot[y][z]));
          }
        }
        const float4 a = w.pl[x][own], b = w.pl[y][own], d = w.pl[z][own];
        w.vx[slot][own] = make_vertex(a, b, d, co,
                                      (uint32_t)x | ((uint32_t)y << 4) | ((uint32_t)z << 8) |
                                          (adj << 12));
        zero = cur != 3 && det3x3_f(a, b, d) == 0.f;
      }
      const uint32_t zm = __ballot_sync(kAll, zero);
      if (zm) {  // a clip's vertex whose planes are dependent ends its cell
        const int lo = max(excl - base, 0), hi = min(excl + want - base, 32);
        if (hi > lo && ((zm >> lo) & (hi - lo == 32 ? kAll : (1u << (hi - lo)) - 1u)))
          status = kNeedsPerturb;
      }
    }
    __syncwarp();
    if (want > 0) {
      nv += want;
      if (np > 4) ne += want;
      want = 0;
      // the rest of the group is culled again where a vertex fell outside
      if (status == kSuccess && bounds()) {
        cand = 0;
        fin = 0;
        skip = last + 1;
        pos -= 4;
        fetch_group();
      }
      if (out != kRun || status != kSuccess) {
        active = false;
        done = true;
        fin = 0;
      }
    }

    // ---- scan: cull groups of four entries, test the candidates, until few
    // lanes are left without a plane that clips
    for (;;) {
      if (active && (hit | und) == 0u && cand == 0u && fin != 0) {
        active = false;
        done = true;
      }
      const bool busy = active && (hit | und) == 0u;
      const bool to_cull = busy && cand == 0u;
      const int n_cull = __popc(__ballot_sync(kAll, to_cull));
      const int n_test = __popc(__ballot_sync(kAll, busy && cand != 0u));
      const int n_busy = n_cull + n_test;
      const int n_und = __popc(__ballot_sync(kAll, und != 0u));
      if (n_busy + n_und == 0) break;
      if (n_busy < p.scan_lanes &&
          (__any_sync(kAll, hit != 0u) ||
           (more && __popc(__ballot_sync(kAll, !active && lane < p.cell_lanes)) >=
                        p.refill_lanes)))
        break;
      // undecided signs: rare, and long where they end in FP64 or expansions,
      // so they wait for one another
      if (n_und >= p.und_lanes || n_busy < p.scan_lanes) {
        while (und) {
          const int v = __ffs(und) - 1;
          und &= und - 1u;
          const uint32_t b = __float_as_uint(w.vx[v][lane].w);
          const int x = slow_conflict<PRED>(w.pl[b & 15u][lane], w.pl[(b >> 4) & 15u][lane],
                                            w.pl[(b >> 8) & 15u][lane], e);
          if (x & kSignConflict) some |= 1u << v;
          if (x & kSignEscalated) ++cell.esc;
          if (PRED == RPD_PRED_EXACT) {
            if (x & kSignUncertain) ++cell.uncertain;
            if (x & kSignFlip) ++cell.flips;
          }
          if (und == 0u) hit = some;
        }
        if (n_busy == 0) continue;
      }
      // the step that more lanes wait for
      if (n_cull >= n_test) {
        if (to_cull) {
          jc = jn;
          const float4 k4 = kn;
          pos += 4;
          fetch_group();
          const int js[4] = {jc.x, jc.y, jc.z, jc.w};
          const float ks[4] = {k4.x, k4.y, k4.z, k4.w};
          float4 B[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) B[u] = __ldg(p.site4f + max(js[u], 0));
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (fin == 0 && u >= skip) {
              if (js[u] < 0) fin = 2;
              else if (CERT && cert_holds(ks[u], box.R, p.cert_margin)) fin = 1;
            }
            const float4 f = bisector_f(seed, B[u]);
            const float n2 = __fmaf_rn(f.x, f.x, __fmaf_rn(f.y, f.y, f.z * f.z));
            const float nn = sqrt_fast(n2) * (1.0f + 1e-6f);
            const float wp = __fmaf_rn(f.x, c.x, __fmaf_rn(f.y, c.y, __fmaf_rn(f.z, c.z, f.w)));
            const float at = __fmaf_rn(
                f.x, box.mid.x, __fmaf_rn(f.y, box.mid.y, __fmaf_rn(f.z, box.mid.z, wp)));
            const float ext = __fmaf_rn(
                fabsf(f.x), box.half.x,
                __fmaf_rn(fabsf(f.y), box.half.y, fabsf(f.z) * box.half.z));
            const float tol =
                4.8e-7f * __fmaf_rn(nn, cmag + 5.0f * span, fabsf(f.w)) + 1e-30f;
            const bool clear = n2 > 1e-25f && at - ext > tol;
            if (fin == 0 && u >= skip && !clear) cand |= 1u << u;
          }
          skip = 0;
        }
      } else if (busy && cand != 0u) {
        const int u = __ffs(cand) - 1;
        cand &= cand - 1u;
        const int j = u == 0 ? jc.x : (u == 1 ? jc.y : (u == 2 ? jc.z : jc.w));
        const float4 f = bisector_f(seed, __ldg(p.site4f + j));
        const float n2 = __fmaf_rn(f.x, f.x, __fmaf_rn(f.y, f.y, f.z * f.z));
        const float nn = sqrt_fast(n2) * (1.0f + 1e-6f);
        const float wp = __fmaf_rn(f.x, c.x, __fmaf_rn(f.y, c.y, __fmaf_rn(f.z, c.z, f.w)));
        const float tol = n2 > 1e-25f
                              ? 4.8e-7f * __fmaf_rn(nn, cmag + span, fabsf(f.w)) + 1e-30f
                              : INFINITY;
        uint32_t m = 0, un = 0;
        for (int v = 0; v < nv; ++v) {
          const float4 x = w.vx[v][lane];
          const float s = __fmaf_rn(f.x, x.x, __fmaf_rn(f.y, x.y, __fmaf_rn(f.z, x.z, wp)));
          const float b = __fmaf_rn(nn, eps_of(x.w), tol);
          if (s < -b) m |= 1u << v;
          else if (!(s > b)) un |= 1u << v;
        }
        cell.pred += (uint32_t)nv;
        if (m | un) {
          last = u;
          e = f;
          je = j;
          und = un;
          some = m;
          if (un == 0u) hit = m;
        }
      }
    }

    // ---- clip: the reference's update, one cell a lane
    if (hit) {
      uint32_t m = hit;
      hit = 0;
      const int cur = np;
      do {
        if (cur >= kTP) {
          out = kBack;
          break;
        }
        w.pl[cur][lane] = e;
        w.id[cur - 4][lane] = je;
        np = cur + 1;
        // conflicting vertices swapped to the tail
        int n2 = nv, i = 0;
        for (;;) {
          const uint32_t rest = (m >> i) << i;
          if (rest == 0u) break;
          i = __ffs(rest) - 1;
          if (i >= n2) break;
          --n2;
          const float4 a = w.vx[i][lane], b = w.vx[n2][lane];
          w.vx[i][lane] = b;
          w.vx[n2][lane] = a;
          m = ((m >> n2) & 1u) ? m : (m & ~(1u << i));
        }
        int nr = nv - n2;
        nv = n2;
        if (n2 == 0) {
          status = kNoIntersection;
          break;
        }
        // the cavity's boundary (compute_boundary, rpd_clip.cu) as a circular
        // list over plane ids, a byte each; only the removed vertices' planes
        // are needed, and a vertex taken is overwritten by the last one
        uint8_t* const nx = reinterpret_cast<uint8_t*>(&w.next[0][lane]);
        auto at_plane = [&](int a) { return nx + ((a >> 2) << 7) + (a & 3); };
        auto planes_of = [&](int v) -> float& { return w.vx[v][lane].w; };
#pragma unroll
        for (int k = 0; k < 4; ++k) w.next[k][lane] = 0xffffffffu;
        int first;
        {
          const uint32_t tb = __float_as_uint(planes_of(n2));
          const int a = tb & 15u, b = (tb >> 4) & 15u, d = (tb >> 8) & 15u;
          *at_plane(a) = (uint8_t)b;
          *at_plane(b) = (uint8_t)d;
          *at_plane(d) = (uint8_t)a;
          first = a;
          --nr;
          planes_of(n2) = planes_of(n2 + nr);
        }
        int iter = 0, at = n2;
        while (nr > 0 && iter++ < 200) {  // (65,535 tries in the reference)
          const uint32_t tb = __float_as_uint(planes_of(at));
          const int a = tb & 15u, b = (tb >> 4) & 15u, d = (tb >> 8) & 15u;
          uint8_t *const pa = at_plane(a), *const pb = at_plane(b), *const pd = at_plane(d);
          int na = *pa, nb = *pb, nd = *pd;
          const bool oa = nb == a, ob = nd == b, oc = na == d;
          if (!(oa || ob || oc) || (!oa && !ob && nb != kEnd) || (!ob && !oc && nd != kEnd) ||
              (!oc && !oa && na != kEnd)) {
            ++at;
            if (at == n2 + nr) at = n2;
            continue;
          }
          if (!oa) na = b;
          if (!ob) nb = d;
          if (!oc) nd = a;
          if (oa && ob) {
            if (first == b) first = nb;
            nb = kEnd;
          }
          if (ob && oc) {
            if (first == d) first = nd;
            nd = kEnd;
          }
          if (oc && oa) {
            if (first == a) first = na;
            na = kEnd;
          }
          *pa = (uint8_t)na;
          *pb = (uint8_t)nb;
          *pd = (uint8_t)nd;
          --nr;
          planes_of(at) = planes_of(n2 + nr);
          at = n2;
        }
        if (nr > 0) {  // a cavity that does not close: the general kernel's
          out = kBack;
          break;
        }
        if (first != kEnd) {
          // the boundary closes, and its edges and vertices fit
          int cir = first, len = 0;
          bool bad = false;
          seq = 0;
          do {
            seq |= (uint64_t)cir << (4 * len);
            cir = *at_plane(cir);
            ++len;
            bad = cir == kEnd || len >= kTP;
          } while (!bad && cir != first);
          if (cir != first || ne + len > kTE || nv + len > kTV) {
            out = kBack;
            break;
          }
          want = len;
        }
      } while (false);
      if (out != kRun || status != kSuccess) {
        active = false;
        done = true;
        fin = 0;
      }
    }
    __syncwarp();
  }

  for (int o = 16; o > 0; o >>= 1) {
    n_pred += __shfl_xor_sync(kAll, n_pred, o);
    n_esc += __shfl_xor_sync(kAll, n_esc, o);
  }
  if (lane == 0) {
    atomicAdd(p.counters + 0, (unsigned long long)n_pred);
    atomicAdd(p.counters + 1, (unsigned long long)n_esc);
  }
}

// First passes on whole base lists, in the two modes that filter (FP64 mode
// evaluates every sign in FP64, whose pipe bounds it either way), from
// kThreadsPairs pairs on.  Below, one lane's serial clips take longer than a
// warp's (clip stage, us, thread / warp per cell): 14k pairs 112 / 78 (id
// order) and 68 / 80 (certified), 25k 170 / 193 and 143 / 162, 195k
// 475 / 1350, 4.05M (certified) 5400 / 18180.  Cells of many planes (many
// sites in few tets) still gain, although the warps take back up to half of
// them: 17.6 pairs a tet 1260 / 1342 (id order), 475 / 843 (certified).
constexpr long long kThreadsPairs = 20000;

// The exact-lists rounds' re-clips likewise (46.6k cells with rows of up to 512
// entries: the rounds' time 1.27 -> 1.10 ms; 10.7k cells 0.36 / 0.43 ms), but for
// the last round, whose complete rows have no keys.
bool clip_threads_takes(const ClipParams& p, int pred_mode) {
  const bool first = !p.site_row && !p.pair_index;
  const bool again = p.site_row && p.pair_index && !p.ext_complete;
  return (pred_mode == RPD_PRED_FP32_FILTER || pred_mode == RPD_PRED_EXACT) && (first || again) &&
         !p.site_klen && !p.pair_klen && !p.consumed && !p.lazy_cert && p.n_work >= kThreadsPairs;
}

template <int PRED, bool CERT, bool EXT>
static cudaError_t launch_one(ClipParams p, int num_sms, cudaStream_t st) {
  const size_t smem = sizeof(WarpStore) * kTWarps;
  cudaError_t e = cudaFuncSetAttribute(clip_threads_kernel<PRED, CERT, EXT>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // fewer pairs than lanes on the chip: fewer cells a warp, so that all of
  // its warps work and their lanes diverge less
  const long long warps = (long long)num_sms * kTBlocks * kTWarps;
  p.cell_lanes = (int)std::min<long long>(32, std::max<long long>(4, (p.n_work + warps - 1) / warps));
  // of 32 lanes, swept on the 1M-tet workload (clip stage, ms; the first two
  // before the box culling): new pairs at 4 / 8 / 12 / 16 / 24 idle ones 9.1 /
  // 8.4 / 8.0 / 7.7 / 7.7, clipping below 4 / 8 / 12 / 16 scanning ones 7.9 / 7.7 /
  // 7.8 / 8.1; undecided signs end in the filter mostly (1 / 2 / 8 / 24 lanes
  // 5.45 / 5.47 / 5.75 / 5.89), in exact arithmetic on exact ties (146k-tet
  // lattice, by expansions: 13.2 / 12.7 / 9.8 / 8.3)
  auto part = [&](int of32) { return std::max(1, p.cell_lanes * of32 / 32); };
  p.refill_lanes = part(16);
  p.scan_lanes = part(8);
  p.und_lanes = part(PRED == RPD_PRED_EXACT ? 24 : 2);
  const long long per_block = (long long)kTWarps * p.cell_lanes;
  const long long blocks =
      std::min<long long>((long long)num_sms * kTBlocks, (p.n_work + per_block - 1) / per_block);
  if (blocks < 1) return cudaSuccess;
  clip_threads_kernel<PRED, CERT, EXT><<<(unsigned)blocks, kTWarps * 32, smem, st>>>(p);
  note_launches(1);
  return cudaGetLastError();
}

template <int PRED, bool CERT>
static cudaError_t launch_list(const ClipParams& p, int num_sms, cudaStream_t st) {
  return p.site_row ? launch_one<PRED, CERT, true>(p, num_sms, st)
                    : launch_one<PRED, CERT, false>(p, num_sms, st);
}

cudaError_t launch_clip_threads(const ClipParams& p, int pred_mode, int certify, int num_sms,
                                cudaStream_t st) {
  if (pred_mode == RPD_PRED_EXACT)
    return certify ? launch_list<RPD_PRED_EXACT, true>(p, num_sms, st)
                   : launch_list<RPD_PRED_EXACT, false>(p, num_sms, st);
  return certify ? launch_list<RPD_PRED_FP32_FILTER, true>(p, num_sms, st)
                 : launch_list<RPD_PRED_FP32_FILTER, false>(p, num_sms, st);
}

}  // namespace rpd
