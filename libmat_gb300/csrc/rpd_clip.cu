// rpd_clip.cu -- warp-cooperative convex-cell clipping on sm_103a.
//
// One warp owns one cell: the tet (or a box) clipped by the power bisectors
// of one site's neighbour list, in list order.  The cell's planes, dual
// triangles (vertices), edges and boundary links live in shared memory in
// the reference's representation (convex_cell.h:73-115, :117-185), so the
// records it emits are the reference's ConvexCell contents.
//
// Semantics follow src/rpd3d/convex_cell.cu exactly:
//   cell = tet                         :116-214
//   bisector plane (FP32)              :561-592
//   conflict predicate, tie = none     :437-500 (FP64 det4x4 of float planes)
//   conflict partition (swap to tail)  :706-721
//   cavity boundary walk               :618-678
//   new edges / vertices / perturb     :524-554, :604-616, :274-316
//   per-list driver and drop rules     :1166-1337
// What is GB300-specific is the execution: the plane coefficients of 32
// neighbours are built by 32 lanes at once; while the cell has <= 16
// vertices each predicate step tests several consecutive planes against all
// vertices in one ballot and jumps to the first plane that clips anything
// (planes that clip nothing leave the cell unchanged, so skipping them is
// exact); predicate signs come from an FP32 cofactor filter with a proven
// error bound and fall back to the reference's FP64 determinant only when
// undecided; the topology update of a clipping plane runs on lane 0 while
// the vertex cofactors of the new vertices are rebuilt in parallel.
//
// This translation unit is compiled with -fmad=false: every float/double
// expression below that restates a reference formula is evaluated one IEEE
// rounding at a time, as in the reference's source.  FMA is used only where
// written explicitly (the filter).

#include <cuda_runtime.h>

#include "rpd_clip_pred.cuh"
#include "rpd_common.cuh"
#include "rpd_df64.cuh"
#include "rpd_kernels.cuh"

namespace rpd {

// ------------------------------------------------------------------------
// shared-memory cell
// ------------------------------------------------------------------------
struct __align__(16) WarpCell {
  float4 pl[kMaxP];  // plane (a, b, c, d), inside: a x + b y + c z + d >= 0
  // of each vertex: its cofactors and the 3x3 permanents matching them
  // (filter), or the four FP64 minors of its planes (FP64 predicates)
  float4 K[kMaxT];
  float4 M[kMaxT];
  float rad[kMaxT];  // bound on each vertex's distance to the seed (certificate)
  int2 id2[kMaxP];
  uchar4 ver[kMaxT];
  uchar4 edge[kMaxE];
  uint8_t h[kMaxP];
  uint8_t bnext[kMaxP];
  uint8_t perm[kMaxT];  // during a clip: the slot each surviving vertex came from
  float4 cand[32];      // the planes of the list chunk being tested, one per lane
};

struct CellState {
  int nb_v, nb_p, nb_e;
  int status;
  int kept;  // vertices that survived the last clip (slots [0, kept))
};

// FP64 predicates: a vertex's minors, kept where the filter keeps K and M.  A
// predicate is then 7 FP64 operations instead of 45, rounded as the reference
// rounds them.  (The FP64 pipe bounds this mode: 48k tets, 88M predicates, clip
// stage 11.96 -> 5.17 ms.)
__device__ __forceinline__ Minors load_minors(const WarpCell& c, int vi) {
  const double2 a = reinterpret_cast<const double2*>(c.K)[vi];
  const double2 b = reinterpret_cast<const double2*>(c.M)[vi];
  return {a.x, a.y, b.x, b.y};
}
// what the predicates (and with RAD the certificate) need of vertex vi
template <int PRED, bool RAD>
__device__ __forceinline__ void set_vertex(WarpCell& c, int vi, float4 p1, float4 p2, float4 p3,
                                           float3 S) {
  if (uses_filter(PRED) || RAD) {
    float4 K, M;
    vertex_cofactors(p1, p2, p3, K, M);
    if (uses_filter(PRED)) {
      c.K[vi] = K;
      c.M[vi] = M;
    }
    if (RAD) c.rad[vi] = vertex_radius(K, M, S);
  }
  if (!uses_filter(PRED)) {
    const Minors m = det4x4_minors(p1, p2, p3);
    reinterpret_cast<double2*>(c.K)[vi] = make_double2(m.m234, m.m134);
    reinterpret_cast<double2*>(c.M)[vi] = make_double2(m.m124, m.m123);
  }
}

// conflict of the vertex in slot vi with plane e; dup = planes identical to e
template <int PRED>
__device__ __forceinline__ bool in_conflict(const WarpCell& c, int vi, float4 e,
                                            uint64_t dup, PredCount& pc) {
  if (dup != 0ull) {  // rare: the plane equals one of the cell's
    const uchar4 v = c.ver[vi];
    if (dup & ((1ull << v.x) | (1ull << v.y) | (1ull << v.z))) return false;
  }
  ++pc.pred;
  if (uses_filter(PRED)) {
    int s = filter_sign(c.K[vi], c.M[vi], e);
    if (s != 0) return s > 0;
    ++pc.esc;
    const uchar4 v = c.ver[vi];
    if (PRED == RPD_PRED_EXACT) {
      const int x = exact_conflict(c.pl[v.x], c.pl[v.y], c.pl[v.z], e, c.M[vi]);
      if (pc.exact && (x & kSignUncertain)) {
        atomicAdd(pc.exact, 1ull);
        if (x & kSignFlip) atomicAdd(pc.exact + 1, 1ull);
      }
      return x & kSignConflict;
    }
    return det4x4_ref(c.pl[v.x], c.pl[v.y], c.pl[v.z], e) > 0.0;
  }
  return det4x4_of(load_minors(c, vi), e) > 0.0;
}

// ------------------------------------------------------------------------
// topology update (convex_cell.cu:618-774)
// ------------------------------------------------------------------------
// cavity boundary as a circular list over plane ids (convex_cell.cu:618-678)
// (bnext must be all kEnd on entry; the warp clears it before lane 0 runs)
__device__ void compute_boundary(WarpCell& c, int nb_v, int& nb_r, int& first,
                                 int& status) {
  first = kEnd;
  int nb_iter = 0;
  int t = nb_v;
  while (nb_r > 0) {
    if (nb_iter++ > 65535) {
      status = kInconsistentBoundary;
      return;
    }
    uchar4 tr = c.ver[t];
    uint8_t p[3] = {tr.x, tr.y, tr.z};
    bool in_border[3], opp[3];
    for (int e = 0; e < 3; ++e) in_border[e] = c.bnext[p[e]] != kEnd;
    for (int e = 0; e < 3; ++e) opp[e] = c.bnext[p[(e + 1) % 3]] == p[e];
    bool simple = true;
    for (int e = 0; e < 3; ++e)
      if (!opp[e] && !opp[(e + 1) % 3] && in_border[(e + 1) % 3]) simple = false;
    if (!opp[0] && !opp[1] && !opp[2]) {
      if (first == kEnd) {
        for (int e = 0; e < 3; ++e) c.bnext[p[e]] = p[(e + 1) % 3];
        first = p[0];
      } else {
        simple = false;
      }
    }
    if (!simple) {
      t++;
      if (t == nb_v + nb_r) t = nb_v;
      continue;
    }
    for (int e = 0; e < 3; ++e)
      if (!opp[e]) c.bnext[p[e]] = p[(e + 1) % 3];
    for (int e = 0; e < 3; ++e)
      if (opp[e] && opp[(e + 1) % 3]) {
        if (first == p[(e + 1) % 3]) first = c.bnext[p[(e + 1) % 3]];
        c.bnext[p[(e + 1) % 3]] = kEnd;
      }
    int last = nb_v + nb_r - 1;
    uchar4 tmp = c.ver[t];
    c.ver[t] = c.ver[last];
    c.ver[last] = tmp;
    t = nb_v;
    nb_r--;
  }
}

// Adds plane e (already written to slot nb_p by the caller) and applies the
// clip whose conflicting vertex slots are in mask[3], by lane 0, for the box
// kernel: only the polytope (no edges, adjacency counts or perturbation
// check; the cell kernel's update is clip_full, by the whole warp).
__device__ void apply_clip_box(WarpCell& c, CellState& s, const uint32_t* mask_in) {
  // conflict bits of vertex slots 0..95 in registers (32-bit words)
  uint32_t m0 = mask_in[0], m1 = mask_in[1], m2 = mask_in[2];
  const int cur = s.nb_p;
  s.nb_p++;
  // conflict partition, the reference's swap-to-tail loop.  Only the dual
  // triangles move here; perm records where each slot's vertex came from,
  // and the warp moves the cofactors afterwards (the conflict bit of a slot
  // at or past the shrinking end is never read again)
  int nb_v = s.nb_v, nb_r = 0, i = 0;
  while (i < nb_v) {
    // the next conflicting slot from i on (bits at or past nb_v are stale
    // and end the loop)
    {
      uint32_t w = i < 32 ? m0 : (i < 64 ? m1 : m2);
      w &= ~0u << (i & 31);
      int base = i & ~31;
      while (w == 0u && base < 64) {
        base += 32;
        w = base == 32 ? m1 : m2;
      }
      if (w == 0u) break;
      i = base + __ffs(w) - 1;
      if (i >= nb_v) break;
    }
    const uint32_t wi = i < 32 ? m0 : (i < 64 ? m1 : m2);
    if ((wi >> (i & 31)) & 1u) {
      nb_v--;
      const uchar4 tv = c.ver[i];
      c.ver[i] = c.ver[nb_v];
      c.ver[nb_v] = tv;
      const uint8_t pv = c.perm[i];
      c.perm[i] = c.perm[nb_v];
      c.perm[nb_v] = pv;
      const uint32_t wn = nb_v < 32 ? m0 : (nb_v < 64 ? m1 : m2);
      const uint32_t bit = 1u << (i & 31);
      const uint32_t nw = ((wn >> (nb_v & 31)) & 1u) ? (wi | bit) : (wi & ~bit);
      if (i < 32) m0 = nw;
      else if (i < 64) m1 = nw;
      else m2 = nw;
      nb_r++;
    } else {
      i++;
    }
  }
  s.nb_v = nb_v;
  s.kept = nb_v;
  if (nb_v == 0) {
    s.status = kNoIntersection;
    return;
  }
  int first;
  if (nb_r == 1) {
    // one vertex removed: the cavity is its triangle, and the walk would
    // link its three planes in order, starting at the first
    const uchar4 tr = c.ver[nb_v];
    c.bnext[tr.x] = tr.y;
    c.bnext[tr.y] = tr.z;
    c.bnext[tr.z] = tr.x;
    first = tr.x;
  } else {
    compute_boundary(c, nb_v, nb_r, first, s.status);
  }
  if (s.status != kSuccess) return;
  if (first == kEnd) return;
  // new vertices around the cavity boundary
  int cir = first;
  do {
    const int nx = c.bnext[cir];
    if (s.nb_v + 1 >= kMaxT) {
      s.status = kTriangleOverflow;
      return;
    }
    c.ver[s.nb_v] = make_uchar4((uint8_t)cur, (uint8_t)cir, (uint8_t)nx, 0);
    s.nb_v++;
    cir = nx;
  } while (cir != first);
}

__device__ __forceinline__ void broadcast_state(CellState& s) {
  s.nb_v = __shfl_sync(0xffffffffu, s.nb_v, 0);
  s.nb_p = __shfl_sync(0xffffffffu, s.nb_p, 0);
  s.nb_e = __shfl_sync(0xffffffffu, s.nb_e, 0);
  s.status = __shfl_sync(0xffffffffu, s.status, 0);
  s.kept = __shfl_sync(0xffffffffu, s.kept, 0);
}

__device__ __forceinline__ uint64_t shfl64(uint64_t v, int src) {
  uint32_t lo = __shfl_sync(0xffffffffu, (uint32_t)v, src);
  uint32_t hi = __shfl_sync(0xffffffffu, (uint32_t)(v >> 32), src);
  return ((uint64_t)hi << 32) | lo;
}

// the cell radius: the largest of the vertices' cached bounds
__device__ __forceinline__ float cell_radius(const WarpCell& c, int nb_v, int lane) {
  float r = 0.f;
  for (int v = lane; v < nb_v; v += 32) r = fmaxf(r, c.rad[v]);
  for (int o = 16; o > 0; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
  return r;
}

// the same bound from the planes alone (no cached cofactors: plain FP64
// clipping, which keeps none)
__device__ __forceinline__ float cell_radius_fresh(const WarpCell& c, int nb_v, int lane,
                                                   float3 S) {
  float r = 0.f;
  for (int v = lane; v < nb_v; v += 32) {
    const uchar4 t = c.ver[v];
    float4 K, M;
    vertex_cofactors(c.pl[t.x], c.pl[t.y], c.pl[t.z], K, M);
    r = fmaxf(r, vertex_radius(K, M, S));
  }
  for (int o = 16; o > 0; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
  return r;
}

// set_vertex of vertex slots [from, to)
template <int PRED, bool RAD>
__device__ __forceinline__ void refresh_cofactors(WarpCell& c, int from, int to, int lane,
                                                  float3 S) {
  for (int v = from + lane; v < to; v += 32) {
    uchar4 t = c.ver[v];
    set_vertex<PRED, RAD>(c, v, c.pl[t.x], c.pl[t.y], c.pl[t.z], S);
  }
}

struct Cert {
  const float* keys;  // key of each list entry (CERT), ascending
  float3 S;           // seed
  float margin;       // absolute part of the certificate's margin
  bool lazy;          // test the certificate once, after the whole (short) list
  bool certified;
  int consumed;       // list entries taken before the certificate held
  float R;            // eager: the cell radius bound after the last clip
};

// ------------------------------------------------------------------------
// one clip of the cell kernel, by the whole warp
// ------------------------------------------------------------------------
// The reference's update (convex_cell.cu:618-774) is sequential: the
// swap-to-tail partition of the conflicting vertices, the walk around the
// cavity, then one edge and one vertex per boundary plane.  The warp
// computes the same result:
//  * partition: the swap-to-tail loop is a fixed permutation of the
//    conflict bits.  With n vertices, C the conflicting slots, n' = n - |C|
//    and T the surviving slots in [n', n):
//      a slot v < n' outside C keeps its vertex;
//      the j-th slot of C below n' takes the j-th highest slot of T;
//      tail slot p >= n' takes the lowest slot of C if p = n - 1, the
//      vertex of slot p + 1 if that slot conflicts, and otherwise the
//      (rho + 1)-th lowest slot of C, rho the slots of T above p;
//    each lane gathers its slot (cells of up to 32 vertices; lane 0 runs
//    the loop itself for larger ones);
//  * boundary: the cavity of one removed vertex is its triangle; otherwise
//    lane 0 walks it (compute_boundary) and lists its planes in order;
//  * lane k makes edge k and vertex k along the boundary, with the vertex's
//    cofactors and radius bound, and the status is the one the sequential
//    loop stops with: the first vertex with a zero determinant needs
//    perturbation unless a triangle overflow comes strictly before it.

// position of the j-th (1-based) lowest set bit of m (m has at least j)
__device__ __forceinline__ int select_bit(uint32_t m, int j) {
  int pos = 0;
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const int c = __popc(m & ((1u << w) - 1u));
    if (c < j) {
      j -= c;
      m >>= w;
      pos += w;
    }
  }
  return pos;
}

// the swap-to-tail partition run by one thread (cells of more than 32
// vertices); returns the survivors' count
template <bool RAD>
__device__ __noinline__ int partition_serial(WarpCell& c, int nb_v, uint32_t m0, uint32_t m1,
                                             uint32_t m2) {
  int i = 0;
  while (i < nb_v) {
    const uint32_t wi = i < 32 ? m0 : (i < 64 ? m1 : m2);
    if ((wi >> (i & 31)) & 1u) {
      nb_v--;
      const uchar4 tv = c.ver[i];
      c.ver[i] = c.ver[nb_v];
      c.ver[nb_v] = tv;
      const float4 k = c.K[i];
      c.K[i] = c.K[nb_v];
      c.K[nb_v] = k;
      const float4 mm = c.M[i];
      c.M[i] = c.M[nb_v];
      c.M[nb_v] = mm;
      if (RAD) {
        const float r = c.rad[i];
        c.rad[i] = c.rad[nb_v];
        c.rad[nb_v] = r;
      }
      const uint32_t wn = nb_v < 32 ? m0 : (nb_v < 64 ? m1 : m2);
      const uint32_t bit = 1u << (i & 31);
      const uint32_t nw = ((wn >> (nb_v & 31)) & 1u) ? (wi | bit) : (wi & ~bit);
      if (i < 32) m0 = nw;
      else if (i < 64) m1 = nw;
      else m2 = nw;
    } else {
      i++;
    }
  }
  return nb_v;
}

// Adds plane e with id2 `id` as plane s.nb_p and clips the cell by it; the
// conflicting vertex slots are in mask[3] (warp-uniform).  All lanes.
template <int PRED, bool RAD>
__device__ __forceinline__ void clip_full(WarpCell& c, CellState& s, const uint32_t* mask,
                                          float4 e, int2 id, int lane, float3 S) {
  const int cur = s.nb_p;
  if (lane == 0) {
    c.pl[cur] = e;
    c.h[cur] = 1;
    c.id2[cur] = id;
  }
  s.nb_p = cur + 1;
  const int n = s.nb_v;
  int n2;
  if (n <= 32) {
    const uint32_t valid = n == 32 ? ~0u : ((1u << n) - 1u);
    const uint32_t C = mask[0] & valid;
    n2 = n - __popc(C);  // at most n - 1: the plane conflicts somewhere
    const uint32_t low = (1u << n2) - 1u;
    const uint32_t T = ~C & valid & ~low;
    const int v = lane;
    int src = v;
    if (v < n2) {
      if ((C >> v) & 1u) {
        const int j = __popc(C & ((1u << v) - 1u)) + 1;
        src = select_bit(T, __popc(T) - j + 1);
      }
    } else if (v == n - 1) {
      src = __ffs(C) - 1;
    } else if (v < n) {
      if ((C >> (v + 1)) & 1u) src = v + 1;
      else src = select_bit(C, __popc(T >> (v + 1)) + 1);
    }
    const bool move = v < n && src != v;
    uchar4 t;
    float4 K, M;
    float rd = 0.f;
    if (move) {
      t = c.ver[src];
      if (v < n2) {
        K = c.K[src];
        M = c.M[src];
        if (RAD) rd = c.rad[src];
      }
    }
    __syncwarp();
    if (move) {
      c.ver[v] = t;
      if (v < n2) {
        c.K[v] = K;
        c.M[v] = M;
        if (RAD) c.rad[v] = rd;
      }
    }
  } else {
    if (lane == 0) n2 = partition_serial<RAD>(c, n, mask[0], mask[1], mask[2]);
    n2 = __shfl_sync(0xffffffffu, n2, 0);
  }
  __syncwarp();
  s.nb_v = n2;
  s.kept = n2;
  if (n2 == 0) {
    s.status = kNoIntersection;
    return;
  }
  const int nb_r = n - n2;
  int len = 3;
  uchar4 tr = make_uchar4(0, 0, 0, 0);
  if (nb_r == 1) {
    // the cavity is the removed vertex's triangle, its planes in order
    tr = c.ver[n2];
  } else {
    if (lane < kMaxP / 4) reinterpret_cast<uint32_t*>(c.bnext)[lane] = 0xffffffffu;
    __syncwarp();
    int st = s.status, L = 0;
    if (lane == 0) {
      int first, r = nb_r;
      compute_boundary(c, n2, r, first, st);
      if (st == kSuccess && first != kEnd) {
        // the boundary holds at most nb_p - 1 planes
        int cir = first;
        do {
          c.perm[L++] = (uint8_t)cir;
          cir = c.bnext[cir];
        } while (cir != first && L < kMaxP);
        if (cir != first) st = kInconsistentBoundary;
      }
    }
    st = __shfl_sync(0xffffffffu, st, 0);
    len = __shfl_sync(0xffffffffu, L, 0);
    s.status = st;
    if (st != kSuccess || len == 0) return;
  }
  __syncwarp();  // tr and the boundary are read before new vertices land
  if (s.nb_e + len > kMaxE) {
    s.status = kEdgeOverflow;
    return;
  }
  const uint8_t hcur = c.h[cur];
  const int nb_e = s.nb_e;
  int zero_k = kMaxP;  // first boundary vertex whose three planes are dependent
  for (int k = lane; k < len; k += 32) {
    int cir, nx;
    if (nb_r == 1) {
      cir = k == 0 ? tr.x : (k == 1 ? tr.y : tr.z);
      nx = k == 0 ? tr.y : (k == 1 ? tr.z : tr.x);
    } else {
      cir = c.perm[k];
      nx = c.perm[k + 1 == len ? 0 : k + 1];
    }
    const float4 pcir = c.pl[cir], pnx = c.pl[nx];
    const uint8_t hcir = c.h[cir], hnx = c.h[nx];
    // cur > cir: the new plane has the largest index
    c.edge[nb_e + k] = make_uchar4((uint8_t)cir, (uint8_t)cur, hcur > hcir ? hcur : hcir, 0);
    // the largest count of the vertex's three edges.  The reference looks
    // each edge up in the cell's edge list (find_edge_id,
    // convex_cell.cu:511-522); an edge's count is fixed when it is made: the
    // tet's own count for the six initial edges (convex_cell.cu:193-211),
    // max(h_a, h_b) for every edge made by new_edge (:604-616), and two
    // existing planes never become adjacent later
    uint8_t adj = hcur > hcir ? hcur : hcir;
    if (hnx > adj) adj = hnx;
    if (cir < 4 && nx < 4) {
      const uint8_t te = c.edge[cTetEdgeSlot[cir][nx]].z;
      if (te > adj) adj = te;
    }
    const int slot = n2 + k;
    if (slot + 1 < kMaxT) {
      c.ver[slot] = make_uchar4((uint8_t)cur, (uint8_t)cir, (uint8_t)nx, adj);
      set_vertex<PRED, RAD>(c, slot, e, pcir, pnx, S);
    }
    if (det3x3_f(e, pcir, pnx) == 0.f && k < zero_k) zero_k = k;
  }
  for (int o = 16; o > 0; o >>= 1) zero_k = min(zero_k, __shfl_xor_sync(0xffffffffu, zero_k, o));
  const int k_of = max(kMaxT - 1 - n2, 0);  // first vertex that would overflow
  if (zero_k < len && zero_k <= k_of) s.status = kNeedsPerturb;
  else if (k_of < len) s.status = kTriangleOverflow;
  s.nb_e = nb_e + len;
  s.nb_v = n2 + len;
}

// ------------------------------------------------------------------------
// the neighbour loop shared by the cell kernel and the box kernel
// ------------------------------------------------------------------------
// make_plane(j) builds the plane of list entry j (bisector, or offset
// bisector for the box kernel).  With CERT the list is in ascending key
// order and clipping stops as soon as the certificate holds.
template <int PRED, bool FULL, bool CERT, class MakePlane>
__device__ void clip_list(WarpCell& c, CellState& s, const int32_t* list, int k,
                          int seed_id, MakePlane make_plane, int lane,
                          PredCount& pc, Cert& cert) {
  constexpr bool kCof = uses_filter(PRED) || CERT;
  const bool eager = CERT && !cert.lazy;
  float R = INFINITY;
  if (eager) R = cell_radius(c, s.nb_v, lane);
  cert.consumed = k;
  for (int base = 0; base < k && s.status == kSuccess; base += 32) {
    int j = (base + lane < k) ? __ldg(list + base + lane) : -1;
    uint32_t valid = __ballot_sync(0xffffffffu, j != -1);
    int count = (~valid == 0u) ? 32 : (__ffs(~valid) - 1);  // up to first -1
    float key_mine = 0.f;
    if (eager && lane < count) key_mine = __ldg(cert.keys + base + lane);
    // the lane's plane goes to shared memory (the tests read it from there;
    // no register holds it through the chunk), with the planes already in
    // the cell that equal it
    uint64_t dup_mine = 0;
    {
      float4 e_mine = make_float4(0.f, 0.f, 0.f, 0.f);
      if (lane < count) e_mine = make_plane(j);
      __syncwarp();  // the previous chunk's planes are no longer read
      c.cand[lane] = e_mine;
      for (int p = 0; p < s.nb_p; ++p)
        if (plane_eq(e_mine, c.pl[p])) dup_mine |= 1ull << p;
    }
    __syncwarp();
    bool any_dup = __any_sync(0xffffffffu, dup_mine != 0ull);
    int r = 0;
    while (r < count) {
      if (eager) {
        float kr = __shfl_sync(0xffffffffu, key_mine, r);
        if (cert_holds(kr, R, cert.margin)) {
          cert.certified = true;
          cert.consumed = base + r;
          return;
        }
      }
      if (s.nb_p >= kMaxP) {  // new_plane fails before any evaluation
        s.status = kVertexOverflow;
        break;
      }
      uint32_t mask[3] = {0u, 0u, 0u};
      int hit = -1;
      if (s.nb_v <= 32) {
        int lgV = s.nb_v <= 4 ? 2 : (s.nb_v <= 8 ? 3 : (s.nb_v <= 16 ? 4 : 5));
        int V = 1 << lgV;
        int pi = lane >> lgV, vi = lane & (V - 1);
        int pidx = r + pi;
        const float4 e = c.cand[pidx & 31];
        uint64_t dup = any_dup ? shfl64(dup_mine, pidx & 31) : 0ull;
        bool cf = false;
        if (pidx < count && vi < s.nb_v) cf = in_conflict<PRED>(c, vi, e, dup, pc);
        uint32_t m = __ballot_sync(0xffffffffu, cf);
        if (m == 0u) {
          r += 32 >> lgV;
          continue;
        }
        int pf = (__ffs(m) - 1) >> lgV;
        mask[0] = (V == 32) ? m : ((m >> (pf << lgV)) & ((1u << V) - 1u));
        hit = r + pf;
      } else {
        const float4 e = c.cand[r];
        uint64_t dup = any_dup ? shfl64(dup_mine, r) : 0ull;
        bool any = false;
        for (int w = 0; w < 3; ++w) {
          int vi = lane + 32 * w;
          bool cf = false;
          if (vi < s.nb_v) cf = in_conflict<PRED>(c, vi, e, dup, pc);
          mask[w] = __ballot_sync(0xffffffffu, cf);
          any |= mask[w] != 0u;
        }
        if (!any) {
          r += 1;
          continue;
        }
        hit = r;
      }
      // the plane of list entry `hit` clips: write it and update topology
      const float4 e = c.cand[hit];
      int jn = __shfl_sync(0xffffffffu, j, hit);
      if (FULL) {
        clip_full<PRED, CERT>(c, s, mask, e,
                              make_int2(seed_id < jn ? seed_id : jn, seed_id < jn ? jn : seed_id),
                              lane, cert.S);
        __syncwarp();
        if (eager && s.status == kSuccess) R = cell_radius(c, s.nb_v, lane);
        if (plane_eq(c.cand[lane], e)) dup_mine |= 1ull << (s.nb_p - 1);
        any_dup = __any_sync(0xffffffffu, dup_mine != 0ull);
        if (s.status != kSuccess) break;
        r = hit + 1;
        continue;
      }
      if (lane < kMaxP / 4) reinterpret_cast<uint32_t*>(c.bnext)[lane] = 0xffffffffu;
      if (kCof && !FULL)
        for (int v = lane; v < s.nb_v; v += 32) c.perm[v] = (uint8_t)v;
      __syncwarp();
      if (lane == 0) {
        const int cur = s.nb_p;
        c.pl[cur] = e;
        c.h[cur] = 1;
        c.id2[cur] = make_int2(seed_id < jn ? seed_id : jn, seed_id < jn ? jn : seed_id);
        apply_clip_box(c, s, mask);
      }
      __syncwarp();
      broadcast_state(s);
      // the surviving vertices' cofactors follow their dual triangles: a
      // survivor moved into slot v < kept came from a slot >= kept (the
      // partition only swaps with its shrinking end), so sources and
      // targets never overlap
      if (kCof && !FULL && s.status == kSuccess) {
        for (int v = lane; v < s.kept; v += 32) {
          const int src = c.perm[v];
          if (src != v) {
            c.K[v] = c.K[src];
            c.M[v] = c.M[src];
            if (CERT) c.rad[v] = c.rad[src];
          }
        }
        __syncwarp();
      }
      // the vertices created by this clip are exactly those whose first
      // plane is the new one; the surviving ones kept their cofactors
      if (kCof && s.status == kSuccess) {
        const int cur = s.nb_p - 1;
        for (int v = lane; v < s.nb_v; v += 32) {
          uchar4 t = c.ver[v];
          if (t.x == cur) {
            float4 K, M;
            vertex_cofactors(c.pl[t.x], c.pl[t.y], c.pl[t.z], K, M);
            c.K[v] = K;
            c.M[v] = M;
            if (CERT) c.rad[v] = vertex_radius(K, M, cert.S);
          }
        }
      }
      __syncwarp();
      if (eager && s.status == kSuccess) R = cell_radius(c, s.nb_v, lane);
      // later planes of this chunk identical to the new one
      if (plane_eq(c.cand[lane], e)) dup_mine |= 1ull << (s.nb_p - 1);
      any_dup = __any_sync(0xffffffffu, dup_mine != 0ull);
      if (s.status != kSuccess) break;
      r = hit + 1;
    }
    if (count < 32) {  // the list ended (-1) inside this chunk
      cert.consumed = base + count;
      break;
    }
  }
  cert.R = R;
}

// End of a cell's list without the certificate holding on the way (status
// success).  A shortened list (learned or per-site lengths) that ran out
// first: the cell is clipped again with its whole list
// (kSecurityRadiusNotReached marks it).  A whole list: the sites missing from
// it have keys >= its completeness bound, so one test against the bound can
// still certify the cell; otherwise such a site may cut it, and the cell is
// flagged, its radius recorded for a longer list.  Lists of all power
// neighbours, as libmat's triangulation gives, leave no such cells.  Out of
// line: it runs for a few cells, and keeps the hot loop's code small.
// pointers of the list metadata finish_list reads (by value: a noinline
// call must not take the address of the kernel's parameters or state)
struct ListMeta {
  const int32_t* nbr;
  const float* keys;
  const int32_t* site_row;
  const int32_t* ext_len;
  const float* ext_bound;
  const float* nbr_bound;
  unsigned long long* misses;
  int k;
};

// returns 1: flagged uncertified (recheck_cells_kernel takes it up), 2: a
// short list missed (re-clip whole), 0
template <bool CERT, bool EXT>
__device__ __forceinline__ int finish_list(const WarpCell& c, int nb_v, ListMeta m, int sid,
                                          int klen, bool lazy, float R_eager, float margin,
                                          int lane, float3 S) {
  int full;
  float bound;
  const int row = EXT ? __ldg(m.site_row + sid) : -1;
  if (row >= 0) {
    full = __ldg(m.ext_len + row);
    bound = __ldg(m.ext_bound + row);
  } else {
    full = m.k;
    bound = m.nbr_bound ? __ldg(m.nbr_bound + sid) : INFINITY;
  }
  // (only base lists are shortened)
  if (CERT && klen < full && __ldg(m.nbr + (long long)sid * m.k + klen) != -1) {
    bool ok = false;
    if (lazy) {
      // one certificate test after the whole short list
      float R = cell_radius(c, nb_v, lane);
      ok = cert_holds(__ldg(m.keys + (long long)sid * m.k + klen), R, margin);
    }
    if (ok) return 0;
    if (m.misses && lane == 0) atomicAdd(m.misses, 1ull);
    return 2;
  }
  if (klen != full || !(bound < INFINITY) || (!CERT && !m.nbr_bound)) return 0;
  // the FP32 radius bounds (cached, or from the planes): a cell they do not
  // certify is flagged, and recheck_cells_kernel bounds it again with FP64
  // where they are loose
  float R;
  if (CERT && !lazy) R = R_eager;
  else if (CERT) R = cell_radius(c, nb_v, lane);
  else R = cell_radius_fresh(c, nb_v, lane, S);
  return cert_holds(bound, R, margin) ? 0 : 1;
}

// intersection of three float planes, double-float Cramer (box kernel):
// per coordinate a float interval [lo, hi] around the double-float value
__device__ void vertex_of_float_planes(float4 a4, float4 b4, float4 c4, float* lo, float* hi) {
  df ax = df_make(a4.x, 0.f), ay = df_make(a4.y, 0.f), az = df_make(a4.z, 0.f),
     aw = df_make(a4.w, 0.f);
  df bx = df_make(b4.x, 0.f), by = df_make(b4.y, 0.f), bz = df_make(b4.z, 0.f),
     bw = df_make(b4.w, 0.f);
  df cx = df_make(c4.x, 0.f), cy = df_make(c4.y, 0.f), cz = df_make(c4.z, 0.f),
     cw = df_make(c4.w, 0.f);
  df mxy = minor2(bx, by, cx, cy), mxz = minor2(bx, bz, cx, cz), mxw = minor2(bx, bw, cx, cw);
  df myz = minor2(by, bz, cy, cz), myw = minor2(by, bw, cy, cw), mzw = minor2(bz, bw, cz, cw);
  df Dw = df_add_s(df_sub_s(df_mul(ax, myz), df_mul(ay, mxz)), df_mul(az, mxy));
  df Dx = df_add_s(df_sub_s(df_mul(ay, mzw), df_mul(az, myw)), df_mul(aw, myz));
  df Dy = df_add_s(df_sub_s(df_mul(ax, mzw), df_mul(az, mxw)), df_mul(aw, mxz));
  df Dz = df_add_s(df_sub_s(df_mul(ax, myw), df_mul(ay, mxw)), df_mul(aw, mxy));
  const df inv = df_recip(Dw);
  const df X[3] = {df_neg(df_mul(Dx, inv)), df_mul(Dy, inv), df_neg(df_mul(Dz, inv))};
  for (int k = 0; k < 3; ++k) {
    lo[k] = __fadd_rd(X[k].hi, X[k].lo);
    hi[k] = __fadd_ru(X[k].hi, X[k].lo);
  }
}

// MINB > 0 caps registers so that MINB blocks of 128 threads fit on an SM
// (occupancy variants chosen by the autotuner)
// EXT: sites may have extended rows (the exact-lists rounds); the first
// pass, on base lists only, runs without that code
template <int PRED, bool CERT, int MINB, bool EXT>
__global__ void __launch_bounds__(MINB > 0 ? 128 : kClipMaxThreads, MINB > 0 ? MINB : 1)
    clip_cells_kernel(ClipParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const int wid = threadIdx.x >> 5;
  WarpCell& c = reinterpret_cast<WarpCell*>(smem_raw)[wid];
  PredCount pc = {0u, 0u, p.exact_counters};
  unsigned int n_uncert = 0;  // lane-uniform
  const long long n_work = p.n_work_dev ? (long long)*p.n_work_dev : p.n_work;

  for (;;) {
    long long q = 0;
    if (lane == 0) q = (long long)atomicAdd(p.work, 1ull);
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q >= n_work) break;
    if (p.pair_index) q = __ldg(p.pair_index + q);
    const int t = __ldg(p.pair_tet + q);
    const int sid = __ldg(p.pair_site + q);
    const float4 seed = __ldg(p.site4f + sid);

    // ---- cell = tet (convex_cell.cu:116-214); the tet's float vertices and
    // vertex counts come packed per tet (one dependent load less)
    if (lane < 4) {
      const float4 q0 = __ldg(p.tet_xyz + 3ll * t), q1 = __ldg(p.tet_xyz + 3ll * t + 1),
                   q2 = __ldg(p.tet_xyz + 3ll * t + 2);
      const float3 t0 = make_float3(q0.x, q0.y, q0.z), t1 = make_float3(q0.w, q1.x, q1.y),
                   t2 = make_float3(q1.z, q1.w, q2.x), t3 = make_float3(q2.y, q2.z, q2.w);
      // face `lane` (cFaceLv): (2,1,3), (0,2,3), (1,0,3), (0,1,2), selected
      // without indexing a local array by lane
      const float3 fa = lane == 0 ? t2 : (lane == 1 ? t0 : (lane == 2 ? t1 : t0));
      const float3 fb = lane == 0 ? t1 : (lane == 1 ? t2 : (lane == 2 ? t0 : t1));
      const float3 fc = lane == 3 ? t2 : t3;
      c.pl[lane] = tri2plane_f(fa, fb, fc);
      c.h[lane] = (uint8_t)__ldg(p.f_adjs + 4 * t + lane);
      c.id2[lane] = make_int2(__ldg(p.f_ids + 4 * t + lane), -1);
    } else if (lane < 8) {
      int i = lane - 4;
      const uchar4 va = __ldg(p.tet_vadj + t);
      const uint8_t vi = i == 0 ? va.x : (i == 1 ? va.y : (i == 2 ? va.z : va.w));
      c.ver[i] = make_uchar4((uint8_t)cTetTri[i][0], (uint8_t)cTetTri[i][1],
                             (uint8_t)cTetTri[i][2], vi);
    } else if (lane < 14) {
      int e = lane - 8;
      c.edge[e] = make_uchar4((uint8_t)cEdgeFaces[e][0], (uint8_t)cEdgeFaces[e][1],
                              __ldg(p.e_adj6 + 6 * (long long)t + e), 0);
    }
    __syncwarp();
    CellState s;
    s.nb_v = 4;
    s.nb_p = 4;
    s.nb_e = 6;
    s.status = kSuccess;
    {
      refresh_cofactors<PRED, CERT>(c, 0, 4, lane, make_float3(seed.x, seed.y, seed.z));
      __syncwarp();
    }

    // ---- clip by the site's neighbour list: its base row, or the extended
    // row it was given after an earlier pass left one of its cells
    // uncertified
    const float4* site4f = p.site4f;
    auto make_plane = [&](int j) { return bisector_f(seed, __ldg(site4f + j)); };
    const int32_t* list;
    const float* keys;
    int klen;
    bool complete = false;  // a row of every site (id order, no keys)
    {
      const int row = EXT ? __ldg(p.site_row + sid) : -1;
      if (row >= 0) {
        const long long off = __ldg(p.ext_off + row);
        list = p.ext_nbr + off;
        klen = __ldg(p.ext_len + row);
        complete = !(__ldg(p.ext_bound + row) < INFINITY);
        keys = (p.ext_keys && !complete) ? p.ext_keys + off : nullptr;
      } else {
        list = p.nbr + (long long)sid * p.k;
        keys = p.keys ? p.keys + (long long)sid * p.k : nullptr;
        klen = p.k;
        if (p.site_klen) klen = min(klen, __ldg(p.site_klen + sid));
        if (p.pair_klen) klen = min(klen, __ldg(p.pair_klen + q));
      }
    }
    Cert cert;
    cert.keys = CERT ? keys : nullptr;
    cert.S = make_float3(seed.x, seed.y, seed.z);
    cert.margin = p.cert_margin;
    cert.lazy = p.lazy_cert != 0 || complete;
    cert.certified = false;
    clip_list<PRED, true, CERT>(c, s, list, klen, sid, make_plane, lane, pc, cert);
    bool uncert = false;
    if (s.status == kSuccess && !cert.certified) {
      ListMeta m;
      m.nbr = p.nbr;
      m.keys = p.keys;
      m.site_row = p.site_row;
      m.ext_len = p.ext_len;
      m.ext_bound = p.ext_bound;
      m.nbr_bound = p.nbr_bound;
      m.misses = p.misses;
      m.k = p.k;
      const int r = finish_list<CERT, EXT>(c, s.nb_v, m, sid, klen, cert.lazy, cert.R, cert.margin,
                                      lane, make_float3(seed.x, seed.y, seed.z));
      uncert = r == 1;
      if (r == 2) s.status = kSecurityRadiusNotReached;
    }
    if (p.consumed && lane == 0) p.consumed[q] = cert.consumed;
    n_uncert += uncert ? 1u : 0u;

    // ---- emit
    rpd_cell_header hd;
    hd.tet_id = t;
    hd.site_id = sid;
    hd.status = s.status;
    hd.nb_v = hd.nb_p = hd.nb_e = 0;
    hd.flags = uncert ? RPD_CELL_UNCERTIFIED : 0;
    hd.offset = 0;
    hd.volume = 0.0;
    if (s.status == kSuccess) {
      PayloadLayout L(s.nb_v, s.nb_p, s.nb_e);
      unsigned long long off = 0;
      if (lane == 0) off = atomicAdd(p.payload_cursor, (unsigned long long)L.total);
      off = __shfl_sync(0xffffffffu, off, 0);
      if (off + L.total > p.payload_cap) {
        hd.status = kPayloadFull;
      } else {
        uint8_t* dst = p.payload + off;
        for (int i = lane; i < s.nb_p; i += 32) {
          reinterpret_cast<float4*>(dst + L.plane)[i] = c.pl[i];
          reinterpret_cast<int2*>(dst + L.id2)[i] = c.id2[i];
        }
        for (int i = lane; i < s.nb_v; i += 32)
          reinterpret_cast<uchar4*>(dst + L.ver)[i] = c.ver[i];
        for (int i = lane; i < s.nb_e; i += 32)
          reinterpret_cast<uchar4*>(dst + L.edge)[i] = c.edge[i];
        for (int i = lane; i < (int)al16(s.nb_p); i += 32)
          dst[L.h + i] = i < s.nb_p ? c.h[i] : 0;
        // pad bytes of the id2 / ver / edge sections
        for (int i = 2 * s.nb_p + lane; i < (int)(al16(8u * s.nb_p) / 4); i += 32)
          reinterpret_cast<int32_t*>(dst + L.id2)[i] = 0;
        for (int i = s.nb_v + lane; i < (int)(al16(4u * s.nb_v) / 4); i += 32)
          reinterpret_cast<uint32_t*>(dst + L.ver)[i] = 0u;
        for (int i = s.nb_e + lane; i < (int)(al16(4u * s.nb_e) / 4); i += 32)
          reinterpret_cast<uint32_t*>(dst + L.edge)[i] = 0u;
        // coordinates, volume and topology hash: cell_epilogue_kernel
        hd.nb_v = (uint8_t)s.nb_v;
        hd.nb_p = (uint8_t)s.nb_p;
        hd.nb_e = (uint8_t)s.nb_e;
        hd.offset = off;
      }
    }
    if (lane == 0) p.headers[q] = hd;
    __syncwarp();
  }
  // statistics
  for (int o = 16; o > 0; o >>= 1) {
    pc.pred += __shfl_xor_sync(0xffffffffu, pc.pred, o);
    pc.esc += __shfl_xor_sync(0xffffffffu, pc.esc, o);
  }
  if (lane == 0) {
    atomicAdd(p.counters + 0, (unsigned long long)pc.pred);
    atomicAdd(p.counters + 1, (unsigned long long)pc.esc);
    if (n_uncert && p.uncertified) atomicAdd(p.uncertified, (unsigned long long)n_uncert);
  }
}

// ------------------------------------------------------------------------
// recheck of the cells flagged uncertified: the radius bound again, from
// the emitted record's planes, FP64 for the vertices whose FP32 bound is
// loose; a cell it certifies loses the flag, the others give their site's
// longer list its length (site_need, the largest radius of the site's
// flagged cells)
// ------------------------------------------------------------------------
__global__ void __launch_bounds__(128) recheck_cells_kernel(RecheckParams p) {
  const int lane = threadIdx.x & 31;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long n = *p.n_dev;
  for (long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n;
       w += n_warps) {
    const long long q = __ldg(p.idx + w);
    rpd_cell_header h = p.headers[q];
    const int sid = h.site_id;
    const float4 seed = __ldg(p.site4f + sid);
    const float3 S = make_float3(seed.x, seed.y, seed.z);
    const int row = p.site_row ? __ldg(p.site_row + sid) : -1;
    const float bound = row >= 0 ? __ldg(p.ext_bound + row) : __ldg(p.nbr_bound + sid);
    const PayloadLayout L(h.nb_v, h.nb_p, h.nb_e);
    const float4* pl = reinterpret_cast<const float4*>(p.payload + h.offset + L.plane);
    const uchar4* ver = reinterpret_cast<const uchar4*>(p.payload + h.offset + L.ver);
    float r = 0.f;
    for (int v = lane; v < h.nb_v; v += 32) {
      const uchar4 t = ver[v];
      const float4 a = pl[t.x], b = pl[t.y], d = pl[t.z];
      float4 K, M;
      vertex_cofactors(a, b, d, K, M);
      r = fmaxf(r, vertex_radius_p(K, M, S, a, b, d));
    }
    for (int o = 16; o > 0; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
    if (lane == 0) {
      // a complete list (bound infinite) certifies any cell
      if (!(bound < INFINITY) || cert_holds(bound, r, p.margin)) {
        p.headers[q].flags = (uint8_t)(h.flags & ~RPD_CELL_UNCERTIFIED);
      } else {
        if (p.site_need) atomicMax(p.site_need + sid, __float_as_uint(r));
        if (p.kept_idx) p.kept_idx[atomicAdd(p.kept_count, 1ull)] = (int32_t)q;
      }
    }
  }
}

cudaError_t launch_recheck_cells(const RecheckParams& p, int num_sms, cudaStream_t st) {
  recheck_cells_kernel<<<(unsigned)(num_sms * 16), 128, 0, st>>>(p);
  note_launches(1);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// box kernel: bounding box of a site's cell grown by an offset, used to
// enumerate candidate tets (see rpd_pairs.cu)
// ------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 6) site_box_kernel(BoxParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const int wid = threadIdx.x >> 5;
  WarpCell& c = reinterpret_cast<WarpCell*>(smem_raw)[wid];
  PredCount pc = {0u, 0u, nullptr};
  const int warps_total = (gridDim.x * blockDim.x) >> 5;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < p.n_site; i += warps_total) {
    float lo[3] = {p.box_lo.x, p.box_lo.y, p.box_lo.z};
    float hi[3] = {p.box_hi.x, p.box_hi.y, p.box_hi.z};
    if (p.flags[p.site_base + i] != 1u) {
      if (lane == 0) {
        p.site_box[2 * i] = make_float4(1.f, 1.f, 1.f, 0.f);  // empty box
        p.site_box[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.offset_r1 > 0.f) {
          p.site_box1[2 * i] = make_float4(1.f, 1.f, 1.f, 0.f);
          p.site_box1[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        p.site_nplanes[i] = 0;
      }
      continue;
    }
    const float4 seed = p.site4f[p.site_base + i];
    // own: the second class's region by a clip of its own, because the first
    // class's is empty
    for (bool own = false;;) {
      // box planes x>=lo, x<=hi, y>=lo, y<=hi, z>=lo, z<=hi
      if (lane < 6) {
        int ax = lane >> 1;
        float4 pl = make_float4(0.f, 0.f, 0.f, 0.f);
        float* q = reinterpret_cast<float*>(&pl);
        if ((lane & 1) == 0) {
          q[ax] = 1.f;
          pl.w = -lo[ax];
        } else {
          q[ax] = -1.f;
          pl.w = hi[ax];
        }
        c.pl[lane] = pl;
      } else if (lane < 14) {
        // corner (sx, sy, sz): planes X = sx, Y = 2 + sy, Z = 4 + sz, ordered
        // (X, Z, Y) for even parity and (X, Y, Z) for odd parity: the eight
        // dual triangles are then consistently oriented with the same sign as
        // the tet's (det4x4 of the triangle's planes with (0,0,0,1) < 0), so
        // "det > 0" means "outside" for both
        int v = lane - 6;
        int sx = v & 1, sy = (v >> 1) & 1, sz = (v >> 2) & 1;
        uint8_t X = (uint8_t)sx, Y = (uint8_t)(2 + sy), Z = (uint8_t)(4 + sz);
        c.ver[v] = ((sx + sy + sz) & 1) == 0 ? make_uchar4(X, Z, Y, 0) : make_uchar4(X, Y, Z, 0);
      }
      __syncwarp();
      CellState s;
      s.nb_v = 8;
      s.nb_p = 6;
      s.nb_e = 0;
      s.status = kSuccess;
      refresh_cofactors<RPD_PRED_FP32_FILTER, false>(c, 0, 8, lane, make_float3(0.f, 0.f, 0.f));
      __syncwarp();
      const float4* site4f = p.site4f;
      const float R = own ? p.offset_r1 : p.offset_r, E = p.offset_e;
      auto make_plane = [&](int j) {
        float4 b = __ldg(site4f + j);
        float4 e = bisector_f(seed, b);
        float D = sqrtf(e.x * e.x + e.y * e.y + e.z * e.z);
        // push the plane outwards by R plus the float error of the rule's
        // power distances (E / 2D) plus a relative slack
        float slack = 1e-5f * (fabsf(e.w) + D * p.coord_scale);
        float d = e.w + R * D + 0.5f * E + slack;
        if (!(D > 0.f) || !(d < 3.0e38f)) return make_float4(0.f, 0.f, 0.f, 1.f);  // no constraint
        return make_float4(e.x, e.y, e.z, d);
      };
      // any subset of the planes gives a superset polytope; the nearest k_box
      // bisectors bound the cell well and keep the box clip small
      Cert nocert;
      nocert.keys = nullptr;
      nocert.certified = false;
      clip_list<RPD_PRED_FP32_FILTER, false, false>(c, s, p.nbr + (long long)i * p.k,
                                                    own ? p.k_box1 : p.k_box, p.site_base + i,
                                                    make_plane, lane, pc, nocert);
      float bl[3], bh[3];
      if (s.status == kSuccess) {
        bl[0] = bl[1] = bl[2] = 3.0e38f;
        bh[0] = bh[1] = bh[2] = -3.0e38f;
        for (int v = lane; v < s.nb_v; v += 32) {
          uchar4 tr = c.ver[v];
          float xl[3], xh[3];
          vertex_of_float_planes(c.pl[tr.x], c.pl[tr.y], c.pl[tr.z], xl, xh);
          for (int k = 0; k < 3; ++k) {
            if (!(xl[k] == xl[k]) || !(xh[k] == xh[k])) {  // degenerate vertex
              xl[k] = lo[k];
              xh[k] = hi[k];
            }
            bl[k] = fminf(bl[k], xl[k]);
            bh[k] = fmaxf(bh[k], xh[k]);
          }
        }
        for (int o = 16; o > 0; o >>= 1)
          for (int k = 0; k < 3; ++k) {
            bl[k] = fminf(bl[k], __shfl_xor_sync(0xffffffffu, bl[k], o));
            bh[k] = fmaxf(bh[k], __shfl_xor_sync(0xffffffffu, bh[k], o));
          }
        for (int k = 0; k < 3; ++k) {
          float m = 1e-3f * (bh[k] - bl[k]) + p.abs_margin;
          bl[k] = fmaxf(bl[k] - m, lo[k]);
          bh[k] = fminf(bh[k] + m, hi[k]);
        }
      } else if (s.status == kNoIntersection) {
        bl[0] = bl[1] = bl[2] = 1.f;
        bh[0] = bh[1] = bh[2] = 0.f;
      } else {
        for (int k = 0; k < 3; ++k) {
          bl[k] = lo[k];
          bh[k] = hi[k];
        }
      }
      const bool empty = s.status == kNoIntersection;
      if (lane == 0) {
        float4* box = own ? p.site_box1 : p.site_box;
        box[2 * i] = make_float4(bl[0], bl[1], bl[2], own ? 1.f : 0.f);
        box[2 * i + 1] = make_float4(bh[0], bh[1], bh[2], 0.f);
      }
      if (empty && !own && p.offset_r1 > 0.f) {
        __syncwarp();
        own = true;
        continue;
      }
      // the planes that bound the grown cell (referenced by a vertex): the pair
      // search tests grid cells and tet centroids against them
      int npl = 0;
      unsigned long long bounding = 0ull;
      if (s.status == kSuccess) {
        unsigned long long m = 0ull;
        for (int v = lane; v < s.nb_v; v += 32) {
          uchar4 tr = c.ver[v];
          m |= (1ull << tr.x) | (1ull << tr.y) | (1ull << tr.z);
        }
        const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)m);
        const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)(m >> 32));
        const unsigned long long act = ((unsigned long long)hi << 32) | lo;
        bounding = act;
        // any subset of them bounds a superset of the grown cell: beyond the
        // storage, the first kBoxPlanes are kept
        npl = min(__popcll(act), kBoxPlanes);
        for (int q = lane; q < s.nb_p; q += 32) {
          const int rank = __popcll(act & ((1ull << q) - 1ull));
          if (((act >> q) & 1ull) && rank < kBoxPlanes)
            p.site_planes[(long long)i * kBoxPlanes + rank] = c.pl[q];
        }
      }
      if (lane == 0) p.site_nplanes[i] = npl;
      if (!own && p.offset_r1 > 0.f) {
        // The larger class's region from this one: pushing every bounding plane
        // out by delta stays inside the polytope scaled about the seed by
        // lambda = 1 + delta / h, h the seed's least distance to those planes
        // (a point x of it has x / lambda on their inner side, since (h_m +
        // delta) / lambda <= h_m).  It saves that class's clip, 0.63 ms of the
        // 1M-tet workload for 0.5 % of its tets.  A seed outside or close to a
        // plane gets the whole region, whose grid cells the planes then cull.
        const float delta = (p.offset_r1 - p.offset_r) * (1.0f + 1e-4f);
        float h = INFINITY;
        if (s.status == kSuccess) {
          for (int q = lane; q < s.nb_p; q += 32)
            if ((bounding >> q) & 1ull) {
              const float4 e = c.pl[q];
              const float tol = 4e-6f * ((fabsf(e.x) + fabsf(e.y) + fabsf(e.z)) * p.coord_scale +
                                         fabsf(e.w));
              const float v = e.x * seed.x + e.y * seed.y + e.z * seed.z + e.w - tol;
              h = fminf(h, v / sqrtf(e.x * e.x + e.y * e.y + e.z * e.z));
            }
          for (int o = 16; o > 0; o >>= 1) h = fminf(h, __shfl_xor_sync(0xffffffffu, h, o));
        }
        if (lane == 0) {
          const bool scaled = s.status == kSuccess && h > 1e-2f * delta && h < INFINITY;
          const float lam = scaled ? 1.0f + delta / h * (1.0f + 1e-4f) : 0.f;
          const float sd[3] = {seed.x, seed.y, seed.z};
          float l1[3], h1[3];
          for (int k = 0; k < 3; ++k) {
            l1[k] = lo[k];
            h1[k] = hi[k];
            if (scaled) {
              const float m = 1e-3f * lam * (bh[k] - bl[k]) + p.abs_margin;
              l1[k] = fmaxf(sd[k] - lam * (sd[k] - bl[k]) - m, lo[k]);
              h1[k] = fminf(sd[k] + lam * (bh[k] - sd[k]) + m, hi[k]);
            }
          }
          p.site_box1[2 * i] = make_float4(l1[0], l1[1], l1[2], 0.f);
          p.site_box1[2 * i + 1] = make_float4(h1[0], h1[1], h1[2], 0.f);
        }
      }
      __syncwarp();
      break;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    pc.pred += __shfl_xor_sync(0xffffffffu, pc.pred, o);
    pc.esc += __shfl_xor_sync(0xffffffffu, pc.esc, o);
  }
  if (lane == 0 && p.counters) {
    atomicAdd(p.counters + 0, (unsigned long long)pc.pred);
    atomicAdd(p.counters + 1, (unsigned long long)pc.esc);
  }
}

size_t clip_smem_per_warp() { return sizeof(WarpCell); }

template <int PRED, bool CERT, int MINB>
static int occ_of(int warps) {
  size_t smem = sizeof(WarpCell) * warps;
  int n = 0;
  cudaFuncSetAttribute(clip_cells_kernel<PRED, CERT, MINB, false>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, clip_cells_kernel<PRED, CERT, MINB, false>,
                                                warps * 32, smem);
  return n > 0 ? n : 1;
}

template <int PRED, bool CERT>
static int occ_variant(int variant, int warps) {
  if (variant == 1) return occ_of<PRED, CERT, 6>(4);
  if (variant == 2) return occ_of<PRED, CERT, 8>(4);
  return occ_of<PRED, CERT, 0>(warps);
}

int clip_blocks_per_sm_cert(int pred_mode, int certify, int warps, int variant) {
  if (pred_mode == RPD_PRED_FP32_FILTER)
    return certify ? occ_variant<RPD_PRED_FP32_FILTER, true>(variant, warps)
                   : occ_variant<RPD_PRED_FP32_FILTER, false>(variant, warps);
  if (pred_mode == RPD_PRED_EXACT)
    return certify ? occ_variant<RPD_PRED_EXACT, true>(variant, warps)
                   : occ_variant<RPD_PRED_EXACT, false>(variant, warps);
  return certify ? occ_variant<RPD_PRED_FP64, true>(variant, warps)
                 : occ_variant<RPD_PRED_FP64, false>(variant, warps);
}

int clip_blocks_per_sm(int pred_mode, int warps) {
  return clip_blocks_per_sm_cert(pred_mode, 0, warps, 0);
}

int box_blocks_per_sm(int warps) {
  size_t smem = sizeof(WarpCell) * warps;
  int n = 0;
  cudaFuncSetAttribute(site_box_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, site_box_kernel, warps * 32, smem);
  return n > 0 ? n : 1;
}

template <int PRED, bool CERT, int MINB, bool EXT>
static void launch_one(const ClipParams& p, int blocks, int warps, cudaStream_t st) {
  size_t smem = sizeof(WarpCell) * warps;
  cudaFuncSetAttribute(clip_cells_kernel<PRED, CERT, MINB, EXT>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  clip_cells_kernel<PRED, CERT, MINB, EXT><<<blocks, warps * 32, smem, st>>>(p);
  note_launches(1);
}

// the re-clips with extended rows (few cells) use one register budget (80:
// six blocks of four warps per SM), whatever the first pass's variant
template <int PRED, bool CERT>
static void launch_variant(const ClipParams& p, int variant, int blocks, int warps,
                           cudaStream_t st) {
  if (p.site_row) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    launch_one<PRED, CERT, 6, true>(p, (sms > 0 ? sms : 1) * 6, 4, st);
  } else if (variant == 1) {
    launch_one<PRED, CERT, 6, false>(p, blocks, 4, st);
  } else if (variant == 2) {
    launch_one<PRED, CERT, 8, false>(p, blocks, 4, st);
  } else {
    launch_one<PRED, CERT, 0, false>(p, blocks, warps, st);
  }
}

cudaError_t launch_clip_cells(const ClipParams& p, int pred_mode, int certify, int variant,
                              int blocks, int warps, cudaStream_t st) {
  if (pred_mode == RPD_PRED_FP32_FILTER) {
    if (certify) launch_variant<RPD_PRED_FP32_FILTER, true>(p, variant, blocks, warps, st);
    else launch_variant<RPD_PRED_FP32_FILTER, false>(p, variant, blocks, warps, st);
  } else if (pred_mode == RPD_PRED_EXACT) {
    if (certify) launch_variant<RPD_PRED_EXACT, true>(p, variant, blocks, warps, st);
    else launch_variant<RPD_PRED_EXACT, false>(p, variant, blocks, warps, st);
  } else {
    if (certify) launch_variant<RPD_PRED_FP64, true>(p, variant, blocks, warps, st);
    else launch_variant<RPD_PRED_FP64, false>(p, variant, blocks, warps, st);
  }
  return cudaGetLastError();
}

cudaError_t launch_site_box(const BoxParams& p, int blocks, int warps, cudaStream_t st) {
  size_t smem = sizeof(WarpCell) * warps;
  cudaFuncSetAttribute(site_box_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  site_box_kernel<<<blocks, warps * 32, smem, st>>>(p);
  note_launches(1);
  return cudaGetLastError();
}

}  // namespace rpd
