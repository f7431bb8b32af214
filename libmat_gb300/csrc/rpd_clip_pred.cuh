// rpd_clip_pred.cuh -- the clippers' arithmetic: the reference's planes and
// determinants, the FP32 filter with its error bound, the FP64 and exact
// escalations, the vertex radius bounds and the certificate's test.  Included
// by the translation units that clip cells, which are compiled with
// -fmad=false: every expression that restates a reference formula is
// evaluated one IEEE rounding at a time; FMA appears only where written.
#pragma once

#include "rpd_common.cuh"
#include "rpd_kernels.cuh"

namespace rpd {

// local faces / edges of a tet (convex_cell.h:25-29, convex_cell.cu:193-211)
static __constant__ int8_t cFaceLv[4][3] = {{2, 1, 3}, {0, 2, 3}, {1, 0, 3}, {0, 1, 2}};
static __constant__ int8_t cEdgeFaces[6][2] = {{2, 3}, {1, 3}, {1, 2}, {0, 3}, {0, 2}, {0, 1}};
static __constant__ int8_t cTetTri[4][3] = {{1, 3, 2}, {0, 2, 3}, {0, 3, 1}, {0, 1, 2}};
// slot of the initial edge between tet faces (lo, hi), lo < hi < 4
static __constant__ int8_t cTetEdgeSlot[4][4] = {{-1, 5, 4, 3}, {5, -1, 2, 1}, {4, 2, -1, 0}, {3, 1, 0, -1}};

// ------------------------------------------------------------------------
// reference arithmetic (no contraction)
// ------------------------------------------------------------------------
__device__ __forceinline__ float4 tri2plane_f(float3 v0, float3 v1, float3 v2) {
  float ax = v1.x - v0.x, ay = v1.y - v0.y, az = v1.z - v0.z;
  float bx = v2.x - v0.x, by = v2.y - v0.y, bz = v2.z - v0.z;
  float nx = ay * bz - az * by;
  float ny = az * bx - ax * bz;
  float nz = ax * by - ay * bx;
  return make_float4(nx, ny, nz, -(v0.x * nx + v0.y * ny + v0.z * nz));
}

__device__ __forceinline__ float4 bisector_f(float4 S, float4 B) {
  float dx = S.x - B.x, dy = S.y - B.y, dz = S.z - B.z;
  float ax = S.x + B.x, ay = S.y + B.y, az = S.z + B.z;
  float dot = (ax * dx + ay * dy + az * dz) + (B.w - S.w);
  return make_float4(dx, dy, dz, -dot / 2.f);
}

// det4x4_ref(p1, p2, p3, e) = m234 e.x - m134 e.y + m124 e.z - m123 e.w: the
// minors of the vertex's planes do not depend on e, and the reference rounds
// them before e comes in
struct Minors {
  double m234, m134, m124, m123;
};
__device__ __forceinline__ Minors det4x4_minors(float4 p1, float4 p2, float4 p3) {
  double a11 = p1.x, a12 = p2.x, a13 = p3.x;
  double a21 = p1.y, a22 = p2.y, a23 = p3.y;
  double a31 = p1.z, a32 = p2.z, a33 = p3.z;
  double a41 = p1.w, a42 = p2.w, a43 = p3.w;
  double m12 = a21 * a12 - a11 * a22;
  double m13 = a31 * a12 - a11 * a32;
  double m14 = a41 * a12 - a11 * a42;
  double m23 = a31 * a22 - a21 * a32;
  double m24 = a41 * a22 - a21 * a42;
  double m34 = a41 * a32 - a31 * a42;
  Minors m;
  m.m123 = m23 * a13 - m13 * a23 + m12 * a33;
  m.m124 = m24 * a13 - m14 * a23 + m12 * a43;
  m.m134 = m34 * a13 - m14 * a33 + m13 * a43;
  m.m234 = m34 * a23 - m24 * a33 + m23 * a43;
  return m;
}
__device__ __forceinline__ double det4x4_of(const Minors& m, float4 e) {
  double a14 = e.x, a24 = e.y, a34 = e.z, a44 = e.w;
  return (m.m234 * a14 - m.m134 * a24 + m.m124 * a34 - m.m123 * a44);
}
__device__ __forceinline__ double det4x4_ref(float4 p1, float4 p2, float4 p3, float4 e) {
  return det4x4_of(det4x4_minors(p1, p2, p3), e);
}

// float det3x3 of the three plane normals (convex_cell.cu:274-316, the w
// of the homogeneous vertex); zero means the vertex needs a perturbation
__device__ __forceinline__ float det3x3_f(float4 a, float4 b, float4 c) {
  float t1 = b.y * c.z - b.z * c.y;
  float t2 = a.y * c.z - a.z * c.y;
  float t3 = a.y * b.z - a.z * b.y;
  return a.x * t1 - b.x * t2 + c.x * t3;
}

// ------------------------------------------------------------------------
// FP32 filter: det4x4(p1,p2,p3,e) = sum_r e_r K_r, K_r the signed 3x3
// minors of the vertex planes.  |fl(K_r) - K_r| <= gamma_5 M_r (M_r the 3x3
// permanent), the FMA dot adds gamma_4 sum|e_r K_r|; the bound also covers
// the reference's FP64 evaluation (gamma_9 in double times the 4x4
// permanent), so a decided sign is the sign of the reference's FP64 det.
// ------------------------------------------------------------------------
// A result below 2^-126 is rounded to a multiple of 2^-149, whatever its size:
// the 2x2 minors are then off by up to 2^-149 and the determinant by
// 2^-149 (|a1| + |b1| + |c1|) + 3 2^-150 more than in proportion to the
// permanent.  The permanents therefore start from kMinorFloor in place of
// zero, which in 6 u times them is at least four times that, and they stay
// clear of the subnormals themselves (above 2^-100 the floor does not show).
// Without it the lanes' clipper gives 6,106 of 195,492 pairs other records in a
// scene of 1.5e-5 units (48k tets), 47 in one of 3e-5.
constexpr float kMinorFloor = 2.3509887e-38f;  // 2^-125
__device__ __forceinline__ void minor3(float a1, float b1, float c1, float a2,
                                       float b2, float c2, float a3, float b3,
                                       float c3, float& det, float& perm) {
  float u1 = __fmaf_rn(b2, c3, -(b3 * c2));
  float u2 = __fmaf_rn(a2, c3, -(a3 * c2));
  float u3 = __fmaf_rn(a2, b3, -(a3 * b2));
  det = __fmaf_rn(a1, u1, __fmaf_rn(-b1, u2, c1 * u3));
  float v1 = __fmaf_rn(fabsf(b2), fabsf(c3), __fmaf_rn(fabsf(b3), fabsf(c2), kMinorFloor));
  float v2 = __fmaf_rn(fabsf(a2), fabsf(c3), __fmaf_rn(fabsf(a3), fabsf(c2), kMinorFloor));
  float v3 = __fmaf_rn(fabsf(a2), fabsf(b3), __fmaf_rn(fabsf(a3), fabsf(b2), kMinorFloor));
  perm = __fmaf_rn(fabsf(a1), v1,
                   __fmaf_rn(fabsf(b1), v2, __fmaf_rn(fabsf(c1), v3, kMinorFloor)));
}

__device__ __forceinline__ void vertex_cofactors(float4 p1, float4 p2, float4 p3,
                                                 float4& K, float4& M) {
  float d;
  minor3(p1.y, p1.z, p1.w, p2.y, p2.z, p2.w, p3.y, p3.z, p3.w, d, M.x);
  K.x = -d;
  minor3(p1.x, p1.z, p1.w, p2.x, p2.z, p2.w, p3.x, p3.z, p3.w, d, M.y);
  K.y = d;
  minor3(p1.x, p1.y, p1.w, p2.x, p2.y, p2.w, p3.x, p3.y, p3.w, d, M.z);
  K.z = -d;
  minor3(p1.x, p1.y, p1.z, p2.x, p2.y, p2.z, p3.x, p3.y, p3.z, d, M.w);
  K.w = d;
}

constexpr float kFiltC1 = 5.0f * 5.9604645e-08f;
constexpr float kFiltC2 = 6.0f * 5.9604645e-08f;
constexpr float kFiltAbs = 1e-30f;

// +1 / -1 decided, 0 undecided.  Bound: c1 sum|e_r K_r| (rounding of the
// dot) + c2 sum|e_r| M_r (rounding of the cofactors, and of the reference's
// own FP64 evaluation, both proportional to the 4x4 permanent
// sum_r |e_r| M_r)
__device__ __forceinline__ int filter_sign(float4 K, float4 M, float4 e) {
  float s = __fmaf_rn(e.w, K.w, __fmaf_rn(e.z, K.z, __fmaf_rn(e.y, K.y, e.x * K.x)));
  float t = __fmaf_rn(fabsf(e.w), fabsf(K.w),
                      __fmaf_rn(fabsf(e.z), fabsf(K.z),
                                __fmaf_rn(fabsf(e.y), fabsf(K.y), fabsf(e.x) * fabsf(K.x))));
  float pm = __fmaf_rn(fabsf(e.w), M.w,
                       __fmaf_rn(fabsf(e.z), M.z, __fmaf_rn(fabsf(e.y), M.y, fabsf(e.x) * M.x)));
  float b = __fmaf_rn(kFiltC1, t, kFiltC2 * pm) + kFiltAbs;
  return s > b ? 1 : (s < -b ? -1 : 0);
}

// ------------------------------------------------------------------------
// FP64 error bound and exact sign of det4x4 (RPD_PRED_EXACT)
// ------------------------------------------------------------------------
// |det4x4_ref - exact| <= gamma_8 P, P the same expression over absolute
// values: products of two floats are exact in FP64 and at most 8 other
// operations lie on any path.  P = sum_r |e_r| M_r with the permanents M of
// the vertex's planes, which the filter holds in FP32 to 6 u and not below
// kMinorFloor: the sum starts from the floor as well, which covers what its
// terms lose in the subnormals.
__device__ __forceinline__ double det4x4_bound(float4 M, float4 e) {
  const float pm = __fmaf_rn(fabsf(e.w), M.w,
                             __fmaf_rn(fabsf(e.z), M.z,
                                       __fmaf_rn(fabsf(e.y), M.y,
                                                 __fmaf_rn(fabsf(e.x), M.x, kMinorFloor))));
  return 10.0 * 1.1102230246251565e-16 * (1.0 + 2e-6) * (double)pm + 1e-300;
}

// The sign of the exact determinant from its 24 products, in straight-line
// arithmetic: a product of four floats is the product of two exact FP64
// products, so a multiplication and an FMA give it exactly as hi + lo (no
// product of four floats overflows, and no residual underflows).  The terms
// are summed in two levels of TwoSum; what falls off the second is only
// summed in magnitude (`lost`).  The sign is that of the sum where it exceeds
// twice `lost`, or where nothing was lost; returns 2 where neither holds (the
// expansions decide then).  Expansions took 4,800 SM cycles a sign (local
// arrays, a path of its own for every lane); 146k-tet lattice, 482k exact
// signs: clip stage 8.2 -> 5.4 ms.
static __device__ __noinline__ int det4x4_sum_sign(float4 p1, float4 p2, float4 p3, float4 e) {
  const double A[4] = {p1.x, p1.y, p1.z, p1.w}, B[4] = {p2.x, p2.y, p2.z, p2.w};
  const double C[4] = {p3.x, p3.y, p3.z, p3.w}, E[4] = {e.x, e.y, e.z, e.w};
  double s = 0.0, c = 0.0, lost = 0.0;
  auto second = [&](double x) {
    const double t = c + x, v = t - c;
    lost += fabs((c - (t - v)) + (x - v));
    c = t;
  };
  auto first = [&](double x) {
    const double t = s + x, v = t - s;
    second((s - (t - v)) + (x - v));
    s = t;
  };
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j == i) continue;
      const double ab = A[i] * B[j];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k == i || k == j) continue;
        const int l = 6 - i - j - k;
        const int inversions = (i > j) + (i > k) + (i > l) + (j > k) + (j > l) + (k > l);
        const double f = (inversions & 1) ? -C[k] * E[l] : C[k] * E[l];
        const double hi = ab * f;
        first(hi);
        second(fma(ab, f, -hi));
      }
    }
  const double t = s + c;
  if (lost == 0.0 || fabs(t) > 2.0 * lost) return t > 0.0 ? 1 : (t < 0.0 ? -1 : 0);
  return 2;
}

// Exact sign by floating-point expansions (Shewchuk, "Adaptive precision
// floating-point arithmetic and fast robust geometric predicates", Discrete
// Comput. Geom. 18, 1997): TwoSum, TwoProduct (with FMA),
// FAST-EXPANSION-SUM and SCALE-EXPANSION, both with zero elimination.
// Expansions are nonoverlapping, in increasing magnitude.
__device__ __forceinline__ void ex_two_sum(double a, double b, double& x, double& y) {
  x = a + b;
  const double bv = x - a;
  const double av = x - bv;
  y = (a - av) + (b - bv);
}
__device__ __forceinline__ void ex_fast_two_sum(double a, double b, double& x, double& y) {
  x = a + b;
  y = b - (x - a);
}
__device__ __forceinline__ void ex_two_prod(double a, double b, double& x, double& y) {
  x = a * b;
  y = fma(a, b, -x);
}

static __device__ int ex_sum(int elen, const double* e, int flen, const double* f, double* h) {
  int ei = 0, fi = 0, hi = 0;
  double en = e[0], fn = f[0], Q, Qn, hh;
  if ((fn > en) == (fn > -en)) {
    Q = en;
    en = ++ei < elen ? e[ei] : 0.0;
  } else {
    Q = fn;
    fn = ++fi < flen ? f[fi] : 0.0;
  }
  if (ei < elen && fi < flen) {
    if ((fn > en) == (fn > -en)) {
      ex_fast_two_sum(en, Q, Qn, hh);
      en = ++ei < elen ? e[ei] : 0.0;
    } else {
      ex_fast_two_sum(fn, Q, Qn, hh);
      fn = ++fi < flen ? f[fi] : 0.0;
    }
    Q = Qn;
    if (hh != 0.0) h[hi++] = hh;
    while (ei < elen && fi < flen) {
      if ((fn > en) == (fn > -en)) {
        ex_two_sum(Q, en, Qn, hh);
        en = ++ei < elen ? e[ei] : 0.0;
      } else {
        ex_two_sum(Q, fn, Qn, hh);
        fn = ++fi < flen ? f[fi] : 0.0;
      }
      Q = Qn;
      if (hh != 0.0) h[hi++] = hh;
    }
  }
  while (ei < elen) {
    ex_two_sum(Q, en, Qn, hh);
    en = ++ei < elen ? e[ei] : 0.0;
    Q = Qn;
    if (hh != 0.0) h[hi++] = hh;
  }
  while (fi < flen) {
    ex_two_sum(Q, fn, Qn, hh);
    fn = ++fi < flen ? f[fi] : 0.0;
    Q = Qn;
    if (hh != 0.0) h[hi++] = hh;
  }
  if (Q != 0.0 || hi == 0) h[hi++] = Q;
  return hi;
}

static __device__ int ex_scale(int elen, const double* e, double b, double* h) {
  int hi = 0;
  double Q, hh, p1, p0, sum;
  ex_two_prod(e[0], b, Q, hh);
  if (hh != 0.0) h[hi++] = hh;
  for (int i = 1; i < elen; ++i) {
    ex_two_prod(e[i], b, p1, p0);
    ex_two_sum(Q, p0, sum, hh);
    if (hh != 0.0) h[hi++] = hh;
    ex_fast_two_sum(p1, sum, Q, hh);
    if (hh != 0.0) h[hi++] = hh;
  }
  if (Q != 0.0 || hi == 0) h[hi++] = Q;
  return hi;
}

// 2x2 minor a*b - c*d of floats (both products exact in FP64)
__device__ __forceinline__ int ex_minor2(double a, double b, double c, double d, double* h) {
  double x, y;
  ex_two_sum(a * b, -(c * d), x, y);
  int n = 0;
  if (y != 0.0) h[n++] = y;
  if (x != 0.0 || n == 0) h[n++] = x;
  return n;
}

// u*a - v*b + w*c for expansions u, v, w (<= lu, lv, lw terms)
static __device__ int ex_combine3(const double* u, int lu, double a, const double* v, int lv, double b,
                           const double* w, int lw, double c, double* h) {
  double t1[24], t2[24], t3[24], t12[48];
  const int n1 = ex_scale(lu, u, a, t1);
  const int n2 = ex_scale(lv, v, -b, t2);
  const int n3 = ex_scale(lw, w, c, t3);
  const int n12 = ex_sum(n1, t1, n2, t2, t12);
  return ex_sum(n12, t12, n3, t3, h);
}

// exact sign of det4x4_ref's determinant (same matrix, no rounding)
static __device__ __noinline__ int det4x4_exact_sign(float4 p1, float4 p2, float4 p3, float4 e) {
  const double a11 = p1.x, a12 = p2.x, a13 = p3.x, a14 = e.x;
  const double a21 = p1.y, a22 = p2.y, a23 = p3.y, a24 = e.y;
  const double a31 = p1.z, a32 = p2.z, a33 = p3.z, a34 = e.z;
  const double a41 = p1.w, a42 = p2.w, a43 = p3.w, a44 = e.w;
  double m12[2], m13[2], m14[2], m23[2], m24[2], m34[2];
  const int l12 = ex_minor2(a21, a12, a11, a22, m12);
  const int l13 = ex_minor2(a31, a12, a11, a32, m13);
  const int l14 = ex_minor2(a41, a12, a11, a42, m14);
  const int l23 = ex_minor2(a31, a22, a21, a32, m23);
  const int l24 = ex_minor2(a41, a22, a21, a42, m24);
  const int l34 = ex_minor2(a41, a32, a31, a42, m34);
  double m123[12], m124[12], m134[12], m234[12];
  const int l123 = ex_combine3(m23, l23, a13, m13, l13, a23, m12, l12, a33, m123);
  const int l124 = ex_combine3(m24, l24, a13, m14, l14, a23, m12, l12, a43, m124);
  const int l134 = ex_combine3(m34, l34, a13, m14, l14, a33, m13, l13, a43, m134);
  const int l234 = ex_combine3(m34, l34, a23, m24, l24, a33, m23, l23, a43, m234);
  // m234 a14 - m134 a24 + m124 a34 - m123 a44
  double t1[24], t2[24], t3[24], t4[24], s12[48], s34[48], d[96];
  const int n1 = ex_scale(l234, m234, a14, t1);
  const int n2 = ex_scale(l134, m134, -a24, t2);
  const int n3 = ex_scale(l124, m124, a34, t3);
  const int n4 = ex_scale(l123, m123, -a44, t4);
  const int n12 = ex_sum(n1, t1, n2, t2, s12);
  const int n34 = ex_sum(n3, t3, n4, t4, s34);
  const int n = ex_sum(n12, s12, n34, s34, d);
  const double top = d[n - 1];
  return top > 0.0 ? 1 : (top < 0.0 ? -1 : 0);
}

__device__ __forceinline__ bool plane_eq(float4 a, float4 b) {
  return a.x == b.x && a.y == b.y && a.z == b.z && a.w == b.w;
}

// predicate statistics of a thread: evaluated, escalated to FP64; and where
// the escalations of RPD_PRED_EXACT count their FP64-uncertain / exact-flip
// cases
struct PredCount {
  uint32_t pred, esc;
  unsigned long long* exact;
};

__host__ __device__ constexpr bool uses_filter(int pred) {
  return pred == RPD_PRED_FP32_FILTER || pred == RPD_PRED_EXACT;
}

// RPD_PRED_EXACT: the predicates the filter cannot decide, out of line
// (rare); M the permanents of the three planes.  kSignConflict where they
// conflict, kSignUncertain where the FP64 sign is not certified by its error
// bound (decided exactly), kSignFlip where the exact sign differs from it
enum SignBits { kSignConflict = 1, kSignUncertain = 2, kSignFlip = 4, kSignEscalated = 8 };
static __device__ __noinline__ int exact_conflict(float4 p1, float4 p2, float4 p3, float4 e,
                                                  float4 M) {
  const double d = det4x4_ref(p1, p2, p3, e);
  if (fabs(d) > det4x4_bound(M, e)) return d > 0.0 ? kSignConflict : 0;
  int xs = det4x4_sum_sign(p1, p2, p3, e);
  if (xs == 2) xs = det4x4_exact_sign(p1, p2, p3, e);
  return kSignUncertain | (xs > 0 ? kSignConflict : 0) | ((xs > 0) != (d > 0.0) ? kSignFlip : 0);
}

// ------------------------------------------------------------------------
// security-radius certificate (lists in ascending bisector distance)
// ------------------------------------------------------------------------
// Every vertex x of the cell satisfies x = K_xyz / K_w (K its cofactors), so
// |x - S| <= (|K_xyz - K_w S| + e) / (|K_w| - e_w) with e, e_w the cofactor
// error bounds (gamma_5 times the permanents M) and the rounding of the
// translation.  A neighbour j whose power bisector lies at distance d_j from
// the seed S cannot clip a cell inside the ball B(S, R): every point x of
// the ball has exact bisector value >= |n_j| (d_j - |x - S|) > 0, and the
// margin below covers the float rounding of the key d_j, of the float plane
// itself (<= 9uL + 4u|w_i - w_j| / |n_j| for coordinates below L), and of the
// predicate.  Keys ascend along the list, so one test of the next key
// certifies every remaining neighbour.
__device__ __forceinline__ float vertex_radius(float4 K, float4 M, float3 S) {
  const float g = 6.0f * 5.9604645e-08f;
  float ew = g * M.w;
  float aw = fabsf(K.w);
  if (!(aw > ew)) return INFINITY;
  float nx = __fmaf_rn(-K.w, S.x, K.x), ny = __fmaf_rn(-K.w, S.y, K.y),
        nz = __fmaf_rn(-K.w, S.z, K.z);
  float ex = g * (M.x + fabsf(S.x) * M.w) + 2.4e-7f * fabsf(nx);
  float ey = g * (M.y + fabsf(S.y) * M.w) + 2.4e-7f * fabsf(ny);
  float ez = g * (M.z + fabsf(S.z) * M.w) + 2.4e-7f * fabsf(nz);
  float ax = fabsf(nx) + ex, ay = fabsf(ny) + ey, az = fabsf(nz) + ez;
  const float n2 = ax * ax + ay * ay + az * az;
  float n = sqrtf(n2);
  if (n2 < 1e-30f) {
    // the squares underflow, to a radius of zero that certifies any cell
    // (48k tets in 1e-3 units and less; some vertices from 3e-2 down)
    constexpr float up = 1.2676506e30f;  // 2^100
    ax *= up;
    ay *= up;
    az *= up;
    n = sqrtf(ax * ax + ay * ay + az * az) * (1.0f / up);
  }
  return n * (1.0f + 1e-6f) / (aw - ew) * (1.0f + 1e-6f);
}

// The same bound in FP64, for a vertex whose FP32 bound is loose or void
// (|K_w| close to its error: nearly parallel planes, as at the faces of
// sliver tets).  Products of two floats are exact in double and every 3x3
// minor rounds at most 3 times, so each cofactor is within 4 eps of its
// permanent (eps = 2^-53); the translation by S and the norm add a few eps.
static __device__ __noinline__ float vertex_radius_d(float4 p1, float4 p2, float4 p3, float3 S) {
  const double x1 = p1.x, y1 = p1.y, z1 = p1.z, w1 = p1.w;
  const double x2 = p2.x, y2 = p2.y, z2 = p2.z, w2 = p2.w;
  const double x3 = p3.x, y3 = p3.y, z3 = p3.z, w3 = p3.w;
  // det3 of rows (a_i, b_i, c_i) and its permanent
  auto d3 = [](double a1, double b1, double c1, double a2, double b2, double c2, double a3,
               double b3, double c3, double& perm) {
    perm = fabs(a1) * (fabs(b2 * c3) + fabs(b3 * c2)) + fabs(b1) * (fabs(a2 * c3) + fabs(a3 * c2)) +
           fabs(c1) * (fabs(a2 * b3) + fabs(a3 * b2));
    return a1 * (b2 * c3 - b3 * c2) - b1 * (a2 * c3 - a3 * c2) + c1 * (a2 * b3 - a3 * b2);
  };
  double Mx, My, Mz, Mw;
  const double Kx = -d3(y1, z1, w1, y2, z2, w2, y3, z3, w3, Mx);
  const double Ky = d3(x1, z1, w1, x2, z2, w2, x3, z3, w3, My);
  const double Kz = -d3(x1, y1, w1, x2, y2, w2, x3, y3, w3, Mz);
  const double Kw = d3(x1, y1, z1, x2, y2, z2, x3, y3, z3, Mw);
  const double eps = 1.1102230246251565e-16;
  const double ew = 4.0 * eps * Mw;
  const double aw = fabs(Kw);
  if (!(aw > 2.0 * ew)) return INFINITY;
  const double sx = S.x, sy = S.y, sz = S.z;
  const double nx = Kx - Kw * sx, ny = Ky - Kw * sy, nz = Kz - Kw * sz;
  const double ex = 4.0 * eps * (Mx + fabs(sx) * Mw) + 2.0 * eps * fabs(nx);
  const double ey = 4.0 * eps * (My + fabs(sy) * Mw) + 2.0 * eps * fabs(ny);
  const double ez = 4.0 * eps * (Mz + fabs(sz) * Mw) + 2.0 * eps * fabs(nz);
  const double ax = fabs(nx) + ex, ay = fabs(ny) + ey, az = fabs(nz) + ez;
  const double r = sqrt(ax * ax + ay * ay + az * az) * (1.0 + 8.0 * eps) / (aw - ew);
  return __double2float_ru(r * (1.0 + 8.0 * eps));
}

// the radius bound of a vertex: FP32 where it is tight (its upper and lower
// bounds within 2^-10 of each other), else FP64 -- the FP32 cofactors of
// nearly parallel planes (the faces of sliver tets) cancel, and their error
// terms can exceed the distance itself
__device__ __forceinline__ float vertex_radius_p(float4 K, float4 M, float3 S, float4 p1,
                                                 float4 p2, float4 p3) {
  const float g = 6.0f * 5.9604645e-08f;
  const float ew = g * M.w, aw = fabsf(K.w);
  if (aw > 64.0f * ew) {
    const float nx = __fmaf_rn(-K.w, S.x, K.x), ny = __fmaf_rn(-K.w, S.y, K.y),
                nz = __fmaf_rn(-K.w, S.z, K.z);
    const float e = g * (M.x + M.y + M.z + (fabsf(S.x) + fabsf(S.y) + fabsf(S.z)) * M.w) +
                    2.4e-7f * (fabsf(nx) + fabsf(ny) + fabsf(nz));
    const float n = sqrtf(nx * nx + ny * ny + nz * nz);
    if (e < n * (1.0f / 2048.0f)) return vertex_radius(K, M, S);
  }
  return vertex_radius_d(p1, p2, p3, S);
}

__device__ __forceinline__ bool cert_holds(float key, float R, float margin) {
  return key * (1.0f - 64.0f * 5.9604645e-08f) - margin > R;
}

}  // namespace rpd
