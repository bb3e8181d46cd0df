// Device functions of the SBR path: closest hit, reception sphere, image
// correction and the received field.  Reference behaviour is cited per
// function (paths relative to SBRSolver_rev2/).
#pragma once

#include <cfloat>
#include <climits>
#include <cuda_runtime.h>

#include "sbr_device.h"
#include "sbr_soft64.cuh"

namespace sbr {

constexpr double kEps64 = 1.1920928955078125e-07;  // FLT_EPSILON as double, Constants.h:13
constexpr float kEps32 = 1.1920928955078125e-07f;
// FP32 filter margin factor of the triangle tests, 2^-18: with unit roundoff
// e = 2^-24, the rounded inputs (2e per product) and the rounding of each
// operation give |dh| <= 7e |d||e2| for h = d x e2, |ds| <= 2e (|o| + |v1|) for
// s = o - v1, hence errors under 11e |e1||e2||d| of a = e1 . h, 12e of
// U = s . h, and with |dq| <= 9e for q = s x e1, 13e of V = d . q and
// W = e2 . q, each relative to the magnitudes the margins are formed from.
// 64e leaves a factor of four and more.  The factor was 2^-14 before: the
// level-10 terrain solve then left 14 % of its contenders to FP64 for their
// edges (now 2 %) and sent 8,738 rays with more than eight contenders to the
// one-pass search (now 15).
constexpr float kFiltK = 3.814697265625e-06f;
// The image correction's filters keep 2^-14: their direction is the
// difference of two rounded points, with an error relative to the points.
constexpr float kCorrK = 6.103515625e-05f;
constexpr float kBoxK = 6.103515625e-05f;  // 2^-14 |origin|: FP32 box expansion
// Margin factor of the FP32 reception test: |dist - radius| and the
// projection are decided in FP32 only when they clear this times the
// magnitudes involved (|segment start| + |receiver| + 1 + unfolded length).
// Bounding every rounding of the FP32 evaluation and of its rounded inputs
// against the FP64 test gives under 30 * 2^-24 of the same magnitudes.
#ifndef SBR_REC_K
#define SBR_REC_K 1.52587890625e-05f  // 2^-16
#endif
constexpr float kRecK = SBR_REC_K;
// Relative slack when a bound on a contender's t is compared with another
// hit's t: a contender whose lower bound exceeds t * (1 + kTieSlack) lies
// farther along the ray, so its FP64 distance is larger (distances of one ray
// are t |d| to within a few FP64 ulps); the slack covers that and the FP32
// rounding of the product.
#ifndef SBR_TIE_SLACK
#define SBR_TIE_SLACK 9.5367431640625e-07f  // 2^-20
#endif
constexpr float kTieSlack = SBR_TIE_SLACK;

struct Hit {
  double t, dist;
  double p[3];
  int rank;  // index in depth-first triangle order, INT_MAX = no hit
  int leaf;
};

// Products, quotients and roots of the FP64 tests: on the FP64 pipe, or in
// integer arithmetic (sbr_soft64.cuh; the same bits for operands in its range).
struct Pipe64 {
  static constexpr bool kSoft = false;
  static __device__ __forceinline__ double mul(double a, double b) { return x64::mul(a, b); }
  // 1.0 / a (Triangle.cpp): the correctly rounded reciprocal is the same
  // double as the correctly rounded quotient 1.0 / a
  static __device__ __forceinline__ double rcp(double a) { return __drcp_rn(a); }
  static __device__ __forceinline__ double sqrt(double a) { return x64::sqrt_(a); }
};
struct Soft64 {
  static constexpr bool kSoft = true;
  static __device__ __forceinline__ double mul(double a, double b) { return soft64::mul(a, b); }
  static __device__ __forceinline__ double rcp(double a) { return soft64::rcp(a); }
  static __device__ __forceinline__ double sqrt(double a) { return soft64::sqrt(a); }
};
// The dot and cross products of the integer form are functions: they are used
// nine times, and inline their products alone are 20 KB of code, in a kernel
// (k_trace) whose warps wait for instructions a third of the time.
struct D3 {
  double x, y, z;
};
__device__ __noinline__ double dot_soft(double a0, double a1, double a2, double b0, double b1,
                                        double b2) {
  return x64::add(x64::add(soft64::mul(a0, b0), soft64::mul(a1, b1)), soft64::mul(a2, b2));
}
__device__ __noinline__ D3 cross_soft(double a0, double a1, double a2, double b0, double b1,
                                      double b2) {
  return D3{x64::sub(soft64::mul(a1, b2), soft64::mul(a2, b1)),
            x64::sub(soft64::mul(a2, b0), soft64::mul(a0, b2)),
            x64::sub(soft64::mul(a0, b1), soft64::mul(a1, b0))};
}
template <class A>
__device__ __forceinline__ double dot64(const double* a, const double* b) {
  if (A::kSoft) return dot_soft(a[0], a[1], a[2], b[0], b[1], b[2]);
  return x64::dot(a, b);
}
template <class A>
__device__ __forceinline__ void cross64(const double* a, const double* b, double* r) {
  if (A::kSoft) {
    const D3 v = cross_soft(a[0], a[1], a[2], b[0], b[1], b[2]);
    r[0] = v.x;
    r[1] = v.y;
    r[2] = v.z;
  } else {
    x64::cross(a, b, r);
  }
}

// Triangle::RayIntersects (Triangle.cpp:80-124), FP64, reference operation
// order.  uv_sure: the FP32 filter has shown that the reference's tests of u
// and v accept (tri_classify), so they are not formed.  It returns early
// for a parallel ray, for u and v together (formed side by side) and for t.
// Comparisons are integer ones, which decide alike without the FP64 pipe.
template <class A>
__device__ __forceinline__ bool mt64_t(const Tri64& T, const double* o, const double* d,
                                       bool uv_sure, double& t, double* P, double& dist) {
  using x64::add;
  double h[3], s[3], q[3];
  cross64<A>(d, T.e2, h);
  const double a = dot64<A>(T.e1, h);
  if (soft64::magnitude_below(a, kEps64)) return false;
  const double f = A::rcp(a);
  x64::sub3(o, T.v1, s);
  cross64<A>(s, T.e1, q);
  if (!uv_sure) {
    const double u = A::mul(f, dot64<A>(s, h));
    const double v = A::mul(f, dot64<A>(d, q));
    if (soft64::negative(u) || soft64::above(u, 1.0) || soft64::negative(v) ||
        soft64::above(add(u, v), 1.0))
      return false;
  }
  const double tt = A::mul(f, dot64<A>(T.e2, q));
  if (!soft64::above(tt, kEps64)) return false;
  P[0] = add(o[0], A::mul(d[0], tt));
  P[1] = add(o[1], A::mul(d[1], tt));
  P[2] = add(o[2], A::mul(d[2], tt));
  double w[3];
  x64::sub3(P, o, w);
  dist = A::sqrt(dot64<A>(w, w));
  t = tt;
  return true;
}
__device__ __forceinline__ bool mt64(const Tri64& T, const double* o, const double* d, double& t,
                                     double* P, double& dist) {
  return mt64_t<Pipe64>(T, o, d, false, t, P, dist);
}

// mt64 out of line, for the rare ray outside soft64's range: the arguments go
// by value, so the caller's ray stays in registers.
struct Mt64Result {
  bool ok;
  double t, dist, p[3];
};
__device__ __noinline__ Mt64Result mt64_call(const Tri64* T, double ox, double oy, double oz,
                                             double dx, double dy, double dz) {
  const double o[3] = {ox, oy, oz}, d[3] = {dx, dy, dz};
  Mt64Result r;
  r.ok = mt64(*T, o, d, r.t, r.p, r.dist);
  return r;
}

// Same test on a CorrTri (image correction looks triangles up by mesh position).
__device__ __forceinline__ bool mt64c(const CorrTri& T, const double* o, const double* d,
                                      double* P) {
  Tri64 t;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t.v1[i] = T.v1[i];
    t.e1[i] = T.e1[i];
    t.e2[i] = T.e2[i];
  }
  double tt, dist;
  return mt64(t, o, d, tt, P, dist);
}

// BVHNode::IntersectsAABB (BVH/BVHNode.h:64-85), FP64, with std::min/std::max
// argument order so NaN slabs are ignored exactly as the reference ignores them.
__device__ __forceinline__ bool slab64(const double* bb, const double* o, const double* d) {
  using namespace x64;
  double tmax = __longlong_as_double(0x7ff0000000000000ll);
  double tmin = -tmax;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double t1 = div(sub(bb[i], o[i]), d[i]);
    const double t2 = div(sub(bb[3 + i], o[i]), d[i]);
    const double tn = (t2 < t1) ? t2 : t1;
    const double tf = (t1 < t2) ? t2 : t1;
    tmax = (tf < tmax) ? tf : tmax;
    tmin = (tmin < tn) ? tn : tmin;
    if (tmin > tmax) return false;
  }
  return true;
}

// BVH::RayIntersects (BVH/BVH.h:276-328) exactly: depth-first, both children,
// children[0] first, strict '<' on distance so the first visited wins ties.
__device__ __noinline__ bool exact_closest(const DevScene& sc, const double* o, const double* d,
                                           Hit& best, unsigned* overflow) {
  int stack[kStack];
  int sp = 0;
  stack[sp++] = 0;
  best.rank = INT_MAX;
  best.dist = __longlong_as_double(0x7ff0000000000000ll);
  while (sp > 0) {
    const int n = stack[--sp];
    const RefNode& nd = sc.ref[n];
    if (!slab64(nd.bb, o, d)) continue;
    if (nd.c0 >= 0) {
      if (sp + 2 > kStack) {
        atomicOr(overflow, kOvStack);
        return false;
      }
      stack[sp++] = nd.c1;
      stack[sp++] = nd.c0;
    } else {
      for (int r = nd.first; r < nd.first + nd.count; ++r) {
        double t, P[3], dist;
        if (mt64(sc.tri64[r], o, d, t, P, dist) && dist < best.dist) {
          best.dist = dist;
          best.t = t;
          best.p[0] = P[0];
          best.p[1] = P[1];
          best.p[2] = P[2];
          best.rank = r;
          best.leaf = n;
        }
      }
    }
  }
  return best.rank != INT_MAX;
}

// FP32 Moller-Trumbore filter with error margins.  Returns false only when
// the FP64 test certainly rejects; otherwise tlo is a lower bound on t.
__device__ __forceinline__ bool tri_filter(const Tri32& T, const float3& o, const float3& d,
                                           float no, float nd, float& tlo) {
  const float hx = d.y * T.e2[2] - d.z * T.e2[1];
  const float hy = d.z * T.e2[0] - d.x * T.e2[2];
  const float hz = d.x * T.e2[1] - d.y * T.e2[0];
  const float a = T.e1[0] * hx + T.e1[1] * hy + T.e1[2] * hz;
  const float sx = o.x - T.v1[0], sy = o.y - T.v1[1], sz = o.z - T.v1[2];
  float U = sx * hx + sy * hy + sz * hz;
  const float qx = sy * T.e1[2] - sz * T.e1[1];
  const float qy = sz * T.e1[0] - sx * T.e1[2];
  const float qz = sx * T.e1[1] - sy * T.e1[0];
  float V = d.x * qx + d.y * qy + d.z * qz;
  float W = T.e2[0] * qx + T.e2[1] * qy + T.e2[2] * qz;
  const float ns = no + T.nv1;
  const float ea = kCorrK * T.ne1 * T.ne2 * nd;
  const float eU = kCorrK * ns * nd * T.ne2;
  const float eV = kCorrK * ns * T.ne1 * nd;
  const float eW = kCorrK * ns * T.ne1 * T.ne2;
  const float A = fabsf(a);
  if (A <= kEps32 + ea) {  // near-parallel: the FP64 test decides
    tlo = 0.0f;
    return true;
  }
  if (a < 0.0f) {
    U = -U;
    V = -V;
    W = -W;
  }
  if (U < -eU || V < -eV) return false;
  if (U > A + ea + eU) return false;
  if (U + V > A + ea + eU + eV) return false;
  const float thi = (W + eW) / (A - ea);
  if (thi <= kEps32 * 0.5f) return false;
  tlo = (W - eW) / (A + ea);
  return true;
}

// tri_filter's terms that depend only on the origin o and the triangle, for many
// rays from one image source towards many receivers (line_may_cross).
struct TriFrom {
  float sx, sy, sz;  // o - v1
  float qx, qy, qz;  // (o - v1) x e1
  float W;           // e2 . q
  float ns;          // |o| + |v1|
};

__device__ __forceinline__ TriFrom tri_from(const Tri32& T, const float3& o, float no) {
  TriFrom F;
  F.sx = o.x - T.v1[0];
  F.sy = o.y - T.v1[1];
  F.sz = o.z - T.v1[2];
  F.qx = F.sy * T.e1[2] - F.sz * T.e1[1];
  F.qy = F.sz * T.e1[0] - F.sx * T.e1[2];
  F.qz = F.sx * T.e1[1] - F.sy * T.e1[0];
  F.W = T.e2[0] * F.qx + T.e2[1] * F.qy + T.e2[2] * F.qz;
  F.ns = no + T.nv1;
  return F;
}

// As tri_filter, also telling what the FP64 test certainly decides: 0 = it
// misses, else kMayHit, with kSureUV when its tests of u and v accept and
// kSureHit when it hits.  [tlo, thi] bounds t.
constexpr int kMayHit = 1, kSureHit = 2, kSureUV = 4;
__device__ __forceinline__ int tri_classify(const Tri32& T, const float3& o, const float3& d,
                                            float no, float nd, float& tlo, float& thi) {
  const float hx = d.y * T.e2[2] - d.z * T.e2[1];
  const float hy = d.z * T.e2[0] - d.x * T.e2[2];
  const float hz = d.x * T.e2[1] - d.y * T.e2[0];
  const float a = T.e1[0] * hx + T.e1[1] * hy + T.e1[2] * hz;
  const float sx = o.x - T.v1[0], sy = o.y - T.v1[1], sz = o.z - T.v1[2];
  float U = sx * hx + sy * hy + sz * hz;
  const float qx = sy * T.e1[2] - sz * T.e1[1];
  const float qy = sz * T.e1[0] - sx * T.e1[2];
  const float qz = sx * T.e1[1] - sy * T.e1[0];
  float V = d.x * qx + d.y * qy + d.z * qz;
  float W = T.e2[0] * qx + T.e2[1] * qy + T.e2[2] * qz;
  const float k = kFiltK * (no + T.nv1), kd = k * nd;
  const float eU = kd * T.ne2, eV = kd * T.ne1, eW = k * T.ne2 * T.ne1;
  const float ea = kFiltK * nd * T.ne1 * T.ne2;
  const float A = fabsf(a);
  U = copysignf(1.0f, a) * U;
  V = copysignf(1.0f, a) * V;
  W = copysignf(1.0f, a) * W;
  // one decision at the end: the lanes of a warp reject for different reasons
  const bool miss = U < -eU || V < -eV || U + V > A + ea + eU + eV ||
                    W + eW <= (kEps32 * 0.5f) * (A - ea);
  if (A <= kEps32 + ea) {  // near-parallel: the FP64 test decides
    tlo = 0.0f;
    thi = INFINITY;
    return kMayHit;
  }
  if (miss) return 0;
  // (approximate quotients: the margins exceed W's and a's errors by more than
  // 2^-19 of W and A, the quotient's error is 2^-22)
  thi = __fdividef(W + eW, A - ea);
  tlo = __fdividef(W - eW, A + ea);
  const bool uv = U > eU && V > eV && U + V < A - ea - eU - eV;
  return kMayHit | (uv ? (tlo > 2.0f * kEps32 ? kSureUV | kSureHit : kSureUV) : 0);
}

__device__ __forceinline__ void load_node(const Node32* nodes, int i, float4& f0, float4& f1,
                                          float4& f2, int2& ch) {
  const float4* p = reinterpret_cast<const float4*>(nodes + i);
  f0 = __ldg(p);
  f1 = __ldg(p + 1);
  f2 = __ldg(p + 2);
  const float4 f3 = __ldg(p + 3);
  ch = make_int2(__float_as_int(f3.x), __float_as_int(f3.y));
}

__device__ __forceinline__ void slab32(float lx, float ly, float lz, float hx, float hy, float hz,
                                       const float3& o, const float3& inv, float m, float& tn,
                                       float& tf) {
  const float ax = ((lx - m) - o.x) * inv.x, bx = ((hx + m) - o.x) * inv.x;
  const float ay = ((ly - m) - o.y) * inv.y, by = ((hy + m) - o.y) * inv.y;
  const float az = ((lz - m) - o.z) * inv.z, bz = ((hz + m) - o.z) * inv.z;
  tn = fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fminf(az, bz));
  tf = fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fmaxf(az, bz));
}

struct TraceStats {
  unsigned fp64_tri, fallback;
};

// The reference's slab test (slab64) decided in FP32 where the error bounds
// allow: 1 = accepted, 0 = rejected, -1 = within the error bounds (run
// slab64).  Box bounds are float values (they come from float vertices), so
// only the origin, direction and the arithmetic carry FP32 error; each
// slab parameter t = (b - o) / d is within
//   e = 2^-20 (|lo| + |hi| + 2|o|) / |d|
// of its FP64 value.  A flat axis (lo == hi) gives one FP64 value t for both
// planes, so the FP64 test accepts iff the other axes' intervals contain it.
// inv = 1/d in FP32: a product with it differs from the quotient by a few
// ulps, far inside e.
// zeros: axes whose direction component is exactly 0 and whose planes lie on
// either side of the origin; their FP64 interval is everything.
__device__ __forceinline__ int slab_certain(const float* bb, int flatmask, const float3& o,
                                            const float3& d, const float3& inv, int zeros) {
  const float K = 9.5367431640625e-07f;  // 2^-20
  float A_lo = -INFINITY, A_hi = -INFINITY, B_lo = INFINITY, B_hi = INFINITY;
  float v = 0.0f, ev = 0.0f;
  int flat = 0;
  if (flatmask & 8) return -1;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float da = a == 0 ? d.x : (a == 1 ? d.y : d.z);
    const float oa = a == 0 ? o.x : (a == 1 ? o.y : o.z);
    const float ia = a == 0 ? inv.x : (a == 1 ? inv.y : inv.z);
    if (zeros >> a & 1) continue;
    if (da == 0.0f) return -1;
    const float lo = bb[a], hi = bb[3 + a];
    const float t1 = (lo - oa) * ia, t2 = (hi - oa) * ia;
    const float e = K * (fabsf(lo) + fabsf(hi) + 2.0f * fabsf(oa)) * fabsf(ia);
    if (!isfinite(t1) || !isfinite(t2) || !isfinite(e)) return -1;
    if (flatmask & (1 << a)) {
      if (flat++) return -1;
      v = t1;
      ev = e;
      continue;
    }
    const float tn = fminf(t1, t2), tf = fmaxf(t1, t2);
    A_lo = fmaxf(A_lo, tn - e);
    A_hi = fmaxf(A_hi, tn + e);
    B_lo = fminf(B_lo, tf - e);
    B_hi = fminf(B_hi, tf + e);
  }
  if (flat) {
    if (A_hi < v - ev && v + ev < B_lo) return 1;
    if (v + ev < A_lo || v - ev > B_hi || A_lo > B_hi) return 0;
    return -1;
  }
  if (A_hi < B_lo) return 1;
  if (A_lo > B_hi) return 0;
  return -1;
}

// Whether every box from `leaf` up to the root of the reference BVH passes the
// reference's slab test, i.e. whether the reference's traversal reaches the
// leaf.  An ancestor's box contains the leaf's, and FP64 subtraction and
// division by one direction component are monotone, so each of the ancestor's
// slab intervals contains the leaf's exactly as computed, and the leaf's own
// test decides for the whole chain.  A zero component gives an infinite
// interval for every box whose planes lie on either side of the origin, the
// ancestors' with the leaf's; only where a plane of the leaf goes through the
// origin or past it (0 / 0, which the reference's min/max ignore) is the chain
// walked.  The leaf's test is FP32 with error bounds (slab_certain), FP64
// inside them.  Walking the chain for every hit (about 10 boxes in the urban
// canyon, 16 on the terrain) cost the level-9 canyon solve 0.35 ms, and the
// FP64 walk for the 0.3 % of its rays with a zero component, which held their
// whole warp through 600 FP64 instructions, another 2.3 ms (level-7 plan: 0.37
// of 0.60 ms).
__device__ __forceinline__ bool zero64(double x) {
  return (__double_as_longlong(x) << 1) == 0;
}
// slab64 out of line (see mt64_call).
__device__ __noinline__ bool slab_call(const double* bb, double ox, double oy, double oz, double dx,
                                       double dy, double dz) {
  const double o[3] = {ox, oy, oz}, d[3] = {dx, dy, dz};
  return slab64(bb, o, d);
}
__device__ __forceinline__ bool leaf_reachable(const DevScene& sc, int leaf, const double* o,
                                               const double* d, const float3& o32,
                                               const float3& d32, const float3& inv) {
  const RefNode& L = sc.ref[leaf];
  int zeros = 0;
  bool beside = false;  // a zero component, and the origin not strictly between the planes
#pragma unroll
  for (int a = 0; a < 3; ++a)
    if (zero64(d[a])) {
      // fb holds the planes exactly and rounding is monotone, so a rounded
      // origin strictly between them comes from one that is
      const float oa = a == 0 ? o32.x : (a == 1 ? o32.y : o32.z);
      zeros |= 1 << a;
      beside |= (L.flat & 8) || !(oa > L.fb[a] && oa < L.fb[3 + a]);
    }
  if (beside) {
    for (int n = leaf; n >= 0; n = sc.ref[n].parent)
      if (!slab_call(sc.ref[n].bb, o[0], o[1], o[2], d[0], d[1], d[2])) return false;
    return true;
  }
  const int v = slab_certain(L.fb, L.flat, o32, d32, inv, zeros);
  return v < 0 ? slab_call(L.bb, o[0], o[1], o[2], d[0], d[1], d[2]) : v != 0;
}

// exact_closest for k_trace, out of line: the ray and the hit go by value (see
// mt64_call).
__device__ __noinline__ Hit exact_call(const DevScene& sc, double ox, double oy, double oz,
                                       double dx, double dy, double dz, unsigned* overflow) {
  const double o[3] = {ox, oy, oz}, d[3] = {dx, dy, dz};
  Hit best;
  if (!exact_closest(sc, o, d, best, overflow)) best.rank = INT_MAX;
  return best;
}

// Closest hit with the reference's result.  FP32 ordered traversal over the
// reference BVH (boxes widened by box_margin so no box the FP64 test accepts
// is missed), FP32 triangle filter, FP64 test for every triangle the filter
// cannot rule out, lexicographic (distance, depth-first rank) minimum - the
// reference's strict '<' in visit order.  The winner is accepted only if the
// reference's slab tests reach its leaf; otherwise the ray is re-run with the
// reference-order traversal.
__device__ __noinline__ bool closest_hit(const DevScene& sc, const double* o, const double* d,
                                         Hit& best, TraceStats& st, unsigned* overflow) {
  const float3 o32 = make_float3(float(o[0]), float(o[1]), float(o[2]));
  const float3 d32 = make_float3(float(d[0]), float(d[1]), float(d[2]));
  const float3 inv = make_float3(1.0f / d32.x, 1.0f / d32.y, 1.0f / d32.z);
  const float no = sqrtf(o32.x * o32.x + o32.y * o32.y + o32.z * o32.z);
  const float nd = sqrtf(d32.x * d32.x + d32.y * d32.y + d32.z * d32.z);
  const float m = sc.box_margin + kBoxK * no;
  best.rank = INT_MAX;
  best.dist = __longlong_as_double(0x7ff0000000000000ll);
  best.t = best.dist;
  float tcut = INFINITY;  // boxes entered beyond this cannot hold a better hit

  int stack[kStack];
  int sp = 0;
  int pending_leaf = -1;
  constexpr int kCand = 8;
  int cand_r[kCand], cand_leaf[kCand];
  float cand_t[kCand];
  int ncand = 0;
  if (sc.root_leaf) pending_leaf = 0;
  else stack[sp++] = 0;
  bool stack_overflow = false;

  while (true) {
    if (pending_leaf >= 0) {
      const RefNode& L = sc.ref[pending_leaf];
      for (int r = L.first; r < L.first + L.count; ++r) {
        float tlo, thi;
        const int k = tri_classify(sc.tri32[r], o32, d32, no, nd, tlo, thi);
        if (k == 0 || tlo > tcut) continue;
        if (ncand < kCand) {
          cand_r[ncand] = r;
          cand_leaf[ncand] = pending_leaf;
          cand_t[ncand] = tlo;
          ++ncand;
          if (k & kSureHit) tcut = fminf(tcut, thi * (1.0f + kTieSlack) + 1e-30f);
        } else {
          // too many contenders: resolve this one now
          ++st.fp64_tri;
          double t, P[3], dist;
          if (mt64(sc.tri64[r], o, d, t, P, dist) &&
              (dist < best.dist || (dist == best.dist && r < best.rank))) {
            best.dist = dist;
            best.t = t;
            best.p[0] = P[0];
            best.p[1] = P[1];
            best.p[2] = P[2];
            best.rank = r;
            best.leaf = pending_leaf;
            tcut = fminf(tcut, float(t) * (1.0f + kTieSlack) + 1e-30f);
          }
        }
      }
      pending_leaf = -1;
    }
    if (sp == 0) break;
    const int ni = stack[--sp];
    if (ni < 0) {  // a leaf deferred as the farther child
      pending_leaf = ~ni;
      continue;
    }
    float4 f0, f1, f2;
    int2 ch;
    load_node(sc.node32, ni, f0, f1, f2, ch);
    float tn0, tf0, tn1, tf1;
    slab32(f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, o32, inv, m, tn0, tf0);
    slab32(f1.z, f1.w, f2.x, f2.y, f2.z, f2.w, o32, inv, m, tn1, tf1);
    const bool h0 = tn0 <= tf0 && tf0 >= 0.0f && tn0 <= tcut;
    const bool h1 = tn1 <= tf1 && tf1 >= 0.0f && tn1 <= tcut;
    int first = 0, second = 0;
    bool has_first = false, has_second = false;
    if (h0 && h1) {
      has_first = has_second = true;
      if (tn1 < tn0) {
        first = ch.y;
        second = ch.x;
      } else {
        first = ch.x;
        second = ch.y;
      }
    } else if (h0) {
      has_first = true;
      first = ch.x;
    } else if (h1) {
      has_first = true;
      first = ch.y;
    }
    if (has_second) {
      if (sp >= kStack) {
        stack_overflow = true;
        break;
      }
      stack[sp++] = second;  // internal node or ~leaf
    }
    if (has_first) {
      if (first < 0) {
        pending_leaf = ~first;
      } else {
        if (sp >= kStack) {
          stack_overflow = true;
          break;
        }
        stack[sp++] = first;
      }
    }
  }

  // Resolve the contenders exactly, nearest lower bound first, until none
  // can reach the best exact distance.
  for (int i = 1; i < ncand; ++i) {  // insertion sort by tlo (ncand <= kCand)
    const float kt = cand_t[i];
    const int kr = cand_r[i], kl = cand_leaf[i];
    int j = i - 1;
    while (j >= 0 && cand_t[j] > kt) {
      cand_t[j + 1] = cand_t[j];
      cand_r[j + 1] = cand_r[j];
      cand_leaf[j + 1] = cand_leaf[j];
      --j;
    }
    cand_t[j + 1] = kt;
    cand_r[j + 1] = kr;
    cand_leaf[j + 1] = kl;
  }
  for (int i = 0; i < ncand; ++i) {
    if (best.rank != INT_MAX && cand_t[i] > float(best.t) * (1.0f + kTieSlack) + 1e-30f) break;
    const int r = cand_r[i];
    ++st.fp64_tri;
    double t, P[3], dist;
    if (mt64(sc.tri64[r], o, d, t, P, dist) &&
        (dist < best.dist || (dist == best.dist && r < best.rank))) {
      best.dist = dist;
      best.t = t;
      best.p[0] = P[0];
      best.p[1] = P[1];
      best.p[2] = P[2];
      best.rank = r;
      best.leaf = cand_leaf[i];
    }
  }
  if (stack_overflow ||
      (best.rank != INT_MAX && !leaf_reachable(sc, best.leaf, o, d, o32, d32, inv))) {
    ++st.fallback;
    return exact_closest(sc, o, d, best, overflow);
  }
  return best.rank != INT_MAX;
}

// closest_hit for k_trace, likewise.
__device__ __noinline__ Hit closest_call(const DevScene& sc, double ox, double oy, double oz,
                                         double dx, double dy, double dz, Counters* ctr) {
  const double o[3] = {ox, oy, oz}, d[3] = {dx, dy, dz};
  Hit best;
  TraceStats st{0, 0};
  if (!closest_hit(sc, o, d, best, st, &ctr->overflow)) best.rank = INT_MAX;
  if (st.fp64_tri) atomicAdd(&ctr->fp64_tri, (unsigned long long)st.fp64_tri);
  if (st.fallback) atomicAdd(&ctr->fallback, (unsigned long long)st.fallback);
  return best;
}

// ---- split closest hit: FP32 candidate search, then FP64 resolution -------
//
// The same decision as closest_hit, cut in two so that the FP32 traversal
// (divergent: rays visit very different numbers of nodes) and the FP64
// resolution (dense FP64 work) run in separate kernels.  The search keeps up
// to kCand contender triangles per ray (depth-first rank, FP32 lower bound on
// t); more contenders, or a stack overflow, send the ray to the
// reference-order FP64 traversal.
constexpr int kCand = 8;
constexpr unsigned char kFindFallback = 0xFF;
// ncand of a ray: its contenders (0..kCand), with kCandUnsafe if its origin or
// direction is outside soft64's range; kFindFallback as a whole.
constexpr int kCandCount = 0x0F, kCandUnsafe = 0x40;
constexpr unsigned kContUV = 0x80000000u;  // contender's rank: u and v are sure (kSureUV)

// A ray prepared for the search BVH's slab tests: along axis a a plane at b is
// crossed at b * inv[a] + off, with off_near / off_far holding -(o +- m) / d,
// the box expansion m folded in.  One fused operation per plane, no near/far
// exchange: the near plane of a box is its low one where d > 0, else its high
// one, picked by address.  Rounding (off to 2 units, the product with inv's
// error common to both terms) moves a plane by under 5 * 2^-24 (|b| + |o| + m),
// far inside m = 2^-14 (extent + 1 + |o|).  A component below 1e-18 counts as
// 1e-18: products stay finite and a box is kept iff the origin is within m of
// its slab, as with an infinite reciprocal.
struct SlabRay {
  float inv[3], off_near[3], off_far[3];
  int near;  // bit a: the near plane along axis a is the high one
};
__device__ __forceinline__ SlabRay slab_ray(const float3& o, const float3& d, float m) {
  SlabRay r;
  r.near = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float oa = a == 0 ? o.x : (a == 1 ? o.y : o.z);
    const float da = a == 0 ? d.x : (a == 1 ? d.y : d.z);
    const float inv = 1.0f / (fabsf(da) < 1e-18f ? copysignf(1e-18f, da) : da);
    const float sm = copysignf(m, da);
    r.inv[a] = inv;
    r.off_near[a] = -(oa + sm) * inv;
    r.off_far[a] = -(oa - sm) * inv;
    r.near |= signbit(da) ? 1 << a : 0;
  }
  return r;
}

// Four planes of an axis take two packed FP32 operations, each product and sum
// rounded as fmaf rounds it: the search is bound by instruction issue (79 % of
// the issue slots; level-9 canyon 4.27 -> 4.13 ms, level-10 terrain 8.87 ->
// 8.63).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long r, x = *reinterpret_cast<unsigned long long*>(&a),
                        y = *reinterpret_cast<unsigned long long*>(&b),
                        z = *reinterpret_cast<unsigned long long*>(&c);
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
  return *reinterpret_cast<float2*>(&r);
}
// The children of a four-wide node that the ray's slab test keeps within
// [0, tcut], nearest first; returns how many (c[0..n), entered at t[0..n)).
__device__ __forceinline__ int visit_node4(const Node4* node, const SlabRay& r, float tcut,
                                           int c[4], float t[4]) {
  const float4* p = reinterpret_cast<const float4*>(node);
  const int sx = r.near & 1 ? 3 : 0, sy = r.near & 2 ? 3 : 0, sz = r.near & 4 ? 3 : 0;
  const float4 bnx = __ldg(p + sx), bny = __ldg(p + 1 + sy), bnz = __ldg(p + 2 + sz);
  const float4 bfx = __ldg(p + 3 - sx), bfy = __ldg(p + 4 - sy), bfz = __ldg(p + 5 - sz);
  const int4 cr = __ldg(reinterpret_cast<const int4*>(p + 6));
  auto visit = [&](float ax, float ay, float az, float bx, float by, float bz, int child,
                   float& t) -> int {
    const float tn = fmaxf(fmaxf(ax, ay), fmaxf(az, 0.0f));
    const float tf = fminf(fminf(bx, by), fminf(bz, tcut));
    const bool h = tn <= tf;  // an absent child's planes are at infinity the wrong way round
    t = h ? tn : INFINITY;
    return h ? child : kEmptyChild;
  };
  auto planes = [](const float4& b, float inv, float off) {
    const float2 i2 = make_float2(inv, inv), o2 = make_float2(off, off);
    const float2 l = fma2(make_float2(b.x, b.y), i2, o2), h = fma2(make_float2(b.z, b.w), i2, o2);
    return make_float4(l.x, l.y, h.x, h.y);
  };
  const float4 nx = planes(bnx, r.inv[0], r.off_near[0]), ny = planes(bny, r.inv[1], r.off_near[1]),
               nz = planes(bnz, r.inv[2], r.off_near[2]), fx = planes(bfx, r.inv[0], r.off_far[0]),
               fy = planes(bfy, r.inv[1], r.off_far[1]), fz = planes(bfz, r.inv[2], r.off_far[2]);
  c[0] = visit(nx.x, ny.x, nz.x, fx.x, fy.x, fz.x, cr.x, t[0]);
  c[1] = visit(nx.y, ny.y, nz.y, fx.y, fy.y, fz.y, cr.y, t[1]);
  c[2] = visit(nx.z, ny.z, nz.z, fx.z, fy.z, fz.z, cr.z, t[2]);
  c[3] = visit(nx.w, ny.w, nz.w, fx.w, fy.w, fz.w, cr.w, t[3]);
  auto order = [](float& ta, int& ca, float& tb, int& cb) {
    if (tb < ta) {
      const float t = ta;
      ta = tb;
      tb = t;
      const int x = ca;
      ca = cb;
      cb = x;
    }
  };
  order(t[0], c[0], t[1], c[1]);  // sorting network for four
  order(t[2], c[2], t[3], c[3]);
  order(t[0], c[0], t[2], c[2]);
  order(t[1], c[1], t[3], c[3]);
  order(t[1], c[1], t[2], c[2]);
  return int(c[0] != kEmptyChild) + int(c[1] != kEmptyChild) + int(c[2] != kEmptyChild) +
         int(c[3] != kEmptyChild);
}

// Whether the reference's test of the triangle a ray starts on certainly
// fails (so its FP64 test can be skipped).  The ray's origin is the hit
// point the parent ray's FP64 test produced on that triangle, within about
// 1e-15 |P| of its plane; leaving at |cos| >= 1e-2 the reference's t for it
// is then below 1e-10 for |P| < 1e5, far under the t > FLT_EPSILON it
// requires (Triangle.cpp:113).
// o32, d32: the ray's origin and direction rounded to FP32 (conversions from
// FP64 occupy the FP64 pipe like an FP64 add, so a ray's are made once).
__device__ __forceinline__ bool origin_rejected(const Tri32& T, const float3& o32,
                                                const float3& d32) {
  const float ox = o32.x, oy = o32.y, oz = o32.z;
  if (!(fabsf(ox) < 1e5f && fabsf(oy) < 1e5f && fabsf(oz) < 1e5f)) return false;
  const float nx = T.e1[1] * T.e2[2] - T.e1[2] * T.e2[1];
  const float ny = T.e1[2] * T.e2[0] - T.e1[0] * T.e2[2];
  const float nz = T.e1[0] * T.e2[1] - T.e1[1] * T.e2[0];
  const float dx = d32.x, dy = d32.y, dz = d32.z;
  const float dn = dx * nx + dy * ny + dz * nz;
  const float nn = sqrtf(nx * nx + ny * ny + nz * nz), dd = sqrtf(dx * dx + dy * dy + dz * dz);
  return fabsf(dn) >= 1e-2f * nn * dd;
}

// HitReceptionSphere (RTSolver.cpp:805-863), FP64 in the reference's order.
__device__ __forceinline__ bool reception64(const double* s, const double* t, const double* c,
                                            double path_len, double tan_beta) {
  using namespace x64;
  double rd[3], w[3];
  sub3(t, s, rd);
  sub3(c, s, w);
  double t0 = div(dot(rd, w), sqn(rd));
  if (t0 < 0) return false;
  if (t0 >= 1) t0 = 1;
  double P[3] = {add(s[0], mul(t0, rd[0])), add(s[1], mul(t0, rd[1])), add(s[2], mul(t0, rd[2]))};
  const double unfolded = add(path_len, norm(P));
  const double radius = mul(unfolded, tan_beta);
  double e[3];
  sub3(c, P, e);
  return norm(e) <= radius;
}

// FP32 reception filter: 1 = captured, 0 = not captured, -1 = within the
// error margin (decide with reception64).
__device__ __forceinline__ int reception32(const float3& s, const float3& u, float len, float S,
                                           const float3& c, float tanb) {
  const float wx = c.x - s.x, wy = c.y - s.y, wz = c.z - s.z;
  const float lam = u.x * wx + u.y * wy + u.z * wz;
  const float ns = sqrtf(s.x * s.x + s.y * s.y + s.z * s.z);
  const float nc = sqrtf(c.x * c.x + c.y * c.y + c.z * c.z);
  const float mag = ns + nc + 1.0f;
  const float ml = kRecK * mag;
  if (lam < -ml) return 0;
  if (lam <= ml) return -1;
  const float lc = fminf(lam, len);
  const float px = s.x + lc * u.x, py = s.y + lc * u.y, pz = s.z + lc * u.z;
  const float np = sqrtf(px * px + py * py + pz * pz);
  const float ex = c.x - px, ey = c.y - py, ez = c.z - pz;
  const float dist = sqrtf(ex * ex + ey * ey + ez * ez);
  const float rad = (S + np) * tanb;
  const float mr = kRecK * (mag + S + np);
  if (dist > rad + mr) return 0;
  if (dist < rad - mr) return 1;
  return -1;
}

}  // namespace sbr
