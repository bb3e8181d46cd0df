// Path stage: duplicate removal by coplanar key (RTSolver.cpp:435-459), the
// corrected geometry and field of each survivor (FieldCompute.cpp:71-151)
// and the per-receiver sum in (launch, BFS) order (FieldCompute.cpp:11-25).
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "sbr_device.h"
#include "sbr_field.cuh"
#include "sbr_kernels.cuh"
#include "sbr_common.cuh"
#include "sbr_trace.cuh"
#include "sbr_capture.cuh"

namespace sbr {

// ---- correction / dedup -----------------------------------------------------

struct PathBuf {
  int n;            // rays
  int tri[kMaxDepth + 1];
  int kind[kMaxDepth + 1];
  double pts[kMaxDepth + 2][3];
};

// Path of a class: tri of each ray (ray i ends on tri[i]; the last ray ends at
// the receiver) and kind of each ray's start.
__device__ __forceinline__ bool class_path(const ClassInfo* info, uint32_t cls, PathBuf& pb) {
  int depth = 0;
  int tri_rev[kMaxDepth], kind_rev[kMaxDepth];
  for (uint32_t c = cls; !is_root_class(c); c = info[c].parent) {
    if (depth >= kMaxDepth) return false;
    tri_rev[depth] = info[c].tri;
    kind_rev[depth] = info[c].kind;
    ++depth;
  }
  pb.n = depth + 1;
  pb.kind[0] = 0;
  for (int i = 0; i < depth; ++i) {
    pb.tri[i] = tri_rev[depth - 1 - i];   // rank of the triangle hit by ray i
    pb.kind[i + 1] = kind_rev[depth - 1 - i];
  }
  pb.tri[depth] = -1;
  return true;
}

// GetImageSources + MultiPathCorrection / DirectPathCorrection
// (RTSolver.cpp:330-433) for a path whose correction succeeded when it was
// captured (correct_event; k_direct for the direct path): fills pb.pts with
// the corrected points.
__device__ bool correct_path(const DevScene& sc, const int* rank_to_id, const TxParams& P,
                             const double* rxp, PathBuf& pb) {
  using namespace x64;
  const double* tx = P.tx;
  if (pb.n == 1) {  // the exact segment Tx -> Rx (RTSolver.cpp:385-387)
    for (int a = 0; a < 3; ++a) {
      pb.pts[0][a] = tx[a];
      pb.pts[1][a] = rxp[a];
    }
    return true;
  }
  const int n = pb.n;
  double img[kMaxDepth + 1][3];
  for (int a = 0; a < 3; ++a) img[0][a] = tx[a];
  for (int i = 0; i + 1 < n; ++i) {
    const CorrTri& T = sc.corr[rank_to_id[pb.tri[i]]];
    if (pb.kind[i + 1] == 1) {  // ImagePoint (RTSolver.cpp:910-924)
      double w[3];
      sub3(img[i], T.v1, w);
      const double dist = dot(T.n, w);
      for (int a = 0; a < 3; ++a) img[i + 1][a] = sub(img[i][a], mul(mul(2.0, dist), T.n[a]));
    } else {
      for (int a = 0; a < 3; ++a) img[i + 1][a] = img[i][a];
    }
  }
  double target[3] = {rxp[0], rxp[1], rxp[2]};
  for (int a = 0; a < 3; ++a) pb.pts[n][a] = rxp[a];
  for (int i = n - 1; i >= 1; --i) {
    const CorrTri& T = sc.corr[rank_to_id[pb.tri[i - 1]]];
    double d[3], P3[3];
    sub3(target, img[i], d);
    if (!mt64c(T, img[i], d, P3)) return false;
    for (int a = 0; a < 3; ++a) {
      pb.pts[i][a] = P3[a];
      target[a] = P3[a];
    }
  }
  for (int a = 0; a < 3; ++a) pb.pts[0][a] = tx[a];
  return true;
}

// Whether the reference's closest hit along d from o (BVH.h:276-328) lies no
// farther than o + d.  Its minimum is no farther exactly if some triangle that
// it reaches and hits is, so the search stops at the first one: FP32 search of
// the search BVH within t <= 1, where a sure hit clearly nearer than t = 1
// blocks if its leaf is reachable, and FP64 decides the rest.
__device__ bool direct_blocked(const DevScene& sc, const double* o, const double* d,
                               Counters* ctr) {
  const float3 o32 = make_float3(float(o[0]), float(o[1]), float(o[2]));
  const float3 d32 = make_float3(float(d[0]), float(d[1]), float(d[2]));
  const float no = sqrtf(o32.x * o32.x + o32.y * o32.y + o32.z * o32.z);
  const float nd = sqrtf(d32.x * d32.x + d32.y * d32.y + d32.z * d32.z);
  const float3 inv = make_float3(1.0f / d32.x, 1.0f / d32.y, 1.0f / d32.z);
  const SlabRay slab = slab_ray(o32, d32, sc.box_margin + kBoxK * no);
  const float tcut = 1.0f + 4.0f * kTieSlack;
  int stack[kStack];
  int sp = 0;
  stack[sp++] = 0;  // the search root is always a node
  while (sp > 0) {
    const int ni = stack[--sp];
    if (ni >= 0) {
      int c[4];
      float t[4];
      const int n = visit_node4(sc.snode4 + ni, slab, tcut, c, t);
      if (sp + n > kStack) {  // a deep stack: the one-pass search
        const Hit h = closest_call(sc, o[0], o[1], o[2], d[0], d[1], d[2], ctr);
        return h.rank != INT_MAX && !(x64::norm(d) < h.dist);
      }
      for (int k = n - 1; k >= 0; --k) stack[sp++] = c[k];
      continue;
    }
    const int first = ~ni >> 3, count = ~ni & 7;
    for (int j = first; j < first + count; ++j) {
      float tlo, thi;
      const int k = tri_classify(sc.stri[j], o32, d32, no, nd, tlo, thi);
      if (!k || tlo > tcut) continue;
      const int rk = __ldg(sc.srank + j);
      const Tri64& T = sc.tri64[rk];
      if (!((k & kSureHit) && thi < 1.0f - 4.0f * kTieSlack)) {
        const Mt64Result m = mt64_call(&T, o[0], o[1], o[2], d[0], d[1], d[2]);
        if (!m.ok || !(m.dist < __longlong_as_double(0x7ff0000000000000ll)) ||
            x64::norm(d) < m.dist)
          continue;
      }
      if (leaf_reachable(sc, T.node, o, d, o32, d32, inv)) return true;
    }
  }
  return false;
}

// DirectPathCorrection (RTSolver.cpp:375-394) once per receiver: the direct
// path survives iff the reference's BVH query from the transmitter along
// (rx - tx) finds nothing closer than the receiver.  A chain of dependent
// loads per receiver, so one warp per block spreads few receivers over the
// chip.  With the closest-hit search of the reference BVH (whose SAH build
// leaves a leaf of 401 triangles in the canyon) it took 0.8 ms for 400 as for
// 10,000 receivers, and a level-7 solve waited 0.5 ms for it.
__global__ void __launch_bounds__(32) k_direct(const __grid_constant__ DevScene sc, const TxParams* txp,
                                               const double* rx, const int* rx_req, int n_rx,
                                               unsigned char* ok, Counters* ctr) {
  for (int gi = blockIdx.x * blockDim.x + threadIdx.x; gi < n_rx; gi += gridDim.x * blockDim.x) {
    const double* tx = txp[rx_req[gi]].tx;
    const double* c = rx + 3 * size_t(gi);
    const double o[3] = {tx[0], tx[1], tx[2]};
    double d[3];
    x64::sub3(c, o, d);
    ok[gi] = direct_blocked(sc, o, d, ctr) ? 0 : 1;
  }
}

// RemoveDuplicatePath (RTSolver.cpp:435-459): the first corrected path in
// (launch, BFS) order wins each (receiver, coplanar key).
__device__ __forceinline__ unsigned long long dedup_key(const ClassInfo* info, const Corrected& e) {
  const uint32_t cop = is_root_class(e.cls) ? kRootClass : info[e.cls].cop;
  return (unsigned long long)e.rx << 32 | cop;
}

__global__ void k_dedup(const Corrected* list, unsigned long long cap, const ClassInfo* info,
                        HashTable dedup, unsigned long long* dedup_rank, Counters* ctr) {
  const unsigned long long n = min(ctr->corrected, cap);
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const Corrected e = list[i];
    const uint32_t ds = ht_insert(dedup, dedup_key(info, e), &ctr->overflow, kOvDedup, &ctr->used_dd,
                                &ctr->lost_dd);
    if (ds != 0xFFFFFFFFu) atomicMin(&dedup_rank[ds], e.rank);
  }
}

struct Survivor {
  uint32_t cls, rx;
  unsigned long long rank;
};

__global__ void k_select(const Corrected* list, unsigned long long cap, const ClassInfo* info,
                         HashTable dedup, const unsigned long long* dedup_rank, Survivor* surv,
                         unsigned long long surv_cap, Counters* ctr) {
  const unsigned long long n = min(ctr->corrected, cap);
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const Corrected e = list[i];
    const uint32_t ds = ht_find(dedup, dedup_key(info, e));
    if (ds == 0xFFFFFFFFu || dedup_rank[ds] != e.rank) continue;
    const unsigned long long k = atomicAdd(&ctr->survivors, 1ull);
    if (k < surv_cap) surv[k] = Survivor{e.cls, e.rx, e.rank};
    else atomicOr(&ctr->overflow, kOvSurv);
  }
}

// ---- field ---------------------------------------------------------------

struct FieldArgs {
  DevScene sc;
  const TxParams* txp;
  const double* rx;
  const int* rx_req;
  const ClassInfo* cls_info;
  const int* rank_to_id;
  const Survivor* surv;
  Counters* ctr;
  unsigned long long cap;
  FieldConsts K;
  int precision;        // -1: each request's own; 0: FP64 for all (the FP64 shadow)
  double* path_field;   // 6 per survivor
  int* path_nray;
  int* path_tri;        // (kMaxDepth + 1) per survivor: triangle id
  int* path_cop;
  int* path_kind;
  int* path_near_edge;  // 1 if an interaction point is within 1e-6 of its triangle's edge
  double* path_pts;     // (kMaxDepth + 2) * 3 per survivor
  SegTerms* seg;        // (kMaxDepth + 1) per survivor
  int* path_mat;        // (kMaxDepth + 1) per survivor: material of each ray's start
  // k_seg's tasks, path << 5 | segment: every segment's direction, every
  // interaction (Counters::seg_tasks, int_tasks of them)
  uint32_t* seg_list;
  uint32_t* int_list;
  // FP32 field mode: bound on each component's absolute error per survivor
  // (0: computed in FP64; -1: no bound, the FP32-phase study mode)
  double* path_bound;
  const int* rx_flag;   // receivers whose paths k_escalate recomputes in FP64
  unsigned long long* fstat;  // [0] paths whose field FP32 mode took in FP64, [1] receivers
};

// FP32 field mode: a path whose condition number (path_combine's kappa)
// exceeds this is computed in FP64.
constexpr float kKappaMax32 = 32.0f;
// path_bound of a path whose FP64 field is still to come (k_escalate).
constexpr double kBoundRedo = -2.0;

// Barycentric distance of a point (on the triangle's plane) from the
// triangle's edges is below tol: min(u, v, 1-u-v) < tol.
__device__ __forceinline__ int near_edge(const CorrTri& T, const double* p, double tol) {
  double w[3] = {p[0] - T.v1[0], p[1] - T.v1[1], p[2] - T.v1[2]};
  const double d00 = T.e1[0] * T.e1[0] + T.e1[1] * T.e1[1] + T.e1[2] * T.e1[2];
  const double d01 = T.e1[0] * T.e2[0] + T.e1[1] * T.e2[1] + T.e1[2] * T.e2[2];
  const double d11 = T.e2[0] * T.e2[0] + T.e2[1] * T.e2[1] + T.e2[2] * T.e2[2];
  const double d20 = w[0] * T.e1[0] + w[1] * T.e1[1] + w[2] * T.e1[2];
  const double d21 = w[0] * T.e2[0] + w[1] * T.e2[1] + w[2] * T.e2[2];
  const double den = d00 * d11 - d01 * d01;
  if (!(den > 0)) return 1;
  const double u = (d11 * d20 - d01 * d21) / den, v = (d00 * d21 - d01 * d20) / den;
  return fmin(fmin(u, v), 1.0 - u - v) < tol ? 1 : 0;
}

// Field stage, one kernel per part: k_path corrects each survivor's path
// (FP64 image correction, sequential along the path) and writes its points,
// triangles and kinds; k_seg computes every segment's terms (one thread per
// segment); k_combine carries each path's field along it.
__global__ void k_path(FieldArgs A) {
  const unsigned long long ns = min(A.ctr->survivors, A.cap);
  const unsigned lane = threadIdx.x & 31u;
  for (unsigned long long i0 = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) & ~31ull;
       i0 < ns; i0 += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long i = i0 + lane;
    int n = 0;
    if (i < ns) {
      const Survivor sv = A.surv[i];
      const TxParams& P = A.txp[A.rx_req[sv.rx]];
      PathBuf pb;
      class_path(A.cls_info, sv.cls, pb);
      correct_path(A.sc, A.rank_to_id, P, A.rx + 3 * size_t(sv.rx), pb);
      A.path_nray[i] = n = pb.n;
      const size_t b = size_t(i) * (kMaxDepth + 1);
      for (int r = 0; r < pb.n; ++r) {
        const int t = pb.tri[r];
        A.path_tri[b + r] = t >= 0 ? A.rank_to_id[t] : -1;
        A.path_cop[b + r] = t >= 0 ? A.sc.tri64[t].cop : -1;
        A.path_kind[b + r] = pb.kind[r];
        // the hit triangle's own material (the ray's hit record carries it)
        A.path_mat[b + r] = r > 0 ? A.sc.tri64[pb.tri[r - 1]].mat : 0;
      }
      const size_t bp = size_t(i) * (kMaxDepth + 2) * 3;
      for (int r = 0; r <= pb.n; ++r)
        for (int a = 0; a < 3; ++a) A.path_pts[bp + 3 * r + a] = pb.pts[r][a];
      // interaction point r+1 lies on the triangle the correction intersected
      int near = 0;
      for (int r = 0; r + 1 < pb.n; ++r)
        near |= near_edge(A.sc.corr[A.rank_to_id[pb.tri[r]]], pb.pts[r + 1], 1e-6);
      A.path_near_edge[i] = near;
    }
    __syncwarp();
    // the path's segments and its interactions (all segments but the first)
    int incl = n, m = n > 0 ? 1 : 0;  // segments; paths
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o), w = __shfl_up_sync(0xffffffffu, m, o);
      if (int(lane) >= o) {
        incl += v;
        m += w;
      }
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31), paths = __shfl_sync(0xffffffffu, m, 31);
    unsigned long long bs = 0, bi = 0;
    if (lane == 0) {
      bs = atomicAdd(&A.ctr->seg_tasks, (unsigned long long)total);
      bi = atomicAdd(&A.ctr->int_tasks, (unsigned long long)(total - paths));
    }
    bs = __shfl_sync(0xffffffffu, bs, 0) + (incl - n);
    bi = __shfl_sync(0xffffffffu, bi, 0) + (incl - n) - (m - (n > 0 ? 1 : 0));
    for (int r = 0; r < n; ++r) {
      A.seg_list[bs + r] = uint32_t(i) << 5 | uint32_t(r);
      if (r > 0) A.int_list[bi + r - 1] = uint32_t(i) << 5 | uint32_t(r);
    }
  }
}

// The path inputs of path i for the field functions: points, frames of the
// triangles each ray ends on, kinds and materials of each ray's start.
struct PathView {
  int n;
  const double (*pts)[3];
  const double* frames[kMaxDepth + 1];
  int kind[kMaxDepth + 1];
  int mat[kMaxDepth + 1];
};

// (of its rays [from, to) where the caller reads no other).
__device__ __forceinline__ void path_view(const FieldArgs& A, unsigned long long i, PathView& v,
                                          int from = 0, int to = kMaxDepth + 1) {
  v.n = A.path_nray[i];
  v.pts = reinterpret_cast<const double(*)[3]>(A.path_pts + size_t(i) * (kMaxDepth + 2) * 3);
  const size_t b = size_t(i) * (kMaxDepth + 1);
  for (int r = from; r < min(v.n, to); ++r) {
    // frames by the id's position in the caller's mesh vector, as the
    // reference looks them up (FieldCompute.cpp:107)
    const int id = A.path_tri[b + r];
    v.frames[r] = id >= 0 ? A.sc.corr[id].cs : nullptr;
    v.kind[r] = A.path_kind[b + r];
    v.mat[r] = A.path_mat[b + r];
  }
}

// One thread per direction task, then one per interaction task.  Chains of
// FP64 instructions (angles, complex functions), so the two parts of a segment
// run side by side, and the tasks are dense: by (path, segment slot) a batch of
// 9,567 paths kept 5 of 32 lanes busy.
__global__ void k_seg(FieldArgs A) {
  const unsigned long long ns_t = A.ctr->seg_tasks, ni_t = A.ctr->int_tasks;
  const unsigned long long first_i = (ns_t + 31) & ~31ull;  // no warp holds both kinds
  for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       k < first_i + ni_t; k += (unsigned long long)gridDim.x * blockDim.x) {
    if (k >= ns_t && k < first_i) continue;
    const bool inter = k >= first_i;
    const uint32_t task = inter ? A.int_list[k - first_i] : A.seg_list[k];
    const unsigned long long i = task >> 5;
    const int r = int(task & 31u);
    const Survivor sv = A.surv[i];
    const TxParams& P = A.txp[A.rx_req[sv.rx]];
    PathView v;
    path_view(A, i, v, max(r - 1, 0), r + 1);
    const PatternTab pat{P.pat, P.pat_nt, P.pat_np, P.pat_dt, P.pat_dp};
    const int prec = A.precision < 0 ? P.precision : A.precision;
    SegTerms& t = A.seg[i * (kMaxDepth + 1) + r];
    const int part = inter ? kSegInteraction : kSegDirection;
    if (!inter && r == 0) {  // no interaction at the start
      t.fp64_fresnel = 0;
      t.ctm[0] = t.cte[0] = 1.0;
      t.ctm[1] = t.cte[1] = 0.0;
    }
    if (prec != 0)
      seg_terms<float>(r, v.pts, v.frames, v.kind, v.mat, A.sc.mats, P.txcs, P.freq, P.pt,
                       P.antenna, P.fresnel != 0, A.K, t, &pat, part);
    else
      seg_terms<double>(r, v.pts, v.frames, v.kind, v.mat, A.sc.mats, P.txcs, P.freq, P.pt,
                        P.antenna, P.fresnel != 0, A.K, t, &pat, part);
  }
}

__global__ void k_combine(FieldArgs A) {
  const unsigned long long ns = min(A.ctr->survivors, A.cap);
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < ns;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const Survivor sv = A.surv[i];
    const TxParams& P = A.txp[A.rx_req[sv.rx]];
    PathView v;
    path_view(A, i, v);
    const SegTerms* seg = A.seg + size_t(i) * (kMaxDepth + 1);
    Cx<double> e[3];
    const int prec = A.precision < 0 ? P.precision : A.precision;
    double bound = 0.0;
    if (prec == 2) {
      path_combine<float, true>(v.n, seg, v.pts, v.frames, v.kind, P.txcs, P.freq, A.K, e);
      bound = -1.0;
    } else if (prec == 1) {
      float kappa = 0.0f;
      path_combine<float>(v.n, seg, v.pts, v.frames, v.kind, P.txcs, P.freq, A.K, e, &kappa);
      bool pole = false;
      for (int r = 0; r < v.n; ++r) pole |= seg[r].fp64_fresnel != 0;
      if (pole || !(kappa <= kKappaMax32)) {
        bound = kBoundRedo;  // an ill-conditioned path: k_escalate takes it in FP64
      } else {
        // each component errs by at most (7 kappa) ulps of |E| (measured on
        // every path of the urban canyon); the bound takes 16 kappa, plus
        // the FP32 rounding of the path field when the sum reads it
        const double mag = sqrt(e[0].re * e[0].re + e[0].im * e[0].im + e[1].re * e[1].re +
                                e[1].im * e[1].im + e[2].re * e[2].re + e[2].im * e[2].im);
        bound = (16.0 * double(kappa) + 1.0) * 0x1p-24 * mag;
      }
    } else {
      path_combine<double>(v.n, seg, v.pts, v.frames, v.kind, P.txcs, P.freq, A.K, e);
    }
    if (A.path_bound) A.path_bound[i] = bound;
    for (int j = 0; j < 3; ++j) {
      A.path_field[6 * i + 2 * j] = e[j].re;
      A.path_field[6 * i + 2 * j + 1] = e[j].im;
    }
  }
}

// FP32 field mode: terms and field again in FP64, first (receivers = false) for
// the ill-conditioned paths k_combine marked, then for every path of the
// receivers k_rx_sum could not certify (it then sums those in FP64).  One warp
// per path, a lane per segment: one thread going through a path's segments
// took 280 and 140 us in the canyon with slab walls (its whole field stage
// 0.54 ms, now 0.30).
__global__ void k_escalate(FieldArgs A, bool receivers) {
  const unsigned long long ns = min(A.ctr->survivors, A.cap);
  const int lane = threadIdx.x & 31;
  for (unsigned long long i = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5;
       i < ns; i += ((unsigned long long)gridDim.x * blockDim.x) >> 5) {
    const Survivor sv = A.surv[i];
    const double state = A.path_bound[i];
    // (bound 0: taken in FP64 already)
    if (receivers ? !A.rx_flag[sv.rx] || state == 0.0 : state != kBoundRedo) continue;
    const TxParams& P = A.txp[A.rx_req[sv.rx]];
    PathView v;
    path_view(A, i, v);
    SegTerms* seg = A.seg + size_t(i) * (kMaxDepth + 1);
    const PatternTab pat{P.pat, P.pat_nt, P.pat_np, P.pat_dt, P.pat_dp};
    if (lane < v.n)
      seg_terms<double>(lane, v.pts, v.frames, v.kind, v.mat, A.sc.mats, P.txcs, P.freq, P.pt,
                        P.antenna, P.fresnel != 0, A.K, seg[lane], &pat);
    __syncwarp();
    if (lane == 0) {
      Cx<double> e[3];
      path_combine<double>(v.n, seg, v.pts, v.frames, v.kind, P.txcs, P.freq, A.K, e);
      for (int j = 0; j < 3; ++j) {
        A.path_field[6 * i + 2 * j] = e[j].re;
        A.path_field[6 * i + 2 * j + 1] = e[j].im;
      }
      A.path_bound[i] = 0.0;
      atomicAdd(&A.fstat[0], 1ull);
    }
    __syncwarp();
  }
}

// ---- per-receiver ordered sum -------------------------------------------

// Paths and their rays per receiver (counts, rays).
__global__ void k_surv_hist(const Survivor* surv, const Counters* ctr, unsigned long long cap,
                            const int* path_nray, int* counts, int* rays) {
  const unsigned long long ns = min(ctr->survivors, cap);
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < ns;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    atomicAdd(&counts[surv[i].rx], 1);
    atomicAdd(&rays[surv[i].rx], path_nray[i]);
  }
}

__global__ void k_surv_scatter(const Survivor* surv, const Counters* ctr, unsigned long long cap,
                               const int* starts, int* cursor, int* order) {
  const unsigned long long ns = min(ctr->survivors, cap);
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < ns;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const uint32_t r = surv[i].rx;
    order[starts[r] + atomicAdd(&cursor[r], 1)] = int(i);
  }
}

// Sort each receiver's survivors by (launch, BFS) rank and sum their fields in
// that order: FP64, or compensated FP32 (Neumaier) for the FP32 precisions.
// precision -1 takes each receiver's request precision, 0 forces FP64.
//
// FP32 field mode (precision 1, with path_bound): the receiver's error bound
// is the sum of its paths' bounds plus the compensated sum's own rounding
// (2 ulps of the result).  The receiver is certified when that bound is
// within half the field tolerance (1e-4 relative magnitude) of each
// component, or, for a component below 1e-9 of the receiver's largest, of
// that largest one; bound[r] then states it.  Otherwise rx_flag[r] is set:
// k_escalate recomputes its paths in FP64 and a second call (only = rx_flag,
// force_precision 0) sums it in FP64, with bound 0.
__global__ void k_rx_sum(const Survivor* surv, const int* starts, int* order, int n_rx,
                         const double* path_field, int force_precision, const int* rx_req,
                         const TxParams* txp, double* field, const double* path_bound = nullptr,
                         double* bound = nullptr, int* rx_flag = nullptr,
                         unsigned long long* fstat = nullptr, const int* only = nullptr,
                         const int* path_nray = nullptr, const int* ray_starts = nullptr,
                         unsigned* ray_offset = nullptr) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rx; r += gridDim.x * blockDim.x) {
    if (only && !only[r]) continue;
    const int precision = force_precision < 0 ? txp[rx_req[r]].precision : force_precision;
    const int b = starts[r], e = starts[r + 1];
    for (int i = b + 1; i < e; ++i) {
      const int v = order[i];
      const unsigned long long key = surv[v].rank;
      int j = i - 1;
      while (j >= b && surv[order[j]].rank > key) {
        order[j + 1] = order[j];
        --j;
      }
      order[j + 1] = v;
    }
    // where the result's ray arrays hold each path's rays (the rays are scanned
    // behind the paths, from the paths' total)
    if (ray_offset) {
      unsigned o = unsigned(ray_starts[r]) - unsigned(ray_starts[0]);
      for (int i = b; i < e; ++i) {
        ray_offset[i] = o;
        o += unsigned(path_nray[order[i]]);
      }
    }
    if (precision != 0) {  // both FP32 modes: compensated FP32 sum
      float s[6] = {0, 0, 0, 0, 0, 0}, c[6] = {0, 0, 0, 0, 0, 0};
      double B = 0.0;
      for (int i = b; i < e; ++i) {
        for (int k = 0; k < 6; ++k) {
          const float x = float(path_field[6 * size_t(order[i]) + k]);
          const float t = s[k] + x;
          c[k] += fabsf(s[k]) >= fabsf(x) ? (s[k] - t) + x : (x - t) + s[k];
          s[k] = t;
        }
        if (path_bound) {
          const double pb = path_bound[order[i]];
          B = (pb < 0.0 || B < 0.0) ? -1.0 : B + pb;
        }
      }
      double f[6];
      for (int k = 0; k < 6; ++k) f[k] = field[6 * size_t(r) + k] = double(s[k]) + double(c[k]);
      if (path_bound && bound) {
        if (precision != 1 || B < 0.0) {
          bound[r] = -1.0;  // FP32-phase study mode: no bound
        } else {
          double mag[3], big = 0.0;
          for (int j = 0; j < 3; ++j) {
            mag[j] = sqrt(f[2 * j] * f[2 * j] + f[2 * j + 1] * f[2 * j + 1]);
            big = fmax(big, mag[j]);
          }
          B = B * (1.0 + 1e-6) + 0x1p-23 * big;
          bool ok = true;
          for (int j = 0; j < 3; ++j)
            ok &= B <= 0.5e-4 * (mag[j] > 1e-9 * big ? mag[j] : big);
          bound[r] = B;
          if (!ok) {
            rx_flag[r] = 1;
            atomicAdd(&fstat[1], 1ull);
          }
        }
      }
    } else {
      double s[6] = {0, 0, 0, 0, 0, 0};
      for (int i = b; i < e; ++i)
        for (int k = 0; k < 6; ++k) s[k] = __dadd_rn(s[k], path_field[6 * size_t(order[i]) + k]);
      for (int k = 0; k < 6; ++k) field[6 * size_t(r) + k] = s[k];
      if (bound) bound[r] = 0.0;
    }
  }
}

// ---- the result, as the host keeps it -------------------------------------

// What a solve returns, written by the device straight into pinned host memory
// (ResultArgs::out): head, segments per request, fields, then the paths in
// receiver order with their rays packed.  The last part's size is known on the
// device only; if it does not fit, the host makes room and launches again.
struct ResultHead {
  Counters c;
  unsigned long long fstat[2];
  long long rays;
  int rx_bad, fits;
};
struct ResultLayout {  // byte offsets
  size_t seg, field, bound, field64, paths;
  __host__ __device__ size_t points(size_t ns) const { return paths + ns * sizeof(sbr_path); }
  __host__ __device__ size_t tri(size_t ns, size_t rays) const {
    return points(ns) + rays * 6 * sizeof(double);
  }
  __host__ __device__ size_t end(size_t ns, size_t rays) const {
    return tri(ns, rays) + 3 * rays * sizeof(int);
  }
};
struct ResultArgs {
  FieldArgs f;  // survivors, path arrays
  const int* order;
  const unsigned* ray_offset;  // by position in order
  const int* ray_starts;
  const unsigned long long* seg_tx;
  const double *field, *bound, *field64;  // field64 may be null
  const int* rx_bad;
  int n_req, rx_total;
  ResultLayout at;
  unsigned char* out;
  size_t room;
};

// One warp per path, after the grid's threads have copied the fixed part: bound
// by the latency of a few dependent loads and of the last store.  In its place a
// synchronisation told the host the sizes, 13 copies fetched the arrays as the
// field stage leaves them (17 slots a path), a blocking copy followed, and the
// host put the paths together: a call of 3,000 receivers and 3,148 paths took
// 0.88 ms, now 0.65; 24 requests with 98,304 receivers 15.1 ms, now 13.6.
__global__ void __launch_bounds__(256) k_result(const __grid_constant__ ResultArgs A) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  ResultHead* const head = reinterpret_cast<ResultHead*>(A.out);
  const bool overflow = A.f.ctr->overflow != 0;
  const size_t ns = overflow ? 0 : size_t(min(A.f.ctr->survivors, A.f.cap));
  const size_t rays = overflow || ns == 0 ? 0 : size_t(unsigned(A.ray_starts[A.rx_total]) - unsigned(A.ray_starts[0]));
  const bool fits = A.at.end(ns, rays) <= A.room;
  for (unsigned i = t; i < sizeof(Counters) / 8; i += nt)
    reinterpret_cast<unsigned long long*>(&head->c)[i] =
        reinterpret_cast<const unsigned long long*>(A.f.ctr)[i];
  if (t == 0) {
    head->fstat[0] = A.f.fstat[0];
    head->fstat[1] = A.f.fstat[1];
    head->rays = (long long)rays;
    head->rx_bad = *A.rx_bad;
    head->fits = fits;
  }
  if (overflow) return;  // this solve will be repeated
  unsigned long long* const seg = reinterpret_cast<unsigned long long*>(A.out + A.at.seg);
  for (unsigned i = t; i < unsigned(A.n_req); i += nt) seg[i] = A.seg_tx[i];
  double2* const field = reinterpret_cast<double2*>(A.out + A.at.field);
  double2* const field64 = reinterpret_cast<double2*>(A.out + A.at.field64);
  double* const bound = reinterpret_cast<double*>(A.out + A.at.bound);
  for (size_t i = t; i < 3 * size_t(A.rx_total); i += nt) {
    field[i] = reinterpret_cast<const double2*>(A.field)[i];
    if (A.field64) field64[i] = reinterpret_cast<const double2*>(A.field64)[i];
  }
  for (unsigned i = t; i < unsigned(A.rx_total); i += nt) bound[i] = A.bound[i];
  if (!fits) return;
  unsigned long long* const paths = reinterpret_cast<unsigned long long*>(A.out + A.at.paths);
  double* const points = reinterpret_cast<double*>(A.out + A.at.points(ns));
  int* const tri = reinterpret_cast<int*>(A.out + A.at.tri(ns, rays));
  constexpr int kWords = sizeof(sbr_path) / 8;
  static_assert(sizeof(sbr_path) == 88 && kWords <= 32, "a lane writes a word of a path");
  const unsigned lane = lane_id();
  for (size_t k = t >> 5; k < ns; k += nt >> 5) {
    const int i = A.order[k];
    const Survivor sv = A.f.surv[i];
    const int n = A.f.path_nray[i];
    const size_t o = A.ray_offset[k];
    const int req = A.f.rx_req[sv.rx];
    auto two = [](int lo, int hi) {
      return (unsigned long long)(unsigned)hi << 32 | (unsigned)lo;
    };
    if (lane < kWords) {
      unsigned long long w;
      if (lane == 0) w = two(req, int(sv.rx) - A.f.txp[req].rx_first);
      else if (lane == 1) w = two(n, int(sv.rank & ((1u << kHeapBits) - 1)));
      else if (lane == 2) w = sv.rank >> kHeapBits;
      else if (lane == 3) w = o;
      else if (lane == 10) w = two(A.f.path_near_edge[i], 0);
      else w = __double_as_longlong(A.f.path_field[6 * size_t(i) + lane - 4]);
      paths[k * kWords + lane] = w;
    }
    const size_t b = size_t(i) * (kMaxDepth + 1), q = size_t(i) * (kMaxDepth + 2) * 3;
    if (lane < unsigned(n)) {
      tri[o + lane] = A.f.path_tri[b + lane];
      tri[rays + o + lane] = A.f.path_cop[b + lane];
      tri[2 * rays + o + lane] = A.f.path_kind[b + lane];
    }
    for (int e = lane; e < 6 * n; e += 32)  // ray r: points r and r + 1
      points[6 * o + e] = A.f.path_pts[q + 3 * (e / 6) + e % 6];
  }
}

}  // namespace sbr
