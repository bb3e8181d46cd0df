// Trace stage: the reference's RayLaunch (RTSolver.cpp:128-257) as a
// wavefront, one bounce depth per launch pair: k_find (FP32 candidate search
// on the search BVH) and k_trace (FP64 resolution against the reference BVH,
// tree node, children, path-class interning).
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "sbr_device.h"
#include "sbr_field.cuh"
#include "sbr_kernels.cuh"
#include "sbr_common.cuh"

namespace sbr {

// ---- trace ------------------------------------------------------------------

struct TraceArgs {
  DevScene sc;
  const TxParams* txp;
  int n_tx;
  const double* const* dirs;  // per level
  const RayRec* in;
  RayRec* out;
  unsigned long long out_cap;
  NodeHot* nodes;
  NodeCold* nodes_cold;
  unsigned long long node_cap;
  HashTable cls_tab, cop_tab;
  ClassInfo* cls_info;
  ClassCap* cls_cap;
  uint32_t* cls_list;  // slots of the classes interned, in interning order
  const int* tri_cop;  // coplanar id by rank
  Counters* ctr;
  unsigned long long* seg_per_tx;  // executed segments per request
  int depth;
  long long n_root;    // total launches (depth 0)
  long long lo, hi;    // this launch covers rays [lo, hi) of the depth
  const uint2* cand;   // contenders of those rays (k_find)
  const unsigned char* ncand;
  const RayF32* ray32; // FP32 copies of those rays (k_find)
  unsigned long long* work;  // rays of the chunk handed out (zero at launch)
};

__device__ __forceinline__ int find_request(const TxParams* txp, int n_tx, long long g) {
  int lo = 0, hi = n_tx - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (txp[mid].launch_first <= g) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// The capture-stage record of a class with image source img (FP64) whose
// last ray starts on the triangle at mesh position tpos: the FP32 image source
// and correction-filter terms (the cone follows in k_class_cones).
__device__ void write_class_cap(const DevScene& sc, const double* img, int tpos, ClassCap& cc) {
  const Tri32 T = sc.corr32[tpos];
  const float3 o = make_float3(float(img[0]), float(img[1]), float(img[2]));
  const float no = sqrtf(o.x * o.x + o.y * o.y + o.z * o.z);
  const TriFrom F = tri_from(T, o, no);
  cc.img[0] = o.x;
  cc.img[1] = o.y;
  cc.img[2] = o.z;
  cc.tpos = tpos;
  cc.F[0] = F.sx; cc.F[1] = F.sy; cc.F[2] = F.sz;
  cc.F[3] = F.qx; cc.F[4] = F.qy; cc.F[5] = F.qz;
  cc.F[6] = F.W; cc.F[7] = F.ns;
}

// Correction cones of the interned classes (one thread per class-table
// slot, after the trace): three planes through the image source and the
// last triangle's edges, formed in FP64 and rounded to FP32, so a plane's
// error is its FP32 rounding alone.  Bound by the FP64 pipe: some 60
// instructions per class (its lengths' FP64 roots and quotients made them 330;
// the level-10 terrain's 1.36M classes 0.71 ms, now 0.55).
__global__ void k_class_cones(const uint32_t* list, const Counters* ctr, uint32_t cap,
                              const ClassInfo* info, DevScene sc, ClassCap* caps) {
  if (ctr->overflow & kOvTrace) return;  // this solve will be repeated
  const unsigned long long n = min(ctr->cls_listed, (unsigned long long)cap);
  for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < n;
       k += (unsigned long long)gridDim.x * blockDim.x) {
    const uint32_t s = list[k];
    const ClassInfo& ci = info[s];
    const CorrTri& T = sc.corr[sc.rank_to_id[ci.tri]];
    ClassCap& cc = caps[s];
    const double* im = ci.img;
    // the vertices and the centroid from the image source
    double v[3][3], g[3];
    for (int a = 0; a < 3; ++a) {
      v[0][a] = T.v1[a] - im[a];
      v[1][a] = v[0][a] + T.e1[a];
      v[2][a] = v[0][a] + T.e2[a];
      g[a] = (v[0][a] + v[1][a] + v[2][a]) * (1.0 / 3.0);
    }
    // lengths enter margins and thresholds only: FP32, rounded up
    auto norm32 = [](const double* x) {
      const float a = soft64::to_f32(x[0]), b = soft64::to_f32(x[1]), c = soft64::to_f32(x[2]);
      return sqrtf(a * a + b * b + c * c) * (1.0f + 1e-6f);
    };
    const float tmag = norm32(im) + norm32(T.v1) + norm32(T.e1) + norm32(T.e2) + 1.0f;
    const float len[3] = {norm32(v[0]), norm32(v[1]), norm32(v[2])};
    for (int k = 0; k < 3; ++k) {
      const double* a = v[k];
      const double* b = v[k == 2 ? 0 : k + 1];
      const double n[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2],
                           a[0] * b[1] - a[1] * b[0]};
      const float nn = norm32(n);
      // orient towards the triangle's centroid, which lies inside the cone
      const double gc = n[0] * g[0] + n[1] * g[1] + n[2] * g[2];
      const float sg = soft64::negative(gc) ? -1.0f : 1.0f;
      const double off = n[0] * im[0] + n[1] * im[1] + n[2] * im[2];
      for (int c = 0; c < 3; ++c) cc.n[k][c] = sg * soft64::to_f32(n[c]);
      cc.n[k][3] = sg * soft64::to_f32(off);
      cc.nn[k] = nn;
      cc.w[k] = nn * tmag;
      // FP64 forms n to within 2^-50 |a||b| and gc to within that times the
      // distance: the plane is used where both are far below what they are
      // compared with (n's FP32 rounding, gc's sign)
      const float ga = fabsf(soft64::to_f32(gc));
      cc.gc[k] = nn > 1e-6f * (len[k] * len[k == 2 ? 0 : k + 1]) && ga > 4e-9f * cc.w[k] ? ga : 0.0f;
    }
  }
}

// Records an interned class's slot for k_class_cones (the list has the class
// table's capacity, which bounds the classes).
__device__ __forceinline__ void list_class(const TraceArgs& A, uint32_t cls) {
  const unsigned long long k = atomicAdd(&A.ctr->cls_listed, 1ull);
  if (k <= A.cls_tab.mask) A.cls_list[k] = cls;
}

// Every thread that interns a class writes the same values (they depend
// only on the key), so concurrent writers agree.
__device__ __forceinline__ void write_class(ClassInfo& ci, const double* img, uint32_t parent,
                                            int tri, uint32_t cop, int kind, int depth) {
  ci.img[0] = img[0];
  ci.img[1] = img[1];
  ci.img[2] = img[2];
  ci.img32[0] = float(img[0]);
  ci.img32[1] = float(img[1]);
  ci.img32[2] = float(img[2]);
  ci.parent = parent;
  ci.tri = tri;
  ci.cop = cop;
  ci.kind = uint8_t(kind);
  ci.depth = uint8_t(depth);
  ci.pad0 = ci.pad1 = 0;
  ci.pad2 = 0;
}

// Records of the freshly interned class `cls`: reached from class `parent` by
// an interaction of `kind` on the triangle of depth-first rank `rank`.  A
// reflection's image source is ImagePoint (RTSolver.cpp:910-924) of the
// parent's (the transmitter for a launch) across the triangle the reference
// finds at this id's position of its mesh vector; a transmission keeps it.
__device__ __noinline__ void intern_class(const TraceArgs& A, uint32_t cls, uint32_t parent,
                                          const double* tx, int rank, uint32_t cop, int kind) {
  const double* pimg = is_root_class(parent) ? tx : A.cls_info[parent].img;
  const int mpos = A.sc.rank_to_id[rank];
  double img[3] = {pimg[0], pimg[1], pimg[2]};
  if (kind == 1) {
    const CorrTri& M = A.sc.corr[mpos];
    double w[3];
    x64::sub3(pimg, M.v1, w);
    const double dist = x64::dot(M.n, w);
    for (int a = 0; a < 3; ++a)
      img[a] = x64::sub(pimg[a], x64::mul(x64::mul(2.0, dist), M.n[a]));
  }
  write_class(A.cls_info[cls], img, parent, rank, cop, kind, A.depth + 1);
  write_class_cap(A.sc, img, mpos, A.cls_cap[cls]);
  list_class(A, cls);
}

// Number of rays entering bounce depth `depth` (known on the device only).
__device__ __forceinline__ long long rays_at_depth(const Counters* ctr, int depth, long long n_root,
                                                   unsigned long long cap) {
  return depth == 0 ? n_root : (long long)min(ctr->queue[depth], cap);
}

// Index of the first node of bounce depth `depth`: every ray makes one tree
// node, and ray i of a depth makes node node_base + i, so no counter hands
// the nodes out and the records are written in ray order.
__device__ __forceinline__ unsigned long long node_base(const Counters* ctr, int depth,
                                                        long long n_root, unsigned long long cap) {
  unsigned long long b = 0;
  for (int d = 0; d < depth; ++d) b += (unsigned long long)rays_at_depth(ctr, d, n_root, cap);
  return b;
}

// Launch ray g of the batch: origin and direction (FP64).
__device__ __forceinline__ void root_ray(const TxParams* txp, int n_tx, const double* const* dirs,
                                         long long g, double* o, double* d, int& q, long long& li) {
  q = find_request(txp, n_tx, g);
  const TxParams& P = txp[q];
  li = g - P.launch_first;
  const double* dd = dirs[P.level] + 3 * li;
  for (int a = 0; a < 3; ++a) {
    o[a] = P.tx[a];
    d[a] = dd[a];
  }
}

// Origin and direction of ray i of bounce depth `depth`.
__device__ __forceinline__ void load_ray_line(const TxParams* txp, int n_tx,
                                              const double* const* dirs, const RayRec* in,
                                              int depth, long long i, double* o, double* d) {
  if (depth == 0) {
    int q;
    long long li;
    root_ray(txp, n_tx, dirs, i, o, d, q, li);
  } else {
    for (int a = 0; a < 3; ++a) {
      o[a] = in[i].o[a];
      d[a] = in[i].d[a];
    }
  }
}

// Ray i of bounce depth `depth`: a launch ray (depth 0) or a queued child.
__device__ __forceinline__ void load_ray(const TxParams* txp, int n_tx, const double* const* dirs,
                                         const RayRec* in, int depth, long long i, RayRec& r) {
  if (depth == 0) {
    int q;
    long long li;
    root_ray(txp, n_tx, dirs, i, r.o, r.d, q, li);
    r.total = 0.0;
    r.S = 0.0;
    r.parent = 0xFFFFFFFFu;
    r.orank = -1;
    r.cls = kRootBase + uint32_t(q);
    r.cop = kRootClass;
    r.launch = uint32_t(li);
    r.heap = 1;
    r.rc = r.tc = 0;
    r.tx = uint32_t(q);
  } else {
    r = in[i];
  }
}

// The tree node ni of a resolved ray (RTSolver.cpp:142-257): its record (hot
// FP32 part and cold FP64 part).  A ray that hits nothing ends at
// src + 1e10 d (a launch) or src + 100 d (RTSolver.cpp:231,249).
__device__ __forceinline__ void emit_node(NodeHot* nodes, NodeCold* cold,
                                          unsigned long long cap, Counters* ctr,
                                          unsigned long long ni, const RayRec& r, bool root,
                                          const float3& o32, const float3& d32, bool soft,
                                          bool hit, const Hit& h) {
  if (ni < cap) {
    NodeCold n;
    NodeHot m;
    n.s[0] = r.o[0]; n.s[1] = r.o[1]; n.s[2] = r.o[2];
    if (hit) {
      n.t[0] = h.p[0]; n.t[1] = h.p[1]; n.t[2] = h.p[2];
      m.len = soft64::to_f32(h.dist);
    } else {
      const double sc = root ? 1E10 : 1E2;  // RTSolver.cpp:231,249
      for (int a = 0; a < 3; ++a)
        n.t[a] = x64::add(r.o[a], soft ? soft64::mul(r.d[a], sc) : x64::mul(r.d[a], sc));
      m.len = float(sc);
    }
    n.S = r.S;
    n.pad = 0.0;
    m.s[0] = o32.x; m.s[1] = o32.y; m.s[2] = o32.z;
    m.S = soft64::to_f32(r.S);
    m.u[0] = d32.x; m.u[1] = d32.y; m.u[2] = d32.z;
    m.parent = r.parent;
    m.cls = r.cls;
    m.launch = r.launch;
    m.heap = r.heap;
    m.tx = r.tx;
    m.pad0 = m.pad1 = m.pad2 = 0;
    cold[ni] = n;
    nodes[ni] = m;
  } else {
    atomicOr(&ctr->overflow, kOvNodes);
  }
}

// Executed segments per request, counted by each lane and added when the
// request changes (a lane's rays are mostly one request's).
struct SegmentCount {
  uint32_t tx;
  unsigned n;
  __device__ __forceinline__ void flush(unsigned long long* per_tx) {
    if (n) atomicAdd(&per_tx[tx], (unsigned long long)n);
    n = 0;
  }
  // The whole warp: one atomic per request present.
  __device__ __forceinline__ void warp_flush(unsigned long long* per_tx) {
    unsigned left = __ballot_sync(0xffffffffu, n != 0);
    while (left) {
      const int lead = __ffs(left) - 1;
      const uint32_t t = __shfl_sync(0xffffffffu, tx, lead);
      const bool mine = n != 0 && tx == t;
      const unsigned sum = __reduce_add_sync(0xffffffffu, mine ? n : 0);
      if (int(lane_id()) == lead) atomicAdd(&per_tx[tx], (unsigned long long)sum);
      left &= ~__ballot_sync(0xffffffffu, mine);
    }
    n = 0;
  }
  __device__ __forceinline__ void add(unsigned long long* per_tx, uint32_t t) {
    if (t != tx) flush(per_tx);
    tx = t;
    ++n;
  }
};

// The next rays of the chunk for the idle lanes `im`: the j-th idle lane gets
// the j-th of them (>= n: none left; exhausted, the same on every lane, when
// the counter has passed the end).  Exactly as many as there are idle lanes
// are taken, so that the warps together move through the chunk in order and
// the children are queued near their neighbours': handing each warp a window
// of 32 to 256 rays cost the level-9 canyon solve 1.4 ms in the next depths'
// scattered rays, far more than the atomics it saved.
__device__ __forceinline__ long long next_rays(unsigned long long* counter, unsigned im,
                                               unsigned lane, long long n, bool& exhausted) {
  const int want = __popc(im), leader = __ffs(im) - 1;
  unsigned long long base = 0;
  if (int(lane) == leader) base = atomicAdd(counter, (unsigned long long)want);
  base = __shfl_sync(0xffffffffu, base, leader);
  if ((long long)base + want >= n) exhausted = true;
  return (long long)base + __popc(im & ((1u << lane) - 1u));
}

// x64::normalize for components in soft64's range.
__device__ __forceinline__ void normalize_soft(const double* a, double* r) {
  const double z = dot64<Soft64>(a, a);
  if (soft64::bits(z) != 0) {  // a sum of squares: never -0
    const double s = soft64::sqrt(z);
    const uint64_t x = soft64::rcp_of(s);
    for (int i = 0; i < 3; ++i) r[i] = soft64::div_by(a[i], s, x);
  } else {
    for (int i = 0; i < 3; ++i) r[i] = a[i];
  }
}

// ---- FP32 candidate search (persistent, rays refilled per warp) ----------
//
// Each lane traverses one ray at a time.  Lanes whose ray is finished take a
// new one from the chunk's work counter (one atomic per warp, when at least
// half the warp is idle or nobody is busy), so warps stay full while rays of
// very different lengths finish at different times.  The search tree is
// four-wide; a step is one node visit (four child boxes) or up to
// tris_per_step triangle tests, so lanes in a leaf and lanes between nodes
// advance at a similar pace.  The FP32 copy of each ray it loads is kept for
// k_trace (ray32).
struct FindArgs {
  DevScene sc;
  const TxParams* txp;
  int n_tx;
  const double* const* dirs;
  RayRec* in;  // reflected rays get their direction normalised here
  const Counters* ctr;
  unsigned long long in_cap;
  long long n_root;
  int depth;
  long long lo, hi;            // this launch covers rays [lo, hi) of the depth
  unsigned long long* work;    // rays of the chunk handed out (zero at launch)
  uint2* cand;                 // kCand per ray of the chunk
  unsigned char* ncand;        // contenders per ray, kFindFallback = exact traversal
  RayF32* ray32;               // FP32 copy per ray of the chunk
  int steps;                   // traversal steps between refills
  int refill;                  // idle lanes that trigger a refill
  int tris_per_step;           // triangles of a leaf tested per step (1 or 2)
};

// Defaults of the search's tunables (the autotuner may choose others).
constexpr int kFindSteps = 32;
constexpr int kFindRefill = 16;

__global__ void __launch_bounds__(128, 8) k_find(FindArgs A) {
  if (A.ctr->overflow & kOvTrace) return;  // this solve will be repeated
  const long long n_all = rays_at_depth(A.ctr, A.depth, A.n_root, A.in_cap);
  const long long n = min(n_all, A.hi) - A.lo;
  if (n <= 0) return;
  const unsigned lane = lane_id();
  bool exhausted = false;
  long long ray = -1;
  float3 o32 = make_float3(0, 0, 0), d32 = o32;
  SlabRay slab = {};
  float no = 0.0f, nd = 0.0f, tcut = INFINITY;
  int2 stack[kStack];  // child ref, entry distance (bits)
  int sp = 0, cur = 0, nc = 0, orank = -1;
  bool fail = false, safe = false;
  uint2* out = nullptr;
  while (true) {
    const unsigned im = __ballot_sync(0xffffffffu, ray < 0);
    if ((__popc(im) >= A.refill || im == 0xffffffffu) && !exhausted) {
      const long long k = next_rays(A.work, im, lane, n, exhausted);
      if (ray < 0 && k < n) {
        ray = k;
        double o[3], d[3];
        orank = -1;
        if (A.depth == 0) {
          int q;
          long long li;
          root_ray(A.txp, A.n_tx, A.dirs, A.lo + k, o, d, q, li);
        } else {
          RayRec& r = A.in[A.lo + k];
          for (int a = 0; a < 3; ++a) {
            o[a] = r.o[a];
            d[a] = r.d[a];
          }
          if (r.heap & 1) {
            // a reflected ray (heap 2h+1) arrives with Reflect(d, n) not yet
            // normalised: normalise it here, where a refill runs on at least
            // half the warp's lanes, and store it for k_trace
            double v[3] = {d[0], d[1], d[2]};
            if (soft64::safe(v[0]) && soft64::safe(v[1]) && soft64::safe(v[2]))
              normalize_soft(v, d);
            else
              x64::normalize(v, d);
            for (int a = 0; a < 3; ++a) r.d[a] = d[a];
          }
          orank = r.orank;
        }
        o32 = make_float3(soft64::to_f32(o[0]), soft64::to_f32(o[1]), soft64::to_f32(o[2]));
        d32 = make_float3(soft64::to_f32(d[0]), soft64::to_f32(d[1]), soft64::to_f32(d[2]));
        safe = soft64::safe(o[0]) && soft64::safe(o[1]) && soft64::safe(o[2]) &&
               soft64::safe(d[0]) && soft64::safe(d[1]) && soft64::safe(d[2]);
        {
          float4* f = reinterpret_cast<float4*>(A.ray32 + k);
          f[0] = make_float4(o32.x, o32.y, o32.z, 0.0f);
          f[1] = make_float4(d32.x, d32.y, d32.z, 0.0f);
        }
        no = sqrtf(o32.x * o32.x + o32.y * o32.y + o32.z * o32.z);
        nd = sqrtf(d32.x * d32.x + d32.y * d32.y + d32.z * d32.z);
        slab = slab_ray(o32, d32, A.sc.box_margin + kBoxK * no);
        tcut = INFINITY;
        sp = 0;
        cur = 0;  // the search root is always a node
        nc = 0;
        fail = false;
        out = A.cand + size_t(k) * kCand;
      }
      __syncwarp();
    }
    if (__ballot_sync(0xffffffffu, ray >= 0) == 0) break;  // every lane is out of rays
    if (ray < 0) continue;
    bool done = false;
    for (int it = 0; it < A.steps && !done; ++it) {
      // A step is either a node visit or leaf tests, for all lanes: leaves are
      // tested when half of the lanes hold one, and every fourth step.  Taking
      // both kinds in each step ran the triangle test with 11 lanes, the node
      // visit with 21: level-9 canyon search 4.55 ms against 3.80, level-10
      // terrain 9.3 against 8.0 (a third of the lanes: 3.86 and 8.1; every
      // eighth step: 3.93 and 7.9).
      const unsigned active = __activemask();
      const unsigned leaves = __ballot_sync(active, cur < 0);
      const bool leaf_step = leaves && (2 * __popc(leaves) >= __popc(active) || (it & 3) == 3);
      if (leaf_step != (cur < 0)) continue;
      if (leaf_step) {
        // up to tris_per_step triangles of the leaf per step
        for (int q = 0; q < A.tris_per_step && cur != kEmptyChild; ++q) {
          const int j = ~cur >> 3, left = (~cur & 7) - 1;
          cur = left > 0 ? ~((j + 1) << 3 | left) : kEmptyChild;
          float tlo, thi;
          const Tri32 T = A.sc.stri[j];
          const int k = tri_classify(T, o32, d32, no, nd, tlo, thi);
          if (k == 0 || tlo > tcut) continue;
          const int rk = __ldg(A.sc.srank + j);
          // the triangle the ray starts on, left at a clear angle: the
          // reference's test of it certainly fails (origin_rejected); such a
          // contender is never a sure hit, so dropping it changes no cut
          if (rk == orank && origin_rejected(T, o32, d32)) continue;
          if (nc == kCand) {
            fail = done = true;
            break;
          }
          out[nc++] = make_uint2(unsigned(rk) | (k & kSureUV ? kContUV : 0u),
                                 __float_as_uint(tlo));
          if (k & kSureHit) tcut = fminf(tcut, thi * (1.0f + kTieSlack) + 1e-30f);
        }
      } else {
        // a four-wide node: the children the ray's slab test keeps (within
        // tcut), nearest first; it goes on with the nearest, the farther ones
        // go on the stack
        int c[4];
        float t[4];
        const int need = visit_node4(A.sc.snode4 + cur, slab, tcut, c, t);
        if (sp + need > kStack) {
          fail = done = true;
          break;
        }
        if (need > 3) stack[sp++] = make_int2(c[3], __float_as_int(t[3]));
        if (need > 2) stack[sp++] = make_int2(c[2], __float_as_int(t[2]));
        if (need > 1) stack[sp++] = make_int2(c[1], __float_as_int(t[1]));
        cur = c[0];
      }
      // The next child off the stack that a hit found since has not cut off,
      // taken in this step: a lane starts each step with a node or a leaf in
      // hand.  A cut-off child cost a node visit before, a postponed leaf a
      // step of its own (level-9 canyon search 4.13 ms, now 3.96; level-10
      // terrain 8.6, now 8.35).
      while (cur == kEmptyChild) {
        if (sp == 0) {
          done = true;
          break;
        }
        const int2 e = stack[--sp];
        if (__int_as_float(e.y) <= tcut) cur = e.x;
      }
    }
    if (done) {
      A.ncand[ray] = fail ? kFindFallback : (unsigned char)(safe ? nc : nc | kCandUnsafe);
      ray = -1;
    }
  }
}

// Resident blocks of k_trace per SM (register budget 65536 / (128 x this)).
// Level-9 canyon, k_trace in all: 4 blocks 5.28 ms, 5 5.38 (spills), 6 5.97, 3
// 5.80; its warps wait for memory and for instructions alike.
#ifndef SBR_TRACE_BLOCKS
#define SBR_TRACE_BLOCKS 4
#endif

// Reflect(d, n) with the FP64 pipe's products (see mt64_call).
__device__ __noinline__ D3 reflect_call(const double* n, double dx, double dy, double dz) {
  const double d[3] = {dx, dy, dz};
  const double dn2 = 2.0 * x64::dot(n, d);
  return D3{x64::sub(dx, x64::mul(n[0], dn2)), x64::sub(dy, x64::mul(n[1], dn2)),
            x64::sub(dz, x64::mul(n[2], dn2))};
}

// Queue slots of the active lanes' children, one atomic: the transmitted rays
// first, then the reflected ones, so that a warp of the next depth finds rays
// that go the same way.
__device__ __forceinline__ void reserve_children(unsigned long long* queue, bool do_t, bool do_r,
                                                 unsigned long long& slot_t,
                                                 unsigned long long& slot_r) {
  const unsigned mask = __activemask();
  const unsigned bt = __ballot_sync(mask, do_t), br = __ballot_sync(mask, do_r);
  const unsigned lt = (1u << lane_id()) - 1u;
  const int leader = __ffs(mask) - 1;
  unsigned long long base = 0;
  if (lane_id() == unsigned(leader) && (bt | br))
    base = atomicAdd(queue, (unsigned long long)(__popc(bt) + __popc(br)));
  base = __shfl_sync(mask, base, leader);
  slot_t = base + __popc(bt & lt);
  slot_r = base + __popc(bt) + __popc(br & lt);
}

// The tree node of a resolved ray and its children (RTSolver.cpp:142-257):
// node record (node ni), reflected and transmitted rays, path-class interning.
// The three table probes are begun together: one memory latency, not three.
__device__ __forceinline__ void finish_ray(const TraceArgs& A, unsigned long long ni,
                                           const RayRec& r, const float3& o32, const float3& d32,
                                           bool soft, bool hit, const Hit& h) {
  const TxParams& P = A.txp[r.tx];
  // children (RTSolver.cpp:186-221)
  const bool do_r = hit && r.rc < P.R, do_t = hit && r.tc < P.T;
  HashProbe p_cop, p_t, p_r;
  if (do_r || do_t) {
    p_cop = ht_probe(A.cop_tab, (unsigned long long)r.cop << 32 | uint32_t(A.tri_cop[h.rank]));
    const unsigned long long key = (unsigned long long)r.cls << 32 | uint32_t(h.rank) << 1;
    if (do_t) p_t = ht_probe(A.cls_tab, key | 1u);
    if (do_r) p_r = ht_probe(A.cls_tab, key);
  }
  unsigned long long slot_t, slot_r;
  reserve_children(&A.ctr->queue[A.depth + 1], do_t, do_r, slot_t, slot_r);
  emit_node(A.nodes, A.nodes_cold, A.node_cap, A.ctr, ni, r, A.depth == 0, o32, d32, soft,
            hit, h);
  if (do_r || do_t) {
    const double cum = x64::add(r.total, h.dist);  // node pathLength
    RayRec c;
    c.o[0] = h.p[0]; c.o[1] = h.p[1]; c.o[2] = h.p[2];
    c.total = cum;
    c.S = x64::add(r.S, cum);
    c.parent = uint32_t(ni);
    c.launch = r.launch;
    c.tx = r.tx;
    c.orank = h.rank;
    const uint32_t cop_cls = ht_insert(A.cop_tab, p_cop, &A.ctr->overflow, kOvCop,
                                       &A.ctr->used_cop, &A.ctr->lost_cop);
    c.cop = cop_cls;
    if (do_t) {  // transmitted: same direction, heap 2h, same image source
      c.d[0] = r.d[0]; c.d[1] = r.d[1]; c.d[2] = r.d[2];
      c.heap = r.heap * 2;
      c.rc = r.rc;
      c.tc = r.tc + 1;
      bool fresh = false;
      c.cls = ht_insert(A.cls_tab, p_t, &A.ctr->overflow, kOvClass, &A.ctr->used_cls,
                        &A.ctr->lost_cls, &fresh);
      if (fresh)  // only the thread that interned the class writes its records
        intern_class(A, c.cls, r.cls, P.tx, h.rank, cop_cls, 2);
      if (slot_t < A.out_cap) A.out[slot_t] = c;
      else atomicOr(&A.ctr->overflow, kOvQueue);
    }
    if (do_r) {  // reflected: Reflect(d, n), heap 2h+1; k_find normalises it
      const double* n = A.sc.tri64[h.rank].n;
      // (2 n) dn and n (2 dn) are the same number rounded once
      if (soft) {
        const double dn2 = 2.0 * dot64<Soft64>(n, r.d);
        for (int a = 0; a < 3; ++a) c.d[a] = x64::sub(r.d[a], soft64::mul(n[a], dn2));
      } else {
        const D3 v = reflect_call(n, r.d[0], r.d[1], r.d[2]);
        c.d[0] = v.x;
        c.d[1] = v.y;
        c.d[2] = v.z;
      }
      c.heap = r.heap * 2 + 1;
      c.rc = r.rc + 1;
      c.tc = r.tc;
      bool fresh = false;
      c.cls = ht_insert(A.cls_tab, p_r, &A.ctr->overflow, kOvClass, &A.ctr->used_cls,
                        &A.ctr->lost_cls, &fresh);
      if (fresh) intern_class(A, c.cls, r.cls, P.tx, h.rank, cop_cls, 1);
      if (slot_r < A.out_cap) A.out[slot_r] = c;
      else atomicOr(&A.ctr->overflow, kOvQueue);
    }
  }
}

// The untested contender with the lowest bound on t (the first of equal ones,
// as a stable sort would give): its index, or -1 when none is left.
__device__ __forceinline__ int next_contender(const uint2* cand, int nc, unsigned tested, float& t,
                                              int& code) {
  int k = -1;
#pragma unroll 1
  for (int j = 0; j < nc; ++j) {
    if (tested >> j & 1u) continue;
    const uint2 e = cand[j];
    const float tj = __uint_as_float(e.y);
    if (k < 0 || tj < t) {
      k = j;
      t = tj;
      code = int(e.x);
    }
  }
  return k;
}

// FP64 resolution of the contenders k_find left: they are tested in
// ascending order of their FP32 lower bound on t until none can reach the
// best exact distance; the answer is the lexicographic minimum (distance,
// depth-first rank), the reference's strict '<' in visit order, accepted if
// its leaf is reachable in the reference BVH (leaf_reachable), else the ray
// takes the reference-order traversal.  The kernel
// is persistent: each lane holds one ray and runs at most one
// triangle test per round, so the warp's instructions serve every
// lane that has a test due, whether it is a ray's first contender or a later
// one.  A lane whose ray is resolved writes the node and children in the
// same round and takes a new ray; a ray needing a
// second test no longer holds the whole warp through a second pass of the
// test with a few lanes.  The warp is brought together after each part of a
// round.  kRoot: the launch rays (depth 0).  A lane keeps only the ray's
// origin and direction and the best hit between rounds; the rest of its
// record is read again when it is resolved.
template <bool kRoot>
__global__ void __launch_bounds__(128, SBR_TRACE_BLOCKS)
    k_trace(const __grid_constant__ TraceArgs A) {
  if (A.ctr->overflow & kOvTrace) return;  // this solve will be repeated
  const long long n_all = rays_at_depth(A.ctr, A.depth, A.n_root, A.out_cap);
  const long long n = min(n_all, A.hi) - A.lo;
  if (n <= 0) return;
  const unsigned lane = lane_id();
  unsigned fp64_tri = 0, fallback = 0;
  SegmentCount seg{0, 0};
  bool exhausted = false;
  const unsigned long long base = node_base(A.ctr, A.depth, A.n_root, A.out_cap) + A.lo;
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&A.ctr->nodes, (unsigned long long)n);
  long long c = -1;  // the lane's ray (index in the chunk), -1 = none
  double o[3] = {0, 0, 0}, d[3] = {0, 0, 0};
  int nc = 0;
  unsigned tested = 0;      // contenders already tested (bit mask)
  int next = -1, code = 0;  // the contender due: its index (-1 none), rank | kContUV
  float tn = 0.0f;          // and lower bound on t
  float tbest = 0.0f;       // FP32 copy of best.t
  Hit best;
  best.rank = INT_MAX;
  best.leaf = -1;
  best.t = 0.0;
  while (true) {
    // Refill: the idle lanes take the next window of rays (the j-th idle
    // lane the window's j-th ray, so the loads stay in order).  A ray k_find
    // left without a contender hits nothing: its lane writes the node at once
    // and stays idle, so such rays never hold a lane through a round of FP64
    // tests.  This repeats until no lane is idle or the chunk is done.
    unsigned im = __ballot_sync(0xffffffffu, c < 0);
    while (im && !exhausted) {
      const long long k = next_rays(A.work, im, lane, n, exhausted);
      if (c < 0 && k < n) {
        nc = A.ncand[k];
        if (!(nc & kCandCount)) {
          RayRec r;
          load_ray(A.txp, A.n_tx, A.dirs, A.in, kRoot ? 0 : 1, A.lo + k, r);
          const float4* f = reinterpret_cast<const float4*>(A.ray32 + k);
          const float4 fo = f[0], fd = f[1];
          Hit none;
          seg.add(A.seg_per_tx, r.tx);
          emit_node(A.nodes, A.nodes_cold, A.node_cap, A.ctr, base + k, r, kRoot,
                    make_float3(fo.x, fo.y, fo.z), make_float3(fd.x, fd.y, fd.z),
                    !(nc & kCandUnsafe), false, none);
        } else {
          load_ray_line(A.txp, A.n_tx, A.dirs, A.in, kRoot ? 0 : 1, A.lo + k, o, d);
          c = k;
          tested = 0;
          next = nc != kFindFallback
                     ? next_contender(A.cand + size_t(k) * kCand, nc & kCandCount, 0u, tn, code)
                     : -1;
          best.rank = INT_MAX;
          best.dist = __longlong_as_double(0x7ff0000000000000ll);
        }
      }
      __syncwarp();
      im = __ballot_sync(0xffffffffu, c < 0);
    }
    if (__ballot_sync(0xffffffffu, c >= 0) == 0) break;  // every lane is out of rays
    const bool soft = A.sc.soft && !(nc & kCandUnsafe);
    if (c >= 0 && next >= 0) {  // the contender due
      const int rk = code & ~int(kContUV);
      ++fp64_tri;
      const Tri64& T = A.sc.tri64[rk];
      double t, P[3], dist;
      bool ok;
      if (soft) {
        ok = mt64_t<Soft64>(T, o, d, code < 0, t, P, dist);
      } else {
        const Mt64Result m = mt64_call(&T, o[0], o[1], o[2], d[0], d[1], d[2]);
        ok = m.ok;
        t = m.t;
        dist = m.dist;
        for (int a = 0; a < 3; ++a) P[a] = m.p[a];
      }
      if (ok && (soft64::less(dist, best.dist) ||
                 (soft64::same(dist, best.dist) && rk < best.rank))) {
        best.dist = dist;
        tbest = soft64::to_f32(t);
        best.p[0] = P[0];
        best.p[1] = P[1];
        best.p[2] = P[2];
        best.rank = rk;
      }
    }
    __syncwarp();
    bool done = false, hit = false;
    if (c >= 0) {
      if (nc == kFindFallback) {  // more contenders than kept, or a deep stack: one-pass search
        best = closest_call(A.sc, o[0], o[1], o[2], d[0], d[1], d[2], A.ctr);
        hit = best.rank != INT_MAX;
        done = true;
      } else {
        // resolved when no further contender can reach the best exact distance
        tested |= 1u << next;
        next = (nc & kCandCount) > 1
                   ? next_contender(A.cand + size_t(c) * kCand, nc & kCandCount, tested, tn, code)
                   : -1;
        done = next < 0 ||
               !(best.rank == INT_MAX || tn <= tbest * (1.0f + kTieSlack) + 1e-30f);
        hit = done && best.rank != INT_MAX;
      }
    }
    __syncwarp();
    if (done) {
      RayRec r;
      load_ray(A.txp, A.n_tx, A.dirs, A.in, kRoot ? 0 : 1, A.lo + c, r);
      const float4* f = reinterpret_cast<const float4*>(A.ray32 + c);
      const float4 fo = f[0], fd = f[1];
      const float3 o32 = make_float3(fo.x, fo.y, fo.z), d32 = make_float3(fd.x, fd.y, fd.z);
      for (int a = 0; a < 3; ++a) {
        r.o[a] = o[a];
        r.d[a] = d[a];
      }
      if (hit && nc != kFindFallback) {
        const float3 i32 = make_float3(1.0f / d32.x, 1.0f / d32.y, 1.0f / d32.z);
        if (!leaf_reachable(A.sc, A.sc.tri64[best.rank].node, o, d, o32, d32, i32)) {
          ++fallback;
          best = exact_call(A.sc, o[0], o[1], o[2], d[0], d[1], d[2], &A.ctr->overflow);
          hit = best.rank != INT_MAX;
        }
      }
      seg.add(A.seg_per_tx, r.tx);
      finish_ray(A, base + c, r, o32, d32, soft, hit, best);
      c = -1;
    }
    __syncwarp();
  }
  seg.warp_flush(A.seg_per_tx);
  fp64_tri = __reduce_add_sync(0xffffffffu, fp64_tri);
  if (lane == 0 && fp64_tri) atomicAdd(&A.ctr->fp64_tri, (unsigned long long)fp64_tri);
  if (fallback) atomicAdd(&A.ctr->fallback, (unsigned long long)fallback);
}

}  // namespace sbr
