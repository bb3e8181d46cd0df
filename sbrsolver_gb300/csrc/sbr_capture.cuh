// Capture stage: RayCapture's reception-sphere test (RTSolver.cpp:259-297,
// 805-863) for every tree node against the receivers near its segment, with
// the first step of image correction as a prefilter; k_capture_finish makes
// the FP64 decisions (exact reception test, MultiPathCorrection, suppression
// by a capturing ancestor) for what the FP32 tests could not settle.
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "sbr_device.h"
#include "sbr_field.cuh"
#include "sbr_kernels.cuh"
#include "sbr_common.cuh"
#include "sbr_trace.cuh"

namespace sbr {

// ---- capture ----------------------------------------------------------------

struct CaptureArgs {
  DevScene sc;
  const NodeHot* nodes;
  const NodeCold* nodes_cold;
  const TxParams* txp;
  const RxGrid* grids;  // per request, all receivers; then per request, those with a direct
                        // path, for the launch rays' own segments
  int n_tx;
  const GridBuild* gb;
  const double* rx;
  const ClassInfo* cls_info;
  const ClassCap* cls_cap;
  const unsigned char* direct_ok;
  Corrected* corr_list;
  unsigned long long corr_cap;
  Counters* ctr;
  unsigned long long node_cap;
  uint2* pairs;                // (node, receiver | unsure << 31) for k_capture_finish
  unsigned long long pair_cap;
  HashTable corr_cache;        // (class, receiver) -> its image correction's outcome
  unsigned char* corr_val;     // per slot: 0 not known yet, 1 fails, 2 succeeds
  unsigned long long* work;    // nodes handed out to warps (zero at launch)
};

// MultiPathCorrection (RTSolver.cpp:330-373) for one capture, walking the
// path class from the receiver back to the transmitter: the line from each
// ray's image source to its current target must cross the triangle at that
// id's mesh position.  FP32 filter first (nearly every correction fails at
// its first test); the FP64 test in the reference's order decides the rest
// and yields the exact intersection that becomes the next target.
__device__ __forceinline__ bool correct_event(const DevScene& sc, const ClassInfo* info,
                                             uint32_t cls, const float3& c32, const double* c64,
                                             unsigned& n64) {
  double tgt[3] = {c64[0], c64[1], c64[2]};
  float3 t32 = c32;
  for (uint32_t c = cls; !is_root_class(c);) {
    const ClassInfo& ci = info[c];
    const int mpos = sc.rank_to_id[ci.tri];
    const float3 o = make_float3(ci.img32[0], ci.img32[1], ci.img32[2]);
    const float3 d = make_float3(t32.x - o.x, t32.y - o.y, t32.z - o.z);
    const float no = sqrtf(o.x * o.x + o.y * o.y + o.z * o.z);
    const float nd = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
    float tlo;
    if (!tri_filter(sc.corr32[mpos], o, d, no, nd, tlo)) return false;
    ++n64;
    double dd[3], P3[3];
    x64::sub3(tgt, ci.img, dd);
    if (!mt64c(sc.corr[mpos], ci.img, dd, P3)) return false;
    tgt[0] = P3[0];
    tgt[1] = P3[1];
    tgt[2] = P3[2];
    t32 = make_float3(float(P3[0]), float(P3[1]), float(P3[2]));
    c = ci.parent;
  }
  return true;
}

// Exact decision for a test inside the FP32 margin (reception64 on the
// node's FP64 record).
__device__ __noinline__ int capture_exact(const NodeCold* cold, uint32_t idx, const double* c64,
                                          double tanb) {
  const NodeCold& n = cold[idx];
  return reception64(n.s, n.t, c64, n.S, tanb) ? 1 : 0;
}

// A warp works through batches of nodes.  Each node's segment is clipped to
// the region that can hold its captures and cut into chunks (each receiver is
// owned by the chunk its projection falls in); each chunk's capsule is
// rasterised over the receiver grid one row of cells per lane; a row is one
// contiguous run of receivers, and the lanes stride over the concatenation of
// the rows' runs.  A capture counts unless an ancestor of the node captures
// the same receiver (RTSolver.cpp:277-284).
constexpr int kCapWarps = 4;
// Nodes staged per warp at a time (at most 32: one per lane; 16 leaves more
// of the SM's shared memory to L1 for the receiver grid).
#ifndef SBR_CAP_BATCH
#define SBR_CAP_BATCH 16
#endif
constexpr int kCapBatch = SBR_CAP_BATCH;

// Upper bound on sqrt(x) from the hardware reciprocal square root (relative
// error below 2^-21), for the capture stage's conservative ranges and
// margins, which all carry slack far beyond that.
__device__ __forceinline__ float sqrt_up(float x) {
  if (!(x > 0.0f)) return 0.0f;
  if (isinf(x)) return x;
  return x * rsqrtf(x) * 1.00000095367431640625f;  // 1 + 2^-20
}

// Correction cone of a class: the points c for which the line from the
// image source img towards c crosses the class's last triangle T
// (MultiPathCorrection's first test for a capture at c; RTSolver.cpp:356).
// Three planes through img and T's edges, n_k . p >= n_k . img, formed once
// per class in FP64 and rounded to FP32 (k_class_cones); k_capture_fast loosens
// each by 2 m_k, m_k = 2^-21 |n_k| (cmax + |img| + |T| + 1).  The FP32 test
// of a point p (|p| <= cmax) or of a cell corner errs by under
// 10 * 2^-24 |n_k| (cmax + |img| + |T|): the plane's rounding, the rounding
// of p, and the dot product.  A plane counts as long as FP64 settles its
// orientation (k_class_cones); under the loosening a thin cone is merely
// thicker than it could be.  (Dropping every cone with the centroid within
// four 2^-19 margins of a plane left 71 % of the level-10 terrain's receiver
// candidates, behind small triangles seen at a grazing angle, without one:
// k_capture_fast 13.0 ms, with them 12.1.)
// The reference's FP64 test accepts
// only points inside the exact cone, so receivers outside the loosened one
// are skipped without changing a result.

constexpr float kConeK = 4.76837158203125e-07f;  // 2^-21

// Whether the box [lo, hi] may hold a point of the cone.
__device__ __forceinline__ bool cone_meets_box(const float* cone, const float* lo, const float* hi) {
  for (int k = 0; k < 3; ++k) {
    float mx = 0.0f, mag = fabsf(cone[4 * k + 3]) + 1.0f;
    for (int a = 0; a < 3; ++a) {
      mx += fmaxf(cone[4 * k + a] * lo[a], cone[4 * k + a] * hi[a]);
      mag += fabsf(cone[4 * k + a]) * fmaxf(fabsf(lo[a]), fabsf(hi[a]));
    }
    if (mx < cone[4 * k + 3] - 1e-3f * mag) return false;  // slack >> FP32 error of mx
  }
  return true;
}

// Narrows the cell range [x0, x1] of the grid row at (i1, i2) along the other
// two axes to the cells whose box can hold a point inside the cone; an empty
// row gets x0 > x1.  cone[12 + k]: 1 / the row component of plane k's normal.
__device__ __forceinline__ void cone_cells(const float* cone, const RxGrid& g, float inv_cell,
                                           int i1, int i2, int& x0, int& x1) {
  const int ar = g.ax[0], am = g.ax[1], al = g.ax[2];
  const float y0 = g.org[am] + i1 * g.cell, y1 = y0 + g.cell;
  const float z0 = g.org[al] + i2 * g.cell, z1 = z0 + g.cell;
  for (int k = 0; k < 3; ++k) {
    const float nx = cone[4 * k + ar], ny = cone[4 * k + am], nz = cone[4 * k + al],
                off = cone[4 * k + 3];
    // need nx*x >= off - max over the row's band of (ny*y + nz*z)
    const float r = off - fmaxf(ny * y0, ny * y1) - fmaxf(nz * z0, nz * z1);
    const float slack = 1e-3f * g.cell;
    if (nx > 0.0f) {
      const float xl = r * cone[12 + k];  // x >= xl
      if (isfinite(xl)) x0 = max(x0, int(floorf((xl - g.org[ar] - slack) * inv_cell)));
    } else if (nx < 0.0f) {
      const float xh = r * cone[12 + k];  // x <= xh
      if (isfinite(xh)) x1 = min(x1, int(floorf((xh - g.org[ar] + slack) * inv_cell)));
    } else if (r > 0.0f) {
      x1 = x0 - 1;
    }
  }
}

struct AncRec {
  float s[3], S, u[3], len;
  uint32_t idx, pad[3];
};

// A node's segment clipped to the region that can hold a capture of this
// request's receivers, cut into chunks (nchunk = 0: nothing to test).
struct NodeSpan {
  float lo, hi, step, ns;  // ns = |segment start|
  int nchunk, use_cone;
};

// The receivers that can fall inside the node's reception spheres lie within
// rb of its segment (rb bounds the sphere radius (S + |P|) tan(beta), with
// |P| <= (cmax + S tan b) / (1 - tan b) for any capturing point).  All
// ranges are widened well beyond their FP32 rounding.
template <class Node>
__device__ __forceinline__ NodeSpan node_span(const Node& nd, const RxGrid& g, int use_cone) {
  NodeSpan sp{0.0f, -1.0f, 0.0f, 0.0f, 0, use_cone};
  if (g.n <= 0) return sp;
  const float3 s = make_float3(nd.s[0], nd.s[1], nd.s[2]);
  const float3 u = make_float3(nd.u[0], nd.u[1], nd.u[2]);
  const float len = nd.len, S = nd.S;
  const float tanb = g.tanb, cmax = g.cmax;
  const float pmax = __fdividef(cmax + S * tanb, fmaxf(1e-6f, 1.0f - tanb)) * 1.0001f + 1.0f;
  const float su = s.x * u.x + s.y * u.y + s.z * u.z;
  const float ss = s.x * s.x + s.y * s.y + s.z * s.z;
  sp.ns = sqrt_up(ss);
  const float disc = su * su - (ss - pmax * pmax);
  float lo = 0.0f, hi = -1.0f;
  if (disc >= 0.0f) {
    const float sq = sqrt_up(disc);
    lo = fmaxf(0.0f, -su - sq);
    hi = fminf(len, -su + sq);
  }
  const float rbg = (S + pmax) * tanb * 1.0001f + 1e-3f;  // bound over the whole segment
  for (int a = 0; a < 3 && lo <= hi; ++a) {
    const float sa = a == 0 ? s.x : (a == 1 ? s.y : s.z);
    const float ua = a == 0 ? u.x : (a == 1 ? u.y : u.z);
    const float bl = g.bmin[a] - rbg, bh = g.bmax[a] + rbg;
    if (fabsf(ua) < 1e-20f) {
      if (sa < bl || sa > bh) hi = -1.0f;
    } else {
      // slack: 1 mm plus 2^-20 relative, beyond the reciprocal's rounding
      const float ia = __frcp_rn(ua);
      const float t1 = (bl - sa) * ia, t2 = (bh - sa) * ia;
      const float tn = fminf(t1, t2), tf = fmaxf(t1, t2);
      lo = fmaxf(lo, tn - 1e-3f - 9.5367431640625e-07f * fabsf(tn));
      hi = fminf(hi, tf + 1e-3f + 9.5367431640625e-07f * fabsf(tf));
    }
  }
  if (!(lo <= hi)) return sp;
  // chunks about as long as the sphere's radius at the middle of the span: a
  // chunk's receivers come from a radius around it, and shorter ones would
  // read the same receivers again and again (level 2, 3 km of receivers on a
  // line: 12 m chunks under 900 m spheres, 1.8 ms of capture)
  const float r0 = (S + sqrt_up(ss + 2.0f * lo * su + lo * lo)) * tanb;
  const float r1 = (S + sqrt_up(ss + 2.0f * hi * su + hi * hi)) * tanb;
  const float lc = fmaxf(g.chunk_len, 0.5f * (r0 + r1));
  int nchunk = int(ceilf(__fdividef(hi - lo, lc)));
  nchunk = max(1, min(nchunk, 4096));
  sp.lo = lo;
  sp.hi = hi;
  sp.nchunk = nchunk;
  sp.step = __fdividef(hi - lo, float(nchunk));
  return sp;
}

// Chunk ch of a node's span: its parameter range [a, b], the radius rb
// around it that can hold a capture, the reception test's error margin mr,
// and the receiver-grid cell box around it (nrows = 0: nothing to test,
// including a box wholly outside the correction cone).
struct ChunkBox {
  float a, b, rb, mr;
  int c0[3], c1[3];
  int nrows;
};

template <class Node>
__device__ __forceinline__ ChunkBox chunk_box(const Node& nd, const RxGrid& g,
                                              const NodeSpan& sp, int ch, float cmax, float tanb,
                                              bool use_cone, const float* cone) {
  ChunkBox cb;
  const float3 s = make_float3(nd.s[0], nd.s[1], nd.s[2]);
  const float3 u = make_float3(nd.u[0], nd.u[1], nd.u[2]);
  const float S = nd.S;
  cb.a = sp.lo + ch * sp.step;
  cb.b = (ch == sp.nchunk - 1) ? sp.hi : sp.lo + (ch + 1) * sp.step;
  const float pa[3] = {s.x + cb.a * u.x, s.y + cb.a * u.y, s.z + cb.a * u.z};
  const float pb[3] = {s.x + cb.b * u.x, s.y + cb.b * u.y, s.z + cb.b * u.z};
  const float npmax = fmaxf(sqrt_up(pa[0] * pa[0] + pa[1] * pa[1] + pa[2] * pa[2]),
                            sqrt_up(pb[0] * pb[0] + pb[1] * pb[1] + pb[2] * pb[2]));
  cb.mr = kRecK * (sp.ns + cmax + S + npmax + 1.0f);
  // |P| is convex along the chunk: the larger end bounds it
  cb.rb = (S + npmax) * tanb * 1.0002f + g.cell * 0.01f + 2e-3f + cb.mr;
  for (int k = 0; k < 3; ++k) {
    cb.c0[k] = max(0, int(floorf((fminf(pa[k], pb[k]) - cb.rb - g.org[k]) * g.inv_cell)));
    cb.c1[k] = min(g.dim[k] - 1, int(floorf((fmaxf(pa[k], pb[k]) + cb.rb - g.org[k]) * g.inv_cell)));
  }
  int e[3];  // cells along each axis
  for (int k = 0; k < 3; ++k) e[k] = cb.c1[k] - cb.c0[k] + 1;
  cb.nrows = 0;
  if (e[0] > 0 && e[1] > 0 && e[2] > 0)
    cb.nrows = g.ax[0] == 0 ? e[1] * e[2] : (g.ax[0] == 1 ? e[0] * e[2] : e[0] * e[1]);
  if (use_cone && cb.nrows) {  // the chunk's cells all outside the cone: skip it
    float blo[3], bhi[3];
    for (int k = 0; k < 3; ++k) {
      blo[k] = g.org[k] + cb.c0[k] * g.cell;
      bhi[k] = g.org[k] + (cb.c1[k] + 1) * g.cell;
    }
    if (!cone_meets_box(cone, blo, bhi)) cb.nrows = 0;
  }
  return cb;
}

// Next batch of `b` nodes for the calling warp (all lanes get the same base).
__device__ __forceinline__ unsigned long long next_batch(unsigned long long* work, int lane,
                                                         int b) {
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(work, (unsigned long long)b);
  return __shfl_sync(0xffffffffu, base, 0);
}

// The capture stage of solves that count its stages: every capture is counted,
// in the plain order of tests (k_capture_fast serves all others).
__global__ void __launch_bounds__(32 * kCapWarps, 4) k_capture(CaptureArgs A) {
  __shared__ AncRec anc[kCapWarps][kMaxDepth];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  if (A.ctr->overflow & kOvTrace) return;  // this solve will be repeated
  const unsigned long long n_nodes = min(A.ctr->nodes, A.node_cap);
  unsigned long long events = 0, cand = 0, anc_tests = 0;
  unsigned n64 = 0;
  // Nodes are taken B at a time: each lane loads one node's record and forms its
  // span; the warp then works through them from shared memory.
  constexpr int B = kCapBatch;
  __shared__ NodeHot s_nh[kCapWarps][B];
  __shared__ NodeSpan s_sp[kCapWarps][B];   // clipped span and chunking
  __shared__ ChunkBox s_ck[kCapWarps][B];   // the span's first chunk
  // Batches of B nodes are handed out by a work counter, one atomic per warp
  // and batch, so warps that drew short segments take more batches.
  for (unsigned long long base = next_batch(A.work, lane, B); base < n_nodes;
       base = next_batch(A.work, lane, B)) {
    {
      const unsigned long long my = base + lane;
      if (lane < B && my < n_nodes) {
        const NodeHot h = A.nodes[my];
        s_nh[warp][lane] = h;
        const float cmax = A.gb[h.tx].cmax;
        const NodeSpan sp = node_span(h, A.grids[h.tx], 0);
        s_sp[warp][lane] = sp;
        if (sp.nchunk > 0)
          s_ck[warp][lane] = chunk_box(h, A.grids[h.tx], sp, 0, cmax, A.txp[h.tx].tan_beta32,
                                       false, nullptr);
      }
      __syncwarp();
    }
    const int n_here = int(min((unsigned long long)B, n_nodes - base));
    for (int jj = 0; jj < n_here; ++jj) {
      const unsigned long long i = base + jj;
      const NodeHot nd = s_nh[warp][jj];
      const TxParams& P = A.txp[nd.tx];
      const RxGrid& g = A.grids[nd.tx];
      const float3 s = make_float3(nd.s[0], nd.s[1], nd.s[2]);
      const float3 u = make_float3(nd.u[0], nd.u[1], nd.u[2]);
      const float len = nd.len, S = nd.S;
      // Reciprocals for the cell-range arithmetic below.  Every range there is
      // widened by at least 2e-3 m + cell/100, far more than the few ulps a
      // product with a reciprocal differs from the quotient.
      const int ar = g.ax[0], am = g.ax[1], al = g.ax[2];
      const NodeHot& sn = s_nh[warp][jj];  // in shared memory: indexed by axis
      const float sr = sn.s[ar], sm = sn.s[am], sl = sn.s[al];
      const float ur = sn.u[ar], um = sn.u[am], ul = sn.u[al];
      const float inv_um = __frcp_rn(um), inv_ul = __frcp_rn(ul);
      const float inv_cell = g.inv_cell;
      // Stage the ancestor chain: every capture is checked against it.
      int na = 0;
      if (lane == 0) {
        for (uint32_t p = nd.parent; p != 0xFFFFFFFFu && p < A.node_cap && na < kMaxDepth;) {
          const NodeHot a = A.nodes[p];
          AncRec& r = anc[warp][na++];
          r.s[0] = a.s[0]; r.s[1] = a.s[1]; r.s[2] = a.s[2]; r.S = a.S;
          r.u[0] = a.u[0]; r.u[1] = a.u[1]; r.u[2] = a.u[2]; r.len = a.len;
          r.idx = p;
          p = a.parent;
        }
      }
      na = __shfl_sync(FULL, na, 0);
      __syncwarp();
      const NodeSpan sp = s_sp[warp][jj];
      if (sp.nchunk > 0) {
        const float tanb = P.tan_beta32;
        const float cmax = A.gb[nd.tx].cmax;
        const float ns = sp.ns;
        const int nchunk = sp.nchunk;
        // error margins of the FP32 reception test, from per-node bounds
        const float ml = kRecK * (ns + cmax + 1.0f);
        {
          for (int ch = 0; ch < nchunk; ++ch) {
            if (ch > 0) {  // every lane forms the same box
              const ChunkBox next = chunk_box(nd, g, sp, ch, cmax, tanb, false, nullptr);
              __syncwarp();
              if (lane == 0) s_ck[warp][jj] = next;
              __syncwarp();
            }
            const ChunkBox& cb = s_ck[warp][jj];
            const float a = cb.a, b = cb.b, rb = cb.rb, mr = cb.mr;
            const int ny = cb.c1[am] - cb.c0[am] + 1;
            const int nrows = cb.nrows;
            for (int rbase = 0; rbase < nrows; rbase += 32) {
              // this lane's row: the part of the chunk within rb of its band
              int beg = 0, cnt = 0;
              const int ridx = rbase + lane;
              if (ridx < nrows) {
                // one layer of cells (receivers on a plane) needs no division
                const bool flat = cb.c1[al] == cb.c0[al];
                const int im = cb.c0[am] + (flat ? ridx : ridx % ny);
                const int il = cb.c0[al] + (flat ? 0 : ridx / ny);
                const float y0 = g.org[am] + im * g.cell - rb, y1 = g.org[am] + (im + 1) * g.cell + rb;
                const float z0 = g.org[al] + il * g.cell - rb, z1 = g.org[al] + (il + 1) * g.cell + rb;
                float la = a, lb = b;
                bool ok = true;
                if (fabsf(um) > 1e-20f) {
                  const float t1 = (y0 - sm) * inv_um, t2 = (y1 - sm) * inv_um;
                  la = fmaxf(la, fminf(t1, t2));
                  lb = fminf(lb, fmaxf(t1, t2));
                } else if (sm < y0 || sm > y1) {
                  ok = false;
                }
                if (fabsf(ul) > 1e-20f) {
                  const float t1 = (z0 - sl) * inv_ul, t2 = (z1 - sl) * inv_ul;
                  la = fmaxf(la, fminf(t1, t2));
                  lb = fminf(lb, fmaxf(t1, t2));
                } else if (sl < z0 || sl > z1) {
                  ok = false;
                }
                if (ok && la <= lb) {
                  const float xa = sr + la * ur, xb = sr + lb * ur;
                  int x0 = max(cb.c0[ar], int(floorf((fminf(xa, xb) - rb - g.org[ar]) * inv_cell)));
                  int x1 = min(cb.c1[ar], int(floorf((fmaxf(xa, xb) + rb - g.org[ar]) * inv_cell)));
                  if (x0 <= x1) {
                    const int row = (il * g.dim[am] + im) * g.dim[ar];
                    beg = g.cell_start[row + x0];
                    cnt = g.cell_start[row + x1 + 1] - beg;
                  }
                }
              }
              // concatenate the 32 rows' receiver runs
              int incl = cnt;
              for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += v;
              }
              const int total = __shfl_sync(FULL, incl, 31);
              for (int kb = 0; kb < total; kb += 32) {
                const int k = kb + lane;
                // row holding item k: first lane whose inclusive count exceeds k
                int rl = 0;
                for (int step2 = 16; step2; step2 >>= 1) {
                  const int v = __shfl_sync(FULL, incl, rl + step2 - 1);
                  if (v <= k) rl += step2;
                }
                const int rincl = __shfl_sync(FULL, incl, rl);
                const int rcnt = __shfl_sync(FULL, cnt, rl);
                const int rbeg = __shfl_sync(FULL, beg, rl);
                if (k >= total) continue;
                const int j = rbeg + (k - (rincl - rcnt));
                const float4 c4 = g.rx32[j];
                const float3 c = make_float3(c4.x, c4.y, c4.z);
                const float wx = c.x - s.x, wy = c.y - s.y, wz = c.z - s.z;
                const float lam = u.x * wx + u.y * wy + u.z * wz;
                if (ch > 0 && lam < a) continue;            // owned by an earlier chunk
                if (ch < nchunk - 1 && lam >= b) continue;  // owned by a later chunk
                const int gi = __float_as_int(c4.w);
                const double* c64 = A.rx + 3 * size_t(gi);
                ++cand;
                int v;
                if (lam < a || lam > b) {
                  // outside the chunk's own range: full-margin test
                  v = reception32(s, u, len, S, c, tanb);
                } else if (lam < -ml) {
                  v = 0;
                } else if (lam <= ml) {
                  v = -1;
                } else {
                  const float lcl = fminf(lam, len);
                  const float px = s.x + lcl * u.x, py = s.y + lcl * u.y, pz = s.z + lcl * u.z;
                  const float np = sqrt_up(px * px + py * py + pz * pz);
                  const float ex = c.x - px, ey = c.y - py, ez = c.z - pz;
                  const float d2 = ex * ex + ey * ey + ez * ez;
                  const float rad = (S + np) * tanb;
                  const float rh = rad + mr, rl2 = rad - mr;
                  v = d2 > rh * rh ? 0 : ((rl2 > 0.0f && d2 < rl2 * rl2) ? 1 : -1);
                }
                if (v < 0) {
                  ++n64;
                  v = capture_exact(A.nodes_cold, uint32_t(i), c64, P.tan_beta);
                }
                if (!v) continue;
                // RayCapture deletes a captured node's subtree, so an ancestor
                // capturing the same receiver suppresses this one.
                auto suppressed = [&]() {
                  for (int q = 0; q < na; ++q) {
                    const AncRec& r = anc[warp][q];
                    ++anc_tests;
                    int w = reception32(make_float3(r.s[0], r.s[1], r.s[2]),
                                        make_float3(r.u[0], r.u[1], r.u[2]), r.len, r.S, c, tanb);
                    if (w < 0) {
                      ++n64;
                      w = capture_exact(A.nodes_cold, r.idx, c64, P.tan_beta);
                    }
                    if (w) return true;
                  }
                  return false;
                };
                if (suppressed()) continue;
                ++events;
                const bool ok = is_root_class(nd.cls)
                                    ? A.direct_ok[gi] != 0
                                    : correct_event(A.sc, A.cls_info, nd.cls, c, c64, n64);
                if (!ok) continue;
                const unsigned long long kk = atomicAdd(&A.ctr->corrected, 1ull);
                if (kk < A.corr_cap)
                  A.corr_list[kk] = Corrected{uint32_t(gi), nd.cls,
                                              (unsigned long long)nd.launch << kHeapBits | nd.heap};
                else
                  atomicOr(&A.ctr->overflow, kOvCorr);
              }
            }
          }
        }
      }
      __syncwarp();
    }
    __syncwarp();  // the next batch overwrites the staged records
  }
  for (int o = 16; o; o >>= 1) {
    events += __shfl_xor_sync(FULL, events, o);
    cand += __shfl_xor_sync(FULL, cand, o);
    anc_tests += __shfl_xor_sync(FULL, anc_tests, o);
    n64 += __shfl_xor_sync(FULL, n64, o);
  }
  if (lane == 0) {
    if (events) atomicAdd(&A.ctr->events, events);
    if (cand) atomicAdd(&A.ctr->cand, cand);
    if (anc_tests) atomicAdd(&A.ctr->anc, anc_tests);
    if (n64) atomicAdd(&A.ctr->fp64_capture, (unsigned long long)n64);
  }
}

// Items of a work counter handed to a warp, a window at a time: every warp of
// the grid asks the same counter, which serves an atomic in about 0.65 ns, so
// a warp takes a part of what was left when it last asked (whole batches of 32,
// or `smallest`, a caller's smaller batch) and the windows shrink towards the
// end, where an uneven last one would leave warps waiting.  At most 64 items:
// costly nodes lie next to each other, and a warp that drew 256 of them held up
// the level-10 terrain's capture (12.2 ms; 128: 8.0, 64 and 32: 7.1).
struct WorkWindow {
  unsigned long long* counter;
  long long next, end, n;  // the window's rest; items in all
  float share;
  int smallest;
  __device__ __forceinline__ WorkWindow(unsigned long long* c, long long items, int least)
      : counter(c), next(0), end(0), n(items), smallest(least) {
    share = 0.125f / (32.0f * float(gridDim.x) * float(blockDim.x >> 5));
  }
  // Fetches a window if the last one is used up; false when no item is left
  // (the same on every lane; the whole warp calls).
  __device__ __forceinline__ bool refill() {
    if (next < end) return true;
    if (next >= n && end > 0) return false;
    const int size = min(64, max(smallest, 32 * int(float(n - next) * share)));
    unsigned long long base = 0;
    if (lane_id() == 0) base = atomicAdd(counter, (unsigned long long)size);
    next = (long long)__shfl_sync(0xffffffffu, base, 0);
    end = min(next + size, n);
    return next < n;
  }
};

// ---- fast path, flattened over the nodes of a batch ------------------------
//
// Receivers are found as k_capture finds them (chunks, cell boxes, margins), but
// the correction's first test comes before the reception test: the line from the
// class's image source to the receiver must cross the class's last triangle, which
// an FP32 filter refutes for ~99.9 % of receivers, and the loosened cone for whole
// rows of cells.  The (node, receiver) pairs left go to k_capture_finish.
// The warp stages B nodes (one lane each: node record, class record, last
// triangle, loosened correction cone, clipped span), then works through the
// whole batch at three flattened levels instead of node by node: the batch's
// (node, chunk) items with one lane per item (cell box, cone test), those
// items' rows of cells with one lane per row (the row's receiver run), and
// those rows' receivers with one lane per receiver (correction prefilter,
// FP32 reception test).  Each level is an inclusive prefix count over the
// lanes; an item finds its parent by a binary search over the counts.  A
// node with a handful of candidates (about six per node at level 9) thus no
// longer holds all 32 lanes through its own chunk, row and receiver passes.

__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += x;
  }
  return v;
}

// The first lane whose inclusive count exceeds k (0 <= k < the total).
__device__ __forceinline__ int warp_find(int incl, int k) {
  int rl = 0;
  for (int step = 16; step; step >>= 1) {
    const int v = __shfl_sync(0xffffffffu, incl, rl + step - 1);
    if (v <= k) rl += step;
  }
  return rl;
}

constexpr int kFastB = 32;  // nodes staged per warp and batch (one per lane)

// What the fast path keeps of a node in shared memory.
struct StagedNode {
  float s[3], S, u[3], len;
  uint32_t cls, grid;  // grid: its receivers' grid (CaptureArgs::grids)
};

// The correction prefilter of a node's class as a candidate needs it: the image
// source, the last triangle's edges, tri_from's terms and the margins' factors
// (tri_filter's, the ones that depend on the class alone multiplied
// beforehand).  Five 16-byte loads a candidate instead of 23 words of two
// records, and the cones an odd number of words apart: the kernel is bound by
// issue and L1 (level-9 canyon 5.05 -> 4.89 ms, 24 requests 2.53 -> 2.45, level-10
// terrain 5.25 -> 5.15).  Seven blocks an SM, with 48 pairs gathered instead of
// 64 to fit, took 5.01 ms in the canyon and 0.155 for 0.141 ms on a line of
// receivers.
struct __align__(16) LineFilter {
  float img[3], W, e1[3], ka, e2[3], ku, s[3], kv, q[3], kw;
};
__device__ __forceinline__ LineFilter line_filter(const ClassCap& c, const Tri32& T) {
  LineFilter L;
  const float ns = c.F[7];
  for (int a = 0; a < 3; ++a) {
    L.img[a] = c.img[a];
    L.e1[a] = T.e1[a];
    L.e2[a] = T.e2[a];
    L.s[a] = c.F[a];
    L.q[a] = c.F[3 + a];
  }
  L.W = c.F[6];
  L.ka = kCorrK * T.ne1 * T.ne2;
  L.ku = kCorrK * ns * T.ne2;
  L.kv = kCorrK * ns * T.ne1;
  L.kw = kCorrK * ns * T.ne1 * T.ne2;
  return L;
}
// tri_filter of the line from the image source to c, without its bound on t.
__device__ __forceinline__ bool line_may_cross(const LineFilter& L, const float3& c) {
  const float dx = c.x - L.img[0], dy = c.y - L.img[1], dz = c.z - L.img[2];
  const float nd = sqrt_up(dx * dx + dy * dy + dz * dz);
  const float hx = dy * L.e2[2] - dz * L.e2[1];
  const float hy = dz * L.e2[0] - dx * L.e2[2];
  const float hz = dx * L.e2[1] - dy * L.e2[0];
  const float a = L.e1[0] * hx + L.e1[1] * hy + L.e1[2] * hz;
  const float sg = copysignf(1.0f, a), A = fabsf(a);
  const float U = sg * (L.s[0] * hx + L.s[1] * hy + L.s[2] * hz);
  const float V = sg * (dx * L.q[0] + dy * L.q[1] + dz * L.q[2]);
  const float W = sg * L.W;
  const float ea = L.ka * nd, eU = L.ku * nd, eV = L.kv * nd;
  const bool parallel = A <= kEps32 + ea;  // the FP64 test decides
  return parallel || (U >= -eU && V >= -eV && U <= A + ea + eU && U + V <= A + ea + eU + eV &&
                      W + L.kw > (kEps32 * 0.5f) * (A - ea));
}

// Pairs for k_capture_finish, gathered per warp so that one atomic on the pair
// counter (which every warp of the grid adds to) serves more than 32 of them.
constexpr int kPairBuf = 64;
__device__ __forceinline__ void flush_pairs(const CaptureArgs& A, const uint2* buf, int& n,
                                            int lane) {
  __syncwarp();
  unsigned long long base = 0;
  if (lane == 0 && n) base = atomicAdd(&A.ctr->pairs, (unsigned long long)n);
  base = __shfl_sync(0xffffffffu, base, 0);
  if (lane == 0 && base + n > A.pair_cap) atomicOr(&A.ctr->overflow, kOvPairs);
  for (int j = lane; j < n; j += 32)
    if (base + j < A.pair_cap) A.pairs[base + j] = buf[j];
  n = 0;
  __syncwarp();
}

// Resident blocks per SM (register budget 65536 / (128 x this)).
#ifndef SBR_CAP_BLOCKS
#define SBR_CAP_BLOCKS 6
#endif
__global__ void __launch_bounds__(32 * kCapWarps, SBR_CAP_BLOCKS) k_capture_fast(CaptureArgs A) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  if (A.ctr->overflow & kOvTrace) return;  // this solve will be repeated
  const unsigned long long n_nodes = min(A.ctr->nodes, A.node_cap);
  unsigned long long cand = 0;
  constexpr int B = kFastB;
  __shared__ StagedNode s_nh[kCapWarps][B];
  __shared__ uint2 s_pr[kCapWarps][kPairBuf];
  int n_pr = 0;  // pairs gathered (the same on every lane)
  __shared__ LineFilter s_lf[kCapWarps][B];  // the class's correction prefilter
  __shared__ float s_cn[kCapWarps][B][15];   // loosened correction cone (odd: no bank conflicts)
  __shared__ NodeSpan s_sp[kCapWarps][B];    // clipped span and chunking
  __shared__ ChunkBox s_ck[kCapWarps][32];  // the current 32 (node, chunk) items
  // fewer nodes than the grid's lanes: fewer nodes per warp, so that each
  // node's chunks still find a warp of their own (184 nodes of up to 250
  // chunks on 6 warps took 1.9 ms)
  const long long warps = (long long)gridDim.x * kCapWarps;
  const int batch = int(min((long long)B, max(1ll, ((long long)n_nodes + warps - 1) / warps)));
  for (WorkWindow work(A.work, (long long)n_nodes, batch); work.refill();) {
    const unsigned long long base = work.next;
    const int n_here = int(min((long long)batch, work.end - work.next));
    work.next += n_here;
    int nck = 0;  // chunks of this lane's node
    {
      const unsigned long long my = base + lane;
      if (lane < n_here) {
        const NodeHot h = A.nodes[my];
        const uint32_t gi = h.tx + (is_root_class(h.cls) ? A.n_tx : 0);
        s_nh[warp][lane] = StagedNode{{h.s[0], h.s[1], h.s[2]}, h.S, {h.u[0], h.u[1], h.u[2]},
                                      h.len, h.cls, gi};
        const RxGrid& g = A.grids[gi];
        const float cmax = g.cmax;
        const int ar = g.ax[0];
        int cone_ok = 0;
        if (!is_root_class(h.cls)) {
          const ClassCap c = A.cls_cap[h.cls];
          s_lf[warp][lane] = line_filter(c, A.sc.corr32[c.tpos]);
          // the cone's planes loosened by 2 m, m = 2^-21 |n| (cmax + |img| + |T| + 1)
          float* cn = s_cn[warp][lane];
          cone_ok = 1;
          for (int k = 0; k < 3; ++k) {
            const float m = kConeK * (c.nn[k] * cmax + c.w[k]);
            cone_ok &= (c.gc[k] > 0.0f && isfinite(m)) ? 1 : 0;
            cn[4 * k + 0] = c.n[k][0];
            cn[4 * k + 1] = c.n[k][1];
            cn[4 * k + 2] = c.n[k][2];
            cn[4 * k + 3] = c.n[k][3] - 2.0f * m;
            cn[12 + k] = 1.0f / (ar == 0 ? c.n[k][0] : (ar == 1 ? c.n[k][1] : c.n[k][2]));
          }
        }
        const NodeSpan sp = node_span(h, g, cone_ok);
        s_sp[warp][lane] = sp;
        nck = sp.nchunk;
      }
      __syncwarp();
    }
    const int ck_incl = warp_incl_scan(nck, lane);
    const int n_ck = __shfl_sync(FULL, ck_incl, 31);
    for (int k0 = 0; k0 < n_ck; k0 += 32) {
      // level 1: one lane per (node, chunk) item
      const int k = k0 + lane;
      const int j = warp_find(ck_incl, min(k, n_ck - 1));
      const int j_incl = __shfl_sync(FULL, ck_incl, j), j_n = __shfl_sync(FULL, nck, j);
      int nrows = 0;
      if (k < n_ck) {
        const int ch = k - (j_incl - j_n);
        const StagedNode& nd = s_nh[warp][j];
        const NodeSpan& sp = s_sp[warp][j];
        const RxGrid& g = A.grids[nd.grid];
        const ChunkBox cb = chunk_box(nd, g, sp, ch, g.cmax, g.tanb, sp.use_cone != 0,
                                      s_cn[warp][j]);
        nrows = cb.nrows;
        s_ck[warp][lane] = cb;
        s_ck[warp][lane].nrows = j | ch << 8;  // node (batch index), chunk
      }
      __syncwarp();
      const int r_incl = warp_incl_scan(nrows, lane);
      const int n_r = __shfl_sync(FULL, r_incl, 31);
      for (int r0 = 0; r0 < n_r; r0 += 32) {
        // level 2: one lane per row of cells: the part of its chunk within rb
        // of the row's y/z band, cut to the cone, as a run of receivers
        const int r = r0 + lane;
        const int ci = warp_find(r_incl, min(r, n_r - 1));
        const int ci_incl = __shfl_sync(FULL, r_incl, ci), ci_n = __shfl_sync(FULL, nrows, ci);
        int beg = 0, cnt = 0;
        if (r < n_r) {
          const int ridx = r - (ci_incl - ci_n);
          const ChunkBox& cb = s_ck[warp][ci];
          const int jn = cb.nrows & 0xff;
          const StagedNode& nd = s_nh[warp][jn];
          const RxGrid& g = A.grids[nd.grid];
          const int ar = g.ax[0], am = g.ax[1], al = g.ax[2];
          const float sr = nd.s[ar], sm = nd.s[am], sl = nd.s[al];
          const float ur = nd.u[ar], um = nd.u[am], ul = nd.u[al];
          // Reciprocals for the cell-range arithmetic: every range is widened
          // by at least 2e-3 m + cell/100, far more than the few ulps a product
          // with a reciprocal differs from the quotient.
          const float inv_um = __frcp_rn(um), inv_ul = __frcp_rn(ul);
          const float rb = cb.rb;
          const int ny = cb.c1[am] - cb.c0[am] + 1;
          // one layer of cells (receivers on a plane) needs no division
          const bool flat = cb.c1[al] == cb.c0[al];
          const int im = cb.c0[am] + (flat ? ridx : ridx % ny);
          const int il = cb.c0[al] + (flat ? 0 : ridx / ny);
          const float y0 = g.org[am] + im * g.cell - rb, y1 = g.org[am] + (im + 1) * g.cell + rb;
          const float z0 = g.org[al] + il * g.cell - rb, z1 = g.org[al] + (il + 1) * g.cell + rb;
          float la = cb.a, lb = cb.b;
          bool ok = true;
          if (fabsf(um) > 1e-20f) {
            const float t1 = (y0 - sm) * inv_um, t2 = (y1 - sm) * inv_um;
            la = fmaxf(la, fminf(t1, t2));
            lb = fminf(lb, fmaxf(t1, t2));
          } else if (sm < y0 || sm > y1) {
            ok = false;
          }
          if (fabsf(ul) > 1e-20f) {
            const float t1 = (z0 - sl) * inv_ul, t2 = (z1 - sl) * inv_ul;
            la = fmaxf(la, fminf(t1, t2));
            lb = fminf(lb, fmaxf(t1, t2));
          } else if (sl < z0 || sl > z1) {
            ok = false;
          }
          if (ok && la <= lb) {
            const float inv_cell = g.inv_cell;
            const float xa = sr + la * ur, xb = sr + lb * ur;
            int x0 = max(cb.c0[ar], int(floorf((fminf(xa, xb) - rb - g.org[ar]) * inv_cell)));
            int x1 = min(cb.c1[ar], int(floorf((fmaxf(xa, xb) + rb - g.org[ar]) * inv_cell)));
            if (s_sp[warp][jn].use_cone && x0 <= x1)
              cone_cells(s_cn[warp][jn], g, inv_cell, im, il, x0, x1);
            if (x0 <= x1) {
              const int row = (il * g.dim[am] + im) * g.dim[ar];
              beg = g.cell_start[row + x0];
              cnt = g.cell_start[row + x1 + 1] - beg;
            }
          }
        }
        const int c_incl = warp_incl_scan(cnt, lane);
        const int n_c = __shfl_sync(FULL, c_incl, 31);
        for (int q0 = 0; q0 < n_c; q0 += 32) {
          // level 3: one lane per candidate receiver
          const int q = q0 + lane;
          const int rl = warp_find(c_incl, min(q, n_c - 1));
          const int rincl = __shfl_sync(FULL, c_incl, rl);
          const int rcnt = __shfl_sync(FULL, cnt, rl);
          const int rbeg = __shfl_sync(FULL, beg, rl);
          const int rci = __shfl_sync(FULL, ci, rl);
          uint2 pair = make_uint2(0, 0);
          auto passes = [&]() -> bool {
            if (q >= n_c) return false;
            const int ckn = s_ck[warp][rci].nrows;
            const int jn = ckn & 0xff, ch = ckn >> 8;
            const StagedNode& nd = s_nh[warp][jn];
            const NodeSpan& sp = s_sp[warp][jn];
            const float a = s_ck[warp][rci].a, b = s_ck[warp][rci].b, mr = s_ck[warp][rci].mr;
            const RxGrid& g = A.grids[nd.grid];
            const float3 s = make_float3(nd.s[0], nd.s[1], nd.s[2]);
            const float3 u = make_float3(nd.u[0], nd.u[1], nd.u[2]);
            const float4 c4 = g.rx32[rbeg + (q - (rincl - rcnt))];
            const float3 c = make_float3(c4.x, c4.y, c4.z);
            const float wx = c.x - s.x, wy = c.y - s.y, wz = c.z - s.z;
            const float lam = u.x * wx + u.y * wy + u.z * wz;
            if (ch > 0 && lam < a) return false;                 // owned by an earlier chunk
            if (ch < sp.nchunk - 1 && lam >= b) return false;    // owned by a later chunk
            const int gi = __float_as_int(c4.w);
            ++cand;
            // MultiPathCorrection's last step must cross the class's last
            // triangle: FP32 filter from the image source towards the receiver
            if (!is_root_class(nd.cls) && !line_may_cross(s_lf[warp][jn], c)) return false;
            const float tanb = g.tanb;
            const float len = nd.len, S = nd.S;
            int v;
            if (lam < a || lam > b) {
              // outside the chunk's own range: full-margin test
              v = reception32(s, u, len, S, c, tanb);
            } else {
              const float ml = kRecK * (sp.ns + g.cmax + 1.0f);
              if (lam < -ml) {
                v = 0;
              } else if (lam <= ml) {
                v = -1;
              } else {
                const float lcl = fminf(lam, len);
                const float px = s.x + lcl * u.x, py = s.y + lcl * u.y, pz = s.z + lcl * u.z;
                const float np = sqrt_up(px * px + py * py + pz * pz);
                const float ex = c.x - px, ey = c.y - py, ez = c.z - pz;
                const float d2 = ex * ex + ey * ey + ez * ez;
                const float rad = (S + np) * tanb;
                const float rh = rad + mr, rl2 = rad - mr;
                v = d2 > rh * rh ? 0 : ((rl2 > 0.0f && d2 < rl2 * rl2) ? 1 : -1);
              }
            }
            if (v == 0) return false;
            pair = make_uint2(uint32_t(base + jn), uint32_t(gi) | (v < 0 ? 0x80000000u : 0u));
            return true;
          };
          // the exact reception test, image correction and ancestor
          // suppression run densely in k_capture_finish
          const bool pass = passes();
          const unsigned pm = __ballot_sync(FULL, pass);
          if (pass) s_pr[warp][n_pr + __popc(pm & ((1u << lane) - 1u))] = pair;
          n_pr += __popc(pm);
          if (n_pr > kPairBuf - 32) flush_pairs(A, s_pr[warp], n_pr, lane);
        }
      }
      __syncwarp();  // the next group of items overwrites s_ck
    }
    __syncwarp();  // the next batch overwrites the staged records
  }
  flush_pairs(A, s_pr[warp], n_pr, lane);
  for (int o = 16; o; o >>= 1) cand += __shfl_xor_sync(FULL, cand, o);
  if (lane == 0 && cand) atomicAdd(&A.ctr->cand, cand);
}

// The FP64 part of capture for the pairs k_capture could not settle in FP32:
// the exact reception test where the FP32 one was unsure, then image
// correction (MultiPathCorrection / DirectPathCorrection) and suppression by
// an ancestor capturing the same receiver (RTSolver.cpp:277-284), as in
// k_capture.  One thread per pair keeps the FP64 pipe busy with full warps.
__global__ void __launch_bounds__(128) k_capture_finish(CaptureArgs A) {
  if (A.ctr->overflow & (kOvTrace | kOvPairs)) return;  // this solve will be repeated
  const unsigned long long n = min(A.ctr->pairs, A.pair_cap);
  unsigned n64 = 0;
  unsigned long long anc_tests = 0;
  for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < n;
       k += (unsigned long long)gridDim.x * blockDim.x) {
    const uint2 pr = A.pairs[k];
    const uint32_t i = pr.x;
    const int gi = int(pr.y & 0x7fffffffu);
    const NodeHot nd = A.nodes[i];
    const TxParams& P = A.txp[nd.tx];
    const double* c64 = A.rx + 3 * size_t(gi);
    if (pr.y >> 31) {
      ++n64;
      if (!capture_exact(A.nodes_cold, i, c64, P.tan_beta)) continue;
    }
    const float3 c = make_float3(float(c64[0]), float(c64[1]), float(c64[2]));
    bool ok;
    if (is_root_class(nd.cls)) {
      ok = A.direct_ok[gi] != 0;
    } else {
      // The correction depends only on the class and the receiver, and the
      // reception spheres are wide (beta = acos(-1/sqrt 5) / (3 (L + 1))), so
      // many nodes of one class capture the same receiver: the outcome is
      // kept per (class, receiver) and each is computed about once.
      const unsigned long long key = (unsigned long long)nd.cls << 32 | uint32_t(gi);
      bool fresh = false;
      const uint32_t slot = ht_claim(A.corr_cache, key, 32, fresh);
      unsigned char known = 0;
      if (slot != 0xFFFFFFFFu && !fresh)
        known = *reinterpret_cast<volatile unsigned char*>(&A.corr_val[slot]);
      if (known) {
        ok = known == 2;
      } else {
        ok = correct_event(A.sc, A.cls_info, nd.cls, c, c64, n64);
        if (slot != 0xFFFFFFFFu) {
          A.corr_val[slot] = ok ? 2 : 1;
          if (fresh) atomicAdd(&A.ctr->used_cc, 1ull);
        }
      }
    }
    if (!ok) continue;
    const float tanb = P.tan_beta32;
    bool sup = false;
    for (uint32_t p = nd.parent; p != 0xFFFFFFFFu && p < A.node_cap;) {
      const NodeHot a = A.nodes[p];
      ++anc_tests;
      int w = reception32(make_float3(a.s[0], a.s[1], a.s[2]), make_float3(a.u[0], a.u[1], a.u[2]),
                          a.len, a.S, c, tanb);
      if (w < 0) {
        ++n64;
        w = capture_exact(A.nodes_cold, p, c64, P.tan_beta);
      }
      if (w) {
        sup = true;
        break;
      }
      p = a.parent;
    }
    if (sup) continue;
    const unsigned long long kk = atomicAdd(&A.ctr->corrected, 1ull);
    if (kk < A.corr_cap)
      A.corr_list[kk] =
          Corrected{uint32_t(gi), nd.cls, (unsigned long long)nd.launch << kHeapBits | nd.heap};
    else
      atomicOr(&A.ctr->overflow, kOvCorr);
  }
  for (int o = 16; o; o >>= 1) {
    anc_tests += __shfl_xor_sync(0xffffffffu, anc_tests, o);
    n64 += __shfl_xor_sync(0xffffffffu, n64, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (anc_tests) atomicAdd(&A.ctr->anc, anc_tests);
    if (n64) atomicAdd(&A.ctr->fp64_capture, (unsigned long long)n64);
  }
}

}  // namespace sbr
