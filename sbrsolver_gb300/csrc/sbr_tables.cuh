// The scene's triangle and node tables on the device, formed there from the
// host's records: by depth-first rank (Tri64, Tri32 and their ids), by mesh
// position (CorrTri and its FP32 copy), and the reference BVH's nodes.
//
// The records pass through a buffer of kTableChunk triangles; each thread takes
// one record and writes its rows of the tables.  Bound by the host's copy into
// the buffer (over 100 GB/s).  For 580k triangles the tables' part of scene
// creation took 34 ms when the host's cores formed them, mostly the first touch
// of 300 MB of vectors that were copied and dropped; now 9.7, of which 6 go to
// the four-wide search nodes, still formed on the host.
#pragma once

#include <cuda_runtime.h>

#include "sbr_device.h"
#include "sbr_host.h"
#include "sbr_soft64.cuh"

namespace sbr {
namespace tables {

constexpr int kTableChunk = 1 << 16;

__global__ void __launch_bounds__(256) k_invert(const int* p, int n, int* inverse) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    inverse[p[i]] = i;
}

__device__ __forceinline__ void edges(const HostTri& t, double* e1, double* e2) {
  for (int a = 0; a < 3; ++a) {
    e1[a] = x64::sub(t.v2[a], t.v1[a]);
    e2[a] = x64::sub(t.v3[a], t.v1[a]);
  }
}

__device__ __forceinline__ Tri32 filter_copy(const double* v1, const double* e1, const double* e2) {
  Tri32 f;
  for (int a = 0; a < 3; ++a) {
    f.v1[a] = float(v1[a]);
    f.e1[a] = float(e1[a]);
    f.e2[a] = float(e2[a]);
  }
  // lengths, a little above
  f.nv1 = __fmul_rn(float(x64::norm(v1)), 1.0001f);
  f.ne1 = __fmul_rn(float(x64::norm(e1)), 1.0001f);
  f.ne2 = __fmul_rn(float(x64::norm(e2)), 1.0001f);
  return f;
}

// found[0]: a triangle outside soft64's range; found[1]: the number of coplanar
// ids (their largest + 1).
__global__ void __launch_bounds__(256)
    k_rank_tables(const HostTri* t, int first, int n, const int* rank_of, Tri64* t64, Tri32* t32,
                  int* cop, int* rank_to_id, int* found) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const HostTri& s = t[i];
    const int r = rank_of[first + i];
    double e1[3], e2[3];
    edges(s, e1, e2);
    Tri64& d = t64[r];
    bool ok = true;
    for (int a = 0; a < 3; ++a) {
      d.v1[a] = s.v1[a];
      d.e1[a] = e1[a];
      d.e2[a] = e2[a];
      d.n[a] = s.n[a];
      ok &= soft64::safe(s.v1[a]) && soft64::safe(e1[a]) && soft64::safe(e2[a]) &&
            soft64::safe(s.n[a]);
    }
    d.id = s.id;
    d.cop = s.cop;
    d.mat = s.mat;
    d.node = -1;  // its leaf: k_ref_nodes
    t32[r] = filter_copy(s.v1, e1, e2);
    cop[r] = s.cop;
    rank_to_id[r] = s.id;
    if (!ok) found[0] = 1;
    const unsigned m = __activemask();
    const int n_cop = __reduce_max_sync(m, s.cop + 1);
    if ((threadIdx.x & 31) == __ffs(m) - 1) atomicMax(&found[1], n_cop);
  }
}

__global__ void __launch_bounds__(256)
    k_mesh_tables(const HostTri* t, int first, int n, const int* position_of, CorrTri* corr,
                  Tri32* corr32) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const HostTri& s = t[i];
    const int p = position_of[first + i];
    double e1[3], e2[3];
    edges(s, e1, e2);
    CorrTri& d = corr[p];
    for (int a = 0; a < 3; ++a) {
      d.v1[a] = s.v1[a];
      d.e1[a] = e1[a];
      d.e2[a] = e2[a];
      d.n[a] = s.n[a];
    }
    for (int a = 0; a < 9; ++a) d.cs[a] = s.cs[a];
    d.mat = s.mat;
    d.pad = 0;
    corr32[p] = filter_copy(s.v1, e1, e2);
  }
}

__global__ void __launch_bounds__(256)
    k_ref_nodes(const HostNode* h, int first, int n, RefNode* ref, Tri64* t64) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const HostNode& s = h[i];
    RefNode r;
    r.flat = 0;
    for (int a = 0; a < 6; ++a) {
      r.bb[a] = s.bb[a];
      r.fb[a] = float(s.bb[a]);
    }
    for (int a = 0; a < 3; ++a) {
      // boxes of float vertices are floats; a non-float bound (empty box
      // sentinel) disables the FP32 decision for that node
      if (double(r.fb[a]) != s.bb[a] || double(r.fb[3 + a]) != s.bb[3 + a]) r.flat |= 8;
      if (s.bb[a] == s.bb[3 + a]) r.flat |= 1 << a;
    }
    r.c0 = s.c0;
    r.c1 = s.c1;
    r.first = s.first;
    r.count = s.count;
    r.parent = s.parent;
    ref[first + i] = r;
    if (s.c0 < 0)
      for (int k = s.first; k < s.first + s.count; ++k) t64[k].node = first + i;
  }
}

__global__ void __launch_bounds__(256) k_node32(const RefNode* ref, int n, Node32* node) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    Node32 m = {};
    if (ref[i].c0 >= 0) {
      for (int k = 0; k < 2; ++k) {
        const int c = k == 0 ? ref[i].c0 : ref[i].c1;
        float* lo = k == 0 ? m.lo0 : m.lo1;
        float* hi = k == 0 ? m.hi0 : m.hi1;
        for (int a = 0; a < 3; ++a) {
          // outward rounding keeps the FP32 box around the FP64 one
          lo[a] = nextafterf(ref[c].fb[a], -INFINITY);
          hi[a] = nextafterf(ref[c].fb[3 + a], INFINITY);
        }
        m.child[k] = ref[c].c0 >= 0 ? c : ~c;
      }
    }
    node[i] = m;
  }
}

__global__ void __launch_bounds__(256)
    k_search_tris(const Tri32* t32, const int* order, int n, Tri32* out) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
    out[j] = t32[order[j]];
}

}  // namespace tables
}  // namespace sbr
