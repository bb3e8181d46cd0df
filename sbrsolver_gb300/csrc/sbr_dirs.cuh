// Launch directions on the device: the subdivided icosahedron of
// icosphere() (sbr_host.cpp; RTSolver.cpp:742-803), same vertices in the same
// order, bit for bit.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "sbr_device.h"
#include "sbr_grid.cuh"

namespace sbr {
namespace dirs {

// The mesh is held as half-edges: half-edge 3 t + k runs from corner k of face
// t to corner k + 1, `from` holds its start vertex, `mate` the half-edge of the
// face across it, which runs the other way.  A midpoint is numbered where its
// edge comes first in face order, so by a scan over "before my mate", and both
// tables of the next level follow from the old ones without a search:
//   face t becomes (corner k, m_k, m_k+2) as 4 t + k, k = 0..2, and
//   (m_0, m_1, m_2) as 4 t + 3, m_k being the midpoint of half-edge k.
struct Mesh {
  const int *from, *mate;
};

__global__ void __launch_bounds__(256) k_edge_first(const int* mate, int n, int* first) {
  for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < n; h += gridDim.x * blockDim.x)
    first[h] = h < mate[h];
}

// One thread per half-edge: the midpoint where it is numbered here, and this
// half-edge's part of the next level's tables (none after the last level).
// Bound by the FP64 pipe (three divisions and a square root a vertex, 76
// cycles a warp instruction).  With the host's hash table of edges the first
// solve of a scene took 3.9 ms at level 6, 73 at level 8 and 2,269 at level 10;
// now 0.35, 0.85 and 4.6.
__global__ void __launch_bounds__(256)
    k_edge_split(Mesh m, const int* rank, int n, int n_vert, double* v, int* from, int* mate) {
  for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < n; h += gridDim.x * blockDim.x) {
    const int t = h / 3, k = h % 3, k1 = (k + 1) % 3, k2 = (k + 2) % 3;
    const int o = m.mate[h], a = m.from[h];
    const int mid = n_vert + rank[min(h, o)];
    if (h < o) {
      const int b = m.from[3 * t + k1];
      double s[3], r[3];
      for (int x = 0; x < 3; ++x) s[x] = x64::add(v[3 * size_t(a) + x], v[3 * size_t(b) + x]);
      x64::normalize(s, r);
      for (int x = 0; x < 3; ++x) v[3 * size_t(mid) + x] = r[x];
    }
    if (!from) continue;
    const int ot = o / 3, ok = o % 3;
    const int corner = 3 * (4 * t + k), next = 3 * (4 * t + k1), inner = 3 * (4 * t + 3);
    from[corner] = a;
    from[corner + 1] = mid;
    from[next + 2] = mid;
    from[inner + k] = mid;
    mate[corner] = 3 * (4 * ot + (ok + 1) % 3) + 2;  // first half, the mate's second
    mate[next + 2] = 3 * (4 * ot + ok);              // second half, the mate's first
    mate[corner + 1] = inner + k2;
    mate[inner + k2] = corner + 1;
  }
}

// The directions: each vertex normalised once more.
__global__ void __launch_bounds__(256) k_unit(double* v, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double s[3], r[3];
    for (int x = 0; x < 3; ++x) s[x] = v[3 * size_t(i) + x];
    x64::normalize(s, r);
    for (int x = 0; x < 3; ++x) v[3 * size_t(i) + x] = r[x];
  }
}

// Scratch of subdivide: two levels' tables, the last one's ranks, a scan's
// sums (0.9 bytes a byte of directions).
inline size_t last_edges(int level) { return level > 0 ? size_t(60) << (2 * (level - 1)) : 0; }
inline size_t scratch_ints(int level) {
  const size_t n = last_edges(level);
  return 3 * n + 1 + 2 * std::max<size_t>(60, n / 4) + n / kScanTile + 1;
}

// The directions of a level into v (10 * 4^level + 2 of them), from the
// icosahedron's vertices and half-edges on the host.
inline void subdivide(int level, const double* v0, const int* from0, const int* mate0, double* v,
                      int* scratch, int sms, cudaStream_t st) {
  const size_t n_last = last_edges(level);
  int* const rank = scratch;
  int* const sums = rank + n_last + 1;
  int* const big = sums + n_last / kScanTile + 1;  // from, mate of the last level
  int* const small = big + 2 * n_last;             // of the one before
  cudaMemcpyAsync(v, v0, 36 * sizeof(double), cudaMemcpyHostToDevice, st);
  int n_vert = 12, n = 60;
  for (int l = 0; l < level; ++l, n *= 4) {
    const bool last = l + 1 == level, odd = (level - 1 - l) & 1;
    int* const cur = odd ? small : big;
    int* const next = odd ? big : small;
    if (l == 0) {
      cudaMemcpyAsync(cur, from0, 60 * sizeof(int), cudaMemcpyHostToDevice, st);
      cudaMemcpyAsync(cur + 60, mate0, 60 * sizeof(int), cudaMemcpyHostToDevice, st);
    }
    const Mesh m{cur, cur + n};
    const int grid = std::min((n + 255) / 256, sms * 16);
    k_edge_first<<<grid, 256, 0, st>>>(m.mate, n, rank);
    scan_ints(rank, rank, n, sums, st);
    k_edge_split<<<grid, 256, 0, st>>>(m, rank, n, n_vert, v, last ? nullptr : next,
                                       last ? nullptr : next + 4 * size_t(n));
    n_vert += n / 2;
  }
  k_unit<<<std::min((n_vert + 255) / 256, sms * 16), 256, 0, st>>>(v, n_vert);
}

}  // namespace dirs
}  // namespace sbr
