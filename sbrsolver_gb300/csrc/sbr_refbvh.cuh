// The reference BVH (BVH/BVH.h:135-230) built on the device, node for node
// and leaf order for leaf order equal to the host build (sbr_host.cpp).
//
// The reference splits a node by sorting its object list with std::sort
// along x, then y, then z (keys: triangle box centres, many of them equal),
// sweeping box surface areas over each order for the cheapest split, and
// sorting once more along the best axis.  Objects with equal keys end up in
// the order std::sort's introsort leaves them in, and that order shapes the
// tree (which objects go left, the leaf order, hence the closest-hit ties).
// This file restates that introsort so that every comparison, exchange and
// move is the one std::sort (libstdc++) makes:
//   * segments longer than 16 with depth budget left: the median of
//     (f + 1, middle, l - 1) is exchanged to the front, then an unguarded
//     Hoare partition of [f + 1, l) around it; both parts continue with one
//     unit of depth budget less (initially 2 floor(log2 n));
//   * a segment out of depth budget is heap sorted (heap built over the
//     whole segment, then popped), as std::partial_sort(f, l, l) does;
//   * segments of at most 16 are left for a final insertion sort.
// Three facts make it parallel without changing any of those steps:
//   * the two parts of a partition are sorted independently, so the
//     segments of all nodes of a tree level are processed together;
//   * a partition is the sequence of exchanges of the k-th left stop (the
//     k-th position, left to right, whose key is not less than the pivot)
//     with the k-th right stop (right to left, key not greater than the
//     pivot) for as long as the left stop lies left of the right stop; those
//     exchanges touch distinct positions, and the cut is the first left stop
//     that does not (or the last right stop exchanged, if that is smaller);
//   * the final insertion sort never moves an element past a partition
//     boundary (everything left of one is not greater than everything right
//     of it), so it is an insertion sort of each segment of at most 16 alone.
// A CPU restatement of these steps reproduced std::sort on 20,000 random
// inputs with many equal keys; the GPU tests compare the device tree with
// the host tree on every test scene.
#pragma once

#include <cstdint>

namespace sbr {
namespace refbvh {

constexpr int kTile = 1024;        // elements per block of the partition rounds
constexpr int kTileThreads = 256;  // 4 consecutive elements per thread
constexpr int kSmallMax = 2048;    // longest segment one block sorts in shared memory
constexpr int kShortMax = 256;     // segments up to this long take one warp
constexpr int kSmallWarps = 8;     // warps for the longer ones
constexpr int kInsertion = 16;     // segments this short wait for insertion sort

struct __align__(16) SortSeg {
  int f, l, d, tile0;  // range [f, l), depth budget, first tile (partition rounds)
};

// Node of the tree, in the order levels create them.
struct __align__(16) RNode {
  double bb[6];      // box, as the host forms it (min xyz, max xyz)
  int f, l;          // objects [f, l) of the build order
  int c0, c1;        // children, -1 for a leaf
};

// What one level decides for each of its nodes.
struct __align__(16) NodeBest {
  double cost;  // best split cost so far (starts at the leaf cost n)
  int axis;     // -1: no split beats the leaf
  int split;    // objects left of the split
};

// Control words: sort list counts and the next level's sizes.
enum Ctl {
  kBig = 0, kBigNext, kSmall, kShort, kTiny, kHeap, kTiles, kTilesNext, kNodes, kActiveNext,
  kSweepTiles, kTiledNodes, kSmallNodes, kError, kCtlWords
};

__device__ __forceinline__ int floor_log2(int n) { return 31 - __clz(n); }


// Sort keys: the reference sorts by box centres, (min + max) / 2 in FP64 of
// the box of float vertices.  The sum orders like its half, and the integer
// like the sum (-0 and +0 alike; the coordinates are finite), so the sort's
// comparisons stay off the FP64 pipe, where each takes a warp ~76 cycles
// (with the sweeps' integer products the canyon's tree 11.6 -> 10.2 ms).
typedef long long Key;
__device__ __forceinline__ Key centre_key(const float4& lo, const float4& hi, int a) {
  const float l = a == 0 ? lo.x : (a == 1 ? lo.y : lo.z);
  const float h = a == 0 ? hi.x : (a == 1 ? hi.y : hi.z);
  const long long b = __double_as_longlong(__dadd_rn(double(l), double(h)));
  return b >= 0 ? b : -(b & 0x7fffffffffffffffll);
}

// Surface area of a box as the host computes it (sbr_host.cpp
// surface_area): 0 for a box that is flat or empty along any axis, else
// 2 (dx dy + dy dz + dz dx) with every operation rounded on its own (products
// and conversions in integer arithmetic where the extents allow).
__device__ __forceinline__ double surface_area(float lx, float ly, float lz, float hx, float hy,
                                               float hz) {
  if (hx <= lx || hy <= ly || hz <= lz) return 0.0;
  using soft64::from_f32;
  const double dx = __dsub_rn(from_f32(hx), from_f32(lx));
  const double dy = __dsub_rn(from_f32(hy), from_f32(ly));
  const double dz = __dsub_rn(from_f32(hz), from_f32(lz));
  double s;
  if (soft64::safe(dx) && soft64::safe(dy) && soft64::safe(dz))
    s = __dadd_rn(__dadd_rn(soft64::mul(dx, dy), soft64::mul(dy, dz)), soft64::mul(dz, dx));
  else
    s = __dadd_rn(__dadd_rn(__dmul_rn(dx, dy), __dmul_rn(dy, dz)), __dmul_rn(dz, dx));
  return __dadd_rn(s, s);
}

// Cost of splitting n objects after the i-th, 2 + (i sa1 + (n - i) sa2) / sr
// with each operation rounded on its own; sr = SA(node box).
struct SplitCost {
  double sr;
  uint64_t x;  // its mantissa's reciprocal
  bool soft;   // sr is nonzero and in range: areas of extents in soft64's range, and
               // n times them, are too
  __device__ __forceinline__ explicit SplitCost(double s) : sr(s), x(0) {
    const uint32_t e = uint32_t(soft64::bits(s) >> 52) & 0x7ffu;
    soft = e > 1023 - 300 && e < 1023 + 260;
    if (soft) x = soft64::rcp_of(s);
  }
  __device__ __forceinline__ double operator()(int i, int n, double sa1, double sa2) const {
    auto in_range = [](double v) {  // 0, or within [2^-300, 2^260)
      const uint32_t e = uint32_t(soft64::bits(v) >> 52) & 0x7ffu;
      return soft64::bits(v) == 0 || (e > 1023 - 300 && e < 1023 + 260);
    };
    if (soft && in_range(sa1) && in_range(sa2)) {
      const double num = __dadd_rn(soft64::mul(soft64::from_int(i), sa1),
                                   soft64::mul(soft64::from_int(n - i), sa2));
      return __dadd_rn(2.0, soft64::div_by(num, sr, x));
    }
    const double num = __dadd_rn(__dmul_rn(double(i), sa1), __dmul_rn(double(n - i), sa2));
    return __dadd_rn(2.0, __ddiv_rn(num, sr));
  }
};

// ---- per-triangle boxes ----------------------------------------------------

// Box of each triangle's float vertices, as std::min / std::max over the
// three (the first of equal values wins, which fixes the sign of a zero);
// lo.w carries the triangle id.
__global__ void k_boxes(const float* v, int nt, float4* lo, float4* hi) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const float* p = v + 9 * size_t(t);
  float l[3], h[3];
  for (int a = 0; a < 3; ++a) {
    l[a] = p[a];
    h[a] = p[a];
    if (p[3 + a] < l[a]) l[a] = p[3 + a];
    if (p[6 + a] < l[a]) l[a] = p[6 + a];
    if (h[a] < p[3 + a]) h[a] = p[3 + a];
    if (h[a] < p[6 + a]) h[a] = p[6 + a];
  }
  lo[t] = make_float4(l[0], l[1], l[2], __int_as_float(t));
  hi[t] = make_float4(h[0], h[1], h[2], 0.0f);
}

// ---- the sort --------------------------------------------------------------

template <class K, class I>
__device__ __forceinline__ void swap_pair(K* key, I* idx, int a, int b) {
  const K k = key[a];
  key[a] = key[b];
  key[b] = k;
  const int i = idx[a];
  idx[a] = idx[b];
  idx[b] = i;
}

// Exchanges the median of (a, b, c) into r, with the reference sort's
// comparisons in its order.
template <class K, class I>
__device__ __forceinline__ void median_to_first(K* key, I* idx, int r, int a, int b, int c) {
  if (key[a] < key[b]) {
    if (key[b] < key[c]) swap_pair(key, idx, r, b);
    else if (key[a] < key[c]) swap_pair(key, idx, r, c);
    else swap_pair(key, idx, r, a);
  } else if (key[a] < key[c]) {
    swap_pair(key, idx, r, a);
  } else if (key[b] < key[c]) {
    swap_pair(key, idx, r, c);
  } else {
    swap_pair(key, idx, r, b);
  }
}

// Insertion sort of [f, l): each element moves left past strictly greater
// ones (the final pass of std::sort restricted to one segment).
template <class K, class I>
__device__ void insertion_sort(K* key, I* idx, int f, int l) {
  for (int i = f + 1; i < l; ++i) {
    const K k = key[i];
    const int x = idx[i];
    int j = i;
    while (j > f && k < key[j - 1]) {
      key[j] = key[j - 1];
      idx[j] = idx[j - 1];
      --j;
    }
    key[j] = k;
    idx[j] = x;
  }
}

// Heap sort of [0, n) in the steps std::partial_sort(f, l, l) takes: the
// heap is built by sifting each parent from the last down to the root
// (the hole goes down to the larger child, the right one on ties, to the
// bottom, then the value climbs back), then the root is popped n - 1 times.
template <class K, class I>
__device__ void heap_push(K* key, I* idx, long hole, long top, K v, int vi) {
  long parent = (hole - 1) / 2;
  while (hole > top && key[parent] < v) {
    key[hole] = key[parent];
    idx[hole] = idx[parent];
    hole = parent;
    parent = (hole - 1) / 2;
  }
  key[hole] = v;
  idx[hole] = vi;
}
template <class K, class I>
__device__ void heap_adjust(K* key, I* idx, long hole, long len, K v, int vi) {
  const long top = hole;
  long child = hole;
  while (child < (len - 1) / 2) {
    child = 2 * (child + 1);
    if (key[child] < key[child - 1]) child--;
    key[hole] = key[child];
    idx[hole] = idx[child];
    hole = child;
  }
  if ((len & 1) == 0 && child == (len - 2) / 2) {
    child = 2 * (child + 1);
    key[hole] = key[child - 1];
    idx[hole] = idx[child - 1];
    hole = child - 1;
  }
  heap_push(key, idx, hole, top, v, vi);
}
template <class K, class I>
__device__ void heap_sort(K* key, I* idx, long n) {
  if (n >= 2)
    for (long parent = (n - 2) / 2;; --parent) {
      heap_adjust(key, idx, parent, n, key[parent], idx[parent]);
      if (parent == 0) break;
    }
  for (long last = n; last > 1;) {
    --last;
    const K v = key[last];
    const int vi = idx[last];
    key[last] = key[0];
    idx[last] = idx[0];
    heap_adjust(key, idx, 0, last, v, vi);
  }
}

// Files a segment of the sort: nothing to do (<= 1), insertion list (<= 16),
// heap list (no depth budget left), a warp's list (<= kSmallMax), else the
// partition rounds (with its tiles reserved).
// small: capacity small_cap; segments of at most kShortMax are filed from
// its end, longer ones from its start.
__device__ __forceinline__ void file_segment(int f, int l, int d, SortSeg* big, SortSeg* small,
                                             int small_cap, SortSeg* tiny, SortSeg* heap, int* ctl,
                                             int big_slot, int tiles_slot) {
  const int n = l - f;
  if (n <= 1) return;
  if (n <= kInsertion) {
    tiny[atomicAdd(ctl + kTiny, 1)] = SortSeg{f, l, d, 0};
  } else if (d == 0) {
    heap[atomicAdd(ctl + kHeap, 1)] = SortSeg{f, l, d, 0};
  } else if (n <= kShortMax) {  // the short ones fill the small list from its end
    small[small_cap - 1 - atomicAdd(ctl + kShort, 1)] = SortSeg{f, l, d, 0};
  } else if (n <= kSmallMax) {
    small[atomicAdd(ctl + kSmall, 1)] = SortSeg{f, l, d, 0};
  } else {
    const int tiles = (n + kTile - 1) / kTile;
    const int t0 = atomicAdd(ctl + tiles_slot, tiles);
    big[atomicAdd(ctl + big_slot, 1)] = SortSeg{f, l, d, t0};
  }
}

// Initial segments: the objects of each listed node (a split node only,
// for the final sort along its best axis).
__global__ void k_file_nodes(const RNode* nodes, const int* active, int m, const NodeBest* best,
                             SortSeg* big, SortSeg* small, int small_cap, SortSeg* tiny,
                             SortSeg* heap, int* ctl) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= m) return;
  if (best && best[a].axis < 0) return;
  const RNode& nd = nodes[active[a]];
  const int n = nd.l - nd.f;
  if (n < 2) return;
  file_segment(nd.f, nd.l, 2 * floor_log2(n), big, small, small_cap, tiny, heap, ctl, kBig,
               kTiles);
}

// Sum over a block (every thread gets it); sh: one entry a warp.
__device__ __forceinline__ int2 block_sum2(int2 v, int2* sh) {
  v.x = __reduce_add_sync(0xffffffffu, v.x);
  v.y = __reduce_add_sync(0xffffffffu, v.y);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  v = make_int2(0, 0);
  for (int w = 0; w < int(blockDim.x >> 5); ++w) {
    v.x += sh[w].x;
    v.y += sh[w].y;
  }
  return v;
}

// A partition round is four launches that take the counts of their lists from
// the device (parity p of the list counts and of the lists themselves; k_cut
// files the next round's segments under the other parity), so rounds follow
// each other without the host.  With the host reading the counts back after
// each round of seven launches the 580k-triangle terrain's 403 rounds took
// 27.2 ms, now 12.

// Round step 1: the median of three to the front of every big segment, its
// tiles' entries of the tile map, and the other parity's counts to zero.
__global__ void __launch_bounds__(128) k_pivot(const SortSeg* big, int* ctl, int p, Key* key,
                                               int* idx, int* tile_seg) {
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl[kBig + (p ^ 1)] = ctl[kTiles + (p ^ 1)] = 0;
  const int n_big = ctl[kBig + p];
  for (int s = blockIdx.x; s < n_big; s += gridDim.x) {
    const SortSeg g = big[s];
    if (threadIdx.x == 0)
      median_to_first(key, idx, g.f, g.f + 1, g.f + (g.l - g.f) / 2, g.l - 1);
    const int tiles = (g.l - g.f + kTile - 1) / kTile;
    for (int t = threadIdx.x; t < tiles; t += blockDim.x) tile_seg[g.tile0 + t] = s;
  }
}

// Stop flags of position p of segment g around pivot key pk: left stops in
// [f + 1, l), right stops in [f, l).
__device__ __forceinline__ void stop_flags(const Key* key, const SortSeg& g, Key pk, int p,
                                           int& lf, int& rf) {
  lf = rf = 0;
  if (p >= g.l) return;
  const Key k = key[p];
  lf = p > g.f && !(k < pk);
  rf = !(pk < k);
}

// Block-wide exclusive sum of one value per thread; returns the total.
__device__ __forceinline__ int block_exclusive(int v, int& excl, int* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (w == 0) {
    int t = lane < int(blockDim.x >> 5) ? sh[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    sh[32 + lane] = t;  // inclusive over warps
  }
  __syncthreads();
  const int before = w ? sh[32 + w - 1] : 0;
  excl = before + x - v;
  const int total = sh[32 + (blockDim.x >> 5) - 1];
  __syncthreads();
  return total;
}

// Round step 2: stop counts per tile (left, right).
__global__ void __launch_bounds__(kTileThreads)
    k_count(const SortSeg* big, const int* ctl, int p, const int* tile_seg, const Key* key,
            int2* cnt) {
  __shared__ int2 sh[kTileThreads / 32];
  const int n_tiles = ctl[kTiles + p];
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const SortSeg g = big[tile_seg[tile]];
    const Key pk = key[g.f];
    const int base = g.f + (tile - g.tile0) * kTile + threadIdx.x * (kTile / kTileThreads);
    int2 n = make_int2(0, 0);
    for (int j = 0; j < kTile / kTileThreads; ++j) {
      int lf, rf;
      stop_flags(key, g, pk, base + j, lf, rf);
      n.x += lf;
      n.y += rf;
    }
    n = block_sum2(n, sh);
    if (threadIdx.x == 0) cnt[tile] = n;
  }
}

// Round step 3: the stops' positions, left stops ascending in lpos[f ..],
// right stops descending in rpos[f ..].  A tile's block adds up the counts of
// the segment's tiles itself (one thread a segment did, in a launch of its own).
__global__ void __launch_bounds__(kTileThreads)
    k_stops(const SortSeg* big, const int* ctl, int p, const int* tile_seg, const Key* key,
            const int2* cnt, int2* totals, int* lpos, int* rpos) {
  __shared__ int sh[64];
  __shared__ int2 sh2[kTileThreads / 32];
  const int n_tiles = ctl[kTiles + p];
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int s = tile_seg[tile];
    const SortSeg g = big[s];
    const Key pk = key[g.f];
    int2 before = make_int2(0, 0), after = before;
    for (int t = g.tile0 + threadIdx.x; t < g.tile0 + (g.l - g.f + kTile - 1) / kTile;
         t += blockDim.x) {
      const int2 c = cnt[t];
      int2& to = t < tile ? before : after;
      to.x += c.x;
      to.y += c.y;
    }
    before = block_sum2(before, sh2);
    after = block_sum2(after, sh2);
    const int n_r = before.y + after.y;
    if (tile == g.tile0 && threadIdx.x == 0) totals[s] = make_int2(before.x + after.x, n_r);
    const int base = g.f + (tile - g.tile0) * kTile + threadIdx.x * (kTile / kTileThreads);
    int lf[kTile / kTileThreads], rf[kTile / kTileThreads];
    int nl = 0, nr = 0;
    for (int j = 0; j < kTile / kTileThreads; ++j) {
      stop_flags(key, g, pk, base + j, lf[j], rf[j]);
      nl += lf[j];
      nr += rf[j];
    }
    int el, er;
    block_exclusive(nl, el, sh);
    block_exclusive(nr, er, sh);
    int rl = before.x + el, rr = before.y + er;
    for (int j = 0; j < kTile / kTileThreads; ++j) {
      if (lf[j]) lpos[g.f + rl++] = base + j;
      if (rf[j]) rpos[g.f + (n_r - 1 - rr++)] = base + j;
    }
  }
}

// Round step 4: the exchanges (k-th left stop with k-th right stop while the
// left one lies left of the right one), and by the first tile's first warp the
// cut of the segment and its two parts filed.
__global__ void __launch_bounds__(kTileThreads)
    k_cut(const SortSeg* big, int* ctl, int p, const int* tile_seg, const int2* totals,
          const int* lpos, const int* rpos, Key* key, int* idx, SortSeg* big_next, SortSeg* small,
          int small_cap, SortSeg* tiny, SortSeg* heap) {
  const int n_tiles = ctl[kTiles + p];
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int s = tile_seg[tile];
    const SortSeg g = big[s];
    const int nl = totals[s].x, nr = totals[s].y, m = min(nl, nr);
    const int k0 = (tile - g.tile0) * kTile;
    for (int k = k0 + threadIdx.x; k < min(m, k0 + kTile); k += blockDim.x) {
      const int a = lpos[g.f + k], b = rpos[g.f + k];
      if (a < b) swap_pair(key, idx, a, b);
    }
    if (tile != g.tile0 || threadIdx.x >= 32) continue;
    const int lane = threadIdx.x;
    int lo = 0, hi = m;  // first k whose left stop is not left of its right stop
    while (lo < hi) {    // 32 probes at a time
      const int step = (hi - lo + 31) / 32, k = lo + lane * step;
      const int c = __popc(__ballot_sync(0xffffffffu, k < hi && lpos[g.f + k] < rpos[g.f + k]));
      hi = min(hi, lo + c * step);
      if (c) lo += (c - 1) * step + 1;
    }
    if (lane) continue;
    const int K = lo;
    int cut = K < nl ? lpos[g.f + K] : g.l;
    if (K >= 1) cut = min(cut, rpos[g.f + K - 1]);
    if (cut <= g.f || cut >= g.l) {  // the sentinel argument guarantees both parts
      atomicOr(ctl + kError, 1);
      continue;
    }
    for (int h = 0; h < 2; ++h)
      file_segment(h ? cut : g.f, h ? g.l : cut, g.d - 1, big_next, small, small_cap, tiny, heap,
                   ctl, kBig + (p ^ 1), kTiles + (p ^ 1));
  }
}

// A block per segment of at most kCap, sorted in shared memory: the segments a
// partition leaves are independent, so the block's warps take one each, round
// by round (a partition by the warp, its exchanges spread over the lanes);
// segments of at most 16 wait for the end, when they are insertion sorted,
// one per thread.  A chain of shared-memory passes: with one warp for all of
// a segment's partitions the canyon's tree spent 4.3 ms here, with eight 2.1.
struct SortPart {
  short f, l, d, pad;
};
template <int kCap>  // at most kCap / kInsertion parts at one time
constexpr size_t small_smem() {
  return size_t(kCap) * (8 + 4 + 2 + 2 + 4) + 2 * sizeof(SortPart) * (kCap / kInsertion);
}

// segs: the list; n_segs: its count; from_end > 0: the list is read from
// its end (entry from_end - 1 - s, from_end being the list's capacity).
template <int kCap, int kWarps>
__global__ void __launch_bounds__(32 * kWarps) k_small(const SortSeg* segs, const int* n_segs,
                                                       int from_end, Key* key, int* idx,
                                                       int* ctl) {
  extern __shared__ __align__(16) unsigned char smem[];
  Key* sk = reinterpret_cast<Key*>(smem);
  int* si = reinterpret_cast<int*>(sk + kCap);
  int* tiny = si + kCap;
  short* lps = reinterpret_cast<short*>(tiny + kCap);
  short* rps = lps + kCap;
  SortPart* parts[2];
  parts[0] = reinterpret_cast<SortPart*>(rps + kCap);
  parts[1] = parts[0] + kCap / kInsertion;
  __shared__ int n_parts[2], n_tiny, bad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int n = *n_segs;
  for (int s = blockIdx.x; s < n; s += gridDim.x) {
    const SortSeg g = segs[from_end > 0 ? from_end - 1 - s : s];
    const int len = g.l - g.f;
    for (int i = threadIdx.x; i < len; i += blockDim.x) {
      sk[i] = key[g.f + i];
      si[i] = idx[g.f + i];
    }
    if (threadIdx.x == 0) {
      parts[0][0] = SortPart{0, short(len), short(g.d), 0};
      n_parts[0] = 1;
      n_parts[1] = 0;
      n_tiny = 0;
      bad = 0;
    }
    __syncthreads();
    // a segment's part is longer than kInsertion; a depth budget of at most
    // 2 log2 n ends the rounds
    for (int cur = 0; n_parts[cur] > 0; cur ^= 1) {
      for (int q = warp; q < n_parts[cur]; q += kWarps) {
        const SortPart t = parts[cur][q];
        const int f = t.f, l = t.l, d = t.d;
        if (d == 0) {
          if (lane == 0) heap_sort(sk + f, si + f, l - f);
          __syncwarp();
          continue;
        }
        short *lp = lps + f, *rp = rps + f;  // the parts' ranges are disjoint
        if (lane == 0) median_to_first(sk, si, f, f + 1, f + (l - f) / 2, l - 1);
        __syncwarp();
        const Key pk = sk[f];
        int nl = 0, nr = 0;
        for (int b = f + 1; b < l; b += 32) {
          const int p = b + lane;
          const bool fl = p < l && !(sk[p] < pk);
          const unsigned m = __ballot_sync(0xffffffffu, fl);
          if (fl) lp[nl + __popc(m & below)] = short(p);
          nl += __popc(m);
        }
        for (int b = l - 1; b >= f; b -= 32) {
          const int p = b - lane;
          const bool fr = p >= f && !(pk < sk[p]);
          const unsigned m = __ballot_sync(0xffffffffu, fr);
          if (fr) rp[nr + __popc(m & below)] = short(p);
          nr += __popc(m);
        }
        __syncwarp();
        const int mk = min(nl, nr);
        int K = 0;
        for (int b = 0; b < mk; b += 32) {
          const int k = b + lane;
          const unsigned m = __ballot_sync(0xffffffffu, k < mk && lp[k] < rp[k]);
          K += __popc(m);
          if (m != 0xffffffffu) break;
        }
        for (int k = lane; k < K; k += 32) swap_pair(sk, si, lp[k], rp[k]);
        int cut = K < nl ? int(lp[K]) : l;
        if (K >= 1) cut = min(cut, int(rp[K - 1]));
        if (lane == 0) {
          if (cut <= f || cut >= l) {  // the sentinel argument guarantees both parts
            bad = 1;
          } else {
            for (int h = 0; h < 2; ++h) {
              const int pf = h == 0 ? f : cut, pl = h == 0 ? cut : l;
              if (pl - pf > kInsertion)
                parts[cur ^ 1][atomicAdd(&n_parts[cur ^ 1], 1)] =
                    SortPart{short(pf), short(pl), short(d - 1), 0};
              else if (pl - pf >= 2)
                tiny[atomicAdd(&n_tiny, 1)] = pf | ((pl - pf) << 16);
            }
          }
        }
        __syncwarp();
      }
      __syncthreads();
      if (threadIdx.x == 0) n_parts[cur] = 0;
      __syncthreads();
    }
    if (threadIdx.x == 0 && bad) atomicOr(ctl + kError, 2);
    for (int j = threadIdx.x; j < n_tiny; j += blockDim.x) {
      const int f = tiny[j] & 0xffff, c = tiny[j] >> 16;
      insertion_sort(sk, si, f, f + c);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < len; i += blockDim.x) {
      key[g.f + i] = sk[i];
      idx[g.f + i] = si[i];
    }
    __syncthreads();
  }
}

// Insertion sort of the short segments the partition rounds left.
__global__ void k_tiny(const SortSeg* segs, const int* n_segs, Key* key, int* idx) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= *n_segs) return;
  insertion_sort(key, idx, segs[s].f, segs[s].l);
}

// Heap sort of the segments the partition rounds ran out of depth on.
__global__ void k_heap(const SortSeg* segs, const int* n_segs, Key* key, int* idx) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= *n_segs) return;
  heap_sort(key + segs[s].f, idx + segs[s].f, segs[s].l - segs[s].f);
}

// ---- one tree level ------------------------------------------------------

// Sort keys: position p of an active node (of a split node, for the final
// sort) gets its box centre along the axis; every position starts as itself
// in the permutation.
__global__ void k_keys(const float4* lo, const float4* hi, const int* node_of,
                       const NodeBest* best, int axis, int n, Key* key, int* idx) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  idx[p] = p;
  const int a = node_of[p];
  if (a < 0) return;
  const int ax = best ? best[a].axis : axis;
  if (ax < 0) return;
  key[p] = centre_key(lo[p], hi[p], ax);
}

// The build order after a sort: records moved along the permutation.
__global__ void k_gather(const float4* lo, const float4* hi, const int* idx, int n, float4* lo2,
                         float4* hi2) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int q = idx[p];
  lo2[p] = lo[q];
  hi2[p] = hi[q];
}

// ---- per-level node work on warp tiles ------------------------------------
//
// A node's objects [f, l) are cut into tiles of kWarpTile consecutive
// objects (a node has at least one tile, a tile never spans two nodes); a
// warp works on a tile, 8 consecutive objects per lane.
constexpr int kSweepItems = 8;
constexpr int kWarpTile = 32 * kSweepItems;

struct BoxF {
  float l[3], h[3];
};

__device__ __forceinline__ BoxF box_merge(const BoxF& a, const BoxF& b) {
  BoxF r;
  for (int c = 0; c < 3; ++c) {
    r.l[c] = fminf(a.l[c], b.l[c]);
    r.h[c] = fmaxf(a.h[c], b.h[c]);
  }
  return r;
}

__device__ __forceinline__ BoxF box_empty() {
  BoxF r;
  for (int c = 0; c < 3; ++c) {
    r.l[c] = INFINITY;
    r.h[c] = -INFINITY;
  }
  return r;
}

__device__ __forceinline__ BoxF box_shfl_up(const BoxF& x, int o) {
  BoxF y;
  for (int c = 0; c < 3; ++c) {
    y.l[c] = __shfl_up_sync(0xffffffffu, x.l[c], o);
    y.h[c] = __shfl_up_sync(0xffffffffu, x.h[c], o);
  }
  return y;
}

__device__ __forceinline__ BoxF box_shfl_down(const BoxF& x, int o) {
  BoxF y;
  for (int c = 0; c < 3; ++c) {
    y.l[c] = __shfl_down_sync(0xffffffffu, x.l[c], o);
    y.h[c] = __shfl_down_sync(0xffffffffu, x.h[c], o);
  }
  return y;
}

__device__ __forceinline__ BoxF rec_box(const float4& L, const float4& H) {
  return BoxF{{L.x, L.y, L.z}, {H.x, H.y, H.z}};
}

// The box bounds as the host's node box takes them: the least lower bound
// (greatest upper bound), the later object winning between equal values, so
// that the sign of a zero is the host's.
struct ExactBox {
  float v[6];
  int p[6];  // object position the value came from, -1: none yet
};

__device__ __forceinline__ bool exact_better(int c, float v, int p, float bv, int bp) {
  if (p < 0) return false;
  if (bp < 0) return true;
  return c < 3 ? (v < bv || (v == bv && p > bp)) : (v > bv || (v == bv && p > bp));
}

__device__ __forceinline__ void exact_add(ExactBox& b, int c, float v, int p) {
  if (exact_better(c, v, p, b.v[c], b.p[c])) {
    b.v[c] = v;
    b.p[c] = p;
  }
}

__device__ __forceinline__ void exact_warp_reduce(ExactBox& b) {
  for (int o = 16; o; o >>= 1)
    for (int c = 0; c < 6; ++c) {
      const float v = __shfl_down_sync(0xffffffffu, b.v[c], o);
      const int p = __shfl_down_sync(0xffffffffu, b.p[c], o);
      exact_add(b, c, v, p);
    }
}

struct __align__(16) TileBest {
  double cost;
  int i, pad;
};

constexpr int kNodeSmall = 16;  // nodes this small are handled by one thread each

// Tiles of every active node of more than kNodeSmall objects (per node its
// first tile and tile count, per tile its node), and the lists of those
// nodes and of the small ones.
__global__ void k_level_tiles(const RNode* nodes, const int* active, int m, int2* node_tiles,
                              int* tile_node, int* tiled, int* small_nodes, int* ctl) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= m) return;
  const RNode& nd = nodes[active[a]];
  const int n = nd.l - nd.f;
  if (n <= kNodeSmall) {
    small_nodes[atomicAdd(ctl + kSmallNodes, 1)] = a;
    node_tiles[a] = make_int2(0, 0);
    return;
  }
  const int nt = (n + kWarpTile - 1) / kWarpTile;
  const int t0 = atomicAdd(ctl + kSweepTiles, nt);
  node_tiles[a] = make_int2(t0, nt);
  tiled[atomicAdd(ctl + kTiledNodes, 1)] = a;
  for (int t = 0; t < nt; ++t) tile_node[t0 + t] = a;
}

// A small node's set-up, one thread each: its positions marked, its box
// formed object by object as the host forms it (box = std::min(object, box),
// std::max(object, box)), the surface area and the leaf cost as the best.
__global__ void k_small_node_box(RNode* nodes, const int* active, const int* small_nodes, int k,
                                 const float4* lo, const float4* hi, int* node_of,
                                 double* sa_root, NodeBest* best) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= k) return;
  const int a = small_nodes[j];
  RNode& nd = nodes[active[a]];
  float b[6] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
  for (int p = nd.f; p < nd.l; ++p) {
    node_of[p] = a;
    const float4 L = lo[p], H = hi[p];
    const float x[6] = {L.x, L.y, L.z, H.x, H.y, H.z};
    for (int c = 0; c < 3; ++c) {
      if (!(b[c] < x[c])) b[c] = x[c];
      if (!(x[3 + c] < b[3 + c])) b[3 + c] = x[3 + c];
    }
  }
  for (int c = 0; c < 6; ++c) nd.bb[c] = double(b[c]);
  sa_root[a] = surface_area(b[0], b[1], b[2], b[3], b[4], b[5]);
  best[a] = NodeBest{double(nd.l - nd.f), -1, -1};
}

// A small node's sweep over one axis order, one thread each, in the
// reference loop's order: prefix areas, then suffix areas with the costs,
// a cost kept when it is below the best so far.
__global__ void k_small_node_sweep(const RNode* nodes, const int* active, const int* small_nodes,
                                   int k, const float4* lo, const float4* hi,
                                   const double* sa_root, int axis, NodeBest* best) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= k) return;
  const int a = small_nodes[j];
  const RNode& nd = nodes[active[a]];
  const int n = nd.l - nd.f;
  if (n < 3) return;
  double sa1[kNodeSmall];
  BoxF run = box_empty();
  for (int i = 0; i < n; ++i) {
    run = box_merge(run, rec_box(lo[nd.f + i], hi[nd.f + i]));
    sa1[i] = surface_area(run.l[0], run.l[1], run.l[2], run.h[0], run.h[1], run.h[2]);
  }
  double sa2[kNodeSmall];
  run = box_empty();
  for (int i = n - 1; i >= 0; --i) {
    run = box_merge(run, rec_box(lo[nd.f + i], hi[nd.f + i]));
    sa2[i] = surface_area(run.l[0], run.l[1], run.l[2], run.h[0], run.h[1], run.h[2]);
  }
  NodeBest b = best[a];
  const SplitCost split(sa_root[a]);
  for (int i = 1; i < n - 1; ++i) {
    const double cost = split(i, n, sa1[i], sa2[i]);
    if (cost < b.cost) b = NodeBest{cost, axis, i};
  }
  best[a] = b;
}

// Level set-up per tile: positions marked with their node, and the tile's
// share of the node box (taken in the order the objects arrive in).
__global__ void k_tile_exact_box(const RNode* nodes, const int* active, const int2* node_tiles,
                                 const int* tile_node, int n_tiles, const float4* lo,
                                 const float4* hi, int* node_of, ExactBox* tbox) {
  const int tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (tile >= n_tiles) return;
  const int a = tile_node[tile];
  const RNode& nd = nodes[active[a]];
  const int b = nd.f + (tile - node_tiles[a].x) * kWarpTile + lane * kSweepItems;
  ExactBox e;
  for (int c = 0; c < 6; ++c) {
    e.v[c] = 0.0f;
    e.p[c] = -1;
  }
  for (int j = 0; j < kSweepItems; ++j) {
    const int p = b + j;
    if (p >= nd.l) break;
    node_of[p] = a;
    const float4 L = lo[p], H = hi[p];
    const float x[6] = {L.x, L.y, L.z, H.x, H.y, H.z};
    for (int c = 0; c < 6; ++c) exact_add(e, c, x[c], p);
  }
  exact_warp_reduce(e);
  if (lane == 0) tbox[tile] = e;
}

// Node box from its tiles, its surface area, and the leaf cost as the best
// so far; a warp per node.
__global__ void k_node_box(RNode* nodes, const int* active, const int* tiled, int k,
                           const int2* node_tiles, const ExactBox* tbox, double* sa_root,
                           NodeBest* best) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= k) return;
  const int a = tiled[w];
  const int2 nt = node_tiles[a];
  ExactBox e;
  for (int c = 0; c < 6; ++c) {
    e.v[c] = 0.0f;
    e.p[c] = -1;
  }
  for (int t = lane; t < nt.y; t += 32) {
    const ExactBox& x = tbox[nt.x + t];
    for (int c = 0; c < 6; ++c) exact_add(e, c, x.v[c], x.p[c]);
  }
  exact_warp_reduce(e);
  if (lane == 0) {
    RNode& nd = nodes[active[a]];
    for (int c = 0; c < 6; ++c) nd.bb[c] = double(e.v[c]);
    sa_root[a] = surface_area(e.v[0], e.v[1], e.v[2], e.v[3], e.v[4], e.v[5]);
    best[a] = NodeBest{double(nd.l - nd.f), -1, -1};
  }
}

// Box of each tile's objects (in the current order).
__global__ void k_tile_boxes(const RNode* nodes, const int* active, const int2* node_tiles,
                             const int* tile_node, int n_tiles, const float4* lo,
                             const float4* hi, BoxF* tagg) {
  const int tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (tile >= n_tiles) return;
  const int a = tile_node[tile];
  const RNode& nd = nodes[active[a]];
  const int b = nd.f + (tile - node_tiles[a].x) * kWarpTile + lane * kSweepItems;
  BoxF x = box_empty();
  for (int j = 0; j < kSweepItems && b + j < nd.l; ++j) x = box_merge(x, rec_box(lo[b + j], hi[b + j]));
  for (int o = 16; o; o >>= 1) x = box_merge(x, box_shfl_down(x, o));
  if (lane == 0) tagg[tile] = x;
}

// Per node, the box of the objects before each of its tiles (pre) and
// after it (post); a warp per node, 32 tiles at a time.
__global__ void k_tile_carries(const int* tiled, int k, const int2* node_tiles, const BoxF* tagg,
                               BoxF* pre, BoxF* post) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= k) return;
  const int a = tiled[w];
  const int2 nt = node_tiles[a];
  BoxF run = box_empty();
  for (int c = 0; c < nt.y; c += 32) {
    const int t = c + lane;
    BoxF x = t < nt.y ? tagg[nt.x + t] : box_empty();
    for (int o = 1; o < 32; o <<= 1) {
      const BoxF y = box_shfl_up(x, o);
      if (lane >= o) x = box_merge(y, x);
    }
    BoxF ex = box_shfl_up(x, 1);
    if (lane == 0) ex = box_empty();
    if (t < nt.y) pre[nt.x + t] = box_merge(run, ex);
    BoxF last;
    for (int k = 0; k < 3; ++k) {
      last.l[k] = __shfl_sync(0xffffffffu, x.l[k], 31);
      last.h[k] = __shfl_sync(0xffffffffu, x.h[k], 31);
    }
    run = box_merge(run, last);
  }
  run = box_empty();
  for (int c = 0; c < nt.y; c += 32) {  // from the last tile backwards
    const int t = nt.y - 1 - (c + lane);
    BoxF x = t >= 0 ? tagg[nt.x + t] : box_empty();
    for (int o = 1; o < 32; o <<= 1) {
      const BoxF y = box_shfl_up(x, o);
      if (lane >= o) x = box_merge(y, x);
    }
    BoxF ex = box_shfl_up(x, 1);
    if (lane == 0) ex = box_empty();
    if (t >= 0) post[nt.x + t] = box_merge(run, ex);
    BoxF last;
    for (int k = 0; k < 3; ++k) {
      last.l[k] = __shfl_sync(0xffffffffu, x.l[k], 31);
      last.h[k] = __shfl_sync(0xffffffffu, x.h[k], 31);
    }
    run = box_merge(run, last);
  }
}

// The reference's sweep over one axis order (BVH.h:135-230), a warp per
// tile: for object i of the node, the surface area of the box of objects
// 0..i (sa1) and of objects i..n-1 (sa2), the cost
// 2 + (i sa1 + (n - i) sa2) / SA(node box) for 1 <= i <= n - 2 (each operation
// rounded on its own), and the tile's cheapest split below the leaf cost,
// the first one among equal costs.
__global__ void k_tile_sweep(const RNode* nodes, const int* active, const int2* node_tiles,
                             const int* tile_node, int n_tiles, const float4* lo,
                             const float4* hi, const BoxF* pre, const BoxF* post,
                             const double* sa_root, TileBest* tbest) {
  const int tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (tile >= n_tiles) return;
  const int a = tile_node[tile];
  const RNode& nd = nodes[active[a]];
  const int n = nd.l - nd.f;
  const int i0 = (tile - node_tiles[a].x) * kWarpTile + lane * kSweepItems;  // object index
  BoxF bx[kSweepItems];
  BoxF mine = box_empty();
  for (int j = 0; j < kSweepItems; ++j) {
    bx[j] = i0 + j < n ? rec_box(lo[nd.f + i0 + j], hi[nd.f + i0 + j]) : box_empty();
    mine = box_merge(mine, bx[j]);
  }
  // boxes of the lanes before / after this one
  BoxF up = mine, down = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const BoxF y = box_shfl_up(up, o);
    if (lane >= o) up = box_merge(y, up);
    const BoxF z = box_shfl_down(down, o);
    if (lane + o < 32) down = box_merge(down, z);
  }
  BoxF before = box_shfl_up(up, 1), after = box_shfl_down(down, 1);
  if (lane == 0) before = box_empty();
  if (lane == 31) after = box_empty();
  double sa1[kSweepItems];
  BoxF run = box_merge(pre[tile], before);
  for (int j = 0; j < kSweepItems; ++j) {
    run = box_merge(run, bx[j]);
    sa1[j] = surface_area(run.l[0], run.l[1], run.l[2], run.h[0], run.h[1], run.h[2]);
  }
  const SplitCost split(sa_root[a]);
  const double leaf = double(n);
  double bc = INFINITY;
  int bi = INT_MAX;
  run = box_merge(post[tile], after);
  for (int j = kSweepItems - 1; j >= 0; --j) {
    run = box_merge(run, bx[j]);
    const int i = i0 + j;
    if (i >= 1 && i <= n - 2) {
      const double sa2 = surface_area(run.l[0], run.l[1], run.l[2], run.h[0], run.h[1], run.h[2]);
      const double cost = split(i, n, sa1[j], sa2);
      if (cost < leaf && (cost < bc || (cost == bc && i < bi))) {
        bc = cost;
        bi = i;
      }
    }
  }
  for (int o = 16; o; o >>= 1) {
    const double oc = __shfl_down_sync(0xffffffffu, bc, o);
    const int oi = __shfl_down_sync(0xffffffffu, bi, o);
    if (oc < bc || (oc == bc && oi < bi)) {
      bc = oc;
      bi = oi;
    }
  }
  if (lane == 0) tbest[tile] = TileBest{bc, bi, 0};
}

// The node's cheapest split of this axis, kept if it beats the best so far
// (earlier axes win ties, as the strict < of the reference's loop decides);
// a warp per node.
__global__ void k_node_best(const int* tiled, int k, const int2* node_tiles, const TileBest* tbest,
                            int axis, NodeBest* best) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= k) return;
  const int a = tiled[w];
  const int2 nt = node_tiles[a];
  double bc = INFINITY;
  int bi = INT_MAX;
  for (int t = lane; t < nt.y; t += 32) {
    const TileBest x = tbest[nt.x + t];
    if (x.cost < bc || (x.cost == bc && x.i < bi)) {
      bc = x.cost;
      bi = x.i;
    }
  }
  for (int o = 16; o; o >>= 1) {
    const double oc = __shfl_down_sync(0xffffffffu, bc, o);
    const int oi = __shfl_down_sync(0xffffffffu, bi, o);
    if (oc < bc || (oc == bc && oi < bi)) {
      bc = oc;
      bi = oi;
    }
  }
  if (lane == 0 && bi != INT_MAX && bc < best[a].cost) best[a] = NodeBest{bc, axis, bi};
}

// Children of the split nodes (after the final sort), and the next level's
// active list.
__global__ void k_children(RNode* nodes, const int* active, int m, const NodeBest* best,
                           int* next, int* ctl) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= m) return;
  if (best[a].axis < 0) return;
  RNode& nd = nodes[active[a]];
  const int c = atomicAdd(ctl + kNodes, 2);
  nodes[c].f = nd.f;
  nodes[c].l = nd.f + best[a].split;
  nodes[c].c0 = nodes[c].c1 = -1;
  nodes[c + 1].f = nd.f + best[a].split;
  nodes[c + 1].l = nd.l;
  nodes[c + 1].c0 = nodes[c + 1].c1 = -1;
  nd.c0 = c;
  nd.c1 = c + 1;
  const int k = atomicAdd(ctl + kActiveNext, 2);
  next[k] = c;
  next[k + 1] = c + 1;
}

// Triangle ids in build order.
__global__ void k_ids(const float4* lo, int n, int* ids) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) ids[p] = __float_as_int(lo[p].w);
}

}  // namespace refbvh
}  // namespace sbr
