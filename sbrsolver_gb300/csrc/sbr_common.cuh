// Warp-level helpers and the device hash tables shared by the SBR kernels.
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "sbr_device.h"
#include "sbr_field.cuh"
#include "sbr_kernels.cuh"

namespace sbr {

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

// Open addressing with linear probing.  Tables are kept at most half full
// (the host grows them between solves from the occupancy counters), so a
// probe run longer than kMaxProbe means the table is too small: the insert
// reports overflow and the solve is repeated with a larger table.
constexpr uint32_t kMaxProbe = 256;

// A key, its home slot and what that slot held when the probe was begun: a
// caller with several inserts begins them all before it finishes the first.
struct HashProbe {
  unsigned long long key, first;
  uint32_t slot;
};
__device__ __forceinline__ HashProbe ht_probe(HashTable t, unsigned long long key) {
  HashProbe p;
  p.key = key;
  p.slot = uint32_t(mix64(key)) & t.mask;
  p.first = *reinterpret_cast<volatile unsigned long long*>(&t.keys[p.slot]);
  return p;
}

// The insert past the home slot (out of line: most probes end there).
__device__ __noinline__ uint32_t ht_insert_on(unsigned long long* keys, uint32_t mask,
                                              unsigned long long key, uint32_t h,
                                              unsigned long long first, unsigned* ov,
                                              unsigned bit, unsigned long long* used,
                                              unsigned long long* lost, bool* fresh) {
  const HashTable t{keys, mask};
  const uint32_t lim = min(kMaxProbe, t.mask + 1);
  for (uint32_t i = 0; i < lim; ++i) {
    const unsigned long long k =
        i == 0 ? first : *reinterpret_cast<volatile unsigned long long*>(&t.keys[h]);
    if (k == key) return h;
    if (k == kEmptyKey) {
      unsigned long long old = atomicCAS(&t.keys[h], kEmptyKey, key);
      if (old == kEmptyKey) {
        atomicAdd(used, 1ull);
        if (fresh) *fresh = true;
        return h;
      }
      if (old == key) return h;
    }
    h = (h + 1) & t.mask;
  }
  atomicOr(ov, bit);
  atomicAdd(lost, 1ull);
  return 0xFFFFFFFFu;
}
__device__ __forceinline__ uint32_t ht_insert(HashTable t, const HashProbe& p, unsigned* ov,
                                              unsigned bit, unsigned long long* used,
                                              unsigned long long* lost, bool* fresh = nullptr) {
  if (p.first == p.key) return p.slot;
  return ht_insert_on(t.keys, t.mask, p.key, p.slot, p.first, ov, bit, used, lost, fresh);
}
__device__ __forceinline__ uint32_t ht_insert(HashTable t, unsigned long long key, unsigned* ov,
                                              unsigned bit, unsigned long long* used,
                                              unsigned long long* lost, bool* fresh = nullptr) {
  return ht_insert(t, ht_probe(t, key), ov, bit, used, lost, fresh);
}

// Find or claim key's slot in a table that may fill up: the slot, or
// 0xFFFFFFFF when a probe run of `limit` slots finds neither (the caller then
// works without the table).  fresh: this call claimed the slot.
__device__ __forceinline__ uint32_t ht_claim(HashTable t, unsigned long long key, uint32_t limit,
                                             bool& fresh) {
  fresh = false;
  uint32_t h = uint32_t(mix64(key)) & t.mask;
  const uint32_t lim = min(limit, t.mask + 1);
  for (uint32_t i = 0; i < lim; ++i) {
    unsigned long long k = *reinterpret_cast<volatile unsigned long long*>(&t.keys[h]);
    if (k == key) return h;
    if (k == kEmptyKey) {
      const unsigned long long old = atomicCAS(&t.keys[h], kEmptyKey, key);
      if (old == kEmptyKey) {
        fresh = true;
        return h;
      }
      if (old == key) return h;
    }
    h = (h + 1) & t.mask;
  }
  return 0xFFFFFFFFu;
}

__device__ __forceinline__ uint32_t ht_find(HashTable t, unsigned long long key) {
  uint32_t h = uint32_t(mix64(key)) & t.mask;
  const uint32_t lim = min(kMaxProbe, t.mask + 1);
  for (uint32_t i = 0; i < lim; ++i) {
    unsigned long long k = t.keys[h];
    if (k == key) return h;
    if (k == kEmptyKey) return 0xFFFFFFFFu;
    h = (h + 1) & t.mask;
  }
  return 0xFFFFFFFFu;
}

// Sets every range of the list to its byte value, all in one launch: a solve
// clears some twenty tables and counters, and as separate fills and memsets
// they cost a small solve more than its capture.
struct FillRange {
  unsigned char* p;
  unsigned long long bytes;
  unsigned value;  // the byte, four times
};
constexpr int kFillRanges = 24;
struct FillList {
  FillRange r[kFillRanges];
  int n;
};
__global__ void __launch_bounds__(256) k_fill(const __grid_constant__ FillList L) {
  const unsigned long long t0 = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
  for (int k = 0; k < L.n; ++k) {
    const FillRange R = L.r[k];
    const unsigned long long words = R.bytes >> 4;
    uint4* w = reinterpret_cast<uint4*>(R.p);  // allocations are 256-byte aligned
    for (unsigned long long i = t0; i < words; i += step)
      w[i] = make_uint4(R.value, R.value, R.value, R.value);
    if (t0 < (R.bytes & 15)) R.p[(words << 4) + t0] = (unsigned char)R.value;
  }
}

}  // namespace sbr
