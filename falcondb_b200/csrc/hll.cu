// Sizing pass over an INT64 key column, for hash and direct-addressed tables:
// a distinct-count estimate from a HyperLogLog sketch (Flajolet, Fusy,
// Gandouet, Meunier, "HyperLogLog: the analysis of a near-optimal cardinality
// estimation algorithm", 2007; 2^12 registers, standard error about 1.6 %),
// and in the same pass the smallest and largest non-NULL key (NULL = a clear
// validity bit, or INT64_MIN, which GROUP BY reads as NULL), and, when asked, how many
// of them fall into each hash partition (gb_partition).  One pass over the keys plus an
// 18 KB device-to-host copy; synchronises the context stream.
#include <cmath>
#include <vector>

#include "common.cuh"
#include "engine.h"
#include "gtable.cuh"

namespace fdb {

constexpr int kHllBits = 12;
constexpr int kHllRegs = 1 << kHllBits;

// regs[0..kHllRegs) then range[0] = min order key (atomicMin from ~0),
// range[1] = max order key (atomicMax from 0) of the non-NULL keys.
struct KeyStatsOut {
  unsigned int regs[kHllRegs];
  unsigned long long range[2];
  unsigned int parts[kGbParts];
  unsigned int counted;  // parts[] are the keys' counts
};

// Whether the key's register was empty.
__device__ __forceinline__ bool hll_add(unsigned int* r, uint64_t h) {
  const uint32_t idx = (uint32_t)(h >> (64 - kHllBits));
  const uint64_t w = (h << kHllBits) | (1ull << (kHllBits - 1));  // bounds the run of zeros
  return atomicMax(&r[idx], (unsigned int)__clzll((long long)w) + 1u) == 0;
}

struct KeyColumn {
  const int64_t* keys;
  const uint64_t* validity;
  uint64_t voff, n;
  __device__ __forceinline__ bool valid(int64_t k, uint64_t row) const {
    if (k == INT64_MIN) return false;
    if (!validity) return true;
    const uint64_t b = voff + row;
    return (validity[b >> 6] >> (b & 63)) & 1ull;
  }
};

// Whether the column's keys look worth counting per partition: one more shared
// atomic per key (20M keys: 50 us, 43 without), used only by a GROUP BY of 32,768
// groups or more (gb_partitions).  512 keys, the same for every CTA, in pairs
// of neighbours spread over the column, decide:
//   * too few values: the valid ones among the pairs' first keys fill less than 226
//     registers in 256 (32,768 values fill 247 +- 3; 1300 values 226, Zipf keys fewer);
//   * runs of equal keys, more than some 27 long (GbHashOp's CTA tables then take in
//     most rows: 20M sorted ids of 50 rows each 0.88 ms, 0.95 by partitions).
// All threads call, with r[] empty and block-wide ordered; r[] keeps the keys.
constexpr int kLookThreads = 256;
__device__ __forceinline__ bool parts_look_useful(const KeyColumn& c, const longlong2* pairs, uint64_t np,
                                                  uint64_t head, unsigned int* r) {
  const uint64_t p = (np / kLookThreads) * threadIdx.x + (threadIdx.x * 0x9E3779B1u >> 8) % (uint32_t)(np / kLookThreads);
  const longlong2 k = pairs[p];
  const bool vx = c.valid(k.x, head + 2 * p), vy = c.valid(k.y, head + 2 * p + 1);
  const bool fresh = vx && hll_add(r, mix64((uint64_t)k.x ^ (1ull << 63)));
  const int values = __syncthreads_count(fresh), valid = __syncthreads_count(vx);
  const int runs = __syncthreads_count(vx && vy && k.x == k.y);
  return values * 256 >= valid * 226 && runs * 256 <= valid * 246;
}

// Each thread takes 4 aligned pairs of keys per round (4 x 16-byte loads in
// flight), so the pass runs near HBM speed; keys before the first 16-byte
// boundary and after the last full pair are read one by one by thread 0 of
// block 0 and the grid's tail.
template <bool kParts>
__device__ __forceinline__ void key_stats_rows(const KeyColumn& c, unsigned int* r, unsigned int* parts, uint64_t head,
                                               KeyStatsOut* out) {
  const int64_t* __restrict__ keys = c.keys;
  const uint64_t n = c.n;
  uint64_t lo = ~0ull, hi = 0;
  auto take = [&](int64_t k, uint64_t row) {
    const uint64_t h = mix64((uint64_t)k ^ (1ull << 63));
    hll_add(r, h);
    if (c.valid(k, row)) {
      const uint64_t o = i64_ord_key(k);
      lo = o < lo ? o : lo;
      hi = o > hi ? o : hi;
      if (kParts) atomicAdd(&parts[gb_partition(h)], 1u);
    }
  };
  if (blockIdx.x == 0 && threadIdx.x == 0)
    for (uint64_t i = 0; i < head; ++i) take(keys[i], i);
  const longlong2* pairs = reinterpret_cast<const longlong2*>(keys + head);
  const uint64_t np = (n - head) / 2;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  for (; p + 3 * stride < np; p += 4 * stride) {
    longlong2 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = __ldcs(pairs + p + u * stride);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint64_t row = head + 2 * (p + u * stride);
      take(v[u].x, row);
      take(v[u].y, row + 1);
    }
  }
  for (; p < np; p += stride) {
    const longlong2 v = __ldcs(pairs + p);
    take(v.x, head + 2 * p);
    take(v.y, head + 2 * p + 1);
  }
  // Tail: the last key when n - head is odd.
  if (blockIdx.x == 0 && threadIdx.x == 0 && ((n - head) & 1)) take(keys[n - 1], n - 1);
  lo = warp_min_u64(lo);
  hi = warp_max_u64(hi);
  if ((threadIdx.x & 31) == 0) {
    if (lo != ~0ull) atomicMin(&out->range[0], (unsigned long long)lo);
    if (hi != 0) atomicMax(&out->range[1], (unsigned long long)hi);
  }
}

__global__ void __launch_bounds__(kLookThreads) key_stats_kernel(KeyColumn c, bool want_parts, KeyStatsOut* out) {
  __shared__ unsigned int r[kHllRegs];
  __shared__ unsigned int parts[kGbParts];
  for (int i = threadIdx.x; i < kHllRegs; i += blockDim.x) r[i] = 0;
  for (int i = threadIdx.x; i < (int)kGbParts; i += blockDim.x) parts[i] = 0;
  __syncthreads();
  // Head: rows before the first 16-byte aligned key.
  const uint64_t head = umin64(c.n, (uint64_t)((16 - ((uintptr_t)c.keys & 15)) & 15) / 8);
  const bool count =
      want_parts && parts_look_useful(c, reinterpret_cast<const longlong2*>(c.keys + head), (c.n - head) / 2, head, r);
  if (count)
    key_stats_rows<true>(c, r, parts, head, out);
  else
    key_stats_rows<false>(c, r, parts, head, out);
  __syncthreads();
  for (int i = threadIdx.x; i < kHllRegs; i += blockDim.x)
    if (r[i]) atomicMax(&out->regs[i], r[i]);
  if (!count) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) out->counted = 1;
  for (int i = threadIdx.x; i < (int)kGbParts; i += blockDim.x)
    if (parts[i]) atomicAdd(&out->parts[i], parts[i]);
}

static uint64_t hll_estimate(const unsigned int* h, uint64_t n) {
  double z = 0.0;
  int zeros = 0;
  for (int i = 0; i < kHllRegs; ++i) {
    z += std::ldexp(1.0, -(int)h[i]);
    zeros += h[i] == 0;
  }
  const double m = kHllRegs, alpha = 0.7213 / (1.0 + 1.079 / m);
  double e = alpha * m * m / z;
  if (e <= 2.5 * m && zeros > 0) e = m * std::log(m / zeros);  // small-range correction
  return std::min<uint64_t>(n, (uint64_t)std::ceil(e));
}

KeyStats key_stats_i64(Ctx& c, const fdb_dev_column& key, uint64_t n, bool parts) {
  KeyStats s;
  if (n == 0) {
    s.distinct = 1;
    return s;
  }
  if (!key.values) fail(FDB_E_ARG, "column without values");
  KeyStatsOut* d = static_cast<KeyStatsOut*>(c.scratch_take(sizeof(KeyStatsOut)));
  FDB_CUDA(cudaMemsetAsync(d, 0, sizeof(KeyStatsOut), c.stream));
  FDB_CUDA(cudaMemsetAsync(&d->range[0], 0xFF, 8, c.stream));
  const unsigned grid = (unsigned)umin64((n / 2 + 255) / 256 + 1, (uint64_t)c.sm_count * 8);
  const KeyColumn col{static_cast<const int64_t*>(key.values), key.validity, key.validity_offset, n};
  key_stats_kernel<<<grid, kLookThreads, 0, c.stream>>>(col, parts && n >= 4 * kLookThreads && n < (1ull << 32), d);
  FDB_CUDA(cudaGetLastError());
  KeyStatsOut h;
  HostReads reads(c);
  reads.add(&h, d, sizeof(h));
  reads.wait();
  s.distinct = n <= 4096 ? n : hll_estimate(h.regs, n);
  if (h.range[0] <= h.range[1]) {
    s.has_range = true;
    s.kmin = (int64_t)(h.range[0] ^ (1ull << 63));
    s.kmax = (int64_t)(h.range[1] ^ (1ull << 63));
  }
  if (h.counted) s.parts.assign(h.parts, h.parts + kGbParts);
  return s;
}

uint64_t estimate_distinct_i64(Ctx& c, const void* keys, uint64_t n) {
  if (n <= 4096) return n ? n : 1;
  fdb_dev_column k{};
  k.dtype = FDB_INT64;
  k.values = keys;
  return key_stats_i64(c, k, n).distinct;
}

}  // namespace fdb
