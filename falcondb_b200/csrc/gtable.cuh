// Open-addressing aggregate table shared by the int64-key GROUP BY kernels
// (one query: k_groupby.cu; many queries in one launch: k_batch.cu).
//
// A slot holds one group: key ^ 2^63 (so the all-zero slot is empty and a
// table is cleared with cudaMemset), COUNT(*), SUM and the MIN / MAX order
// keys of the value.  MIN is kept as the bitwise NOT of its order key so that
// both MIN and MAX are atomicMax from a zero identity.  The key INT64_MIN reads
// as NULL (aggregate.rs:867, 1207) and has a slot of its own outside the table.
#pragma once
#include "common.cuh"

namespace fdb {

struct GSlot {          // 40 bytes; all-zero = empty
  uint64_t key;         // key ^ 2^63
  unsigned long long count;
  double sum;
  unsigned long long nmin;  // ~order key of MIN (atomicMax)
  unsigned long long max;   // order key of MAX
};

constexpr uint32_t kSmemSlots = 1024;      // CTA table slots (power of two)
#ifndef FDB_GB_SMEM_PROBE
#define FDB_GB_SMEM_PROBE 4
#endif
constexpr uint32_t kSmemProbe = FDB_GB_SMEM_PROBE;  // probes before a row spills to global
constexpr uint32_t kGlobalProbeLimit = 1u << 16;

// Hash partitions of a key (the top bits of mix64 of the stored key).
constexpr uint32_t kGbParts = 512;
__device__ __forceinline__ uint32_t gb_partition(uint64_t hash) { return (uint32_t)(hash >> 55); }
static_assert(kGbParts == 1u << 9, "gb_partition takes nine bits");

__device__ __forceinline__ void gslot_accum(GSlot* s, double v, bool has_v) {
  atomicAdd(&s->count, 1ull);
  if (has_v) {
    atomicAdd(&s->sum, v);
    if (!isnan(v)) {
      const uint64_t k = f64_ord_key(v);
      atomicMax(&s->nmin, (unsigned long long)~k);
      atomicMax(&s->max, (unsigned long long)k);
    }
  }
}

// Shared-memory (CTA table) slots count rows with a 32-bit atomic on the low
// word of `count`: shared memory has a native 32-bit atomic add, while its
// 64-bit integer and FP64 adds are compare-and-swap loops that serialise on a
// hot slot.  A CTA sees fewer than 2^32 rows of one query, and readers take
// the whole 64-bit word (high word zero).
__device__ __forceinline__ void sslot_accum(GSlot* s, double v, bool has_v) {
  atomicAdd(reinterpret_cast<unsigned int*>(&s->count), 1u);
  if (has_v) {
    atomicAdd(&s->sum, v);
    if (!isnan(v)) {
      const uint64_t k = f64_ord_key(v);
      atomicMax(&s->nmin, (unsigned long long)~k);
      atomicMax(&s->max, (unsigned long long)k);
    }
  }
}

__device__ __forceinline__ void gslot_merge(GSlot* s, const GSlot& v) {
  atomicAdd(&s->count, v.count);
  atomicAdd(&s->sum, v.sum);
  atomicMax(&s->nmin, v.nmin);
  atomicMax(&s->max, v.max);
}

// Find or claim the slot of `skey` (nonzero) in a global table of mask+1
// slots.  A table that is too small (more groups than slots) fails fast: the
// probe is capped, the error word is set, and every later lookup sees the
// error word and gives up at once, so the kernel still ends promptly.
__device__ __forceinline__ GSlot* gtable_find(GSlot* table, uint64_t mask, uint64_t skey, int* err) {
  if (*reinterpret_cast<volatile int*>(err) != 0) return nullptr;
  uint64_t h = mix64(skey) & mask;
  const uint64_t limit = umin64(mask + 1, kGlobalProbeLimit);
  for (uint64_t probe = 0; probe < limit; ++probe) {
    GSlot* s = table + h;
    const uint64_t cur = *reinterpret_cast<volatile uint64_t*>(&s->key);
    if (cur == skey) return s;
    if (cur == 0) {
      const uint64_t prev = atomicCAS(reinterpret_cast<unsigned long long*>(&s->key), 0ull,
                                      (unsigned long long)skey);
      if (prev == 0 || prev == skey) return s;
    }
    h = (h + 1) & mask;
  }
  atomicExch(err, kErrCapacity);
  return nullptr;
}

// gtable_find for a caller that has already loaded `cur`, the key word of the
// key's home slot h = mix64(skey) & mask (so that several lookups can have
// their first load in flight together).
__device__ __forceinline__ GSlot* gtable_find_from(GSlot* table, uint64_t mask, uint64_t skey, uint64_t h,
                                                   uint64_t cur, int* err) {
  const uint64_t limit = umin64(mask + 1, kGlobalProbeLimit);
  for (uint64_t probe = 0; probe < limit; ++probe) {
    GSlot* s = table + h;
    if (probe) cur = *reinterpret_cast<volatile uint64_t*>(&s->key);
    if (cur == skey) return s;
    if (cur == 0) {
      const uint64_t prev = atomicCAS(reinterpret_cast<unsigned long long*>(&s->key), 0ull,
                                      (unsigned long long)skey);
      if (prev == 0 || prev == skey) return s;
    }
    h = (h + 1) & mask;
  }
  atomicExch(err, kErrCapacity);
  return nullptr;
}

// The CTA's shared-memory slot of `skey`, claiming one if free within
// kSmemProbe probes; nullptr when the key has no room there.
__device__ __forceinline__ GSlot* smem_table_slot(GSlot* tab, uint64_t skey) {
  uint32_t h = (uint32_t)mix64(skey) & (kSmemSlots - 1);
  for (uint32_t probe = 0; probe < kSmemProbe; ++probe) {
    GSlot* s = tab + h;
    const uint64_t cur = *reinterpret_cast<volatile uint64_t*>(&s->key);
    if (cur == skey) return s;
    if (cur == 0) {
      const uint64_t prev = atomicCAS(reinterpret_cast<unsigned long long*>(&s->key), 0ull,
                                      (unsigned long long)skey);
      if (prev == 0 || prev == skey) return s;
    }
    h = (h + 1) & (kSmemSlots - 1);
  }
  return nullptr;
}

// The output row of a live slot (key given as stored, XOR 2^63).
__device__ __forceinline__ fdb_group_i64 gslot_group(uint64_t skey, const GSlot& s) {
  fdb_group_i64 g;
  g.key = (int64_t)(skey ^ (1ull << 63));
  g.count = (int64_t)s.count;
  g.sum = s.sum;
  g.min = s.nmin ? f64_from_ord_key(~s.nmin) : __longlong_as_double(0x7ff8000000000000ll);
  g.max = s.max ? f64_from_ord_key(s.max) : __longlong_as_double(0x7ff8000000000000ll);
  return g;
}

// The lanes of a warp whose rows go to the same CTA slot (j; -1: none), merged
// before the shared-memory atomics: the first of them gets their number and the
// sum of their values, the others 0 rows.  All 32 lanes call.  The method is the
// known one for reducing by key within a warp: a match gives each lane its peers, and
// in each round a lane adds its next live peer's value and every other peer drops out.
struct SlotRows {
  uint32_t rows;
  double sum;
};
__device__ __forceinline__ SlotRows warp_slot_rows(int j, double v, int lane) {
  const unsigned peers = __match_any_sync(0xffffffffu, j >= 0 ? j : -1 - lane);
  const unsigned below = peers & ((1u << lane) - 1u);
  unsigned above = peers & ~((2u << lane) - 1u);
  uint32_t rank = __popc(below);
  SlotRows r;
  r.rows = below ? 0u : (uint32_t)__popc(peers);
  r.sum = v;
  while (__any_sync(0xffffffffu, above != 0)) {  // halves every group's live lanes
    const double x = __shfl_sync(0xffffffffu, r.sum, above ? __ffs(above) - 1 : lane);
    if (above) r.sum += x;
    above &= __ballot_sync(0xffffffffu, (rank & 1u) == 0);
    rank >>= 1;
  }
  if (j < 0) r.rows = 0;
  return r;
}

// Whether a warp's rows are worth merging: at least kMergeLanes of them meet
// another row in their slot.  Lanes of one slot retry its SUM one after another,
// while merging costs every row a match and a few shuffles: 30M rows of 64
// queries with 2000 Zipf(1.1) keys (8 lanes) 790 us without it, 612 with; 50 Zipf
// keys 995 and 310; one key 3630 and 294; 5M rows of 200 uniform keys (2 lanes) 76
// without, 89 with.  The line lies between, where neither side is far ahead (3 and
// 5 differ by 4 us on the last, 0 on the others).
constexpr int kMergeLanes = 5;
__device__ __forceinline__ bool warp_slots_repeat(int j, int lane) {
  const unsigned peers = __match_any_sync(0xffffffffu, j >= 0 ? j : -1 - lane);
  return __popc(__ballot_sync(0xffffffffu, (peers & ((1u << lane) - 1u)) != 0)) >= kMergeLanes;
}

// ---------------------------------------------------------------------------
// CTA table keyed by 64-bit keys, structure of arrays: kSmemSlots slots and the
// NULL group's (the last).
//   * Random slots spread over all 32 banks (a 40-byte record's fields fall on
//     few).
//   * MIN / MAX take their 64-bit atomic, a compare-and-swap loop in shared
//     memory, only when the value improves on the slot.  The first test reads one
//     word of lower bounds of both order keys' top 16 bits, stored after the keys
//     are raised (a store that loses a race only lowers a bound).
// The FLOAT64 SUM stays a compare-and-swap loop; where keys are skewed a warp's
// rows are merged first (warp_slot_rows).  Without that it was what cost most: one
// table of 4096 slots per SM, which takes in every row of 2000 Zipf(1.1) keys, was
// slower than three of 1024 that send a third of them to the global table (1.5
// against 0.84 ms for 30M rows), and columns of sums per thread for the six most
// frequent keys brought it to 1.0 only.
// ---------------------------------------------------------------------------
struct HTab {
  uint64_t key[kSmemSlots + 1];             // 0 = empty
  double sum[kSmemSlots + 1];
  unsigned long long nmin[kSmemSlots + 1];  // ~order key of MIN
  unsigned long long max[kSmemSlots + 1];   // order key of MAX
  uint32_t mm16[kSmemSlots + 1];            // top 16 bits of nmin (low half) and max (high half)
  uint32_t count[kSmemSlots + 1];           // a CTA sees fewer than 2^32 rows
};
static_assert(sizeof(HTab) % 8 == 0, "cleared by 8-byte words");

__device__ __forceinline__ void htab_clear(HTab& t) {
  uint64_t* w = reinterpret_cast<uint64_t*>(&t);
  for (uint32_t i = threadIdx.x; i < sizeof(t) / 8; i += blockDim.x) w[i] = 0;
}

// The slot of skey, claiming one if free within kSmemProbe probes; -1 when the
// key has no room there.
__device__ __forceinline__ int htab_slot(HTab& t, uint64_t skey) {
  uint32_t h = (uint32_t)mix64(skey) & (kSmemSlots - 1);
  for (uint32_t probe = 0; probe < kSmemProbe; ++probe) {
    const uint64_t cur = *reinterpret_cast<volatile uint64_t*>(&t.key[h]);
    if (cur == skey) return (int)h;
    if (cur == 0) {
      const uint64_t prev = atomicCAS(reinterpret_cast<unsigned long long*>(&t.key[h]), 0ull, (unsigned long long)skey);
      if (prev == 0 || prev == skey) return (int)h;
    }
    h = (h + 1) & (kSmemSlots - 1);
  }
  return -1;
}

// A row's value into slot j, with g's rows (warp_slot_rows of the warp's slots).
__device__ __forceinline__ void htab_accum(HTab& t, uint32_t j, const SlotRows& g, double v, bool has_v) {
  if (g.rows) {
    atomicAdd(&t.count[j], g.rows);
    if (__double_as_longlong(g.sum) != 0) atomicAdd(&t.sum[j], g.sum);
  }
  if (!has_v || isnan(v)) return;
  const unsigned long long k = f64_ord_key(v);
  const uint32_t w = *reinterpret_cast<volatile uint32_t*>(&t.mm16[j]);
  volatile uint16_t* bound = reinterpret_cast<volatile uint16_t*>(&t.mm16[j]);
  const uint32_t n16 = (uint32_t)(~k >> 48), k16 = (uint32_t)(k >> 48);
  if (n16 >= (w & 0xFFFFu) && ~k > *reinterpret_cast<volatile unsigned long long*>(&t.nmin[j])) {
    atomicMax(&t.nmin[j], ~k);
    bound[0] = (uint16_t)n16;
  }
  if (k16 >= (w >> 16) && k > *reinterpret_cast<volatile unsigned long long*>(&t.max[j])) {
    atomicMax(&t.max[j], k);
    bound[1] = (uint16_t)k16;
  }
}

__device__ __forceinline__ GSlot htab_group(const HTab& t, uint32_t j) {
  return GSlot{t.key[j], t.count[j], t.sum[j], t.nmin[j], t.max[j]};
}

}  // namespace fdb
