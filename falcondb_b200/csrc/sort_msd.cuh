// Sample sort of (key, position) pairs: the path of ORDER BY and DISTINCT for
// keys that rarely repeat (the radix passes of k_sort.cu take the others).
//
// The LSD radix sort reads and writes every pair once per key byte that varies
// (226 bytes per row for a float column) and is bound by the instructions of
// its stable ranking.  Here one or two scatter passes put the pairs into buckets
// of about 1500 whose key ranges come from a sample, and a CTA sorts each bucket
// in shared memory: 8 + 12, 12 + 12 and 12 + 4 bytes per row.  No pass has to be
// stable, because pairs are compared by (key, position) in the last one, so a
// pair's place in its tile is the return value of one shared-memory atomic.
//
//   msd_sample_kernel   one CTA: up to 16384 sampled keys give the bucket map, a
//                       table over 4096 equal steps of the sample's range (its
//                       tails cut off) with about the same share of the samples
//                       in every bucket.  Keys that repeat too often for the
//                       buckets' capacity stop the sort here.
//   msd_split_kernel    tiles of 4096 pairs: bucket by one table read, reorder in
//                       shared memory, write runs to the buckets' regions.
//   msd_subsample / split again   above 409,600 pairs, inside each bucket.
//   msd_leaf_kernel     one CTA per bucket: a slot per pair by linear
//                       interpolation over the bucket's range, then each pair
//                       counts the pairs of its own slot that come before it.  A
//                       bucket whose keys crowd into few slots is sorted by a
//                       bitonic network instead, or, when it is the whole
//                       input, by a stable counting sort.
//
//   msd_over_*_kernel   leaves of two-level sorts that hold more pairs than their
//                       region: what the region has no room for is spilled to a
//                       list, the region's pairs join it, and the list (a few per
//                       cent of the pairs) is sorted by radix passes.  These are
//                       values with some 2400 to 40,000 of 100M rows, too few for
//                       the sample to see, and other clusters of close keys.
//
// A first-level bucket that overflows its region, or more spilled pairs than the
// list takes, sets a state word; the kernels after it return at once and the
// caller runs the radix passes instead.
#pragma once
#include <type_traits>

#include "common.cuh"

namespace fdb {

constexpr int kMsdThreads = 512;
constexpr int kMsdItems = 8;
constexpr uint32_t kMsdTile = kMsdThreads * kMsdItems;  // pairs per tile
constexpr uint32_t kMsdMaxB = 512;                      // buckets per level
constexpr uint32_t kMsdSteps = 4096;                    // steps of a bucket map
constexpr int kMsdSampleItems = 8;                      // samples per thread (of 1024) of a map
constexpr int kMsdLeafThreads = 256;
constexpr int kMsdLeafItems = 9;                        // pairs per thread of most leaves; up to
constexpr uint32_t kMsdLeafMost = kMsdLeafThreads * kMsdLeafItems;  // this many pairs, and a leaf's
constexpr int kMsdBigItems = 16;                        // capacity is this, so that four CTAs'
constexpr uint32_t kMsdLeafCap = 3968;                  // shared memory still fit an SM
constexpr uint32_t kMsdSlots = 4096;                    // leaf slots
constexpr uint32_t kMsdCrowd = 32;                      // pairs per slot before another sort takes over
constexpr uint32_t kMsdLeafRows = 1600;                 // the most rows a leaf holds on average
static_assert(kMsdMaxB <= kMsdThreads, "one thread per bucket in a tile's scan");
static_assert(kMsdSlots == 16 * kMsdLeafThreads, "a thread's slots are two 16-byte words");
static_assert(kMsdLeafCap <= kMsdLeafThreads * kMsdBigItems, "a leaf fits its threads' items");

// State words, nonzero when the sort stopped: set by the sample, by a
// first-level overflow, by the second-level samples, by more spilled pairs than
// there is room for.  A kernel reads only the words that kernels before it write,
// so all its threads see the same.
constexpr int kMsdRepeats = 0, kMsdOverflow1 = 1, kMsdUneven2 = 2, kMsdOverflow2 = 3, kMsdStates = 4;
// Counters: leaves of more than kMsdLeafMost pairs; pairs that their leaf's region
// had no room for, and those leaves; pairs in steps that nearly fill a leaf.
constexpr int kMsdBigCount = 8, kMsdSpilled = 9, kMsdOverLeaves = 10, kMsdUnevenPairs = 11;

__device__ __forceinline__ bool msd_stopped(const uint32_t* state, int words) {
  uint32_t x = 0;
  for (int i = 0; i < words; ++i) x |= state[i];
  return x != 0;
}

// A bucket map: a key's offset x = (key - base) >> shift (32 bits, clamped to
// the range's ends), its step umulhi(x, mul) of kMsdSteps, and the step's part.
// Part p has the offsets [first[p], first[p + 1]).
struct MsdMap {
  uint64_t base;
  uint32_t shift, mul;
  uint16_t part[kMsdSteps];
  uint32_t first[kMsdMaxB + 4];
};

__device__ __forceinline__ uint32_t msd_step(uint64_t key, uint64_t base, uint32_t shift, uint32_t mul) {
  const uint64_t d = (key - base) >> shift;
  const uint32_t x = key < base ? 0u : ((uint32_t)(d >> 32) ? 0xFFFFFFFFu : (uint32_t)d);
  return min(__umulhi(x, mul), kMsdSteps - 1);
}

// A leaf as its CTA needs it: its pairs, where they start in the output, and the
// slots' scale (offset (key - base) >> shift, slot umulhi(offset, mul)).
// `measure`: the leaf also holds keys outside its map's range, so the scale has
// to come from its own smallest and largest key.
struct MsdLeaf {
  uint64_t base;
  uint32_t count, out;
  uint32_t shift, mul, measure, _pad;
};

// The scale of the key range [base, base + range].
__device__ __forceinline__ void msd_scale(uint64_t range, uint32_t* shift, uint32_t* mul) {
  const uint32_t over = (uint32_t)(range >> 32);
  *shift = over ? 32 - __clz(over) : 0;
  const uint64_t offsets = (range >> *shift) + 1;  // at most 2^32
  *mul = (uint32_t)min((uint64_t)0xFFFFFFFFu, ((uint64_t)kMsdSlots << 32) / offsets);
}

__device__ __forceinline__ uint32_t msd_hash(uint64_t key) {
  return ((uint32_t)key * 0x85EBCA6Bu) ^ ((uint32_t)(key >> 32) * 0x9E3779B1u);
}

// Exclusive block scan over kThreads threads (32 words of sm); one barrier.
template <int kThreads>
__device__ __forceinline__ uint32_t msd_block_scan(uint32_t v, uint32_t* sm) {
  constexpr int kWarps = kThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sm[warp] = x;
  __syncthreads();
  uint32_t s = lane < kWarps ? sm[lane] : 0u;
#pragma unroll
  for (int o = 1; o < kWarps; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += y;
  }
  const uint32_t base = __shfl_sync(0xffffffffu, s, warp ? warp - 1 : 0);
  return (warp ? base : 0u) + x - v;
}

// Ascending (key, position) order of n pairs in shared memory, by the whole
// block: a bitonic network over p2 = 2^k >= n pairs whose missing ones count as
// larger than any other.  Every merge is ascending (its first step pairs i with
// the mirror image of i in its block), so the missing pairs never move.
__device__ __forceinline__ void msd_bitonic_pairs(uint64_t* k, uint32_t* v, uint32_t n, uint32_t p2) {
  for (uint32_t size = 2; size <= p2; size <<= 1)
    for (uint32_t step = size >> 1; step > 0; step >>= 1) {
      for (uint32_t t = threadIdx.x; t < p2 / 2; t += blockDim.x) {
        const uint32_t i = 2 * t - (t & (step - 1));
        const uint32_t j = step == size >> 1 ? (i | (size - 1)) - (i & (step - 1)) : i + step;
        if (j >= n) continue;
        const uint64_t a = k[i], b = k[j];
        const uint32_t x = v[i], y = v[j];
        if (a > b || (a == b && x > y)) {
          k[i] = b;
          k[j] = a;
          v[i] = y;
          v[j] = x;
        }
      }
      __syncthreads();
    }
}

// Position of sample j of 2^log_samples <= m in [0, m): one per stratum.
__device__ __forceinline__ uint32_t msd_sample_pos(uint32_t j, int log_samples, uint32_t m) {
  const uint32_t a = (uint32_t)(((uint64_t)j * m) >> log_samples), b = (uint32_t)(((uint64_t)(j + 1) * m) >> log_samples);
  uint32_t h = (j + 1) * 0x9E3779B1u;
  h = (h ^ (h >> 15)) * 0x85EBCA6Bu;
  h ^= h >> 13;
  return a + __umulhi(h, b - a);
}

struct MsdMapSmem {
  uint32_t hist[kMsdSteps];
  uint32_t scan[32];
  uint64_t lo[32], hi[32];
  uint32_t lo_step, hi_step, heaviest;
};

// The bucket map of the block's 2^log_samples samples (kItems in each of the
// first `per` threads) for `parts` buckets; returns the samples in the fullest step
// (what the map cannot split).  As long as the range of all but half a bucket's
// share at either end is under three quarters of the range, the range is cut to
// that (outliers go to the end steps).
template <int kItems>
__device__ __forceinline__ uint32_t msd_build_map(MsdMapSmem& S, const uint64_t (&k)[kItems], uint32_t per,
                                                  int log_samples, uint32_t parts, MsdMap* map) {
  constexpr uint32_t kPer = kMsdSteps / 1024;
  const uint32_t tid = threadIdx.x, samples = 1u << log_samples;
  uint64_t lo = ~0ull, hi = 0;
#pragma unroll
  for (int i = 0; i < kItems; ++i)
    if (tid < per) {
      lo = min(lo, k[i]);
      hi = max(hi, k[i]);
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((tid & 31) == 0) {
    S.lo[tid >> 5] = lo;
    S.hi[tid >> 5] = hi;
  }
  if (tid == 0) S.heaviest = 0;
  __syncthreads();
  lo = S.lo[tid & 31];
  hi = S.hi[tid & 31];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  uint64_t base = lo, range = hi - lo;
  const uint32_t tail = samples / (2 * parts);
  uint32_t shift = 0, mul = 0, c[kPer], before = 0;
  for (int round = 0;; ++round) {
    const uint32_t over = (uint32_t)(range >> 32);
    shift = over ? 32 - __clz(over) : 0;
    const uint64_t steps = (range >> shift) + 1;  // offsets, at most 2^32
    mul = (uint32_t)min((uint64_t)0xFFFFFFFFu, ((uint64_t)kMsdSteps << 32) / steps);
    reinterpret_cast<uint4*>(S.hist)[tid] = make_uint4(0, 0, 0, 0);
    if (tid == 0) {
      S.lo_step = 0;
      S.hi_step = kMsdSteps - 1;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kItems; ++i)
      if (tid < per) atomicAdd(&S.hist[msd_step(k[i], base, shift, mul)], 1u);
    __syncthreads();
    const uint4 h = reinterpret_cast<const uint4*>(S.hist)[tid];
    c[0] = h.x;
    c[1] = h.y;
    c[2] = h.z;
    c[3] = h.w;
    before = msd_block_scan<1024>(c[0] + c[1] + c[2] + c[3], S.scan);
    uint32_t cum = before;
#pragma unroll
    for (uint32_t q = 0; q < kPer; ++q) {
      const uint32_t next = cum + c[q];
      if (cum <= tail && next > tail) S.lo_step = tid * kPer + q;
      if (cum < samples - tail && next >= samples - tail) S.hi_step = tid * kPer + q;
      cum = next;
    }
    __syncthreads();
    const uint32_t a = S.lo_step, b = S.hi_step;
    if (round == 7 || steps <= kMsdSteps || b < a || (b - a + 1) * 4 >= kMsdSteps * 3) break;
    // Step s starts at offset ceil(s * 2^32 / mul).
    const uint64_t xa = (((uint64_t)a << 32) + mul - 1) / mul;
    const uint64_t xb = min(steps, (((uint64_t)(b + 1) << 32) + mul - 1) / mul);
    base += xa << shift;
    range = ((xb - xa) << shift) - 1;
    __syncthreads();
  }
  // A step goes to the part that the middle of its samples falls in.
  uint32_t cum = before, fullest = 0, part[kPer];
#pragma unroll
  for (uint32_t q = 0; q < kPer; ++q) {
    part[q] = min(parts - 1, (uint32_t)(((uint64_t)(cum + c[q] / 2) * parts) >> log_samples));
    fullest = max(fullest, c[q]);
    cum += c[q];
  }
  reinterpret_cast<uint2*>(map->part)[tid] = make_uint2(part[0] | part[1] << 16, part[2] | part[3] << 16);
  reinterpret_cast<uint4*>(S.hist)[tid] = make_uint4(part[0], part[1], part[2], part[3]);
  fullest = __reduce_max_sync(0xffffffffu, fullest);
  if ((tid & 31) == 0) atomicMax(&S.heaviest, fullest);
  __syncthreads();
  for (uint32_t s = tid; s < kMsdSteps; s += 1024) {
    const uint32_t p0 = s ? S.hist[s - 1] + 1 : 0, p1 = S.hist[s];
    if (p0 > p1) continue;
    const uint32_t x = (uint32_t)min((uint64_t)0xFFFFFFFFu, (((uint64_t)s << 32) + mul - 1) / mul);
    for (uint32_t p = p0; p <= p1; ++p) map->first[p] = x;
  }
  for (uint32_t p = S.hist[kMsdSteps - 1] + 1 + tid; p <= parts; p += 1024) map->first[p] = 0xFFFFFFFFu;
  if (tid == 0) {
    map->base = base;
    map->shift = shift;
    map->mul = mul;
  }
  return S.heaviest;
}

// The sort stops, for the radix passes, when at most `few_bytes` bytes of the
// sampled keys vary, when some key has `run` + 1 equal samples (a sampled share of
// about 1024 pairs, but at least four samples: 49,000 of 100M pairs), when equal
// samples are so many that most keys have 16 pairs or more (8 samples^2 / m: keys
// of r pairs each give samples^2 r / 2m), or when one step of the map holds far
// more than a bucket.  K keys of r pairs among others that do not repeat go unseen
// up to about K r^2 = 2.8e9 (m / 1e8)^2, which is 1.2 % of 100M pairs at r = 2400
// and fewer above: what spills.  The first eighth of the samples is looked at by
// itself, so that clear cases stop after one round trip to memory.
constexpr uint32_t kMsdSeen = 2 * 1024 * kMsdSampleItems;  // hash slots of the equal-sample check
struct MsdSampleSmem {
  MsdMapSmem map;
  uint64_t keys[1024 * kMsdSampleItems];  // thread tid's sample i at i * 1024 + tid
  uint16_t seen[kMsdSeen];
  uint32_t count[kMsdSeen / 8];
  uint32_t equal;
  uint32_t any[4];  // OR of the keys' halves, then of their complements'
};
static_assert(kMsdSeen == 1u << 14, "hash bits of the equal-sample check");

// One CTA, kItems samples per thread: the equal-sample check takes the first
// kMsdSampleItems of them, the map all.  Clears the state's `counters` words under
// its first reads, which saves a sort of few values the launch that the sample costs
// it (420,000 rows of 12 values: 65 us, 70 with a memset and the sums of one block;
// 68 by the radix passes without a sample).
template <class Src, int kItems>
__global__ void __launch_bounds__(1024) msd_sample_kernel(Src src, uint32_t m, int log_samples, uint32_t parts,
                                                          uint32_t run, int few_bytes, MsdMap* map, uint32_t* state,
                                                          uint32_t counters) {
  extern __shared__ __align__(128) unsigned char msd_smem[];
  MsdSampleSmem& S = *reinterpret_cast<MsdSampleSmem*>(msd_smem);
  constexpr int kChecked = kMsdSampleItems;
  static_assert(kItems >= kChecked, "the check's samples are among the map's");
  const uint32_t tid = threadIdx.x, samples = 1u << log_samples, per = samples / kItems;  // threads with samples
  const bool in = tid < per;
  uint64_t k[kItems];
  k[0] = in ? src.key(msd_sample_pos(tid * kItems, log_samples, m)) : 0;
  for (uint32_t j = tid; j < counters / 4; j += 1024) reinterpret_cast<uint4*>(state)[j] = make_uint4(0, 0, 0, 0);
  if (tid < 4) S.any[tid] = 0;
  if (tid == 4) S.equal = 0;
  for (uint32_t j = tid; j < kMsdSeen / 8; j += 1024) S.count[j] = 0;
  __syncthreads();
  // Equal samples: the last sample written to a key's hash slot stands for it.
  bool heavy = false;
  uint32_t limit = 0;
  auto check = [&](auto first_item, auto last_item) {
    constexpr int first = decltype(first_item)::value, last = decltype(last_item)::value;
#pragma unroll
    for (int i = first; i < last; ++i)
      if (in) {
        S.keys[i * 1024 + tid] = k[i];
        S.seen[msd_hash(k[i]) >> 18] = (uint16_t)(i * 1024 + tid);
      }
    __syncthreads();
    uint32_t n = 0;
#pragma unroll
    for (int i = first; i < last; ++i)
      if (in) {
        const uint32_t h = msd_hash(k[i]) >> 18, w = S.seen[h];
        if (w != i * 1024 + tid && S.keys[w] == k[i]) {
          ++n;
          heavy |= atomicAdd(&S.count[h / 8], 1u) + 1 >= run;
        }
      }
    n = __reduce_add_sync(0xffffffffu, n);
    if ((tid & 31) == 0 && n) atomicAdd(&S.equal, n);
    limit = (uint32_t)(8.0f * (float)(per * last) * (float)(per * last) / (float)m) + 4;
  };
  const uint32_t lo = (uint32_t)k[0], hi = (uint32_t)(k[0] >> 32);
  const uint32_t any[4] = {__reduce_or_sync(0xffffffffu, in ? lo : 0u), __reduce_or_sync(0xffffffffu, in ? hi : 0u),
                           __reduce_or_sync(0xffffffffu, in ? ~lo : 0u), __reduce_or_sync(0xffffffffu, in ? ~hi : 0u)};
  if ((tid & 31) < 4) atomicOr(&S.any[tid & 3], any[tid & 3]);
  check(std::integral_constant<int, 0>(), std::integral_constant<int, 1>());
  int stop = __syncthreads_or(heavy);
  const uint64_t vary = (uint64_t)(S.any[1] & S.any[3]) << 32 | (S.any[0] & S.any[2]);
  int bytes = 0;
#pragma unroll
  for (int b = 0; b < 8; ++b) bytes += ((vary >> (8 * b)) & 0xFF) != 0;
  if (stop || bytes <= few_bytes || S.equal > limit) {
    if (tid == 0) state[kMsdRepeats] = 1;
    return;
  }
#pragma unroll
  for (int i = 1; i < kItems; ++i)
    k[i] = in ? src.key(msd_sample_pos(tid * kItems + i, log_samples, m)) : 0;
  check(std::integral_constant<int, 1>(), std::integral_constant<int, kChecked>());
  stop = __syncthreads_or(heavy);
  if (stop || S.equal > limit) {
    if (tid == 0) state[kMsdRepeats] = 1;
    return;
  }
  const uint32_t fullest = msd_build_map(S.map, k, per, log_samples, parts, map);
  if (tid == 0 && (uint64_t)fullest * parts > samples + samples / 2) state[kMsdRepeats] = 1;
}

// One CTA per first-level bucket: the map of its second level, from up to
// `max_samples` of its own keys.  CTA 0 also writes how many tiles the buckets
// before each one have (first[b], b <= gridDim.x).
template <int kItems>
__global__ void __launch_bounds__(1024) msd_subsample_kernel(const uint64_t* keys, const uint32_t* cursor, uint32_t cap,
                                                             uint32_t parts, uint32_t spill_cap, MsdMap* maps,
                                                             uint32_t* first, uint32_t* state) {
  __shared__ MsdMapSmem S;
  if (msd_stopped(state, kMsdOverflow1 + 1)) return;
  const uint32_t tid = threadIdx.x;
  if (blockIdx.x == 0) {
    const uint32_t t = tid < gridDim.x ? (cursor[tid] + kMsdTile - 1) / kMsdTile : 0u;
    const uint32_t s = msd_block_scan<1024>(t, S.scan);
    if (tid <= gridDim.x) first[tid] = s;
    __syncthreads();
  }
  const uint32_t n = cursor[blockIdx.x];
  if (n == 0) return;
  const int log_samples = 31 - __clz(min(n, 1024u * kItems));
  if ((1u << log_samples) < kItems) {  // a bucket this small: any map will do
    if (tid == 0) {
      MsdMap& M = maps[blockIdx.x];
      M.base = 0;
      M.shift = 32;
      M.mul = kMsdSteps;
    }
    for (uint32_t s = tid; s < kMsdSteps; s += 1024) maps[blockIdx.x].part[s] = 0;
    for (uint32_t p = tid; p <= parts; p += 1024) maps[blockIdx.x].first[p] = p ? 0xFFFFFFFFu : 0u;
    return;
  }
  const uint32_t per = (1u << log_samples) / kItems;
  const uint64_t* src = keys + (size_t)blockIdx.x * cap;
  uint64_t k[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    k[i] = tid < per ? src[msd_sample_pos(tid * kItems + i, log_samples, n)] : 0;
  }
  const uint32_t fullest = msd_build_map(S, k, per, log_samples, parts, maps + blockIdx.x);
  // A step that alone nearly fills a leaf (small buckets never do) will spill.
  const uint32_t pairs = (uint32_t)(((uint64_t)fullest * n) >> log_samples);
  if (tid == 0 && pairs > kMsdLeafCap * 3 / 4 && atomicAdd(&state[kMsdUnevenPairs], pairs) + pairs > spill_cap)
    state[kMsdUneven2] = 1;
}

struct MsdSplitSmem {
  uint64_t keys[kMsdTile];
  uint32_t pos[kMsdTile];
  uint16_t part[kMsdTile];
  uint16_t map[kMsdSteps];
  uint32_t count[kMsdMaxB];
  uint32_t start[kMsdMaxB];
  uint32_t base[kMsdMaxB];
  uint32_t scan[32];
};

// The second level reads the first's pairs, of whatever column.
struct MsdNoSource {
  __device__ __forceinline__ uint64_t key(uint32_t) const { return 0; }
};
struct MsdSpill {
  uint64_t* keys;
  uint32_t* pos;
  uint32_t cap;
};

// Pairs of one level scattered into `parts` buckets each.  First level
// (kSecond false): tile blockIdx.x of the source, buckets 0 .. parts - 1.
// Second level: the tiles of the first level's buckets (kin, vin, in_count,
// in_cap, first), bucket b's parts being buckets b * parts ...  Bucket x's
// pairs go to kout / vout [x * cap, ...), counted in cursor[x].  Second-level
// pairs beyond their region go to the spill list.  Bound by
// shared memory (a table read, one atomic and two or three stores at random
// places per pair: the LSU data pipe is 72 % busy) and by the write of short
// runs; 0.67 and 0.78 ms for 100M pairs, 3.0 TB/s.  At three CTAs per SM the 40
// registers do not hold eight keys and eight places: 36 to 88 bytes spill.
template <class Src, bool kSecond>
__global__ void __launch_bounds__(kMsdThreads, 3)
    msd_split_kernel(Src src, uint32_t m, const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                     const uint32_t* __restrict__ in_count, uint32_t in_cap, const uint32_t* __restrict__ first,
                     uint32_t nfirst, const MsdMap* __restrict__ maps, uint32_t parts, uint32_t cap,
                     uint64_t* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t* cursor, MsdSpill spill,
                     uint32_t* state) {
  extern __shared__ __align__(128) unsigned char msd_smem[];
  MsdSplitSmem& S = *reinterpret_cast<MsdSplitSmem*>(msd_smem);
  if (msd_stopped(state, kSecond ? kMsdUneven2 + 1 : kMsdRepeats + 1)) return;
  const uint32_t tid = threadIdx.x;
  uint32_t bucket = 0, n, t0;
  if (kSecond) {
    if (blockIdx.x >= first[nfirst]) return;
    uint32_t lo = 0, hi = nfirst;  // first[lo] <= blockIdx.x < first[hi]
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (first[mid] <= blockIdx.x)
        lo = mid;
      else
        hi = mid;
    }
    bucket = lo;
    t0 = (blockIdx.x - first[bucket]) * kMsdTile;
    n = min(kMsdTile, in_count[bucket] - t0);
  } else {
    t0 = blockIdx.x * kMsdTile;
    n = min(kMsdTile, m - t0);
  }
  const size_t in0 = (size_t)bucket * in_cap + t0;
  uint64_t k[kMsdItems];
#pragma unroll
  for (int j = 0; j < kMsdItems; ++j) {
    const uint32_t i = j * kMsdThreads + tid;
    k[j] = 0;
    if (i < n) k[j] = kSecond ? __ldcs(kin + in0 + i) : src.key(t0 + i);
  }
  const MsdMap& M = maps[bucket];
  const uint64_t base = M.base;
  const uint32_t shift = M.shift, mul = M.mul;
  if (tid < parts) S.count[tid] = 0;
  for (uint32_t i = tid; i < kMsdSteps / 8; i += kMsdThreads)
    reinterpret_cast<uint4*>(S.map)[i] = reinterpret_cast<const uint4*>(M.part)[i];
  __syncthreads();
  // Bucket of each pair, and its arrival number there (bucket << 16 | number).
  uint32_t br[kMsdItems];
#pragma unroll
  for (int j = 0; j < kMsdItems; ++j) {
    const bool in = j * kMsdThreads + tid < n;
    const uint32_t x = S.map[msd_step(k[j], base, shift, mul)];
    // A warp whose pairs all go to one bucket (sorted input) adds once.
    const uint32_t x0 = __shfl_sync(0xffffffffu, x, 0);
    uint32_t r = 0;
    if (__all_sync(0xffffffffu, in && x == x0)) {
      if ((tid & 31) == 0) r = atomicAdd(&S.count[x], 32u);
      r = __shfl_sync(0xffffffffu, r, 0) + (tid & 31);
    } else if (in) {
      r = atomicAdd(&S.count[x], 1u);
    }
    br[j] = x << 16 | r;
  }
  __syncthreads();
  const uint32_t c = tid < parts ? S.count[tid] : 0u;
  uint32_t g = 0;
  if (c) g = atomicAdd(&cursor[bucket * parts + tid], c);  // its round trip runs under the scan
  const uint32_t s = msd_block_scan<kMsdThreads>(c, S.scan);
  if (tid < parts) {
    S.start[tid] = s;
    if (!kSecond && g + c > cap) atomicExch(state + kMsdOverflow1, 1u);
    S.base[tid] = g - s;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kMsdItems; ++j) {
    const uint32_t i = j * kMsdThreads + tid;
    if (i < n) {
      const uint32_t x = br[j] >> 16, p = S.start[x] + (br[j] & 0xFFFFu);
      S.keys[p] = k[j];
      if (kSecond) {
        S.pos[p] = __ldcs(vin + in0 + i);
        S.part[p] = (uint16_t)x;
      } else {
        S.pos[p] = x << 16 | i;  // the bucket beside the place in the tile
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kMsdItems; ++j) {
    const uint32_t p = j * kMsdThreads + tid;
    if (p < n) {
      const uint32_t w = S.pos[p], x = kSecond ? S.part[p] : w >> 16, o = S.base[x] + p;
      if (o < cap) {
        const size_t at = (size_t)(bucket * parts + x) * cap + o;
        kout[at] = S.keys[p];
        vout[at] = kSecond ? w : t0 + (w & 0xFFFFu);
      } else if (kSecond) {
        const unsigned act = __activemask();  // one atomic for the lanes that are here
        const int lane = tid & 31, first_lane = __ffs(act) - 1;
        uint32_t q = 0;
        if (lane == first_lane) q = atomicAdd(state + kMsdSpilled, (uint32_t)__popc(act));
        q = __shfl_sync(act, q, first_lane) + __popc(act & ((1u << lane) - 1u));
        if (q < spill.cap) {
          spill.keys[q] = S.keys[p];
          spill.pos[q] = w;
        } else {
          atomicExch(state + kMsdOverflow2, 1u);
        }
      }
    }
  }
}

// Describes the leaves: CTA b those of first-level bucket b (`parts` of them, of
// map b); with one level, CTA 0 all.  above[] counts the buckets' pairs.  Lists
// the big leaves from big[0] on, and those with more pairs than their region
// (`cap`) from big[leaves - 1] down.
__global__ void __launch_bounds__(kMsdThreads) msd_leaves_kernel(const uint32_t* above, const uint32_t* count,
                                                                 uint32_t cap, const MsdMap* maps, uint32_t parts,
                                                                 MsdLeaf* leaves, uint32_t* big, uint32_t* state) {
  __shared__ uint32_t sm[32];
  __shared__ uint32_t before;
  if (msd_stopped(state, kMsdStates)) return;
  const uint32_t tid = threadIdx.x;
  if (tid == 0) before = 0;
  __syncthreads();
  uint32_t a = tid < blockIdx.x ? above[tid] : 0u;  // at most 512 buckets
  a = __reduce_add_sync(0xffffffffu, a);
  if ((tid & 31) == 0 && a) atomicAdd(&before, a);
  const uint32_t c = tid < parts ? count[blockIdx.x * parts + tid] : 0u;
  const uint32_t s = msd_block_scan<kMsdThreads>(c, sm);
  __syncthreads();
  if (tid >= parts) return;
  MsdLeaf l;
  l.count = c;
  l.out = before + s;
  l.shift = l.mul = l.measure = l._pad = 0;
  l.base = 0;
  if (c) {
    const MsdMap& M = maps[blockIdx.x];
    const uint32_t x0 = M.first[tid], x1 = M.first[tid + 1];
    l.measure = x0 == 0 || x1 == 0xFFFFFFFFu;  // the end steps also hold what lies outside
    if (!l.measure) {
      l.base = M.base + ((uint64_t)x0 << M.shift);
      msd_scale(((uint64_t)(x1 - x0) << M.shift) - 1, &l.shift, &l.mul);
    }
  }
  leaves[blockIdx.x * parts + tid] = l;
  if (c > cap)
    big[gridDim.x * parts - 1 - atomicAdd(state + kMsdOverLeaves, 1u)] = blockIdx.x * parts + tid;
  else if (c > kMsdLeafMost)
    big[atomicAdd(state + kMsdBigCount, 1u)] = blockIdx.x * parts + tid;
}

template <int kItems>
struct MsdLeafSmem {
  static constexpr uint32_t kCap = kItems == kMsdLeafItems ? kMsdLeafMost : kMsdLeafCap;
  uint64_t keys[kCap];  // the output rows once every pair has its place
  uint32_t pos[kCap];
  uint16_t slot[kMsdSlots + 8];  // counts, then where each slot starts
  uint32_t scan[32];
  uint32_t hi_min, hi_max, lo_min, lo_max, crowded;
};

// A CTA's stable counting sort of up to kMsdLeafCap pairs, for a leaf that is the
// whole input and whose keys crowd: 12 bits of (key - smallest) per pass.  Each
// warp counts its own 512 pairs in order (the lanes of one digit by a match), so
// pairs keep their order; a thread then owns 16 digits, whose counts lie 9 words
// from its neighbour's (no bank conflicts).  ORDER BY 3000
// rows of 12 values, the whole call: 30 us, 76 through the bitonic network, 60
// through the radix passes; DISTINCT 47, 93, 82.
constexpr int kMsdCountWarps = kMsdLeafThreads / 32;
constexpr int kMsdCountBits = 12, kMsdCountPasses = 3;
struct MsdCountSmem {
  uint32_t count[kMsdCountWarps][kMsdLeafThreads * 9];  // digit d: half word (d & 1) of word d / 16 * 9 + d / 2 % 8
  uint64_t lo[kMsdCountWarps], hi[kMsdCountWarps];
};
static_assert(1 << kMsdCountBits == 16 * kMsdLeafThreads, "a thread owns sixteen digits");

// The pairs (k[j], j * 256 + tid) sorted into S, keys less the smallest; false,
// with nothing of use there, when the keys' range needs more than
// kMsdCountPasses passes.
template <int kItems>
__device__ __forceinline__ bool msd_count_sort(const uint64_t (&k)[kItems], uint32_t n, MsdLeafSmem<kItems>& S,
                                               MsdCountSmem& C) {
  constexpr int T = kMsdLeafThreads;
  static_assert(kItems * 32 * kMsdCountWarps >= (int)kMsdLeafCap, "a warp's pairs");
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, below = (1u << lane) - 1u;
  uint64_t lo = ~0ull, hi = 0;
#pragma unroll
  for (int j = 0; j < kItems; ++j)
    if (j * T + tid < n) {
      lo = min(lo, k[j]);
      hi = max(hi, k[j]);
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) {
    C.lo[warp] = lo;
    C.hi[warp] = hi;
  }
  __syncthreads();
  for (int w = 0; w < kMsdCountWarps; ++w) {
    lo = min(lo, C.lo[w]);
    hi = max(hi, C.hi[w]);
  }
  const uint64_t range = hi - lo;
  if (range >> (kMsdCountBits * kMsdCountPasses)) return false;
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const uint32_t i = j * T + tid;
    if (i < n) {
      S.keys[i] = k[j] - lo;
      S.pos[i] = i;
    }
  }
  for (int shift = 0; range >> shift; shift += kMsdCountBits) {
    for (int i = 0; i < kMsdCountWarps * 9; ++i) (&C.count[0][0])[i * T + tid] = 0;
    __syncthreads();
    uint64_t x[kItems];
    uint32_t v[kItems], at[kItems];  // at: the digit's half word << 16 | rank among the warp's pairs of it
    uint16_t* mine = reinterpret_cast<uint16_t*>(C.count[warp]);
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      const uint32_t i = warp * (kItems * 32) + r * 32 + lane;
      x[r] = i < n ? S.keys[i] : 0;
      v[r] = i < n ? S.pos[i] : 0;
      const uint32_t d = (uint32_t)(x[r] >> shift) & ((1u << kMsdCountBits) - 1);
      const unsigned peers = __match_any_sync(0xffffffffu, i < n ? d : 0xFFFFFFFFu);
      const uint32_t h = 2 * ((d >> 4) * 9 + ((d >> 1) & 7)) + (d & 1);
      const int leader = __ffs(peers) - 1;
      uint32_t before = 0;
      if (i < n && (int)lane == leader) {
        before = mine[h];
        mine[h] = (uint16_t)(before + __popc(peers));
      }
      before = __shfl_sync(0xffffffffu, before, leader);
      at[r] = h << 16 | (before + __popc(peers & below));
      __syncwarp();
    }
    __syncthreads();
    uint32_t sum = 0;
    for (int q = 0; q < 8; ++q)
#pragma unroll
      for (int w = 0; w < kMsdCountWarps; ++w) {
        const uint32_t c = C.count[w][tid * 9 + q];
        sum += (c & 0xFFFFu) + (c >> 16);
      }
    uint32_t run = msd_block_scan<T>(sum, S.scan);
    for (int q = 0; q < 8; ++q) {
      uint32_t c[kMsdCountWarps], s[kMsdCountWarps];
#pragma unroll
      for (int w = 0; w < kMsdCountWarps; ++w) {
        c[w] = C.count[w][tid * 9 + q];
        s[w] = run;
        run += c[w] & 0xFFFFu;
      }
#pragma unroll
      for (int w = 0; w < kMsdCountWarps; ++w) {
        C.count[w][tid * 9 + q] = s[w] | run << 16;
        run += c[w] >> 16;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r)
      if (warp * (kItems * 32) + r * 32 + lane < n) {
        const uint32_t p = mine[at[r] >> 16] + (at[r] & 0xFFFFu);
        S.keys[p] = x[r];
        S.pos[p] = v[r];
      }
    __syncthreads();
  }
  __syncthreads();
  return true;
}

// Sorts a leaf of n pairs (kDirect: the pairs of the source).  kHeads false:
// writes src.row(position) of the leaf's pairs in order.  kHeads: sets bit
// src.row(position) of `mask` for the first position of every key.  Bound by
// latency and issue (about 200 instructions per 32 pairs at 49 % issue), so few
// threads take a leaf, its loads are all issued first, most leaves' shared
// memory is sized for 2304 pairs (five CTAs per SM), and pairs are compared in
// slot order, where neighbouring lanes read neighbouring words.
template <class Src, bool kHeads, bool kDirect, int kItems>
__device__ __forceinline__ void msd_leaf(const Src& src, const MsdLeaf& l, const uint64_t* __restrict__ keys,
                                         const uint32_t* __restrict__ pos, uint32_t* __restrict__ rows,
                                         unsigned long long* mask, MsdLeafSmem<kItems>& S,
                                         MsdCountSmem* counts = nullptr) {
  constexpr int T = kMsdLeafThreads;
  const uint32_t tid = threadIdx.x, n = l.count, out0 = l.out;
  uint32_t shift = l.shift, mul = l.mul;
  uint64_t base = l.base;
  // The positions are read with the keys where registers allow.
  constexpr bool kEarly = !kDirect && kItems == kMsdLeafItems;
  uint32_t v[kEarly ? kItems : 1];
  auto position = [&](int j, uint32_t i) -> uint32_t {
    if constexpr (kDirect) return i;
    else if constexpr (kEarly) return v[j];
    else return __ldcs(pos + i);
  };
  uint64_t k[kItems];
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    if (j * T >= n) break;
    const uint32_t i = j * T + tid;
    k[j] = 0;
    if (i < n) {
      k[j] = kDirect ? src.key(i) : __ldcs(keys + i);
      if constexpr (kEarly) v[j] = __ldcs(pos + i);
    }
  }
  if (tid == 0) S.crowded = 0;
  reinterpret_cast<uint4*>(S.slot)[tid] = make_uint4(0, 0, 0, 0);
  reinterpret_cast<uint4*>(S.slot)[tid + T] = make_uint4(0, 0, 0, 0);
  if (l.measure) {  // the range of the high halves, or of the low ones when all agree
    if (tid == 0) {
      S.hi_min = S.lo_min = 0xFFFFFFFFu;
      S.hi_max = S.lo_max = 0;
    }
    __syncthreads();
    uint32_t a = 0xFFFFFFFFu, b = 0;
#pragma unroll
    for (int j = 0; j < kItems; ++j)
      if (j * T + tid < n) {
        a = min(a, (uint32_t)(k[j] >> 32));
        b = max(b, (uint32_t)(k[j] >> 32));
      }
    a = __reduce_min_sync(0xffffffffu, a);
    b = __reduce_max_sync(0xffffffffu, b);
    if ((tid & 31) == 0) {
      atomicMin(&S.hi_min, a);
      atomicMax(&S.hi_max, b);
    }
    __syncthreads();
    const bool low = S.hi_min == S.hi_max;
    if (low) {
      a = 0xFFFFFFFFu;
      b = 0;
#pragma unroll
      for (int j = 0; j < kItems; ++j)
        if (j * T + tid < n) {
          a = min(a, (uint32_t)k[j]);
          b = max(b, (uint32_t)k[j]);
        }
      a = __reduce_min_sync(0xffffffffu, a);
      b = __reduce_max_sync(0xffffffffu, b);
      if ((tid & 31) == 0) {
        atomicMin(&S.lo_min, a);
        atomicMax(&S.lo_max, b);
      }
      __syncthreads();
    }
    base = (uint64_t)S.hi_min << 32 | (low ? S.lo_min : 0u);
    msd_scale(((uint64_t)S.hi_max << 32 | (low ? S.lo_max : 0xFFFFFFFFu)) - base, &shift, &mul);
  }
  auto slot_of = [&](uint64_t key) { return __umulhi((uint32_t)((key - base) >> shift), mul); };
  __syncthreads();
  uint32_t arrival[(kItems + 3) / 4];  // each pair's arrival number in its slot, a byte each
  bool crowded = false;
#pragma unroll
  for (int q = 0; q < (kItems + 3) / 4; ++q) arrival[q] = 0;
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    if (j * T >= n) break;
    if (j * T + tid < n) {
      const uint32_t s = slot_of(k[j]), half = (s & 1u) * 16;
      const uint32_t r = (atomicAdd(reinterpret_cast<uint32_t*>(S.slot) + (s >> 1), 1u << half) >> half) & 0xFFFFu;
      crowded |= r >= kMsdCrowd;
      arrival[j / 4] |= (r & 0xFFu) << (j % 4 * 8);
    }
  }
  if (crowded) S.crowded = 1;
  __syncthreads();

  if (S.crowded) {
    bool sorted = false;
    if constexpr (kDirect) sorted = msd_count_sort(k, n, S, *counts);
    if (!sorted) {
      uint32_t p2 = 32;
      while (p2 < n) p2 <<= 1;
#pragma unroll
      for (int j = 0; j < kItems; ++j) {
        const uint32_t i = j * T + tid;
        if (i < n) {
          S.keys[i] = k[j];
          S.pos[i] = position(j, i);
        }
      }
      __syncthreads();
      msd_bitonic_pairs(S.keys, S.pos, n, p2);
    }
    for (uint32_t i = tid; i < n; i += T) {
      const uint32_t row = src.row(S.pos[i]);
      if (!kHeads)
        rows[out0 + i] = row;
      else if (i == 0 || S.keys[i] != S.keys[i - 1])
        atomicOr(&mask[row >> 6], 1ull << (row & 63));
    }
    return;
  }

  // Each thread's sixteen slots are two 16-byte words of half words.
  uint4 q8[2] = {reinterpret_cast<const uint4*>(S.slot)[2 * tid], reinterpret_cast<const uint4*>(S.slot)[2 * tid + 1]};
  uint32_t* w = &q8[0].x;
  uint32_t t = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint32_t lo = w[q] & 0xFFFFu, hi = w[q] >> 16;
    w[q] = t | (t + lo) << 16;
    t += lo + hi;
  }
  const uint32_t s0 = msd_block_scan<T>(t, S.scan) * 0x10001u;
#pragma unroll
  for (int q = 0; q < 8; ++q) w[q] += s0;
  reinterpret_cast<uint4*>(S.slot)[2 * tid] = q8[0];
  reinterpret_cast<uint4*>(S.slot)[2 * tid + 1] = q8[1];
  if (tid == 0) S.slot[kMsdSlots] = (uint16_t)n;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    if (j * T >= n) break;
    const uint32_t i = j * T + tid;
    if (i < n) {
      const uint32_t p = S.slot[slot_of(k[j])] + ((arrival[j / 4] >> (j % 4 * 8)) & 0xFFu);
      S.keys[p] = k[j];
      S.pos[p] = position(j, i);
    }
  }
  __syncthreads();
  // The pair at p, in slot order: its place is its slot's start plus the slot's
  // pairs that come first.
  uint32_t place[(kItems + 1) / 2];
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    if (j * T >= n) break;
    const uint32_t p = j * T + tid;
    if (p < n) {
      const uint64_t key = S.keys[p];
      const uint32_t s = slot_of(key), q0 = S.slot[s], q1 = S.slot[s + 1];
      uint32_t less = q0;
      bool again = false;  // an equal key comes first
      if (q1 - q0 > 1)
        for (uint32_t q = q0; q < q1; ++q) {
          const uint64_t x = S.keys[q];
          if (x < key) {
            ++less;
          } else if (x == key && S.pos[q] < S.pos[p]) {
            ++less;
            again = true;
          }
        }
      if (j & 1)
        place[j / 2] |= less << 16;
      else
        place[j / 2] = less;
      if (kHeads && !again) {
        const uint32_t row = src.row(S.pos[p]);
        atomicOr(&mask[row >> 6], 1ull << (row & 63));
      }
    }
  }
  if (kHeads) return;
  __syncthreads();
  uint32_t* out = reinterpret_cast<uint32_t*>(S.keys);
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    if (j * T >= n) break;
    const uint32_t p = j * T + tid;
    if (p < n) out[(place[j / 2] >> (j % 2 * 16)) & 0xFFFFu] = S.pos[p];
  }
  __syncthreads();
  for (uint32_t i = tid; i < n; i += T) rows[out0 + i] = src.row(out[i]);
}

// The leaves of at most kMsdLeafMost pairs, one per CTA.
template <class Src, bool kHeads>
__global__ void __launch_bounds__(kMsdLeafThreads, 5)
    msd_leaf_kernel(Src src, const uint64_t* __restrict__ keys, const uint32_t* __restrict__ pos,
                    const MsdLeaf* __restrict__ leaves, uint32_t cap, uint32_t* __restrict__ rows,
                    unsigned long long* mask, const uint32_t* state) {
  extern __shared__ __align__(128) unsigned char msd_smem[];
  if (msd_stopped(state, kMsdStates)) return;
  const MsdLeaf l = leaves[blockIdx.x];
  if (l.count == 0 || l.count > min(kMsdLeafMost, cap)) return;
  const size_t in0 = (size_t)blockIdx.x * cap;
  msd_leaf<Src, kHeads, false, kMsdLeafItems>(src, l, keys + in0, pos + in0, rows, mask,
                                              *reinterpret_cast<MsdLeafSmem<kMsdLeafItems>*>(msd_smem));
}

// The larger leaves (big[], counted in the state words), and kDirect: the
// m <= kMsdLeafCap pairs of the source by one CTA.
struct MsdDirectSmem {
  MsdLeafSmem<kMsdBigItems> leaf;
  MsdCountSmem counts;
};
template <class Src, bool kHeads, bool kDirect>
__global__ void __launch_bounds__(kMsdLeafThreads, kDirect ? 1 : 4)
    msd_big_leaf_kernel(Src src, uint32_t m, const uint64_t* __restrict__ keys, const uint32_t* __restrict__ pos,
                        const MsdLeaf* __restrict__ leaves, const uint32_t* __restrict__ big, uint32_t cap,
                        uint32_t* __restrict__ rows, unsigned long long* mask, const uint32_t* state) {
  extern __shared__ __align__(128) unsigned char msd_smem[];
  auto& S = *reinterpret_cast<MsdLeafSmem<kMsdBigItems>*>(msd_smem);
  if constexpr (kDirect) {
    MsdLeaf l{};
    l.count = m;
    l.measure = 1;
    msd_leaf<Src, kHeads, true, kMsdBigItems>(src, l, nullptr, nullptr, rows, mask, S,
                                              &reinterpret_cast<MsdDirectSmem*>(msd_smem)->counts);
  } else {
    if (msd_stopped(state, kMsdStates)) return;
    const uint32_t nbig = state[kMsdBigCount];
    for (uint32_t b = blockIdx.x; b < nbig; b += gridDim.x) {
      const MsdLeaf l = leaves[big[b]];
      const size_t in0 = (size_t)big[b] * cap;
      msd_leaf<Src, kHeads, false, kMsdBigItems>(src, l, keys + in0, pos + in0, rows, mask, S);
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------
// The leaves with more pairs than their region: over[0], over[-1], ...  100M rows
// with ten values of 5000 rows, or a hundred: 2.85 and 2.92 ms in all (8.69 and
// 8.67 when one such leaf sent every row to the radix passes, which alone take
// 7.8); 30M with ten 1.26 ms (2.90).
// ---------------------------------------------------------------------------

// CTA b adds the region of the b-th of them to the spill list.
__global__ void __launch_bounds__(256) msd_over_collect_kernel(const uint64_t* __restrict__ keys,
                                                               const uint32_t* __restrict__ pos, uint32_t cap,
                                                               const uint32_t* over, MsdSpill spill, uint32_t* state) {
  __shared__ uint32_t base;
  if (threadIdx.x == 0) base = atomicAdd(state + kMsdSpilled, cap);
  __syncthreads();
  const size_t in0 = (size_t)over[-(ptrdiff_t)blockIdx.x] * cap;
  for (uint32_t i = threadIdx.x; i < cap; i += blockDim.x)
    if (base + i < spill.cap) {
      spill.keys[base + i] = keys[in0 + i];
      spill.pos[base + i] = pos[in0 + i];
    }
}

// Radix pairs of the n listed pairs: (position, index) without `order`, then, in
// the order that these sorted to, (key, position): radix passes are stable, so
// equal keys end up by position.  What varies as the other key kernels have it.
__global__ void __launch_bounds__(256) msd_over_keys_kernel(MsdSpill spill, const uint32_t* __restrict__ order,
                                                            uint32_t n, uint64_t* __restrict__ keys,
                                                            uint32_t* __restrict__ vals, unsigned long long* vary) {
  unsigned long long o = 0, a = ~0ull;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t at = order ? order[i] : i;
    const uint64_t k = order ? spill.keys[at] : spill.pos[at];
    keys[i] = k;
    vals[i] = order ? spill.pos[at] : i;
    o |= k;
    a &= k;
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    o |= __shfl_xor_sync(0xffffffffu, o, s);
    a &= __shfl_xor_sync(0xffffffffu, a, s);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicOr(&vary[0], o);
    atomicOr(&vary[1], ~a);
  }
}

// CTA b writes the b-th leaf's part of the sorted list, as msd_leaf would: leaves
// follow one another in key order, so it starts after the pairs of the listed
// leaves of smaller number.
template <class Src, bool kHeads>
__global__ void __launch_bounds__(256) msd_over_write_kernel(Src src, const uint32_t* over, uint32_t nover,
                                                             const MsdLeaf* __restrict__ leaves,
                                                             const uint64_t* __restrict__ keys,
                                                             const uint32_t* __restrict__ pos,
                                                             uint32_t* __restrict__ rows, unsigned long long* mask) {
  __shared__ uint32_t start;
  const uint32_t leaf = over[-(ptrdiff_t)blockIdx.x];
  if (threadIdx.x == 0) start = 0;
  __syncthreads();
  uint32_t before = 0;
  for (uint32_t j = threadIdx.x; j < nover; j += blockDim.x) {
    const uint32_t other = over[-(ptrdiff_t)j];
    if (other < leaf) before += leaves[other].count;
  }
  if (before) atomicAdd(&start, before);
  __syncthreads();
  const uint32_t n = leaves[leaf].count, out0 = leaves[leaf].out, in0 = start;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const uint32_t row = src.row(pos[in0 + i]);
    if (!kHeads)
      rows[out0 + i] = row;
    else if (i == 0 || keys[in0 + i] != keys[in0 + i - 1])
      atomicOr(&mask[row >> 6], 1ull << (row & 63));
  }
}

}  // namespace fdb
