// Quantile binning on the device: QuantizeDense / TransformDense
// (src/core/binned_dataset.cpp:95-238) for a matrix that then stays resident.
//
// Semantics (the same as the host restatement in quantize.cpp): NaN is missing (bin 0 plus
// a missing flag); Inf is an error; float64 input must fit float32. Per feature, with m
// non-missing values and desired = min(max_bins, m), the boundary candidates are the
// order statistics at ranks ceil(part * m / desired) - 1 for part = 1..desired-1, kept
// when below the maximum and above the previous kept boundary; a value's bin is the
// number of boundaries below it (lower_bound).
//
// No sort: the order statistics come from a three-round radix selection over the 32-bit
// order-preserving image of each float (16 + 8 + 8 bits; missing rows and the padding of a
// column to 32 rows hold the largest key, which no value has). Round one counts the top 16
// bits of every value of a feature; each target rank then names its bucket, and the next
// round counts the next 8 bits of the values in those buckets only (at most 256 target
// buckets per feature), and so on. Each round's 65,536 counters fit a CTA's shared memory as
// 16-bit halves, and a CTA takes at most 65,535 rows of one feature, so a half cannot
// overflow; a membership bitmap with prefix counts names a value's bucket.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

#include "host_types.h"

using namespace mpsb;

namespace {

constexpr int kTargets = 256;        // at most max_bins order statistics per feature
constexpr uint32_t kMissingKey = 0xFFFFFFFFu;
constexpr uint32_t kDigits = 65536;  // counters of a round: 2^16 buckets, or 256 slots x 2^8
constexpr uint32_t kErrInf = 1u;      // an Inf in the input
constexpr uint32_t kErrRange = 2u;    // a float64 value outside the float32 range

// Order-preserving image of a float: unsigned order of keys = numeric order of values
// (-0 sorts just below +0; both compare equal as floats, see the transform).
__device__ __forceinline__ uint32_t order_key(float x) {
  const uint32_t b = __float_as_uint(x);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

__device__ __forceinline__ uint64_t quantile_rank(uint64_t part, uint64_t total, uint64_t divisor) {
  const uint64_t whole = part * (total / divisor);  // binned_dataset.cpp:83-95
  const uint64_t numerator = part * (total % divisor);
  return whole + numerator / divisor + (numerator % divisor != 0 ? 1 : 0) - 1;
}

// Input element (row, feature) at byte offset row * rs + feature * cs; returns false with
// an error bit for values the reference rejects.
template <class T, bool ALIGNED>
__device__ __forceinline__ T load_raw(const uint8_t* data, uint64_t rs, uint64_t cs, uint64_t r, uint32_t f) {
  const uint8_t* p = data + r * rs + uint64_t(f) * cs;
  T x;
  if constexpr (ALIGNED) x = __ldg(reinterpret_cast<const T*>(p));
  else memcpy(&x, p, sizeof x);  // a byte at a time
  return x;
}
template <class T>
__device__ __forceinline__ float checked_value(T x, uint32_t* err) {
  if (isnan(x)) return __uint_as_float(0x7FC00000u);
  if (isinf(x)) *err |= kErrInf;
  else if (fabs(x) > T(3.4028234663852886e38)) *err |= kErrRange;
  return float(x);  // correctly rounded, as the host's static_cast
}

// Input matrix -> feature-major order keys (columns of `stride` >= n keys, the rest missing)
// and, where `missing` is given, flags of stride n; through a tile of 128 rows x 32 features,
// so both the row-major reads and the feature-major writes are coalesced. Sixteen loads in
// flight per thread; a CTA takes tiles in turn and adds its missing counts once (added per
// tile, the features' counters, sixteen to a cache line, set the time: 700 us for
// 1,000,000 x 100 with 5 % missing, 338 now; 577 in 32 x 32 tiles).
constexpr uint32_t kKeyRows = 128;
template <class T, bool ALIGNED>
__global__ void __launch_bounds__(256) keys_kernel(const uint8_t* data, uint64_t rs, uint64_t cs, uint32_t n, uint32_t features, size_t stride, uint32_t* keys,
                                                   uint8_t* missing, unsigned long long* miss_count,
                                                   uint32_t* error) {
  __shared__ float tile[kKeyRows][33];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t f0 = blockIdx.y * 32;
  uint32_t err = 0, gone[4] = {};
  // Lanes walk the matrix's contiguous direction: features for row-major input, rows for
  // column-major input (the tile is indexed [row][feature] either way).
  const bool row_major = cs < rs;
  for (uint32_t r0 = blockIdx.x * kKeyRows; r0 < n; r0 += gridDim.x * kKeyRows) {
    T v[16];
#pragma unroll
    for (uint32_t k = 0; k < 16; ++k) {  // past an edge: the last row or feature again, unused
      const uint32_t i = warp * 16 + k;  // row, or (column-major) feature i / 4 and 32 rows
      const uint32_t r = row_major ? i : (i & 3u) * 32 + lane, f = row_major ? lane : i >> 2;
      v[k] = load_raw<T, ALIGNED>(data, rs, cs, min(r0 + r, n - 1), min(f0 + f, features - 1));
    }
#pragma unroll
    for (uint32_t k = 0; k < 16; ++k) {
      const uint32_t i = warp * 16 + k;
      const uint32_t r = row_major ? i : (i & 3u) * 32 + lane, f = row_major ? lane : i >> 2;
      const float x = checked_value<T>(v[k], &err);
      tile[r][f] = r0 + r < n ? x : __uint_as_float(0x7FC00000u);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const uint32_t f = f0 + warp * 4 + q;
      if (f >= features) break;
#pragma unroll
      for (uint32_t k = 0; k < kKeyRows / 32; ++k) {
        const uint32_t r = r0 + k * 32 + lane;
        if (r >= stride) break;
        const float x = tile[k * 32 + lane][warp * 4 + q];
        const bool nan = isnan(x);
        keys[size_t(f) * stride + r] = nan ? kMissingKey : order_key(x);
        if (r < n) {
          if (missing != nullptr) missing[size_t(f) * n + r] = nan ? 1 : 0;
          gone[q] += nan ? 1u : 0u;
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) {
    const uint32_t f = f0 + warp * 4 + q, sum = __reduce_add_sync(0xffffffffu, gone[q]);
    if (lane == 0 && sum) atomicAdd(&miss_count[f], (unsigned long long)sum);
  }
  if (err) atomicOr(error, err);
}

// Rounds of the selection: counts of a digit of one feature's keys over a chunk of its rows
// (at most 65,535: the counters are 16-bit halves). LEVEL 0: the top 16 bits. LEVEL 1 and 2:
// the next 8 bits of the keys whose higher bits are a target's, counted per target bucket
// (slot): the bucket's bit in bits1 (top 16 bits) or bits2 (slot, next 8 bits), its slot the
// set bits before it. hist: [features][kDigits].
// Reads each key once, 64 bytes in flight per thread; 1,000,000 x 100 takes 102, 218 and 205
// us for the three rounds (11 + 11 + 10 bits with global counters and 4-byte loads: 502, 600,
// 680).
constexpr uint32_t kDigitThreads = 1024;
constexpr uint32_t kBitWords = kDigits / 32;
constexpr size_t digit_smem(int level) { return kDigits * 2 + size_t(level) * kBitWords * 6; }

struct BucketSlots {  // in shared memory: membership bits, and the bits set before each word
  uint32_t* bits;
  uint16_t* before;

  // Every thread of the CTA; `warp_sum` holds 33 words.
  __device__ void load(const uint32_t* src, uint32_t* warp_sum) {
    static_assert(kBitWords == 2 * kDigitThreads, "two words per thread");
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint2 w = reinterpret_cast<const uint2*>(src)[threadIdx.x];
    const uint32_t own = __popc(w.x) + __popc(w.y);
    uint32_t incl = own;
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= uint32_t(off)) incl += y;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    uint32_t base = incl - own;
    for (uint32_t q = 0; q < warp; ++q) base += warp_sum[q];
    reinterpret_cast<uint2*>(bits)[threadIdx.x] = w;
    before[2 * threadIdx.x] = uint16_t(base);
    before[2 * threadIdx.x + 1] = uint16_t(base + __popc(w.x));
    __syncthreads();
  }
  __device__ bool find(uint32_t bucket, uint32_t* slot) const {
    const uint32_t w = bits[bucket >> 5], bit = bucket & 31u;
    if (!((w >> bit) & 1u)) return false;
    *slot = before[bucket >> 5] + __popc(w & ((1u << bit) - 1u));
    return true;
  }
};

template <int LEVEL>
__global__ void __launch_bounds__(kDigitThreads, 1) count_digits_kernel(const uint32_t* keys, size_t stride,
                                                                        uint32_t chunk, const uint32_t* bits1,
                                                                        const uint32_t* bits2, uint32_t* hist) {
  extern __shared__ __align__(16) uint32_t cnt[];  // [kDigits / 2], then the bucket tables
  __shared__ uint32_t warp_sum[33];
  const uint32_t f = blockIdx.y, tid = threadIdx.x;
  BucketSlots one, two;
  one.bits = cnt + kDigits / 2;
  one.before = reinterpret_cast<uint16_t*>(one.bits + kBitWords);
  two.bits = reinterpret_cast<uint32_t*>(one.before + kBitWords);
  two.before = reinterpret_cast<uint16_t*>(two.bits + kBitWords);
  for (uint32_t i = tid; i < kDigits / 8; i += kDigitThreads) reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0, 0, 0, 0);
  if (LEVEL >= 1) one.load(bits1 + size_t(f) * kBitWords, warp_sum);
  if (LEVEL >= 2) two.load(bits2 + size_t(f) * kBitWords, warp_sum);
  __syncthreads();
  auto tally = [&](uint32_t k) {
    uint32_t at = k >> 16;
    if (LEVEL >= 1) {
      uint32_t slot;
      if (!one.find(at, &slot)) return;
      at = slot * 256 + ((k >> 8) & 255u);
      if (LEVEL >= 2) {
        if (!two.find(at, &slot)) return;
        at = slot * 256 + (k & 255u);
      }
    }
    atomicAdd(&cnt[at >> 1], 1u << ((at & 1u) * 16));
  };
  const size_t r0 = size_t(blockIdx.x) * chunk;
  const uint32_t quads = r0 < stride ? uint32_t(min(size_t(chunk), stride - r0) / 4) : 0u;
  const uint4* src = reinterpret_cast<const uint4*>(keys + size_t(f) * stride + r0);
  for (uint32_t q0 = tid; q0 < quads; q0 += 4 * kDigitThreads) {
    uint4 v[4];
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
      const uint32_t q = q0 + u * kDigitThreads;
      v[u] = q < quads ? __ldg(src + q) : make_uint4(kMissingKey, kMissingKey, kMissingKey, kMissingKey);
    }
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
      if (q0 + u * kDigitThreads >= quads) break;
      tally(v[u].x);
      tally(v[u].y);
      tally(v[u].z);
      tally(v[u].w);
    }
  }
  __syncthreads();
  uint32_t* out = hist + size_t(f) * kDigits;
  for (uint32_t i = tid; i < kDigits / 2; i += kDigitThreads) {
    const uint32_t w = cnt[i];
    if (w & 0xFFFFu) atomicAdd(out + 2 * i, w & 0xFFFFu);
    if (w >> 16) atomicAdd(out + 2 * i + 1, w >> 16);
  }
}

// Per feature selection state between rounds.
struct Select {
  uint32_t m;                  // non-missing values
  uint32_t n_targets;          // desired (ranks of parts 1..desired-1, then the maximum)
  uint32_t rank[kTargets];     // residual rank inside the current bucket
  uint32_t prefix[kTargets];   // key bits chosen so far
  uint16_t slot[kTargets];     // bucket slot of the current round
};

// Exclusive count of the block's flags before the thread, and the total (flags in the first
// kTargets threads only).
__device__ __forceinline__ uint32_t flags_before(bool flag, uint32_t* warp_sum, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t ballot = __ballot_sync(0xffffffffu, flag);
  if (lane == 0 && warp < kTargets / 32) warp_sum[warp] = uint32_t(__popc(ballot));
  __syncthreads();
  uint32_t before = uint32_t(__popc(ballot & ((1u << lane) - 1u))), all = 0;
#pragma unroll
  for (int w = 0; w < kTargets / 32; ++w) {
    if (w < warp) before += warp_sum[w];
    all += warp_sum[w];
  }
  *total = all;
  __syncthreads();  // warp_sum may be written again
  return before;
}

// After round one: targets, their top-16-bit buckets and residual ranks, slots of the
// distinct buckets (ranks are non-decreasing, so equal buckets are adjacent) and the
// buckets' membership bits. A block per feature: 64 counters at a time are summed by a warp,
// the 1,024 sums scanned, and a warp per target searches them and then its 64 counters.
__global__ void __launch_bounds__(1024) select_top_kernel(const uint32_t* hist, uint32_t max_bins, Select* sel,
                                                          uint32_t* bits) {
  __shared__ uint32_t s_incl[1024], s_warp[32], s_bucket[kTargets], warp_sum[kTargets / 32];
  const uint32_t f = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint2* h = reinterpret_cast<const uint2*>(hist + size_t(f) * kDigits);
  auto pair_of = [&](uint32_t group) {
    uint2 v = __ldg(h + group * 32 + lane);
    if (group == 1023 && lane == 31) v.y = 0;  // the missing keys' bucket
    return v;
  };
  auto inclusive = [&](uint32_t x) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= uint32_t(off)) x += y;
    }
    return x;
  };
  uint32_t own = 0;
#pragma unroll 8
  for (uint32_t g = 0; g < 32; ++g) {
    const uint2 v = pair_of(warp * 32 + g);
    const uint32_t sum = __reduce_add_sync(0xffffffffu, v.x + v.y);
    if (lane == g) own = sum;
  }
  uint32_t incl = inclusive(own);
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t m = 0;
  for (uint32_t q = 0; q < 32; ++q) {
    if (q == warp) incl += m;
    m += s_warp[q];
  }
  s_incl[threadIdx.x] = incl;
  __syncthreads();
  Select& S = sel[f];
  const uint32_t desired = m < max_bins ? m : max_bins;
  if (threadIdx.x == 0) {
    S.m = m;
    S.n_targets = desired;
  }
  for (uint32_t j = warp; j < desired; j += 32) {
    const uint32_t rank = j + 1 < desired ? uint32_t(quantile_rank(j + 1, m, desired)) : m - 1;
    uint32_t lo = 0, hi = 1023;  // first group whose counts pass the rank
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (s_incl[mid] > rank) hi = mid; else lo = mid + 1;
    }
    uint32_t rest = rank - (lo ? s_incl[lo - 1] : 0u);
    const uint2 v = pair_of(lo);
    const uint32_t x = inclusive(v.x + v.y);
    const uint32_t who = uint32_t(__ffs(__ballot_sync(0xffffffffu, x > rest))) - 1u;
    if (lane == who) {
      rest -= x - (v.x + v.y);
      const uint32_t odd = rest >= v.x ? 1u : 0u;
      S.rank[j] = rest - (odd ? v.x : 0u);
      S.prefix[j] = s_bucket[j] = lo * 64 + 2 * lane + odd;
    }
  }
  __syncthreads();
  const uint32_t k = threadIdx.x;
  const bool live = k < desired;
  const bool starts = live && k > 0 && s_bucket[k] != s_bucket[k - 1];
  uint32_t total;
  const uint32_t s = flags_before(starts, warp_sum, &total) + (starts ? 1u : 0u);
  if (live) {
    S.slot[k] = uint16_t(s);
    if (k == 0 || starts) atomicOr(bits + size_t(f) * kBitWords + (s_bucket[k] >> 5), 1u << (s_bucket[k] & 31u));
  }
}

// Selection of rounds two and three, a warp per target: the digit of its slot's 256 counters
// that holds the residual rank, and the rank inside it.
__global__ void __launch_bounds__(256) select_digit_kernel(const uint32_t* hist, Select* sel) {
  const uint32_t f = blockIdx.x;
  Select& S = sel[f];
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t j = blockIdx.y * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (j >= S.n_targets) return;
  const uint4* h = reinterpret_cast<const uint4*>(hist + size_t(f) * kDigits + size_t(S.slot[j]) * 256);
  const uint4 p = __ldg(h + 2 * lane), q = __ldg(h + 2 * lane + 1);
  const uint32_t c[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
  uint32_t own = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) own += c[k];
  uint32_t incl = own;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= uint32_t(off)) incl += y;
  }
  // The lane whose counters hold the rank (a slot's counters hold more values than its ranks).
  uint32_t rest = S.rank[j];
  const uint32_t over = __ballot_sync(0xffffffffu, incl > rest);
  const uint32_t who = over ? uint32_t(__ffs(over)) - 1u : 31u;
  if (lane != who) return;
  rest -= incl - own;
  uint32_t digit = 0;
#pragma unroll
  for (uint32_t k = 0; k < 7; ++k) {
    if (digit == k && rest >= c[k]) {
      rest -= c[k];
      digit = k + 1;
    }
  }
  S.rank[j] = rest;
  S.prefix[j] = (S.prefix[j] << 8) | (who * 8 + digit);
}

// Slots of the distinct 24-bit prefixes after round two (equal prefixes are adjacent) and
// their membership bits: a thread per target, block per feature.
__global__ void __launch_bounds__(kTargets) assign_slots_kernel(Select* sel, uint32_t* bits) {
  __shared__ uint32_t warp_sum[kTargets / 32];
  const uint32_t f = blockIdx.x, k = threadIdx.x;
  Select& S = sel[f];
  const bool live = k < S.n_targets;
  const uint32_t prefix = live ? S.prefix[k] : 0u;
  const bool starts = live && k > 0 && prefix != S.prefix[k - 1];
  uint32_t total;
  const uint32_t s = flags_before(starts, warp_sum, &total) + (starts ? 1u : 0u);
  if (live) {
    const uint32_t bucket = uint32_t(S.slot[k]) * 256 + (prefix & 255u);
    if (k == 0 || starts) atomicOr(bits + size_t(f) * kBitWords + (bucket >> 5), 1u << (bucket & 31u));
    S.slot[k] = uint16_t(s);
  }
}

// Boundaries from the selected order statistics (BuildBoundaries, binned_dataset.cpp:97-118):
// a candidate is kept when below the maximum and above the last kept one, that is above the
// candidate before it (the candidates are non-decreasing). A thread per candidate, block
// per feature.
__global__ void __launch_bounds__(kTargets) finish_kernel(const Select* sel, float* bounds, uint32_t* counts) {
  __shared__ uint32_t warp_sum[kTargets / 32];
  const uint32_t f = blockIdx.x, k = threadIdx.x;
  const Select& S = sel[f];
  const uint32_t nt = S.n_targets;
  bool keep = false;
  float c = 0.0f;
  if (k + 1 < nt) {
    c = key_value(S.prefix[k]);
    keep = c < key_value(S.prefix[nt - 1]) && (k == 0 || c > key_value(S.prefix[k - 1]));
  }
  uint32_t total;
  const uint32_t at = flags_before(keep, warp_sum, &total);
  if (keep) bounds[size_t(f) * kTargets + at] = c;
  if (k == 0) counts[f] = total;
}

// bin = lower_bound(boundaries, value) in float order (so -0 and +0 bin alike): the 255
// boundaries as a search tree in level order (+inf past the last), whose upper levels' few
// nodes lie side by side in different shared-memory banks; the leaf reached is the count of
// boundaries below the value.
constexpr uint32_t kTreeNodes = 256;  // node 0 unused
__device__ __forceinline__ void load_tree(const float* bounds, uint32_t nb, float* tree, uint32_t first,
                                          uint32_t step) {
  for (uint32_t k = first; k < kTreeNodes; k += step) {
    if (k == 0) continue;
    const uint32_t level = 31u - uint32_t(__clz(k));
    const uint32_t at = ((2 * (k - (1u << level)) + 1) << (7 - level)) - 1;  // in order
    tree[k] = at < nb ? bounds[at] : INFINITY;
  }
}
__device__ __forceinline__ uint32_t tree_bin(const float* tree, float x) {
  uint32_t k = 1;
#pragma unroll
  for (int level = 0; level < 8; ++level) k = 2 * k + (tree[k] < x ? 1u : 0u);
  return k - kTreeNodes;
}

// Keys -> the u8 dataset's three copies of the bins (row-major rows of nfb * 32 bytes, column
// blocks, feature-major), missing rows at kMissingSlot: 128 rows of a feature block at a time.
// Each warp bins four features of the tile, 16 keys in flight per lane; the two row layouts
// leave through shared memory in 16-byte pieces. 1,000,000 x 100: 357 us; binning to an
// intermediate copy (750 us) and packing it (327 us) before.
__global__ void __launch_bounds__(256) bin_pack_kernel(const uint32_t* keys, size_t stride, uint32_t n,
                                                       uint32_t features, const float* bounds,
                                                       const uint32_t* counts, uint8_t* out, uint8_t* out_blocked,
                                                       uint8_t* out_fm) {
  constexpr uint32_t kPitch = 36;  // bytes per tile row: nine words, no bank conflicts
  __shared__ float tree[kBlockFeatures][kTreeNodes];
  __shared__ __align__(16) uint8_t tile[128 * kPitch];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t fb = blockIdx.y, nfb = gridDim.y;
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) {
    const uint32_t f = fb * kBlockFeatures + warp * 4 + q;
    if (f < features) load_tree(bounds + size_t(f) * kTargets, counts[f], tree[warp * 4 + q], lane, 32);
  }
  __syncthreads();
  for (uint32_t r0 = blockIdx.x * 128; r0 < n; r0 += gridDim.x * 128) {
    uint32_t key[4][4];
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const uint32_t f = fb * kBlockFeatures + warp * 4 + q;
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t r = r0 + k * 32 + lane;
        key[q][k] = f < features && r < n ? __ldg(keys + size_t(f) * stride + r) : kMissingKey;
      }
    }
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const uint32_t c = warp * 4 + q, f = fb * kBlockFeatures + c;
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t r = k * 32 + lane;
        uint32_t bin = 0;
        if (f < features) {
          bin = key[q][k] == kMissingKey ? uint32_t(kMissingSlot) : tree_bin(tree[c], key_value(key[q][k]));
          if (r0 + r < n) out_fm[size_t(f) * n + r0 + r] = uint8_t(bin);
        }
        tile[r * kPitch + c] = uint8_t(bin);
      }
    }
    __syncthreads();
    const uint32_t r = threadIdx.x >> 1, half = (threadIdx.x & 1u) * 16, row = r0 + r;
    if (row < n) {
      const uint32_t* w = reinterpret_cast<const uint32_t*>(tile + r * kPitch + half);
      const uint4 v = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4*>(out + (size_t(row) * nfb + fb) * kBlockFeatures + half) = v;
      *reinterpret_cast<uint4*>(out_blocked + (size_t(fb) * n + row) * kBlockFeatures + half) = v;
    }
    __syncthreads();
  }
}

// Feature-major bins (missing rows 0) and missing flags of stride n, for the datasets whose
// bins fit u8 but whose missing slot does not (256 bins and missing values).
__global__ void __launch_bounds__(256) transform_kernel(const uint32_t* keys, size_t stride, uint32_t n,
                                                        const float* bounds, const uint32_t* counts,
                                                        uint8_t* bins, uint8_t* missing) {
  __shared__ float tree[kTreeNodes];
  const uint32_t f = blockIdx.y;
  load_tree(bounds + size_t(f) * kTargets, counts[f], tree, threadIdx.x, blockDim.x);
  __syncthreads();
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const uint32_t key = __ldg(keys + size_t(f) * stride + r);
    const bool gone = key == kMissingKey;
    bins[size_t(f) * n + r] = gone ? 0 : uint8_t(tree_bin(tree, key_value(key)));
    missing[size_t(f) * n + r] = gone ? 1 : 0;
  }
}

struct Scratch {
  DevArena mem;
  explicit Scratch(const mpsb_cuda_backend* b) { mem.pool = b->pool; }
  template <class T>
  T* alloc(size_t count) {
    return static_cast<T*>(mem.alloc(count * sizeof(T)));
  }
};

void check_view(const void* data, int scalar_type, uint64_t rows, uint32_t features, uint64_t rs,
                uint64_t cs, uint64_t* extent) {
  if (data == nullptr) throw DataError("Input matrix data must not be null");
  if (rows == 0 || features == 0) throw DataError("Input matrix must contain at least one row and one feature");
  if (scalar_type != 1 && scalar_type != 2) throw DataError("Input scalar type is not supported");
  if (rows >= 0xFFFFFFFFull) throw UnsupportedError("the CUDA backend indexes rows with uint32");
  const uint64_t item = scalar_type == 2 ? 8 : 4;
  if (rs < item || cs < item) throw DataError("Input matrix stride is smaller than the element size");
  uint64_t a, b, c;
  if (__builtin_mul_overflow(rows - 1, rs, &a) || __builtin_mul_overflow(uint64_t(features - 1), cs, &b) ||
      __builtin_add_overflow(a, b, &c) || __builtin_add_overflow(c, item, &c))
    throw DataError("input matrix maximum offset: multiplication overflow");
  *extent = c;
}

// Order keys of an uploaded matrix: columns of `stride` keys and, for more than 256 bins,
// missing flags.
struct Keys {
  uint32_t* keys = nullptr;
  uint8_t* missing = nullptr;
  size_t stride = 0;
  uint32_t n = 0, features = 0;
  std::vector<uint64_t> missing_count;
};

// Upload the matrix and turn it into keys. wide: unpadded columns, with missing flags.
Keys make_keys(mpsb_cuda_backend* b, Scratch& ss, const void* data, int scalar_type, uint64_t rows,
               uint32_t features, uint64_t rs, uint64_t cs, bool wide) {
  uint64_t extent = 0;
  check_view(data, scalar_type, rows, features, rs, cs, &extent);
  cudaStream_t s = b->stream;
  uint8_t* raw = ss.alloc<uint8_t>(extent);
  CK(cudaMemcpyAsync(raw, data, extent, cudaMemcpyHostToDevice, s));
  Keys k;
  k.n = uint32_t(rows);
  k.features = features;
  k.stride = wide ? rows : (rows + 31) / 32 * 32;
  k.keys = ss.alloc<uint32_t>(k.stride * features);
  if (wide) k.missing = ss.alloc<uint8_t>(size_t(rows) * features);
  unsigned long long* miss = ss.alloc<unsigned long long>(features);
  CK(cudaMemsetAsync(miss, 0, features * sizeof(unsigned long long), s));
  CK(cudaMemsetAsync(b->error.p, 0, sizeof(uint32_t), s));
  const uint32_t blocks = (features + 31) / 32;
  const dim3 grid(std::max(1u, std::min(uint32_t((rows + kKeyRows - 1) / kKeyRows), uint32_t(b->sm_count) * 8 / blocks + 1)),
                  blocks);
  // Strides of whole elements (the upload starts aligned): one load per value.
  const uint64_t size = scalar_type == 1 ? 4 : 8;
  const bool aligned = rs % size == 0 && cs % size == 0;
  auto kernel = scalar_type == 1 ? (aligned ? keys_kernel<float, true> : keys_kernel<float, false>)
                                 : (aligned ? keys_kernel<double, true> : keys_kernel<double, false>);
  kernel<<<grid, 256, 0, s>>>(raw, rs, cs, k.n, features, k.stride, k.keys, k.missing, miss, b->error.as<uint32_t>());
  CK(cudaGetLastError());
  k.missing_count.assign(features, 0);
  CK(cudaMemcpyAsync(k.missing_count.data(), miss, features * sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
  const uint32_t e = b->take_error();  // synchronizes the stream
  if (e & kErrInf) throw DataError("Input matrix contains Inf");
  if (e & kErrRange) throw DataError("float64 input value exceeds the finite float32 range");
  return k;
}

// The counting passes of a selection over u8 bins: chunks of one feature, enough for two CTAs
// per SM where the rows allow, at most 65,535 rows each.
template <int LEVEL>
void count_digits(mpsb_cuda_backend* b, const Keys& k, const uint32_t* bits1, const uint32_t* bits2, uint32_t* hist) {
  static std::atomic<unsigned long long> configured{0};  // one bit per device
  CK(opt_in_dynamic_smem(configured, count_digits_kernel<LEVEL>, digit_smem(LEVEL)));
  const size_t want = (k.stride * k.features + 2 * size_t(b->sm_count) - 1) / (2 * size_t(b->sm_count));
  const uint32_t chunk = uint32_t(std::min<size_t>(65504, std::max<size_t>(4096, (want + 31) / 32 * 32)));
  const dim3 grid(uint32_t((k.stride + chunk - 1) / chunk), k.features);
  count_digits_kernel<LEVEL><<<grid, kDigitThreads, digit_smem(LEVEL), b->stream>>>(k.keys, k.stride, chunk, bits1,
                                                                                 bits2, hist);
  CK(cudaGetLastError());
}

// A resident dataset's host tables and its per-feature device arrays, without bins.
mpsb_cuda_dataset* start_dataset(mpsb_cuda_backend* b, uint32_t rows, uint32_t features,
                                 std::vector<uint32_t> bin_count, std::vector<uint64_t> missing_count) {
  cudaStream_t s = b->stream;
  std::unique_ptr<mpsb_cuda_dataset> d(new mpsb_cuda_dataset);
  d->backend = b;
  d->n_rows = rows;
  d->features = features;
  d->nfb = (features + kBlockFeatures - 1) / kBlockFeatures;
  d->h_bin_count = std::move(bin_count);
  d->h_has_missing.assign(features, 0);
  for (uint32_t f = 0; f < features; ++f) d->h_has_missing[f] = missing_count[f] ? 1 : 0;
  // 256 bins and missing values in one feature: the wide layout's missing slot.
  d->slots = dataset_slots(d->h_bin_count.data(), d->h_has_missing.data(), features);
  d->missing_count = std::move(missing_count);
  d->bin_count.alloc(features * sizeof(uint32_t));
  d->has_missing.alloc(features);
  CK(cudaMemcpyAsync(d->bin_count.p, d->h_bin_count.data(), features * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(d->has_missing.p, d->h_has_missing.data(), features, cudaMemcpyHostToDevice, s));
  return d.release();
}

// The dataset of feature-major bins (u8 or u16: `width` bytes) and missing flags.
mpsb_cuda_dataset* finish_packed(mpsb_cuda_backend* b, std::unique_ptr<mpsb_cuda_dataset> d, const void* bins_fm,
                               uint32_t width, const uint8_t* missing) {
  const uint32_t rows = d->n_rows, features = d->features;
  if (d->slots == uint32_t(kSlots)) {  // more than 256 bins asked for, no feature has them
    d->bins.alloc(size_t(d->nfb) * rows * kBlockFeatures);
    d->bins_blocked.alloc(size_t(d->nfb) * rows * kBlockFeatures);
    d->bins_fm.alloc(size_t(features) * rows);
    CK(launch_pack_bins(bins_fm, width, missing, d->bin_count.as<uint32_t>(), rows, features, d->nfb,
                        d->bins.as<uint8_t>(), d->bins_blocked.as<uint8_t>(), d->bins_fm.as<uint8_t>(),
                        b->error.as<uint32_t>(), b->stream));
    if (b->take_error()) throw DataError("Binned value exceeds the feature histogram range");
    attach_bins_tmap(d.get());
    return d.release();
  }
  d->bins16.alloc(size_t(d->nfb) * rows * kBlockFeatures * sizeof(uint16_t));
  d->bins16_fm.alloc(size_t(features) * rows * sizeof(uint16_t));
  for (uint32_t fb = 0; fb < d->nfb; ++fb) {
    const size_t first = size_t(fb) * kBlockFeatures * rows;
    CK(launch_pack_bins16_block(static_cast<const uint8_t*>(bins_fm) + first * width, width, missing + first,
                                d->bin_count.as<uint32_t>(), rows, features, fb, d->slots, d->bins16.as<uint16_t>(),
                                d->bins16_fm.as<uint16_t>(), b->error.as<uint32_t>(), b->stream));
  }
  if (b->take_error()) throw DataError("Binned value exceeds the feature histogram range");
  return d.release();
}

// The dataset of at most 256 bins a feature from its keys and boundaries ([features][kTargets]
// with their counts, on the device).
mpsb_cuda_dataset* finish_narrow(mpsb_cuda_backend* b, Scratch& ss, const Keys& k, const float* bounds,
                                 const uint32_t* counts, std::vector<uint32_t> bin_count) {
  std::unique_ptr<mpsb_cuda_dataset> d(start_dataset(b, k.n, k.features, std::move(bin_count), k.missing_count));
  cudaStream_t s = b->stream;
  const uint32_t n = k.n;
  if (d->slots != uint32_t(kSlots)) {
    uint8_t* bins_fm = ss.alloc<uint8_t>(size_t(k.features) * n);
    uint8_t* missing = ss.alloc<uint8_t>(size_t(k.features) * n);
    const dim3 grid(std::max(1u, std::min((n + 255) / 256, uint32_t(b->sm_count) * 8 / k.features + 1)), k.features);
    transform_kernel<<<grid, 256, 0, s>>>(k.keys, k.stride, n, bounds, counts, bins_fm, missing);
    CK(cudaGetLastError());
    return finish_packed(b, std::move(d), bins_fm, 1, missing);
  }
  d->bins.alloc(size_t(d->nfb) * n * kBlockFeatures);
  d->bins_blocked.alloc(size_t(d->nfb) * n * kBlockFeatures);
  d->bins_fm.alloc(size_t(k.features) * n);
  const dim3 grid(std::max(1u, std::min((n + 127) / 128, uint32_t(b->sm_count) * 6 / d->nfb + 1)), d->nfb);
  bin_pack_kernel<<<grid, 256, 0, s>>>(k.keys, k.stride, n, k.features, bounds, counts, d->bins.as<uint8_t>(),
                                       d->bins_blocked.as<uint8_t>(), d->bins_fm.as<uint8_t>());
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(s));
  attach_bins_tmap(d.get());
  return d.release();
}

// ---- More than 256 bins per feature -------------------------------------------------
// The selection above keeps one target slot per boundary (at most 256). Wide schemas
// sort each feature's order keys instead (a stable LSD radix sort, eight passes of 4-bit
// digits, every feature in the same launches) and read the order statistics at their
// ranks; missing rows carry the key 0xFFFFFFFF, above every finite value's, so they sort
// last and the first m keys of a feature are its non-missing values in order.
constexpr int kSortThreads = 256;
constexpr uint32_t kSortTile = 4096;  // keys per (feature, tile) block

// Digit counts of one (tile, feature): cnt[(f * 16 + digit) * tiles + tile].
__global__ void __launch_bounds__(kSortThreads) sort_count_kernel(const uint32_t* keys, uint32_t n,
                                                                  uint32_t tiles, int shift, uint32_t* cnt) {
  __shared__ uint32_t c[16];
  const uint32_t f = blockIdx.y, t = blockIdx.x;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 16) c[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t* k = keys + size_t(f) * n;
  const uint32_t lo = t * kSortTile, hi = min(n, lo + kSortTile);
  uint32_t mine = 0;  // lane v < 16 counts digit v for its warp
  for (uint32_t base = lo + (threadIdx.x & ~31u); base < hi; base += kSortThreads) {
    const uint32_t i = base + uint32_t(lane);
    const bool valid = i < hi;
    const uint32_t d = valid ? (k[i] >> shift) & 15u : 16u;
#pragma unroll
    for (uint32_t v = 0; v < 16; ++v) {
      const uint32_t m = __ballot_sync(0xffffffffu, d == v);
      if (uint32_t(lane) == v) mine += uint32_t(__popc(m));
    }
  }
  if (lane < 16 && mine) atomicAdd(&c[lane], mine);
  __syncthreads();
  if (threadIdx.x < 16) cnt[(size_t(f) * 16 + threadIdx.x) * tiles + t] = c[threadIdx.x];
}

// Exclusive prefix of one feature's counts in (digit, tile) order, in place.
__global__ void __launch_bounds__(1024) sort_scan_kernel(uint32_t* cnt, uint32_t tiles) {
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t carry;
  const uint32_t f = blockIdx.x;
  uint32_t* c = cnt + size_t(f) * 16 * tiles;
  const uint32_t total = 16 * tiles;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t base = 0; base < total; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < total ? c[i] : 0u;
    uint32_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      const uint32_t w = lane < int(blockDim.x >> 5) ? warp_sum[lane] : 0u;
      uint32_t z = w;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, z, off);
        if (lane >= off) z += y;
      }
      warp_sum[lane] = z - w;  // exclusive
    }
    __syncthreads();
    const uint32_t before = carry;
    if (i < total) c[i] = before + warp_sum[warp] + x - v;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = before + warp_sum[warp] + x;
    __syncthreads();
  }
}

// Stable scatter of one (tile, feature) by the digit at `shift`: the tile's keys in
// rounds of kSortThreads; a key's place is its digit's offset for the tile, plus the
// earlier keys of the tile with that digit (previous rounds, earlier warps of the round,
// lower lanes of its warp).
__global__ void __launch_bounds__(kSortThreads) sort_scatter_kernel(const uint32_t* in, uint32_t* out,
                                                                    uint32_t n, uint32_t tiles, int shift,
                                                                    const uint32_t* off) {
  constexpr int W = kSortThreads / 32;
  __shared__ uint32_t run[16];
  __shared__ uint32_t wcount[W][16];
  const uint32_t f = blockIdx.y, t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 16) run[threadIdx.x] = off[(size_t(f) * 16 + threadIdx.x) * tiles + t];
  const uint32_t* k = in + size_t(f) * n;
  uint32_t* o = out + size_t(f) * n;
  const uint32_t lo = t * kSortTile, hi = min(n, lo + kSortTile);
  const uint32_t lt = (1u << lane) - 1u;
  __syncthreads();
  for (uint32_t base = lo; base < hi; base += kSortThreads) {
    const uint32_t i = base + threadIdx.x;
    const bool valid = i < hi;
    const uint32_t key = valid ? k[i] : 0u;
    const uint32_t d = valid ? (key >> shift) & 15u : 16u;
    uint32_t rank = 0;
#pragma unroll
    for (uint32_t v = 0; v < 16; ++v) {
      const uint32_t m = __ballot_sync(0xffffffffu, d == v);
      if (d == v) rank = uint32_t(__popc(m & lt));
      if (uint32_t(lane) == v) wcount[warp][v] = uint32_t(__popc(m));
    }
    __syncthreads();
    if (valid) {
      uint32_t before = run[d] + rank;
      for (int w = 0; w < warp; ++w) before += wcount[w][d];
      if (before < n) o[before] = key;  // always: the counts come from the same keys
    }
    __syncthreads();
    if (threadIdx.x < 16) {
      uint32_t sum = 0;
      for (int w = 0; w < W; ++w) sum += wcount[w][threadIdx.x];
      run[threadIdx.x] += sum;
    }
    __syncthreads();
  }
}

// Boundaries of one feature from its sorted keys (BuildBoundaries, binned_dataset.cpp:
// 97-118): candidate p (1 <= p < desired) is the value at rank QuantileRank(p, m, desired)
// and is kept when below the maximum and above the previous candidate. The candidates are
// non-decreasing, so "above the last kept boundary" is "above the previous candidate" for
// every candidate below the maximum. A block per feature; kept candidates are compacted
// in order by a block prefix sum.
__global__ void __launch_bounds__(1024) wide_bounds_kernel(const uint32_t* sorted, uint32_t n,
                                                           const uint64_t* miss_count, uint32_t max_bins,
                                                           float* bounds, uint32_t* counts) {
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t carry;
  const uint32_t f = blockIdx.x;
  const uint32_t* k = sorted + size_t(f) * n;
  const uint32_t m = n - uint32_t(miss_count[f]);
  const uint32_t desired = m < max_bins ? m : max_bins;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const float maximum = m ? key_value(k[m - 1]) : 0.0f;
  const uint32_t parts = desired > 1 ? desired - 1 : 0;  // candidates p = 1 .. desired - 1
  float* out = bounds + size_t(f) * (max_bins - 1);
  for (uint32_t base = 0; base < parts; base += blockDim.x) {
    const uint32_t p = base + threadIdx.x + 1;
    bool keep = false;
    float c = 0.0f;
    if (p <= parts) {
      c = key_value(k[quantile_rank(p, m, desired)]);
      keep = c < maximum && (p == 1 || c > key_value(k[quantile_rank(p - 1, m, desired)]));
    }
    const uint32_t ballot = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) warp_sum[warp] = uint32_t(__popc(ballot));
    __syncthreads();
    if (warp == 0) {
      const uint32_t w = lane < int(blockDim.x >> 5) ? warp_sum[lane] : 0u;
      uint32_t z = w;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, z, off);
        if (lane >= off) z += y;
      }
      warp_sum[lane] = z - w;
    }
    __syncthreads();
    const uint32_t before = carry;
    if (keep) out[before + warp_sum[warp] + uint32_t(__popc(ballot & ((1u << lane) - 1u)))] = c;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = before + warp_sum[warp] + uint32_t(__popc(ballot));
    __syncthreads();
  }
  if (threadIdx.x == 0) counts[f] = carry;
}

// Wide transform: bin = lower_bound over the feature's boundaries (global memory, up to
// 65535 per feature at bounds + f * stride); missing rows get bin 0 (their flag marks them).
__global__ void transform_wide_kernel(const uint32_t* keys, const uint8_t* missing, uint32_t n,
                                      const float* bounds, size_t stride, const uint32_t* counts,
                                      uint16_t* bins) {
  const uint32_t f = blockIdx.y;
  const uint32_t nb = counts[f];
  const float* b = bounds + size_t(f) * stride;
  const size_t base = size_t(f) * n;
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    uint32_t bin = 0;
    if (!missing[base + r]) {
      const float x = key_value(keys[base + r]);
      uint32_t lo = 0, hi = nb;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(b + mid) < x) lo = mid + 1; else hi = mid;
      }
      bin = lo;
    }
    bins[base + r] = uint16_t(bin);
  }
}

// Sorts every feature's keys (missing rows last) into `sorted`; `tmp` is a buffer of the
// same size. Eight passes, the first out of the keys: the last one ends in `sorted`.
void sort_feature_keys(cudaStream_t s, Scratch& ss, const uint32_t* keys, uint32_t n, uint32_t features,
                       uint32_t* sorted, uint32_t* tmp) {
  const uint32_t tiles = (n + kSortTile - 1) / kSortTile;
  uint32_t* cnt = ss.alloc<uint32_t>(size_t(features) * 16 * tiles);
  const uint32_t* in = keys;
  uint32_t* out = tmp;
  for (int shift = 0; shift < 32; shift += 4) {
    sort_count_kernel<<<dim3(tiles, features), kSortThreads, 0, s>>>(in, n, tiles, shift, cnt);
    CK(cudaGetLastError());
    sort_scan_kernel<<<features, 1024, 0, s>>>(cnt, tiles);
    CK(cudaGetLastError());
    sort_scatter_kernel<<<dim3(tiles, features), kSortThreads, 0, s>>>(in, out, n, tiles, shift, cnt);
    CK(cudaGetLastError());
    in = out;
    out = out == tmp ? sorted : tmp;
  }
}

// QuantizeDense for max_bins > 256 on the device: u16 feature-major bins in `bins_fm`,
// boundaries [features][max_bins - 1] in `bounds` with their counts.
void quantize_wide(cudaStream_t s, Scratch& ss, const uint32_t* keys,
                   const std::vector<uint64_t>& missing_count, uint32_t n, uint32_t features,
                   uint32_t max_bins, float* bounds, uint32_t* counts, uint16_t* bins_fm) {
  const size_t cells = size_t(n) * features;
  uint32_t* sorted = ss.alloc<uint32_t>(cells);
  uint32_t* tmp = ss.alloc<uint32_t>(cells);
  sort_feature_keys(s, ss, keys, n, features, sorted, tmp);
  uint64_t* d_miss = ss.alloc<uint64_t>(features);
  CK(cudaMemcpyAsync(d_miss, missing_count.data(), features * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
  wide_bounds_kernel<<<features, 1024, 0, s>>>(sorted, n, d_miss, max_bins, bounds, counts);
  CK(cudaGetLastError());
}

// The device's feature-major copy as the reference lays bins out: missing rows (at the
// dataset's missing slot) become bin 0 plus a flag.
template <typename T>
void export_bins(const mpsb_cuda_dataset* d, T* bins, uint8_t* missing) {
  dataset_ready(d);
  d->backend->activate();
  cudaStream_t s = d->backend->stream;
  const size_t cells = size_t(d->n_rows) * d->features;
  const bool wide = d->slots != uint32_t(kSlots);
  std::vector<uint16_t> b16(wide ? cells : 0);
  std::vector<uint8_t> b8(wide ? 0 : cells);
  if (wide)
    CK(cudaMemcpyAsync(b16.data(), d->bins16_fm.p, cells * sizeof(uint16_t), cudaMemcpyDeviceToHost, s));
  else
    CK(cudaMemcpyAsync(b8.data(), d->bins_fm.p, cells, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  const uint32_t missing_slot = d->slots - 1;
  for (uint32_t f = 0; f < d->features; ++f) {
    for (uint32_t r = 0; r < d->n_rows; ++r) {
      const size_t i = size_t(f) * d->n_rows + r;
      const uint32_t v = wide ? uint32_t(b16[i]) : uint32_t(b8[i]);
      const bool miss = d->h_has_missing[f] && v == missing_slot;
      if (missing) missing[i] = miss ? 1 : 0;
      bins[i] = T(miss ? 0u : v);
    }
  }
}

}  // namespace

extern "C" {

int mpsb_cuda_dataset_quantize(mpsb_cuda_backend* b, const void* data, int scalar_type,
                               uint64_t rows, uint32_t features, uint64_t row_stride,
                               uint64_t col_stride, uint32_t max_bins, mpsb_cuda_dataset** out) {
  return guard([&] {
    if (!b || !out) throw TrainingError("null argument");
    if (max_bins < 2 || max_bins > 65536) throw DataError("max_bins must be in [2, 65536]");
    if (features > 65535) throw UnsupportedError("device binning takes at most 65535 features");
    b->activate();
    cudaStream_t s = b->stream;
    Scratch ss(b);
    const bool wide = max_bins > uint32_t(kTargets);
    Keys k = make_keys(b, ss, data, scalar_type, rows, features, row_stride, col_stride, wide);
    const uint32_t n = k.n;
    // Schema on the host: per feature the boundary count and `stride` boundary slots.
    std::vector<uint32_t> h_counts(features);
    std::vector<float> h_bounds;
    size_t stride = 0;
    std::unique_ptr<mpsb_cuda_dataset> d;
    if (wide) {
      stride = max_bins - 1;
      float* bounds = ss.alloc<float>(size_t(features) * stride);
      uint32_t* counts = ss.alloc<uint32_t>(features);
      uint16_t* bins16 = ss.alloc<uint16_t>(size_t(features) * n);
      quantize_wide(s, ss, k.keys, k.missing_count, n, features, max_bins, bounds, counts, bins16);
      const dim3 grid(std::max(1u, std::min((n + 255) / 256, uint32_t(b->sm_count) * 4 / std::max(1u, features) + 1)),
                      features);
      transform_wide_kernel<<<grid, 256, 0, s>>>(k.keys, k.missing, n, bounds, stride, counts, bins16);
      CK(cudaGetLastError());
      h_bounds.resize(size_t(features) * stride);
      CK(cudaMemcpyAsync(h_counts.data(), counts, features * 4, cudaMemcpyDeviceToHost, s));
      CK(cudaMemcpyAsync(h_bounds.data(), bounds, h_bounds.size() * 4, cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      std::vector<uint32_t> bin_count(features);
      for (uint32_t f = 0; f < features; ++f) bin_count[f] = h_counts[f] + 1;
      d.reset(start_dataset(b, n, features, bin_count, k.missing_count));
      d.reset(finish_packed(b, std::move(d), bins16, 2, k.missing));
    } else {
      // Three rounds' counters and two rounds' membership bits, cleared together.
      const size_t digits = size_t(features) * kDigits, words = size_t(features) * kBitWords;
      uint32_t* hist = ss.alloc<uint32_t>(3 * digits + 2 * words);
      uint32_t *bits1 = hist + 3 * digits, *bits2 = bits1 + words;
      Select* sel = ss.alloc<Select>(features);
      float* bounds = ss.alloc<float>(size_t(features) * kTargets);
      uint32_t* counts = ss.alloc<uint32_t>(features);
      CK(cudaMemsetAsync(hist, 0, (3 * digits + 2 * words) * sizeof(uint32_t), s));
      const dim3 targets(features, kTargets / 8);  // eight targets (warps) per block
      count_digits<0>(b, k, nullptr, nullptr, hist);
      select_top_kernel<<<features, 1024, 0, s>>>(hist, max_bins, sel, bits1);
      CK(cudaGetLastError());
      count_digits<1>(b, k, bits1, nullptr, hist + digits);
      select_digit_kernel<<<targets, 256, 0, s>>>(hist + digits, sel);
      CK(cudaGetLastError());
      assign_slots_kernel<<<features, kTargets, 0, s>>>(sel, bits2);
      CK(cudaGetLastError());
      count_digits<2>(b, k, bits1, bits2, hist + 2 * digits);
      select_digit_kernel<<<targets, 256, 0, s>>>(hist + 2 * digits, sel);
      CK(cudaGetLastError());
      finish_kernel<<<features, kTargets, 0, s>>>(sel, bounds, counts);
      CK(cudaGetLastError());
      // Schema back to the host.
      stride = kTargets;
      h_bounds.resize(size_t(features) * kTargets);
      std::vector<Select> h_sel(features);
      CK(cudaMemcpyAsync(h_counts.data(), counts, features * 4, cudaMemcpyDeviceToHost, s));
      CK(cudaMemcpyAsync(h_bounds.data(), bounds, h_bounds.size() * 4, cudaMemcpyDeviceToHost, s));
      CK(cudaMemcpyAsync(h_sel.data(), sel, features * sizeof(Select), cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      std::vector<uint32_t> bin_count(features);
      for (uint32_t f = 0; f < features; ++f) {
        bin_count[f] = h_counts[f] + 1;
        if (k.missing_count[f] + h_sel[f].m != rows) throw BackendError("device binning lost rows");
      }
      d.reset(finish_narrow(b, ss, k, bounds, counts, bin_count));
    }
    d->max_bins = max_bins;
    d->boundary_offset.resize(features);
    uint64_t off = 0;
    for (uint32_t f = 0; f < features; ++f) {
      d->boundary_offset[f] = off;
      d->boundaries.insert(d->boundaries.end(), h_bounds.begin() + size_t(f) * stride,
                           h_bounds.begin() + size_t(f) * stride + h_counts[f]);
      off += h_counts[f];
    }
    d->boundary_count = h_counts;
    d->has_schema = true;
    *out = d.release();
  });
}

int mpsb_cuda_dataset_transform(mpsb_cuda_backend* b, const mpsb_cuda_dataset* schema,
                                const void* data, int scalar_type, uint64_t rows,
                                uint32_t features, uint64_t row_stride, uint64_t col_stride,
                                mpsb_cuda_dataset** out) {
  return guard([&] {
    if (!b || !schema || !out) throw TrainingError("null argument");
    dataset_ready(schema);
    if (!schema->has_schema) throw TrainingError("the schema dataset holds no bin boundaries");
    if (features != schema->features)
      throw DataError("Prediction input feature count does not match the binned schema");
    b->activate();
    cudaStream_t s = b->stream;
    Scratch ss(b);
    const bool wide = schema->max_bins > uint32_t(kTargets);
    Keys k = make_keys(b, ss, data, scalar_type, rows, features, row_stride, col_stride, wide);
    const uint32_t n = k.n;
    const size_t stride = wide ? schema->max_bins - 1 : size_t(kTargets);
    std::vector<float> h_bounds(size_t(features) * stride, 0.0f);
    for (uint32_t f = 0; f < features; ++f)
      std::copy(schema->boundaries.begin() + schema->boundary_offset[f],
                schema->boundaries.begin() + schema->boundary_offset[f] + schema->boundary_count[f],
                h_bounds.begin() + size_t(f) * stride);
    float* bounds = ss.alloc<float>(h_bounds.size());
    uint32_t* counts = ss.alloc<uint32_t>(features);
    CK(cudaMemcpyAsync(bounds, h_bounds.data(), h_bounds.size() * 4, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(counts, schema->boundary_count.data(), features * 4, cudaMemcpyHostToDevice, s));
    const dim3 grid(std::max(1u, std::min((n + 255) / 256, uint32_t(b->sm_count) * 4 / std::max(1u, features) + 1)),
                    features);
    std::unique_ptr<mpsb_cuda_dataset> d;
    if (wide) {
      uint16_t* bins16 = ss.alloc<uint16_t>(size_t(features) * n);
      transform_wide_kernel<<<grid, 256, 0, s>>>(k.keys, k.missing, n, bounds, stride, counts, bins16);
      CK(cudaGetLastError());
      d.reset(start_dataset(b, n, features, schema->h_bin_count, k.missing_count));
      d.reset(finish_packed(b, std::move(d), bins16, 2, k.missing));
    } else {
      d.reset(finish_narrow(b, ss, k, bounds, counts, schema->h_bin_count));
    }
    d->max_bins = schema->max_bins;
    d->boundaries = schema->boundaries;
    d->boundary_offset = schema->boundary_offset;
    d->boundary_count = schema->boundary_count;
    d->has_schema = true;
    *out = d.release();
  });
}

uint64_t mpsb_cuda_dataset_boundary_total(const mpsb_cuda_dataset* d) {
  return d ? d->boundaries.size() : 0;
}

int mpsb_cuda_dataset_schema(const mpsb_cuda_dataset* d, float* boundaries,
                             uint64_t* boundary_offset, uint32_t* boundary_count,
                             uint32_t* bin_count, uint64_t* missing_count) {
  return guard([&] {
    if (!d) throw TrainingError("null argument");
    if (!d->has_schema) throw TrainingError("the dataset holds no bin boundaries");
    if (boundaries) std::copy(d->boundaries.begin(), d->boundaries.end(), boundaries);
    if (boundary_offset) std::copy(d->boundary_offset.begin(), d->boundary_offset.end(), boundary_offset);
    if (boundary_count) std::copy(d->boundary_count.begin(), d->boundary_count.end(), boundary_count);
    if (bin_count) std::copy(d->h_bin_count.begin(), d->h_bin_count.end(), bin_count);
    if (missing_count) std::copy(d->missing_count.begin(), d->missing_count.end(), missing_count);
  });
}

int mpsb_cuda_dataset_export(const mpsb_cuda_dataset* d, uint8_t* bins, uint8_t* missing) {
  return guard([&] {
    if (!d || !bins) throw TrainingError("null argument");
    for (uint32_t f = 0; f < d->features; ++f)
      if (d->h_bin_count[f] > 256)
        throw UnsupportedError("the dataset has more than 256 bins per feature: export it as u16");
    export_bins(d, bins, missing);
  });
}

int mpsb_cuda_dataset_export16(const mpsb_cuda_dataset* d, uint16_t* bins, uint8_t* missing) {
  return guard([&] {
    if (!d || !bins) throw TrainingError("null argument");
    export_bins(d, bins, missing);
  });
}

}  // extern "C"
