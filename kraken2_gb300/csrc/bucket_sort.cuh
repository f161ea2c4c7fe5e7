// Sorts many buckets of 64-bit keys at once, a thread block to a bucket in
// shared memory, and drops repeats: the library build's sequence blocks and
// the -K counters' hash ranges.
//
// A bucket's keys go to shared memory by zone -- 4,096 of them, in the order
// the caller wants first, spread as evenly as the keys allow (a hash, uniform
// bits), so that a zone holds about one key and a thread sorts a zone by
// insertion.  Two passes over the keys and one over the zones: about two warp
// instructions a key (with 256 zones, ranked by a warp each, it was thirteen).
// Zones of more than kThreadZone keys -- repeats, uneven keys -- are ranked
// by a warp.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "k2g_device.cuh"
#include "radix_sort.cuh"

namespace k2g {
namespace {

constexpr int kSortThreads = 512;
constexpr int kZones = 4096;
constexpr uint32_t kThreadZone = 20;      // keys of a zone sorted by one thread
constexpr uint32_t kSmallBlock = 8064;    // keys; three thread blocks to an SM
constexpr uint32_t kLargeBlock = 25600;   // 200 KB of keys
constexpr uint32_t kBigZones = kLargeBlock / (kThreadZone + 1) + 1;

// Keys, zone ends (16 bits each), big zones.
inline size_t bucket_sort_smem(uint32_t cap) {
  return (size_t)cap * 8 + kZones * 2 + (cap / (kThreadZone + 1) + 1) * 2 + 16;
}

struct ZoneMurmur {   // MurmurHash3 mod 256, then the key's four top bits
  int shift;
  __device__ __forceinline__ uint32_t operator()(uint64_t key) const {
    return ((uint32_t)murmur3(key) & 0xFFu) << 4 | ((uint32_t)(key >> shift) & 15u);
  }
};
struct ZoneBits {     // twelve bits of the key
  int shift;
  __device__ __forceinline__ uint32_t operator()(uint64_t key) const { return (uint32_t)(key >> shift) & 0xFFFu; }
};

constexpr uint64_t kNoKey = ~0ull;   // (no key has all bits set)

// One thread: a zone's keys in order, repeats dropped (kNoKey behind them).
__device__ __forceinline__ void sort_zone(uint64_t *z, uint32_t m) {
  uint32_t d = 1;
  for (uint32_t i = 1; i < m; i++) {
    const uint64_t x = z[i];
    uint32_t j = d;
    uint64_t y = 0;
    while (j && (y = z[j - 1]) > x) j--;
    if (j && y == x) continue;
    for (uint32_t t = d; t > j; t--) z[t] = z[t - 1];
    z[j] = x;
    d++;
  }
  for (; d < m; d++) z[d] = kNoKey;
}

// One warp: the same for a zone of any size.  Most are large by repeats of a few
// keys, which are taken out first, one after another, as long as each makes up a
// sixteenth of what is left (28M keys of 10,000 distinct ones 5.69 -> 0.81 ms); the
// rest and one of each are sorted by a bitonic sort whose every exchange puts the
// lesser key first (keys past m count as the greatest); kNoKey takes the place of
// repeats.
__device__ __forceinline__ void sort_big_zone(uint64_t *z, uint32_t m) {
  const uint32_t lane = threadIdx.x & 31;
  {
    uint32_t left = m, taken = 0, gone = m;
    uint64_t mine = kNoKey;   // lane i: the i-th key taken out
    while (left > 32 && taken < 32 && gone * 16 >= left) {
      const uint64_t key = z[0];
      __syncwarp();
      uint32_t kept = 0;
      for (uint32_t i0 = 0; i0 < left; i0 += 32) {
        const uint64_t x = i0 + lane < left ? z[i0 + lane] : key;
        const uint32_t others = __ballot_sync(0xffffffffu, x != key);
        if (x != key) z[kept + __popc(others & ((1u << lane) - 1))] = x;
        kept += __popc(others);
        __syncwarp();
      }
      if (lane == taken) mine = key;
      taken++;
      gone = left - kept;
      left = kept;
    }
    if (lane < taken) z[left + lane] = mine;
    for (uint32_t i = left + taken + lane; i < m; i += 32) z[i] = kNoKey;
    m = left + taken;
    __syncwarp();
  }
  auto exchange = [&](uint32_t a, uint32_t b) {
    if (b >= m) return;
    const uint64_t x = z[a], y = z[b];
    if (x > y) {
      z[a] = y;
      z[b] = x;
    }
  };
  uint32_t half = 1;   // half of m, as a power of two
  while (2 * half < m) half *= 2;
  for (uint32_t k = 1; k <= half; k *= 2) {
    // runs of k are sorted: the second of each two runs backwards, then both apart
    for (uint32_t i = lane; i < half; i += 32) {
      const uint32_t t = i & (k - 1), run = (i - t) * 2;
      exchange(run + t, run + 2 * k - 1 - t);
    }
    __syncwarp();
    for (uint32_t j = k / 2; j; j /= 2) {
      for (uint32_t i = lane; i < half; i += 32) {
        const uint32_t t = i & (j - 1), run = (i - t) * 2;
        exchange(run + t, run + t + j);
      }
      __syncwarp();
    }
  }
  uint64_t last = kNoKey;
  for (uint32_t i0 = 0; i0 < m; i0 += 32) {
    const uint64_t x = i0 + lane < m ? z[i0 + lane] : kNoKey;
    uint64_t before = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) before = last;
    last = __shfl_sync(0xffffffffu, x, 31);
    if (x == before && i0 + lane < m) z[i0 + lane] = kNoKey;
  }
}

// Bucket b = keys[start[b], start[b + 1]): sorted in place, repeats dropped,
// n_distinct[b] left.  Buckets of lo < keys <= cap (lo 0: from none on); the
// others return.
template <class Zone>
__global__ void __launch_bounds__(kSortThreads)
bucket_sort_kernel(const uint32_t *start, uint64_t *keys, uint32_t lo, uint32_t cap, uint32_t *n_distinct,
                   Zone zone) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kWarps = kSortThreads / 32, kPer = kZones / kSortThreads;
  static_assert(kPer == 8, "a thread scans its zones as one 16-byte word");
  uint64_t *key = reinterpret_cast<uint64_t *>(smem);
  uint32_t *count2 = reinterpret_cast<uint32_t *>(smem + (size_t)cap * 8);   // two zones a word
  uint16_t *end = reinterpret_cast<uint16_t *>(count2);
  uint16_t *big = end + kZones;
  __shared__ uint32_t s_warp[kWarps], s_big;
  const uint32_t b = blockIdx.x, base = start[b], n = start[b + 1] - base;
  if (n <= lo && lo) return;
  if (n > cap) return;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (!n) {
    if (tid == 0) n_distinct[b] = 0;
    return;
  }
  reinterpret_cast<uint4 *>(count2)[tid] = make_uint4(0, 0, 0, 0);
  if (tid == 0) s_big = 0;
  __syncthreads();
  const uint64_t *x = keys + base;
#pragma unroll 2
  for (uint32_t i = tid; i < n; i += kSortThreads) {
    const uint32_t z = zone(x[i]);
    atomicAdd(&count2[z >> 1], 1u << (16 * (z & 1)));
  }
  __syncthreads();
  {   // counts to starts
    uint4 c4 = reinterpret_cast<uint4 *>(count2)[tid];
    uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w}, sum = 0;
#pragma unroll
    for (int u = 0; u < 4; u++) sum += (c[u] & 0xFFFFu) + (c[u] >> 16);
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if ((int)lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t at = incl - sum;
    for (uint32_t w = 0; w < warp; w++) at += s_warp[w];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t lo16 = at, hi16 = at + (c[u] & 0xFFFFu);
      at = hi16 + (c[u] >> 16);
      c[u] = lo16 | hi16 << 16;
    }
    reinterpret_cast<uint4 *>(count2)[tid] = make_uint4(c[0], c[1], c[2], c[3]);
  }
  __syncthreads();
#pragma unroll 2
  for (uint32_t i = tid; i < n; i += kSortThreads) {
    const uint64_t v = x[i];
    const uint32_t z = zone(v), old = atomicAdd(&count2[z >> 1], 1u << (16 * (z & 1)));
    key[z & 1 ? old >> 16 : old & 0xFFFFu] = v;
  }
  __syncthreads();   // (a zone's start is its end now)
  for (uint32_t z = tid; z < kZones; z += kSortThreads) {
    const uint32_t from = z ? end[z - 1] : 0, m = end[z] - from;
    if (m > kThreadZone) big[atomicAdd(&s_big, 1u)] = (uint16_t)z;
    else if (m > 1) sort_zone(key + from, m);
  }
  __syncthreads();
  for (uint32_t i = warp; i < s_big; i += kWarps) {
    const uint32_t z = big[i], from = z ? end[z - 1] : 0;
    sort_big_zone(key + from, end[z] - from);
  }
  __syncthreads();
  // what is left, packed: a run of the keys per warp
  const uint32_t run = (n + 32 * kWarps - 1) / (32 * kWarps) * 32, r0 = min(n, warp * run), r1 = min(n, r0 + run);
  uint32_t have = 0;
  for (uint32_t i0 = r0; i0 < r1; i0 += 32)
    have += __popc(__ballot_sync(0xffffffffu, i0 + lane < r1 && key[i0 + lane] != kNoKey));
  if (lane == 0) s_warp[warp] = have;
  __syncthreads();
  uint32_t at = 0, total = 0;
  for (uint32_t w = 0; w < kWarps; w++) {
    if (w < warp) at += s_warp[w];
    total += s_warp[w];
  }
  if (tid == 0) n_distinct[b] = total;
  uint64_t *out = keys + base;
  for (uint32_t i0 = r0; i0 < r1; i0 += 32) {
    const uint64_t v = i0 + lane < r1 ? key[i0 + lane] : kNoKey;
    const uint32_t in = __ballot_sync(0xffffffffu, v != kNoKey);
    if (v != kNoKey) out[at + __popc(in & ((1u << lane) - 1))] = v;
    at += __popc(in);
  }
}

// Keys are dealt into buckets by the bits from `shift` up.  A pass over slices
// of the keys with a counter per bucket in shared memory counts them (a global
// atomic per key took 0.50 ms for 28M keys, this 0.04).  Then they are dealt
// to at most 2^kDealDigit places at a time -- in two steps where there are
// more buckets -- tile by tile: a tile's keys are put in the order of their
// places in shared memory and written out run by run.  (Straight to 2^13
// buckets, a random sector a key, took 0.57 ms for 28M keys; 0.21 both steps.)
constexpr int kDealThreads = 1024;
constexpr int kDealBits = 15;   // 2^15 counters are 128 KB
constexpr int kDealDigit = 7, kDealDigitMost = kDealBits - kDealDigit;
constexpr int kDealPer = 8, kDealTile = kDealThreads * kDealPer;

__global__ void __launch_bounds__(kDealThreads)
bucket_count_kernel(const uint64_t *k, uint64_t n, uint64_t slice, int shift, uint32_t nb, uint32_t *count) {
  extern __shared__ uint32_t h[];
  const uint64_t i0 = min(n, blockIdx.x * slice), i1 = min(n, i0 + slice);
  for (uint32_t b = threadIdx.x; b < nb; b += kDealThreads) h[b] = 0;
  __syncthreads();
  // (a thread adds up a bucket's keys while they follow one another: one key
  // over and over would leave the additions to one address)
  uint32_t last = 0, run = 0;
#pragma unroll 4
  for (uint64_t i = i0 + threadIdx.x; i < i1; i += kDealThreads) {
    const uint32_t b = (uint32_t)(k[i] >> shift);
    if (b != last) {
      if (run) atomicAdd(&h[last], run);
      last = b;
      run = 0;
    }
    run++;
  }
  if (run) atomicAdd(&h[last], run);
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < nb; b += kDealThreads)
    if (h[b]) atomicAdd(&count[b], h[b]);
}

__global__ void bucket_largest_kernel(const uint32_t *count, uint32_t n, uint32_t *largest) {
  uint32_t m = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) m = max(m, count[i]);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(largest, m);
}

// First places of the `n` groups of `per` buckets.
__global__ void bucket_cursor_kernel(const uint32_t *start, uint32_t per, uint32_t n, uint32_t *cursor) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) cursor[i] = start[i * per];
}

// Parent p holds keys[start[p * per], start[(p + 1) * per]); its keys go to the
// `digits` (a power of two) cursors cursor[p * digits ..] by the bits from
// shift up.  Block b works on parent b % parents.  Nothing is dealt where the
// largest bucket is too large to be sorted.
__global__ void __launch_bounds__(kDealThreads)
bucket_deal_kernel(const uint64_t *keys, const uint32_t *start, uint32_t parents, uint32_t per, int shift,
                   uint32_t digits, const uint32_t *largest, uint32_t *cursor, uint64_t *out) {
  if (*largest > kLargeBlock) return;
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t *s_key = reinterpret_cast<uint64_t *>(smem);
  constexpr int kMost = 1 << (kDealDigit > kDealDigitMost ? kDealDigit : kDealDigitMost);
  __shared__ uint32_t s_count[kMost], s_first[kMost], s_warp[kMost / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, p = blockIdx.x % parents;
  const uint32_t lo = start[p * per], hi = start[(p + 1) * per];
  const uint64_t stride = (uint64_t)(gridDim.x / parents) * kDealTile;
  for (uint64_t t0 = lo + (uint64_t)(blockIdx.x / parents) * kDealTile; t0 < hi; t0 += stride) {
    const uint32_t n = (uint32_t)min((uint64_t)kDealTile, hi - t0);
    __syncthreads();   // (the tile before is done with)
    if (tid < digits) s_count[tid] = 0;
    __syncthreads();
    uint64_t x[kDealPer];
    uint32_t at[kDealPer];
#pragma unroll
    for (int u = 0; u < kDealPer; u++) {
      const uint32_t i = u * kDealThreads + tid;
      if (i < n) x[u] = keys[t0 + i];
    }
#pragma unroll
    for (int u = 0; u < kDealPer; u++)
      if (u * kDealThreads + tid < n) at[u] = atomicAdd(&s_count[(uint32_t)(x[u] >> shift) & (digits - 1)], 1u);
    __syncthreads();
    // where each digit's keys lie in the tile (s_first) and, less that, go to
    uint32_t c = 0, incl = 0;
    if (tid < kMost) {
      c = tid < digits ? s_count[tid] : 0;
      incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += y;
      }
      if (lane == 31) s_warp[tid >> 5] = incl;
    }
    __syncthreads();
    if (tid < digits) {
      uint32_t first = incl - c;
      for (uint32_t w = 0; w < tid >> 5; w++) first += s_warp[w];
      s_first[tid] = first;
      s_count[tid] = (c ? atomicAdd(&cursor[p * digits + tid], c) : 0u) - first;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kDealPer; u++)
      if (u * kDealThreads + tid < n) s_key[s_first[(uint32_t)(x[u] >> shift) & (digits - 1)] + at[u]] = x[u];
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kDealPer; u++) {
      const uint32_t i = u * kDealThreads + tid;
      if (i < n) {
        const uint64_t v = s_key[i];
        out[s_count[(uint32_t)(v >> shift) & (digits - 1)] + i] = v;   // (modulo 2^32)
      }
    }
  }
}

// Keys to a bucket, where the number of buckets is free: 2,250 to kBucketKeys,
// and up to kBucketKeysMost with 2^15 buckets.
constexpr uint64_t kBucketKeys = 4500, kBucketKeysMost = 6000;

// Device words of a deal over nb buckets.
struct BucketMem {
  uint32_t nb;
  uint32_t *start;      // [nb + 1]
  uint32_t *largest;    // (behind start[nb])
  uint32_t *place;      // [nb + 1]
  uint32_t *distinct;   // [nb]
  uint32_t *sums;
  static uint64_t words(uint32_t nb) { return 3ull * nb + 3 + nb / rsort::kScanChunk + 2; }
  BucketMem(uint32_t *mem, uint32_t n)
      : nb(n), start(mem), largest(start + n + 1), place(largest + 1), distinct(place + n + 1), sums(distinct + n) {}
};

// Deals keys[0, n) (n < 2^32, each key >> shift below nb = 2^bits, bits <=
// kDealBits) into buckets, bucket b at start[b]: in alt, or back in keys where
// that took two steps (*dealt).  *largest: the largest bucket; above kLargeBlock
// the keys stay where they are.
inline cudaError_t deal_to_buckets(uint64_t *keys, uint64_t *alt, uint64_t n, int shift, int bits, const BucketMem &m,
                                   int device, uint64_t **dealt, uint32_t *largest, cudaStream_t st) {
  cudaError_t e;
#define TRY(x) if ((e = (x)) != cudaSuccess) return e
  int sms = 0;
  TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  // (a slice of several keys per counter)
  const uint64_t slice = std::max<uint64_t>((n + sms - 1) / sms, 4096);
  TRY(cudaFuncSetAttribute(bucket_count_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 << kDealBits));
  TRY(cudaFuncSetAttribute(bucket_deal_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDealTile * 8));
  TRY(cudaMemsetAsync(m.start, 0, (m.nb + 2) * 4ull, st));
  bucket_count_kernel<<<(unsigned)((n + slice - 1) / slice), kDealThreads, m.nb * 4, st>>>(keys, n, slice, shift, m.nb,
                                                                                         m.start);
  bucket_largest_kernel<<<(m.nb + 255) / 256, 256, 0, st>>>(m.start, m.nb, m.largest);
  note_launches(2);
  TRY(rsort::exclusive_scan(m.start, m.nb + 1, m.sums, st));
  const int low = bits > kDealDigit ? bits - kDealDigit : 0;   // bits left for the second step
  auto step = [&](const uint64_t *in, uint64_t *out, uint32_t parents, int digit_bits, int at) {
    const uint32_t digits = 1u << digit_bits, cursors = parents * digits;
    bucket_cursor_kernel<<<(cursors + 255) / 256, 256, 0, st>>>(m.start, m.nb / cursors, cursors, m.place);
    // (two blocks to an SM, and a few for every parent)
    const uint64_t tiles = n / parents / kDealTile + 1;
    const uint32_t each = (uint32_t)std::min<uint64_t>(tiles, (2 * sms + parents - 1) / parents);
    bucket_deal_kernel<<<parents * each, kDealThreads, kDealTile * 8, st>>>(in, m.start, parents, m.nb / parents, at,
                                                                            digits, m.largest, m.place, out);
    note_launches(2);
  };
  step(keys, alt, 1, bits - low, shift + low);
  if (low) step(alt, keys, 1u << kDealDigit, low, shift);
  *dealt = low ? keys : alt;
  TRY(cudaGetLastError());
  TRY(cudaMemcpyAsync(largest, m.largest, 4, cudaMemcpyDeviceToHost, st));
#undef TRY
  return cudaStreamSynchronize(st);
}

// Sorts the buckets; `largest` bounds their sizes (at most kLargeBlock).
template <class Zone>
cudaError_t bucket_sort(const uint32_t *start, uint32_t n_buckets, uint64_t largest, uint64_t *keys,
                        uint32_t *n_distinct, Zone zone, cudaStream_t st) {
  const uint32_t caps[3] = {0, kSmallBlock, kLargeBlock};
  for (int i = 1; i < 3; i++) {
    if (i > 1 && largest <= caps[i - 1]) break;
    const size_t smem = bucket_sort_smem(caps[i]);
    auto kern = bucket_sort_kernel<Zone>;
    // (the limit is the kernel's, whichever thread calls: always the largest)
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bucket_sort_smem(kLargeBlock));
    if (e != cudaSuccess) return e;
    kern<<<n_buckets, kSortThreads, smem, st>>>(start, keys, caps[i - 1], caps[i], n_distinct, zone);
    note_launches();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace
}  // namespace k2g
