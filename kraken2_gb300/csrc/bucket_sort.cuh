// Sorts many buckets of 64-bit keys (below 2^63) at once, a thread block to a
// bucket in shared memory, and drops repeats: the library build's sequence
// blocks and the -K counters' hash ranges.
//
// A bucket's keys go to shared memory by zone -- 256 of them, in the order the
// caller wants first, spread evenly (a hash or uniform bits) -- and a warp
// ranks a zone's few keys by comparing all with all: about 5 instructions a
// key at 25 keys a zone, against a radix pass over memory per 8 bits.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "k2g_device.cuh"

namespace k2g {
namespace {

constexpr int kSortThreads = 512;
constexpr int kZones = 256;
constexpr uint32_t kSmallBlock = 8064;    // keys; three thread blocks to an SM
constexpr uint32_t kLargeBlock = 25600;   // 200 KB of keys

inline size_t bucket_sort_smem(uint32_t cap) { return (size_t)cap * 8 + kZones * 12 + 16; }

struct ZoneMurmur {   // MurmurHash3 mod 256
  __device__ __forceinline__ uint32_t operator()(uint64_t key) const { return (uint32_t)murmur3(key) & 0xFFu; }
};
struct ZoneBits {     // eight bits of the key
  int shift;
  __device__ __forceinline__ uint32_t operator()(uint64_t key) const { return (uint32_t)(key >> shift) & 0xFFu; }
};

// Distinct keys of a zone holding more than 128 keys, one after
// another from the smallest (warp-wide); out may be null (count only).
__device__ __forceinline__ uint32_t select_distinct(const uint64_t *z, uint32_t n, uint64_t *out) {
  const uint32_t lane = threadIdx.x & 31;
  uint64_t last = 0;
  uint32_t d = 0;
  for (;;) {
    uint64_t best = ~0ull;
    for (uint32_t i = lane; i < n; i += 32) {
      const uint64_t x = z[i];
      if ((!d || x > last) && x < best) best = x;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) best = min64(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (best == ~0ull) return d;   // (keys have fewer than 64 bits)
    if (out && lane == 0) out[d] = best;
    last = best;
    d++;
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
  uint64_t *key = reinterpret_cast<uint64_t *>(smem);
  uint32_t *hist = reinterpret_cast<uint32_t *>(smem + (size_t)cap * 8), *first = hist + kZones, *dist = first + kZones;
  const uint32_t b = blockIdx.x, base = start[b], n = start[b + 1] - base;
  if (n <= lo && lo) return;
  if (n > cap) return;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = kSortThreads / 32;
  if (!n) {
    if (threadIdx.x == 0) n_distinct[b] = 0;
    return;
  }
  for (uint32_t i = threadIdx.x; i < kZones; i += kSortThreads) hist[i] = 0;
  __syncthreads();
  const uint64_t *x = keys + base;
  for (uint32_t i = threadIdx.x; i < n; i += kSortThreads) atomicAdd(&hist[zone(x[i])], 1u);
  __syncthreads();
  auto scan = [&](const uint32_t *in, uint32_t *out) {   // exclusive, by the first warp
    uint32_t carry = 0;
    for (int i0 = 0; i0 < kZones; i0 += 32) {
      const uint32_t v = in[i0 + lane];
      uint32_t x = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if ((int)lane >= o) x += y;
      }
      out[i0 + lane] = carry + x - v;
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
    return carry;
  };
  if (warp == 0) scan(hist, first);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < kZones; i += kSortThreads) dist[i] = first[i];   // cursors
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n; i += kSortThreads) {
    const uint64_t v = x[i];
    key[atomicAdd(&dist[zone(v)], 1u)] = v;
  }
  __syncthreads();
  // every zone sorted in place, repeats dropped
  for (uint32_t z = warp; z < kZones; z += warps) {
    const uint32_t m = hist[z];
    uint64_t *zk = key + first[z];
    uint32_t d = 0;
    if (m <= 32) {
      const uint64_t v = lane < m ? zk[lane] : ~0ull;
      uint32_t less = 0;
      bool again = false;
      for (uint32_t j = 0; j < m; j++) {
        const uint64_t x = __shfl_sync(0xffffffffu, v, j);
        less |= x < v ? 1u << j : 0u;
        again |= x == v && j < lane;
      }
      const bool own = lane < m && !again;
      const uint32_t keepers = __ballot_sync(0xffffffffu, own);
      __syncwarp();
      if (own) zk[__popc(less & keepers)] = v;
      d = __popc(keepers);
    } else if (m <= 128) {
      uint64_t v[4];
      uint32_t own = 0, rank[4] = {0, 0, 0, 0};
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const uint32_t i = 32 * t + lane;
        v[t] = i < m ? zk[i] : ~0ull;
        bool again = i >= m;
        for (uint32_t j = 0; j < i && j < m; j++) again |= zk[j] == v[t];
        own |= again ? 0u : 1u << t;
      }
      __syncwarp();
      uint32_t keepers[4];
#pragma unroll
      for (int t = 0; t < 4; t++) {
        keepers[t] = __ballot_sync(0xffffffffu, (own >> t) & 1u);
        d += __popc(keepers[t]);
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        for (uint32_t k = keepers[u]; k; k &= k - 1) {
          const uint64_t x = zk[32 * u + __ffs(k) - 1];
#pragma unroll
          for (int t = 0; t < 4; t++) rank[t] += x < v[t] ? 1u : 0u;
        }
      __syncwarp();
#pragma unroll
      for (int t = 0; t < 4; t++)
        if ((own >> t) & 1u) zk[rank[t]] = v[t];
    } else {
      d = select_distinct(zk, m, nullptr);
    }
    __syncwarp();
    if (lane == 0) dist[z] = d;
  }
  __syncthreads();
  __shared__ uint32_t place[kZones];
  if (warp == 0) {
    const uint32_t total = scan(dist, place);
    if (lane == 0) n_distinct[b] = total;
  }
  __syncthreads();
  for (uint32_t z = warp; z < kZones; z += warps) {
    uint64_t *out = keys + base + place[z];
    const uint64_t *zk = key + first[z];
    if (hist[z] > 128) select_distinct(zk, hist[z], out);
    else
      for (uint32_t i = lane; i < dist[z]; i += 32) out[i] = zk[i];
  }
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
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<n_buckets, kSortThreads, smem, st>>>(start, keys, caps[i - 1], caps[i], n_distinct, zone);
    note_launches();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace
}  // namespace k2g
