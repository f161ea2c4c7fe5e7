// Order-exact build insert: the table k2g_build_insert(..., ordered = 1)
// leaves is the one sequential SetMinimizerLCA in list order produces
// (src/build_db.h:187-194 over src/compact_hash.h:395-462), cell for cell.
//
// Why it parallelises: with linear probing an insert only reads and writes
// cells of the run of occupied cells (cluster) its home lies in, in the final
// table.  So:
//   1. snapshot the table, then insert everything unordered (CAS + LCA) -- this
//      predicts the final occupancy;
//   2. tag every pair with the start of its predicted cluster and sort by
//      (cluster start, list position);
//   3. one thread per cluster restores the cluster from the snapshot and
//      replays its pairs in list order.  Where the exact replay needs more
//      cells than predicted it may take the free cells after its cluster
//      (no other cluster owns them); reaching the next cluster flags it;
//   4. flagged clusters are replayed again merged with their neighbours by a
//      single thread, and the size is recounted.
// Only the order of pairs whose compacted keys collide along a probe path
// can change the outcome, so flags are rare.
//
// A cluster in which every pair went to its home cell needs neither step 2
// nor 3: the first pair that a sequential insert places elsewhere would find
// its home taken by another key, whose home it is too or which was there
// before, and then the unordered pass would have moved one of the two as well;
// the values are LCAs, in any order the same (unless the taxonomy has several
// roots: an LCA of 0 empties a cell, so such tables keep all pairs).  The
// unordered pass marks the cells that pairs were moved to, and only the pairs
// of clusters with marks are sorted and replayed: three in ten of the 15.7M of
// 48 Mbp at a load of 0.26 (whole build 4.9 -> 3.9 ms), nearly all at 0.85
// (14.7 -> 14.3) -- unless step 4 is likely, which needs all of them
// (merges_expected).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "k2g_device.cuh"
#include "k2g_internal.h"
#include "radix_sort.cuh"

namespace k2g {
namespace {

constexpr int kIndexBits = 30;                  // pairs per round: < 2^30
constexpr uint64_t kNoRegion = ~0ull;
constexpr uint32_t kFlagCap = 1u << 20;         // clusters that may need a merged replay

template <class C>
struct OrderedView {
  TableView t;
  typename C::T *cells;
  const typename C::T *snap;  // the table before this round (null: all zero)
  const uint32_t *occ;        // bitmap: occupied after the unordered pass
  const uint32_t *parent;
  const uint64_t *keys;
  const uint32_t *taxids;
  uint64_t n;
  __device__ __forceinline__ typename C::T before(uint64_t c) const { return snap ? snap[c] : typename C::T(0); }
};

template <class C>
__device__ __forceinline__ bool occupied1(const OrderedView<C> &v, uint64_t c) {
  return (v.occ[c >> 5] >> (c & 31)) & 1u;
}
__device__ __forceinline__ uint64_t next_cell(const TableView &t, uint64_t c) {
  return c + 1 == t.capacity ? 0 : c + 1;
}
__device__ __forceinline__ uint64_t prev_cell(const TableView &t, uint64_t c) {
  return c == 0 ? t.capacity - 1 : c - 1;
}

// (a warp reads 32 cells side by side for a word; a thread for each word, its
// reads 128 bytes apart, took 84 us for 24M cells; 20 now)
template <class C>
__global__ void occ_kernel(const typename C::T *cells, TableView t, uint32_t *occ) {
  constexpr int kWords = 4;   // reads in flight per lane
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t n_words = (t.capacity + 31) / 32, stride = (uint64_t)gridDim.x * (blockDim.x >> 5) * kWords;
  for (uint64_t w = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * kWords; w < n_words; w += stride) {
    typename C::T cell[kWords];
#pragma unroll
    for (int u = 0; u < kWords; u++) {
      const uint64_t c = (w + u) * 32 + lane;
      cell[u] = c < t.capacity ? cells[c] : 0;
    }
#pragma unroll
    for (int u = 0; u < kWords; u++) {
      const uint32_t bits = __ballot_sync(0xffffffffu, C::value(cell[u], t) != 0);
      if (lane == u && w + u < n_words) occ[w + u] = bits;
    }
  }
}

// Start of the cluster of cell s.
template <class C>
__device__ __forceinline__ uint64_t cluster_start(const OrderedView<C> &v, uint64_t s, uint32_t *status) {
  uint64_t steps = 0;
  while (occupied1(v, prev_cell(v.t, s))) {
    s = prev_cell(v.t, s);
    if (++steps >= v.t.capacity) {
      atomicOr(status, STATUS_BUILD_FULL);
      break;
    }
  }
  return s;
}

// (cluster start << kIndexBits | list position) per pair; pairs with taxid 0
// are not inserted and sort last.
template <class C>
__global__ void region_kernel(OrderedView<C> v, uint64_t *out, uint32_t *status) {
  for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < v.n;
       j += (uint64_t)gridDim.x * blockDim.x) {
    if (!v.taxids[j]) {
      out[j] = kNoRegion;
      continue;
    }
    out[j] = (cluster_start(v, fast_mod(murmur3(v.keys[j]), v.t.div), status) << kIndexBits) | j;
  }
}

// Whether a pair was moved to a cell of the cluster of the occupied cell c.
template <class C>
__device__ __forceinline__ bool cluster_moved(const OrderedView<C> &v, const uint32_t *moved, uint64_t c) {
  // the cluster's cells in c's word of the bitmaps, then the rest one by one
  const uint32_t b = (uint32_t)(c & 31), free = ~v.occ[c >> 5];
  const uint32_t under = free & ((1u << b) - 1), over = b < 31 ? free >> (b + 1) : 0;
  const uint32_t lo = under ? 32 - __clz(under) : 0, hi = over ? b + __ffs(over) - 1 : 31;
  if (moved[c >> 5] & (0xFFFFFFFFu >> (31 - hi)) & (0xFFFFFFFFu << lo)) return true;
  auto marked = [&](uint64_t x) { return (moved[x >> 5] >> (x & 31)) & 1u; };
  uint64_t left = v.t.capacity;   // (a full table is one endless cluster)
  if (!lo)
    for (uint64_t x = prev_cell(v.t, c - b); occupied1(v, x); x = prev_cell(v.t, x))
      if (marked(x) || !--left) return true;
  if (hi == 31 || c - b + hi == v.t.capacity - 1)
    for (uint64_t x = next_cell(v.t, c - b + hi); occupied1(v, x); x = next_cell(v.t, x))
      if (marked(x) || !--left) return true;
  return false;
}

constexpr int kPickThreads = 256;
constexpr uint32_t kPickTile = 1024;   // pairs per block

// The pairs of clusters with marks: a bitmap, and their number per tile.
template <class C>
__global__ void __launch_bounds__(kPickThreads)
pick_kernel(OrderedView<C> v, const uint32_t *moved, uint32_t *picked, uint32_t *tile_cnt) {
  __shared__ uint32_t s_n;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  uint32_t mine = 0;
#pragma unroll
  for (int u = 0; u < (int)kPickTile / kPickThreads; u++) {
    const uint64_t j = blockIdx.x * (uint64_t)kPickTile + u * kPickThreads + threadIdx.x;
    const bool take = j < v.n && v.taxids[j] && cluster_moved(v, moved, fast_mod(murmur3(v.keys[j]), v.t.div));
    const uint32_t word = __ballot_sync(0xffffffffu, take);
    if ((threadIdx.x & 31) == 0) {
      picked[j >> 5] = word;
      mine += __popc(word);
    }
  }
  if (mine) atomicAdd(&s_n, mine);
  __syncthreads();
  if (threadIdx.x == 0) tile_cnt[blockIdx.x] = s_n;
}

// region_kernel's words of the picked pairs, in list order.
template <class C>
__global__ void __launch_bounds__(kPickThreads)
picked_region_kernel(OrderedView<C> v, const uint32_t *picked, const uint32_t *tile_off, uint64_t *out,
                     uint32_t *status) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t words = __popc(picked[blockIdx.x * (uint64_t)(kPickTile / 32) + lane]);   // (32 words a tile)
#pragma unroll
  for (int u = 0; u < (int)kPickTile / kPickThreads; u++) {
    const uint32_t w = (u * kPickThreads + threadIdx.x) >> 5;
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < w ? words : 0u);
    const uint64_t j = blockIdx.x * (uint64_t)kPickTile + w * 32 + lane;
    const uint32_t word = picked[j >> 5];
    if ((word >> lane) & 1u)
      out[tile_off[blockIdx.x] + before + __popc(word & ((1u << lane) - 1))] =
          (cluster_start(v, fast_mod(murmur3(v.keys[j]), v.t.div), status) << kIndexBits) | j;
  }
}

// Sequential SetMinimizerLCA of one pair against the cells as they are.
// Cells from `start` for `limit` offsets belong to this replay; beyond them
// only cells that were free after the unordered pass may be taken.  Returns
// false when the probe reaches a cell owned by another cluster.
template <class C>
__device__ bool replay_one(const OrderedView<C> &v, uint64_t start, uint64_t &limit, uint64_t key,
                           uint32_t taxid) {
  const uint64_t hc = murmur3(key);
  const uint64_t ck = hc >> v.t.key_shift;
  uint64_t c = fast_mod(hc, v.t.div);
  for (uint64_t step = 0; step < v.t.capacity; step++) {
    const uint64_t off = c >= start ? c - start : c + v.t.capacity - start;
    if (off >= limit) {
      // past the cells this replay owns: a free cell extends them, a
      // cell of another cluster ends the replay
      if (off > limit || occupied1(v, c)) return false;
      limit = off + 1;
    }
    const typename C::T cell = v.cells[c];
    const uint32_t val = C::value(cell, v.t);
    if (!val || C::match(cell, ck, v.t)) {
      const uint32_t nv = val ? lca(v.parent, val, taxid) : taxid;
      v.cells[c] = C::make(ck, nv, v.t);
      return true;
    }
    c = next_cell(v.t, c);
  }
  return false;
}

// One thread per cluster: restore from the snapshot, replay in list order.
template <class C>
__global__ void replay_kernel(OrderedView<C> v, const uint64_t *sorted, uint64_t n_sorted,
                              uint64_t *flags, unsigned long long *n_flags) {
  const uint64_t pmask = (1ull << kIndexBits) - 1;
  for (uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; p < n_sorted;
       p += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t key = sorted[p];
    if (key == kNoRegion) continue;
    const uint64_t s = key >> kIndexBits;
    if (p > 0 && (sorted[p - 1] >> kIndexBits) == s) continue;   // not the first of its cluster
    // the cluster's cells after the unordered pass
    uint64_t len = 1;
    for (uint64_t c = next_cell(v.t, s); occupied1(v, c) && len < v.t.capacity; c = next_cell(v.t, c))
      len++;
    for (uint64_t o = 0, c = s; o < len; o++, c = next_cell(v.t, c)) v.cells[c] = v.before(c);
    uint64_t limit = len;
    bool ok = true;
    for (uint64_t q = p; q < n_sorted && sorted[q] != kNoRegion && (sorted[q] >> kIndexBits) == s; q++) {
      const uint64_t j = sorted[q] & pmask;
      if (!replay_one(v, s, limit, v.keys[j], v.taxids[j])) {
        ok = false;
        break;
      }
    }
    if (!ok) {
      const unsigned long long at = atomicAdd(n_flags, 1ull);
      if (at < kFlagCap) flags[at] = s;
    }
  }
}

__device__ uint64_t lower_bound_region(const uint64_t *sorted, uint64_t n, uint64_t s) {
  uint64_t lo = 0, hi = n;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (sorted[mid] < (s << kIndexBits)) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Merged replays of the flagged clusters, one after another (a single
// thread: flags are rare).  The flagged list is sorted by cluster start.
// A merged group spans clusters [s0 .. ]; it grows by the next cluster until
// its replay fits.  `scratch` holds list positions (capacity scratch_cap).
template <class C>
__global__ void fixup_kernel(OrderedView<C> v, const uint64_t *sorted, uint64_t n_sorted,
                             const uint64_t *flags, uint64_t n_flags, uint64_t *scratch,
                             uint64_t scratch_cap, uint32_t *status) {
  if (threadIdx.x || blockIdx.x) return;
  const uint64_t pmask = (1ull << kIndexBits) - 1;
  uint64_t covered_until = 0;   // offsets of the table already redone (non-wrapping groups)
  bool any = false;
  for (uint64_t fi = 0; fi < n_flags; fi++) {
    const uint64_t s0 = flags[fi];
    if (any && s0 < covered_until) continue;
    uint64_t n_clusters = 2;
    for (;;) {
      // extent: n_clusters clusters from s0, plus the free cells after each
      // that a first-pass replay may have taken (non-empty, not occupied
      // after the unordered pass)
      uint64_t c = s0, len = 0, items = 0;
      uint64_t starts[64];
      int ns = 0;
      bool too_many = false;
      for (uint64_t k = 0; k < n_clusters; k++) {
        if (ns < 64) starts[ns++] = c;
        else too_many = true;
        while (occupied1(v, c) && len < v.t.capacity) { c = next_cell(v.t, c); len++; }
        while (!occupied1(v, c) && C::value(v.cells[c], v.t) && len < v.t.capacity) {
          c = next_cell(v.t, c);
          len++;
        }
        if (k + 1 < n_clusters)   // skip free cells to the next cluster
          while (!occupied1(v, c) && len < v.t.capacity) { c = next_cell(v.t, c); len++; }
      }
      if (too_many || len >= v.t.capacity) {
        atomicOr(status, STATUS_BUILD_FULL);
        return;
      }
      // restore the extent, gather its pairs
      for (uint64_t o = 0, x = s0; o < len; o++, x = next_cell(v.t, x)) v.cells[x] = v.before(x);
      for (int k = 0; k < ns; k++) {
        for (uint64_t q = lower_bound_region(sorted, n_sorted, starts[k]);
             q < n_sorted && sorted[q] != kNoRegion && (sorted[q] >> kIndexBits) == starts[k]; q++) {
          if (items == scratch_cap) {
            atomicOr(status, STATUS_BUILD_FULL);
            return;
          }
          scratch[items++] = sorted[q] & pmask;
        }
      }
      // list order (heap sort of the gathered positions)
      for (uint64_t i = items / 2; i-- > 0;) {
        uint64_t r = i;
        while (2 * r + 1 < items) {
          uint64_t ch = 2 * r + 1;
          if (ch + 1 < items && scratch[ch + 1] > scratch[ch]) ch++;
          if (scratch[r] >= scratch[ch]) break;
          const uint64_t tmp = scratch[r]; scratch[r] = scratch[ch]; scratch[ch] = tmp;
          r = ch;
        }
      }
      for (uint64_t e = items; e-- > 1;) {
        uint64_t tmp = scratch[0]; scratch[0] = scratch[e]; scratch[e] = tmp;
        uint64_t r = 0;
        while (2 * r + 1 < e) {
          uint64_t ch = 2 * r + 1;
          if (ch + 1 < e && scratch[ch + 1] > scratch[ch]) ch++;
          if (scratch[r] >= scratch[ch]) break;
          tmp = scratch[r]; scratch[r] = scratch[ch]; scratch[ch] = tmp;
          r = ch;
        }
      }
      // replay; the extent owns its cells, free cells after it may be taken
      uint64_t limit = len;
      bool ok = true;
      for (uint64_t i = 0; i < items && ok; i++)
        ok = replay_one(v, s0, limit, v.keys[scratch[i]], v.taxids[scratch[i]]);
      if (ok) {
        covered_until = s0 + limit;
        any = true;
        break;
      }
      n_clusters++;
    }
  }
}

template <class C>
__global__ void count_kernel(const typename C::T *cells, TableView t, unsigned long long *size) {
  constexpr int kAhead = 8;
  uint64_t mine = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < t.capacity; c += kAhead * stride) {
    typename C::T cell[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; u++) cell[u] = c + u * stride < t.capacity ? cells[c + u * stride] : 0;
#pragma unroll
    for (int u = 0; u < kAhead; u++) mine += C::value(cell[u], t) != 0;
  }
  for (int o = 16; o; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(size, (unsigned long long)mine);
}

int grid(int device, uint64_t n) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return (int)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)sms * 16));
}

int bits_of(uint64_t x) {
  int b = 0;
  while (b < 64 && (x >> b)) b++;
  return b;
}

// Whether some cluster of a batch of n pairs is likely to need a merged replay,
// for which all pairs have to be sorted; then the pairs of clusters with marks
// are not sorted first.  Where the first such clusters appear at loads of 0.40,
// 0.66 and 0.85, for 1.3M to 157M pairs and 10 to 22 key bits, fits their number
// going with n / 4^key_bits and the power 5.3 of 1 / (1 - load).  The line lies
// where the sort in vain costs as much as the picking gains: of 15.7M pairs at
// 0.66 the picking took 6.6 ms with 12 bits, where some need it, 5.1 all sorted;
// with 13, where none do, 5.0 and 5.1; at 0.85 14.1 and 11.4 with 16 bits, 10.2
// and 11.1 with 22; at 0.40 4.5 and 3.9 with 10, 3.2 and 3.7 with 11; of 157M at
// 0.66 72.6 and 61.2 with 13, 58.8 and 60.3 with 14.
bool merges_expected(uint64_t n, uint64_t size, uint64_t capacity, uint32_t key_bits) {
  const double free_share = std::max(1.0 - (double)size / (double)capacity, 0.01);
  const double expected = 0.005 * std::ldexp((double)n, -2 * (int)key_bits) / std::pow(free_share, 5.3);
  return expected > 0.38;
}

template <class T>
struct DevBuf {
  int device;
  cudaStream_t st;
  T *p = nullptr;
  DevBuf(int d, cudaStream_t s) : device(d), st(s) {}
  DevBuf(const DevBuf &) = delete;
  ~DevBuf() { free(); }
  void free() {
    if (p) cudaFreeAsync(p, st);
    p = nullptr;
  }
  cudaError_t alloc(uint64_t n) {
    return scratch_alloc(reinterpret_cast<void **>(&p), std::max<uint64_t>(n, 1) * sizeof(T), device, st);
  }
};

}  // namespace

// One round (fewer than 2^30 pairs) of the order-exact insert over cells of
// layout C.
template <class C>
k2g_status insert_ordered(k2g_db *db, typename C::T *cells, const uint64_t *d_keys,
                          const uint32_t *d_taxids, uint64_t n, cudaStream_t st) {
  using T = typename C::T;
  const TableView t = db->table_view();
  const uint64_t cap = db->capacity;
  if (bits_of(cap) + kIndexBits > 64) return fail(K2G_ERR_UNSUPPORTED, "table too large for the ordered insert");
  const int dev = db->device;
  DevBuf<T> snap(dev, st);
  DevBuf<uint32_t> occ(dev, st), status(dev, st), moved(dev, st);
  DevBuf<uint64_t> keys(dev, st), alt(dev, st), flags(dev, st), scratch(dev, st);
  DevBuf<uint32_t> hist(dev, st), sums(dev, st), picked(dev, st), tiles(dev, st);
  DevBuf<unsigned long long> ctr(dev, st);
  if (!db->blank) K2G_CUDA_TRY(snap.alloc(cap));   // (the first batch of a build needs none)
  const uint64_t words = (cap + 31) / 32, n_tiles = (n + kPickTile - 1) / kPickTile;
  K2G_CUDA_TRY(occ.alloc(words));
  K2G_CUDA_TRY(status.alloc(1));
  K2G_CUDA_TRY(ctr.alloc(2));
  K2G_CUDA_TRY(flags.alloc(kFlagCap));
  if (db->one_root) {
    K2G_CUDA_TRY(moved.alloc(words));
    K2G_CUDA_TRY(cudaMemsetAsync(moved.p, 0, words * 4, st));
  }
  if (snap.p) K2G_CUDA_TRY(cudaMemcpyAsync(snap.p, cells, cap * sizeof(T), cudaMemcpyDeviceToDevice, st));
  // 1. unordered pass (validates values and capacity)
  K2G_CUDA_TRY(insert_unordered(db, d_keys, d_taxids, n, status.p, moved.p, st));
  uint32_t st_word = 0;
  unsigned long long n_flags = 0;
  uint64_t size = 0;
  K2G_CUDA_TRY(cudaMemcpyAsync(&st_word, status.p, 4, cudaMemcpyDeviceToHost, st));
  K2G_CUDA_TRY(cudaMemcpyAsync(&size, db->d_size, 8, cudaMemcpyDeviceToHost, st));
  K2G_CUDA_TRY(cudaStreamSynchronize(st));
  const k2g_status s = insert_status(st_word);
  if (s != K2G_OK) return s;
  const bool pick = db->one_root && !merges_expected(n, size, cap, (uint32_t)db->key_bits);
  K2G_CUDA_TRY(cudaMemsetAsync(status.p, 0, 4, st));
  K2G_CUDA_TRY(cudaMemsetAsync(ctr.p, 0, 16, st));
  occ_kernel<C><<<grid(db->device, 8 * words), 256, 0, st>>>(cells, t, occ.p);
  note_launches();
  K2G_CUDA_TRY(cudaGetLastError());
  // 2. cluster of each pair, sorted
  OrderedView<C> v{t, cells, snap.p, occ.p, db->d_parent, d_keys, d_taxids, n};
  uint64_t *sorted = nullptr, n_sorted = n;
  // by cluster start alone: the list positions below it are in order already,
  // and the sort is stable (pairs that are not inserted have all bits set,
  // above any cell number)
  auto sort_pairs = [&]() -> k2g_status {
    K2G_CUDA_TRY(alt.alloc(n_sorted));
    K2G_CUDA_TRY(hist.alloc(rsort::hist_entries(n_sorted)));
    K2G_CUDA_TRY(sums.alloc(rsort::sum_entries(n_sorted) + 1));
    K2G_CUDA_TRY(rsort::sort_u64(keys.p, alt.p, n_sorted, kIndexBits + bits_of(cap), hist.p, sums.p, st, &sorted,
                                 kIndexBits));
    return K2G_OK;
  };
  auto sort_all = [&]() -> k2g_status {
    n_sorted = n;
    K2G_CUDA_TRY(keys.alloc(n));
    region_kernel<C><<<grid(db->device, n), 256, 0, st>>>(v, keys.p, status.p);
    note_launches();
    K2G_CUDA_TRY(cudaGetLastError());
    return sort_pairs();
  };
  auto sort_picked = [&]() -> k2g_status {
    K2G_CUDA_TRY(picked.alloc(n_tiles * (kPickTile / 32)));
    K2G_CUDA_TRY(tiles.alloc(n_tiles + 1));
    K2G_CUDA_TRY(sums.alloc(n_tiles / rsort::kScanChunk + 2));
    K2G_CUDA_TRY(cudaMemsetAsync(tiles.p + n_tiles, 0, 4, st));
    pick_kernel<C><<<(unsigned)n_tiles, kPickThreads, 0, st>>>(v, moved.p, picked.p, tiles.p);
    note_launches();
    K2G_CUDA_TRY(cudaGetLastError());
    K2G_CUDA_TRY(rsort::exclusive_scan(tiles.p, n_tiles + 1, sums.p, st));
    uint32_t m = 0;
    K2G_CUDA_TRY(cudaMemcpyAsync(&m, tiles.p + n_tiles, 4, cudaMemcpyDeviceToHost, st));
    K2G_CUDA_TRY(cudaStreamSynchronize(st));
    sums.free();
    n_sorted = m;
    if (!m) return K2G_OK;
    K2G_CUDA_TRY(keys.alloc(m));
    picked_region_kernel<C><<<(unsigned)n_tiles, kPickThreads, 0, st>>>(v, picked.p, tiles.p, keys.p, status.p);
    note_launches();
    K2G_CUDA_TRY(cudaGetLastError());
    return sort_pairs();
  };
  const k2g_status by = pick ? sort_picked() : sort_all();
  if (by != K2G_OK) return by;
  // 3. per-cluster replays
  if (n_sorted) {
    replay_kernel<C><<<grid(db->device, n_sorted), 256, 0, st>>>(v, sorted, n_sorted, flags.p, ctr.p);
    note_launches();
    K2G_CUDA_TRY(cudaGetLastError());
  }
  K2G_CUDA_TRY(cudaMemcpyAsync(&n_flags, ctr.p, 8, cudaMemcpyDeviceToHost, st));
  K2G_CUDA_TRY(cudaMemcpyAsync(&st_word, status.p, 4, cudaMemcpyDeviceToHost, st));
  K2G_CUDA_TRY(cudaStreamSynchronize(st));
  if (st_word) return fail(K2G_ERR_CAPACITY, "compact hash table capacity exceeded");
  if (n_flags > kFlagCap) return fail(K2G_ERR_BUDGET, "too many clusters need a merged replay");
  // 4. merged replays of flagged clusters, in cluster order
  if (n_flags) {
    if (pick) {   // (their neighbours may be clusters without marks)
      keys.free();
      alt.free();
      hist.free();
      sums.free();
      const k2g_status all = sort_all();
      if (all != K2G_OK) return all;
    }
    std::vector<uint64_t> fl(n_flags);
    K2G_CUDA_TRY(cudaMemcpyAsync(fl.data(), flags.p, n_flags * 8, cudaMemcpyDeviceToHost, st));
    K2G_CUDA_TRY(cudaStreamSynchronize(st));
    std::sort(fl.begin(), fl.end());
    // (on this stream: the kernel below need not wait for another's copy)
    K2G_CUDA_TRY(cudaMemcpyAsync(flags.p, fl.data(), n_flags * 8, cudaMemcpyHostToDevice, st));
    const uint64_t scratch_cap = std::min<uint64_t>(n, 1ull << 24);
    K2G_CUDA_TRY(scratch.alloc(scratch_cap));
    fixup_kernel<C><<<1, 32, 0, st>>>(v, sorted, n_sorted, flags.p, n_flags, scratch.p, scratch_cap, status.p);
    note_launches();
    K2G_CUDA_TRY(cudaGetLastError());
    K2G_CUDA_TRY(cudaMemcpyAsync(&st_word, status.p, 4, cudaMemcpyDeviceToHost, st));
    K2G_CUDA_TRY(cudaStreamSynchronize(st));
    if (st_word) return fail(K2G_ERR_CAPACITY, "compact hash table capacity exceeded");
  }
  // size: occupied cells
  K2G_CUDA_TRY(cudaMemsetAsync(db->d_size, 0, 8, st));
  count_kernel<C><<<grid(db->device, cap), 256, 0, st>>>(cells, t,
                                                          reinterpret_cast<unsigned long long *>(db->d_size));
  note_launches();
  K2G_CUDA_TRY(cudaGetLastError());
  K2G_CUDA_TRY(cudaStreamSynchronize(st));
  return K2G_OK;
}

k2g_status build_insert_ordered(k2g_db *db, const uint64_t *d_keys, const uint32_t *d_taxids,
                                uint64_t n, cudaStream_t st) {
  if (db->d_wide) return insert_ordered<CellWide>(db, db->d_wide, d_keys, d_taxids, n, st);
  return insert_ordered<Cell32>(db, db->d_cells, d_keys, d_taxids, n, st);
}

}  // namespace k2g
