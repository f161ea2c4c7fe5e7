// Classification of short fragments, one warp per group of fragments.
//
// A group is up to kWcReads consecutive fragments.  Its warp runs the whole
// path -- scan, table lookups, hit lists, ResolveTree -- with everything in
// between in registers and 8 KB of shared memory, so a call is one launch
// with no device scratch:
//   pack     16 bases per lane to 2-bit words in shared memory: forward
//            (first base high) and complement (first base low), so that an
//            l-mer and its reverse complement are each two funnel shifts;
//   scan     8 l-mer positions per lane.  The lanes' work items are the
//            positions that end an l-mer of some sequence, numbered through
//            the group, so lanes stay full whatever the read lengths; window
//            minima come from prefix and suffix minima of blocks of four.
//            The starts of token groups (src/classify.cc:797-838) become
//            entries (key, fragment, token position) in token order;
//   probe    one entry per lane, three table sectors in flight per lane; walks
//            that leave their home sector are listed and finished together
//            (src/compact_hash.h:355-392; a sector of every listed walk at a
//            time, all lanes in step, was 13 % slower);
//   replay   32 entries at a time: equal neighbours join into hit-list runs
//            (src/classify.cc:950-991), every finished run adds its tokens to
//            its fragment's taxon map, hits are counted by ballots;
//   resolve  one fragment's taxa across the lanes; "x is an ancestor of y" is
//            an interval test on preorder numbers, so ResolveTree
//            (src/classify.cc:710-762) needs no walks to the root.
//
// What bounds it: on tables beyond L2 the random 32-byte table loads and the
// integer ALU together (150 bp reads on a 2 GB table: DRAM 68 % busy, ALU pipe
// 62 %, 696 warp instructions a read); where the table fits L2 the ALU alone.
// Against the staged scan / probe / resolve kernels it replaces for such
// calls: 8M x 150 bp on a 16 GB table 16.5 -> 9.4 ms (39 G sectors/s of the
// 49 G/s a bare random gather reaches), 500k pairs over related genomes 2.75
// -> 1.34 ms, 1,000 reads 118 -> 18 us (one launch instead of seven).
#pragma once

#include "classify_core.cuh"
#include "classify_split.h"

namespace k2g {

// Warps per block and blocks per SM that the registers are fitted to, and table
// sectors in flight per lane of a probe: 2 x 14 and 3.  On 2M x 150 bp reads, 4
// GB table: 2.30 ms; 2 x 12 and 4: 2.37, 2 x 12 and 5: 2.51, 2 x 16 and 2 (with
// half the entries): 2.38.  An SM holds 13 blocks of them, 26 warps: a block's
// shared memory is 15.6 KB and 1 KB goes with it, of 228.
constexpr int kWcWarps = 2, kWcBlocks = 14;
constexpr int kWcReads = 8;           // most fragments per group
constexpr int kWcEntries = 320;       // entries held before a probe and replay
constexpr int kWcLogSlots = 7, kWcSlots = 1 << kWcLogSlots;   // taxon map slots per warp, shared out among its fragments
constexpr int kWcWindow = 2048;       // bases packed at a time
constexpr int kWcPos = 8;             // l-mer positions per lane
// Longest sequence taken: token positions of a fragment fit kEPosBits.
constexpr uint64_t kWcMaxLen = 1ull << 26;

// Entry kinds (two bits of an entry's meta word: kind, fragment, position).
enum : uint32_t { E_KEY = 0, E_AMBIG = 1, E_BORDER = 2, E_CONT = 3 };
constexpr uint32_t kEPosBits = 27;

struct WcArgs {
  ClassifyArgs a;
  const uint2 *span;      // per taxon: preorder number, one past its subtree's last
  uint32_t log_reads;     // fragments per group = 1 << log_reads <= kWcReads
  uint64_t n_groups;
  // Pieces of long fragments (classify_split.h), one warp each, before the
  // groups: a piece's tokens are those of a read of its own that starts k - 1
  // bases before its cut.  a.pieces and a.n_pieces say which slots hold one;
  // the groups pass over the fragments in a.split_mark.
  uint64_t piece_slots;
};

// One warp's shared memory: what every form of the classification uses ...
struct WcBase {
  // An entry: key (two words, in the top bits; ~0 where nothing is looked
  // up), meta, value.  The replay then keeps its run heads (code, meta) in
  // the first two words.
  uint4 entry[kWcEntries];
  uint32_t mkey[kWcSlots], mcnt[kWcSlots];
  uint4 seq[2 * kWcReads];            // sequences with work: start, length, first item, fragment and tokens before
                                      // (bit 3 of the last: a border comes first)
  uint64_t run_base[kWcReads];
  uint32_t tokens[kWcReads], hits[kWcReads], n_runs[kWcReads];
  uint32_t n_taxa[kWcReads], a_slot[kWcReads];   // taxa of the map, and a slot of them
  uint32_t over, stopped;             // fragment bits
};

// ... and the packed bases of the nucleotide scan.  After a scan the same
// words list the entries whose walk goes on (16 bits each).
struct WcShared : WcBase {
  static constexpr bool kFrames = false, kMany = false;
  uint32_t be[kWcWindow / 16 + 4];
  uint32_t le[kWcWindow / 16 + 4];    // [3] holds the window's first word
  uint32_t inv[kWcWindow / 32 + 4];   // bit per base: not A/C/G/T; [2] is the first word
  __device__ __forceinline__ uint16_t *list() { return reinterpret_cast<uint16_t *>(be); }
};

// The same for fragments of kManyBases and more that stay whole (pairs): those
// with more taxa than a map in shared memory holds are resolved from a map in
// their run region (wc_resolve_many).  A type of its own, since the mere call
// made the other kernels up to 1 % slower; shorter ones gain nothing by it
// (5,000 pairs of 2 x 2 kb with a taxon a k-mer 1.11 and 1.12 ms, 1,000 of 2 x
// 10 kb 41.9 and 10.5).
struct WcSharedMany : WcShared {
  static constexpr bool kMany = true;
};
constexpr uint64_t kManyBases = 8192;

__device__ __forceinline__ uint32_t below(int n) { return n >= 32 ? 0xFFFFFFFFu : (1u << n) - 1u; }
__device__ __forceinline__ int last_bit(uint32_t m) { return 31 - __clz(m); }

// 16 bases to 2 bits each: the first base in the top bits (be), and
// complemented with the first base in the low bits (le).  The result is zero
// exactly when all of them are A/C/G/T, either case.
__device__ __forceinline__ uint32_t wc_pack(const uint4 &v, uint32_t &be, uint32_t &le) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t top[4], odd = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t codes = ((w[i] >> 1) ^ (w[i] >> 2)) & 0x03030303u;
    top[i] = codes * 0x01041040u;                     // four codes gathered into the top byte
    // the letters of the codes, in byte order 0, 2, 1, 3
    const uint32_t want = __byte_perm(0x74676361u, 0u, (codes | (codes >> 12)) & 0xFFFFu);
    odd |= want ^ __byte_perm(w[i] | 0x20202020u, 0u, 0x3120u);
  }
  const uint32_t x = __byte_perm(__byte_perm(top[0], top[1], 0x0073), __byte_perm(top[2], top[3], 0x0073), 0x5410);
  le = ~x;
  const uint32_t r = __brev(x);
  be = ((r >> 1) & 0x55555555u) | ((r & 0x55555555u) << 1);
  return odd;
}

// Bit i set where base i of 16 is not A/C/G/T.
__device__ __forceinline__ uint32_t wc_bad_bases(const uint4 &v) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t bad = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t codes = ((w[i] >> 1) ^ (w[i] >> 2)) & 0x03030303u;
    const uint32_t no = acgt_bytes(w[i], codes) ^ 0x01010101u;
    bad |= ((no * 0x10204080u) >> 28) << (4 * i);     // four flags gathered into a nibble
  }
  return bad;
}

// Bit i set where the quality byte i of 16 is below the threshold.
__device__ __forceinline__ uint32_t wc_low_quality(const uint4 &q, uint32_t qthr4, bool qall) {
  if (qall) return 0xFFFFu;
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  uint32_t bad = 0;
#pragma unroll
  for (int i = 0; i < 4; i++)
    bad |= (((__vcmplts4(w[i], qthr4) & 0x01010101u) * 0x10204080u) >> 28) << (4 * i);
  return bad;
}

// Window minima: m[j] of the five candidates ending at position j, the first
// four positions' reaching into the lane below.
__device__ __forceinline__ void wc_window5(const uint64_t (&c)[kWcPos], uint64_t (&m)[kWcPos]) {
  const uint64_t s6 = min64(c[6], c[7]), s5 = min64(c[5], s6), s4 = min64(c[4], s5);
  const uint64_t p3 = __shfl_up_sync(0xffffffffu, c[7], 1), p2 = __shfl_up_sync(0xffffffffu, s6, 1),
                 p1 = __shfl_up_sync(0xffffffffu, s5, 1), p0 = __shfl_up_sync(0xffffffffu, s4, 1);
  const uint64_t q1 = min64(c[0], c[1]), q2 = min64(q1, c[2]), q3 = min64(q2, c[3]);
  m[0] = min64(p0, c[0]);
  m[1] = min64(p1, q1);
  m[2] = min64(p2, q2);
  m[3] = min64(p3, q3);
  const uint64_t t2 = min64(c[2], c[3]), t1 = min64(c[1], t2);
  const uint64_t u1 = min64(c[4], c[5]), u2 = min64(u1, c[6]), u3 = min64(u2, c[7]);
  m[4] = min64(q3, c[4]);
  m[5] = min64(t1, u1);
  m[6] = min64(t2, u2);
  m[7] = min64(c[3], u3);
}

// The walk of CompactHashTable::Get over one 32-byte sector of the table:
// the value where it ends (0: absent), or kWalkOn.  Cells [off, lim) count.
constexpr uint32_t kWalkOn = 0xFFFFFFFFu;

template <bool WIDE>
__device__ __forceinline__ uint32_t wc_sector(const TableView &t, const Sector &s, uint64_t hc,
                                              uint32_t off, uint32_t lim) {
  const uint32_t c[8] = {s.lo.x, s.lo.y, s.lo.z, s.lo.w, s.hi.x, s.hi.y, s.hi.z, s.hi.w};
  uint32_t res = kWalkOn;
  if constexpr (WIDE) {
    const uint64_t ck = hc >> t.key_shift;
#pragma unroll
    for (int i = 3; i >= 0; i--) {
      const uint64_t cell = ((uint64_t)c[2 * i + 1] << 32) | c[2 * i];
      const uint32_t v = c[2 * i] & t.value_mask;
      const bool match = (uint64_t)(uint32_t)(cell >> t.value_bits) == ck;
      const bool in = (uint32_t)i >= off && (uint32_t)i < lim;
      res = (in && (match || !v)) ? v : res;
    }
  } else {
    const uint32_t ckv = (uint32_t)(hc >> t.key_shift) << t.value_bits;
#pragma unroll
    for (int i = 7; i >= 0; i--) {
      const uint32_t x = c[i] ^ ckv;                             // the value, where the key matches
      const uint32_t u = (c[i] & t.value_mask) ? x : 0u;         // 0: an empty cell
      const bool in = (uint32_t)i >= off && (uint32_t)i < lim;
      res = (in && u <= t.value_mask) ? u : res;
    }
  }
  return res;
}

template <bool WIDE>
__device__ __forceinline__ Sector wc_load(const TableView &t, uint64_t cell) {
  if constexpr (WIDE) return load_sector(reinterpret_cast<const uint32_t *>(t.wide), cell * 2);
  else return load_sector(t.cells, cell);
}

// The rest of a walk, from the sector starting at `base`.  A walk that meets
// every sector (a full table) finds nothing.
template <bool WIDE>
__device__ __forceinline__ uint32_t wc_walk(const TableView &t, uint64_t hc, uint64_t base) {
  constexpr uint32_t N = WIDE ? 4 : 8;
  uint32_t v = kWalkOn;
  for (uint64_t step = 0; step <= t.capacity / N + 1; step++) {
    const uint64_t left = t.capacity - base;
    v = wc_sector<WIDE>(t, wc_load<WIDE>(t, base), hc, 0, left < N ? (uint32_t)left : N);
    if (v != kWalkOn) return v;
    base = left <= N ? 0 : base + N;
  }
  return 0;
}

// A taxon -> tokens map: open addressing over `mask` + 1 slots, key 0 empty.
struct WcMap {
  uint32_t *key, *cnt;
  uint32_t mask, step;   // slot i at key[i * step], cnt[i * step]
  __device__ __forceinline__ uint32_t home(uint32_t taxon) const { return ((taxon * 0x9E3779B1u) >> 16) & mask; }
  // Adds n tokens; the slot, kOld | the slot where the taxon was there
  // already, or ~0 when the map is full.
  static constexpr uint32_t kOld = 0x80000000u;
  __device__ __forceinline__ uint32_t add(uint32_t taxon, uint32_t n) const {
    uint32_t i = home(taxon);
    for (uint32_t probes = 0; probes <= mask; probes++) {
      const uint32_t old = atomicCAS(&key[i * step], 0u, taxon);
      if (old == 0 || old == taxon) {
        atomicAdd(&cnt[i * step], n);
        return old ? i | kOld : i;
      }
      i = (i + 1) & mask;
    }
    return 0xFFFFFFFFu;
  }
  __device__ __forceinline__ uint32_t get(uint32_t taxon) const {
    uint32_t i = home(taxon);
    for (uint32_t probes = 0; probes <= mask; probes++) {
      const uint32_t k = key[i * step];
      if (k == taxon) return cnt[i * step];
      if (k == 0) return 0;
      i = (i + 1) & mask;
    }
    return 0;
  }
};

__device__ __forceinline__ bool in_span(uint2 s, uint32_t pre) { return s.x <= pre && pre < s.y; }

// The call once the highest score's taxa are known to span the preorder
// numbers [lo, hi], `from` being the taxon numbered lo: their LCA, climbed
// until the tokens of its subtree reach `required` (sum_of and in_tree give
// the tokens of a taxon and of a subtree).
template <class SumOf, class InTree>
__device__ __forceinline__ uint32_t wc_climb(const uint32_t *parent, const uint2 *span, uint32_t from,
                                             uint32_t hi, uint32_t required, SumOf sum_of,
                                             InTree in_tree) {
  uint32_t call = from;
  while (call && hi >= __ldg(&span[call].y)) call = __ldg(parent + call);
  uint32_t score = sum_of(call);
  while (call && score < required) {
    score = in_tree(__ldg(span + call));
    if (score >= required) break;
    call = __ldg(parent + call);
  }
  return call;
}

// ResolveTree over `many` <= 32 distinct taxa, in the first lanes (t = 0: none).
__device__ __forceinline__ uint32_t wc_resolve(const uint32_t *parent, const uint2 *span, uint32_t t,
                                               uint32_t n, int many, uint32_t required) {
  const uint2 sp = t ? __ldg(span + t) : make_uint2(0xFFFFFFFFu, 0u);
  uint32_t score = 0;
  for (int i = 0; i < many; i++) {
    const uint2 x = make_uint2(__shfl_sync(0xffffffffu, sp.x, i), __shfl_sync(0xffffffffu, sp.y, i));
    const uint32_t c = __shfl_sync(0xffffffffu, n, i);
    if (t && in_span(x, sp.x)) score += c;
  }
  const uint32_t most = __reduce_max_sync(0xffffffffu, score);
  const bool top = t && score == most;
  const uint32_t lo = __reduce_min_sync(0xffffffffu, top ? sp.x : 0xFFFFFFFFu);
  const uint32_t hi = __reduce_max_sync(0xffffffffu, top ? sp.x : 0u);
  const uint32_t at = __ballot_sync(0xffffffffu, top && sp.x == lo);
  const uint32_t from = __shfl_sync(0xffffffffu, t, __ffs(at) - 1);
  return wc_climb(
      parent, span, from, hi, required,
      [&](uint32_t x) { return __reduce_add_sync(0xffffffffu, t && t == x ? n : 0u); },
      [&](uint2 x) { return __reduce_add_sync(0xffffffffu, t && in_span(x, sp.x) ? n : 0u); });
}

// The highest score seen by a lane, and the taxa that reach it.
struct WcBest {
  uint32_t score = 0, lo = 0xFFFFFFFFu, hi = 0, from = 0;
  __device__ __forceinline__ void see(uint32_t taxon, uint32_t pre, uint32_t s) {
    if (s > score) {
      score = s;
      lo = hi = pre;
      from = taxon;
    } else if (s == score) {
      if (pre < lo) {
        lo = pre;
        from = taxon;
      }
      hi = max(hi, pre);
    }
  }
  // the same over the warp; false when nothing was seen
  __device__ __forceinline__ bool join() {
    const uint32_t most = __reduce_max_sync(0xffffffffu, score);
    if (!most) return false;
    const uint32_t all_lo = __reduce_min_sync(0xffffffffu, score == most ? lo : 0xFFFFFFFFu);
    hi = __reduce_max_sync(0xffffffffu, score == most ? hi : 0u);
    const uint32_t at = __ballot_sync(0xffffffffu, score == most && lo == all_lo);
    from = __shfl_sync(0xffffffffu, from, __ffs(at) - 1);
    return true;
  }
};

// ResolveTree over a map of any size, a taxon per lane at a time: its score
// from its path to the root.
static __device__ __noinline__ uint32_t wc_resolve_map(const uint32_t *parent, const uint2 *span, WcMap m,
                                                       uint32_t required) {
  const uint32_t lane = threadIdx.x & 31;
  WcBest best;
  for (uint32_t i = lane; i <= m.mask; i += 32) {
    const uint32_t t = m.key[i * m.step];
    if (!t) continue;
    uint32_t score = 0;
    for (uint32_t x = t; x; x = __ldg(parent + x)) score += m.get(x);
    best.see(t, __ldg(&span[t].x), score);
  }
  __syncwarp();
  if (!best.join()) return 0;
  return wc_climb(parent, span, best.from, best.hi, required, [&](uint32_t x) { return x ? m.get(x) : 0u; },
                  [&](uint2 x) {
                    uint32_t sum = 0;
                    for (uint32_t i = lane; i <= m.mask; i += 32) {
                      const uint32_t t = m.key[i * m.step];
                      if (t && in_span(x, __ldg(&span[t].x))) sum += m.cnt[i * m.step];
                    }
                    __syncwarp();
                    return __reduce_add_sync(0xffffffffu, sum);
                  });
}

// A hit-list run as this warp wrote it.
__device__ __forceinline__ uint2 wc_run(const uint64_t *runs, uint32_t i) {
  const uint64_t x = *const_cast<const volatile uint64_t *>(runs + i);
  const uint32_t t = (uint32_t)(x >> 32);
  return make_uint2(t < K2G_CODE_AMBIGUOUS ? t : 0u, (uint32_t)x);
}

// ResolveTree from a fragment's runs, for one with more taxa than any map at
// hand holds: quadratic in the runs, spread over the lanes.
static __device__ __noinline__ uint32_t wc_resolve_runs(const uint32_t *parent, const uint2 *span,
                                                        const uint64_t *runs, uint32_t count,
                                                        uint32_t required) {
  const uint32_t lane = threadIdx.x & 31;
  WcBest best;
  for (uint32_t i0 = 0; i0 < count; i0 += 32) {
    const uint2 it = i0 + lane < count ? wc_run(runs, i0 + lane) : make_uint2(0, 0);
    const uint32_t pre = it.x ? __ldg(&span[it.x].x) : 0;
    uint32_t score = 0;
    for (uint32_t j = 0; j < count; j++) {
      const uint2 o = wc_run(runs, j);
      if (o.x && it.x && in_span(__ldg(span + o.x), pre)) score += o.y;
    }
    if (it.x) best.see(it.x, pre, score);
  }
  if (!best.join()) return 0;
  auto sum = [&](auto pick) {
    uint32_t s = 0;
    for (uint32_t i = lane; i < count; i += 32) {
      const uint2 o = wc_run(runs, i);
      if (o.x && pick(o.x)) s += o.y;
    }
    __syncwarp();
    return __reduce_add_sync(0xffffffffu, s);
  };
  return wc_climb(parent, span, best.from, best.hi, required,
                  [&](uint32_t x) { return sum([&](uint32_t t) { return t == x; }); },
                  [&](uint2 x) { return sum([&](uint32_t t) { return in_span(x, __ldg(&span[t].x)); }); });
}

// ResolveTree over a map of `taxa` > 0 taxa in shared memory; `list` holds 32.
__device__ __forceinline__ uint32_t wc_resolve_slots(const uint32_t *parent, const uint2 *span, const WcMap &m,
                                                     uint32_t taxa, uint2 *list, uint32_t required) {
  if (taxa > 32) return wc_resolve_map(parent, span, m, required);
  const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
  int n = 0;
  for (uint32_t i0 = 0; i0 <= m.mask; i0 += 32) {
    const uint32_t t = i0 + lane <= m.mask ? m.key[i0 + lane] : 0;
    const uint32_t b = __ballot_sync(0xffffffffu, t != 0);
    if (t) list[n + __popc(b & lt)] = make_uint2(t, m.cnt[i0 + lane]);
    n += __popc(b);
  }
  __syncwarp();
  const uint2 x = (int)lane < n ? list[lane] : make_uint2(0, 0);
  return wc_resolve(parent, span, x.x, x.y, n, required);
}

// ResolveTree from a fragment's runs, for one with more taxa than any map in
// shared memory holds: a map in the unused part of its run region of `region`
// words -- left zero -- or, where that is too small, the runs themselves (200
// pairs of 2 x 50 kb with thousands of taxa each: 905 ms from the runs alone,
// 42 with the map).
static __device__ __noinline__ uint32_t wc_resolve_many(const uint32_t *parent, const uint2 *span, uint64_t *runs,
                                                        uint32_t count, uint32_t region, uint32_t required) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t room = region > count ? region - count : 0;
  uint32_t slots = 32;
  while (slots < 65536 && 2 * slots <= room) slots *= 2;
  if (slots <= room) {
    uint64_t *at = runs + count;
    uint32_t *mem = reinterpret_cast<uint32_t *>(at);
    const WcMap big{mem, mem + 1, slots - 1, 2};
    for (uint32_t i = lane; i < slots; i += 32) at[i] = 0;
    __syncwarp();
    bool full = false;
    for (uint32_t i = lane; i < count; i += 32) {
      const uint2 x = wc_run(runs, i);
      if (x.x && big.add(x.x, x.y) == 0xFFFFFFFFu) full = true;
    }
    __syncwarp();
    uint32_t call = 0;
    full = __any_sync(0xffffffffu, full);
    if (!full) call = wc_resolve_map(parent, span, big, required);
    __syncwarp();
    for (uint32_t i = lane; i < slots; i += 32) at[i] = 0;
    __syncwarp();
    if (!full) return call;
  }
  return wc_resolve_runs(parent, span, runs, count, required);
}

// ---- the kernel --------------------------------------------------------------

template <bool WIDE, bool HITS, class Shared>
struct Wc {
  const ClassifyArgs &a;
  Shared &s;
  const int lane;
  const uint32_t lt;            // lanes below
  uint64_t f0;                  // first fragment of the group
  uint32_t log_slots;           // taxon map slots per fragment
  uint32_t first_pos;           // position of a fragment's first token
  uint32_t key_shift;           // keys are held in the top bits
  uint64_t toggle_top;
  // carried from one replay to the next (the same in all lanes): the run
  // still open (its fragment ~0: none), the runs its fragment has before it,
  // and the value of the last key
  uint32_t open_code = 0, open_meta = 0xFFFFFFFFu, open_rank = 0, key_taxon = 0;

  // the last unambiguous minimizer of the scan, and its sequence
  uint64_t seen_min = 0;
  uint32_t seen_seq = 0xFFFFFFFFu;

  // Where token groups start among the lane's positions, given their window
  // minima, which of them end a k-mer (emit) and which of those k-mers are
  // ambiguous.  head: the lane's first position is its sequence's first;
  // repeated: lane 0 repeats the item before the pass, its first k - l minima
  // miss the candidates before it; sq: the lane's sequence; n_in: lanes with
  // an item.  cont: starts that continue the last key's taxon.  next_*: the
  // scan state after the pass.
  __device__ __forceinline__ uint32_t starts(const uint64_t (&m)[kWcPos], uint32_t emit, uint32_t amb, bool head,
                                             bool repeated, bool dirty, uint32_t sq, int n_in, uint32_t skip,
                                             uint32_t &cont, uint64_t &next_min, uint32_t &next_seq) const {
    uint32_t start = 0;
    next_min = seen_min;
    next_seq = seen_seq;
    if (!dirty) {
      const uint64_t pm = __shfl_up_sync(0xffffffffu, m[7], 1);
      start = m[0] != pm ? 1u : 0u;
#pragma unroll
      for (int j = 1; j < kWcPos; j++) start |= m[j] != m[j - 1] ? 1u << j : 0u;
      if (head) start |= 1u << skip;   // a sequence's first minimizer is new
      start &= emit;
      next_min = __shfl_sync(0xffffffffu, m[7], n_in - 1);
      next_seq = __shfl_sync(0xffffffffu, sq, n_in - 1);
      return start;
    }
    const uint32_t clear = emit & ~amb & (lane == 0 && repeated ? 0xFFu << skip : 0xFFu);
    uint64_t lm = 0;
#pragma unroll
    for (int j = 0; j < kWcPos; j++) lm = (clear >> j) & 1u ? m[j] : lm;
    // the last unambiguous minimizer before this lane, in its sequence
    const uint32_t have = __ballot_sync(0xffffffffu, clear != 0);
    const int src = (have & lt) ? last_bit(have & lt) : 0;
    uint64_t run_min = __shfl_sync(0xffffffffu, lm, src);
    uint32_t run_seq = __shfl_sync(0xffffffffu, sq, src);
    if (!(have & lt)) {
      run_min = seen_min;
      run_seq = seen_seq;
    }
    bool known = run_seq == sq && !head;
    bool prev_amb = (__shfl_up_sync(0xffffffffu, amb, 1) >> (kWcPos - 1)) & 1u;
    bool fresh = head;
#pragma unroll
    for (int j = 0; j < kWcPos; j++) {
      const bool is_amb = (amb >> j) & 1u, at = (emit >> j) & 1u;
      const bool is_new = !is_amb && !(known && run_min == m[j]);
      if (at && (fresh || is_amb != prev_amb || is_new)) start |= 1u << j;
      if (!is_amb && !is_new) cont |= 1u << j;
      known = known || (at && !is_amb);
      run_min = at && !is_amb ? m[j] : run_min;
      fresh = fresh && !at;
      prev_amb = at ? is_amb : prev_amb;
    }
    if (have) {
      next_min = __shfl_sync(0xffffffffu, lm, last_bit(have));
      next_seq = __shfl_sync(0xffffffffu, sq, last_bit(have));
    }
    return start;
  }

  // Appends the lanes' token groups to the entries, in token order; false
  // (and nothing appended) when they do not fit.  tag: the sequence's word
  // (WcBase::seq); tok0: the token position of the lane's first position.
  __device__ __forceinline__ bool add(int &ne, const uint64_t (&m)[kWcPos], uint32_t start, uint32_t amb,
                                      uint32_t cont, bool border, uint32_t tag, uint32_t tok0, bool dirty) {
    const uint32_t adds = __popc(start) + (border ? 1u : 0u);
    uint32_t upto = adds;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, upto, d);
      if (lane >= d) upto += x;
    }
    const int total = (int)__shfl_sync(0xffffffffu, upto, 31);
    if (ne + total > kWcEntries) return false;
    uint4 *at = s.entry + (uint32_t)ne + upto - adds;
    const uint32_t rtag = (tag & 7u) << kEPosBits;
    const uint32_t meta = rtag + tok0;
    if (border) *at++ = make_uint4(~0u, ~0u, (E_BORDER << 30) | rtag | ((tag >> 4) - 1), 0);
    if (!dirty) {
#pragma unroll
      for (int j = 0; j < kWcPos; j++)
        if ((start >> j) & 1u) *at++ = make_uint4((uint32_t)m[j], (uint32_t)(m[j] >> 32), meta + j, 0);
    } else {
#pragma unroll
      for (int j = 0; j < kWcPos; j++) {
        const bool is_amb = (amb >> j) & 1u, is_cont = (cont >> j) & 1u;
        const uint64_t key = is_amb || is_cont ? ~0ull : m[j];
        const uint32_t kind = is_amb ? E_AMBIG << 30 : is_cont ? E_CONT << 30 : 0u;
        if ((start >> j) & 1u) *at++ = make_uint4((uint32_t)key, (uint32_t)(key >> 32), kind | (meta + j), 0);
      }
    }
    ne += total;
    return true;
  }

  __device__ __forceinline__ uint64_t key_of(uint64_t top) const { return (top ^ toggle_top) >> key_shift; }
  __device__ __forceinline__ uint64_t top_of(int i) const {
    return *reinterpret_cast<const uint64_t *>(&s.entry[i]);
  }

  __device__ __forceinline__ WcMap map_of(uint32_t r) const {
    return WcMap{s.mkey + (r << log_slots), s.mcnt + (r << log_slots), (1u << log_slots) - 1u, 1u};
  }

  // Get() for every key entry: the home sectors of all, then the walks that
  // go on (about one in five at load 0.7).
  __device__ __forceinline__ void probe(int ne) {
    constexpr int B = 3;
    constexpr uint32_t N = WIDE ? 4 : 8, kLogN = WIDE ? 2 : 3;
    const TableView &t = a.table;
    uint16_t *list = s.list();
    // the table's last sector where it is a partial one: its padding cells
    // look empty, so an absent key found there is looked up once more
    const uint64_t partial = t.capacity & (N - 1) ? t.capacity & ~(uint64_t)(N - 1) : ~0ull;
    int n_list = 0;
    bool redo = false;
#pragma unroll 1
    for (int i0 = 0; i0 < ne; i0 += 32 * B) {
      uint64_t hc[B], idx[B];
      Sector sec[B];
      uint32_t ask = 0;
#pragma unroll
      for (int b = 0; b < B; b++) {
        const int i = i0 + 32 * b + lane;
        const uint64_t top = i < ne ? top_of(i) : ~0ull;
        hc[b] = murmur3(key_of(top));
        // a subsampled minimizer (-M) is not looked up: its value is 0
        const bool look = top != ~0ull && hc[b] >= a.scan.min_hash;
        idx[b] = look ? mod_once(hc[b], t.div) : 0;
        ask |= look ? 1u << b : 0u;
        sec[b] = wc_load<WIDE>(t, idx[b] & ~(uint64_t)(N - 1));
      }
#pragma unroll
      for (int b = 0; b < B; b++) {
        const int i = i0 + 32 * b + lane;
        const bool look = (ask >> b) & 1u;
        const uint32_t v = wc_sector<WIDE>(t, sec[b], hc[b], (uint32_t)idx[b] & (N - 1), N);
        const uint64_t base = idx[b] & ~(uint64_t)(N - 1);
        const bool again = look && !v && base == partial;
        const bool on = look && (v == kWalkOn || again);
        const uint32_t m = __ballot_sync(0xffffffffu, on);
        if (on) list[n_list + __popc(m & lt)] = (uint16_t)(i | (again ? 0x8000 : 0));
        // a walk that goes on leaves its sector's number instead of a value
        if (look) s.entry[i].w = on ? (uint32_t)(base >> kLogN) : v;
        n_list += __popc(m);
        redo |= again;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int e = lane; e < n_list; e += 32) {
      const uint32_t x = list[e], i = x & 0x7FFFu;
      const uint64_t hc = murmur3(key_of(top_of((int)i)));
      uint64_t base = (uint64_t)s.entry[i].w << kLogN;
      uint32_t v = 0;
      if (x & 0x8000u) {
        const uint64_t idx = fast_mod(hc, t.div);
        v = wc_sector<WIDE>(t, wc_load<WIDE>(t, base), hc, (uint32_t)idx & (N - 1), (uint32_t)(t.capacity - base));
      }
      if (!(x & 0x8000u) || v == kWalkOn) v = wc_walk<WIDE>(t, hc, base + N >= t.capacity ? 0 : base + N);
      s.entry[i].w = v;
    }
    __syncwarp();
  }

  // Room for n events, one atomic for the warp.
  __device__ __forceinline__ uint64_t take_events(uint32_t n) {
    unsigned long long base = 0;
    if (lane == 0 && n) base = atomicAdd(a.hits_used, (unsigned long long)n);
    return __shfl_sync(0xffffffffu, base, 0);
  }

  // add_kmer events (src/classify.cc:869-873); the token position is the
  // ordinal (monotone in token order).
  __device__ __forceinline__ void emit_events(bool event, int i, uint32_t r, uint32_t pos, uint32_t v,
                                              uint64_t &base) {
    const uint32_t m = __ballot_sync(0xffffffffu, event);
    if (!m) return;
    if (a.cls.quick) base = take_events(__popc(m));
    const uint64_t at = base + __popc(m & lt);
    base += __popc(m);
    if (!event) return;
    if (at < a.hits_cap) {
      a.hit_keys[at] = key_of(top_of(i));
      a.hit_taxa[at] = v;
      a.hit_order[at] = ((a.frag_base + f0 + r) << 32) | pos;
    } else {
      atomicOr(a.status, STATUS_HITS_OVERFLOW);
    }
  }

  // (a border between frames, or between mates)
  __device__ __forceinline__ uint32_t border_code(uint32_t r, uint32_t pos) const {
    if constexpr (Shared::kFrames) return pos == s.mate_pos[r] ? K2G_CODE_MATE_BORDER : K2G_CODE_FRAME_BORDER;
    else return K2G_CODE_MATE_BORDER;
  }

  // Quick mode: the lookup whose hit reaches the minimum ends its fragment;
  // it and everything after it leave no tokens.  Returns whether the entry
  // stands; `hit` is cleared where it does not (the ending lookup keeps its
  // event).
  __device__ __forceinline__ bool quick_cut(bool act, bool &hit, bool &event, uint32_t r, uint32_t pos) {
    const uint32_t le = lt | (1u << lane);
    const uint32_t up_r = __shfl_up_sync(0xffffffffu, r, 1);
    const uint32_t firsts = __ballot_sync(0xffffffffu, act && (lane == 0 || up_r != r));
    const uint32_t seg = le & ~below(firsts & le ? last_bit(firsts & le) : 0);
    const uint32_t hb = __ballot_sync(0xffffffffu, hit);
    const uint32_t total = s.hits[r] + __popc(hb & seg);
    const bool was = (s.stopped >> r) & 1u;
    const bool stop = hit && !was && (int32_t)total >= a.cls.min_hit_groups;
    const uint32_t sb = __ballot_sync(0xffffffffu, stop);
    const bool first = stop && !(sb & seg & lt);
    act = act && !was && !(sb & seg);
    event = hit && (act || first);
    __syncwarp();
    if (first) {
      s.tokens[r] = pos;
      atomicOr(&s.stopped, 1u << r);
    }
    hit = event;   // the ending lookup counts as a hit group
    return act;
  }

  // Hit-list runs and taxa from the entries [0, ne); with `last`, the open
  // run is written too.
  __device__ __forceinline__ void replay(int ne, bool conts, bool last) {
    uint64_t events = 0;   // where the next event goes
    if (HITS && !a.cls.quick) {
      // every value is a hit: only key entries have one yet
      uint32_t n = 0;
      for (int i0 = 0; i0 < ne; i0 += 32)
        n += __popc(__ballot_sync(0xffffffffu, i0 + lane < ne && s.entry[i0 + lane].w));
      events = take_events(n);
    }
    // 1. an entry unlike the one before it heads a run
    int nh = 0;
    uint32_t prev_code = open_code, prev_r = open_meta == 0xFFFFFFFFu ? 8u : open_meta >> kEPosBits;
#pragma unroll 1
    for (int i0 = 0; i0 < ne; i0 += 32) {
      const int i = i0 + lane;
      bool act = i < ne;
      const uint2 mv = act ? *reinterpret_cast<const uint2 *>(&s.entry[i].z) : make_uint2(0, 0);
      const uint32_t kind = mv.x >> 30, where = mv.x & below(30), r = where >> kEPosBits;
      uint32_t v = mv.y;
      bool hit = v != 0;   // (a value of a key)
      if (conts) {
        // a continued group takes the taxon of the last key before it
        const uint32_t keys = __ballot_sync(0xffffffffu, act && kind == E_KEY);
        const uint32_t x = __shfl_sync(0xffffffffu, v, (keys & lt) ? last_bit(keys & lt) : 0);
        if (kind == E_CONT) v = (keys & lt) ? x : key_taxon;
        if (keys) key_taxon = __shfl_sync(0xffffffffu, v, last_bit(keys));
      }
      bool event = hit;
      if (a.cls.quick) act = quick_cut(act, hit, event, r, where & below(kEPosBits));
      if constexpr (HITS) emit_events(event, i, r, where & below(kEPosBits), v, events);
      if (hit) atomicAdd(&s.hits[r], 1u);
      const uint32_t code = kind == E_AMBIG    ? K2G_CODE_AMBIGUOUS
                            : kind == E_BORDER ? border_code(r, where & below(kEPosBits))
                                               : v;
      const uint32_t acts = __ballot_sync(0xffffffffu, act);
      const int prev = (acts & lt) ? last_bit(acts & lt) : -1;
      const uint32_t pc = __shfl_sync(0xffffffffu, code, prev & 31), pr = __shfl_sync(0xffffffffu, r, prev & 31);
      const bool head = act && (prev < 0 ? prev_r != r || prev_code != code : pr != r || pc != code);
      const uint32_t heads = __ballot_sync(0xffffffffu, head);
      if (head) *reinterpret_cast<uint2 *>(&s.entry[nh + __popc(heads & lt)]) = make_uint2(code, where);
      nh += __popc(heads);
      if (acts) {
        prev_code = __shfl_sync(0xffffffffu, code, last_bit(acts));
        prev_r = __shfl_sync(0xffffffffu, r, last_bit(acts));
      }
      __syncwarp();
    }
    if (!conts) key_taxon = prev_code;   // (keys and borders only)
    // 2. runs: item 0 is the open one, item j the j-th head; each ends where
    // the next begins, or with its fragment
    const int n_items = nh + 1;
#pragma unroll 1
    for (int j0 = 0; j0 < n_items; j0 += 32) {
      const int j = j0 + lane;
      uint2 it = make_uint2(open_code, open_meta), nx = make_uint2(0, 0xFFFFFFFFu);
      if (j > 0 && j <= nh) it = *reinterpret_cast<const uint2 *>(&s.entry[j - 1]);
      if (j < nh) nx = *reinterpret_cast<const uint2 *>(&s.entry[j]);
      const bool ends = j < n_items && it.y != 0xFFFFFFFFu && (j < nh || last);
      const uint32_t start = it.y & below(kEPosBits), r = (it.y >> kEPosBits) & 7u;
      // runs of the fragment before this one (its first run starts at first_pos)
      const uint32_t le = lt | (1u << lane);
      const uint32_t firsts = __ballot_sync(0xffffffffu, j < n_items && it.y != 0xFFFFFFFFu && start == first_pos);
      const uint32_t rank = (firsts & le) ? (uint32_t)(lane - last_bit(firsts & le)) : open_rank + (uint32_t)lane;
      if (ends) {
        const bool same = (nx.y >> kEPosBits) == (it.y >> kEPosBits);
        const uint32_t n = (same ? nx.y & below(kEPosBits) : s.tokens[r]) - start;
        const uint64_t at = s.run_base[r] + rank;
        bool room = at < a.runs_cap;
        // (six frames can have more runs than their fragment's region holds)
        if constexpr (Shared::kFrames) room = room && rank < s.room[r];
        if (room) a.runs[at] = ((uint64_t)it.x << 32) | n;
        else atomicOr(a.status, STATUS_RUNS_OVERFLOW);
        if (!same) s.n_runs[r] = rank + 1;
        if (it.x && it.x < K2G_CODE_AMBIGUOUS) {
          const uint32_t slot = map_of(r).add(it.x, n);
          if (slot == 0xFFFFFFFFu) {
            atomicOr(&s.over, 1u << r);   // resolved from the fragment's runs
          } else if (!(slot & WcMap::kOld)) {
            atomicAdd(&s.n_taxa[r], 1u);
            s.a_slot[r] = (r << log_slots) + slot;
          }
        }
      }
      const int tail = min(31, n_items - 1 - j0);
      const uint32_t tail_rank = __shfl_sync(0xffffffffu, rank, tail);
      if (j0 + 32 >= n_items) {
        if (nh) {
          open_code = __shfl_sync(0xffffffffu, it.x, tail);
          open_meta = __shfl_sync(0xffffffffu, it.y, tail);
        }
        open_rank = tail_rank;
      } else {
        open_rank = tail_rank + 1;
      }
    }
    __syncwarp();
  }

  // The calls and outputs of the group's fragments: lane r writes fragment r
  // where `out` says so; total: the tokens its confidence counts.
  __device__ __forceinline__ void finish(const uint2 *span, bool out, uint64_t total) {
    uint32_t call = 0, required = 0, taxa = 0;
    if (out) {
      required = (uint32_t)ceil(__dmul_rn(a.cls.confidence, (double)total));
      taxa = (s.over >> lane) & 1u ? 0xFFFFFFFFu : s.n_taxa[lane];
      // one taxon: it, or nothing (its ancestors hold no more tokens)
      if (taxa == 1) {
        const uint32_t at = s.a_slot[lane];
        call = s.mcnt[at] >= required ? s.mkey[at] : 0u;
      }
    }
    for (uint32_t todo = __ballot_sync(0xffffffffu, taxa > 1); todo; todo &= todo - 1) {
      const uint32_t r = (uint32_t)__ffs(todo) - 1;
      const uint32_t need = __shfl_sync(0xffffffffu, required, r), many = __shfl_sync(0xffffffffu, taxa, r);
      // (the entries are done with: their memory serves as scratch)
      uint2 *list = reinterpret_cast<uint2 *>(s.entry);
      uint32_t got = 0;
      if (many != 0xFFFFFFFFu) {
        got = wc_resolve_slots(a.parent, span, map_of(r), many, list, need);
      } else {
        // more taxa than its share of the map: count its runs into a larger one
        constexpr uint32_t kBig = 512;
        static_assert(32 * sizeof(uint2) + kBig * 8 <= sizeof(s.entry), "scratch");
        uint32_t *mem = reinterpret_cast<uint32_t *>(list + 32);
        const WcMap big{mem, mem + kBig, kBig - 1, 1};
        for (uint32_t i = lane; i < 2 * kBig; i += 32) mem[i] = 0;
        __syncwarp();
        const uint64_t base = s.run_base[r];
        const uint32_t n = base >= a.runs_cap ? 0u : (uint32_t)min((uint64_t)s.n_runs[r], a.runs_cap - base);
        uint32_t added = 0;
        bool full = false;
        for (uint32_t i = lane; i < n; i += 32) {
          const uint2 x = wc_run(a.runs + base, i);
          const uint32_t slot = x.x ? big.add(x.x, x.y) : WcMap::kOld;
          full |= slot == 0xFFFFFFFFu;
          added += slot < kBig ? 1u : 0u;
        }
        __syncwarp();
        added = __reduce_add_sync(0xffffffffu, added);
        if (__any_sync(0xffffffffu, full)) {
          if constexpr (Shared::kMany) {
            const uint64_t f = f0 + r, per = a.cls.paired ? 2 : 1;
            const uint64_t end = base + (a.seq_off[(f + 1) * per] - a.seq_off[f * per]) + 2;
            got = wc_resolve_many(a.parent, span, a.runs + base, n, (uint32_t)(min(end, a.runs_cap) - base), need);
          } else {
            got = wc_resolve_runs(a.parent, span, a.runs + base, n, need);
          }
        } else {
          got = wc_resolve_slots(a.parent, span, big, added, list, need);
        }
      }
      __syncwarp();
      if (lane == (int)r) call = got;
    }
    if (out) {
      const uint64_t f = f0 + lane;
      const uint32_t groups = s.hits[lane];
      if ((int32_t)groups < a.cls.min_hit_groups) call = 0;
      a.call[f] = call;
      if (a.hit_groups) a.hit_groups[f] = groups;
      if (a.hitlist_off) a.hitlist_off[f] = s.run_base[lane];
      if (a.hitlist_len) a.hitlist_len[f] = s.n_runs[lane];
      if (call && a.taxon_reads) atomicAdd(a.taxon_reads + call, 1ull);
    }
  }
};

// LONG: the call's long fragments come as pieces.  Shared: WcShared, or
// WcSharedMany where long ones stay whole.
template <bool WIDE, bool HITS, bool LONG, class Shared>
__global__ void __launch_bounds__(kWcWarps * 32, kWcBlocks) warp_classify_kernel(WcArgs wa) {
  extern __shared__ __align__(16) unsigned char smem[];
  const ClassifyArgs &a = wa.a;
  // (whole warps return: the block has no barriers)
  const uint64_t task = blockIdx.x * (uint64_t)kWcWarps + (threadIdx.x >> 5);
  bool piece = false;
  uint64_t f0 = 0;
  uint32_t hi = 0, first_pos = 0;     // of a piece: the k-mers ending at k - 1 + first_pos .. hi - 1
  if constexpr (LONG) {
    piece = task < wa.piece_slots;
    if (task >= wa.piece_slots + wa.n_groups || (piece && task >= (uint64_t)*a.n_pieces)) return;
    f0 = (task - wa.piece_slots) << wa.log_reads;
    if (piece) {
      f0 = a.pieces[task].frag;
      first_pos = a.pieces[task].lo - (uint32_t)(a.scan.k - 1);
      hi = a.pieces[task].hi;
      if (!hi) return;
    }
  } else {
    if (task >= wa.n_groups) return;
    f0 = task << wa.log_reads;
  }
  Shared &s = reinterpret_cast<Shared *>(smem)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u, le = lt | (1u << lane);
  const int k = a.scan.k, l = a.scan.l;
  const int nr = piece ? 1 : (int)min((uint64_t)1 << wa.log_reads, a.n_frags - f0);
  const int per = a.cls.paired ? 2 : 1, ns = nr * per;
  const uint32_t key_shift = 64u - 2u * (uint32_t)l;
  Wc<WIDE, HITS, Shared> w{a, s, lane, lt, f0, piece ? kWcLogSlots : kWcLogSlots - wa.log_reads, first_pos, key_shift,
                   a.scan.toggle << key_shift};
  const uint64_t mask_top = (a.scan.spaced_mask ? a.scan.spaced_mask & a.scan.lmer_mask : a.scan.lmer_mask)
                            << key_shift;

  // ---- the group's sequences: lane i holds sequence i
  uint64_t o = lane <= ns ? a.seq_off[f0 * per + (piece ? 0 : lane)] : 0;
  const uint64_t runs_at = o;
  if (piece) o += lane ? hi : first_pos;
  const uint64_t o0 = __shfl_sync(0xffffffffu, o, 0);
  const uint64_t o_end = __shfl_sync(0xffffffffu, o, ns);
  const uint64_t o_next = __shfl_down_sync(0xffffffffu, o, 1);
  // (a fragment that its pieces carry has no part in the group)
  bool mine = lane < ns;
  if constexpr (LONG) mine = mine && (piece || !a.split_mark[f0 + lane / per]);
  const uint32_t len = mine ? (uint32_t)(o_next - o) : 0;
  const uint32_t kmers = len >= (uint32_t)k ? len - (uint32_t)k + 1 : 0;
  const bool mate2 = per == 2 && (lane & 1);
  const uint32_t mate1_kmers = __shfl_up_sync(0xffffffffu, kmers, 1);
  const uint32_t mate2_kmers = __shfl_down_sync(0xffffffffu, kmers, 1);
  // work items: 8 positions each from the first l-mer's end on; a second
  // mate without k-mers keeps one item for the mate border
  const uint32_t items = kmers ? (len - (uint32_t)(l - 1) + kWcPos - 1) / kWcPos : (mate2 && mine ? 1u : 0u);
  uint32_t incl = items;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += x;
  }
  const uint32_t first_item = items ? incl - items : 0xFFFFFFFFu;
  const uint32_t n_items = __shfl_sync(0xffffffffu, incl, 31);
  const uint32_t busy = __ballot_sync(0xffffffffu, items != 0);
  // stream coordinates: bytes from the 16-byte aligned address at or before
  // the group's first base
  const uint8_t *origin = a.bases + o0;
  const uint32_t lead = (uint32_t)((uintptr_t)origin & 15u);
  origin -= lead;
  const uint8_t *qorigin = nullptr;
  if (a.quals && a.cls.min_quality > 0) qorigin = a.quals + o0 - lead;
  const uint32_t stream_end = lead + (uint32_t)(o_end - o0);
  if (items)
    s.seq[__popc(busy & lt)] = make_uint4(lead + (uint32_t)(o - o0), len, first_item,
                                          (uint32_t)(lane / per) | (mate2 ? 8u | ((mate1_kmers + 1) << 4) : first_pos << 4));
  if (lane < ns && lane % per == 0) {
    const int r = lane / per;
    s.run_base[r] = runs_at + 2 * (f0 + r + a.frag_off) + first_pos;
    s.tokens[r] = per == 2 ? kmers + 1 + mate2_kmers : first_pos + kmers;
    s.hits[r] = 0;
    s.n_runs[r] = 0;
    s.n_taxa[r] = 0;
  }
  if (lane == 0) s.over = s.stopped = 0;
#pragma unroll
  for (int i = 0; i < kWcSlots; i += 128) {
    *reinterpret_cast<uint4 *>(&s.mkey[i + 4 * lane]) = make_uint4(0, 0, 0, 0);
    *reinterpret_cast<uint4 *>(&s.mcnt[i + 4 * lane]) = make_uint4(0, 0, 0, 0);
  }
  __syncwarp();

  // ---- scan, with a probe and replay whenever the entries are full
  uint32_t g0 = 0;                    // first item of the pass
  uint32_t win_lo = 0, win_hi = 0;    // bases packed in shared memory
  bool dirty = false;                 // ambiguous bases seen in the group
  int ne = 0;
  bool own0 = true;                   // lane 0's item is not a repeated one
  (void)own0;
  bool done = n_items == 0;
  while (!done) {
    bool full = false;
#pragma unroll 1
    while (!done && !full) {
      // item of this lane: the sequence whose first item is the last at or
      // before it.  A pass that goes on inside a sequence repeats the item
      // before in lane 0, for the lane above.
      const uint32_t g = g0 + (uint32_t)lane;
      const uint32_t rel = first_item - g0;   // (wraps for earlier sequences)
      const uint32_t starts = __reduce_or_sync(0xffffffffu, rel < 32 ? 1u << rel : 0u);
      const uint32_t before = __popc(__ballot_sync(0xffffffffu, first_item < g0));
      const uint32_t sq = before + __popc(starts & le) - 1;
      const uint4 seq = s.seq[sq];
      const bool head = (starts >> lane) & 1u;
      const int p0 = l - 1 + kWcPos * (int)(g - seq.z);
      const int q0 = (int)seq.x + p0;
      const int n_last = (int)min(31u, n_items - 1 - g0);
      const int qb = __shfl_sync(0xffffffffu, q0, n_last) + kWcPos - 1;
      if (qb >= (int)win_hi) {
        // pack the bases from this pass's first on
        win_lo = (uint32_t)(__shfl_sync(0xffffffffu, q0, 0) - (l - 1)) & ~15u;
        win_hi = win_lo + kWcWindow;
        const uint32_t end = min(stream_end, win_hi);
        __syncwarp();
#pragma unroll 1
        for (uint32_t c0 = win_lo; c0 < end; c0 += 32 * 16) {
          const uint32_t c = c0 + 16 * (uint32_t)lane;
          const bool have = c < end;
          const uint4 v = have ? __ldg(reinterpret_cast<const uint4 *>(origin + c))
                               : make_uint4(0x41414141u, 0x41414141u, 0x41414141u, 0x41414141u);
          uint32_t be, lo, bad = 0;
          const uint32_t odd = wc_pack(v, be, lo);
          if (__any_sync(0xffffffffu, odd) || qorigin) {
            bad = wc_bad_bases(v);
            if (qorigin && have) {
              const int thr = 33 + a.cls.min_quality;
              bad |= wc_low_quality(__ldg(reinterpret_cast<const uint4 *>(qorigin + c)),
                                    ((uint32_t)min(thr, 127) & 0xFFu) * 0x01010101u, thr > 127);
            }
            // bytes outside the group's sequences do not count
            if (c < lead) bad &= 0xFFFFu << (lead - c);
            if (c + 16 > stream_end) bad &= have ? 0xFFFFu >> (c + 16 - stream_end) : 0u;
            dirty |= __any_sync(0xffffffffu, bad != 0);
          }
          if (have) {
            const uint32_t j = (c - win_lo) >> 4;
            s.be[j] = be;
            s.le[j + 3] = lo;
            reinterpret_cast<uint16_t *>(s.inv + 2)[j] = (uint16_t)bad;
          }
        }
        __syncwarp();
      }
      // (items behind a gap that the window does not reach wait for a later pass)
      bool in = g < n_items;
      int n_in = 32;
      if constexpr (LONG) {
        in = in && q0 + kWcPos <= (int)win_hi;
        n_in = __popc(__ballot_sync(0xffffffffu, in));
      } else {
        own0 = g0 == 0;
      }
      const bool own = in && (lane > 0 || own0);
      // candidates of the 8 positions, in the top 2l bits
      uint64_t c[kWcPos];
      {
        const uint32_t at = in ? (uint32_t)(q0 - (l - 1)) - win_lo : 0u, wi = at >> 4, sh = 2 * (at & 15u);
        const uint32_t b0 = s.be[wi], b1 = s.be[wi + 1], b2 = s.be[wi + 2], b3 = s.be[wi + 3];
        const uint32_t A = __funnelshift_l(b1, b0, sh), B = __funnelshift_l(b2, b1, sh), C = __funnelshift_l(b3, b2, sh);
        const uint32_t to = in ? (uint32_t)(q0 + kWcPos - 1) - win_lo : 0u, we = to >> 4, ts = 30 - 2 * (to & 15u);
        const uint32_t e0 = s.le[we], e1 = s.le[we + 1], e2 = s.le[we + 2], e3 = s.le[we + 3];
        const uint32_t X = __funnelshift_l(e0, e1, ts), Y = __funnelshift_l(e1, e2, ts), Z = __funnelshift_l(e2, e3, ts);
#pragma unroll
        for (int j = 0; j < kWcPos; j++) {
          const uint32_t fh = j ? __funnelshift_l(B, A, 2 * j) : A, fl = j ? __funnelshift_l(C, B, 2 * j) : B;
          const int t = 2 * (kWcPos - 1 - j);
          const uint32_t rh = t ? __funnelshift_l(Y, Z, t) : Z, rl = t ? __funnelshift_l(X, Y, t) : Y;
          const uint64_t f = ((uint64_t)fh << 32) | fl, r = ((uint64_t)rh << 32) | rl;
          c[j] = ((f < r ? f : r) & mask_top) ^ w.toggle_top;
        }
      }
      // positions of this lane that end a k-mer
      const int n_pos = min(kWcPos, max(0, (int)seq.y - p0));
      uint32_t emit = in ? (1u << n_pos) - 1u : 0u;
      if (head) emit &= 0xFFu << (k - l);
      uint32_t amb = 0;
      if (dirty) {
        // bit i of `v` is base q0 - 34 + i
        const uint32_t b = in ? (uint32_t)(q0 - 34 - (int)win_lo + 64) : 64u;
        const uint32_t *iv = s.inv + (b >> 5);
        const uint32_t i0 = iv[0], i1 = iv[1], i2 = iv[2];
        const uint64_t v = ((uint64_t)__funnelshift_r(i1, i2, b & 31) << 32) | __funnelshift_r(i0, i1, b & 31);
        const uint64_t lm = (1ull << l) - 1, am = (1ull << (k - 1)) - 1;
#pragma unroll
        for (int j = 0; j < kWcPos; j++) {
          if ((v >> (35 + j - l)) & lm) c[j] = ~0ull;
          if ((v >> (36 + j - k)) & am) amb |= 1u << j;
        }
      }
      uint64_t m[kWcPos];
      wc_window5(c, m);
      // token groups
      uint32_t cont = 0;
      uint64_t next_min;
      uint32_t next_seq;
      uint32_t start = w.starts(m, emit, amb, head, !own0, dirty, sq, n_in, (uint32_t)(k - l), cont, next_min, next_seq);
      if (!own) start = 0;
      const uint32_t tok0 = (seq.w >> 4) + (uint32_t)(p0 - (k - 1));
      full = !w.add(ne, m, start, amb, cont, own && head && (seq.w & 8u), seq.w, tok0, dirty);
      if (!full) {   // (else the pass is redone after a replay)
        w.seen_min = next_min;
        w.seen_seq = next_seq;
        done = g0 + (uint32_t)n_in >= n_items;
        if constexpr (LONG) own0 = n_in < 32 && ((starts >> n_in) & 1u);   // the next item begins a sequence
        g0 += (uint32_t)n_in - (LONG && own0 ? 0u : 1u);
      }
    }
    __syncwarp();
    w.probe(ne);
    win_hi = 0;   // the list of the probe lay in the packed words
    w.replay(ne, dirty, done);
    ne = 0;
  }

  if (LONG && piece) {   // the merge resolves its fragment
    if (lane == 0) {
      SplitPiece &pc = a.pieces[task];
      pc.hit_groups = s.hits[0];
      pc.tokens = s.tokens[0] - first_pos;
      pc.n_runs = s.n_runs[0];
    }
    return;
  }

  bool out = lane < nr;
  if constexpr (LONG) out = out && !a.split_mark[f0 + lane];
  uint64_t total = 0;
  if (out) total = s.tokens[lane] - (a.cls.paired ? 1u : 0u);
  w.finish(wa.span, out, total);
}

// ---- the fragments their pieces carried ---------------------------------------

constexpr int kMergeWarps = 4;
constexpr uint32_t kMergeSlots = 512;

struct MergeShared {
  uint32_t mkey[kMergeSlots], mcnt[kMergeSlots];
  uint2 list[32];
};

// One warp per fragment.  The pieces' runs lie in the fragment's run region,
// shifted by the tokens before each piece; they are moved to the front in
// place (a run is never written behind where it is read: a piece has no more
// runs than tokens), equal runs that meet at a cut joining as they would have
// in one pass.  The runs are counted into a taxon map on the way.
static __global__ void __launch_bounds__(kMergeWarps * 32)
warp_merge_kernel(ClassifyArgs a, const uint2 *span, SplitBufs b) {
  __shared__ MergeShared shared[kMergeWarps];
  MergeShared &s = shared[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t n_split = min((uint64_t)b.ctr[1], b.frags_cap);
  const uint32_t k = (uint32_t)a.scan.k;
  const WcMap small{s.mkey, s.mcnt, kMergeSlots - 1, 1};
  for (uint64_t sid = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; sid < n_split;
       sid += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const SplitFrag sf = b.frags[sid];
    if (!sf.n) continue;
    const uint64_t f = sf.frag, o0 = a.seq_off[f], len = a.seq_off[f + 1] - o0;
    const uint64_t base = o0 + 2 * (f + a.frag_off);
    for (uint32_t i = lane; i < kMergeSlots; i += 32) s.mkey[i] = s.mcnt[i] = 0;
    __syncwarp();
    uint32_t hits = 0, w = 0, added = 0;
    bool full = false, have = false;
    uint64_t open = 0;   // the last run so far, not written yet
    for (uint32_t j = 0; j < sf.n; j++) {
      const SplitPiece &pc = b.pieces[sf.first + j];
      hits += pc.hit_groups;
      const uint64_t from = base + (pc.lo - (k - 1));
      // (past runs_cap nothing was written, and the overflow was flagged)
      const uint32_t n = from >= a.runs_cap ? 0u : (uint32_t)min((uint64_t)pc.n_runs, a.runs_cap - from);
      constexpr uint32_t U = 4;
      for (uint32_t i0 = 0; i0 < n; i0 += 32 * U) {
        uint64_t x[U];
#pragma unroll
        for (uint32_t u = 0; u < U; u++) {
          const uint32_t i = i0 + 32 * u + lane;
          x[u] = i < n ? a.runs[from + i] : 0;
        }
        __syncwarp();
        // the first of these joins the open run or follows it
        const uint64_t head = __shfl_sync(0xffffffffu, x[0], 0);
        const bool joins = have && (uint32_t)(head >> 32) == (uint32_t)(open >> 32);
        const uint32_t m = min(32 * U, n - i0);
        if (have && !joins) {
          if (lane == 0) a.runs[base + w] = open;
          w++;
        }
        const uint64_t first = joins ? open + (uint32_t)head : head;
        // all but the last are final
#pragma unroll
        for (uint32_t u = 0; u < U; u++) {
          const uint32_t i = 32 * u + lane;
          if (i + 1 < m) a.runs[base + w + i] = i ? x[u] : first;
          const uint32_t t = (uint32_t)(x[u] >> 32);
          if (i < m && t && t < K2G_CODE_AMBIGUOUS) {
            const uint32_t slot = small.add(t, (uint32_t)x[u]);
            full |= slot == 0xFFFFFFFFu;
            added += slot < kMergeSlots ? 1u : 0u;
          }
        }
        w += m - 1;
        uint64_t last = first;
#pragma unroll
        for (uint32_t u = 0; u < U; u++) {
          const uint64_t y = __shfl_sync(0xffffffffu, x[u], (m - 1) & 31);
          if (m > 1 && (m - 1) >> 5 == u) last = y;
        }
        open = last;
        have = true;
        __syncwarp();
      }
    }
    if (have) {
      if (base + w < a.runs_cap) {
        if (lane == 0) a.runs[base + w] = open;
      } else if (lane == 0) {
        atomicOr(a.status, STATUS_RUNS_OVERFLOW);
      }
      w++;
    }
    __syncwarp();
    const uint32_t total = (uint32_t)(len - (k - 1));
    const uint32_t required = (uint32_t)ceil(__dmul_rn(a.cls.confidence, (double)total));
    added = __reduce_add_sync(0xffffffffu, added);
    uint32_t call = 0;
    if (__any_sync(0xffffffffu, full)) {
      const uint32_t n = base >= a.runs_cap ? 0u : (uint32_t)min((uint64_t)w, a.runs_cap - base);
      call = wc_resolve_many(a.parent, span, a.runs + base, n, base < a.runs_cap ? (uint32_t)(min(base + len + 2, a.runs_cap) - base) : 0u,
                             required);
    } else if (added) {
      call = wc_resolve_slots(a.parent, span, small, added, s.list, required);
    }
    if ((int32_t)hits < a.cls.min_hit_groups) call = 0;
    if (lane == 0) {
      a.call[f] = call;
      if (a.hit_groups) a.hit_groups[f] = hits;
      if (a.hitlist_off) a.hitlist_off[f] = base;
      if (a.hitlist_len) a.hitlist_len[f] = w;
      if (call && a.taxon_reads) atomicAdd(a.taxon_reads + call, 1ull);
    }
    __syncwarp();
  }
}

}  // namespace k2g
