// The distinct minimizers of sequence blocks in the build's order, block by
// block in shared memory (included by build_gather.cu).
//
//   block_scan_kernel   one warp per chunk of k-mer starts: bases packed to 2
//                       bits, eight l-mer positions a lane (the scan of
//                       warp_classify.cuh); run twice, first to count the
//                       candidates and then to write them back to back (a
//                       place for every k-mer would be three times the
//                       memory, and mapping it costs more than the scan);
//   bucket_sort_kernel  (bucket_sort.cuh) one thread block per sequence block:
//                       its candidates to shared memory by zone (MurmurHash3
//                       mod 256, the order's first key, then the top bits of
//                       the value: one or two candidates a zone), each zone
//                       sorted and freed of repeats by one thread;
//   block_pack_kernel   the blocks' lists back to back, with their taxa.
//
// This replaces eleven radix passes over all (minimizer, block) pairs: for 48
// Mbp of related genomes 2.9 ms of scan, passes and removal of repeats before,
// 0.8 ms now; a candidate is written once, read twice and moved once.
#pragma once

#include "bucket_sort.cuh"
#include "warp_classify.cuh"

namespace k2g {
namespace {

constexpr int kScanWarps = 4;
constexpr uint32_t kScanWords = (kChunk + 96) / 16;   // packed bases of a chunk

struct ScanShared {
  uint32_t be[kScanWords + 4], le[kScanWords + 4];    // le[3] holds the first word
  uint32_t inv[kScanWords / 2 + 4];                   // [2] is the first word
};

// Candidates of the chunks that hold k-mer starts (k - l = 4, canonical
// l-mers): the minimizer of every unambiguous k-mer unless the k-mer before
// it in the block has the same one.
// The chunk's go to cand + offs[chunk], or with WRITE false only their number
// to counts.
template <bool WRITE>
__global__ void __launch_bounds__(kScanWarps * 32)
block_scan_kernel(ScanView sv, const uint8_t *bases, const Chunk *chunks, uint64_t n_chunks,
                  uint64_t *cand, uint32_t *counts, const uint32_t *offs, uint32_t sample_below) {
  __shared__ ScanShared shared[kScanWarps];
  const uint64_t ci = blockIdx.x * (uint64_t)kScanWarps + (threadIdx.x >> 5);
  if (ci >= n_chunks) return;
  const Chunk ch = chunks[ci];
  if (ch.kind == kSubblockStart) return;
  ScanShared &s = shared[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int k = sv.k, l = sv.l;
  const uint32_t key_shift = 64u - 2u * (uint32_t)l;
  const uint64_t toggle_top = sv.toggle << key_shift;
  const uint64_t mask_top = (sv.spaced_mask ? sv.spaced_mask & sv.lmer_mask : sv.lmer_mask) << key_shift;
  // a chunk inside a block starts one k-mer early, to know the one before
  const uint32_t early = ch.kind == kContinues ? 1u : 0u;
  const uint32_t len = early + ch.n + (uint32_t)k - 1;
  const uint8_t *origin = bases + (ch.pos - early);
  const uint32_t lead = (uint32_t)((uintptr_t)origin & 15u), end = lead + len;
  origin -= lead;
  bool dirty = false;
#pragma unroll 1
  for (uint32_t c0 = 0; c0 < end; c0 += 32 * 16) {
    const uint32_t c = c0 + 16 * (uint32_t)lane;
    if (c < end) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(origin + c));
      uint32_t be, lo, bad = 0;
      if (wc_pack(v, be, lo)) bad = wc_bad_bases(v);
      if (c < lead) bad &= 0xFFFFu << (lead - c);
      if (c + 16 > end) bad &= 0xFFFFu >> (c + 16 - end);
      const uint32_t j = c >> 4;
      s.be[j] = be;
      s.le[j + 3] = lo;
      reinterpret_cast<uint16_t *>(s.inv + 2)[j] = (uint16_t)bad;
      dirty |= bad != 0;
    }
  }
  dirty = __any_sync(0xffffffffu, dirty);
  __syncwarp();
  const uint32_t n_items = (len - (uint32_t)(l - 1) + kWcPos - 1) / kWcPos;
  uint64_t *out = WRITE ? cand + offs[ci] : nullptr;
  uint32_t n_out = 0;
#pragma unroll 1
  for (uint32_t g0 = 0; g0 < n_items; g0 += 31) {
    if (g0 && g0 + 1 >= n_items) break;   // (only the repeated item is left)
    const uint32_t g = g0 + (uint32_t)lane;
    const bool in = g < n_items;
    const int p0 = l - 1 + kWcPos * (int)g, q0 = (int)lead + p0;
    uint64_t c[kWcPos];
    {
      const uint32_t at = in ? (uint32_t)(q0 - (l - 1)) : 0u, wi = at >> 4, sh = 2 * (at & 15u);
      const uint32_t b0 = s.be[wi], b1 = s.be[wi + 1], b2 = s.be[wi + 2], b3 = s.be[wi + 3];
      const uint32_t A = __funnelshift_l(b1, b0, sh), B = __funnelshift_l(b2, b1, sh), C = __funnelshift_l(b3, b2, sh);
      const uint32_t to = in ? (uint32_t)(q0 + kWcPos - 1) : 0u, we = to >> 4, ts = 30 - 2 * (to & 15u);
      const uint32_t e0 = s.le[we], e1 = s.le[we + 1], e2 = s.le[we + 2], e3 = s.le[we + 3];
      const uint32_t X = __funnelshift_l(e0, e1, ts), Y = __funnelshift_l(e1, e2, ts), Z = __funnelshift_l(e2, e3, ts);
#pragma unroll
      for (int j = 0; j < kWcPos; j++) {
        const uint32_t fh = j ? __funnelshift_l(B, A, 2 * j) : A, fl = j ? __funnelshift_l(C, B, 2 * j) : B;
        const int t = 2 * (kWcPos - 1 - j);
        const uint32_t rh = t ? __funnelshift_l(Y, Z, t) : Z, rl = t ? __funnelshift_l(X, Y, t) : Y;
        const uint64_t f = ((uint64_t)fh << 32) | fl, r = ((uint64_t)rh << 32) | rl;
        c[j] = ((f < r ? f : r) & mask_top) ^ toggle_top;
      }
    }
    // positions that end a k-mer, and those of the chunk's own k-mers
    const int n_pos = min(kWcPos, max(0, (int)len - p0));
    uint32_t emit = in ? (1u << n_pos) - 1u : 0u;
    if (g == 0) emit &= 0xFFu << (k - l);
    uint32_t amb = 0;
    if (dirty) {
      // bit i of v is base q0 - 34 + i
      const uint32_t b = in ? (uint32_t)(q0 - 34 + 64) : 64u;
      const uint32_t *iv = s.inv + (b >> 5);
      const uint64_t v = ((uint64_t)__funnelshift_r(iv[1], iv[2], b & 31) << 32) | __funnelshift_r(iv[0], iv[1], b & 31);
      const uint64_t lm = (1ull << l) - 1, am = (1ull << (k - 1)) - 1;
#pragma unroll
      for (int j = 0; j < kWcPos; j++) {
        if ((v >> (35 + j - l)) & lm) c[j] = ~0ull;
        if ((v >> (36 + j - k)) & am) amb |= 1u << j;
      }
    }
    uint64_t m[kWcPos];
    wc_window5(c, m);
    uint32_t start = 0;
    const uint64_t pm = __shfl_up_sync(0xffffffffu, m[7], 1);
    const uint32_t pa = __shfl_up_sync(0xffffffffu, amb, 1);
    const uint32_t prev_amb = ((amb << 1) | ((pa >> 7) & 1u)) & 0xFFu;
    start = m[0] != pm ? 1u : 0u;
#pragma unroll
    for (int j = 1; j < kWcPos; j++) start |= m[j] != m[j - 1] ? 1u << j : 0u;
    start |= prev_amb;                       // nothing to compare with
    if (g == 0) start |= 1u << (k - l);      // the first k-mer scanned
    start &= emit & ~amb;
    if (lane == 0 && g0) start = 0;          // the repeated item
    if (g == 0 && early) start &= ~(1u << (k - l));   // the k-mer before the chunk
    // (a subsampled table or a capacity estimate keeps some of them)
    if (sample_below || sv.min_hash) {
#pragma unroll
      for (int j = 0; j < kWcPos; j++)
        if (((start >> j) & 1u) && !keep(sv, sample_below, (m[j] ^ toggle_top) >> key_shift)) start &= ~(1u << j);
    }
    const uint32_t adds = __popc(start);
    if constexpr (!WRITE) {
      n_out += adds;   // (summed over the lanes at the end)
      continue;
    }
    uint32_t upto = adds;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, upto, d);
      if (lane >= d) upto += x;
    }
    uint64_t *at = out + n_out + upto - adds;
#pragma unroll
    for (int j = 0; j < kWcPos; j++)
      if ((start >> j) & 1u) *at++ = (m[j] ^ toggle_top) >> key_shift;
    n_out += __shfl_sync(0xffffffffu, upto, 31);
  }
  if constexpr (!WRITE) {
    n_out = __reduce_add_sync(0xffffffffu, n_out);
    if (lane == 0) counts[ci] = n_out;
  }
}

// Where every sequence block's candidates start: chunks lie block after block.
// (start[n_blocks] is set by the host.)
__global__ void block_start_kernel(const Chunk *chunks, uint64_t n_chunks, const uint32_t *offs, uint32_t *start) {
  const uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (c < n_chunks && (c == 0 || chunks[c].block != chunks[c - 1].block)) start[chunks[c].block] = offs[c];
}

// One warp per sequence block: its list to its place, and its taxon.
__global__ void block_pack_kernel(const uint32_t *start, const uint64_t *sorted, const uint32_t *n_distinct,
                                  const uint32_t *place, uint32_t n_blocks, const uint32_t *block_taxon,
                                  uint64_t *out_keys, uint32_t *out_taxa) {
  const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (b >= n_blocks) return;
  const uint64_t *x = sorted + start[b];
  const uint32_t n = n_distinct[b], o = place[b], t = block_taxon[b];
  for (uint32_t i = lane; i < n; i += 32) {
    out_keys[o + i] = x[i];
    out_taxa[o + i] = t;
  }
}

}  // namespace
}  // namespace k2g
