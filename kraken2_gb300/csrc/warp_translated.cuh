// Translated search, one warp per group of fragments (the nucleotide form is
// warp_classify.cuh, which explains the parts they share: entries, probe,
// replay and resolve).
//
// A frame of a mate is a sequence of its own.  The scan packs a mate once to
// 2 bits per base, then its codons to 4-bit residues: the codons that end at
// bases i = c (mod 3) are frame c, and the same codons complemented and read
// backwards are frame c + 3, so one pass over the codons of a class fills two
// arrays, the forward one with the first residue high and the other with the
// first codon low -- an l-mer of either is the top bits of a window that ends
// or begins at its residue.  The lanes take 8 residues each, through the six
// frames of a mate in order; borders (src/classify.cc:785-895) are entries.
//
// A group takes a fragment at a time where mates are longer than the packed
// window holds, frame after frame, a window of each at a time.
//
// What bounds it: integer instructions (2,310 a read of 150 bp, 56 % of the issue
// slots, the ALU pipe at 64 %) and their dependences, with 29 % of the warps
// resident; DRAM is idle.  A warp's lanes share what one thread walked residue by residue before, with
// its frames in local memory: 100,000 x 150 bp, 10 MB table 2.89 -> 0.35 ms.
#pragma once

#include "translated.cuh"
#include "warp_classify.cuh"

namespace k2g {

constexpr int kTxResidues = 512;                  // of a codon class in the packed window
constexpr int kTxBases = 3 * kTxResidues;
constexpr int kTxWords = kTxResidues / 8;
// Longest mate taken: two mates of six frames fit kEPosBits.
constexpr uint64_t kTxMaxLen = 1ull << 24;

struct TxShared : WcBase {
  static constexpr bool kFrames = true, kMany = false;
  uint32_t bases[kTxBases / 16 + 4];              // 2 bits per base, first base low
  uint32_t inv[kTxBases / 32 + 4];                // bit per base: not A/C/G/T
  // per class: residues of the codons (8 a word, the first one high; [4] is
  // the window's first word) and of their complements (the first one low,
  // [4] likewise), and the codons that hold an ambiguous base
  uint32_t fwd[3][kTxWords + 8], rev[3][kTxWords + 8];
  uint32_t bad[3][kTxWords / 4 + 4];              // [1] is the first word
  uint32_t mate_pos[kWcReads], room[kWcReads];    // position of the mate border; runs the region holds
  uint64_t mate_off[4];                           // start and length of each mate of the group
  uint32_t mate_len[4];
  __device__ __forceinline__ uint16_t *list() { return reinterpret_cast<uint16_t *>(fwd); }
};

// (as WcSharedMany, from kTxManyBases on: six frames give more runs a base)
struct TxSharedMany : TxShared {
  static constexpr bool kMany = true;
};
constexpr uint64_t kTxManyBases = 4096;

struct TxWarpArgs {
  ClassifyArgs a;
  const uint2 *span;
  uint32_t log_reads;     // 0 or 1
  uint64_t n_groups;
  uint64_t max_len;       // longest mate the caller says there is
};

// First codon start of the class of frame c (c mod 3), and its codons in a
// mate of len bases.
__device__ __forceinline__ uint32_t tx_first(uint32_t c) { return c == 2 ? 0u : c + 1; }
__device__ __forceinline__ uint32_t tx_codons(uint32_t c, uint32_t len) {
  const uint32_t j0 = tx_first(c);
  return len >= j0 + 3 ? (len - 3 - j0) / 3 + 1 : 0;
}

// Packs bases [b0, b1) of a mate (b1 - b0 <= kTxBases + 16) and returns the
// position of base b0 in s.bases.
template <class S>
__device__ __forceinline__ uint32_t tx_pack_bases(S &s, const ClassifyArgs &a, uint64_t off, uint32_t b0,
                                                  uint32_t b1, bool &bad_any) {
  const uint32_t lane = threadIdx.x & 31;
  const uint8_t *origin = a.bases + off + b0;
  const uint32_t lead = (uint32_t)((uintptr_t)origin & 15u);
  origin -= lead;
  const uint8_t *q = a.quals && a.cls.min_quality > 0 ? a.quals + off + b0 - lead : nullptr;
  const uint32_t end = lead + (b1 - b0);
#pragma unroll 1
  for (uint32_t c0 = 0; c0 < end; c0 += 32 * 16) {
    const uint32_t c = c0 + 16 * lane;
    if (c < end) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(origin + c));
      uint32_t be, le;
      uint32_t bad = 0;
      if (wc_pack(v, be, le)) bad = wc_bad_bases(v);
      if (q) {
        const int thr = 33 + a.cls.min_quality;
        bad |= wc_low_quality(__ldg(reinterpret_cast<const uint4 *>(q + c)),
                              ((uint32_t)min(thr, 127) & 0xFFu) * 0x01010101u, thr > 127);
      }
      s.bases[c >> 4] = ~le;
      reinterpret_cast<uint16_t *>(s.inv)[c >> 4] = (uint16_t)bad;
      bad_any |= bad != 0;
    }
  }
  return lead;
}

// Residues [u0, u1) of class c (u0 a multiple of 8) from the packed bases;
// `at` is where the codon of u0 starts there.
template <class S>
__device__ __forceinline__ void tx_pack_residues(S &s, const uint8_t *lut, uint32_t c, uint32_t word0,
                                                 uint32_t words, uint32_t at) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t w = word0 + lane; w < words; w += 32) {
    const uint32_t b = at + 24 * w, wi = b >> 4, sh = 2 * (b & 15u);
    const uint32_t x0 = s.bases[wi], x1 = s.bases[wi + 1], x2 = s.bases[wi + 2];
    const uint64_t v = ((uint64_t)__funnelshift_r(x1, x2, sh) << 32) | __funnelshift_r(x0, x1, sh);
    const uint32_t i0 = s.inv[b >> 5], i1 = s.inv[(b >> 5) + 1];
    const uint32_t iv = __funnelshift_r(i0, i1, b & 31);
    uint32_t f = 0, r = 0, bad = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t code = lut[(uint32_t)(v >> (6 * i)) & 63u];
      f |= (code & 15u) << (28 - 4 * i);
      r |= (code >> 4) << (4 * i);
      bad |= ((iv >> (3 * i)) & 7u) ? 1u << i : 0u;
    }
    s.fwd[c][w + 4] = f;
    s.rev[c][w + 4] = r;
    reinterpret_cast<uint8_t *>(&s.bad[c][1])[w] = (uint8_t)bad;
  }
}

template <bool WIDE, bool HITS, class Shared>
__global__ void __launch_bounds__(kWcWarps * 32, 10) warp_translated_kernel(TxWarpArgs wa) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint8_t lut[64];   // codon (first base low) -> residue, and of its complement << 4
  {
    // A 0, C 1, G 2, T 3 here; A 0, G 1, C 2, T 3 in codon_aa, first base high
    const uint32_t i = threadIdx.x & 63u;
    auto g = [](uint32_t b) { return b == 1 ? 2u : b == 2 ? 1u : b; };
    const uint32_t b0 = i & 3, b1 = (i >> 2) & 3, b2 = i >> 4;
    const uint32_t f = tx::aa_code((uint8_t)tx::codon_aa((g(b0) << 4) | (g(b1) << 2) | g(b2)));
    const uint32_t r = tx::aa_code((uint8_t)tx::codon_aa((g(3 - b2) << 4) | (g(3 - b1) << 2) | g(3 - b0)));
    lut[i] = (uint8_t)(f | (r << 4));
  }
  __syncthreads();
  const ClassifyArgs &a = wa.a;
  const uint64_t group = blockIdx.x * (uint64_t)kWcWarps + (threadIdx.x >> 5);
  if (group >= wa.n_groups) return;
  Shared &s = reinterpret_cast<Shared *>(smem)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u, le = lt | (1u << lane);
  const int k = a.scan.k, l = a.scan.l;
  const uint64_t f0 = group << wa.log_reads;
  const int nr = (int)min((uint64_t)1 << wa.log_reads, a.n_frags - f0);
  const int per = a.cls.paired ? 2 : 1, nm = nr * per, ns = 6 * nm;
  const uint32_t key_shift = 64u - 4u * (uint32_t)l;
  Wc<WIDE, HITS, Shared> w{a, s, lane, lt, f0, kWcLogSlots - wa.log_reads, 0u, key_shift,
                             a.scan.toggle << key_shift};
  const uint64_t mask_top = (a.scan.spaced_mask ? a.scan.spaced_mask & a.scan.lmer_mask : a.scan.lmer_mask)
                            << key_shift;

  // ---- mates, then their frames: lane i holds frame i % 6 of mate i / 6
  const uint64_t o = lane <= nm ? a.seq_off[f0 * per + lane] : 0;
  const uint64_t o_next = __shfl_down_sync(0xffffffffu, o, 1);
  const uint64_t full_len = lane < nm ? o_next - o : 0;
  // (a mate longer than max_seq_len says: its fragment is refused)
  const uint32_t too_long = __ballot_sync(0xffffffffu, full_len > wa.max_len);
  auto refused = [&](int r) { return (too_long >> (r * per)) & (per == 2 ? 3u : 1u); };
  if (lane < nm) {
    s.mate_off[lane] = o;
    s.mate_len[lane] = refused(lane / per) ? 0u : (uint32_t)full_len;
  }
  if (lane < nm && lane % per == 0) {
    const int r = lane / per;
    s.run_base[r] = o + 2 * (f0 + r + a.frag_off);
    s.hits[r] = s.n_runs[r] = s.n_taxa[r] = 0;
  }
  if (lane == 0) s.over = s.stopped = 0;
#pragma unroll
  for (int i = 0; i < kWcSlots; i += 128) {
    *reinterpret_cast<uint4 *>(&s.mkey[i + 4 * lane]) = make_uint4(0, 0, 0, 0);
    *reinterpret_cast<uint4 *>(&s.mcnt[i + 4 * lane]) = make_uint4(0, 0, 0, 0);
  }
  __syncwarp();
  const int rm = lane / 6, frame = lane - 6 * rm, fr = rm / per;   // mate of the group, its frame, fragment
  const bool mine = lane < ns && !refused(fr);
  const uint32_t cls = (uint32_t)(frame >= 3 ? frame - 3 : frame);
  const uint32_t n_res = mine ? tx_codons(cls, s.mate_len[rm]) : 0;
  const uint32_t kmers = n_res >= (uint32_t)k ? n_res - (uint32_t)k + 1 : 0;
  const int in_frag = lane - 6 * per * fr;                         // frames of the fragment before this one
  const bool opens = in_frag == 0;
  // tokens of the fragment before this frame: k-mers, and a border after
  // each earlier frame
  uint32_t upto = mine ? kmers + 1 : 0;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, upto, d);
    if (lane >= d && in_frag >= d) upto += x;
  }
  const uint32_t tok_base = upto - (mine ? kmers + 1 : 0);
  if (mine && in_frag == 6 * per - 1) s.tokens[fr] = upto - 1;     // (no border after the last frame)
  if (mine && per == 2 && in_frag == 6) s.mate_pos[fr] = tok_base - 1;
  if (mine && per == 1 && opens) s.mate_pos[fr] = 0xFFFFFFFFu;
  if (mine && opens)
    s.room[fr] = s.mate_len[rm] + (per == 2 ? s.mate_len[rm + 1] : 0u) + 2;
  const uint32_t items = kmers ? (n_res - (uint32_t)(l - 1) + kWcPos - 1) / kWcPos : (mine && !opens ? 1u : 0u);
  uint32_t incl = items;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += x;
  }
  const uint32_t first_item = items ? incl - items : 0xFFFFFFFFu;
  const uint32_t n_items = __shfl_sync(0xffffffffu, incl, 31);
  const uint32_t busy = __ballot_sync(0xffffffffu, items != 0);
  // (at most 12 frames: two fragments of one mate, or one pair)
  if (items)
    s.seq[__popc(busy & lt)] = make_uint4((uint32_t)lane, n_res, first_item,
                                          (uint32_t)fr | (opens ? 0u : 8u) | (tok_base << 4));
  __syncwarp();

  // ---- scan
  uint32_t g0 = 0;
  int cur = -1;                       // mate packed whole, or -1
  bool own0 = true, dirty = false;
  int ne = 0;
  bool done = n_items == 0;
  while (!done) {
    bool full = false;
#pragma unroll 1
    while (!done && !full) {
      const uint32_t g = g0 + (uint32_t)lane;
      const uint32_t rel = first_item - g0;
      const uint32_t starts = __reduce_or_sync(0xffffffffu, rel < 32 ? 1u << rel : 0u);
      const uint32_t before = __popc(__ballot_sync(0xffffffffu, first_item < g0));
      const uint32_t sq = before + __popc(starts & le) - 1;
      const uint4 seq = s.seq[sq];
      const bool head = (starts >> lane) & 1u;
      const uint32_t q_rm = seq.x / 6, q_frame = seq.x - 6 * q_rm;
      const bool back = q_frame >= 3;
      const uint32_t q_cls = back ? q_frame - 3 : q_frame;
      const int n = (int)seq.y;
      const int t0 = l - 1 + kWcPos * (int)(g - seq.z);   // residue of the lane's first position
      // the window: the whole mate, or a stretch of one frame's codons
      const int lead_rm = (int)__shfl_sync(0xffffffffu, q_rm, 0);
      const uint32_t mate_len = s.mate_len[lead_rm];
      bool in = g < n_items && (int)q_rm == lead_rm;
      int u_lo = 0;                   // first codon of the class in the window
      if (mate_len <= (uint32_t)kTxBases) {
        if (cur != lead_rm) {
          __syncwarp();
          bool bad = false;
          const uint32_t at = tx_pack_bases(s, a, s.mate_off[lead_rm], 0, mate_len, bad);
          dirty |= __any_sync(0xffffffffu, bad);
          __syncwarp();
          for (uint32_t c = 0; c < 3; c++)
            tx_pack_residues(s, lut, c, 0, (tx_codons(c, mate_len) + 7) / 8, at + tx_first(c));
          __syncwarp();
          cur = lead_rm;
        }
      } else {
        const uint32_t lead_sq = __shfl_sync(0xffffffffu, sq, 0), c = __shfl_sync(0xffffffffu, q_cls, 0);
        const bool lead_back = __shfl_sync(0xffffffffu, back ? 1u : 0u, 0);
        const int lead_n = __shfl_sync(0xffffffffu, n, 0), lead_t = __shfl_sync(0xffffffffu, t0, 0) - (k - 1);
        // codons the pass can reach from its first residue on, a whole window of them
        if (lead_back) u_lo = max(0, ((min(lead_n - 1, lead_n - 1 - lead_t) >> 3) - (kTxWords - 1)) * 8);
        else u_lo = max(0, lead_t) & ~7;
        const int u_hi = min(lead_n, u_lo + kTxResidues);
        __syncwarp();
        bool bad = false;
        const uint32_t b0 = tx_first(c) + 3 * (uint32_t)u_lo;
        const uint32_t at = tx_pack_bases(s, a, s.mate_off[lead_rm], b0, tx_first(c) + 3 * (uint32_t)u_hi, bad);
        dirty |= __any_sync(0xffffffffu, bad);
        __syncwarp();
        tx_pack_residues(s, lut, c, 0, (uint32_t)(u_hi - u_lo + 7) / 8, at);
        __syncwarp();
        cur = -1;
        in = in && sq == lead_sq &&
             (lead_back ? max(0, n - 1 - (t0 + kWcPos - 1)) >= u_lo : t0 + kWcPos <= u_lo + kTxResidues || t0 + kWcPos > n);
        in = in && (lead_back || t0 - (l - 1) < u_lo + kTxResidues - 32);
      }
      const int n_in = __popc(__ballot_sync(0xffffffffu, in));
      const bool own = in && (lane > 0 || own0);
      // candidates: windows of 4-bit residues, the l-mer in the top bits
      uint64_t c[kWcPos];
      {
        // forward: from residue t0 - (l - 1) on; backward: codons n - 1 - t0 + l - 1 and down
        const int r0 = in ? (back ? n - 1 - t0 + l - 1 - u_lo : t0 - (l - 1) - u_lo) : 0;
        const int wi = r0 >> 3;
        const uint32_t sh = back ? 28u - 4u * (uint32_t)(r0 & 7) : 4u * (uint32_t)(r0 & 7);
        const uint32_t *x = (back ? s.rev[q_cls] : s.fwd[q_cls]) + 4 + wi;
        const int d = back ? -1 : 1;
        const uint32_t x0 = x[0], x1 = x[d], x2 = x[2 * d], x3 = x[3 * d];
        const uint32_t A = __funnelshift_l(x1, x0, sh), B = __funnelshift_l(x2, x1, sh), C = __funnelshift_l(x3, x2, sh);
#pragma unroll
        for (int j = 0; j < kWcPos; j++) {
          const uint32_t h = j ? __funnelshift_l(B, A, 4 * j) : A, lw = j ? __funnelshift_l(C, B, 4 * j) : B;
          c[j] = ((((uint64_t)h << 32) | lw) & mask_top) ^ w.toggle_top;
        }
      }
      const int n_pos = min(kWcPos, max(0, n - t0));
      uint32_t emit = in ? (1u << n_pos) - 1u : 0u;
      if (head) emit &= 0xFFu << (k - l);
      uint32_t amb = 0;
      if (dirty) {
        // bit i of v: residue t0 - (k - 2) + i; k + 6 bits
        const int b = in ? (back ? n - 1 - t0 - 7 - u_lo : t0 - (k - 2) - u_lo) + 32 : 32;
        const uint32_t *bw = s.bad[q_cls] + (b >> 5);
        uint32_t v = __funnelshift_r(bw[0], bw[1], b & 31);
        if (back) v = __brev(v) >> (32 - (k + 6));
        const uint32_t lm = ((1u << l) - 1) << (k - 1 - l), am = (1u << (k - 1)) - 1;
#pragma unroll
        for (int j = 0; j < kWcPos; j++) {
          if (v & (lm << j)) c[j] = ~0ull;
          if (v & (am << j)) amb |= 1u << j;
        }
      }
      // window minima: four candidates ending at each position
      uint64_t m[kWcPos];
      {
        const uint64_t d5 = min64(c[5], c[6]), d6 = min64(c[6], c[7]), t5 = min64(d5, c[7]);
        const uint64_t p5 = __shfl_up_sync(0xffffffffu, t5, 1), p6 = __shfl_up_sync(0xffffffffu, d6, 1),
                       p7 = __shfl_up_sync(0xffffffffu, c[7], 1);
        const uint64_t d0 = min64(c[0], c[1]), d1 = min64(c[1], c[2]), d2 = min64(c[2], c[3]),
                       d3 = min64(c[3], c[4]), d4 = min64(c[4], c[5]);
        m[0] = min64(p5, c[0]);
        m[1] = min64(p6, d0);
        m[2] = min64(p7, min64(d0, c[2]));
        m[3] = min64(d0, d2);
        m[4] = min64(d1, d3);
        m[5] = min64(d2, d4);
        m[6] = min64(d3, d5);
        m[7] = min64(d4, d6);
      }
      uint32_t cont = 0;
      uint64_t next_min;
      uint32_t next_seq;
      uint32_t start = w.starts(m, emit, amb, head, !own0, dirty, sq, n_in, (uint32_t)(k - l), cont, next_min, next_seq);
      if (!own) start = 0;
      const uint32_t tok0 = (seq.w >> 4) + (uint32_t)(t0 - (k - 1));
      full = !w.add(ne, m, start, amb, cont, own && head && (seq.w & 8u), seq.w, tok0, dirty);
      if (!full) {
        w.seen_min = next_min;
        w.seen_seq = next_seq;
        done = g0 + (uint32_t)n_in >= n_items;
        own0 = n_in < 32 && ((starts >> n_in) & 1u);
        g0 += (uint32_t)n_in - (own0 ? 0u : 1u);
      }
    }
    __syncwarp();
    w.probe(ne);
    cur = -1;   // the list of the probe lay in the packed words
    w.replay(ne, dirty, done);
    ne = 0;
  }

  // ---- calls
  const bool out = lane < nr && !refused(lane);
  uint64_t total = 0;
  if (out) {
    // (the reference leaves two frame borders uncounted, four for pairs)
    total = s.tokens[lane];
    total -= a.cls.paired ? 5u : 2u;
    s.n_runs[lane] = min(s.n_runs[lane], s.room[lane]);
  }
  __syncwarp();
  w.finish(wa.span, out, total);
  if (lane < nr && !out) {
    atomicOr(a.status, STATUS_RUNS_OVERFLOW);
    a.call[f0 + lane] = 0;
    if (a.hitlist_len) a.hitlist_len[f0 + lane] = 0;
  }
}

}  // namespace k2g
