// k2g_classify_host: classification of reads held in host memory.
//
// The input is cut into chunks of about a twelfth of the call.  Each chunk has
// one of three or four slots, with a stream for its copies in and its classification
// and one for what follows, so its copies overlap the kernels of the others,
// and the host waits for a chunk only when the others are under way.
// The second stream has the higher priority: its short kernels would wait
// behind the classification of the next two chunks, and the slot with them
// (2M x 150 bp: 3.6 ms, 2.9 with it).  Hit-list runs are
// compacted on the device (exclusive scan of the per-fragment run counts,
// then a gather) so only the used runs cross back to the host.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "k2g_internal.h"

namespace k2g {

constexpr int kScanBlock = 1024;

// Block-level exclusive scan of n counts; block totals to sums[].
__global__ void scan_blocks_kernel(const uint32_t *in, uint64_t *out, uint64_t *sums, uint64_t n) {
  __shared__ uint64_t warp_tot[32];
  uint64_t i = blockIdx.x * (uint64_t)kScanBlock + threadIdx.x;
  uint64_t v = i < n ? in[i] : 0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint64_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[w] = x;
  __syncthreads();
  if (w == 0) {
    uint64_t t = warp_tot[lane];
    for (int o = 1; o < 32; o <<= 1) {
      uint64_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    warp_tot[lane] = t;
  }
  __syncthreads();
  uint64_t excl = x - v + (w ? warp_tot[w - 1] : 0);
  if (i < n) out[i] = excl;
  if (threadIdx.x == kScanBlock - 1) sums[blockIdx.x] = excl + v;
}

// Exclusive scan of up to kScanBlock*kScanBlock block sums in one block.
__global__ void scan_sums_kernel(uint64_t *sums, uint64_t nb, uint64_t *total) {
  __shared__ uint64_t buf[kScanBlock];
  uint64_t carry = 0;
  for (uint64_t base = 0; base < nb; base += kScanBlock) {
    uint64_t i = base + threadIdx.x;
    uint64_t v = i < nb ? sums[i] : 0;
    buf[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < kScanBlock; o <<= 1) {
      uint64_t y = threadIdx.x >= (unsigned)o ? buf[threadIdx.x - o] : 0;
      __syncthreads();
      buf[threadIdx.x] += y;
      __syncthreads();
    }
    uint64_t incl = buf[threadIdx.x];
    if (i < nb) sums[i] = carry + incl - v;
    __syncthreads();
    carry += buf[kScanBlock - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// Adds block offsets and gathers each fragment's runs into the dense array.  A
// warp takes `each` fragments: a thread copies a short list, the warp the long
// ones one after another.  (A thread for every list took 0.72 ms for 120k
// fragments of up to 50 kb.  4 fragments a warp where most bases are in long
// ones, not 32, which are six long lists: that host call 2.38 -> 2.32 ms.)
constexpr uint32_t kShortList = 16;

__global__ void gather_runs_kernel(const uint64_t *sparse, const uint64_t *seq_off, int per,
                                   const uint32_t *len, const uint64_t *excl, const uint64_t *sums,
                                   uint64_t n, uint32_t each, uint64_t *dense) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t i = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * each + lane;
  const bool in = i < n && lane < each;
  const uint32_t m = in ? len[i] : 0;
  const uint64_t to = in ? excl[i] + sums[i / kScanBlock] : 0, from = in ? seq_off[i * per] + 2 * i : 0;
  if (m <= kShortList)
    for (uint32_t r = 0; r < m; r++) dense[to + r] = sparse[from + r];
  for (uint32_t todo = __ballot_sync(0xffffffffu, m > kShortList); todo; todo &= todo - 1) {
    const int who = __ffs(todo) - 1;
    const uint32_t k = __shfl_sync(0xffffffffu, m, who);
    const uint64_t o = __shfl_sync(0xffffffffu, to, who), src = __shfl_sync(0xffffffffu, from, who);
#pragma unroll 4
    for (uint32_t r = lane; r < k; r += 32) dense[o + r] = sparse[src + r];
  }
}

__global__ void rebase_kernel(uint64_t *off, uint64_t n, uint64_t base) {
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i < n) off[i] -= base;
}

__global__ void add_block_base_kernel(uint64_t *out, const uint64_t *sums, uint64_t n) {
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] += sums[i / kScanBlock];
}

// Exclusive scan whose value i is d_out[i] + d_sums[i / 1024].
k2g_status block_scan_u32(const uint32_t *d_in, uint64_t n, uint64_t *d_out, uint64_t *d_sums, uint64_t *d_total,
                          cudaStream_t st) {
  if (!n) return K2G_OK;
  uint64_t nb = (n + kScanBlock - 1) / kScanBlock;
  scan_blocks_kernel<<<(unsigned)nb, kScanBlock, 0, st>>>(d_in, d_out, d_sums, n);
  scan_sums_kernel<<<1, kScanBlock, 0, st>>>(d_sums, nb, d_total);
  note_launches(2);
  K2G_CUDA_TRY(cudaGetLastError());
  return K2G_OK;
}
static_assert(kScanBlock == 1024, "users of block_scan_u32 add d_sums[i >> 10]");

k2g_status exclusive_scan_u32(const uint32_t *d_in, uint64_t n, uint64_t *d_out, uint64_t *d_sums,
                              uint64_t *d_total, cudaStream_t st) {
  if (!n) return K2G_OK;
  const k2g_status s = block_scan_u32(d_in, n, d_out, d_sums, d_total, st);
  if (s != K2G_OK) return s;
  add_block_base_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d_out, d_sums, n);
  note_launches();
  K2G_CUDA_TRY(cudaGetLastError());
  return K2G_OK;
}

k2g_status compact_runs(const uint64_t *d_sparse, const uint64_t *d_seq_off, int per,
                        const uint32_t *d_len, uint64_t n, uint64_t *d_excl, uint64_t *d_sums,
                        uint64_t *d_total, uint64_t *d_dense, bool long_lists, cudaStream_t st) {
  uint64_t nb = (n + kScanBlock - 1) / kScanBlock;
  scan_blocks_kernel<<<(unsigned)nb, kScanBlock, 0, st>>>(d_len, d_excl, d_sums, n);
  scan_sums_kernel<<<1, kScanBlock, 0, st>>>(d_sums, nb, d_total);
  note_launches(3);
  const uint32_t each = long_lists ? 4 : 32;
  gather_runs_kernel<<<(unsigned)((n + 8 * each - 1) / (8 * each)), 256, 0, st>>>(d_sparse, d_seq_off, per, d_len, d_excl,
                                                                                d_sums, n, each, d_dense);
  K2G_CUDA_TRY(cudaGetLastError());
  return K2G_OK;
}

}  // namespace k2g

using namespace k2g;

namespace {

// Device buffers of one chunk in flight.  They are kept per device across
// calls (grown when a call needs more), so a call allocates nothing once
// the sizes have been seen.
struct Slot {
  cudaStream_t st = nullptr, out = nullptr;   // in and classified; counted, compacted and out
  cudaEvent_t classified = nullptr;
  cudaEvent_t done = nullptr;      // compacted: the input buffers are free, the number of runs known
  cudaEvent_t left = nullptr;      // copied out: all are
  char *bases = nullptr, *quals = nullptr;
  uint64_t *off = nullptr;
  uint32_t *call = nullptr, *hg = nullptr, *hlen = nullptr;
  uint64_t *sparse = nullptr, *dense = nullptr, *excl = nullptr, *sums = nullptr;
  uint64_t *total = nullptr;       // device: runs of the chunk, then its status word
  uint64_t *h_total = nullptr;     // the same, pinned
  // add_kmer events (only with counters)
  uint64_t *hit_keys = nullptr, *hit_order = nullptr, *hits_used = nullptr;
  uint32_t *hit_taxa = nullptr, *blocks = nullptr;
  uint64_t cap_bases = 0, cap_frags = 0, cap_quals = 0, cap_hits = 0;
  // the chunk under way
  bool copied = false;             // results on their way out
  uint64_t f0 = 0, nf = 0, max_len = 0;
  k2g_reads rd{};
  k2g_results rs{};
};
constexpr int kSlots = 4;

struct HostCache {
  std::mutex mu;
  Slot slots[kSlots];
  unsigned long long *taxon_reads = nullptr;
  uint64_t taxon_cap = 0;
};
HostCache g_host[64];

template <class T>
cudaError_t regrow(T *&p, uint64_t n) {
  if (p) cudaFree(p);
  p = nullptr;
  return device_alloc(&p, std::max<uint64_t>(n, 1) * sizeof(T));
}

// Makes the slot hold chunks of up to fb fragments / bb bases.
cudaError_t fit_slot(Slot &s, uint64_t bb, uint64_t fb, int per, bool quals, uint64_t hits) {
  cudaError_t e;
#define TRY(x) if ((e = (x)) != cudaSuccess) return e
  if (!s.hits_used) {   // (the last of them: after a failure the rest is made)
    int low = 0, high = 0;
    TRY(cudaDeviceGetStreamPriorityRange(&low, &high));
    for (cudaEvent_t *e1 : {&s.classified, &s.done, &s.left})
      if (!*e1) TRY(cudaEventCreateWithFlags(e1, cudaEventDisableTiming));
    if (!s.out) TRY(cudaStreamCreateWithPriority(&s.out, cudaStreamNonBlocking, high));
    if (!s.st) TRY(cudaStreamCreateWithFlags(&s.st, cudaStreamNonBlocking));
    if (!s.h_total) TRY(cudaHostAlloc(&s.h_total, 16, cudaHostAllocDefault));
    if (!s.total) TRY(cudaMalloc(&s.total, 16));
    TRY(cudaMalloc(&s.hits_used, 8));
  }
  if (bb > s.cap_bases || fb > s.cap_frags) {
    bb = std::max(bb, s.cap_bases);
    fb = std::max(fb, s.cap_frags);
    const uint64_t sparse_cap = bb + 2 * fb + 8;
    // (until all of them are there, the slot holds nothing: a call that runs
    // out of memory here leaves it to the next to start over)
    s.cap_bases = s.cap_frags = s.cap_quals = s.cap_hits = 0;
    TRY(regrow(s.bases, bb + 16));
    TRY(regrow(s.off, fb * 2 + 1));
    TRY(regrow(s.call, fb));
    TRY(regrow(s.hg, fb));
    TRY(regrow(s.hlen, fb));
    TRY(regrow(s.sparse, sparse_cap));
    TRY(regrow(s.dense, sparse_cap));
    TRY(regrow(s.excl, fb));
    TRY(regrow(s.sums, (fb + kScanBlock - 1) / kScanBlock + 1));
    TRY(regrow(s.blocks, fb));
    s.cap_bases = bb;
    s.cap_frags = fb;
  }
  if (quals && s.cap_quals < s.cap_bases) {
    s.cap_quals = 0;
    TRY(regrow(s.quals, s.cap_bases + 16));
    s.cap_quals = s.cap_bases;
  }
  if (hits > s.cap_hits) {
    s.cap_hits = 0;
    TRY(regrow(s.hit_keys, hits));
    TRY(regrow(s.hit_taxa, hits));
    TRY(regrow(s.hit_order, hits));
    s.cap_hits = hits;
  }
#undef TRY
  (void)per;
  return cudaSuccess;
}

// Gives a slot's buffers back.
void empty_slot(Slot &s) {
  auto drop = [](auto *&p) {
    if (p) cudaFree(p);
    p = nullptr;
  };
  drop(s.bases); drop(s.quals); drop(s.off); drop(s.call); drop(s.hg); drop(s.hlen); drop(s.sparse); drop(s.dense);
  drop(s.excl); drop(s.sums); drop(s.blocks); drop(s.hit_keys); drop(s.hit_taxa); drop(s.hit_order);
  s.cap_bases = s.cap_frags = s.cap_quals = s.cap_hits = 0;
}

// Largest g in [f, n] with seq_off[g * per] - seq_off[f * per] <= max_bases
// (offsets are non-decreasing).
uint64_t cut_by_bases(const uint64_t *seq_off, int per, uint64_t f, uint64_t n,
                      uint64_t max_bases) {
  const uint64_t b0 = seq_off[f * per];
  uint64_t lo = f, hi = n;
  while (lo < hi) {
    const uint64_t mid = lo + (hi - lo + 1) / 2;
    if (seq_off[mid * per] - b0 <= max_bases) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

}  // namespace

// Host-buffer classification over chunks.  With counters, chunks end at
// reader-block boundaries (frag_block) and each chunk's add_kmer events are
// folded in after it is classified.
static k2g_status host_classify(const k2g_db *db, const char *bases, const char *quals,
                                const uint64_t *seq_off, uint64_t n_frags,
                                const uint32_t *frag_block, k2g_counters *counters,
                                const k2g_classify_params *params, uint32_t *call,
                                uint32_t *hit_groups, uint32_t *hitlist_len, uint64_t *runs,
                                uint64_t *n_runs, uint64_t *taxon_reads) {
  if (!db || !bases || !seq_off || !params || !call) return fail(K2G_ERR_ARG, "null argument");
  if (counters && !frag_block) return fail(K2G_ERR_ARG, "counters need frag_block");
  if (runs && !n_runs) return fail(K2G_ERR_ARG, "runs given without n_runs capacity");
  const uint64_t runs_cap = runs ? *n_runs : 0;
  if (n_runs) *n_runs = 0;
  if (!n_frags) return K2G_OK;
  K2G_CUDA_TRY(cudaSetDevice(db->device));
  const int per = params->paired ? 2 : 1;

  // Chunk plan: about a twelfth of the call (a quarter with hit events, whose
  // counting makes the host wait), 128 MB (64 MB with hit events) of bases or
  // 2M fragments at most, and 16 MB at least, 20 where most are long -- below
  // that a chunk's launches and copies outweigh what overlaps.  2M x 150 bp:
  // 6 chunks 3.01 ms, 8 2.96, 12 2.89, 16 2.90; with hit events 1M x 150 bp: 3
  // to 5 chunks 4.9 to 5.0, 8 5.3.  Long ones (mean 5 kb) among 150 bp, four
  // slots, chunks of 16, 20 and 24 MB at least: 20k and 100k 2.39, 2.30, 2.28
  // ms; 20k and 1k 2.07, 2.03, 1.99; 10k and 50k of 100 bp 1.43, 1.38, 1.42; 8k
  // and 1k 1.06, 1.05, 1.06; 5k and 500k 2.13, 2.11, 2.12; 3k and 20k 0.74,
  // 0.73, 0.73; 20k and 300k of 251 bp 3.24, 3.24, 3.29: 20 is never behind 16.
  const uint64_t all_bases = seq_off[n_frags * per] - seq_off[0];
  const uint64_t least = (long_batch(all_bases, n_frags) ? 20ull : 16ull) << 20;
  const uint64_t max_bases = std::min<uint64_t>(counters ? 64ull << 20 : 128ull << 20,
                                                std::max<uint64_t>(least, all_bases / (counters ? 4 : 12) + 1)),
                 max_frags = 2ull << 20;
  std::vector<uint64_t> cuts{0};
  while (cuts.back() < n_frags) {
    const uint64_t f = cuts.back();
    uint64_t g = std::min(cut_by_bases(seq_off, per, f, n_frags, max_bases), f + max_frags);
    if (g == f) g = f + 1;   // a single oversized fragment forms its own chunk
    if (counters && g < n_frags) {
      // end the chunk at the last block boundary; a block larger than a
      // chunk forms its own chunk
      uint64_t h = g;
      while (h > f && frag_block[h] == frag_block[h - 1]) h--;
      if (h == f) {
        h = g;
        while (h < n_frags && frag_block[h] == frag_block[h - 1]) h++;
      }
      g = h;
    }
    cuts.push_back(g);
  }
  uint64_t chunk_frags = 0, chunk_bases = 0;
  for (size_t c = 0; c + 1 < cuts.size(); c++) {
    chunk_frags = std::max(chunk_frags, cuts[c + 1] - cuts[c]);
    chunk_bases = std::max(chunk_bases, seq_off[cuts[c + 1] * per] - seq_off[cuts[c] * per]);
  }
  // at most one lookup per k-mer; translated, six frames of a third of the
  // bases each (two lookups per base) plus the frames' ends
  const uint64_t hits_cap = !counters ? 0
                            : db->opts.dna_db ? chunk_bases + 4 * chunk_frags + 16
                                              : 2 * chunk_bases + 32 * chunk_frags + 16;

  HostCache &hc = g_host[db->device & 63];
  std::lock_guard<std::mutex> lock(hc.mu);
  Slot *slots = hc.slots;
  const size_t n_chunks = cuts.size() - 1;
  // Three slots, four for long fragments, whose merge waits behind the next
  // chunks' classification (120k mixed ones: 2.54 -> 2.38 ms; short ones the
  // same, with hit events 4.52 -> 4.59).  A third as large as one huge sequence
  // would be memory for nothing.
  size_t n_slots = chunk_bases > (256ull << 20) ? 2 : long_batch(all_bases, n_frags) && !counters ? kSlots : 3;
  int used = (int)std::min(n_chunks, n_slots);
  auto fit = [&]() {
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < used && e == cudaSuccess; i++)
      e = fit_slot(slots[i], chunk_bases, chunk_frags, per, quals != nullptr, hits_cap);
    return e;
  };
  cudaError_t fitted = fit();
  bool more = used > 2;
  for (int i = 2; i < kSlots; i++) more = more || slots[i].bases || slots[i].sparse;
  if (fitted == cudaErrorMemoryAllocation && more) {
    // two slots do, where the others' memory is needed or not there
    (void)cudaGetLastError();
    for (int i = 2; i < kSlots; i++) empty_slot(slots[i]);
    n_slots = 2;
    used = (int)std::min(n_chunks, n_slots);
    fitted = fit();
  }
  K2G_CUDA_TRY(fitted);
  unsigned long long *d_taxon_reads = nullptr;
  if (taxon_reads) {
    if (hc.taxon_cap < db->node_count) {
      hc.taxon_cap = 0;
      K2G_CUDA_TRY(regrow(hc.taxon_reads, db->node_count));
      hc.taxon_cap = db->node_count;
    }
    d_taxon_reads = hc.taxon_reads;
    // zeroed before any stream's first chunk
    K2G_CUDA_TRY(cudaMemsetAsync(d_taxon_reads, 0, db->node_count * 8, slots[0].st));
    K2G_CUDA_TRY(cudaEventRecord(slots[0].done, slots[0].st));
    for (int i = 1; i < used; i++) K2G_CUDA_TRY(cudaStreamWaitEvent(slots[i].st, slots[0].done, 0));
  }

  // Stage 1 of chunk c: copy in.  (Blocks first: they often lie in pageable
  // memory, where the call returns only when the stream has got to the copy.)
  auto copy_in = [&](size_t c) -> k2g_status {
    Slot &s = slots[c % n_slots];
    const uint64_t f0 = cuts[c], nf = cuts[c + 1] - f0;
    const uint64_t b0 = seq_off[f0 * per], nb = seq_off[(f0 + nf) * per] - b0;
    s.f0 = f0;
    s.nf = nf;
    K2G_CUDA_TRY(cudaStreamWaitEvent(s.st, s.done, 0));
    if (counters) {
      K2G_CUDA_TRY(cudaMemcpyAsync(s.blocks, frag_block + f0, nf * 4, cudaMemcpyHostToDevice, s.st));
      K2G_CUDA_TRY(cudaMemsetAsync(s.hits_used, 0, 8, s.st));
    }
    K2G_CUDA_TRY(cudaMemcpyAsync(s.off, seq_off + f0 * per, (nf * per + 1) * 8,
                                 cudaMemcpyHostToDevice, s.st));
    K2G_CUDA_TRY(cudaMemcpyAsync(s.bases, bases + b0, nb, cudaMemcpyHostToDevice, s.st));
    if (quals) K2G_CUDA_TRY(cudaMemcpyAsync(s.quals, quals + b0, nb, cudaMemcpyHostToDevice, s.st));
    K2G_CUDA_TRY(cudaMemsetAsync(s.total, 0, 16, s.st));
    // longest sequence of the chunk (while the copies run)
    s.max_len = 0;
    for (uint64_t i = f0 * per; i < (f0 + nf) * per; i++)
      s.max_len = std::max(s.max_len, seq_off[i + 1] - seq_off[i]);
    return K2G_OK;
  };
  // Stage 2: classify.
  auto classify = [&](size_t c) -> k2g_status {
    Slot &s = slots[c % n_slots];
    const uint64_t f0 = s.f0, nf = s.nf, b0 = seq_off[f0 * per], nb = seq_off[(f0 + nf) * per] - b0;
    // (after the copies: a kernel waits for the blocks of the chunk before,
    // and copies behind it would too)
    K2G_CUDA_TRY(cudaStreamWaitEvent(s.st, s.left, 0));
    rebase_kernel<<<(unsigned)((nf * per + 1 + 255) / 256), 256, 0, s.st>>>(s.off, nf * per + 1, b0);
    note_launches();
    s.rd = k2g_reads{};
    s.rd.d_bases = s.bases;
    s.rd.d_quals = quals ? s.quals : nullptr;
    s.rd.d_seq_off = s.off;
    s.rd.n_frags = nf;
    s.rd.max_seq_len = s.max_len;
    s.rd.total_bases = nb;
    s.rd.frag_base = f0;
    s.rs = k2g_results{};
    s.rs.d_call = s.call;
    s.rs.d_hit_groups = s.hg;
    s.rs.d_hitlist_len = s.hlen;
    s.rs.d_runs = s.sparse;
    s.rs.runs_cap = s.cap_bases + 2 * s.cap_frags + 8;
    s.rs.d_taxon_reads = reinterpret_cast<uint64_t *>(d_taxon_reads);
    s.rs.d_status = reinterpret_cast<uint32_t *>(s.total + 1);
    if (counters) {
      s.rd.d_frag_block = s.blocks;
      s.rs.d_hit_keys = s.hit_keys;
      s.rs.d_hit_taxa = s.hit_taxa;
      s.rs.d_hit_order = s.hit_order;
      s.rs.hits_cap = s.cap_hits;
      s.rs.d_hits_used = s.hits_used;
    }
    // short-read chunks share one execution state (in order, as overlapping
    // them only adds interference); long-read chunks overlap their tails
    // (the one-launch form has no state)
    const void *key = long_batch(nb, nf) ? (const void *)s.st : (const void *)&hc;
    const k2g_status r = classify_keyed(db, &s.rd, params, &s.rs, K2G_MODE_PIPELINED, s.st, key);
    if (r != K2G_OK) return r;
    K2G_CUDA_TRY(cudaEventRecord(s.classified, s.st));
    return K2G_OK;
  };
  // Stage 3: count the events, compact the runs, copy the fixed-size results.
  auto copy_out = [&](size_t c) -> k2g_status {
    Slot &s = slots[c % n_slots];
    K2G_CUDA_TRY(cudaStreamWaitEvent(s.out, s.classified, 0));
    if (counters) {
      const k2g_status r = k2g_counters_add(counters, &s.rd, &s.rs, s.out);
      if (r != K2G_OK) return r;
    }
    const k2g_status r = compact_runs(s.sparse, s.off, per, s.hlen, s.nf, s.excl, s.sums, s.total, s.dense,
                                      long_batch(s.rd.total_bases, s.nf), s.out);
    if (r != K2G_OK) return r;
    K2G_CUDA_TRY(cudaMemcpyAsync(s.h_total, s.total, 16, cudaMemcpyDeviceToHost, s.out));
    K2G_CUDA_TRY(cudaEventRecord(s.done, s.out));
    K2G_CUDA_TRY(cudaMemcpyAsync(call + s.f0, s.call, s.nf * 4, cudaMemcpyDeviceToHost, s.out));
    if (hit_groups)
      K2G_CUDA_TRY(cudaMemcpyAsync(hit_groups + s.f0, s.hg, s.nf * 4, cudaMemcpyDeviceToHost, s.out));
    if (hitlist_len)
      K2G_CUDA_TRY(cudaMemcpyAsync(hitlist_len + s.f0, s.hlen, s.nf * 4, cudaMemcpyDeviceToHost, s.out));
    s.copied = true;
    return K2G_OK;
  };
  // Stage 4: copy the runs, whose number the host now knows (chunk order).
  uint64_t runs_written = 0;
  auto copy_runs = [&](size_t c) -> k2g_status {
    Slot &s = slots[c % n_slots];
    if (!s.copied) return K2G_OK;
    const cudaError_t e = cudaEventSynchronize(s.done);
    s.copied = false;
    if (e != cudaSuccess) return cuda_fail(e, "chunk completion");
    if ((uint32_t)s.h_total[1]) return fail(K2G_ERR_CAPACITY, "classification buffer overflow");
    const uint64_t nr = s.h_total[0];
    if (runs) {
      if (runs_written + nr > runs_cap) return fail(K2G_ERR_CAPACITY, "runs buffer too small");
      K2G_CUDA_TRY(cudaMemcpyAsync(runs + runs_written, s.dense, nr * 8, cudaMemcpyDeviceToHost, s.out));
    }
    K2G_CUDA_TRY(cudaEventRecord(s.left, s.out));
    runs_written += nr;
    return K2G_OK;
  };
  auto all_chunks = [&]() -> k2g_status {
    // with counters, stage 3 of a chunk makes the host wait for its kernels:
    // the next chunk's are in the queue and the copies of the one after it on
    // their way before that (1M x 150 bp: 4.2 -> 2.9 ms
    // for the classification)
    const size_t lag = counters ? 1 : 0, ahead = counters && n_slots > 2 ? 1 : 0;
    for (size_t c = 0; c < n_chunks + ahead + lag; c++) {
      k2g_status r = K2G_OK;
      if (ahead && c >= ahead && c - ahead < n_chunks) r = classify(c - ahead);
      if (r == K2G_OK && c < n_chunks) {
        if (c >= n_slots) r = copy_runs(c - n_slots);
        if (r == K2G_OK) r = copy_in(c);
        if (r == K2G_OK && !ahead) r = classify(c);
      }
      if (r == K2G_OK && c >= ahead + lag) r = copy_out(c - ahead - lag);
      if (r != K2G_OK) return r;
    }
    for (size_t c = n_chunks > n_slots ? n_chunks - n_slots : 0; c < n_chunks; c++) {
      const k2g_status r = copy_runs(c);
      if (r != K2G_OK) return r;
    }
    return K2G_OK;
  };
  const k2g_status status = all_chunks();
  // every copy is done (on an error too: the slots are free for the next call)
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < used; i++) {
    for (cudaStream_t x : {slots[i].st, slots[i].out}) {
      const cudaError_t es = cudaStreamSynchronize(x);
      if (es != cudaSuccess) e = es;
    }
    slots[i].copied = false;
  }
  if (status != K2G_OK) return status;
  if (e != cudaSuccess) return cuda_fail(e, "host classification");
  if (taxon_reads) {
    std::vector<uint64_t> tr(db->node_count);
    K2G_CUDA_TRY(cudaMemcpy(tr.data(), d_taxon_reads, db->node_count * 8, cudaMemcpyDeviceToHost));
    for (uint64_t i = 0; i < db->node_count; i++) taxon_reads[i] += tr[i];
  }
  if (n_runs) *n_runs = runs_written;
  return K2G_OK;
}

extern "C" k2g_status k2g_classify_host(const k2g_db *db, const char *bases, const char *quals,
                                        const uint64_t *seq_off, uint64_t n_frags,
                                        const k2g_classify_params *params, uint32_t *call,
                                        uint32_t *hit_groups, uint32_t *hitlist_len,
                                        uint64_t *runs, uint64_t *n_runs,
                                        uint64_t *taxon_reads) {
  return host_classify(db, bases, quals, seq_off, n_frags, nullptr, nullptr, params, call,
                       hit_groups, hitlist_len, runs, n_runs, taxon_reads);
}

extern "C" k2g_status k2g_classify_host_blocks(const k2g_db *db, const char *bases,
                                               const char *quals, const uint64_t *seq_off,
                                               uint64_t n_frags, const uint32_t *frag_block,
                                               k2g_counters *counters,
                                               const k2g_classify_params *params, uint32_t *call,
                                               uint32_t *hit_groups, uint32_t *hitlist_len,
                                               uint64_t *runs, uint64_t *n_runs,
                                               uint64_t *taxon_reads) {
  return host_classify(db, bases, quals, seq_off, n_frags, frag_block, counters, params, call,
                       hit_groups, hitlist_len, runs, n_runs, taxon_reads);
}
