// The one-launch classification of short fragments (warp_classify.cuh).
#include <algorithm>

#include "k2g_internal.h"
#include "warp_classify.cuh"

namespace k2g {

template <bool WIDE, bool HITS>
static cudaError_t launch_warp(const WcArgs &wa, cudaStream_t st) {
  const uint64_t blocks = (wa.n_groups + kWcWarps - 1) / kWcWarps;
  warp_classify_kernel<WIDE, HITS>
      <<<(unsigned)blocks, kWcWarps * 32, kWcWarps * sizeof(WcShared), st>>>(wa);
  note_launches();
  return cudaGetLastError();
}

bool warp_classify_takes(const ClassifyArgs &a, uint64_t max_len) {
  // (a walk that goes on keeps its sector's number in 32 bits)
  const uint64_t sectors = a.table.capacity / (a.table.wide ? 4 : 8);
  return a.scan.w == 5 && a.scan.revcom_version != 0 && max_len <= kWcMaxLen && sectors < (1ull << 32);
}

cudaError_t warp_classify(const ClassifyArgs &a, const uint2 *span, uint64_t total_bases, int sms,
                          cudaStream_t st) {
  WcArgs wa{a, span, 0, 0};
  // Fragments per group: as many as keep every warp slot of the device busy
  // (24 warps per SM are resident), up to about 1,600 bases (their entries
  // fill the shared-memory list once).
  const double avg = (double)total_bases / (double)a.n_frags;
  while ((2u << wa.log_reads) <= (uint32_t)kWcReads &&
         (a.n_frags >> (wa.log_reads + 1)) >= (uint64_t)sms * 24 &&
         avg * (double)(2u << wa.log_reads) <= 1600.0)
    wa.log_reads++;
  wa.n_groups = (a.n_frags + (1ull << wa.log_reads) - 1) >> wa.log_reads;
  const bool hits = a.hit_keys != nullptr;
  if (a.table.wide) return hits ? launch_warp<true, true>(wa, st) : launch_warp<true, false>(wa, st);
  return hits ? launch_warp<false, true>(wa, st) : launch_warp<false, false>(wa, st);
}

}  // namespace k2g
