// The one-launch classification of short fragments, and long fragments in
// pieces (warp_classify.cuh).
#include <algorithm>

#include "k2g_internal.h"
#include "warp_classify.cuh"

namespace k2g {
namespace {

// Nominal length of a warp's piece, in tuned piece lengths (those are for one
// lane): 2,048 bases by default.  A warp takes about 30 us for that beside
// the others of its SM, so the last pieces to run do not keep the device long.
constexpr uint32_t kWarpPieces = 4;

template <bool WIDE, bool HITS, bool LONG, class Shared>
cudaError_t launch_warp(const WcArgs &wa, cudaStream_t st) {
  const uint64_t blocks = (wa.piece_slots + wa.n_groups + kWcWarps - 1) / kWcWarps;
  warp_classify_kernel<WIDE, HITS, LONG, Shared>
      <<<(unsigned)blocks, kWcWarps * 32, kWcWarps * sizeof(Shared), st>>>(wa);
  note_launches();
  return cudaGetLastError();
}

template <bool LONG, class Shared>
cudaError_t launch(const WcArgs &wa, cudaStream_t st) {
  const bool hits = wa.a.hit_keys != nullptr;
  if (wa.a.table.wide)
    return hits ? launch_warp<true, true, LONG, Shared>(wa, st) : launch_warp<true, false, LONG, Shared>(wa, st);
  return hits ? launch_warp<false, true, LONG, Shared>(wa, st) : launch_warp<false, false, LONG, Shared>(wa, st);
}

}  // namespace

bool warp_classify_takes(const k2g_db *db, const ClassifyArgs &a, uint64_t max_len) {
  // (a walk that goes on keeps its sector's number in 32 bits; with several
  // roots the LCA of taxa one after another is not that of all: an LCA of 0
  // and the next taxon give the taxon)
  const uint64_t sectors = a.table.capacity / (a.table.wide ? 4 : 8);
  return db->one_root && a.scan.w == 5 && a.scan.revcom_version != 0 && max_len <= kWcMaxLen && sectors < (1ull << 32);
}

// Single fragments of two pieces and more are cut (quick mode stops inside a
// fragment, and a pair carries a mate border: those stay whole).
uint32_t warp_piece(int paired, int quick, uint64_t max_len, uint32_t piece_len) {
  const uint32_t piece = std::min(kWarpPieces * piece_len, kPieceLenMax);
  return !paired && !quick && max_len >= 2ull * piece ? piece : 0;
}

cudaError_t warp_classify(const ClassifyArgs &a, const uint2 *span, uint64_t max_len, uint64_t total_bases,
                          uint32_t piece_len, int device, int sms, cudaStream_t st) {
  WcArgs wa{a, span, 0, 0, 0};
  const uint32_t piece = warp_piece(a.cls.paired, a.cls.quick, max_len, piece_len);
  const bool split = piece != 0;
  // Fragments per group: as many as leave 28 groups an SM, up to about 1,600
  // bases (their entries fill the shared-memory list once); 4 where long
  // fragments are cut, since the average says nothing of the others then.
  // (28 an SM, two more than it holds at a time: with 26 a second wave that is
  // nearly empty is avoided at some sizes, 7,904 x 250 bp 29.1 -> 27.0 us and
  // 16,000 x 150 on a table within L2 31.1 -> 29.0, but the larger groups cost
  // more at others, 16,000 x 150 on 400 MB 34.2 -> 36.7 and x 250 51.3 -> 56.0,
  // 31,616 x 150 44.2 -> 47.1.)  Two of up to 170 bases, which one scan pass
  // holds (two of 158) or nearly so, cost little more than one: half as many
  // groups will do for them (5,000 x 150 bp 21.1 -> 18.5 us, x 165 20.7 -> 18.7,
  // 8,000 of 30 to 301 bases 37.8 -> 30.7; from 3,000 down no difference).
  const double avg = (double)total_bases / (double)a.n_frags;
  const uint64_t slots = (uint64_t)sms * kWcWarps * kWcBlocks;
  while ((2u << wa.log_reads) <= (uint32_t)(split ? 4 : kWcReads) &&
         (a.n_frags >> (wa.log_reads + 1)) >= (!wa.log_reads && !split && avg <= 170.0 ? slots / 2 : slots) &&
         (split || avg * (double)(2u << wa.log_reads) <= 1600.0))
    wa.log_reads++;
  wa.n_groups = (a.n_frags + (1ull << wa.log_reads) - 1) >> wa.log_reads;
  if (!split && max_len * (a.cls.paired ? 2 : 1) >= kManyBases) return launch<false, WcSharedMany>(wa, st);
  if (!split) return launch<false, WcShared>(wa, st);

  const uint64_t pc = split_pieces_cap(total_bases, piece), fc = split_frags_cap(total_bases, piece);
  const size_t at_pieces = 64, at_frags = at_pieces + pc * sizeof(SplitPiece),
               at_mark = at_frags + fc * sizeof(SplitFrag);
  unsigned char *mem = nullptr;
  cudaError_t e = scratch_alloc(reinterpret_cast<void **>(&mem), at_mark + a.n_frags, device, st);
  if (e != cudaSuccess) return e;
  SplitBufs b{mem + at_mark, reinterpret_cast<SplitPiece *>(mem + at_pieces), pc,
              reinterpret_cast<SplitFrag *>(mem + at_frags), fc, nullptr, nullptr,
              reinterpret_cast<unsigned long long *>(mem), piece};
  e = cudaMemsetAsync(mem, 0, at_frags, st);
  if (e == cudaSuccess) e = split_plan(a, b, sms, st);
  if (e == cudaSuccess) {
    wa.a.pieces = b.pieces;
    wa.a.n_pieces = b.ctr;
    wa.a.split_mark = b.mark;
    wa.piece_slots = pc;
    e = launch<true, WcShared>(wa, st);
  }
  if (e == cudaSuccess) {
    const uint64_t blocks = std::min<uint64_t>((fc + kMergeWarps - 1) / kMergeWarps, (uint64_t)sms * 12);
    warp_merge_kernel<<<(unsigned)blocks, kMergeWarps * 32, 0, st>>>(a, span, b);
    note_launches();
    e = cudaGetLastError();
  }
  const cudaError_t ef = cudaFreeAsync(mem, st);
  return e != cudaSuccess ? e : ef;
}

}  // namespace k2g
