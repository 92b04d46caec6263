// mutation_grid.h -- how many CTAs the mutation kernel is launched with (host only,
// no CUDA).
#pragma once
#include <algorithm>
#include <cstdint>

namespace dycg {

constexpr int MUT_BLOCK = 512;  // threads of one of its CTAs

// Most CTAs of the mutation kernel. `asked` (dycg_options.mutation_ctas) counts CTAs
// of eight warps, as it always has: two of them are one of this kernel's. Without it,
// random host transactions cost four times as much over tens of GB as within one,
// unless those in flight fall into a narrow window: a CTA on a quarter of the SMs
// takes 2.41 ms of a 100K-update R-MAT 26 snapshot (30 GB), one on half of them 2.71,
// one on each 2.98. At 1.6 GB (R-MAT 21) the three take 0.94-0.96 ms, and below it
// the suffix scans want all the warps (CC on 500K vertices: 3.66 against 3.40 ms a
// pass). Between 1.6 and 30 GB nothing was measured.
inline uint32_t mutation_ctas(uint32_t asked, uint32_t sms, uint64_t arena_bytes) {
  if (asked) return asked / 2 + asked % 2;
  return arena_bytes > (4ull << 30) ? std::max(1u, sms / 4) : sms;
}

// CTAs of one launch. The records are in row order (sorted by ingest) and the rows in
// arena order, so the warps in flight work on a window of consecutive records; capping
// the CTAs narrows that window of the host arena, and the host link serves
// transactions in a narrow window several times faster than ones spread over a
// multi-GB arena. A small batch needs no more CTAs than it has warps' work for, and
// its barriers are cheaper with fewer; but one record can fill a row of any length,
// so there are eight: three records that fill a 2^20-slot row take 1.0 ms with one
// CTA, 0.20 with eight and 0.17 with sixteen, a batch of 32 records 19 us of mutation
// with four or eight CTAs and 20.5 with sixteen.
inline uint32_t mutation_grid(uint32_t records, uint32_t dirs, uint32_t ctas, uint64_t resident) {
  const uint64_t warps = ((uint64_t)records * dirs + 3) / 4;
  return (uint32_t)std::max<uint64_t>(
      1, std::min<uint64_t>({std::max<uint64_t>((warps + 1) / 2, 8), ctas, resident}));
}

}  // namespace dycg
