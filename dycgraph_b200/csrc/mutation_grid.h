// mutation_grid.h -- how many CTAs the mutation kernel is launched with (host only,
// no CUDA).
#pragma once
#include <algorithm>
#include <cstdint>

namespace dycg {

constexpr int MUT_BLOCK = 512;  // threads of one of its CTAs

constexpr uint32_t MUT_RECORDS = 256;            // records one of its CTAs has in flight
constexpr uint64_t MUT_WINDOW = 5ull << 30;      // bytes of arena those of all CTAs should span

// CTAs of one launch, for `records` of the longer kind. `asked`
// (dycg_options.mutation_ctas) is the most and counts CTAs of eight warps, as it always
// has: two of them are one of this kernel's.
//
// Without it: random host transactions cost four times as much over tens of GB as
// within one, unless those in flight fall into a narrow window. The records are in row
// order (sorted by ingest) and the rows in arena order, so those in flight span
// (CTAs x MUT_RECORDS / records) of the arenas, and above 4 GB the CTAs are as many as
// span MUT_WINDOW, a quarter of the SMs at least. R-MAT 26 (30 GB), 100K updates: 2.41
// ms of mutation with a CTA on a quarter of the SMs, 2.71 on half of them, 2.98 on
// each; R-MAT 27 (60 GB), 1M Zipf updates without / with a cache: 7.45 / 6.59 ms with a
// quarter, 6.86 / 5.79 with each. At 1.6 GB (R-MAT 21) the three
// take 0.94-0.96 ms, and below it the suffix scans want all the warps (CC on 500K
// vertices: 3.66 against 3.40 ms a pass). Between 1.6 and 30 GB nothing was measured.
//
// A small batch needs no more CTAs than it has warps' work for, and its barriers are
// cheaper with fewer; but one record can fill a row of any length, so there are eight:
// three records that fill a 2^20-slot row take 1.0 ms with one CTA, 0.20 with eight and
// 0.17 with sixteen, a batch of 32 records 19 us of mutation with four or eight CTAs and
// 20.5 with sixteen.
inline uint32_t mutation_grid(uint32_t records, uint32_t dirs, uint32_t asked, uint32_t sms,
                              uint64_t arena_bytes, uint64_t resident) {
  uint64_t most = sms;
  if (asked) {
    most = asked / 2 + asked % 2;
  } else if (arena_bytes > (4ull << 30)) {
    const double fits = (double)MUT_WINDOW / (double)arena_bytes * records / MUT_RECORDS;
    most = std::min<uint64_t>(sms, std::max<uint64_t>((uint64_t)fits, std::max(1u, sms / 4)));
  }
  const uint64_t warps = ((uint64_t)records * dirs + 3) / 4;
  return (uint32_t)std::max<uint64_t>(
      1, std::min<uint64_t>({std::max<uint64_t>((warps + 1) / 2, 8), most, resident}));
}

}  // namespace dycg
