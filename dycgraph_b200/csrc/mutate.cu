// mutate.cu -- in-place mutation of the pinned host adjacency (with
// write-through to resident HBM pages) by one ingested batch.
//
// Mutation keeps the chunk store's occurrence semantics
// (include/groute/graphs/source_local_chunk_store.h:220-406,
// BuildDeletionPlan :685-739): a deletion requested r times removes r live
// occurrences (fewer if fewer exist: the rest are counted missing), additions
// append occurrences, and a row whose block is full drops its deleted slots and,
// if it outgrew the block, moves to a new power-of-two block at the arena tail.
// Rows stay sorted in their prefix, so a deletion finds its target through the
// HBM fence index and one 128-byte read of the row instead of the reference's
// linear row scan. A deletion sets a bit of the HBM deletion bitmap (no host-link
// write).
//
// One cooperative launch mutates both directions: deletions and the inserted
// slots, a barrier, [long suffixes: two passes with a barrier each], the
// insertions' descriptors, a barrier, [full rows; long ones by the whole grid, with
// barriers of their own]. Bracketed phases run only when the batch needs them,
// which the barriers' published counters decide, so a snapshot needs no host
// synchronisation and a captured one takes the same path. What bounds it is the
// host link's random transactions, one per deletion and one per insertion and
// direction (3.4 ns each over a 1 GB arena: 0.68 ms of the 0.77 ms that phase 1
// takes for 100K updates at R-MAT 21), and the chain of dependent accesses (~6
// us) for small batches: so an 8-lane group serves a deletion (a 128-byte line
// per step), a lane an insertion row, and a small batch spreads over the SMs.
// Mutation per snapshot, before (a warp per record, a launch per step and
// direction, two host synchronisations) -> now: 32 updates 0.115 -> 0.019 ms,
// R-MAT 16 2K 0.140 -> 0.063 (0.10 after some hundred snapshots, when most rows
// are suffix), R-MAT 20 BFS 10K 0.20 -> 0.12, R-MAT 21 100K 1.62 -> 1.14.
#include "frontier.cuh"
#include "internal.h"
#include "mutation_grid.h"

namespace dycg {

namespace {

constexpr uint32_t COMPACT_WARP = 1024;  // longest row that one warp compacts
// Rows above this many slots are copied by the whole grid (copy_long), wherever they
// go. In place, one CTA takes 2048 slots per host round trip; on the way to a new
// block, a chunk's place needs the deletion bits of all slots before it. Mutation of
// a snapshot of 100 records that fills one row, by those forms -> by the grid: 2^13
// slots moved 0.066 -> 0.041 ms, 2^14 in place 0.076 -> 0.040, 2^16 0.25 -> 0.045,
// 2^20 3.9 -> 0.21, 2^23 in place 32 -> 1.5, moved 8.2 -> 0.98. At 2^12 they are level.
constexpr uint32_t LONG_ROW = 1u << 12;

struct Counts {
  uint32_t link = 0, hbm = 0, missing = 0, moved = 0;
};

// Live occurrences of `target` among slots [s, e) of the row at off, by groups
// of W lanes (converged warp; on: the group has work), U slots per lane and
// step: the first `rem` of them, in slot order, get their deletion bit. sorted:
// ids ascend, so a group stops past target; its steps follow the row's 128-byte
// lines, and the fence index tells whether the next line is worth a host
// read. Returns the slots this lane read.
template <int W, int U>
__device__ __forceinline__ uint32_t take_slots(const Adj &A, u64 off, uint32_t s, uint32_t e,
                                               uint32_t target, bool sorted, bool on,
                                               uint32_t &rem) {
  const uint32_t lane = lane_id(), gl = lane & (W - 1);
  const uint32_t gsh = W == 32 ? 0u : lane & ~(W - 1);
  const unsigned gmask = W == 32 ? 0xffffffffu : (1u << W) - 1;
  uint32_t reads = 0;
  bool past = !on;
  while (__any_sync(0xffffffffu, !past && rem && s < e)) {
    const bool go = !past && rem && s < e;
    uint32_t end = min(e, s + W * U);
    if (sorted) {  // to the end of this line
      const u64 line = (((off + s) >> A.fence_shift) + 1) << A.fence_shift;
      end = (uint32_t)min((u64)end, line - off);
    }
    uint32_t d[U], b[U], next = 0;
    if (go && sorted && end < e) next = A.fence[(off + end) >> A.fence_shift];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t x = s + u * W + gl;
      d[u] = 0;
      b[u] = 1;
      if (go && x < end) {
        const u64 p = off + x;
        d[u] = read_dst_rw(A, p);
        b[u] = (*(volatile uint32_t *)(A.tbits + (p >> 5)) >> (p & 31)) & 1u;
        reads++;
      }
    }
    past |= sorted && next > target;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t x = s + u * W + gl;
      const bool in = go && x < end;
      const bool live = in && d[u] == target && !b[u];
      const unsigned lm = (__ballot_sync(0xffffffffu, live) >> gsh) & gmask;
      const unsigned pm =
          (__ballot_sync(0xffffffffu, in && sorted && d[u] > target) >> gsh) & gmask;
      if (live && (uint32_t)__popc(lm & ((1u << gl) - 1)) < rem) {
        const u64 p = off + x;
        atomicOr(A.tbits + (p >> 5), 1u << (p & 31));
      }
      rem -= min((uint32_t)__popc(lm), rem);
      past |= pm != 0;
    }
    s = end;
  }
  return reads;
}

// Slot (row-relative) where the sorted prefix [0, srt) can first hold target:
// the HBM fence index holds the id of the first slot of every 128-byte group
// of slots, an 8-ary search over the row's fences narrows it to one group.
__device__ __forceinline__ uint32_t group_lower_bound(const Adj &A, u64 off, uint32_t srt,
                                                      uint32_t target, bool on) {
  const uint32_t lane = lane_id(), gl = lane & 7, gsh = lane & 24;
  const uint32_t fs = A.fence_shift;
  const u64 flo = (off + (1ull << fs) - 1) >> fs;  // fences inside the prefix
  u64 fhi = on && srt ? ((off + srt - 1) >> fs) + 1 : flo;
  if (fhi < flo) fhi = flo;
  u64 lo = flo, hi = fhi;
  while (__any_sync(0xffffffffu, hi - lo > 8)) {
    const bool go = hi - lo > 8;
    const u64 step = (hi - lo + 7) / 8;
    const u64 f = min(lo + (gl + 1) * step, hi) - 1;
    const unsigned ge = (__ballot_sync(0xffffffffu, go && A.fence[f] >= target) >> gsh) & 255u;
    if (!go) continue;
    if (!ge) {
      lo = hi;
    } else {
      const uint32_t k = __ffs(ge) - 1;
      hi = min(lo + (k + 1) * step, hi);
      lo += k * step;
    }
  }
  const unsigned ge =
      (__ballot_sync(0xffffffffu, lo + gl < hi && A.fence[lo + gl] >= target) >> gsh) & 255u;
  lo = ge ? lo + __ffs(ge) - 1 : hi;
  // the answer lies past slot (lo - 1) << fs, whose id is below target
  const u64 beg = lo > flo ? ((lo - 1) << fs) + 1 : off;
  return beg > off ? (uint32_t)(beg - off) : 0u;
}

__device__ __forceinline__ uint32_t next_pow2_u32(uint32_t x) {
  return x <= 1 ? 1u : 1u << (32 - __clz(x - 1));
}

// The records of a deletion's row, exact at the row's first entry; elsewhere
// as far as the deferral rule asks (DEFER_RECORDS or more, or fewer: exact), so
// that all of a row's records take the same side of it.
__device__ __forceinline__ uint32_t row_records(const Rec *list, uint32_t pos, const Rec &r) {
  uint32_t c = r.z;
  for (uint32_t k = 1; c < DEFER_RECORDS && k <= pos && list[pos - k].x == r.x; k++) c++;
  return c;
}

// Deletions of one direction's list, positions [p0, p0 + per).
__device__ void delete_records(const MutParams &M, uint32_t dir, uint32_t p0, uint32_t per,
                               uint32_t nd, Counts &C) {
  const Adj &A = M.adj[dir];
  const Rec *list = M.dels[dir];
  const uint32_t lane = lane_id(), gl = lane & 7;
  const uint32_t pos = p0 + lane;
  const bool have = lane < per && pos < nd;
  const Rec r = have ? list[pos] : make_uint4(INF32, INF32, 0u, 0u);
  uint32_t len = 0, srt = 0, rowrecs = 0;
  u64 off = 0;
  if (r.w) {
    rowrecs = row_records(list, pos, r);
    off = A.off[r.x];
    len = A.len[r.x];
    srt = A.srt[r.x];
  } else if (have && dir == 0) {
    M.found[pos] = 0;
  }
  const uint32_t rounds = per / 4;
  for (uint32_t t = 0; t < rounds; t++) {
    const uint32_t src = (lane >> 3) * rounds + t;
    const uint32_t row = __shfl_sync(0xffffffffu, r.x, src);
    const uint32_t target = __shfl_sync(0xffffffffu, r.y, src);
    const uint32_t mult = __shfl_sync(0xffffffffu, r.w, src);
    const u64 o = __shfl_sync(0xffffffffu, off, src);
    const uint32_t l = __shfl_sync(0xffffffffu, len, src);
    const uint32_t sp = __shfl_sync(0xffffffffu, srt, src);
    const uint32_t of_row = __shfl_sync(0xffffffffu, rowrecs, src);
    const bool on = mult != 0, many = of_row >= DEFER_RECORDS;
    if (!__any_sync(0xffffffffu, on)) continue;
    uint32_t rem = mult;
    const uint32_t s0 = group_lower_bound(A, o, sp, target, on);
    // (a line holds 16 slots with weights, 32 without)
    uint32_t reads = A.stride == 2 ? take_slots<8, 2>(A, o, s0, sp, target, true, on, rem)
                                   : take_slots<8, 4>(A, o, s0, sp, target, true, on, rem);
    // unsorted suffix: matched later with the row's other records, or a short
    // one by the group, a longer one by the warp
    const uint32_t suffix = l - sp;
    const bool defer = on && (suffix > DEFER_SUFFIX || (suffix > DEFER_SHORT && many));
    const bool tail = on && rem && suffix && !defer;
    reads += take_slots<8, 4>(A, o, sp, l, target, false, tail && suffix <= DEFER_SHORT, rem);
    unsigned wide = __ballot_sync(0xffffffffu, tail && suffix > DEFER_SHORT && gl == 0);
    while (wide) {
      const int w = __ffs(wide) - 1;
      wide &= wide - 1;
      uint32_t wrem = __shfl_sync(0xffffffffu, rem, w);
      const uint32_t wsp = __shfl_sync(0xffffffffu, sp, w);
      const uint32_t x = take_slots<32, 4>(A, __shfl_sync(0xffffffffu, o, w), wsp,
                                        __shfl_sync(0xffffffffu, l, w),
                                        __shfl_sync(0xffffffffu, target, w), false, true, wrem);
      const uint32_t all = __reduce_add_sync(0xffffffffu, x);
      if ((lane & 24) == (uint32_t)w) {
        rem = wrem;
        reads += gl == 0 ? all : 0;
      }
    }
    const bool cached = on && l && A.page_slot[page_of(A, o)] != PAGE_NONE;
    if (cached) C.hbm += 4 * reads; else C.link += 4 * reads;
    for (int k = 4; k; k >>= 1) reads += __shfl_xor_sync(0xffffffffu, reads, k);
    if (gl == 0 && on) {
      const uint32_t at = p0 + src, found = mult - rem;
      if (found) atomicSub(A.live + row, found);
      if (dir == 0) M.found[at] = found;
      if (defer) {
        // matched with all the row's records at once, later (suffix_*); the
        // row's first record announces it
        M.rem[dir][at] = rem;
        M.matches[dir][at] = 0;
        if (at == 0 || list[at - 1].x != row) {
          const uint32_t i1 = at + of_row;  // exact at the row's first entry
          const uint32_t nch = (suffix + SUFFIX_CHUNK - 1) / SUFFIX_CHUNK;
          const uint32_t base = atomicAdd(&M.mctl->q_count[0], nch);
          if (base + nch > M.suffix_cap) {
            atomicCAS(&M.ctl->err, 0u, ERR_QUEUE);
          } else {
            for (uint32_t c = 0; c < nch; c++)
              M.suffix[base + c] = make_uint4(at, i1, c, dir | (nch << 1));
          }
        }
      } else if (dir == 0) {
        C.missing += rem;
      }
      if (reads) atomicAdd(A.page_hits + page_of(A, o + min(s0, l - 1)), reads);
    }
  }
}

// Long suffixes, a warp per SUFFIX_CHUNK slots of a deferred row and pass.
//   COUNT  every live slot is looked up among the row's records (sorted by
//          neighbour): a lane's eight slots are read together and bisected
//          together. Each record's matches are counted, and the slots' records
//          stay in HBM (chunks past suffix_keep are read from the host again).
//   MARK   the matches of the records that want all of theirs are deleted.
// A record that wants fewer than there are (two hubs joined by many occurrences) gets
// the earliest ones. Its suffix is cut into OVER_SEGS segments:
//   HIST   its matches per segment are counted;
//   [over_cut, a warp per record: the segment in which its last one lies, and the
//          deletions within that segment]
//   CUT    its matches in the segments before that are deleted.
// A warp per such record that walked the suffix instead read a good part of it over the
// link for each: 100K Zipf updates on R-MAT 22 took 7.6 ms of mutation without a cache
// and 3.2 with the learned one, now 0.58 and 0.37; a pass of 2,000-update snapshots
// on R-MAT 16, whose rows are suffix for the most part, 1.92 ms, now 1.57.
enum SuffixPass { COUNT, MARK, HIST, CUT };
constexpr uint32_t NO_OVER = 0xFFFFFFFFu;

// Records that want fewer occurrences than match, in buffers of the relocation phase,
// which comes later: the list (record, its row's first chunk, chunks << 1 |
// direction, segment of the cut) and each record's place in it.
__device__ __forceinline__ uint4 *over_list(const MutParams &M) {
  return reinterpret_cast<uint4 *>(M.reloc.rec);
}
__device__ __forceinline__ uint32_t *over_of(const MutParams &M, uint32_t dir) {
  return reinterpret_cast<uint32_t *>(M.reloc.longs) + dir * (M.reloc.cap / M.dirs);
}
__device__ __forceinline__ uint32_t segment_of(uint32_t chunk, uint32_t chunks) {
  return (uint32_t)((u64)chunk * OVER_SEGS / chunks);
}

template <SuffixPass PASS>
__device__ void suffix_chunk(const MutParams &M, uint32_t c, uint32_t window, Counts &C) {
  constexpr int U = SUFFIX_CHUNK / 32;
  const uint4 ch = M.suffix[c];
  const uint32_t dir = ch.w & 1, nch = ch.w >> 1;
  const Adj &A = M.adj[dir];
  const Rec *list = M.dels[dir];
  const uint32_t lane = lane_id();
  // nothing left to look for: the records were found in the prefix (their
  // remainders are in HBM, the suffix is across the link)
  bool wanted = false;
  for (uint32_t i = ch.x + lane; i < ch.y && !wanted; i += 32)
    wanted = list[i].w && M.rem[dir][i];
  if (!__any_sync(0xffffffffu, wanted)) return;
  const uint32_t row = list[ch.x].x;
  const u64 off = A.off[row];
  const uint32_t srt = A.srt[row], len = A.len[row];
  const uint32_t b = srt + ch.z * SUFFIX_CHUNK, e = min(len, b + SUFFIX_CHUNK);
  uint32_t *keep = M.suffix_ids + (u64)c * SUFFIX_CHUNK;
  uint32_t lo[U];  // the slots' records, INF32: none that wants any
  if (PASS != COUNT && c < M.suffix_keep) {
#pragma unroll
    for (int u = 0; u < U; u++) lo[u] = keep[u * 32 + lane];
  } else {
    const uint32_t pg0 = page_of(A, off + b);
    const bool cached = A.page_slot[pg0] != PAGE_NONE;
    uint32_t d[U], same = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t s = b + u * 32 + lane;
      d[u] = INF32;  // past every record's neighbour
      if (s < e) {
        const u64 p = off + s;
        const uint32_t x = read_dst_rw(A, p);
        if (!slot_deleted_rw(A, p)) d[u] = x;
        if (page_of(A, p) == pg0) same++;
        else atomicAdd(A.page_hits + page_of(A, p), 1u);
        if (cached) C.hbm += 4; else C.link += 4;
      }
    }
    same = __reduce_add_sync(0xffffffffu, same);
    if (lane == 0 && same) atomicAdd(A.page_hits + pg0, same);
    // first of the row's entries with neighbour >= d (a run's first entry opens it)
#pragma unroll
    for (int u = 0; u < U; u++) lo[u] = ch.x;
    for (uint32_t width = ch.y - ch.x; width;) {
      const uint32_t half = (width + 1) / 2;
#pragma unroll
      for (int u = 0; u < U; u++) {
        const uint32_t mid = lo[u] + half - 1;
        if (mid < ch.y && list[mid].y < d[u]) lo[u] = mid + 1;
      }
      width -= half;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (d[u] == INF32 || lo[u] >= ch.y || list[lo[u]].y != d[u] || !M.rem[dir][lo[u]])
        lo[u] = INF32;
    if (PASS == COUNT && c < M.suffix_keep) {
#pragma unroll
      for (int u = 0; u < U; u++) keep[u * 32 + lane] = lo[u];
    }
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
    if (lo[u] == INF32) continue;
    bool mark = false;
    if (PASS == COUNT) {
      atomicAdd(M.matches[dir] + lo[u], 1u);
    } else if (PASS == MARK) {
      mark = M.matches[dir][lo[u]] <= M.rem[dir][lo[u]];
    } else {
      const uint32_t id = over_of(M, dir)[lo[u]];
      if (id < window || id - window >= M.over_window) continue;  // (NO_OVER among them)
      const uint32_t seg = segment_of(ch.z, nch);
      if (PASS == HIST) atomicAdd(M.over_hist + (u64)(id - window) * OVER_SEGS + seg, 1u);
      else mark = seg < over_list(M)[id].w;
    }
    if (mark) {
      const u64 p = off + b + u * 32 + lane;
      atomicOr(A.tbits + (p >> 5), 1u << (p & 31));
    }
  }
  if (PASS != MARK) return;
  // this chunk's share of the row's records
  const uint32_t share = (ch.y - ch.x + nch - 1) / nch;
  const uint32_t i0 = ch.x + ch.z * share, i1 = min(ch.y, i0 + share);
  for (uint32_t p0 = i0; p0 < i1; p0 += 32) {
    const uint32_t p = p0 + lane;
    const uint32_t want = p < i1 && list[p].w ? M.rem[dir][p] : 0u;
    const uint32_t match = want ? M.matches[dir][p] : 0u;
    const uint32_t taken = min(want, match);
    if (taken) {
      atomicSub(A.live + row, taken);
      if (dir == 0) M.found[p] += taken;
    }
    if (dir == 0) C.missing += want - taken;
    unsigned over = __ballot_sync(0xffffffffu, match > want && want);
    uint32_t id = 0;
    if (over && lane == 0) id = atomicAdd(&M.mctl->a_pool, (uint32_t)__popc(over));
    id = __shfl_sync(0xffffffffu, id, 0) + __popc(over & ((1u << lane) - 1));
    const bool mine = (over >> lane) & 1u;
    if (p < i1) over_of(M, dir)[p] = mine ? id : NO_OVER;
    if (mine) over_list(M)[id] = make_uint4(p, c - ch.z, nch << 1 | dir, 0u);
    for (; over; over &= over - 1) {  // (the first window's counts)
      const uint32_t o = __shfl_sync(0xffffffffu, id, __ffs(over) - 1);
      if (o < M.over_window) M.over_hist[(u64)o * OVER_SEGS + lane] = 0;
    }
  }
}

// Where the deletions of record `id` of the list end: all of its matches in the
// segments before the cut (CUT marks those), the first few in the cut's own.
__device__ void over_cut(const MutParams &M, uint32_t id, uint32_t window, Counts &C) {
  constexpr int U = SUFFIX_CHUNK / 32;
  static_assert(OVER_SEGS == 32, "a lane per segment");
  const uint4 o = over_list(M)[id];
  const uint32_t dir = o.z & 1, nch = o.z >> 1, lane = lane_id();
  const uint32_t want = M.rem[dir][o.x];
  uint32_t upto = M.over_hist[(u64)(id - window) * OVER_SEGS + lane];
#pragma unroll
  for (int k = 1; k < 32; k *= 2) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, upto, k);
    if (lane >= (uint32_t)k) upto += x;
  }
  // (there are more matches than wanted ones, so some segment goes past them)
  const uint32_t cut = __ffs(__ballot_sync(0xffffffffu, upto > want)) - 1;
  const uint32_t before = __shfl_sync(0xffffffffu, upto, (cut - 1) & 31);
  uint32_t rem = want - (cut ? before : 0u);
  if (lane == 0) over_list(M)[id].w = cut;
  const Adj &A = M.adj[dir];
  const Rec rec = M.dels[dir][o.x];
  const u64 off = A.off[rec.x];
  const uint32_t srt = A.srt[rec.x], len = A.len[rec.x];
  for (uint32_t z = (cut * nch + OVER_SEGS - 1) / OVER_SEGS;
       rem && z < nch && segment_of(z, nch) == cut; z++) {
    const uint32_t c = o.y + z, b = srt + z * SUFFIX_CHUNK;
    bool hit[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t s = b + u * 32 + lane;
      if (c < M.suffix_keep) {
        hit[u] = M.suffix_ids[(u64)c * SUFFIX_CHUNK + u * 32 + lane] == o.x;
      } else {
        hit[u] = s < len && read_dst_rw(A, off + s) == rec.y && !slot_deleted_rw(A, off + s);
        if (s < len) C.link += 4;
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const unsigned m = __ballot_sync(0xffffffffu, hit[u]);
      if (hit[u] && (uint32_t)__popc(m & ((1u << lane) - 1)) < rem) {
        const u64 p = off + b + u * 32 + lane;
        atomicOr(A.tbits + (p >> 5), 1u << (p & 31));
      }
      rem -= min(rem, (uint32_t)__popc(m));
    }
  }
}

// Insertions of one direction's list, a lane per row segment, in two steps.
// First the occurrences of the segments that fit their blocks are written behind
// the rows' slots: nothing looks there before the rows' lengths say so, so the
// host writes go out while the deletions' host reads come in.
__device__ void append_slots(const MutParams &M, uint32_t dir, uint32_t pos, uint32_t na,
                             Counts &C) {
  const Adj &A = M.adj[dir];
  const Rec *list = M.adds[dir];
  const uint32_t bytes = 4u * A.stride;
  const Rec r = pos < na ? list[pos] : make_uint4(INF32, INF32, 0u, 0u);
  const uint32_t count = r.w;
  u64 at = 0;
  bool fits = false;
  if (count) {
    const uint32_t len = A.len[r.x];
    fits = (u64)len + count <= A.cap[r.x];
    at = A.off[r.x] + len;
  }
  // short segments by their lane, long ones by the warp
  const bool lone = fits && count <= 4;
  for (uint32_t j = 0; lone && j < count; j++) {
    const Rec x = j ? list[pos + j] : r;
    const bool c = write_slot(A, at + j, x.y, x.z);
    C.link += bytes;
    if (c) C.hbm += bytes;
  }
  unsigned wide = __ballot_sync(0xffffffffu, fits && !lone);
  while (wide) {
    const int src = __ffs(wide) - 1;
    wide &= wide - 1;
    const uint32_t wp = __shfl_sync(0xffffffffu, pos, src);
    const uint32_t wc = __shfl_sync(0xffffffffu, count, src);
    const u64 wa = __shfl_sync(0xffffffffu, at, src);
    for (uint32_t j = lane_id(); j < wc; j += 32) {
      const Rec x = list[wp + j];
      const bool c = write_slot(A, wa + j, x.y, x.z);
      C.link += bytes;
      if (c) C.hbm += bytes;
    }
  }
}

// Long rows of this launch in two lists (0: those that stay in their block, 1: those
// that move, from the end of the same array), each row with the number of its first
// chunk: one addition gives both places, so the numbers ascend along a list. The
// chunks' counts live in the suffix phase's list, which is over: 4 bytes per 512
// slots of long rows, where that list has 16 per 256 slots of the arena.
constexpr uint32_t LONG_CHUNK = 512;
struct LongRows {
  uint2 *first;      // (relocation record, first chunk) of row 0, row 1 at first[step]
  int step;
  uint32_t *count;   // per chunk: its live slots, then those before it
  uint32_t rows, chunks;
  __device__ uint2 &row(uint32_t i) const { return first[(int)i * step]; }
};
__device__ __forceinline__ LongRows long_rows(const MutParams &M, uint32_t list) {
  const u64 n = *(volatile u64 *)(list ? &M.mctl->a_tail : &M.mctl->a_head);
  return {list ? M.reloc.longs + M.reloc.cap - 1 : M.reloc.longs, list ? -1 : 1,
          reinterpret_cast<uint32_t *>(M.suffix) + (u64)list * M.suffix_cap * 2,
          (uint32_t)(n >> 32), (uint32_t)n};
}
__device__ __forceinline__ void list_long(const MutParams &M, uint32_t list, uint32_t k,
                                          uint32_t len) {
  const u64 at = atomicAdd(list ? &M.mctl->a_tail : &M.mctl->a_head,
                           (1ull << 32) | ((len + LONG_CHUNK - 1) / LONG_CHUNK));
  long_rows(M, list).row(at >> 32) = make_uint2(k, (uint32_t)at);
}

// A block of `slots` slots at the arena tail, or NO_BLOCK when the rest of the arena
// does not hold it. Small blocks are many (a thousand rows may outgrow theirs in one
// launch) and take one addition; a large one that does not fit must leave the rest
// to smaller ones, so it takes a compare-and-swap, and there are few of them.
constexpr u64 NO_BLOCK = ~0ull;
constexpr uint32_t SMALL_BLOCK = 1u << 16;
__device__ __forceinline__ u64 reserve_block(const Adj &A, uint32_t slots) {
  u64 top = *(volatile u64 *)A.top;
  if (slots <= SMALL_BLOCK) {
    if (top + slots > A.arena) return NO_BLOCK;
    top = atomicAdd(A.top, (u64)slots);
    return top + slots <= A.arena ? top : NO_BLOCK;
  }
  while (top + slots <= A.arena) {
    const u64 seen = atomicCAS(A.top, top, top + slots);
    if (seen == top) return top;
    top = seen;
  }
  return NO_BLOCK;
}

// Then, the deletions done, the descriptors. A row that does not fit drops its
// deleted slots on its way to a new power-of-two block (with headroom) at the
// arena tail, or in its own block: when they are half of it (the copy of a block is
// then paid for by half as many appends before the next one; 5/8 and 3/4 took the
// same time in every stream), once the block that its slots ask for would reach into
// the second half of the arena's headroom, whenever the live occurrences and a reserve
// fit, and whenever they fit at all if the arena has no such block left. So a row takes
// space for good only when its live occurrences outgrow its block (2,000-update
// snapshots on R-MAT 16 used to eat the arena in some 5,000 of them), no row asks
// in vain for a larger block than it needs, and no repair reads a slot deleted
// long ago for ever. Rows that change their slots are left to the relocation phase.
__device__ void append_rows(const MutParams &M, uint32_t dir, uint32_t pos, uint32_t na,
                            Counts &C) {
  const Adj &A = M.adj[dir];
  const Rec r = pos < na ? M.adds[dir][pos] : make_uint4(INF32, INF32, 0u, 0u);
  const uint32_t row = r.x, count = r.w;
  if (!count) return;
  const uint32_t len = A.len[row], cap = A.cap[row], live = A.live[row];
  if ((u64)len + count <= cap) {
    A.len[row] = len + count;
    A.live[row] = live + count;
    // appends stay in the unsorted suffix (no host-link read here); an
    // empty row takes its sorted run of appends as its sorted prefix
    if (len == 0) A.srt[row] = count;
    return;
  }
  const auto block = [](u64 slots) { return next_pow2_u32((uint32_t)(slots + slots / 8 + 1)); };
  const u64 need = (u64)live + count, off = A.off[row];
  const uint32_t tight = block(need), roomy = block((u64)len + count);
  const bool scarce = *(volatile u64 *)A.top + roomy > M.scarce[dir];
  bool stays = tight <= cap && (scarce || need <= cap / 2);
  if (!stays) {
    uint32_t ncap = scarce ? tight : roomy;
    u64 noff = reserve_block(A, ncap);
    if (noff == NO_BLOCK && need > cap && tight < ncap) {
      ncap = tight;
      noff = reserve_block(A, ncap);
    }
    stays = noff == NO_BLOCK && need <= cap;
    if (!stays) {
      if (noff == NO_BLOCK) {
        atomicCAS(&M.ctl->err, 0u, ERR_ARENA);
        return;
      }
      const uint32_t nchunk = len > LONG_ROW ? 0 : (len + RELOC_CHUNK - 1) / RELOC_CHUNK;
      const uint32_t cb = nchunk ? atomicAdd(&M.mctl->tile_count, nchunk) : 0;
      const uint32_t k = atomicAdd(&M.mctl->q_count[1], 1u);
      if (k >= M.reloc.cap || cb + nchunk > M.reloc.chunk_cap) {
        atomicCAS(&M.ctl->err, 0u, ERR_ARENA);
        return;
      }
      M.reloc.rec[k] = RelocRec{row, pos, len, dir, off, noff};
      for (uint32_t c = 0; c < nchunk; c++) M.reloc.chunks[cb + c] = make_uint2(k, c);
      if (len > LONG_ROW) list_long(M, 1, k, len);
      A.off[row] = noff;
      A.cap[row] = ncap;
      C.moved++;
      return;
    }
  }
  const uint32_t k = atomicAdd(&M.mctl->q_count[1], 1u);
  if (k >= M.reloc.cap) {
    atomicCAS(&M.ctl->err, 0u, ERR_ARENA);
    return;
  }
  M.reloc.rec[k] = RelocRec{row, pos, len, dir, off, off};
  // a wide row takes a whole CTA, a long one the whole grid
  if (len > LONG_ROW) list_long(M, 0, k, len);
  else if (len > COMPACT_WARP) M.reloc.wide[atomicAdd(&M.mctl->q_count[2], 1u)] = k;
}

// Deleted slots among the first `count` of the row at off (warp-collective).
__device__ __forceinline__ uint32_t dead_slots(const Adj &A, u64 off, uint32_t count) {
  if (!count) return 0;
  const u64 w0 = off >> 5, w1 = (off + count - 1) >> 5;
  uint32_t dead = 0;
  for (u64 w = w0 + lane_id(); w <= w1; w += 32) {
    uint32_t b = *(volatile uint32_t *)(A.tbits + w);
    if (w == w0) b &= ~0u << (off & 31);
    if (w == w1) b &= ~0u >> (31 - ((off + count - 1) & 31));
    dead += __popc(b);
  }
  return __reduce_add_sync(0xffffffffu, dead);
}

// Warp per RELOC_CHUNK slots of a row that moves: its live slots in order,
// behind those of the chunks before it (the bitmap tells how many), eight loads
// in flight per lane.
__device__ void relocate_chunk(const MutParams &M, uint2 ch, Counts &C) {
  const RelocRec rec = M.reloc.rec[ch.x];
  const Adj &A = M.adj[rec.dir];
  const uint32_t bytes = 4u * A.stride;
  const uint32_t b = ch.y * RELOC_CHUNK, e = min(rec.len, b + RELOC_CHUNK);
  u64 to = rec.new_off + b - dead_slots(A, rec.old_off, b);
  constexpr uint32_t PER = 8;
  for (uint32_t s0 = b; s0 < e; s0 += PER * 32) {
    uint2 v[PER];
    bool live[PER];
#pragma unroll
    for (uint32_t t = 0; t < PER; t++) {
      const uint32_t s = s0 + t * 32 + lane_id();
      live[t] = false;
      if (s < e) {
        v[t] = read_pair_rw(A, rec.old_off + s);
        live[t] = !slot_deleted_rw(A, rec.old_off + s);
        C.link += bytes;
      }
    }
#pragma unroll
    for (uint32_t t = 0; t < PER; t++) {
      const unsigned lm = __ballot_sync(0xffffffffu, live[t]);
      if (live[t]) {
        const bool c =
            write_slot(A, to + __popc(lm & ((1u << lane_id()) - 1)), v[t].x, v[t].y);
        C.link += bytes;
        if (c) C.hbm += bytes;
      }
      to += __popc(lm);
    }
  }
}

// The same within a row's own block, by T threads (a warp, or a CTA with sm):
// T * 4 slots at a time are read before the live ones among them are written,
// never past what has been read, and their deletion bits are cleared.
template <uint32_t T>
__device__ void compact_row(const MutParams &M, const RelocRec &rec, uint32_t *sm, Counts &C) {
  const Adj &A = M.adj[rec.dir];
  const uint32_t bytes = 4u * A.stride;
  const uint32_t me = T == 32 ? lane_id() : threadIdx.x, warp = me >> 5;
  constexpr uint32_t PER = 4, W = T / 32;
  u64 to = rec.old_off;
  for (uint32_t s0 = 0; s0 < rec.len; s0 += PER * T) {
    uint2 v[PER];
    unsigned lm[PER];
#pragma unroll
    for (uint32_t t = 0; t < PER; t++) {
      const uint32_t s = s0 + t * T + me;
      const u64 p = rec.old_off + s;
      bool live = false;
      if (s < rec.len) {
        v[t] = read_pair_rw(A, p);
        live = !slot_deleted_rw(A, p);
        if (!live) atomicAnd(A.tbits + (p >> 5), ~(1u << (p & 31)));
        C.link += bytes;
      }
      lm[t] = __ballot_sync(0xffffffffu, live);
      if (T > 32 && lane_id() == 0) sm[t * W + warp] = __popc(lm[t]);
    }
    // every read of this step is done before any write of it
    if (T > 32) __syncthreads();
    else __syncwarp();
#pragma unroll
    for (uint32_t t = 0; t < PER; t++) {
      uint32_t before = 0, all = __popc(lm[t]);
      if (T > 32) {
        all = 0;
        for (uint32_t w = 0; w < W; w++) {
          if (w == warp) before = all;
          all += sm[t * W + w];
        }
      }
      if ((lm[t] >> lane_id()) & 1u) {
        const u64 p = to + before + __popc(lm[t] & ((1u << lane_id()) - 1));
        if (p != rec.old_off + s0 + t * T + me) {
          const bool c = write_slot(A, p, v[t].x, v[t].y);
          C.link += bytes;
          if (c) C.hbm += bytes;
        }
      }
      to += all;
    }
    if (T > 32) __syncthreads();  // (sm is free again)
  }
}

// A row's inserted occurrences behind its live slots, and its descriptor; sorted:
// live slots of its sorted prefix. T threads, me-th of them.
__device__ void finish_row(const MutParams &M, const RelocRec &rec, uint32_t sorted, uint32_t me,
                           uint32_t T) {
  const Adj &A = M.adj[rec.dir];
  const Rec *list = M.adds[rec.dir];
  const uint32_t count = list[rec.seg].w, live = A.live[rec.row];
  for (uint32_t j = me; j < count; j += T) {
    const Rec x = list[rec.seg + j];
    write_slot(A, rec.new_off + live + j, x.y, x.z);
  }
  if (T == 32) __syncwarp();
  else __syncthreads();  // every thread has read the old descriptor
  if (me == 0) {
    A.srt[rec.row] = live ? sorted : count;
    A.len[rec.row] = live + count;
    A.live[rec.row] = live + count;
  }
}

// Warp per listed row: rows that moved get their insertions, short ones that
// stay are compacted first.
__device__ void finish_warp(const MutParams &M, const RelocRec &rec, Counts &C) {
  const Adj &A = M.adj[rec.dir];
  const bool stays = rec.new_off == rec.old_off;
  if (rec.len > (stays ? COMPACT_WARP : LONG_ROW)) return;  // a CTA's or the grid's
  const uint32_t srt = A.srt[rec.row];
  const uint32_t sorted = srt - dead_slots(A, rec.old_off, srt);
  __syncwarp();
  if (stays) compact_row<32>(M, rec, nullptr, C);
  finish_row(M, rec, sorted, lane_id(), 32);
}

// Chunk g of a list: its row's relocation record (x) and its number in the row (y).
__device__ __forceinline__ uint2 long_chunk(const LongRows &L, uint32_t g) {
  uint32_t lo = 0, hi = L.rows;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (L.row(mid).y <= g) lo = mid; else hi = mid;
  }
  const uint2 r = L.row(lo);
  return make_uint2(r.x, g - r.y);
}

// A warp's chunk in registers: its slots, which of them live, and where those go.
constexpr uint32_t LONG_PER = LONG_CHUNK / 32;
struct LongPiece {
  uint2 v[LONG_PER];
  unsigned live[LONG_PER];
  u64 to;
  uint32_t dir;
};
__device__ __forceinline__ void read_long(const MutParams &M, const LongRows &L, uint32_t g,
                                          LongPiece &x, Counts &C) {
  const uint32_t lane = lane_id();
  const uint2 ch = long_chunk(L, g);
  const RelocRec rec = M.reloc.rec[ch.x];
  const Adj &A = M.adj[rec.dir];
  x.dir = rec.dir;
  x.to = rec.new_off + L.count[g];
  const uint32_t b = ch.y * LONG_CHUNK, cnt = min(rec.len - b, LONG_CHUNK);
  const u64 p = rec.old_off + b;
  // the chunk's deletion bits, a word per lane
  const uint32_t sh = (uint32_t)p & 31;
  const uint32_t bits =
      lane * 32 < sh + cnt ? *(volatile uint32_t *)(A.tbits + (p >> 5) + lane) : ~0u;
#pragma unroll
  for (uint32_t t = 0; t < LONG_PER; t++)
    if (t * 32 + lane < cnt) {
      x.v[t] = read_pair_rw(A, p + t * 32 + lane);
      C.link += 4u * A.stride;
    }
#pragma unroll
  for (uint32_t t = 0; t < LONG_PER; t++) {
    const uint32_t lo = __shfl_sync(0xffffffffu, bits, t);
    const uint32_t hi = __shfl_sync(0xffffffffu, bits, t + 1);
    const uint32_t left = cnt > t * 32 ? cnt - t * 32 : 0u;  // slots from here on
    x.live[t] = ~__funnelshift_r(lo, hi, sh) & (left >= 32 ? ~0u : (1u << left) - 1);
  }
}
// Half a chunk at a time goes through shared memory (`half`: the warp's part), so that
// the stores cover whole 128-byte lines however the live slots were scattered: a store
// per 32 slots read left the link with 50-byte writes.
constexpr uint32_t LONG_HALF = LONG_CHUNK / 2;
__device__ __forceinline__ void write_long(const MutParams &M, const LongPiece &x, uint2 *half,
                                           Counts &C) {
  const Adj &A = M.adj[x.dir];
  const uint32_t lane = lane_id();
  u64 to = x.to;
#pragma unroll
  for (uint32_t h = 0; h < 2; h++) {
    uint32_t n = 0;
#pragma unroll
    for (uint32_t t = h * (LONG_PER / 2); t < (h + 1) * (LONG_PER / 2); t++) {
      if ((x.live[t] >> lane) & 1u) half[n + __popc(x.live[t] & ((1u << lane) - 1))] = x.v[t];
      n += __popc(x.live[t]);
    }
    __syncwarp();
    for (u64 p = (to & ~31ull) + lane; p < to + n; p += 32) {
      if (p < to) continue;
      const bool c = write_slot(A, p, half[p - to].x, half[p - to].y);
      C.link += 4u * A.stride;
      if (c) C.hbm += 4u * A.stride;
    }
    __syncwarp();
    to += n;
  }
}

// Long rows by the whole grid: the live slots of every chunk are counted, a CTA per
// row turns the counts into places, and the chunks are copied, a warp each. Rows
// that move are copied as the warps come; rows that stay in steps of as many
// chunks as there are warps, all read before any is written: a live slot's place is
// never past its own, and chunks are taken in order, so what a step overwrites
// has been read, and no copy elsewhere is needed. What bounds it is the host link
// (2^20 slots are 4 MB in and up to 4 out).
__device__ Snap copy_long(const MutParams &M, uint32_t &gen, Counts &C) {
  constexpr uint32_t W = MUT_BLOCK / 32;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const uint32_t gw = warp * gridDim.x + blockIdx.x, nw = gridDim.x * W;
  const LongRows lists[2] = {long_rows(M, 0), long_rows(M, 1)};
  for (const LongRows &L : lists)
    for (uint32_t g = gw; g < L.chunks; g += nw) {
      const uint2 ch = long_chunk(L, g);
      const RelocRec rec = M.reloc.rec[ch.x];
      const uint32_t b = ch.y * LONG_CHUNK, cnt = min(rec.len - b, LONG_CHUNK);
      const uint32_t dead = dead_slots(M.adj[rec.dir], rec.old_off + b, cnt);
      if (lane == 0) L.count[g] = cnt - dead;
    }
  Snap sn = grid_sync(M.mctl, gen, 0, SEL_Q1, M.timeout_ns);
  if (!sn.ok) return sn;
  __shared__ uint32_t s_sum[W];
  for (const LongRows &L : lists)
    for (uint32_t i = blockIdx.x; i < L.rows; i += gridDim.x) {
      const uint2 lr = L.row(i);
      const uint32_t nch = (M.reloc.rec[lr.x].len + LONG_CHUNK - 1) / LONG_CHUNK;
      uint32_t before = 0;
      for (uint32_t c0 = 0; c0 < nch; c0 += MUT_BLOCK) {
        const uint32_t c = c0 + threadIdx.x, x = c < nch ? L.count[lr.y + c] : 0u;
        uint32_t sum = x;  // inclusive over the warp, then over the CTA
#pragma unroll
        for (int o = 1; o < 32; o *= 2) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= (uint32_t)o) sum += y;
        }
        __syncthreads();  // (s_sum is free again)
        if (lane == 31) s_sum[warp] = sum;
        __syncthreads();
        uint32_t all = 0;
        for (uint32_t w = 0; w < W; w++) {
          if (w == warp) sum += all;
          all += s_sum[w];
        }
        if (c < nch) L.count[lr.y + c] = before + sum - x;
        before += all;
      }
    }
  sn = grid_sync(M.mctl, gen, 0, SEL_Q1, M.timeout_ns);
  if (!sn.ok) return sn;
  __shared__ uint2 s_half[W][LONG_HALF];
  LongPiece x;
  for (uint32_t g = gw; g < lists[1].chunks; g += nw) {
    read_long(M, lists[1], g, x, C);
    write_long(M, x, s_half[warp], C);
  }
  for (uint32_t g0 = 0; g0 < lists[0].chunks; g0 += nw) {
    const bool mine = g0 + gw < lists[0].chunks;
    if (mine) read_long(M, lists[0], g0 + gw, x, C);
    sn = grid_sync(M.mctl, gen, 0, SEL_Q1, M.timeout_ns);
    if (!sn.ok) return sn;
    if (mine) write_long(M, x, s_half[warp], C);
  }
  // (every deletion bit and every slot that an insertion takes has been read)
  sn = grid_sync(M.mctl, gen, 0, SEL_Q1, M.timeout_ns);
  if (!sn.ok) return sn;
  for (const LongRows &L : lists)
    for (uint32_t i = blockIdx.x; i < L.rows; i += gridDim.x) {
      const uint2 lr = L.row(i);
      const RelocRec rec = M.reloc.rec[lr.x];
      const Adj &A = M.adj[rec.dir];
      // live slots of the sorted prefix: those of its whole chunks and the rest's
      const uint32_t srt = A.srt[rec.row], c = srt / LONG_CHUNK, part = srt % LONG_CHUNK;
      uint32_t sorted = c * LONG_CHUNK < rec.len ? L.count[lr.y + c] : A.live[rec.row];
      sorted += part - dead_slots(A, rec.old_off + srt - part, part);
      __syncthreads();  // (before any thread clears bits)
      if (rec.new_off == rec.old_off) {
        const u64 w0 = rec.old_off >> 5, w1 = (rec.old_off + rec.len - 1) >> 5;
        for (u64 w = w0 + threadIdx.x; w <= w1; w += MUT_BLOCK) {
          uint32_t b = ~0u;  // the row's bits of this word
          if (w == w0) b &= ~0u << (rec.old_off & 31);
          if (w == w1) b &= ~0u >> (31 - ((rec.old_off + rec.len - 1) & 31));
          if (b == ~0u) A.tbits[w] = 0;
          else atomicAnd(A.tbits + w, ~b);
        }
      }
      finish_row(M, rec, sorted, threadIdx.x, MUT_BLOCK);
    }
  return sn;
}

}  // namespace

__global__ void __launch_bounds__(MUT_BLOCK, 1)
    mutate_kernel(const __grid_constant__ MutParams M) {
  const uint32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const uint32_t nw = (gridDim.x * MUT_BLOCK) >> 5;
  const uint32_t nd = M.deletions ? M.hdr->nd : 0u, na = M.insertions ? M.hdr->na : 0u;
  uint32_t gen = 0;
  Counts C;
  Snap sn{true, 0, 0, 0};
  // 1. deletions, and the insertions' slots. Warps claim their tasks: a hub row's
  // scan must not hold the barrier with the rest of its warp's share behind it
  {
    // deletions per warp: one per 8-lane group while the batch is small
    const u64 all = (u64)nd * M.dirs;
    const uint32_t per = all <= (u64)nw * 4 ? 4u : all <= (u64)nw * 8 ? 8u : 16u;
    const uint32_t dt = (nd + per - 1) / per, at = (na + 31) / 32;
    const uint32_t dall = dt * M.dirs, total = dall + at * M.dirs;
    for (uint32_t t = gw; t < total;) {
      if (t < dall) {
        const uint32_t dir = t >= dt;
        delete_records(M, dir, (t - dir * dt) * per, per, nd, C);
      } else {
        const uint32_t a = t - dall, dir = a >= at;
        append_slots(M, dir, (a - dir * at) * 32 + lane_id(), na, C);
      }
      if (lane_id() == 0) t = nw + atomicAdd(&M.mctl->grab, 1u);
      t = __shfl_sync(0xffffffffu, t, 0);
    }
    sn = grid_sync(M.mctl, gen, 0, SEL_Q0, M.timeout_ns);
  }
  // 2. long suffixes
  if (sn.ok && sn.cnt) {
    const uint32_t ns = sn.cnt <= M.suffix_cap ? sn.cnt : 0u;  // (else: the error is set)
    for (uint32_t i = gw; i < ns; i += nw) suffix_chunk<COUNT>(M, i, 0, C);
    sn = grid_sync(M.mctl, gen, 0, SEL_Q0, M.timeout_ns);
    if (sn.ok) {
      for (uint32_t i = gw; i < ns; i += nw) suffix_chunk<MARK>(M, i, 0, C);
      sn = grid_sync(M.mctl, gen, 0, SEL_Q0, M.timeout_ns);
    }
    const uint32_t over = *(volatile uint32_t *)&M.mctl->a_pool;
    for (uint32_t w = 0; sn.ok && w < over; w += M.over_window) {
      const uint32_t end = min(over - w, M.over_window) + w;
      if (w) {
        for (u64 k = (u64)gw * 32 + lane_id(); k < (u64)(end - w) * OVER_SEGS; k += (u64)nw * 32)
          M.over_hist[k] = 0;
        sn = grid_sync(M.mctl, gen, 0, SEL_Q0, M.timeout_ns);
        if (!sn.ok) break;
      }
      for (uint32_t i = gw; i < ns; i += nw) suffix_chunk<HIST>(M, i, w, C);
      sn = grid_sync(M.mctl, gen, 0, SEL_Q0, M.timeout_ns);
      if (!sn.ok) break;
      for (uint32_t i = w + gw; i < end; i += nw) over_cut(M, i, w, C);
      sn = grid_sync(M.mctl, gen, 0, SEL_Q0, M.timeout_ns);
      if (!sn.ok) break;
      for (uint32_t i = gw; i < ns; i += nw) suffix_chunk<CUT>(M, i, w, C);
      sn = grid_sync(M.mctl, gen, 0, SEL_Q0, M.timeout_ns);
    }
  }
  // 3. the insertions' rows, and the ones that moved
  if (sn.ok && na) {
    const uint32_t at = (na + 31) / 32;
    for (uint32_t t = gw; t < at * M.dirs; t += nw) {
      const uint32_t dir = t >= at;
      append_rows(M, dir, (t - dir * at) * 32 + lane_id(), na, C);
    }
    sn = grid_sync(M.mctl, gen, 0, SEL_Q1, M.timeout_ns);
    if (sn.ok && !*(volatile uint32_t *)&M.ctl->err) {
      for (uint32_t i = gw; i < sn.tiles; i += nw) relocate_chunk(M, M.reloc.chunks[i], C);
      for (uint32_t i = gw; i < sn.cnt; i += nw) finish_warp(M, M.reloc.rec[i], C);
      const uint32_t wide = *(volatile uint32_t *)&M.mctl->q_count[2];
      __shared__ uint32_t sm[4 * MUT_BLOCK / 32];
      for (uint32_t i = blockIdx.x; i < wide; i += gridDim.x) {
        const RelocRec rec = M.reloc.rec[M.reloc.wide[i]];
        const Adj &A = M.adj[rec.dir];
        const uint32_t srt = A.srt[rec.row];
        const uint32_t sorted = srt - dead_slots(A, rec.old_off, srt);
        __syncthreads();  // (before any warp clears bits)
        compact_row<MUT_BLOCK>(M, rec, sm, C);
        finish_row(M, rec, sorted, threadIdx.x, MUT_BLOCK);
      }
      if (*(volatile u64 *)&M.mctl->a_head | *(volatile u64 *)&M.mctl->a_tail)
        sn = copy_long(M, gen, C);
    }
  }
  if (!sn.ok && threadIdx.x == 0) atomicCAS(&M.ctl->err, 0u, ERR_BARRIER);
  const u64 link = warp_sum(C.link), hbm = warp_sum(C.hbm), missing = warp_sum(C.missing),
            moved = warp_sum(C.moved);
  if (lane_id() == 0) {
    if (link) atomicAdd(&M.ctl->stat[ST_MUT_LINK_BYTES], link);
    if (hbm) atomicAdd(&M.ctl->stat[ST_MUT_HBM_BYTES], hbm);
    if (missing) atomicAdd(&M.ctl->stat[ST_MISSING], missing);
    if (moved) atomicAdd(&M.ctl->stat[ST_RELOCATED], moved);
  }
}

cudaError_t launch_mutate(const MutParams &M, uint32_t records, uint32_t ctas, u64 arena_bytes,
                          cudaStream_t s) {
  if (!records) return cudaSuccess;
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mutate_kernel, MUT_BLOCK, 0);
  if (e != cudaSuccess) return e;
  const uint32_t grid =
      mutation_grid(records, M.dirs, ctas, (uint32_t)sms, arena_bytes,
                    (u64)std::max(per_sm, 1) * (u64)sms);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(MUT_BLOCK);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, mutate_kernel, M);
}

}  // namespace dycg
