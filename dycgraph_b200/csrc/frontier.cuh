// frontier.cuh -- bounded grid barrier and the row-expansion engine shared by
// the persistent repair kernels (SSSP/BFS/CC closures and PageRank pushes).
//
// Work distribution (the B200 form of the reference's degree-aware CTA/warp
// scheduler, include/groute/device/cta_scheduler_hybrid.cuh:60-240): while a
// wave has no more rows than the launch has warps, one warp per frontier vertex
// walks its row 32 slots at a time (coalesced 128-byte reads, from the HBM page
// cache or zero-copy from the host arena); larger waves give short rows to
// 8-lane groups, four rows per warp; rows longer than HEAVY are cut into
// TILE-slot tiles that whole CTAs process after a grid barrier, so a
// million-edge hub row spreads over the whole GPU.
#pragma once
#include "common.cuh"

namespace dycg {

constexpr uint32_t SYNC_RESET_TILES = 1;
constexpr uint32_t SYNC_RESET_Q0 = 2;
constexpr uint32_t SYNC_RESET_Q1 = 4;
constexpr uint32_t SYNC_RESET_Q2 = 8;
constexpr uint32_t SYNC_RESET_VMIN = 16;
constexpr uint32_t SYNC_RESET_GRAB = 32;
constexpr uint32_t SYNC_RESET_ASYNC = 64;
constexpr uint32_t SYNC_RESET_RANGES = 128;  // with Q0 / Q1: that queue's range counts too

// What a barrier publishes to every block: one of the queue counters (SEL_*),
// the tile count and the ordered closure's minimum, as they stood when the last
// block arrived.
constexpr uint32_t SEL_Q0 = 0, SEL_Q1 = 1, SEL_Q2 = 2, SEL_AFF = 3;
struct Snap {
  bool ok;         // false: the launch has failed, leave
  uint32_t cnt, tiles, vmin;
};

__device__ __forceinline__ uint4 ld_pub(const uint32_t *p) {
  u64 a, b;  // one 128-bit access: the four words belong together
  asm volatile(
      "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\t"
      "mov.b128 {%0, %1}, t;\n\t}"
      : "=l"(a), "=l"(b)
      : "l"(p)
      : "memory");
  return make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
}
__device__ __forceinline__ void st_pub(uint32_t *p, uint4 v) {
  const u64 a = ((u64)v.y << 32) | v.x, b = ((u64)v.w << 32) | v.z;
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\t"
      "st.relaxed.gpu.global.b128 [%0], t;\n\t}"
      :
      : "l"(p), "l"(a), "l"(b)
      : "memory");
}

// Grid-wide barrier for cooperative launches; gen is the caller's barrier
// generation (0 at launch, the control block is cleared before every launch).
// What bounds it is dependent L2 round trips (~0.6 us each), so there are three:
// the arrival atomic, the last arriver's reads of the counters, and the poll
// that sees its publication -- which carries the counters the blocks need next,
// so nobody reads them again afterwards. Every wait is bounded: past timeout_ns
// the waiting block records ERR_BARRIER and all blocks leave at their next
// barrier. The last arriver applies the requested resets while every other
// block is waiting.
__device__ __forceinline__ Snap grid_sync(Ctl *c, uint32_t &gen, uint32_t flags, uint32_t sel,
                                          u64 timeout_ns) {
  constexpr uint32_t FAILED = 0x80000000u;
  __shared__ uint4 s_pub;
  __syncthreads();
  gen++;
  if (threadIdx.x == 0) {
    __threadfence();
    uint4 p;
    if (atomicAdd(&c->bar_count, 1u) + 1 == gridDim.x) {
      __threadfence();
      const uint4 q = __ldcg(reinterpret_cast<const uint4 *>(c->q_count));
      const uint4 t = __ldcg(reinterpret_cast<const uint4 *>(&c->tile_count));
      p.x = gen | (t.z ? FAILED : 0u);
      p.y = sel == SEL_Q0 ? q.x : sel == SEL_Q1 ? q.y : sel == SEL_Q2 ? q.z : q.w;
      p.z = t.x;
      p.w = ~t.y;
      // (counters that a flag resets are published as they were; a queue that
      // is reset here is never the one selected)
      if (flags & SYNC_RESET_TILES) c->tile_count = 0;
      if (flags & SYNC_RESET_Q0) c->q_count[0] = 0;
      if (flags & SYNC_RESET_Q1) c->q_count[1] = 0;
      if (flags & SYNC_RESET_Q2) c->q_count[2] = 0;
      if (flags & SYNC_RESET_RANGES) {
        const uint32_t par = (flags & SYNC_RESET_Q1) ? 1 : 0;
        for (int b = 0; b < 64; b++) c->qrange[par][b] = 0;
      }
      // the minimum is complete once no tile is left to expand
      if ((flags & SYNC_RESET_VMIN) && (t.x == 0 || (flags & SYNC_RESET_TILES))) c->vmin = 0;
      if (flags & SYNC_RESET_GRAB) c->grab = 0;
      if (flags & SYNC_RESET_ASYNC) {
        c->a_head = 0;
        c->a_tail = 0;
        c->a_pend = 0;
        c->a_pool = 0;
        c->a_tiles = 0;
      }
      c->bar_count = 0;
      __threadfence();
      st_pub(c->pub, p);
    } else {
      const u64 t0 = globaltimer_ns();
      for (uint32_t polls = 1;; polls++) {
        p = ld_pub(c->pub);
        if ((p.x & ~FAILED) == gen) break;
        if (polls % 64 == 0) {
          if (*(volatile uint32_t *)&c->err) {
            p.x = FAILED;
            break;
          }
          if (globaltimer_ns() - t0 > timeout_ns) {
            atomicCAS(&c->err, 0u, ERR_BARRIER);
            p.x = FAILED;
            break;
          }
        }
      }
    }
    __threadfence();
    s_pub = p;
  }
  __syncthreads();
  const uint4 p = s_pub;
  return Snap{!(p.x & FAILED), p.y, p.z, p.w};
}

// Per-thread traffic counters, flushed once per kernel (a thread's share of one
// launch stays far below 2^32: 100 GB over a grid's threads is under 1 MB each).
struct Acc {
  uint32_t link;
  uint32_t hbm;
  uint32_t scanned;
  uint32_t expanded;
  uint32_t improved;
  uint32_t state;  // vertex-state bytes counted by the kernel itself (batched form)
  __device__ void flush(Ctl *c) {
    u64 a = warp_sum(link), b = warp_sum(hbm), s = warp_sum(scanned), e = warp_sum(expanded),
        i = warp_sum(improved), k = warp_sum(state);
    if (lane_id() == 0) {
      if (k) atomicAdd(&c->stat[ST_STATE_BYTES], k);
      if (a) atomicAdd(&c->stat[ST_LINK_BYTES], a);
      if (b) atomicAdd(&c->stat[ST_HBM_ADJ_BYTES], b);
      if (s) atomicAdd(&c->stat[ST_SCANNED], s);
      if (e) atomicAdd(&c->stat[ST_EXPANDED], e);
      if (i) atomicAdd(&c->stat[ST_IMPROVED], i);
    }
  }
};

// One reservation for up to U entries per lane (the warp is converged): the
// ballots give every entry its place, so a lane's U appends cost one atomic
// round trip together.
template <int U>
__device__ __forceinline__ void append_batch(uint32_t *q, uint32_t *count, uint32_t cap,
                                             const bool (&want)[U], const uint32_t (&val)[U],
                                             uint32_t *err) {
  unsigned m[U];
  uint32_t total = 0;
#pragma unroll
  for (int u = 0; u < U; u++) {
    m[u] = __ballot_sync(0xffffffffu, want[u]);
    total += __popc(m[u]);
  }
  if (!total) return;
  const uint32_t lane = lane_id();
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(count, total);
  base = __shfl_sync(0xffffffffu, base, 0);
  if (base + total > cap) {
    if (lane == 0) atomicExch(err, ERR_QUEUE);
    return;
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
    if (want[u]) q[base + __popc(m[u] & ((1u << lane) - 1))] = val[u];
    base += __popc(m[u]);
  }
}

constexpr int UNROLL = 4;  // slots a lane keeps in flight

// Walk slots [b, e) of a row: the warp is cut into groups of G lanes, each with
// its own row v (on: the group has one); a group's lane takes slots
// b + lane, b + lane + stride, ... (stride >= G), UNROLL of them loaded ahead
// of their use, so that each lane keeps several zero-copy reads in flight (a
// host-link read costs ~1-2 us). Op interface (the whole warp calls every
// member, converged; a group without a row passes on = false):
//   bool begin(uint32_t v, bool on, Row&)   -- false: skip the row
//   void edges(uint32_t v, nb[UNROLL], w[UNROLL], valid[UNROLL], Row&, Acc&)
//   void end(uint32_t v, bool on, Row&)     -- on as begin returned it
template <int G, bool WITH_W, class Op>
__device__ __forceinline__ void group_slots(const Adj &A, uint32_t v, bool on, u64 off, uint32_t b,
                                            uint32_t e, uint32_t stride, Op &op, Acc &acc) {
  typename Op::Row r;
  on = op.template begin<G>(v, on, r);
  if (!__any_sync(0xffffffffu, on)) return;
  const uint32_t gl = lane_id() & (G - 1);
  const bool first = gl == 0;
  if (on && first && b == 0) acc.expanded++;
  uint32_t hit_pg = PAGE_NONE, hit_n = 0;  // group leader: pending hotness count
  const uint32_t bytes = WITH_W ? 8u : 4u;
  const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << G) - 1) << (lane_id() & ~(G - 1));
  for (uint32_t s0 = b; __any_sync(0xffffffffu, on && s0 < e); s0 += stride * UNROLL) {
    uint32_t d[UNROLL], w[UNROLL], pg[UNROLL];
    bool in[UNROLL], cached[UNROLL], ok[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      const uint32_t s = s0 + u * stride + gl;
      in[u] = on && s < e;
      d[u] = TOMB;
      w[u] = 0;
      pg[u] = PAGE_NONE;
      cached[u] = false;
      if (in[u]) {
        const u64 p = off + s;
        pg[u] = page_of(A, p);
        if (WITH_W) {
          const uint2 pr = read_pair(A, p, cached[u]);
          d[u] = pr.x;
          w[u] = pr.y;
        } else {
          d[u] = read_dst(A, p, cached[u]);
        }
        if (slot_deleted(A, p)) d[u] |= TOMB;
      }
    }
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      ok[u] = in[u] && !(d[u] & TOMB);
      d[u] &= VMASK;
      if (in[u]) {
        if (cached[u]) acc.hbm += ok[u] ? bytes : 4u;
        else acc.link += ok[u] ? bytes : 4u;
        acc.scanned++;
      }
      // hotness: the leader accumulates the group's slots that share its page
      if (!__any_sync(0xffffffffu, in[u])) continue;
      const uint32_t pg0 = __shfl_sync(0xffffffffu, pg[u], 0, G);
      const unsigned same = __ballot_sync(0xffffffffu, in[u] && pg[u] == pg0) & gmask;
      if (first && same) {
        if (pg0 != hit_pg) {
          if (hit_n) atomicAdd(A.page_hits + hit_pg, hit_n);
          hit_pg = pg0;
          hit_n = 0;
        }
        hit_n += __popc(same);
      }
      if (in[u] && pg[u] != pg0) atomicAdd(A.page_hits + pg[u], 1u);
    }
    op.edges(v, d, w, ok, r, acc);
  }
  if (first && hit_n) atomicAdd(A.page_hits + hit_pg, hit_n);
  op.template end<G>(v, on, r);
}

struct Tiles {
  uint4 *tiles;
  uint32_t cap;
};

// Rows at most this long go to 8-lane groups in waves with more rows than warps.
constexpr uint32_t GROUP_ROW = 64;

// Expand the rows of items[0..cnt) over adjacency A. op.admit(v, on) is asked
// once per item before its row is looked at (false: not now). Ends with a grid
// barrier that publishes counter `sel` and applies `reset_flags`.
// Items are taken statically or, with `claimed`, one at a time from the control
// block's claim counter (reset by the barriers that end the phase), so a warp
// that drew long rows does not hold the wave's barrier while the others idle.
// Static: warp k of every block before warp k + 1 of any, so that a short wave
// spreads over all SMs; one item per warp while the wave fits (its latency is
// one row's), up to four per warp above (short rows leave most of 32 lanes
// idle).
template <bool WITH_W, class Op>
__device__ Snap expand_rows(const Adj &A, const uint32_t *items, uint32_t cnt, Op &op, Acc &acc,
                            Tiles T, Ctl *ctl, uint32_t &gen, uint32_t sel, uint32_t reset_flags,
                            u64 timeout_ns, bool claimed = false) {
  const uint32_t lane = lane_id();
  const uint32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t per = claimed || cnt <= nw ? 1u : cnt <= 2 * nw ? 2u : 4u;
  const uint32_t grp = lane >> 3;
  uint32_t i = gw * per;
  if (claimed) {
    if (lane == 0) i = atomicAdd(&ctl->grab, 1u);
    i = __shfl_sync(0xffffffffu, i, 0);
  }
  while (i < cnt) {
    const bool have = grp < per && i + grp < cnt;
    const uint32_t v = have ? __ldcg(items + i + grp) : 0u;
    if (claimed) {
      if (lane == 0) i = atomicAdd(&ctl->grab, 1u);
      i = __shfl_sync(0xffffffffu, i, 0);
    } else {
      i += nw * per;
    }
    const uint32_t len = have ? A.len[v] : 0u;
    const u64 off = have ? A.off[v] : 0ull;
    const bool on = op.admit(v, have);
    const bool small = per > 1 && len <= GROUP_ROW;
    if (__any_sync(0xffffffffu, on && small))
      group_slots<8, WITH_W>(A, v, on && small, off, 0, len, 8, op, acc);
    // the others one after another, a whole warp each
    unsigned big = __ballot_sync(0xffffffffu, on && !small && (lane & 7) == 0);
    while (big) {
      const int src = __ffs(big) - 1;
      big &= big - 1;
      const uint32_t bv = __shfl_sync(0xffffffffu, v, src);
      const uint32_t bl = __shfl_sync(0xffffffffu, len, src);
      const u64 bo = __shfl_sync(0xffffffffu, off, src);
      if (bl > HEAVY) {
        const uint32_t nt = (bl + TILE - 1) / TILE;
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&ctl->tile_count, nt);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base + nt > T.cap) {
          if (lane == 0) atomicCAS(&ctl->err, 0u, ERR_TILES);
        } else {
          for (uint32_t t = lane; t < nt; t += 32)
            T.tiles[base + t] = make_uint4(bv, t * TILE, min(bl, (t + 1) * TILE), 0);
        }
        continue;
      }
      group_slots<32, WITH_W>(A, bv, true, bo, 0, bl, 32, op, acc);
    }
  }
  // The items have been consumed: the queue resets can apply here. When no row
  // was heavy this barrier's snapshot already holds every append of the
  // expansion and the tile phase (and its barrier) is skipped.
  Snap sn = grid_sync(ctl, gen, reset_flags | SYNC_RESET_GRAB, sel, timeout_ns);
  if (!sn.ok || sn.tiles == 0) return sn;
  const uint32_t nt = min(sn.tiles, T.cap);
  const uint32_t wib = threadIdx.x >> 5;
  __shared__ uint32_t s_tile;
  uint32_t t = blockIdx.x;
  if (claimed) {
    if (threadIdx.x == 0) s_tile = atomicAdd(&ctl->grab, 1u);
    __syncthreads();
    t = s_tile;
  }
  while (t < nt) {
    const uint4 tl = __ldcg(T.tiles + t);
    if (claimed) {
      __syncthreads();  // every warp has read s_tile
      if (threadIdx.x == 0) s_tile = atomicAdd(&ctl->grab, 1u);
      __syncthreads();
      t = s_tile;
    } else {
      t += gridDim.x;
    }
    group_slots<32, WITH_W>(A, tl.x, true, A.off[tl.x], tl.y + wib * 32, tl.z, blockDim.x, op,
                            acc);
  }
  return grid_sync(ctl, gen,
                   SYNC_RESET_TILES | SYNC_RESET_GRAB | (reset_flags & SYNC_RESET_VMIN), sel,
                   timeout_ns);
}

__device__ __forceinline__ u64 ld_key(const u64 *p) {
  return *(const volatile u64 *)p;
}

// With zero-weight edges (CC labels; stored weights may be 0) an equal value
// must not move the parent: a switch to a smaller-id parent of equal value can
// close a cycle in the parent forest, and deletion repair follows parents.
// Lower *addr to cand given a recent read `seen`; true when the value
// decreased (strict CAS form where zero weights are possible, atomicMin with
// parent tie-break otherwise).
template <bool STRICT>
__device__ __forceinline__ bool lower_from(u64 *addr, u64 cand, u64 seen) {
  if (cand >= seen) return false;
  if (STRICT) {
    u64 old = seen;
    while (key_value(cand) < key_value(old)) {
      const u64 prev = atomicCAS(addr, old, cand);
      if (prev == old) return true;
      old = prev;
    }
    return false;
  }
  return key_value(atomicMin(addr, cand)) > key_value(cand);
}

// lower_from split in two so that a lane can issue several independent
// first attempts before it looks at any result: first_lower issues the first
// atomic (false: cand cannot lower `seen`, nothing issued) and leaves its
// result in got; lowered finishes the attempt (the strict form retries from
// the value it lost to, exactly as lower_from's loop does).
template <bool STRICT>
__device__ __forceinline__ bool first_lower(u64 *addr, u64 cand, u64 seen, u64 &got) {
  if (cand >= seen) return false;
  if (STRICT) {
    if (key_value(cand) >= key_value(seen)) return false;
    got = atomicCAS(addr, seen, cand);
  } else {
    got = atomicMin(addr, cand);
  }
  return true;
}
template <bool STRICT>
__device__ __forceinline__ bool lowered(u64 *addr, u64 cand, u64 seen, u64 got) {
  if (!STRICT) return key_value(got) > key_value(cand);
  if (got == seen) return true;
  return lower_from<true>(addr, cand, got);
}

// Zero-weight edges possible: strict value decrease only.
template <uint32_t ALGO, bool STORED>
struct Strict {
  static constexpr bool value = ALGO == ALGO_CC || STORED;
};

}  // namespace dycg
