// repair.cu -- one persistent cooperative kernel repairs SSSP / BFS / CC after
// a snapshot, after the topology mutation kernels have run.
//
// Phases (each ends at a bounded grid barrier):
//   1. deletion seeds: for every deleted (u,v) that removed an occurrence and
//      where u is v's parent, v is affected (reset_del_edges,
//      include/framework/variants/driver.cuh:401-441, IsDeletionDependency
//      api.cuh:42-49; with parents always tight the rule reduces to parent==u).
//      Whoever marks a vertex affected resets its state (reset_affected_values,
//      driver.cuh:448-463).
//   2. invalidation waves: children y of affected x (parent(y)==x) become
//      affected (PushFunctorDB_Del, push_functor.h:1180-1213), over out-rows.
//   3. pull: each affected v takes min over live in-edges of
//      (value(x)+w, parent x) (GpuAffectedPullRelax, framework.cuh:189-263;
//      equal values break toward the smaller parent) and enters the frontier
//      when it has a value; insertion seeds (SeedAddedEdgeFrontier,
//      framework.cuh:297-370).
//   4. closure waves: push relaxation until the frontier is empty
//      (RunExactGpuClosure, framework.cuh:504-616, AccumulateBuffer
//      samples/hybrid_sssp/hybrid_sssp.cu:125-145).
// The reference drives phases 2 and 3 from the host with one synchronisation
// per level/iteration; here the whole repair is a single launch. What bounds it
// on small and ordinary snapshots is latency: the grid barriers and each wave's
// chain of dependent accesses, so phases are merged where their order does not
// matter and a lane's independent accesses are issued together.
#include "frontier.cuh"
#include "internal.h"

namespace dycg {

constexpr int REPAIR_BLOCK = 1024;

struct RepairParams {
  Adj out, in;
  u64 *key;
  uint32_t *mark;
  uint32_t *wtag;
  uint32_t *aff;
  uint32_t *q[2];
  Tiles tiles;
  Ctl *ctl;
  const BatchHdr *hdr;
  const Rec *dels;          // deleted (u,v); del_found: occurrences removed
  const uint32_t *del_found;
  const Rec *adds;          // insertions (u,v,w)
  uint32_t n;
  uint32_t source;
  uint32_t epoch;
  uint32_t tag_base;
  uint32_t phases;
  uint32_t max_waves;
  uint32_t delta;           // ordered closure: expand values < wave min + delta (0: unordered)
  uint32_t *tag_dev;        // non-null: wave tags start at *tag_dev, which the
                            // launch advances past the tags it used
  u64 timeout_ns;
  bool claimed;             // waves' items claimed one at a time (else static)
};

template <uint32_t ALGO>
__device__ __forceinline__ u64 reset_key(uint32_t v) {
  return ALGO == ALGO_CC ? pack_key(v, 0) : KEY_INF;
}

// Children of an affected vertex become affected; whoever marks one resets its
// key at once (nobody needs its old parent any more: an affected vertex enters
// the list once), so no pass over the affected list is spent on that.
template <uint32_t ALGO>
struct InvalidateOp {
  const RepairParams *P;
  struct Row {};
  __device__ bool admit(uint32_t, bool on) { return on; }
  template <int G>
  __device__ bool begin(uint32_t, bool on, Row &) { return on; }
  __device__ void edges(uint32_t x, const uint32_t (&y)[UNROLL], const uint32_t (&)[UNROLL],
                        const bool (&valid)[UNROLL], Row &, Acc &) {
    u64 k[UNROLL];
    uint32_t old[UNROLL];
    bool want[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) k[u] = valid[u] ? ld_key(P->key + y[u]) : 0;
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      want[u] = valid[u] && !(ALGO != ALGO_CC && y[u] == P->source) && key_parent1(k[u]) == x + 1u;
      if (want[u]) old[u] = atomicExch(P->mark + y[u], P->epoch);
    }
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      want[u] = want[u] && old[u] != P->epoch;
      if (want[u]) P->key[y[u]] = reset_key<ALGO>(y[u]);
    }
    append_batch(P->aff, &P->ctl->n_aff, P->n, want, y, &P->ctl->err);
  }
  template <int G>
  __device__ void end(uint32_t, bool, Row &) {}
};

// Ordered closure: ctl->vmin holds the complement of the next wave's minimum
// (so that a cleared control block means "none yet").
__device__ __forceinline__ void note_min(Ctl *ctl, uint32_t value) {
  value = __reduce_min_sync(0xffffffffu, value);
  if (lane_id() == 0 && value != INF32) atomicMax(&ctl->vmin, ~value);
}

// Affected v pulls the best candidate over its live in-edges and enters the
// closure's first frontier when it has a value (a CC vertex always has its own
// id). A vertex lowered later, by an insertion seed of the same phase, enters
// it through that seed.
template <uint32_t ALGO, bool STORED, bool ORDERED>
struct PullOp {
  const RepairParams *P;
  uint32_t tag;
  struct Row {
    u64 best;
  };
  __device__ bool admit(uint32_t, bool on) { return on; }
  template <int G>
  __device__ bool begin(uint32_t, bool on, Row &r) {
    r.best = KEY_INF;
    return on;
  }
  __device__ void edges(uint32_t v, const uint32_t (&x)[UNROLL], const uint32_t (&w)[UNROLL],
                        const bool (&valid)[UNROLL], Row &r, Acc &) {
    u64 k[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) k[u] = valid[u] ? ld_key(P->key + x[u]) : KEY_INF;
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      const uint32_t vx = key_value(k[u]);
      if (vx == INF32) continue;
      const u64 c = (u64)vx + (STORED ? w[u] : rule_weight<ALGO>(x[u], v));
      if (c >= INF32) continue;
      const u64 cand = pack_key((uint32_t)c, x[u] + 1u);
      r.best = cand < r.best ? cand : r.best;
    }
  }
  template <int G>
  __device__ void end(uint32_t v, bool on, Row &r) {
    u64 m = r.best;
    if (G == 32) {
      m = warp_min_all(m);
    } else {
#pragma unroll
      for (int o = G / 2; o; o >>= 1) {
        const u64 x = __shfl_xor_sync(0xffffffffu, m, o);
        m = x < m ? x : m;
      }
    }
    bool want[1] = {on && (lane_id() & (G - 1)) == 0 && (ALGO == ALGO_CC || m != KEY_INF)};
    const uint32_t val[1] = {v};
    if (want[0]) {
      if (m != KEY_INF) lower_from<Strict<ALGO, STORED>::value>(P->key + v, m, ld_key(P->key + v));
      want[0] = atomicExch(P->wtag + v, tag) != tag;
    }
    if (ORDERED)
      note_min(P->ctl, want[0] ? min(key_value(m), ALGO == ALGO_CC ? v : INF32) : INF32);
    append_batch(P->q[0], &P->ctl->q_count[0], P->n, want, val, &P->ctl->err);
  }
};

// Push relaxation of the out-edges of a frontier vertex. In the ordered
// closure only vertices below thr are expanded: the others are
// carried to the next queue, and every carried value and improvement lowers
// the next wave's minimum.
template <uint32_t ALGO, bool STORED, bool ORDERED>
struct RelaxOp {
  const RepairParams *P;
  uint32_t *outq;
  uint32_t *outc;
  uint32_t tag;
  uint32_t thr;
  static constexpr bool STRICT = Strict<ALGO, STORED>::value;
  struct Row {
    uint32_t dv, imp;  // the vertex's value; the lowest value this lane pushed
  };
  __device__ bool admit(uint32_t v, bool on) { return ORDERED ? below<8>(v, on) : on; }
  // groups of G lanes hold the same item
  template <int G>
  __device__ bool below(uint32_t v, bool on) {
    const bool lead = (lane_id() & (G - 1)) == 0;
    const uint32_t d = on ? key_value(ld_key(P->key + v)) : INF32;
    // one read decides for the whole group
    const uint32_t dv = G == 1 ? d : __shfl_sync(0xffffffffu, d, 0, G);
    const bool later = on && dv != INF32 && dv >= thr;
    if (__any_sync(0xffffffffu, later)) {
      const uint32_t val[1] = {v};
      const bool want[1] = {later && lead && atomicExch(P->wtag + v, tag) != tag};
      append_batch(outq, outc, P->n, want, val, &P->ctl->err);
      note_min(P->ctl, later ? dv : INF32);
    }
    return on && dv < thr;
  }
  template <int G>
  __device__ bool begin(uint32_t x, bool on, Row &r) {
    // one read, broadcast: the key may change under concurrent relaxations
    r.dv = __shfl_sync(0xffffffffu, on ? key_value(ld_key(P->key + x)) : INF32, 0, G);
    r.imp = INF32;
    return r.dv != INF32;
  }
  __device__ void edges(uint32_t x, const uint32_t (&y)[UNROLL], const uint32_t (&w)[UNROLL],
                        const bool (&valid)[UNROLL], Row &r, Acc &acc) {
    // a lane's four keys, then its four first attempts, then its four tags:
    // each set of independent accesses in flight together
    u64 cand[UNROLL], cur[UNROLL], got[UNROLL];
    bool want[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      const u64 c = (u64)r.dv + (STORED ? w[u] : rule_weight<ALGO>(x, y[u]));
      cand[u] = valid[u] && c < INF32 ? pack_key((uint32_t)c, x + 1u) : KEY_INF;
      cur[u] = cand[u] != KEY_INF ? ld_key(P->key + y[u]) : 0;
    }
#pragma unroll
    for (int u = 0; u < UNROLL; u++)
      want[u] = first_lower<STRICT>(P->key + y[u], cand[u], cur[u], got[u]);
    uint32_t old[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      want[u] = want[u] && lowered<STRICT>(P->key + y[u], cand[u], cur[u], got[u]);
      if (want[u]) {
        acc.improved++;
        r.imp = min(r.imp, key_value(cand[u]));
        old[u] = atomicExch(P->wtag + y[u], tag);
      }
    }
#pragma unroll
    for (int u = 0; u < UNROLL; u++) want[u] = want[u] && old[u] != tag;
    append_batch(outq, outc, P->n, want, y, &P->ctl->err);
  }
  template <int G>
  __device__ void end(uint32_t, bool, Row &r) {
    if (ORDERED) note_min(P->ctl, r.imp);
  }
};

// 1024-thread CTAs, one per SM: the same warps in flight as four CTAs of 256,
// and a quarter of the arrivals at every grid barrier (512 and 768 threads: the
// same on short waves, 3-9% slower on 100K-update snapshots). Measured with the
// merged phases and the batched accesses, kernel time per snapshot before ->
// now: R-MAT 16 SSSP 2K updates 0.24 -> 0.14 ms, R-MAT 20 BFS 10K 0.24 -> 0.12
// ms, R-MAT 21 SSSP 100K 0.73 -> 0.36 ms, 1024^2 grid SSSP 1K (1,580 ordered
// waves) 39.4 -> 20.2 ms. 1024 threads leave 64 registers each: CC and
// stored-weight SSSP spill 172 and 164 bytes a thread, BFS and rule-weight SSSP 48
// and 44 (ordered: 188 and 196, 80).
template <uint32_t ALGO, bool STORED, bool ORDERED>
__global__ void __launch_bounds__(REPAIR_BLOCK, 1)
    repair_kernel(const __grid_constant__ RepairParams P) {
  Ctl *ctl = P.ctl;
  Acc acc = {0, 0, 0, 0, 0};
  const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t gstride = gridDim.x * blockDim.x;
  const uint32_t lane = lane_id();
  const uint32_t tag_base = P.tag_dev ? *(volatile uint32_t *)P.tag_dev : P.tag_base;
  // short record lists: warp k of every block before warp k + 1 of any
  const uint32_t first = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32;
  uint32_t gen = 0, na = 0, cur = 0;
  Snap sn;
  if (gtid == 0) ctl->stat[ST_T_START] = globaltimer_ns();

  if (P.phases & PH_DELETE) {
    // 1. deletion seeds (warp-uniform loop so appends can aggregate)
    const uint32_t n_del = P.hdr->nd;
    for (uint32_t i0 = first; i0 < n_del; i0 += gstride) {
      const uint32_t i = i0 + lane;
      bool want[1] = {false};
      uint32_t v[1] = {0};
      if (i < n_del && P.del_found[i] != 0) {
        const Rec e = P.dels[i];
        v[0] = e.y;
        if (!(ALGO != ALGO_CC && e.y == P.source) &&
            key_parent1(ld_key(P.key + e.y)) == e.x + 1u) {
          want[0] = atomicExch(P.mark + e.y, P.epoch) != P.epoch;
          if (want[0]) P.key[e.y] = reset_key<ALGO>(e.y);
        }
      }
      append_batch(P.aff, &ctl->n_aff, P.n, want, v, &ctl->err);
    }
    sn = grid_sync(ctl, gen, 0, SEL_AFF, P.timeout_ns);
    // 2. invalidation waves over the growing affected list
    while (sn.ok && sn.cnt != na) {
      InvalidateOp<ALGO> op{&P};
      const uint32_t lo = na;
      na = sn.cnt;
      sn = expand_rows<false>(P.out, P.aff + lo, na - lo, op, acc, P.tiles, ctl, gen, SEL_AFF, 0,
                              P.timeout_ns, P.claimed);
    }
    if (!sn.ok) goto done;
    if (gtid == 0) ctl->tphase[0] = globaltimer_ns();  // seeds + invalidation done
  }
  // 3. insertion seeds and the pull over the affected vertices' in-rows, one
  // phase: whatever either reads is an upper bound of a live path, and every
  // vertex either lowers enters the first frontier
  if (P.phases & PH_INSERT) {
    const uint32_t n_add = P.hdr->na;
    for (uint32_t i0 = first; i0 < n_add; i0 += gstride) {
      const uint32_t i = i0 + lane;
      bool want[1] = {false};
      uint32_t v[1] = {0}, imp = INF32;
      const Rec e = i < n_add ? P.adds[i] : make_uint4(INF32, INF32, 0, 0);
      if (e.x < P.n) {
        v[0] = e.y;
        const uint32_t du = key_value(ld_key(P.key + e.x));
        if (du != INF32) {
          const u64 c = (u64)du + (STORED ? e.z : rule_weight<ALGO>(e.x, e.y));
          if (c < INF32 &&
              lower_from<Strict<ALGO, STORED>::value>(
                  P.key + e.y, pack_key((uint32_t)c, e.x + 1u), ld_key(P.key + e.y))) {
            want[0] = atomicExch(P.wtag + e.y, tag_base) != tag_base;
            imp = (uint32_t)c;
          }
        }
      }
      if (ORDERED) note_min(ctl, imp);
      append_batch(P.q[0], &ctl->q_count[0], P.n, want, v, &ctl->err);
    }
    // the seeds' share of the phase: until the first warp, which has as many as any,
    // is through with its own
    if (gtid == 0) ctl->tphase[1] = globaltimer_ns();
  }
  if (ORDERED && !(P.phases & (PH_DELETE | PH_INSERT))) {
    // static solve: the minimum of the frontier it was given
    const uint32_t cnt = *(volatile uint32_t *)&ctl->q_count[0];
    for (uint32_t i0 = first; i0 < cnt; i0 += gstride)
      note_min(ctl, i0 + lane < cnt ? key_value(ld_key(P.key + P.q[0][i0 + lane])) : INF32);
  }
  if (na) {
    PullOp<ALGO, STORED, ORDERED> op{&P, tag_base};
    sn = expand_rows<STORED>(P.in, P.aff, na, op, acc, P.tiles, ctl, gen, SEL_Q0, SYNC_RESET_VMIN,
                             P.timeout_ns, P.claimed);
  } else {
    sn = grid_sync(ctl, gen, SYNC_RESET_VMIN, SEL_Q0, P.timeout_ns);
  }
  if (!sn.ok) goto done;
  if (gtid == 0) ctl->tphase[2] = globaltimer_ns();  // pull done
  // 4. closure waves. Ordered (P.delta > 0, for high-diameter graphs, the B200 form
  // of the reference's ordered insertion schedule, framework.cuh:537-556): each
  // wave expands only the frontier vertices whose value is below the wave's
  // minimum + delta and carries the rest to the next wave, so a vertex is
  // expanded about once instead of once per improvement. One pass and one
  // barrier per wave: the expanding warps themselves carry what is above the
  // threshold, an item per warp (or group), so that the wave's rows spread over
  // all warps whatever their place in the queue, and the next wave's minimum is
  // kept on the fly and published by the closing barrier. From an item per thread on
  // the carrying is a pass and a barrier of its own: CC on the 4096^2 grid, some ten
  // million items in ~800 waves, took 3.0 ms a wave when asked four at a time per warp
  // (2,422-3,219 ms of repair a snapshot), and takes 0.5 so (the label order, and with
  // it the number of waves, varies from run to run). SSSP there: 338 ms, 331 so.
  if (P.phases & PH_CLOSE) {
    for (uint32_t wave = 0; sn.cnt; wave++) {
      if (wave >= P.max_waves) {
        if (gtid == 0) atomicCAS(&ctl->err, 0u, ERR_WAVES);
        break;
      }
      const uint32_t thr = sn.vmin > INF32 - P.delta ? INF32 : sn.vmin + P.delta;
      RelaxOp<ALGO, STORED, ORDERED> op{&P, P.q[cur ^ 1], &ctl->q_count[cur ^ 1],
                                        tag_base + 1 + wave, thr};
      const uint32_t *items = P.q[cur];
      uint32_t cnt = sn.cnt;
      if (ORDERED && cnt >= gstride) {
        // a long queue, of which most is only carried: a lane asks for each item, and
        // what is left (in the affected list, which the pull has read) is expanded
        for (uint32_t i0 = first; i0 < cnt; i0 += gstride) {
          const uint32_t i = i0 + lane;
          const uint32_t v[1] = {i < cnt ? __ldcg(items + i) : 0u};
          const bool want[1] = {op.template below<1>(v[0], i < cnt)};
          append_batch(P.aff, &ctl->q_count[2], P.n, want, v, &ctl->err);
        }
        sn = grid_sync(ctl, gen, 0, SEL_Q2, P.timeout_ns);
        if (!sn.ok) goto done;
        items = P.aff;
        cnt = sn.cnt;
      }
      sn = expand_rows<STORED>(P.out, items, cnt, op, acc, P.tiles, ctl, gen,
                               cur ? SEL_Q0 : SEL_Q1,
                               (cur ? SYNC_RESET_Q1 : SYNC_RESET_Q0) | SYNC_RESET_VMIN |
                                   (ORDERED ? SYNC_RESET_Q2 : 0u),
                               P.timeout_ns, P.claimed);
      if (!sn.ok) goto done;
      if (gtid == 0) ctl->waves = wave + 1;
      cur ^= 1;
    }
  }
  if (gtid == 0) ctl->tphase[3] = globaltimer_ns();  // closure done
done:
  acc.flush(ctl);
  if (gtid == 0) {
    atomicAdd(&ctl->stat[ST_AFFECTED], (u64) * (volatile uint32_t *)&ctl->n_aff);
    // every block read *tag_dev before the first barrier
    if (P.tag_dev) *P.tag_dev = tag_base + ctl->waves + 2;
  }
}

// Static solve set-up: every key reset, the initial frontier in q[0].
template <uint32_t ALGO>
__global__ void init_state_kernel(u64 *key, uint32_t n, uint32_t source, uint32_t *q0,
                                  Ctl *ctl) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += gridDim.x * blockDim.x) {
    if (ALGO == ALGO_CC) {
      key[v] = pack_key(v, 0);
      q0[v] = v;
    } else {
      key[v] = v == source ? pack_key(0, 0) : KEY_INF;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (ALGO == ALGO_CC) {
      ctl->q_count[0] = n;
    } else if (source < n) {
      q0[0] = source;
      ctl->q_count[0] = 1;
    }
  }
}

template <uint32_t ALGO, bool STORED, bool ORDERED>
static cudaError_t launch_one(const RepairLaunch &L, cudaStream_t s) {
  RepairParams P;
  P.out = L.out;
  P.in = L.in;
  P.key = L.key;
  P.mark = L.mark;
  P.wtag = L.wtag;
  P.aff = L.aff;
  P.q[0] = L.q0;
  P.q[1] = L.q1;
  P.tiles = Tiles{L.tiles, L.tile_cap};
  P.ctl = L.ctl;
  P.hdr = L.hdr;
  P.dels = L.dels;
  P.del_found = L.del_found;
  P.adds = L.adds;
  P.n = L.n;
  P.source = L.source;
  P.epoch = L.epoch;
  P.tag_base = L.tag_base;
  P.phases = L.phases;
  P.max_waves = L.max_waves;
  P.delta = L.delta;
  P.tag_dev = L.tag_dev;
  P.timeout_ns = L.timeout_ns;
  P.claimed = L.sched != 0;
  static int blocks_per_sm = -1;
  if (blocks_per_sm < 0) {
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &blocks_per_sm, repair_kernel<ALGO, STORED, ORDERED>, REPAIR_BLOCK, 0);
    if (e != cudaSuccess) return e;
  }
  const int grid = blocks_per_sm * L.num_sms;
  void *args[] = {&P};
  return cudaLaunchCooperativeKernel((const void *)repair_kernel<ALGO, STORED, ORDERED>, grid,
                                     REPAIR_BLOCK, args, 0, s);
}

// Kernels of their own for the two closures: what only the ordered one needs costs the
// other no registers.
template <uint32_t ALGO, bool STORED>
static cudaError_t launch_closure(const RepairLaunch &L, cudaStream_t s) {
  return L.delta ? launch_one<ALGO, STORED, true>(L, s) : launch_one<ALGO, STORED, false>(L, s);
}

cudaError_t launch_repair(const RepairLaunch &L, cudaStream_t s) {
  switch (L.algo) {
    case ALGO_SSSP:
      return L.stored ? launch_closure<ALGO_SSSP, true>(L, s)
                      : launch_closure<ALGO_SSSP, false>(L, s);
    case ALGO_BFS:
      return launch_closure<ALGO_BFS, false>(L, s);
    case ALGO_CC:
      return launch_closure<ALGO_CC, false>(L, s);
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t launch_init_state(uint32_t algo, u64 *key, uint32_t n, uint32_t source,
                              uint32_t *q0, Ctl *ctl, cudaStream_t s) {
  const int grid = (int)std::min<u64>((n + BLOCK - 1) / BLOCK + 1, 148ull * 16);
  if (algo == ALGO_CC)
    init_state_kernel<ALGO_CC><<<grid, BLOCK, 0, s>>>(key, n, source, q0, ctl);
  else
    init_state_kernel<ALGO_SSSP><<<grid, BLOCK, 0, s>>>(key, n, source, q0, ctl);
  return cudaGetLastError();
}

}  // namespace dycg
