// pr.cu -- signed-residual PageRank on the paged adjacency, one persistent
// cooperative kernel per phase group.
//
// Semantics follow the reference's pr::Runtime (include/framework/pr_residual.cuh):
// unnormalised ranks x = (1-alpha) + alpha * P^T x with dangling mass dropped;
// a vertex is in the frontier while |r| > epsilon (Frontier::Add :21-30);
// Consume (:54-71) moves r into x; Scatter (:74-100) pushes
// alpha * delta / degree along every live occurrence with FP32 atomics. A
// batch changes r by what the reference's two amend passes add up to
// (Engine::UpdatePageRank, framework.cuh:2692-2736: -alpha*x[u]/deg_old(u)
// over the old row of every touched source before the topology changes,
// +alpha*x[u]/deg_new(u) over the new row after), then converges for at most
// max_rounds rounds; unfinished work carries over. The sum is pushed in one
// pass after the mutation: every live occurrence of the new row gets
// alpha*x[u]*(1/deg_new - 1/deg_old), an inserted occurrence another
// alpha*x[u]/deg_old, a deleted one -alpha*x[u]/deg_old. The residuals are
// the same sums (with one rounding instead of two per kept occurrence), but
// a row whose degree did not change pushes nothing, and a kept neighbour gets
// a push ~deg times smaller, so far fewer vertices cross epsilon only to be
// cancelled by the second pass. deg_old is saved per touched source (in the
// delta array, free between snapshots) before the mutation.
#include "frontier.cuh"
#include "internal.h"

namespace dycg {

struct PrParams {
  Adj out;
  float *x;
  float *r;
  float *delta;
  uint32_t *queued;
  uint32_t *q[2];
  const uint32_t *sources;  // touched sources (amend)
  const uint32_t *n_sources;
  const BatchHdr *hdr;
  const Rec *dels;          // deleted (u, v); occurrences found at run heads, 0 elsewhere
  const uint32_t *del_found;
  const Rec *adds;          // inserted occurrences (u >= n: invalid record)
  Tiles tiles;
  Ctl *ctl;
  uint32_t n;
  uint32_t cur;             // queue holding the frontier
  uint32_t phases;          // PR_AMEND and/or PR_CONVERGE
  float eps;
  float alpha;
  uint32_t max_rounds;
  u64 timeout_ns;
};

// Frontier::Add: enqueue on crossing epsilon.
__device__ __forceinline__ bool pr_add(const PrParams *P, uint32_t dst, float c) {
  const float old = atomicAdd(P->r + dst, c);
  const float nv = old + c;
  if (!isfinite(nv)) atomicCAS(&P->ctl->err, 0u, ERR_NONFINITE);
  return fabsf(old) <= P->eps && fabsf(nv) > P->eps && atomicCAS(P->queued + dst, 0u, 1u) == 0u;
}

// Pushes c to UNROLL targets per lane: the atomics first (independent, in
// flight together), then Frontier::Add's crossing test on each result.
__device__ __forceinline__ void push_batch(const PrParams *P, uint32_t *outq, uint32_t *outc,
                                           const uint32_t (&y)[UNROLL],
                                           const bool (&valid)[UNROLL], float c, Acc &acc) {
  float old[UNROLL];
  bool want[UNROLL];
#pragma unroll
  for (int u = 0; u < UNROLL; u++) old[u] = valid[u] ? atomicAdd(P->r + y[u], c) : 0.f;
#pragma unroll
  for (int u = 0; u < UNROLL; u++) {
    want[u] = false;
    if (valid[u]) {
      const float nv = old[u] + c;
      if (!isfinite(nv)) atomicCAS(&P->ctl->err, 0u, ERR_NONFINITE);
      want[u] = fabsf(old[u]) <= P->eps && fabsf(nv) > P->eps &&
                atomicCAS(P->queued + y[u], 0u, 1u) == 0u;
      acc.improved++;
    }
  }
  append_batch(outq, outc, P->n, want, y, &P->ctl->err);
}

// The same without looking at the results (no value comes back from L2): a
// dense round finds its frontier by a scan afterwards.
__device__ __forceinline__ void push_only(const PrParams *P, const uint32_t (&y)[UNROLL],
                                          const bool (&valid)[UNROLL], float c, Acc &acc) {
#pragma unroll
  for (int u = 0; u < UNROLL; u++)
    if (valid[u]) {
      atomicAdd(P->r + y[u], c);
      acc.improved++;
    }
}

// A round is dense when at least 1 in DENSE vertices is in its frontier: its rows
// then hold several times n occurrences, and reading every residual once costs
// less than a returned value, a crossing test and a queue append per push. A
// frontier is the vertices with |r| > eps either way (outside the frontier none
// is above it when a round begins, and a vertex that crossed and came back is
// dropped when it is consumed), so the rounds push the same values. It is worth
// little: 1.67 against 1.71 ms of an R-MAT 18 snapshot's kernel without the rule.
constexpr uint32_t DENSE = 16;

__device__ __forceinline__ uint32_t old_degree(const PrParams *P, uint32_t u) {
  return __float_as_uint(P->delta[u]);
}

// The kept-occurrence share of the amend over a touched source's new row.
struct AmendOp {
  const PrParams *P;
  uint32_t *outq;
  uint32_t *outc;
  struct Row {
    float c;
  };
  __device__ bool admit(uint32_t, bool on) { return on; }
  template <int G>
  __device__ bool begin(uint32_t u, bool on, Row &row) {
    row.c = 0.f;
    if (!on) return false;
    const uint32_t dn = P->out.live[u], dold = old_degree(P, u);
    const float xu = P->x[u];
    if (!dn || dn == dold || xu == 0.f) return false;
    // alpha x (1/dn - 1/dold) = alpha x (dold - dn) / (dn dold), or alpha x / dn
    row.c = dold ? P->alpha * xu * ((float)((int64_t)dold - (int64_t)dn) /
                                    ((float)dn * (float)dold))
                 : P->alpha * xu / (float)dn;
    return row.c != 0.f;
  }
  __device__ void edges(uint32_t, const uint32_t (&y)[UNROLL], const uint32_t (&)[UNROLL],
                        const bool (&valid)[UNROLL], Row &row, Acc &acc) {
    push_batch(P, outq, outc, y, valid, row.c, acc);
  }
  template <int G>
  __device__ void end(uint32_t, bool, Row &) {}
};

struct ScatterOp {
  const PrParams *P;
  uint32_t *outq;
  uint32_t *outc;
  bool dense;
  struct Row {
    float c;
  };
  __device__ bool admit(uint32_t, bool on) { return on; }
  template <int G>
  __device__ bool begin(uint32_t v, bool on, Row &row) {
    row.c = 0.f;
    if (!on) return false;
    const float d = P->delta[v];
    const uint32_t deg = P->out.live[v];
    if (d == 0.f || !deg) return false;
    row.c = P->alpha * d / (float)deg;
    return true;
  }
  __device__ void edges(uint32_t, const uint32_t (&y)[UNROLL], const uint32_t (&)[UNROLL],
                        const bool (&valid)[UNROLL], Row &row, Acc &acc) {
    if (dense) push_only(P, y, valid, row.c, acc);
    else push_batch(P, outq, outc, y, valid, row.c, acc);
  }
  template <int G>
  __device__ void end(uint32_t, bool, Row &) {}
};

// The per-occurrence shares of the amend: -alpha x[u]/deg_old for each
// deleted occurrence, +alpha x[u]/deg_old for each inserted one (together with
// the row pass that makes it alpha x[u]/deg_new). Appends into q[cur].
__device__ void amend_records(const PrParams &P, uint32_t cur, Acc &acc) {
  const uint32_t lane = lane_id();
  const uint32_t first = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32;
  const uint32_t step = gridDim.x * blockDim.x;
  uint32_t *q = P.q[cur], *qc = &P.ctl->q_count[cur];
  const uint32_t nd = P.hdr->nd, na = P.hdr->na;
  for (int adds = 0; adds < 2; adds++) {
    const uint32_t cnt = adds ? na : nd;
    const Rec *list = adds ? P.adds : P.dels;
    for (uint32_t i0 = first; i0 < cnt; i0 += step) {  // warp-uniform
      const uint32_t i = i0 + lane;
      const Rec e = i < cnt ? list[i] : make_uint4(INF32, INF32, 0, 0);
      bool want[1] = {false};
      const uint32_t v[1] = {e.y};
      // (a record has both endpoints in range or neither)
      const uint32_t f = e.x >= P.n ? 0u : adds ? 1u : P.del_found[i];
      if (f) {
        const uint32_t dold = old_degree(&P, e.x);
        const float xu = P.x[e.x];
        if (dold && xu != 0.f) {
          const float c = adds ? P.alpha * xu / (float)dold
                               : -P.alpha * xu * (float)f / (float)dold;
          want[0] = pr_add(&P, e.y, c);
          acc.improved++;
        }
      }
      append_batch(q, qc, P.n, want, v, &P.ctl->err);
    }
  }
}

// Frontier of a dense round: the vertices above epsilon, in vertex order (so
// that the next round's rows are read in arena order), four per lane and append.
__device__ void collect(const PrParams &P, uint32_t next) {
  const uint32_t lane = lane_id();
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  for (u64 v0 = (u64)gw * 32 * UNROLL; v0 < P.n; v0 += (u64)warps * 32 * UNROLL) {
    float rv[UNROLL];
    uint32_t v[UNROLL];
    bool want[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      v[u] = (uint32_t)v0 + u * 32 + lane;
      rv[u] = v[u] < P.n ? __ldcg(P.r + v[u]) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      if (!isfinite(rv[u])) atomicCAS(&P.ctl->err, 0u, ERR_NONFINITE);
      want[u] = fabsf(rv[u]) > P.eps;
      if (want[u]) P.queued[v[u]] = 1;
    }
    append_batch(P.q[next], &P.ctl->q_count[next], P.n, want, v, &P.ctl->err);
  }
}

__global__ void __launch_bounds__(BLOCK) pr_kernel(const __grid_constant__ PrParams P) {
  Ctl *ctl = P.ctl;
  Acc acc = {0, 0, 0, 0, 0};
  const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t gstride = gridDim.x * blockDim.x;
  uint32_t cur = P.cur, gen = 0;
  Snap sn;
  if (P.phases & PR_AMEND) {
    amend_records(P, cur, acc);
    AmendOp op{&P, P.q[cur], &ctl->q_count[cur]};
    sn = expand_rows<false>(P.out, P.sources, *P.n_sources, op, acc, P.tiles, ctl, gen,
                            cur ? SEL_Q1 : SEL_Q0, 0, P.timeout_ns);
  } else {
    sn = grid_sync(ctl, gen, 0, cur ? SEL_Q1 : SEL_Q0, P.timeout_ns);
  }
  if (!sn.ok) goto done;
  if (P.phases & PR_CONVERGE) {
    for (uint32_t round = 0; round < P.max_rounds; round++) {
      const uint32_t cnt = sn.cnt;
      if (cnt == 0) break;
      // Consume
      for (uint32_t i = gtid; i < cnt; i += gstride) {
        const uint32_t v = P.q[cur][i];
        const float rv = P.r[v];
        P.queued[v] = 0;
        if (!isfinite(rv) || !isfinite(P.x[v])) atomicCAS(&ctl->err, 0u, ERR_NONFINITE);
        if (fabsf(rv) > P.eps) {
          P.x[v] += rv;
          P.r[v] = 0.f;
          P.delta[v] = rv;
        } else {
          P.delta[v] = 0.f;
        }
      }
      sn = grid_sync(ctl, gen, cur ? SYNC_RESET_Q0 : SYNC_RESET_Q1, cur ? SEL_Q1 : SEL_Q0,
                     P.timeout_ns);
      if (!sn.ok) goto done;
      // Scatter
      const bool dense = (u64)cnt * DENSE >= P.n;
      ScatterOp op{&P, P.q[cur ^ 1], &ctl->q_count[cur ^ 1], dense};
      sn = expand_rows<false>(P.out, P.q[cur], cnt, op, acc, P.tiles, ctl, gen,
                              cur ? SEL_Q0 : SEL_Q1, cur ? SYNC_RESET_Q1 : SYNC_RESET_Q0,
                              P.timeout_ns);
      if (!sn.ok) goto done;
      if (dense) {
        collect(P, cur ^ 1);
        sn = grid_sync(ctl, gen, 0, cur ? SEL_Q0 : SEL_Q1, P.timeout_ns);
        if (!sn.ok) goto done;
      }
      cur ^= 1;
      if (gtid == 0) ctl->waves = round + 1;
    }
  }
done:
  acc.flush(ctl);
  if (gtid == 0) {
    ctl->pad[0] = cur;
    ctl->pad[1] = *(volatile uint32_t *)&ctl->q_count[cur];
  }
}

__global__ void pr_init_kernel(float *x, float *r, uint32_t *queued, uint32_t *q0, uint32_t n,
                               float base, Ctl *ctl) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += gridDim.x * blockDim.x) {
    x[v] = 0.f;
    r[v] = base;
    queued[v] = 1;
    q0[v] = v;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->q_count[0] = n;
}

cudaError_t launch_pr(const PrLaunch &L, cudaStream_t s) {
  PrParams P;
  P.out = L.out;
  P.x = L.x;
  P.r = L.r;
  P.delta = L.delta;
  P.queued = L.queued;
  P.q[0] = L.q0;
  P.q[1] = L.q1;
  P.sources = L.sources;
  P.n_sources = L.n_sources;
  P.hdr = L.hdr;
  P.dels = L.dels;
  P.del_found = L.del_found;
  P.adds = L.adds;
  P.tiles = Tiles{L.tiles, L.tile_cap};
  P.ctl = L.ctl;
  P.n = L.n;
  P.cur = L.cur;
  P.phases = L.phases;
  P.eps = L.eps;
  P.alpha = L.alpha;
  P.max_rounds = L.max_rounds;
  P.timeout_ns = L.timeout_ns;
  static int blocks_per_sm = -1;
  if (blocks_per_sm < 0) {
    cudaError_t e =
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, pr_kernel, BLOCK, 0);
    if (e != cudaSuccess) return e;
  }
  void *args[] = {&P};
  return cudaLaunchCooperativeKernel((const void *)pr_kernel, blocks_per_sm * L.num_sms, BLOCK,
                                     args, 0, s);
}

cudaError_t launch_pr_init(float *x, float *r, uint32_t *queued, uint32_t *q0, uint32_t n,
                           float base, Ctl *ctl, cudaStream_t s) {
  const int grid = (int)std::min<u64>((n + BLOCK - 1) / BLOCK + 1, 148ull * 16);
  pr_init_kernel<<<grid, BLOCK, 0, s>>>(x, r, queued, q0, n, base, ctl);
  return cudaGetLastError();
}

}  // namespace dycg
