// internal.h -- launcher declarations shared between the kernel files and the
// host engine.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "common.cuh"

namespace dycg {

struct dycg_edge_dev {
  uint32_t u, v, w;
};

// One snapshot's records as the device sees them (written by the host ahead of
// the snapshot's kernels, so a captured snapshot serves any batch of its class).
struct BatchHdr {
  const dycg_edge_dev *dels, *adds;
  uint32_t nd, na;
  uint32_t pad[2];
};

// Entry of an ingested record list (ingest.cu): row, neighbour, weight
// (insertions) or the row's records from this one on (deletions, at run heads),
// and at the first entry of a run its length, else 0 -- equal (row, neighbour)
// for deletions, equal row for insertions. Row INF32: a record with an endpoint
// out of range (sorted last).
typedef uint4 Rec;

constexpr uint32_t PH_DELETE = 1, PH_INSERT = 2, PH_CLOSE = 4;
constexpr uint32_t PR_AMEND = 1, PR_CONVERGE = 2;

struct RepairLaunch {
  Adj out, in;
  u64 *key;
  uint32_t *mark, *wtag, *aff, *q0, *q1;
  uint4 *tiles;
  uint32_t tile_cap;
  Ctl *ctl;
  const BatchHdr *hdr;
  const Rec *dels;            // by source; del_found: occurrences removed, at run heads
  const uint32_t *del_found;
  const Rec *adds;
  uint32_t n, source, epoch, tag_base, phases, max_waves;
  uint32_t delta;  // ordered closure bucket width (0: unordered)
  uint32_t *tag_dev;  // optional device wave-tag counter (replaces tag_base)
  u64 timeout_ns;
  uint32_t algo;
  bool stored;
  int num_sms;
  uint32_t sched;     // frontier items: 0 static, 1 claimed one at a time
};
cudaError_t launch_repair(const RepairLaunch &L, cudaStream_t s);
cudaError_t launch_init_state(uint32_t algo, u64 *key, uint32_t n, uint32_t source,
                              uint32_t *q0, Ctl *ctl, cudaStream_t s);

// Batched repair of Q = 32*nb queries over one graph (multi.cu).
constexpr uint32_t MULTI_MAX_BLOCKS = 8;   // up to 256 queries
constexpr uint32_t MULTI_MIN_TILE = 1024;  // smallest tile (sizes the tile queue)
struct MultiLaunch {
  Adj out, in;
  u64 *key;                     // n * Q, vertex-major
  uint32_t *affm, *inew0, *inew1, *nmask0, *nmask1, *cmask;  // n * nb each
  uint32_t *mark, *wtag, *aff, *q0, *q1;
  uint4 *tiles;
  uint32_t tile_cap;
  Ctl *ctl;
  uint32_t *seq;                // device {epoch, next wave tag}, advanced by each launch
  const BatchHdr *hdr;
  const Rec *dels;
  const uint32_t *del_found;
  const Rec *adds;
  uint32_t n, nb, phases, max_waves;
  uint32_t qratio;              // query lanes when 4*active >= qratio*min(len,32)
  uint32_t pull_qratio;         // the same rule for the pull phase
  uint32_t heavy;               // rows with more work (warp iterations) are tiled
  uint32_t tile;                // tile size, in slots
  uint32_t sched;               // frontier-queue scheme (DYCG_QUEUE_* bits): claimed items,
                                // range-ordered wave queues, asynchronous worklist
  u64 *ring;                    // asynchronous worklist ring (ring_cap items)
  uint32_t ring_cap;
  uint32_t *inq;                // per vertex: an item waits in the ring
  uint32_t *pool;               // mask records of split heavy rows (pool_cap x nb words)
  uint32_t pool_cap;
  u64 timeout_ns;
  uint32_t algo;
  bool stored;
  int num_sms;
};
cudaError_t launch_multi(const MultiLaunch &L, cudaStream_t s);
cudaError_t launch_multi_init(u64 *key, uint32_t n, uint32_t nb, const uint32_t *sources,
                              uint32_t *nmask0, uint32_t *q0, uint32_t *wtag, const uint32_t *seq,
                              Ctl *ctl, uint32_t sched, cudaStream_t s);
// values/parents of query q out of the vertex-major (Q = 32*nb) or
// query-major (Q = 0: key already offset to the query) key array
cudaError_t launch_multi_gather(const u64 *key, uint32_t n, uint32_t Q, uint32_t q,
                                uint32_t *values, uint32_t *parents, cudaStream_t s);

struct PrLaunch {
  Adj out;
  float *x, *r, *delta;
  uint32_t *queued, *q0, *q1;
  const uint32_t *sources, *n_sources;  // touched sources
  const BatchHdr *hdr;
  const Rec *dels;                       // deleted pairs, occurrences found at run heads
  const uint32_t *del_found;
  const Rec *adds;                       // inserted occurrences
  uint4 *tiles;
  uint32_t tile_cap;
  Ctl *ctl;
  uint32_t n, cur, phases;
  float eps, alpha;
  uint32_t max_rounds;
  u64 timeout_ns;
  int num_sms;
};
cudaError_t launch_pr(const PrLaunch &L, cudaStream_t s);
cudaError_t launch_pr_init(float *x, float *r, uint32_t *queued, uint32_t *q0, uint32_t n,
                           float base, Ctl *ctl, cudaStream_t s);

// ingest (ingest.cu)
struct Lists {
  Rec *rec[4];  // deletions by source / destination, insertions by source / destination
};
// Distinct sources of the batch's valid records (tag null: not wanted), with
// their degrees before the mutation for PageRank.
struct Touch {
  uint32_t *tag;
  uint32_t epoch;
  uint32_t *list, *count;
  const uint32_t *live;
  float *old_degree;
};
constexpr uint32_t INGEST_BLOCK_MAX = 8192;  // records of a list one CTA sorts
struct IngestLaunch {
  const BatchHdr *hdr;
  Lists lists;
  uint32_t nd, na;      // records of each kind, or a replayed class's capacities
  uint32_t n;
  bool has_in, with_w;
  u64 *keys, *keys_sorted;  // device-wide form: all lists' keys and weights
  uint32_t *w, *w_sorted;
  void *temp;
  size_t temp_bytes;
  Touch touch;
  Ctl *ctl;
  uint32_t carry_q, carry;  // PageRank: carried frontier (queue, length)
};
size_t ingest_temp_bytes(uint64_t records);
cudaError_t launch_ingest(const IngestLaunch &L, uint32_t *launches, cudaStream_t s);

// mutation (mutate.cu)
// Deletions in rows with a long unsorted suffix are matched with all the row's
// records at once, SUFFIX_CHUNK slots per warp, instead of a suffix scan per
// record, whose cost grows with (records in the row) x (suffix length). It costs
// another phase (~15 us), so it pays from three records on (DEFER_RECORDS) once
// the suffix is longer than a group's two steps (DEFER_SHORT), and for any number
// of records above DEFER_SUFFIX slots (eight dependent host-link steps of a warp).
// Scanning rows up to 1024 slots per record instead took 1.90 ms of a 100K-update
// R-MAT 21 snapshot's mutation, this rule 1.14.
constexpr uint32_t DEFER_SUFFIX = 1024, DEFER_SHORT = 64, DEFER_RECORDS = 3;
constexpr uint32_t SUFFIX_CHUNK = 256;
// Chunks whose slots' records stay in HBM between the passes: one per 1024 arena
// slots, within these (16 to 64 MB). A 1M-update Zipf snapshot on R-MAT 27 has some
// 45,000 without a cache: its suffixes take 8.0 ms with 16,384 of them kept, 2.9 with
// all.
constexpr uint32_t SUFFIX_KEEP_LEAST = 16384, SUFFIX_KEEP_MOST = 65536;
// Records that want fewer occurrences than match in a suffix: segments of the suffix
// that their matches are counted by, and records counted at a time (8 MB of counts).
constexpr uint32_t OVER_SEGS = 32, OVER_WINDOW = 65536;
// Bookkeeping of rows whose block is full: new_off == old_off, compacted in place.
constexpr uint32_t RELOC_CHUNK = 1024;
struct RelocRec {
  uint32_t row, seg, len, dir;
  u64 old_off, new_off;
};
struct Reloc {
  RelocRec *rec;
  uint2 *chunks;      // of rows that move
  uint32_t *wide;     // rows that stay and take a CTA
  uint2 *longs;       // rows that the whole grid copies
  uint32_t cap, chunk_cap;
};
struct MutParams {
  Adj adj[2];                // outgoing, incoming
  uint32_t dirs;             // directions kept: 1 or 2
  bool deletions, insertions;
  const BatchHdr *hdr;
  const Rec *dels[2], *adds[2];
  uint32_t *found;           // occurrences removed per record (by source)
  uint32_t *rem[2], *matches[2];  // long suffixes: wanted and matching occurrences
  uint4 *suffix;             // chunks: first record, end record, chunk, direction | chunks << 1
  uint32_t suffix_cap;
  uint32_t *suffix_ids;      // the first suffix_keep chunks' slots, between the passes
  uint32_t suffix_keep;
  uint32_t *over_hist;       // matches per segment of over_window records at a time
  uint32_t over_window;
  Reloc reloc;
  u64 scarce[2];             // arena top from which full rows stay in their blocks if they can
  Ctl *ctl, *mctl;           // snapshot counters; this launch's barrier and queues
  u64 timeout_ns;
};
// records: the longer of the two kinds (or the class's capacity); ctas: the caller's
// limit (0: none); arena_bytes: of both directions
cudaError_t launch_mutate(const MutParams &M, uint32_t records, uint32_t ctas, u64 arena_bytes,
                          cudaStream_t s);

// cache
// Device-resident admission state: the free-slot count and the plan of the
// last maintenance round (cache.cu plan_kernel), so that ranking, eviction
// and staging run without a host round trip (inside captured graphs too).
struct CachePlan {
  uint32_t free_count;   // free cache slots: free_list[0, free_count)
  uint32_t candidates;   // last round: top-K pages not resident
  uint32_t admit, evict; // last round: pages staged / evicted
  uint32_t first_rank;   // last round: first evicted rank among the candidates
  uint32_t free_base;    // last round: free count before eviction
  uint32_t top;          // last round: free count after eviction
  uint32_t pad;
  u64 loaded, evicted;   // totals
};
struct CacheWork {
  uint32_t *hits;        // == page_hits
  float *score, *score_sorted;
  uint32_t *ids, *ids_sorted, *fa, *fe, *sa, *se, *admit;
  void *temp;
  size_t temp_bytes;
  CachePlan *plan;       // device
  CachePlan *h_plan;     // pinned host copy (read after a synchronisation)
};
struct CachePages {
  const uint32_t *h_out, *h_in;  // host arena words (device-mapped)
  uint32_t pages_out, page_shift, stride;
  uint32_t *cdst;
};
size_t cache_temp_bytes(uint32_t npages);
cudaError_t cache_rank(CacheWork &W, uint32_t npages, uint32_t K, float decay, float min_score,
                       const uint32_t *page_slot, cudaStream_t s);
// plan (refresh gate, at most cap admissions), evict, stage; admissions and
// evictions are also added to the optional device counters. cache_plan and
// cache_stage are its two halves (the staging may run on another stream,
// ordered after the plan).
cudaError_t cache_plan(CacheWork &W, uint32_t npages, uint32_t gate, uint32_t cap,
                       u64 *stat_loaded, u64 *stat_evicted, cudaStream_t s);
cudaError_t cache_stage(CacheWork &W, uint32_t npages, uint32_t *page_slot, uint32_t *free_list,
                        const CachePages &pg, cudaStream_t s);
cudaError_t cache_apply(CacheWork &W, uint32_t npages, uint32_t gate, uint32_t cap,
                        uint32_t *page_slot, uint32_t *free_list, const CachePages &pg,
                        u64 *stat_loaded, u64 *stat_evicted, cudaStream_t s);

// cache given precomputed scores (W.score, W.ids filled): sort, flags, counts
cudaError_t cache_rank_given(CacheWork &W, uint32_t npages, uint32_t K, float min_score,
                             const uint32_t *page_slot, cudaStream_t s);

// learned admission policy (policy.cu)
constexpr int POLICY_F = 8, POLICY_H = 64;
constexpr int POLICY_PARAMS = POLICY_F * POLICY_H + POLICY_H + POLICY_H * POLICY_H + POLICY_H +
                              POLICY_H + 1;
size_t mlp_grad_smem();
// Row-layout features (rows starting in each page, longest of them). With
// period = {counter, every}: only when counter % every == 0 (device values).
cudaError_t launch_page_rows(const u64 *off, const uint32_t *len, uint32_t n, uint32_t page_base,
                             uint32_t page_shift, uint32_t *rows, uint32_t *maxlen,
                             const uint32_t *period, cudaStream_t s);
cudaError_t launch_page_rows_clear(uint32_t *rows, uint32_t *maxlen, uint32_t npages,
                                   const uint32_t *period, cudaStream_t s);
cudaError_t launch_period_step(uint32_t *period, cudaStream_t s);
cudaError_t launch_page_delta(const Rec *recs, const BatchHdr *hdr, bool adds, uint32_t cap,
                              const u64 *off, uint32_t page_base, uint32_t page_shift,
                              uint32_t *delta, cudaStream_t s);
cudaError_t launch_features(const uint32_t *hits, const float *hist, const uint8_t *age,
                            const uint32_t *delta, const uint32_t *rows, const uint32_t *maxlen,
                            uint32_t npages, void *x, cudaStream_t s);
constexpr int POLICY_HORIZON = 3;  // training target: reads over this many snapshots
struct TargetRefs {
  float *t[POLICY_HORIZON];  // raw targets receiving this snapshot's reads (or null)
};
cudaError_t launch_history(uint32_t *hits, float *hist, uint8_t *age, uint32_t npages,
                           const TargetRefs &tg, bool clear, cudaStream_t s);
cudaError_t launch_log1p(const float *in, float *out, u64 n, cudaStream_t s);
// tcgen05 inference; err (optional) receives ERR_BARRIER if a tensor-core
// completion wait ran out
cudaError_t launch_mlp_infer(const void *x, uint32_t n, const float *params, float *score,
                             uint32_t *ids, uint32_t *err, cudaStream_t s);
// tcgen05 loss and gradient; err (optional) as for inference
cudaError_t launch_mlp_grad(const void *x, const float *y, uint64_t total, uint32_t count,
                            uint64_t sample_seed, const float *params, float scale, float *grad,
                            float *loss, uint32_t *err, cudaStream_t s);
cudaError_t launch_adam(float *p, float *g, float *m, float *v, float lr, uint32_t step,
                        cudaStream_t s);
cudaError_t sample_row_edges(const Adj &A, const uint32_t *sources, u64 count, u64 seed,
                             uint32_t n, uint32_t *out, cudaStream_t s);

// build
cudaError_t build_gen_rmat(u64 *keys, u64 draws, u64 seed, uint32_t scale, double a, double b,
                           double c, int symmetrize, cudaStream_t s);
cudaError_t build_gen_grid(u64 *keys, uint32_t side, u64 nshort, uint32_t radius, u64 seed,
                           cudaStream_t s);
cudaError_t build_csr_keys(const u64 *off, const uint32_t *dst, uint32_t n, u64 *keys,
                           cudaStream_t s);
cudaError_t build_swap_keys(const u64 *in, u64 *out, u64 count, cudaStream_t s);
cudaError_t build_sort(void *temp, size_t &bytes, u64 *k_in, u64 *k_out, uint32_t *v_in,
                       uint32_t *v_out, u64 count, cudaStream_t s);
cudaError_t build_scan_u32_to_u64(void *temp, size_t &bytes, const uint32_t *in, u64 *out,
                                  u64 count, cudaStream_t s);
cudaError_t build_scan_u64(void *temp, size_t &bytes, const u64 *in, u64 *out, u64 count,
                           cudaStream_t s);
cudaError_t build_unique(const u64 *k, const uint32_t *vin, u64 count, int dedup,
                         uint32_t *flag, u64 *pos, u64 *out, uint32_t *vout, void *temp,
                         size_t temp_bytes, cudaStream_t s);
cudaError_t build_degrees(const u64 *k, u64 m, uint32_t *deg, cudaStream_t s);
cudaError_t build_caps(const uint32_t *deg, uint32_t n, u64 *cap64, uint32_t *cap,
                       uint32_t *len, uint32_t *srt, uint32_t *live, cudaStream_t s);
cudaError_t build_scatter(const u64 *k, const uint32_t *wv, u64 m, const u64 *off,
                          const u64 *rowstart, uint32_t *hwords, uint32_t stride, uint32_t *fence,
                          uint32_t fence_shift, u64 wseed, uint32_t wlo, uint32_t whi,
                          int weight_from_hash, int swapped, cudaStream_t s);
size_t build_temp_bytes(u64 count, bool pairs);
cudaError_t sample_draw(u64 *pos, u64 count, u64 seed, u64 total, cudaStream_t s);
cudaError_t sample_resolve(const u64 *pos, u64 count, const u64 *pre, uint32_t n, const Adj &A,
                           uint32_t *out, cudaStream_t s);

}  // namespace dycg
