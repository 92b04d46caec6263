// ingest.cu -- GPU ingest of an update batch.
//
// Replaces the reference's CPU GroupedUpdateBatch
// (include/framework/effective_update_batch.h:36-207): the batch's records
// become up to four lists (deletions and insertions, by source and, where an
// incoming adjacency is kept, by destination), each sorted by (row, neighbour)
// with equal records in arrival order. A record list keeps one entry per
// update (Rec: row, neighbour, weight or the row's records, run); the entry that
// opens a run carries the run's length -- equal (u, v) for deletions (its
// multiplicity), equal row for insertions (the row's segment) -- and the others
// carry 0, so nothing is compacted and every consumer works on positions.
//
// Two forms, by the records of the longer kind:
//   up to 8192   one launch, a CTA per list: keys, block radix sort, runs, all in
//                shared memory. What bounds ordinary batches is not the 12 bytes
//                per record but launches and their gaps: four device-wide sorts
//                of a few thousand 64-bit keys took eight passes of ~16 us each,
//                nearly all of it look-back latency.
//   above        one device-wide sort of all lists together (the list number on
//                top of the key), over the bits that vertex ids can have.
// Ingest per snapshot, before -> now: 32 updates 0.16 -> 0.017 ms, R-MAT 16 2K
// 0.17 -> 0.028, R-MAT 20 BFS 10K 0.50 -> 0.08, R-MAT 21 100K 0.70 -> 0.26.
#include <cub/block/block_radix_sort.cuh>
#include <cub/device/device_radix_sort.cuh>

#include "frontier.cuh"
#include "internal.h"

namespace dycg {

namespace {

int grid_for(u64 threads) {
  u64 b = (threads + BLOCK - 1) / BLOCK;
  if (b < 1) b = 1;
  if (b > 148ull * 32) b = 148ull * 32;
  return (int)b;
}

// (row, neighbour) of record r in list `list` (even: by source, odd: by
// destination) as one key of 2 * nbits bits; ~0 (after every valid key, whose
// ids are below n < 2^nbits) for a record with an endpoint out of range.
__device__ __forceinline__ u64 list_key(const dycg_edge_dev &r, uint32_t list, uint32_t n,
                                        uint32_t nbits) {
  if (r.u >= n || r.v >= n) return KEY_INF;
  const uint32_t row = list & 1 ? r.v : r.u, nb = list & 1 ? r.u : r.v;
  return ((u64)row << nbits) | nb;
}

// First position after p whose key leaves p's run (keys ascending, cnt of
// them): doubling steps, then bisection, so a hub row's segment or a heavily
// repeated edge costs its logarithm.
template <class Keys>
__device__ __forceinline__ uint32_t run_end(const Keys &key, uint32_t p, uint32_t cnt,
                                            uint32_t shift) {
  const u64 k = key(p) >> shift;
  uint32_t lo = p, step = 1;  // key(lo) belongs to the run
  while (lo + step < cnt && (key(lo + step) >> shift) == k) {
    lo += step;
    step *= 2;
  }
  uint32_t hi = min(lo + step, cnt);  // key(hi), if any, does not
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if ((key(mid) >> shift) == k) lo = mid; else hi = mid;
  }
  return hi;
}

// The list entry at position p.
template <class Keys>
__device__ __forceinline__ Rec list_entry(const Keys &key, uint32_t p, uint32_t cnt, bool adds,
                                          uint32_t w, uint32_t nbits) {
  const u64 mask = (1ull << nbits) - 1;
  const u64 k = key(p);
  Rec r = make_uint4((uint32_t)((k >> nbits) & mask), (uint32_t)(k & mask), w, 0u);
  if ((k & ((mask << nbits) | mask)) == ((mask << nbits) | mask))
    return make_uint4(INF32, INF32, 0u, 0u);
  const uint32_t shift = adds ? nbits : 0u;
  if (p == 0 || (key(p - 1) >> shift) != (k >> shift)) {
    r.w = run_end(key, p, cnt, shift) - p;
    // deletions: the row's records from here on
    if (!adds) r.z = run_end(key, p, cnt, nbits) - p;
  }
  return r;
}

// A source's first appearance in this batch: counted, listed, and its degree
// before the mutation kept (PageRank amends need it).
__device__ __forceinline__ void note_source(const Touch &T, uint32_t u, Ctl *ctl) {
  if (atomicExch(T.tag + u, T.epoch) == T.epoch) return;
  T.list[atomicAdd(T.count, 1u)] = u;
  if (T.old_degree) T.old_degree[u] = __uint_as_float(T.live[u]);
  atomicAdd(&ctl->stat[ST_TOUCHED], 1ull);
}

}  // namespace

// One CTA per list, up to THREADS * ITEMS records.
template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS)
    ingest_block_kernel(const BatchHdr *hdr, Lists L, uint32_t lists, uint32_t n, uint32_t nbits,
                        Touch T, Ctl *ctl, uint32_t carry_q, uint32_t carry) {
  using Sort = cub::BlockRadixSort<u64, THREADS, ITEMS, uint32_t>;
  extern __shared__ __align__(16) uint8_t ingest_sm[];
  typename Sort::TempStorage &temp = *reinterpret_cast<typename Sort::TempStorage *>(ingest_sm);
  u64 *sk = reinterpret_cast<u64 *>(ingest_sm);                       // sorted keys, then
  uint32_t *si = reinterpret_cast<uint32_t *>(sk + THREADS * ITEMS);  // their arrival order
  const uint32_t list = lists == 4 ? blockIdx.x : blockIdx.x * 2;
  const bool adds = list >= 2;
  const uint32_t cnt = adds ? hdr->na : hdr->nd;
  const dycg_edge_dev *e = adds ? hdr->adds : hdr->dels;
  // PageRank: the frontier carried over from the last batch
  if (blockIdx.x == 0 && threadIdx.x == 0 && carry) ctl->q_count[carry_q] = carry;
  u64 k[ITEMS];
  uint32_t idx[ITEMS], bad = 0;
#pragma unroll
  for (int i = 0; i < ITEMS; i++) {
    idx[i] = threadIdx.x * ITEMS + i;
    k[i] = KEY_INF;
    if (idx[i] < cnt) {
      k[i] = list_key(e[idx[i]], list, n, nbits);
      bad += k[i] == KEY_INF;
    }
  }
  if (!(list & 1)) {
    bad = __reduce_add_sync(0xffffffffu, bad);
    if (lane_id() == 0 && bad) atomicAdd(&ctl->stat[ST_INVALID], (u64)bad);
  }
  if (cnt) Sort(temp).Sort(k, idx, 0, 2 * nbits);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; i++) {
    sk[threadIdx.x * ITEMS + i] = k[i];
    si[threadIdx.x * ITEMS + i] = idx[i];
  }
  __syncthreads();
  const auto key = [&](uint32_t p) { return sk[p]; };
  for (uint32_t p = threadIdx.x; p < cnt; p += THREADS) {
    const Rec r = list_entry(key, p, cnt, adds, adds ? e[si[p]].w : 0u, nbits);
    L.rec[list][p] = r;
    if (T.tag && !(list & 1) && r.x != INF32 && (p == 0 || (key(p - 1) >> nbits) != r.x))
      note_source(T, r.x, ctl);
  }
}

// Keys of every list, list number on top; list l occupies positions
// [l * dcap, ...) for deletions, then acap each for insertions (capacities of
// a replayed size class, or the batch's own counts); positions past the
// batch's count sort last within their list.
__global__ void ingest_keys_kernel(const BatchHdr *hdr, uint32_t lists, uint32_t dcap,
                                   uint32_t acap, uint32_t n, uint32_t nbits, u64 *keys,
                                   uint32_t *w, Ctl *ctl, uint32_t carry_q, uint32_t carry) {
  const uint32_t half = lists / 2;
  const u64 dtot = (u64)half * dcap, total = dtot + (u64)half * acap;
  if (blockIdx.x == 0 && threadIdx.x == 0 && carry) ctl->q_count[carry_q] = carry;
  uint32_t bad = 0;
  for (u64 j = blockIdx.x * (u64)blockDim.x + threadIdx.x; j < total;
       j += (u64)gridDim.x * blockDim.x) {
    const bool adds = j >= dtot;
    const u64 q = adds ? j - dtot : j;
    const uint32_t cap = adds ? acap : dcap;
    const uint32_t dir = q >= cap ? 1u : 0u, i = (uint32_t)(q - (u64)dir * cap);
    const uint32_t cnt = adds ? hdr->na : hdr->nd;
    u64 k = KEY_INF;
    uint32_t x = 0;
    if (i < cnt) {
      const dycg_edge_dev r = (adds ? hdr->adds : hdr->dels)[i];
      k = list_key(r, dir, n, nbits);
      x = r.w;
      bad += k == KEY_INF && dir == 0;
    }
    keys[j] = (k & ((1ull << (2 * nbits)) - 1)) | ((u64)((adds ? half : 0u) + dir) << (2 * nbits));
    if (w) w[j] = x;
  }
  bad = __reduce_add_sync(0xffffffffu, bad);
  if (lane_id() == 0 && bad) atomicAdd(&ctl->stat[ST_INVALID], (u64)bad);
}

__global__ void ingest_lists_kernel(const BatchHdr *hdr, Lists L, uint32_t lists, uint32_t dcap,
                                    uint32_t acap, uint32_t nbits, const u64 *keys,
                                    const uint32_t *w, Touch T, Ctl *ctl) {
  const uint32_t half = lists / 2;
  const u64 dtot = (u64)half * dcap, total = dtot + (u64)half * acap;
  for (u64 j = blockIdx.x * (u64)blockDim.x + threadIdx.x; j < total;
       j += (u64)gridDim.x * blockDim.x) {
    const bool adds = j >= dtot;
    const u64 q = adds ? j - dtot : j;
    const uint32_t cap = adds ? acap : dcap;
    const uint32_t dir = q >= cap ? 1u : 0u, p = (uint32_t)(q - (u64)dir * cap);
    const uint32_t cnt = adds ? hdr->na : hdr->nd;
    if (p >= cnt) continue;
    const u64 *base = keys + (j - p);
    const auto key = [&](uint32_t i) { return base[i]; };
    const Rec r = list_entry(key, p, cnt, adds, w ? w[j] : 0u, nbits);
    L.rec[(adds ? 2u : 0u) + dir][p] = r;
    if (T.tag && dir == 0 && r.x != INF32 && (p == 0 || (key(p - 1) >> nbits) != (key(p) >> nbits)))
      note_source(T, r.x, ctl);
  }
}

template <int THREADS, int ITEMS>
static cudaError_t launch_block(const IngestLaunch &L, uint32_t lists, uint32_t nbits,
                                cudaStream_t s) {
  using Sort = cub::BlockRadixSort<u64, THREADS, ITEMS, uint32_t>;
  const size_t smem =
      std::max(sizeof(typename Sort::TempStorage), (size_t)THREADS * ITEMS * 12);
  if (smem > 48 * 1024) {  // a per-device setting: cheap enough to state on every launch
    const cudaError_t e =
        cudaFuncSetAttribute(ingest_block_kernel<THREADS, ITEMS>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  ingest_block_kernel<THREADS, ITEMS><<<lists, THREADS, smem, s>>>(
      L.hdr, L.lists, lists, L.n, nbits, L.touch, L.ctl, L.carry_q, L.carry);
  return cudaGetLastError();
}

static uint32_t id_bits(uint32_t n) {
  uint32_t b = 1;
  while (b < 31 && (n >> b)) b++;
  return b;
}

size_t ingest_temp_bytes(uint64_t records) {
  size_t a = 0, b = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, a, (const u64 *)nullptr, (u64 *)nullptr,
                                  (const uint32_t *)nullptr, (uint32_t *)nullptr,
                                  (int64_t)records, 0, 64);
  cub::DeviceRadixSort::SortKeys(nullptr, b, (const u64 *)nullptr, (u64 *)nullptr,
                                 (int64_t)records, 0, 64);
  return std::max(a, b);
}

cudaError_t launch_ingest(const IngestLaunch &L, uint32_t *launches, cudaStream_t s) {
  const uint32_t most = std::max(L.nd, L.na);
  *launches = 0;
  if (!most) return cudaSuccess;
  const uint32_t nbits = id_bits(L.n), lists = L.has_in ? 4 : 2;
  *launches = 1;
  // a block sort's time grows with its items per thread and its warps: ~6 us at
  // 128 records, ~25 us at 8192; the device-wide form takes ~120 us there
  if (most <= 128) return launch_block<128, 1>(L, lists, nbits, s);
  if (most <= 1024) return launch_block<256, 4>(L, lists, nbits, s);
  if (most <= 4096) return launch_block<512, 8>(L, lists, nbits, s);
  if (most <= INGEST_BLOCK_MAX) return launch_block<1024, 8>(L, lists, nbits, s);
  const u64 total = (u64)(lists / 2) * ((u64)L.nd + L.na);
  ingest_keys_kernel<<<grid_for(total), BLOCK, 0, s>>>(L.hdr, lists, L.nd, L.na, L.n, nbits,
                                                       L.keys, L.with_w ? L.w : nullptr, L.ctl,
                                                       L.carry_q, L.carry);
  size_t tb = L.temp_bytes;
  const int bits = 2 * nbits + (lists == 4 ? 2 : 1);
  cudaError_t e =
      L.with_w ? cub::DeviceRadixSort::SortPairs(L.temp, tb, L.keys, L.keys_sorted, L.w, L.w_sorted,
                                                 (int64_t)total, 0, bits, s)
               : cub::DeviceRadixSort::SortKeys(L.temp, tb, L.keys, L.keys_sorted, (int64_t)total,
                                                0, bits, s);
  if (e != cudaSuccess) return e;
  ingest_lists_kernel<<<grid_for(total), BLOCK, 0, s>>>(L.hdr, L.lists, lists, L.nd, L.na, nbits,
                                                        L.keys_sorted,
                                                        L.with_w ? L.w_sorted : nullptr, L.touch,
                                                        L.ctl);
  *launches = 3;
  return cudaGetLastError();
}

}  // namespace dycg
