// group.cu -- standalone GPU grouping of an update batch, the device form of
// the reference's GroupedUpdateBatch (include/framework/effective_update_batch.h:
// 36-207): records with an endpoint outside the vertex range are dropped and
// counted, the rest are radix-sorted by (u, v), and each distinct (u, v)
// becomes one output record with its multiplicity, in ascending (u, v) order.
// Optional per-segment counts of the distinct records bin them by source into
// the caller's vertex ranges (the reference's SEGMENT ranges).
//
// Keys hold only the bits that ids below the vertex count can have, so the sort
// takes seven passes instead of eight at 2^24 vertices and four at 2^15. Up to
// GROUP_BLOCK_MAX records one CTA does the whole call in shared memory (what
// bounds a small batch is the number of launches, and it needs no scratch);
// above, a device-wide sort and scan. Segment counts come from the sorted order
// -- a segment is a range of it, so two bisections give its distinct records --
// where one atomic per distinct record on its segment's counter took ~500 of the
// 713 us of a 1M-record R-MAT batch (half of its sources fall into a few
// segments); the batch takes 225-287 now.
#include <cub/block/block_radix_sort.cuh>
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>

#include "../../include/dycg.h"
#include "group.cuh"

namespace dycg {

// (u, v) in 2 * nbits bits; all ones (after every valid key) when out of range.
__device__ __forceinline__ u64 group_key(const dycg_edge &r, uint32_t n, uint32_t nbits) {
  return r.u < n && r.v < n ? ((u64)r.u << nbits) | r.v : KEY_INF;
}

__device__ __forceinline__ void emit_uv(uint32_t *out_uv, uint32_t o, u64 key, uint32_t nbits) {
  out_uv[2 * o] = (uint32_t)(key >> nbits);
  out_uv[2 * o + 1] = (uint32_t)(key & ((1ull << nbits) - 1));
}

// First of cnt ascending values that is >= x.
template <class T, class A>
__device__ __forceinline__ uint32_t first_at_least(const A *a, uint32_t cnt, T x) {
  uint32_t lo = 0, hi = cnt;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) / 2;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Distinct records whose source is below `end`: valid sorted keys, the runs'
// first indices.
__device__ __forceinline__ uint32_t runs_below(const u64 *keys, uint32_t valid,
                                               const uint32_t *start, uint32_t runs, uint32_t end,
                                               uint32_t nbits) {
  const uint32_t p = first_at_least<u64>(keys, valid, (u64)end << nbits);
  return p == valid ? runs : first_at_least<uint32_t>(start, runs, p);
}

// Segment s holds sources in [ends[s - 1], ends[s]).
__device__ __forceinline__ void count_segments(const u64 *keys, uint32_t valid,
                                               const uint32_t *start, uint32_t runs,
                                               const uint32_t *ends, uint32_t nseg,
                                               uint32_t *seg_counts, uint32_t nbits,
                                               uint32_t first, uint32_t step) {
  for (uint32_t s = first; s < nseg; s += step) {
    const uint32_t below = s ? runs_below(keys, valid, start, runs, ends[s - 1], nbits) : 0u;
    const uint32_t upto = runs_below(keys, valid, start, runs, ends[s], nbits);
    seg_counts[s] = upto - min(below, upto);
  }
}

// The same from the records' side, over zeroed counts: the first run of a segment
// counts it.
__device__ __forceinline__ void count_from_runs(const u64 *keys, uint32_t valid,
                                                const uint32_t *start, uint32_t runs,
                                                const uint32_t *ends, uint32_t nseg,
                                                uint32_t *seg_counts, uint32_t nbits,
                                                uint32_t first, uint32_t step) {
  for (uint32_t r = first; r < runs; r += step) {
    const uint32_t u = (uint32_t)(keys[start[r]] >> nbits);
    const uint32_t s = first_at_least<u64>(ends, nseg, (u64)u + 1);
    if (s == nseg) continue;
    const bool opens =
        r == 0 || (s && (uint32_t)(keys[start[r - 1]] >> nbits) < ends[s - 1]);
    if (opens) seg_counts[s] = runs_below(keys, valid, start, runs, ends[s], nbits) - r;
  }
}

// Which of the two: a segment costs two bisections of the records, a run one of the
// segments. The whole call for 300 records at 4096 / 65,536 / 2^20 segments from the
// segments' side 41 / 453 / 7,027 us, from the records' 21 / 23 / 25; for 8192 at
// 16,384 / 65,536 segments 110 / 260 against 92 from the records' at 65,536.
__host__ __device__ __forceinline__ bool from_runs(uint32_t nseg, uint32_t records) {
  return nseg / 2 > records;
}

// The whole call in one CTA: up to THREADS * ITEMS records.
template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS)
    group_block_kernel(const dycg_edge *e, uint32_t cnt, uint32_t n, uint32_t nbits,
                       const uint32_t *seg_ends, uint32_t nseg, uint32_t *out_uv,
                       uint32_t *out_mult, uint32_t *seg_counts, uint32_t *counts) {
  using Sort = cub::BlockRadixSort<u64, THREADS, ITEMS>;
  using Scan = cub::BlockScan<uint32_t, THREADS>;
  extern __shared__ __align__(16) uint8_t group_sm[];
  u64 *sk = reinterpret_cast<u64 *>(group_sm);                          // sorted keys
  uint32_t *ss = reinterpret_cast<uint32_t *>(sk + THREADS * ITEMS);    // runs' first indices
  __shared__ typename Scan::TempStorage scan_temp;
  __shared__ uint32_t s_bad;
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
  u64 k[ITEMS];
  uint32_t bad = 0;
#pragma unroll
  for (int i = 0; i < ITEMS; i++) {
    const uint32_t p = threadIdx.x * ITEMS + i;
    k[i] = KEY_INF;
    if (p < cnt) {
      k[i] = group_key(e[p], n, nbits);
      bad += k[i] == KEY_INF;
    }
  }
  if (bad) atomicAdd(&s_bad, bad);
  Sort(*reinterpret_cast<typename Sort::TempStorage *>(group_sm)).Sort(k, 0, 2 * nbits);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; i++) sk[threadIdx.x * ITEMS + i] = k[i];
  __syncthreads();
  const uint32_t valid = cnt - s_bad;
  uint32_t heads = 0, runs = 0, o = 0;
#pragma unroll
  for (int i = 0; i < ITEMS; i++) {
    const uint32_t p = threadIdx.x * ITEMS + i;
    heads += p < valid && (p == 0 || sk[p - 1] != k[i]);
  }
  Scan(scan_temp).ExclusiveSum(heads, o, runs);
#pragma unroll
  for (int i = 0; i < ITEMS; i++) {
    const uint32_t p = threadIdx.x * ITEMS + i;
    if (p < valid && (p == 0 || sk[p - 1] != k[i])) {
      ss[o] = p;
      emit_uv(out_uv, o++, k[i], nbits);
    }
  }
  __syncthreads();
  for (uint32_t r = threadIdx.x; r < runs; r += THREADS)
    out_mult[r] = (r + 1 < runs ? ss[r + 1] : valid) - ss[r];
  if (seg_counts) {
    if (from_runs(nseg, THREADS * ITEMS))
      count_from_runs(sk, valid, ss, runs, seg_ends, nseg, seg_counts, nbits, threadIdx.x, THREADS);
    else
      count_segments(sk, valid, ss, runs, seg_ends, nseg, seg_counts, nbits, threadIdx.x, THREADS);
  }
  if (threadIdx.x == 0) {
    counts[0] = runs;
    counts[1] = cnt - valid;
  }
}

__global__ void group_keys_kernel(const dycg_edge *e, uint32_t cnt, uint32_t n, uint32_t nbits,
                                  u64 *keys, uint32_t *invalid) {
  uint32_t bad = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt;
       i += gridDim.x * blockDim.x) {
    keys[i] = group_key(e[i], n, nbits);
    bad += keys[i] == KEY_INF;
  }
  bad = __reduce_add_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0 && bad) atomicAdd(invalid, bad);
}

// 1 where a run of equal keys opens (the scan's input, never stored).
struct HeadFlags {
  using difference_type = ptrdiff_t;
  using value_type = uint32_t;
  using pointer = const uint32_t *;
  using reference = uint32_t;
  using iterator_category = std::random_access_iterator_tag;
  const u64 *k;
  ptrdiff_t at;
  __host__ __device__ HeadFlags(const u64 *keys, ptrdiff_t i = 0) : k(keys), at(i) {}
  __device__ uint32_t operator*() const {
    return k[at] != KEY_INF && (at == 0 || k[at - 1] != k[at]);
  }
  __device__ uint32_t operator[](ptrdiff_t i) const { return *HeadFlags(k, at + i); }
  __host__ __device__ HeadFlags operator+(ptrdiff_t i) const { return HeadFlags(k, at + i); }
  __host__ __device__ HeadFlags &operator+=(ptrdiff_t i) {
    at += i;
    return *this;
  }
  __host__ __device__ ptrdiff_t operator-(const HeadFlags &o) const { return at - o.at; }
};

// Run heads in key order: the run number o of head i is pos[i]; record its
// first index and emit its (u, v).
__global__ void group_starts_kernel(const u64 *k, const uint32_t *pos, uint32_t cnt,
                                    uint32_t nbits, uint32_t *start, uint32_t *out_uv,
                                    uint32_t *counts) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt;
       i += gridDim.x * blockDim.x) {
    const u64 key = k[i];
    const bool head = key != KEY_INF && (i == 0 || k[i - 1] != key);
    if (i == cnt - 1) counts[0] = pos[i] + head;
    if (!head) continue;
    start[pos[i]] = i;
    emit_uv(out_uv, pos[i], key, nbits);
  }
}

// Multiplicity of run o = distance to the next run's first index; the last
// run ends at the number of valid keys (invalid ones sort last as KEY_INF).
// One thread per run whatever its length, so a batch of one repeated record
// costs the same as a batch of distinct ones. And the segments' counts.
__global__ void group_mult_kernel(const u64 *keys, const uint32_t *start, uint32_t cnt,
                                  const uint32_t *counts, uint32_t nbits, uint32_t *out_mult,
                                  const uint32_t *seg_ends, uint32_t nseg, uint32_t *seg_counts) {
  const uint32_t runs = counts[0];
  const uint32_t valid = cnt - counts[1];
  const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (uint32_t o = first; o < runs; o += step) {
    const uint32_t end = o + 1 < runs ? start[o + 1] : valid;
    out_mult[o] = end - start[o];
  }
  if (seg_counts) {
    if (from_runs(nseg, cnt))
      count_from_runs(keys, valid, start, runs, seg_ends, nseg, seg_counts, nbits, first, step);
    else
      count_segments(keys, valid, start, runs, seg_ends, nseg, seg_counts, nbits, first, step);
  }
}

static int grid_for(u64 threads) {
  u64 b = (threads + BLOCK - 1) / BLOCK;
  if (b < 1) b = 1;
  if (b > 148ull * 32) b = 148ull * 32;
  return (int)b;
}

size_t group_temp_bytes(uint32_t n) {
  size_t a = 0, b = 0;
  cub::DeviceRadixSort::SortKeys(nullptr, a, (const u64 *)nullptr, (u64 *)nullptr, (int)n, 0, 64);
  cub::DeviceScan::ExclusiveSum(nullptr, b, HeadFlags(nullptr), (uint32_t *)nullptr, (int)n);
  return a > b ? a : b;
}

template <int THREADS, int ITEMS>
static cudaError_t group_block(const dycg_edge *e, uint32_t n, uint32_t nv, uint32_t nbits,
                               const uint32_t *seg_ends, uint32_t nseg, uint32_t *out_uv,
                               uint32_t *out_mult, uint32_t *seg_counts, uint32_t *counts,
                               cudaStream_t s) {
  using Sort = cub::BlockRadixSort<u64, THREADS, ITEMS>;
  const size_t smem = std::max(sizeof(typename Sort::TempStorage), (size_t)THREADS * ITEMS * 12);
  if (smem > 32 * 1024) {  // (with the static part above 48 KB from 4096 records on)
    const cudaError_t x =
        cudaFuncSetAttribute(group_block_kernel<THREADS, ITEMS>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (x != cudaSuccess) return x;
  }
  if (seg_counts && from_runs(nseg, THREADS * ITEMS)) {
    const cudaError_t x = cudaMemsetAsync(seg_counts, 0, (size_t)nseg * sizeof(uint32_t), s);
    if (x != cudaSuccess) return x;
  }
  group_block_kernel<THREADS, ITEMS><<<1, THREADS, smem, s>>>(
      e, n, nv, nbits, seg_ends, nseg, out_uv, out_mult, seg_counts, counts);
  return cudaGetLastError();
}

cudaError_t group_run(const dycg_edge *d_records, uint32_t n, uint32_t num_vertices,
                      const uint32_t *seg_ends, uint32_t nseg, uint32_t *out_uv,
                      uint32_t *out_mult, uint32_t *seg_counts, uint32_t *counts,
                      const GroupScratch &S, cudaStream_t s) {
  cudaError_t e;
  if (!nseg) seg_counts = nullptr;
  uint32_t nbits = 1;  // ids are below num_vertices < 2^nbits, so no valid key is all ones
  while (nbits < 32 && ((u64)num_vertices >> nbits)) nbits++;
  if (n && n <= GROUP_BLOCK_MAX) {
    const auto run = n <= 256    ? group_block<256, 1>
                     : n <= 1024 ? group_block<256, 4>
                     : n <= 4096 ? group_block<512, 8>
                                 : group_block<1024, 8>;
    return run(d_records, n, num_vertices, nbits, seg_ends, nseg, out_uv, out_mult, seg_counts,
               counts, s);
  }
  e = cudaMemsetAsync(counts, 0, 2 * sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  if (seg_counts && (n == 0 || from_runs(nseg, n))) {
    e = cudaMemsetAsync(seg_counts, 0, (size_t)nseg * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
  }
  if (n == 0) return cudaSuccess;
  group_keys_kernel<<<grid_for(n), BLOCK, 0, s>>>(d_records, n, num_vertices, nbits, S.keys_a,
                                                  counts + 1);
  size_t tb = S.temp_bytes;
  e = cub::DeviceRadixSort::SortKeys(S.temp, tb, S.keys_a, S.keys_b, (int)n, 0, 2 * (int)nbits, s);
  if (e != cudaSuccess) return e;
  tb = S.temp_bytes;
  e = cub::DeviceScan::ExclusiveSum(S.temp, tb, HeadFlags(S.keys_b), S.pos, (int)n, s);
  if (e != cudaSuccess) return e;
  group_starts_kernel<<<grid_for(n), BLOCK, 0, s>>>(S.keys_b, S.pos, n, nbits, S.start, out_uv,
                                                    counts);
  group_mult_kernel<<<grid_for(from_runs(nseg, n) ? n : std::max(n, nseg)), BLOCK, 0, s>>>(
      S.keys_b, S.start, n, counts, nbits, out_mult, seg_ends, nseg, seg_counts);
  return cudaGetLastError();
}

}  // namespace dycg

using namespace dycg;

extern "C" int dycg_group_updates(const dycg_edge *d_records, size_t n, uint32_t num_vertices,
                                  const uint32_t *d_segment_ends, uint32_t num_segments,
                                  uint32_t *d_out_uv, uint32_t *d_out_mult,
                                  uint32_t *d_segment_counts, uint32_t *d_counts,
                                  void *stream) {
  if ((n && (!d_records || !d_out_uv || !d_out_mult)) || !d_counts || n > 0x7FFFFFFFull ||
      (num_segments && !d_segment_ends))
    return DYCG_EINVAL;
  cudaStream_t s = (cudaStream_t)stream;
  GroupScratch S{};
  void *base = nullptr;
  if (n > GROUP_BLOCK_MAX) {
    const uint32_t m = (uint32_t)n;
    S.temp_bytes = group_temp_bytes(m);
    const size_t bytes = group_scratch_bytes(m, S.temp_bytes);
    if (cudaMallocAsync(&base, bytes, s) != cudaSuccess) return DYCG_ENOMEM;
    group_carve(base, m, S);
  }
  cudaError_t e = group_run(d_records, (uint32_t)n, num_vertices, d_segment_ends, num_segments,
                            d_out_uv, d_out_mult, d_segment_counts, d_counts, S, s);
  cudaError_t f = base ? cudaFreeAsync(base, s) : cudaSuccess;
  if (e != cudaSuccess || f != cudaSuccess) return DYCG_ECUDA;
  return DYCG_OK;
}
