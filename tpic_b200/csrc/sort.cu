// Stable counting sort of one species' records by cell key.
//
// TPIC sorts with LPFx's direct-cell counting sort: histogram, scan,
// permutation by atomic cursors and one scatter per attribute
// (lpfx/algorithm/particle/device/cuda_hip/sort.hpp:64-260). Its device form
// is unstable within a bin (lpfx/algorithm/particle/device/sort.hpp:372-374);
// its host form (lpfx/algorithm/particle/host/sort.hpp:205-290) is stable.
// This sort produces the stable order, so the permutation, counts and offsets
// are bit-identical to the host sort:
//   1. histogram with warp-aggregated atomics (__match_any_sync),
//   2. exclusive scan of the bins,
//   3. placement by warp-aggregated atomic cursors (stable within a warp),
//   4. per-bin fix-up: each bin's source indices are sorted ascending, which
//      restores the input order among equal keys (a warp ranks them by
//      counting; block bitonic or merge-path sorts for large bins),
//   5. one fused gather of every attribute through the permutation.
// An out-of-range key stops the sort after step 1 (the kernels of steps 2-5
// test the sort's own flag) and is reported through *invalid.
#include "grid_barrier.cuh"
#include "kernels.cuh"

#include <algorithm>
#include <cuda.h>
#include <mutex>

namespace tpicb200 {
namespace {

using CoopBarrier = GridBarrier<true>;

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int kWarpBinCapacity = 256;   // per-warp shared-memory sort
constexpr int kBlockBinCapacity = 8192; // per-block shared-memory sort (32 KB)

// Scratch words after the scan block sums: [0] sort-local invalid flag,
// [1] number of large bins, then the large-bin list.
struct ScanScratch {
  uint32_t* block_sums;
  uint32_t* flag;
  uint32_t* large_count;
  uint32_t* large_bins;
};

__device__ __forceinline__ void aggregated_add(uint32_t* base, int32_t key, bool valid,
                                               uint32_t& position) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned active = __ballot_sync(0xffffffffu, valid);
  const unsigned peers = __match_any_sync(0xffffffffu, valid ? key : -1);
  if (valid) {
    const unsigned group = peers & active;
    const int leader = __ffs(group) - 1;
    const unsigned rank = __popc(group & ((1u << lane) - 1u));
    uint32_t start = 0;
    if ((int)lane == leader) start = atomicAdd(base + key, __popc(group));
    start = __shfl_sync(group, start, leader);
    position = start + rank;
  }
}

__global__ void __launch_bounds__(256) fill_kernel(uint32_t* out, long long n, uint32_t value) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = value;
}

__global__ void __launch_bounds__(256) copy_kernel(uint32_t* out, const uint32_t* __restrict__ in, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = in[i];
}

__device__ __forceinline__ void histogram(const Geom& g, const int32_t* __restrict__ keys, uint32_t count,
                                          uint32_t* counts, uint32_t* flag) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < count; base += stride) {
    const uint32_t i = base + (threadIdx.x & 31);
    const bool in_range = i < count;
    const int32_t key = in_range ? keys[i] : -1;
    const bool ok = key >= 0 && (long long)key < g.bins;
    if (in_range && !ok) atomicExch(flag, 1u);
    uint32_t unused;
    aggregated_add(counts, key, in_range && ok, unused);
  }
}
__global__ void __launch_bounds__(256) histogram_kernel(Geom g, const int32_t* __restrict__ keys, uint32_t count,
                                                        uint32_t* counts, uint32_t* flag) {
  histogram(g, keys, count, counts, flag);
}

__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const uint32_t* __restrict__ counts,
                                                                   long long bins, uint32_t* block_sums,
                                                                   const uint32_t* flag) {
  __shared__ uint32_t scratch[kScanThreads / 32];
  if (*flag) return;
  const long long base = (long long)blockIdx.x * kScanTile;
  uint32_t sum = 0;
#pragma unroll
  for (int r = 0; r < kScanItems; ++r) {
    const long long i = base + threadIdx.x + (long long)r * kScanThreads;
    if (i < bins) sum += counts[i];
  }
  sum = block_sum<kScanThreads>(sum, scratch);
  if (threadIdx.x == 0) block_sums[blockIdx.x] = sum;
}

// Exclusive scan of the block sums by one block of 1024 threads.
__global__ void __launch_bounds__(1024) scan_block_sums_kernel(uint32_t* block_sums, int nblocks,
                                                               const uint32_t* flag) {
  __shared__ uint32_t warp_totals[32];
  if (*flag) return;
  const int per = (nblocks + 1023) / 1024;
  const int first = threadIdx.x * per;
  uint32_t local = 0;
  for (int i = 0; i < per; ++i)
    if (first + i < nblocks) local += block_sums[first + i];
  // Block exclusive scan of `local`.
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inclusive = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inclusive, o);
    if (lane >= o) inclusive += t;
  }
  if (lane == 31) warp_totals[warp] = inclusive;
  __syncthreads();
  if (warp == 0) {
    uint32_t t = warp_totals[lane];
    uint32_t inc = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    warp_totals[lane] = inc - t;
  }
  __syncthreads();
  uint32_t running = warp_totals[warp] + inclusive - local;
  for (int i = 0; i < per; ++i)
    if (first + i < nblocks) {
      const uint32_t v = block_sums[first + i];
      block_sums[first + i] = running;
      running += v;
    }
}

__global__ void __launch_bounds__(kScanThreads) scan_down_kernel(const uint32_t* __restrict__ counts,
                                                                 long long bins,
                                                                 const uint32_t* __restrict__ block_sums,
                                                                 uint32_t* offsets, const uint32_t* flag) {
  __shared__ uint32_t warp_totals[kScanThreads / 32];
  if (*flag) return;
  const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
  uint32_t items[kScanItems];
  uint32_t local = 0;
#pragma unroll
  for (int r = 0; r < kScanItems; ++r) {
    items[r] = base + r < bins ? counts[base + r] : 0u;
    local += items[r];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inclusive = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inclusive, o);
    if (lane >= o) inclusive += t;
  }
  if (lane == 31) warp_totals[warp] = inclusive;
  __syncthreads();
  uint32_t warp_prefix = 0;
  for (int w = 0; w < warp; ++w) warp_prefix += warp_totals[w];
  uint32_t running = block_sums[blockIdx.x] + warp_prefix + inclusive - local;
#pragma unroll
  for (int r = 0; r < kScanItems; ++r) {
    if (base + r < bins) offsets[base + r] = running;
    running += items[r];
  }
  if (base + kScanItems >= bins && base < bins) offsets[bins] = running;
  if (bins == 0 && blockIdx.x == 0 && threadIdx.x == 0) offsets[0] = 0;
}

__device__ __forceinline__ void place(const int32_t* __restrict__ keys, uint32_t count, uint32_t* cursor,
                                      uint32_t* perm) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < count; base += stride) {
    const uint32_t i = base + (threadIdx.x & 31);
    const bool valid = i < count;
    const int32_t key = valid ? keys[i] : -1;
    uint32_t position = 0;
    aggregated_add(cursor, key, valid, position);
    if (valid) perm[position] = i;
  }
}
__global__ void __launch_bounds__(256) place_kernel(const int32_t* __restrict__ keys, uint32_t count,
                                                    uint32_t* cursor, uint32_t* perm, const uint32_t* flag) {
  if (*flag) return;
  place(keys, count, cursor, perm);
}

// The n <= kWarpBinCapacity distinct indices in s, written in increasing order
// to `to` by one warp: an index's place is the number of smaller ones. Every
// lane holds up to eight of them and compares each of the n with all eight.
__device__ __forceinline__ void warp_rank_sort(const uint32_t* s, uint32_t n, uint32_t* to) {
  constexpr int kOwn = kWarpBinCapacity / 32;
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t own[kOwn], rank[kOwn];
#pragma unroll
  for (int r = 0; r < kOwn; ++r) {
    own[r] = 32 * r + lane < n ? s[32 * r + lane] : 0xffffffffu;
    rank[r] = 0;
  }
  for (uint32_t t = 0; t < n; ++t) {
    const uint32_t other = s[t];
#pragma unroll
    for (int r = 0; r < kOwn; ++r) rank[r] += other < own[r] ? 1u : 0u;
  }
#pragma unroll
  for (int r = 0; r < kOwn; ++r)
    if (32 * r + lane < n) to[rank[r]] = own[r];
}

// Bins above kWarpBinCapacity are listed in large_bins; with huge_count those
// above kBlockBinCapacity from its end.
__device__ __forceinline__ void fixup_small(const uint32_t* counts, const uint32_t* offsets, long long bins,
                                            uint32_t* perm, uint32_t* large_count, uint32_t* large_bins,
                                            uint32_t* huge_count, uint32_t (*buffer)[kWarpBinCapacity]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* s = buffer[warp];
  // Neighbouring bins to different blocks: the cells of a line are neighbours.
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  for (long long bin = (long long)gridDim.x * warp + blockIdx.x; bin < bins; bin += warps) {
    const uint32_t n = counts[bin];
    if (n <= 1) continue;
    if (n > (uint32_t)kWarpBinCapacity) {
      if (lane == 0) {
        const bool huge = huge_count && n > (uint32_t)kBlockBinCapacity;
        large_bins[huge ? bins - 1 - atomicAdd(huge_count, 1u) : (long long)atomicAdd(large_count, 1u)] = (uint32_t)bin;
      }
      continue;
    }
    const uint32_t first = offsets[bin];
    bool sorted = true;
    for (uint32_t t = lane; t < n; t += 32) {
      const uint32_t value = perm[first + t];
      s[t] = value;
      if (t > 0 && perm[first + t - 1] > value) sorted = false;
    }
    if (__all_sync(0xffffffffu, sorted)) continue;
    __syncwarp();
    warp_rank_sort(s, n, perm + first);
    __syncwarp();
  }
}

__global__ void __launch_bounds__(256) fixup_small_kernel(const uint32_t* counts, const uint32_t* offsets,
                                                          long long bins, uint32_t* perm, uint32_t* large_count,
                                                          uint32_t* large_bins, const uint32_t* flag) {
  __shared__ uint32_t buffer[8][kWarpBinCapacity];
  if (*flag) return;
  fixup_small(counts, offsets, bins, perm, large_count, large_bins, nullptr, buffer);
}

// The n <= kBlockBinCapacity distinct indices at p in increasing order, by one
// block (bitonic, in shared memory).
__device__ __forceinline__ void block_sort(uint32_t* p, uint32_t n, uint32_t* s) {
  int size = 1;
  while (size < (int)n) size <<= 1;
  for (int t = threadIdx.x; t < size; t += blockDim.x) s[t] = t < (int)n ? p[t] : 0xffffffffu;
  __syncthreads();
  for (int k = 2; k <= size; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = threadIdx.x; t < size; t += blockDim.x) {
        const int partner = t ^ j;
        if (partner > t) {
          const uint32_t a = s[t], b = s[partner];
          const bool up = (t & k) == 0;
          if ((a > b) == up) { s[t] = b; s[partner] = a; }
        }
      }
      __syncthreads();
    }
  for (int t = threadIdx.x; t < (int)n; t += blockDim.x) p[t] = s[t];
  __syncthreads();
}

// Entry t after runs of `width` sorted indices in src[0, n) are merged in pairs
// (merge path: i entries of the first run and d - i of the second precede
// output d).
__device__ __forceinline__ uint32_t merged(const uint32_t* src, uint32_t n, uint32_t width, uint32_t t) {
  const uint32_t run = uint32_t(t / (2ull * width) * (2ull * width));
  const uint32_t a0 = run, a1 = min(n - run, width) + run;
  const uint32_t b1 = uint32_t(min(run + 2ull * width, (unsigned long long)n));
  const uint32_t la = a1 - a0, lb = b1 - a1, d = t - run;
  uint32_t lo = d > lb ? d - lb : 0, hi = d < la ? d : la;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (src[a0 + mid] < src[a1 + d - mid - 1]) lo = mid + 1;
    else hi = mid;
  }
  const uint32_t i = lo, jb = d - i;
  return i < la && (jb >= lb || src[a0 + i] < src[a1 + jb]) ? src[a0 + i] : src[a1 + jb];
}

// One block per large bin. Up to kBlockBinCapacity entries sort in shared
// memory; larger bins merge runs in global memory with merge-path splits,
// ping-ponging with `scratch` (a free array of the output records).
__device__ __forceinline__ void fixup_large(const uint32_t* counts, const uint32_t* offsets, uint32_t* perm,
                                            uint32_t* scratch, const uint32_t* large_count,
                                            const uint32_t* large_bins, uint32_t* s) {
  const uint32_t nlarge = *large_count;
  for (uint32_t item = blockIdx.x; item < nlarge; item += gridDim.x) {
    const uint32_t bin = large_bins[item];
    const uint32_t n = counts[bin], first = offsets[bin];
    if (n <= (uint32_t)kBlockBinCapacity) {
      block_sort(perm + first, n, s);
      continue;
    }
    uint32_t* src = perm + first;
    uint32_t* dst = scratch + first;
    for (unsigned long long width = 1; width < n; width <<= 1) {
      for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) dst[t] = merged(src, n, uint32_t(width), t);
      __syncthreads();
      uint32_t* tmp = src; src = dst; dst = tmp;
    }
    if (src != perm + first)
      for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) perm[first + t] = src[t];
    __syncthreads();
  }
}

// The same for bins above kBlockBinCapacity (listed from the end of the
// large-bin list) by all blocks of a cooperative launch: sorted runs of
// kBlockBinCapacity, then one merge pass over all those bins between two
// barriers, so that a wait is for one pass over the records and never for
// a whole bin: by one block a bin of ten million would outlast the barrier's
// bound. Whole sorts of two bins of 150,000 records 11.0 -> 2.6 ms (separate
// launches of one block a bin: 5.3), of 64 of 20,000 2.7 -> 1.07 (1.07).
// False when a barrier gave up.
__device__ __forceinline__ bool fixup_huge(const uint32_t* counts, const uint32_t* offsets, uint32_t* perm,
                                           uint32_t* scratch, uint32_t nhuge, const uint32_t* last,
                                           uint32_t* s, CoopBarrier& barrier) {
  constexpr uint32_t kRun = kBlockBinCapacity;
  uint32_t longest = 0, run = 0;
  for (uint32_t h = 0; h < nhuge; ++h) {
    const uint32_t bin = *(last - h), n = counts[bin], first = offsets[bin];
    longest = max(longest, n);
    for (uint32_t r = 0; r < n; r += min(kRun, n - r), ++run)
      if (run % gridDim.x == blockIdx.x) block_sort(perm + first + r, min(kRun, n - r), s);
  }
  // f(first, n, begin, end) for this block's share of every bin [first, first + n):
  // chunks of the bins in turn, the bins staged in shared memory.
  auto each_chunk = [&](auto&& f) {
    constexpr uint32_t kBatch = kBlockBinCapacity / 2;
    const uint32_t size = 2 * blockDim.x;
    unsigned long long chunk = 0;
    for (uint32_t h0 = 0; h0 < nhuge; h0 += kBatch) {
      const uint32_t batch = min(kBatch, nhuge - h0);
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < batch; i += blockDim.x) {
        const uint32_t bin = *(last - h0 - i);
        s[2 * i] = offsets[bin];
        s[2 * i + 1] = counts[bin];
      }
      __syncthreads();
      for (uint32_t i = 0; i < batch; ++i) {
        const uint32_t first = s[2 * i], n = s[2 * i + 1], chunks = n / size + (n % size ? 1 : 0);
        for (unsigned long long c = (blockIdx.x + gridDim.x - chunk % gridDim.x) % gridDim.x; c < chunks; c += gridDim.x)
          f(first, n, uint32_t(c * size), uint32_t(min((c + 1) * size, (unsigned long long)n)));
        chunk += chunks;
      }
    }
  };
  // Pass m goes from perm to scratch for even m and back for odd m; a bin that was
  // one run after an odd number of passes is copied back in the pass behind them.
  bool odd = false;
  for (unsigned long long width = kRun; width < longest || odd; width <<= 1, odd = !odd) {
    if (!barrier.wait()) return false;
    each_chunk([&](uint32_t first, uint32_t n, uint32_t begin, uint32_t end) {
      const uint32_t* src = (odd ? scratch : perm) + first;
      uint32_t* dst = (odd ? perm : scratch) + first;
      if (n > width)
        for (uint32_t t = begin + threadIdx.x; t < end; t += blockDim.x) dst[t] = merged(src, n, uint32_t(width), t);
      else if (odd && 2ull * n > width)
        for (uint32_t t = begin + threadIdx.x; t < end; t += blockDim.x) dst[t] = src[t];
    });
  }
  return true;
}

__global__ void __launch_bounds__(1024) fixup_large_kernel(const uint32_t* counts, const uint32_t* offsets,
                                                           uint32_t* perm, uint32_t* scratch,
                                                           const uint32_t* large_count, const uint32_t* large_bins,
                                                           const uint32_t* flag) {
  __shared__ uint32_t s[kBlockBinCapacity];
  if (*flag) return;
  fixup_large(counts, offsets, perm, scratch, large_count, large_bins, s);
}

// The records of both sides of a gather.
template <class Vel>
struct SortRecords {
  const double *irx, *iry, *irz;
  const Vel *iu, *iv, *iw;
  const double* iq;
  const int32_t* ikey;
  const uint64_t* iid;
  double *orx, *ory, *orz;
  Vel *ou, *ov, *ow;
  double* oq;
  int32_t* okey;
  uint64_t* oid;  // null: no ids
  SortRecords(const tpicb200_particles* in, tpicb200_particles* out)
      : irx((const double*)in->rx), iry((const double*)in->ry), irz((const double*)in->rz), iu((const Vel*)in->u),
        iv((const Vel*)in->v), iw((const Vel*)in->w), iq(in->q), ikey(in->cell), iid(in->id), orx((double*)out->rx),
        ory((double*)out->ry), orz((double*)out->rz), ou((Vel*)out->u), ov((Vel*)out->v), ow((Vel*)out->w),
        oq(out->q), okey(out->cell), oid(in->id ? out->id : nullptr) {}
};
template <class Vel>
__device__ __forceinline__ void gather(uint32_t s, uint32_t p, const SortRecords<Vel>& r) {
  const double x = __ldg(r.irx + s), y = __ldg(r.iry + s), z = __ldg(r.irz + s), q = __ldg(r.iq + s);
  const Vel u = __ldg(r.iu + s), v = __ldg(r.iv + s), w = __ldg(r.iw + s);
  const int32_t key = __ldg(r.ikey + s);
  r.orx[p] = x;
  r.ory[p] = y;
  r.orz[p] = z;
  r.ou[p] = u;
  r.ov[p] = v;
  r.ow[p] = w;
  r.oq[p] = q;
  r.okey[p] = key;
  if (r.oid) r.oid[p] = r.iid[s];
}
// Unless a flag is raised, or with no flag through ranks that may be a failed sort's.
template <class Vel, bool kFlag>
__global__ void __launch_bounds__(256) gather_kernel(const uint32_t* __restrict__ perm, uint32_t count,
                                                     SortRecords<Vel> r, const uint32_t* flag) {
  if (kFlag && *flag) return;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < count; p += gridDim.x * blockDim.x) {
    const uint32_t s = perm[p];
    if (kFlag || s < count) gather(s, p, r);
  }
}
cudaError_t launch_gather(int precision, const uint32_t* perm, const tpicb200_particles* in, tpicb200_particles* out,
                          const uint32_t* flag, cudaStream_t s) {
  const uint32_t n = in->count;
  const unsigned blocks = grid_for(n, 256, 148u * 8u);
  auto go = [&](auto kernel, auto records) { kernel<<<blocks, 256, 0, s>>>(perm, n, records, flag); };
  if (precision == TPICB200_PRECISION_DOUBLE)
    go(flag ? gather_kernel<double, true> : gather_kernel<double, false>, SortRecords<double>(in, out));
  else
    go(flag ? gather_kernel<float, true> : gather_kernel<float, false>, SortRecords<float>(in, out));
  count_launches(1);
  return cudaGetLastError();
}

__global__ void report_kernel(const uint32_t* flag, uint32_t* invalid) {
  if (*flag && invalid) atomicAdd(invalid, 1u);
}

}  // namespace

size_t sort_scan_words(long long bins) {
  const long long nblocks = (bins + kScanTile - 1) / kScanTile;
  return size_t(nblocks) + 2 + size_t(bins);
}

namespace {

// The general sort.
cudaError_t enqueue_general(int precision, const Geom& g, const tpicb200_particles* in, tpicb200_particles* out,
                            uint32_t* counts, uint32_t* offsets, uint32_t* cursor, uint32_t* perm,
                            uint32_t* scan_scratch, uint32_t* invalid, cudaStream_t s) {
  const long long bins = g.bins;
  const int nblocks = int((bins + kScanTile - 1) / kScanTile);
  ScanScratch sc{scan_scratch, scan_scratch + nblocks, scan_scratch + nblocks + 1,
                 scan_scratch + nblocks + 2};
  const uint32_t n = in->count;
  cudaError_t e;
  if ((e = cudaMemsetAsync(sc.flag, 0, 2 * sizeof(uint32_t), s)) != cudaSuccess) return e;
  fill_kernel<<<grid_for(bins, 256, 148u * 8u), 256, 0, s>>>(counts, bins, 0u);
  if (n) histogram_kernel<<<grid_for(n, 256, 148u * 8u), 256, 0, s>>>(g, in->cell, n, counts, sc.flag);
  scan_reduce_kernel<<<nblocks, kScanThreads, 0, s>>>(counts, bins, sc.block_sums, sc.flag);
  scan_block_sums_kernel<<<1, 1024, 0, s>>>(sc.block_sums, nblocks, sc.flag);
  scan_down_kernel<<<nblocks, kScanThreads, 0, s>>>(counts, bins, sc.block_sums, offsets, sc.flag);
  copy_kernel<<<grid_for(bins, 256, 148u * 8u), 256, 0, s>>>(cursor, offsets, bins);
  int launches = 7;
  if (n) {
    place_kernel<<<grid_for(n, 256, 148u * 8u), 256, 0, s>>>(in->cell, n, cursor, perm, sc.flag);
    fixup_small_kernel<<<grid_for(bins, 256, 148u * 16u), 256, 0, s>>>(counts, offsets, bins, perm, sc.large_count,
                                                                      sc.large_bins, sc.flag);
    fixup_large_kernel<<<148, 1024, 0, s>>>(counts, offsets, perm, (uint32_t*)out->cell, sc.large_count,
                                            sc.large_bins, sc.flag);
    launches += 3;
    if ((e = launch_gather(precision, perm, in, out, sc.flag, s)) != cudaSuccess) return e;
  }
  report_kernel<<<1, 1, 0, s>>>(sc.flag, invalid);
  count_launches(launches + 1);
  return cudaGetLastError();
}

// ---- The binned sort's cooperative kernels ----

// Exclusive scan of counts[0, bins) into offsets[0, bins] (and cursor, when
// given) by all CTAs: each takes a contiguous range, whose sum it has stored
// in sums[blockIdx.x]; the other CTAs' sums are read after a grid barrier.
constexpr int kCoopThreads = 256;
// One CTA of 1,024 threads an SM: 64 bins of 5,000 records, a block's sort each, 308
// us, with two of 512 382, with two of 256 480 (as separate launches 349).
constexpr int kFallbackThreads = 1024;
__device__ __forceinline__ void coop_range(long long bins, long long& b0, long long& b1) {
  const long long each = (bins + gridDim.x - 1) / gridDim.x;
  b0 = min(blockIdx.x * each, bins);
  b1 = min(b0 + each, bins);
}
template <int kThreads>
__device__ __forceinline__ void coop_scan(const uint32_t* counts, long long bins, const uint32_t* sums,
                                          uint32_t* offsets, uint32_t* cursor) {
  __shared__ uint32_t scratch[kThreads / 32];
  __shared__ uint32_t warp_totals[kThreads / 32];
  constexpr int kItems = 4;
  uint32_t before = 0;
  for (unsigned b = threadIdx.x; b < blockIdx.x; b += kThreads) before += __ldcg(sums + b);
  uint32_t running = block_sum<kThreads>(before, scratch);
  long long b0, b1;
  coop_range(bins, b0, b1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (long long tile = b0; tile < b1; tile += kItems * kThreads) {
    const long long at = tile + (long long)threadIdx.x * kItems;
    uint32_t items[kItems], local = 0;
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      items[r] = at + r < b1 ? __ldcg(counts + at + r) : 0u;
      local += items[r];
    }
    uint32_t inclusive = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inclusive, o);
      if (lane >= o) inclusive += t;
    }
    __syncthreads();
    if (lane == 31) warp_totals[warp] = inclusive;
    __syncthreads();
    uint32_t prefix = running, total = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
      if (w < warp) prefix += warp_totals[w];
      total += warp_totals[w];
    }
    prefix += inclusive - local;
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      if (at + r < b1) {
        offsets[at + r] = prefix;
        if (cursor) cursor[at + r] = prefix;
      }
      prefix += items[r];
    }
    running += total;
  }
  if (b1 == bins && b0 < b1 && threadIdx.x == 0) offsets[bins] = running;
}

// The steps of the general sort by all CTAs; returns early where a barrier gives up.
template <class Vel>
__device__ __forceinline__ void fallback_sort(const Geom& g, uint32_t n, const SortRecords<Vel>& r, uint32_t* counts,
                                              uint32_t* offsets, uint32_t* cursor, uint32_t* perm,
                                              const ScanScratch& sc, uint32_t* invalid, CoopBarrier& barrier,
                                              uint32_t* buffer, uint32_t* scratch) {
  uint32_t* sums = sc.large_bins;  // free until the fix-up
  constexpr int kThreads = kFallbackThreads;
  uint32_t* huge_count = sc.block_sums;
  for (long long b = blockIdx.x * (long long)kThreads + threadIdx.x; b < g.bins; b += (long long)gridDim.x * kThreads)
    counts[b] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) *sc.flag = *sc.large_count = *huge_count = 0;
  if (!barrier.wait()) return;
  histogram(g, r.ikey, n, counts, sc.flag);
  if (!barrier.wait()) return;
  const bool bad = __ldcg(sc.flag) != 0;
  if (!bad) {
    long long b0, b1;
    coop_range(g.bins, b0, b1);
    uint32_t sum = 0;
    for (long long b = b0 + threadIdx.x; b < b1; b += kThreads) sum += __ldcg(counts + b);
    sum = block_sum<kThreads>(sum, scratch);
    if (threadIdx.x == 0) sums[blockIdx.x] = sum;
    if (!barrier.wait()) return;
    coop_scan<kThreads>(counts, g.bins, sums, offsets, cursor);
    if (!barrier.wait()) return;
    place(r.ikey, n, cursor, perm);
    if (!barrier.wait()) return;
    fixup_small(counts, offsets, g.bins, perm, sc.large_count, sc.large_bins, huge_count,
                reinterpret_cast<uint32_t (*)[kWarpBinCapacity]>(buffer));
    if (!barrier.wait()) return;
    uint32_t* free = (uint32_t*)r.okey;
    fixup_large(counts, offsets, perm, free, sc.large_count, sc.large_bins, buffer);
    if (!fixup_huge(counts, offsets, perm, free, *huge_count, sc.large_bins + g.bins - 1, buffer, barrier)) return;
    if (!barrier.wait()) return;
    for (unsigned long long p = blockIdx.x * kThreads + threadIdx.x; p < n; p += gridDim.x * kThreads)
      gather(perm[p], uint32_t(p), r);
  } else if (blockIdx.x == 0 && threadIdx.x == 0 && invalid) {
    atomicAdd(invalid, 1u);
  }
}

// The general sort in one launch, for the binned sort's fallback: enqueued
// behind every binned sort and leaving at once unless the fallback flag is up.
// As the general sort's eleven kernels it cost 25 us of empty launches per
// species and cycle. Its steps are separated by grid barriers, none of which waits
// for more than a pass over the records or the bins; the last CTA to
// leave clears the flags for the next sort. Where a barrier gave up, perm and the
// records are unfinished: that CTA then empties the bins, so that nothing reads
// through them, and counts 1 << 22 in *invalid.
template <class Vel>
__global__ void __launch_bounds__(kFallbackThreads, 1)
    fallback_sort_kernel(Geom g, uint32_t n, SortRecords<Vel> r, uint32_t* counts, uint32_t* offsets, uint32_t* cursor,
                         uint32_t* perm, ScanScratch sc, uint32_t* invalid, BinnedState* state, GridWaits waits) {
  static_assert(kFallbackThreads / 32 * kWarpBinCapacity <= kBlockBinCapacity, "the warps' buffers are the block's");
  __shared__ uint32_t buffer[kBlockBinCapacity];
  __shared__ uint32_t scratch[kFallbackThreads / 32];
  if (state->fallback == 0) return;
  CoopBarrier barrier(state->barrier, waits);
  fallback_sort(g, n, r, counts, offsets, cursor, perm, sc, invalid, barrier, buffer, scratch);
  const CoopBarrier::Exit exit = barrier.leave();
  if (exit == CoopBarrier::kLastOfFailed) {
    for (long long b = threadIdx.x; b <= g.bins; b += kFallbackThreads) {
      if (b < g.bins) counts[b] = 0;
      offsets[b] = 0;
    }
    if (threadIdx.x == 0 && invalid) atomicAdd(invalid, 1u << 22);
  }
  if (exit != CoopBarrier::kOther && threadIdx.x == 0) state->fallback = state->bins_bad = 0;
}

template <class Vel>
cudaError_t launch_fallback(const Geom& g, const tpicb200_particles* in, tpicb200_particles* out, uint32_t* counts,
                            uint32_t* offsets, uint32_t* cursor, uint32_t* perm, uint32_t* scan_scratch,
                            uint32_t* invalid, const BinnedScratch& b, cudaStream_t s) {
  const int nblocks = int((g.bins + kScanTile - 1) / kScanTile);
  ScanScratch sc{scan_scratch, scan_scratch + nblocks, scan_scratch + nblocks + 1, scan_scratch + nblocks + 2};
  Geom geom = g;
  uint32_t n = in->count;
  SortRecords<Vel> r(in, out);
  // One CTA an SM, fewer for little work (a barrier costs with their number);
  // their sums must fit the bins' scratch.
  const long long work = std::max<long long>(g.bins, n);
  const unsigned blocks = unsigned(std::min<long long>(grid_for(work, kFallbackThreads, unsigned(b.sms)), g.bins));
  BinnedState* state = b.state;
  GridWaits waits = b.sort_waits;
  void* args[] = {&geom, &n, &r, &counts, &offsets, &cursor, &perm, &sc, &invalid, &state, &waits};
  count_launches(1);
  return cudaLaunchCooperativeKernel((const void*)fallback_sort_kernel<Vel>, dim3(blocks), dim3(kFallbackThreads), args,
                                     0, s);
}

// ---- Binned sort: the input is grouped by the bins of an earlier sort ----
//
// After the mover a species' records are still grouped by the cells of the
// previous sort, in increasing key order, and almost every record moved to
// one of the 27 cells around its old one. The stable order of a destination
// bin is then: its source cells in increasing key order and, within one
// source, the records in input order. So
//   1. direction codes d < 27 of every record and transfer counts T[d][c]
//      per old interior cell c: from the mover itself (it knows both cells)
//      or from classify_kernel (old cell from the bins, new from the key);
//      periodic_step gives each (source, destination) pair one code on
//      any extent (on an axis of two cells 0 -> 1 is -1 and 1 -> 0 is +1; on
//      an axis of one cell every step is 0);
//   2. validation: the old bins must tile the records in key order;
//   3. counts (thread per bin): counts'[b] = sum_d T[d][b - d];
//   4. scan of the counts;
//   5. bases (thread per interior bin): walking the 27 sources of b in key
//      order, T[d][c] becomes the first output position of c's records that
//      moved by d;
//   6. rank (a warp per run of up to 32 old cells of an x-row): a record's
//      position is its base plus its rank among the earlier records of its
//      cell with the same d, after checking that old cell + d is the cell of
//      its key; one gather then writes the sorted records.
// Any record that did not move to a neighbour, any invalid key, bins that do
// not tile the records or a failed scatter check raise the fallback flag,
// and the general sort, enqueued last and gated on the flag, rewrites the
// whole output (the binned gather is skipped). The output is the same stable
// order either way.

constexpr int kBinnedThreads = 256;
constexpr int kBinnedWarps = kBinnedThreads / 32;

// A warp takes a run (up to g.run_len <= 32 consecutive old interior cells
// of one x-row, run_cells) at a time. The run's records form one contiguous range; lane l
// holds cell l's record range. Writes the cells' first records to `start`
// (empty cells share their successor's start; unused entries are ~0) and
// returns the run's record range.
__device__ __forceinline__ void load_run_bins(const Geom& g, int i0, int len, int j, int k,
                                              const uint32_t* __restrict__ old_counts,
                                              const uint32_t* __restrict__ old_offsets, uint32_t* start,
                                              uint32_t& begin, uint32_t& end) {
  const int lane = threadIdx.x & 31;
  uint32_t off = 0xffffffffu, stop = 0;
  if (lane < len) {
    const int32_t key = g.encode(i0 + lane, j, k);
    off = old_offsets[key];
    stop = off + old_counts[key];
  }
  start[lane] = off;
  begin = __shfl_sync(0xffffffffu, off, 0);
  end = __shfl_sync(0xffffffffu, stop, len - 1);
  __syncwarp();
}

// Cell (offset in the run) of record p: the last cell whose start is at most p.
__device__ __forceinline__ int run_cell(const uint32_t* start, uint32_t p) {
  int c = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1)
    if (start[c + step] <= p) c += step;
  return c;
}

// Direction code of a record of old interior cell (i, j, k) whose key is now
// `key`, or -1 when the key is invalid or not one of the 27 neighbours.
__device__ __forceinline__ int key_move_code(const Geom& g, int i, int j, int k, int32_t key) {
  if (key < 0 || key >= g.bins) return -1;
  int a, b, c;
  g.decode(key, a, b, c);
  if (!g.interior_cell(a, b, c)) return -1;
  return move_code(g, i, j, k, a, b, c);
}

// The old bins copied (the new ones may overwrite them in place), checked, and
// the transfer counts cleared when the mover will add into them. The bins must
// tile the n records in key order: each starts where the one before it ends,
// the first at 0, the last ending at n, records only in interior cells.
__global__ void __launch_bounds__(256) binned_begin_kernel(Geom g, uint32_t n, const uint32_t* in_counts,
                                                           const uint32_t* in_offsets, uint32_t* old_counts,
                                                           uint32_t* old_offsets, uint32_t* transfer,
                                                           long long transfer_words, BinnedState* state) {
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  bool bad = false;
  for (long long b = first; b < g.bins; b += stride) {
    const uint32_t off = in_offsets[b], cnt = in_counts[b], next = in_offsets[b + 1];
    bad = bad || (unsigned long long)off + cnt != next || (b == 0 && off != 0) || (b + 1 == g.bins && next != n);
    if (cnt) {
      int i, j, k;
      g.decode(int32_t(b), i, j, k);
      bad = bad || !g.interior_cell(i, j, k);
    }
    old_counts[b] = cnt;
    old_offsets[b] = off;
    if (b + 1 == g.bins) old_offsets[g.bins] = next;
  }
  for (long long t = first; t < transfer_words; t += stride) transfer[t] = 0;
  if (__syncthreads_or(bad) && threadIdx.x == 0) {
    atomicExch(&state->bins_bad, 1u);
    atomicExch(&state->fallback, 1u);
  }
}

__global__ void __launch_bounds__(kBinnedThreads) classify_kernel(Geom g, const int32_t* __restrict__ keys,
    uint32_t n, const uint32_t* __restrict__ old_counts, const uint32_t* __restrict__ old_offsets,
    uint32_t* __restrict__ transfer, uint16_t* __restrict__ code, BinnedState* state) {
  __shared__ uint32_t starts[kBinnedWarps][kRunCells];
  __shared__ uint32_t hist[kBinnedWarps][27][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long cells = (long long)g.nx * g.ny * g.nz;
  const long long runs = run_count(g);
  bool bad = false;
  uint32_t* start = starts[warp];
  for (long long run = (long long)blockIdx.x * kBinnedWarps + warp; run < runs;
       run += (long long)gridDim.x * kBinnedWarps) {
    int i0, len, j, k;
    run_cells(g, run, i0, len, j, k);
    uint32_t begin, end;
    load_run_bins(g, i0, len, j, k, old_counts, old_offsets, start, begin, end);
#pragma unroll
    for (int d = 0; d < 27; ++d) hist[warp][d][lane] = 0;
    __syncwarp();
    if (begin > end || end > n) {  // bins that do not describe the records: no walk over them
      bad = true;
      continue;
    }
    // Four chunks per step: the key loads of all four are in flight together.
    for (uint32_t p0 = begin; p0 < end; p0 += 128) {
      int32_t key[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint32_t p = p0 + 32 * m + lane;
        key[m] = p < end ? keys[p] : 0;
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        if (p0 + 32 * m >= end) break;
        const uint32_t p = p0 + 32 * m + lane;
        const bool live = p < end;
        int c = 0, d = -1;
        if (live) {
          c = run_cell(start, p);
          d = key_move_code(g, i0 + c, j, k, key[m]);
          if (d < 0) bad = true;
          code[p] = d < 0 ? kNoMove : uint16_t(d | (c << 5));
        }
        const int slot = d < 0 ? -1 : c * 27 + d;
        const unsigned peers = __match_any_sync(0xffffffffu, slot);
        if (slot >= 0 && lane == __ffs(peers) - 1) hist[warp][d][c] += __popc(peers);
        __syncwarp();
      }
    }
    if (lane < len) {
      const long long u = i0 + lane + (long long)g.nx * (j + (long long)g.ny * k);
#pragma unroll
      for (int d = 0; d < 27; ++d) transfer[(long long)d * cells + u] = hist[warp][d][lane];
    }
    __syncwarp();
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicExch(&state->fallback, 1u);
}

// Records that bin b receives.
__device__ __forceinline__ uint32_t binned_count(const Geom& g, const uint32_t* __restrict__ transfer, long long b) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const long long cells = (long long)nx * ny * nz;
  int i, j, k;
  g.decode(int32_t(b), i, j, k);
  uint32_t sum = 0;
  if (g.interior_cell(i, j, k)) {
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
      for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
          // Neighbour offsets are -1..1: a conditional wrap (no modulo).
          int si = i - dx, sj = j - dy, sk = k - dz;
          si = si < 0 ? si + nx : (si >= nx ? si - nx : si);
          sj = sj < 0 ? sj + ny : (sj >= ny ? sj - ny : sj);
          sk = sk < 0 ? sk + nz : (sk >= nz ? sk - nz : sk);
          const int d = (dx + 1) + 3 * (dy + 1) + 9 * (dz + 1);
          sum += transfer[d * cells + si + (long long)nx * (sj + (long long)ny * sk)];
        }
  }
  return sum;
}

// Directions along one axis in increasing source coordinate: the sources of
// destination x are x - d (periodic).
__device__ __forceinline__ void source_order(int x, int n, int (&d)[3]) {
  if (x == 0) { d[0] = 0; d[1] = -1; d[2] = 1; }
  else if (x == n - 1) { d[0] = -1; d[1] = 1; d[2] = 0; }
  else { d[0] = 1; d[1] = 0; d[2] = -1; }
}

__device__ __forceinline__ void binned_bases(const Geom& g, const uint32_t* offsets, uint32_t* transfer) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const long long cells = (long long)nx * ny * nz;
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < cells;
       v += (long long)gridDim.x * blockDim.x) {
    const int i = int(v % nx);
    const long long r = v / nx;
    const int j = int(r % ny), k = int(r / ny);
    int ox[3], oy[3], oz[3];
    source_order(i, nx, ox);
    source_order(j, ny, oy);
    source_order(k, nz, oz);
    // Sources (periodic neighbours x - d) in increasing key order.
    long long index[27];
    uint32_t count[27];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const int dx = ox[a], dy = oy[b], dz = oz[c];
          int si = i - dx, sj = j - dy, sk = k - dz;
          si = si < 0 ? si + nx : (si >= nx ? si - nx : si);
          sj = sj < 0 ? sj + ny : (sj >= ny ? sj - ny : sj);
          sk = sk < 0 ? sk + nz : (sk >= nz ? sk - nz : sk);
          const int e = a + 3 * b + 9 * c;
          index[e] = ((dx + 1) + 3 * (dy + 1) + 9 * (dz + 1)) * cells + si + (long long)nx * (sj + (long long)ny * sk);
          count[e] = transfer[index[e]];
        }
    uint32_t base = offsets[g.encode(i, j, k)];
#pragma unroll
    for (int e = 0; e < 27; ++e) {
      transfer[index[e]] = base;
      base += count[e];
    }
  }
}

// The plan by all CTAs; returns early where a barrier gives up.
__device__ __forceinline__ void binned_plan(const Geom& g, uint32_t* transfer, uint32_t* counts, uint32_t* offsets,
                                            uint32_t* sums, CoopBarrier& barrier, uint32_t* scratch) {
  long long b0, b1;
  coop_range(g.bins, b0, b1);
  uint32_t sum = 0;
  for (long long b = b0 + threadIdx.x; b < b1; b += kCoopThreads) {
    const uint32_t count = binned_count(g, transfer, b);
    counts[b] = count;
    sum += count;
  }
  sum = block_sum<kCoopThreads>(sum, scratch);
  if (threadIdx.x == 0) sums[blockIdx.x] = sum;
  if (!barrier.wait()) return;
  coop_scan<kCoopThreads>(counts, g.bins, sums, offsets, nullptr);
  if (!barrier.wait()) return;
  binned_bases(g, offsets, transfer);
}

// Counts, their scan and the bases in one launch, the passes separated by grid
// barriers; where one gives up the last CTA to leave raises the fallback flag.
// As five kernels they were launch latency on small grids (127 x 65
// x 1 FP64 particle stage 125 us, 111 us with one) and no faster on large ones
// (128^3 cycle 27.1 ms, 26.8 ms with one).
__global__ void __launch_bounds__(kCoopThreads, 2) binned_plan_kernel(Geom g, uint32_t* transfer, uint32_t* counts,
                                                                      uint32_t* offsets, uint32_t* sums,
                                                                      BinnedState* state, GridWaits waits) {
  __shared__ uint32_t scratch[kCoopThreads / 32];
  if (state->fallback) return;
  CoopBarrier barrier(state->barrier, waits);
  binned_plan(g, transfer, counts, offsets, sums, barrier, scratch);
  if (threadIdx.x == 0 && barrier.depart() == CoopBarrier::kLastOfFailed) state->fallback = 1;
}

// The lane mask of a live lane's slot: the live lanes with the same slot
// value (one match instruction; a lane that is not live matches only itself).
__device__ __forceinline__ unsigned slot_group(int slot, bool live) {
  return __match_any_sync(0xffffffffu, live ? slot : -1 - int(threadIdx.x & 31));
}

// Output position of every record: perm[position] = record. The record goes
// to its base plus its rank among the earlier records of its cell with the
// same direction, after the check that its old cell + d is the cell of its
// key; the sorted records are then written by gather_kernel, whose stores
// are coalesced (records that changed cell would otherwise each write
// partial sectors of nine arrays).
__global__ void __launch_bounds__(kBinnedThreads) binned_rank_kernel(Geom g, uint32_t n,
    const uint32_t* __restrict__ old_counts, const uint32_t* __restrict__ old_offsets,
    const uint32_t* __restrict__ transfer, const uint16_t* __restrict__ code, const int32_t* __restrict__ keys,
    uint32_t* __restrict__ perm, BinnedState* state) {
  __shared__ uint32_t starts[kBinnedWarps][kRunCells];
  __shared__ uint32_t cursor[kBinnedWarps][27][33];
  if (state->fallback) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const long long cells = (long long)nx * ny * nz;
  const long long runs = run_count(g);
  const unsigned below = (1u << lane) - 1u;
  bool bad = false;
  for (long long run = (long long)blockIdx.x * kBinnedWarps + warp; run < runs;
       run += (long long)gridDim.x * kBinnedWarps) {
    int i0, len, j, k;
    run_cells(g, run, i0, len, j, k);
    uint32_t begin, end;
    load_run_bins(g, i0, len, j, k, old_counts, old_offsets, starts[warp], begin, end);
    if (lane < len) {
      const long long u = i0 + lane + (long long)nx * (j + (long long)ny * k);
#pragma unroll
      for (int d = 0; d < 27; ++d) cursor[warp][d][lane] = transfer[(long long)d * cells + u];
    }
    __syncwarp();
    // Four chunks per step: their loads are in flight together.
    for (uint32_t p0 = begin; p0 < end; p0 += 128) {
      uint16_t cd[4];
      int32_t key[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint32_t p = p0 + 32 * m + lane;
        cd[m] = p < end ? code[p] : kNoMove;
        key[m] = p < end ? keys[p] : 0;
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        if (p0 + 32 * m >= end) break;
        const uint32_t p = p0 + 32 * m + lane;
        bool live = p < end;
        const int d = cd[m] & 31, c = (cd[m] >> 5) & 31;
        if (live) {
          // The record must land in the cell of its key: its old cell + d.
          int a = i0 + c + (d % 3) - 1, b = j + (d / 3) % 3 - 1, e = k + d / 9 - 1;
          a = a < 0 ? a + nx : (a >= nx ? a - nx : a);
          b = b < 0 ? b + ny : (b >= ny ? b - ny : b);
          e = e < 0 ? e + nz : (e >= nz ? e - nz : e);
          if (cd[m] == kNoMove || d >= 27 || c >= len || g.encode(a, b, e) != key[m]) {
            bad = true;
            live = false;
          }
        }
        const unsigned group = slot_group(c * 27 + d, live);
        if (live) {
          const uint32_t o = cursor[warp][d][c] + __popc(group & below);
          if (o < n) perm[o] = p;
          else bad = true;
        }
        __syncwarp();
        if (live && lane == __ffs(group) - 1) cursor[warp][d][c] += __popc(group);
        __syncwarp();
      }
    }
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(&state->fallback, 1u);
}

}  // namespace

cudaError_t launch_sort(int precision, const Geom& g, const tpicb200_particles* in,
                        tpicb200_particles* out, uint32_t* counts, uint32_t* offsets,
                        uint32_t* cursor, uint32_t* perm, uint32_t* scan_scratch,
                        uint32_t* invalid, cudaStream_t s) {
  out->count = in->count;
  return enqueue_general(precision, g, in, out, counts, offsets, cursor, perm, scan_scratch, invalid, s);
}

cudaError_t launch_sorted_gather(int precision, const uint32_t* perm, const tpicb200_particles* in,
                                 tpicb200_particles* out, cudaStream_t s) {
  out->count = in->count;
  if (!in->count) return cudaSuccess;
  return launch_gather(precision, perm, in, out, nullptr, s);
}

size_t binned_scratch_words(const Geom& g) {
  const long long cells = (long long)g.nx * g.ny * g.nz;
  return sizeof(BinnedState) / 4 + size_t(2 * g.bins + 1) + size_t(27 * cells);
}

// Every periodic grid: on an axis of one or two cells each (source, destination)
// pair still has exactly one direction code (periodic_step), so the sources
// of a destination stay in increasing key order with no two nonempty
// directions sharing a source.
bool binned_sort_applies(const Geom& g) { return g.nx >= 1 && g.ny >= 1 && g.nz >= 1; }

BinnedScratch binned_scratch(const Geom& g, uint32_t* words, uint16_t* codes, GridWaits plan_waits,
                             GridWaits sort_waits, int sms) {
  BinnedScratch b;
  b.sms = sms;
  b.plan_waits = plan_waits;
  b.sort_waits = sort_waits;
  b.state = reinterpret_cast<BinnedState*>(words);
  b.old_counts = words + sizeof(BinnedState) / 4;
  b.old_offsets = b.old_counts + g.bins;
  b.transfer = b.old_offsets + g.bins + 1;
  b.code = codes;
  return b;
}

cudaError_t binned_reset(const BinnedScratch& b) { return cudaMemset(b.state, 0, sizeof(BinnedState)); }

cudaError_t binned_begin(const Geom& g, const BinnedScratch& b, uint32_t n, const uint32_t* in_counts,
                         const uint32_t* in_offsets, bool zero_transfer, cudaStream_t s) {
  const long long words = zero_transfer ? 27LL * g.nx * g.ny * g.nz : 0;
  binned_begin_kernel<<<grid_for(std::max(g.bins, words / 4), 256, 148u * 8u), 256, 0, s>>>(
      g, n, in_counts, in_offsets, b.old_counts, b.old_offsets, b.transfer, words, b.state);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t binned_finish(int precision, const Geom& g, const BinnedScratch& b, bool classify, bool materialize,
                          const tpicb200_particles* in, tpicb200_particles* out, uint32_t* counts,
                          uint32_t* offsets, uint32_t* cursor, uint32_t* perm, uint32_t* scan_scratch,
                          uint32_t* invalid, cudaStream_t s) {
  const long long bins = g.bins;
  const uint32_t n = in->count;
  out->count = n;
  // One warp per run (up to 32 cells of an x-row).
  const unsigned runs_grid = grid_for(run_count(g) * 32, kBinnedThreads, 148u * 8u);
  if (classify) {
    classify_kernel<<<runs_grid, kBinnedThreads, 0, s>>>(g, in->cell, n, b.old_counts, b.old_offsets, b.transfer,
                                                        b.code, b.state);
    count_launches(1);
  }
  const int nblocks = int((bins + kScanTile - 1) / kScanTile);
  ScanScratch sc{scan_scratch, scan_scratch + nblocks, scan_scratch + nblocks + 1, scan_scratch + nblocks + 2};
  cudaError_t e = cudaSuccess;
  {
    Geom geom = g;
    uint32_t *transfer = b.transfer, *sums = sc.large_bins;
    BinnedState* state = b.state;
    GridWaits waits = b.plan_waits;
    void* args[] = {&geom, &transfer, &counts, &offsets, &sums, &state, &waits};
    const unsigned blocks = unsigned(std::min<long long>(grid_for(bins, kCoopThreads, 2u * unsigned(b.sms)), bins));
    e = cudaLaunchCooperativeKernel((const void*)binned_plan_kernel, dim3(blocks), dim3(kCoopThreads), args, 0, s);
    count_launches(1);
  }
  if (e != cudaSuccess) return e;
  binned_rank_kernel<<<runs_grid, kBinnedThreads, 0, s>>>(g, n, b.old_counts, b.old_offsets, b.transfer, b.code,
                                                           in->cell, perm, b.state);
  count_launches(1);
  // The gather writes the records unless a check raised the fallback flag
  // (without `materialize` the caller reads the records through perm).
  if (n && materialize) e = launch_gather(precision, perm, in, out, &b.state->fallback, s);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // The general sort behind the fallback flag: it rewrites every output.
  return precision == TPICB200_PRECISION_DOUBLE
             ? launch_fallback<double>(g, in, out, counts, offsets, cursor, perm, scan_scratch, invalid, b, s)
             : launch_fallback<float>(g, in, out, counts, offsets, cursor, perm, scan_scratch, invalid, b, s);
}

cudaError_t launch_sort_binned(int precision, const Geom& g, const tpicb200_particles* in,
                               const uint32_t* in_counts, const uint32_t* in_offsets, tpicb200_particles* out,
                               uint32_t* counts, uint32_t* offsets, uint32_t* cursor, uint32_t* perm,
                               uint32_t* scan_scratch, const BinnedScratch& b, uint32_t* invalid, cudaStream_t s) {
  if (cudaError_t e = binned_begin(g, b, in->count, in_counts, in_offsets, false, s); e != cudaSuccess) return e;
  return binned_finish(precision, g, b, true, true, in, out, counts, offsets, cursor, perm, scan_scratch, invalid,
                       s);
}

// ---- Sort without a context and without allocation ----
//
// Some callers cannot allocate device memory for a sort: a caller that owns
// no context (the sort needs one only for its scratch), a caller whose device
// memory is held by another allocator's pool, or a loop that must not pay
// cudaMalloc's implicit device synchronisation. For them the general sort runs
// on a fixed file-scope scratch array instead of context buffers, for inputs
// up to TPICB200_SORT_STATIC_MAX_RECORDS records over up to
// TPICB200_SORT_STATIC_MAX_BINS bins; larger inputs are rejected. Every call
// shares the one array, so calls that overlap in time (other streams, other
// host threads) race on it; they must be ordered on one stream.

namespace {

constexpr long long kStaticRecords = TPICB200_SORT_STATIC_MAX_RECORDS;
constexpr long long kStaticBins = TPICB200_SORT_STATIC_MAX_BINS;
constexpr long long kStaticScanWords = (kStaticBins + kScanTile - 1) / kScanTile + 2 + kStaticBins;
// Permutation, cursors, then the scan block sums, flags and large-bin list.
constexpr long long kStaticWords = kStaticRecords + kStaticBins + kStaticScanWords;

static __device__ __align__(256) uint32_t g_static_scratch[kStaticWords];

// The array's address is resolved once per CUDA context: a device's primary
// context, a driver context a caller made current, or the primary context
// created again after cudaDeviceReset each hold their own copy of the array.
// A context's id (cuCtxGetId) is unique for the life of the process, so a
// context created after another was destroyed never reuses its cached
// address. The driver functions are fetched through the runtime, so the
// library needs no link against the driver library.
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);
constexpr int kStaticMaxContexts = 64;
std::mutex g_static_mutex;
struct StaticAddress {
  unsigned long long context_id;
  uint32_t* address;
};
StaticAddress g_static_address[kStaticMaxContexts] = {};
int g_static_used = 0;
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;

cudaError_t current_context_id(unsigned long long* id) {
  CUcontext ctx = nullptr;
  if (g_ctx_get_current(&ctx) != CUDA_SUCCESS) return cudaErrorInvalidResourceHandle;
  if (!ctx) return cudaErrorContextIsDestroyed;
  return g_ctx_get_id(ctx, id) == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidResourceHandle;
}

}  // namespace

long long sort_static_scratch_bytes() { return kStaticWords * 4; }

cudaError_t sort_static_setup(uint32_t** scratch) {
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (!g_ctx_get_current || !g_ctx_get_id) {
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    void* fn = nullptr;
    cudaError_t e = cudaGetDriverEntryPoint("cuCtxGetCurrent", &fn, cudaEnableDefault, &found);
    if (e != cudaSuccess || found != cudaDriverEntryPointSuccess || !fn) return e != cudaSuccess ? e : cudaErrorNotSupported;
    g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(fn);
    e = cudaGetDriverEntryPoint("cuCtxGetId", &fn, cudaEnableDefault, &found);
    if (e != cudaSuccess || found != cudaDriverEntryPointSuccess || !fn) return e != cudaSuccess ? e : cudaErrorNotSupported;
    g_ctx_get_id = reinterpret_cast<CtxGetIdFn>(fn);
  }
  unsigned long long id = 0;
  cudaError_t e = current_context_id(&id);
  uint32_t* fresh = nullptr;
  if (e == cudaErrorContextIsDestroyed) {
    // No context is current yet: resolving the symbol initialises the
    // current device's primary context and makes it current.
    e = cudaGetSymbolAddress((void**)&fresh, g_static_scratch);
    if (e != cudaSuccess) return e;
    e = current_context_id(&id);
  }
  if (e != cudaSuccess) return e;
  for (int i = 0; i < g_static_used; ++i)
    if (g_static_address[i].context_id == id) {
      *scratch = g_static_address[i].address;
      return cudaSuccess;
    }
  // Once per context, with that context current: the array's device address.
  if (!fresh) {
    e = cudaGetSymbolAddress((void**)&fresh, g_static_scratch);
    if (e != cudaSuccess) return e;
  }
  // Contexts beyond the table's size replace the oldest entry.
  const int slot = g_static_used < kStaticMaxContexts ? g_static_used++ : int(id % kStaticMaxContexts);
  g_static_address[slot] = {id, fresh};
  *scratch = fresh;
  return cudaSuccess;
}

cudaError_t launch_sort_static(int precision, const Geom& g, const tpicb200_particles* in, tpicb200_particles* out,
                               uint32_t* counts, uint32_t* offsets, uint32_t* invalid, uint32_t* scratch,
                               cudaStream_t s) {
  if ((long long)in->count > kStaticRecords || g.bins > kStaticBins) return cudaErrorInvalidValue;
  uint32_t* perm = scratch;
  uint32_t* cursor = perm + kStaticRecords;
  uint32_t* scan = cursor + kStaticBins;
  // The general sort clears what must start at zero on every call: its
  // flags and large-bin count (memset), the counts (fill); the cursors are
  // copied from the offsets and the permutation is fully written.
  out->count = in->count;
  return enqueue_general(precision, g, in, out, counts, offsets, cursor, perm, scan, invalid, s);
}

}  // namespace tpicb200
