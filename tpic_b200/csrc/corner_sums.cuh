// Sums over the records of a cell of W_a(record) * value_n(record), the 8
// CIC corners a by N values, on the FP64 tensor cores: what a per-record
// deposition onto the corner nodes adds, one total per cell, corner and value.
//
// A warp stages 32 records (fractions and values) in shared memory; with
// m8n8k4 the 8 corners are the rows of A (each lane forms the weight of its
// corner and record from the staged fractions), the values the columns of B
// and 4 records one step, so a chunk takes 8 steps per 8 values and the totals
// stay in two registers per lane and tile. Records are taken in groups of
// equal cell keys; the totals are kept while consecutive groups have the same
// key, over chunks too, and handed out when it changes, so sorted records cost
// one addition per cell, corner and value. A chunk of many cells (records in no
// order, or few a cell) is a chain of as many groups: above kMost of them each
// lane adds its own record's contributions. Output moments on 64^3, us, by groups
// alone / with kMost / one thread a record and nothing else: 4.2M records in no
// order rho 823 / 199 / 184, rho and J 1,067 / 713 / 616, all ten 1,560 / 1,737 /
// 1,509; within some 25 cells of their place 431 / 170 / 181, 524 / 367 / 434, 737 /
// 629 / 943; sorted 132 / 129 / 228, 152 / 154 / 610, 203 / 207 / 1,321; two a cell
// 64 / 29 / 29, 78 / 55 / 53, 111 / 110 / 106. kMost 32: groups alone.
#pragma once

#include "common.cuh"

namespace tpicb200 {

template <int N, int kMost>
struct CornerSums {
  static constexpr int kTiles = (N + 7) / 8;
  // 36 records a row: the 16 lanes of a shared-memory phase (4 rows x 4
  // records) then touch 16 different 8-byte banks.
  static constexpr int kPitch = 36;
  struct Stage {  // one per warp
    double fraction[3][kPitch];
    double value[N][kPitch];
  };

  double c[kTiles][2];
  int32_t key;  // the cell of the totals held; -1: none

  __device__ __forceinline__ void begin() {
    key = -1;
#pragma unroll
    for (int t = 0; t < kTiles; ++t) c[t][0] = c[t][1] = 0.0;
  }

  // Hands the totals held to sink.add(node, n, total), this lane's share, with
  // node = sink.node(key, corner).
  template <class Sink>
  __device__ __forceinline__ void flush(Sink&& sink) {
    if (key < 0) return;
    const int lane = threadIdx.x & 31;
    const auto node = sink.node(key, lane >> 2);
#pragma unroll
    for (int t = 0; t < kTiles; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = 8 * t + 2 * (lane & 3) + h;
        if (n < N) sink.add(node, n, c[t][h]);
      }
    begin();
  }

  // Whether the records of a chunk are in more than kMost cells. Runs of equal keys
  // bound their number from above and are counted first; a chunk of hardly any runs
  // longer than one record is taken for many cells without a closer look.
  __device__ __forceinline__ bool many(bool ok, int32_t k) const {
    const unsigned lane = threadIdx.x & 31u;
    const int32_t before = __shfl_up_sync(0xffffffffu, k, 1);
    const int runs = __popc(__ballot_sync(0xffffffffu, ok && (lane == 0 || k != before)));
    if (runs <= kMost || runs > 28) return runs > kMost;
    const unsigned same = __match_any_sync(0xffffffffu, k) & __ballot_sync(0xffffffffu, ok);
    return __popc(__ballot_sync(0xffffffffu, ok && int(lane) == __ffs(same) - 1)) > kMost;
  }

  // One chunk: this lane's record (ok: it counts; its key, fractions and
  // values, all finite where their totals are used). Every lane calls it.
  template <class Sink>
  __device__ __forceinline__ void add(Stage& s, bool ok, int32_t k, const double f[3], const double v[N],
                                      Sink&& sink) {
    const int lane = threadIdx.x & 31, row = lane >> 2, col = lane & 3;
    __syncwarp();
#pragma unroll
    for (int a = 0; a < 3; ++a) s.fraction[a][lane] = ok ? f[a] : 0.0;
#pragma unroll
    for (int n = 0; n < N; ++n) s.value[n][lane] = ok ? v[n] : 0.0;
    __syncwarp();
    if constexpr (kMost < 32) {
      if (many(ok, k)) {
        if (ok) {
          // Not unrolled, the cell decoded for each corner: with more registers fewer
          // warps fit, which costs the sorted records more than this saves.
#pragma unroll 1
          for (int a = 0; a < 8; ++a) {
            const double x = s.fraction[0][lane], y = s.fraction[1][lane], z = s.fraction[2][lane];
            const double w = ((a & 1) ? x : 1.0 - x) * ((a & 2) ? y : 1.0 - y) * ((a & 4) ? z : 1.0 - z);
            const auto node = sink.node(k, a);
#pragma unroll
            for (int n = 0; n < N; ++n) sink.add(node, n, w * s.value[n][lane]);
          }
        }
        return;
      }
    }
    unsigned left = __ballot_sync(0xffffffffu, ok);
    while (left) {
      const int32_t group = __shfl_sync(0xffffffffu, k, __ffs(left) - 1);
      const unsigned members = __ballot_sync(0xffffffffu, k == group) & left;
      left &= ~members;
      if (group != key) {
        flush(sink);
        key = group;
      }
#pragma unroll
      for (int step = 0; step < 8; ++step) {
        const unsigned four = (members >> (4 * step)) & 15u;
        if (four == 0) continue;
        const int r = 4 * step + col;
        const double x = s.fraction[0][r], y = s.fraction[1][r], z = s.fraction[2][r];
        const double w = ((row & 1) ? x : 1.0 - x) * ((row & 2) ? y : 1.0 - y) * ((row & 4) ? z : 1.0 - z);
        // Both factors of a record outside the group are zero, so a nonfinite
        // value stays in its own cell's totals.
        const bool member = (four >> col) & 1u;
        const double a = member ? w : 0.0;
#pragma unroll
        for (int t = 0; t < kTiles; ++t) {
          const int n = 8 * t + row;
          dmma_884(c[t], a, member && n < N ? s.value[n < N ? n : 0][r] : 0.0);
        }
      }
    }
  }
};

// Records [first, last) of this warp: consecutive runs of whole chunks, as
// equal as the chunks allow, so that a warp's records are neighbours.
__device__ __forceinline__ void warp_segment(uint32_t count, uint32_t& first, uint32_t& last) {
  const uint32_t warps = gridDim.x * (blockDim.x / 32), warp = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const uint32_t chunks = count / 32 + (count % 32 ? 1 : 0);
  const uint32_t each = chunks / warps, more = chunks % warps;
  const uint32_t c0 = warp * each + min(warp, more), c1 = c0 + each + (warp < more ? 1 : 0);
  first = c0 * 32;
  last = uint32_t(min((unsigned long long)c1 * 32, (unsigned long long)count));
}

}  // namespace tpicb200
