// Per-cell moments of the deposition: their classes and their layout, shared
// by the kernels that form them (mass_tc.cu, moments.cu) and assemble them.
#pragma once

#include "common.cuh"

namespace tpicb200 {

constexpr int kFuse = 2;                     // species per launch
constexpr int kMassMoments = 27 * 9;         // G[t][c] per cell
constexpr int kMoments = kMassMoments + 24;  // + J corner sums [a][c]

// Moment layout: each group of four consecutive cells has one contiguous
// record of kMoments 16-byte words, word q holding entry q of the four cells.
__host__ __device__ constexpr long long moment_index(long long cell, int q) {
  return ((cell >> 2) * kMoments + q) * 4 + (cell & 3);
}

// Monomial class of the corner pair (a, b).
__host__ __device__ constexpr int monomial_class(int a, int b) {
  return ((a & 1) + (b & 1)) + 3 * (((a >> 1) & 1) + ((b >> 1) & 1)) + 9 * (((a >> 2) & 1) + ((b >> 2) & 1));
}

}  // namespace tpicb200
