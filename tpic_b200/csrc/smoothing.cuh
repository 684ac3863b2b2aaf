// Energy-conserving smoothing passes over a tile held in shared memory.
//
// One pass (node_smoothing_kernel, ecsim/fields/node_smoothing_device.hpp:17-36,
// with the operator of ecsim/fields/node_smoothing.hpp:24-52) in arithmetic C
// with each product and sum rounded on its own (no contraction) in the
// reference's order. Op 0 Face7: alpha * centre + beta * faces; op 1
// Binomial27: (8 centre + 4 faces + 2 edges + corners) * (1/64).
#pragma once

#include "common.cuh"

namespace tpicb200 {

__device__ __forceinline__ float rn_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rn_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rn_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double rn_add(double a, double b) { return __dadd_rn(a, b); }

// The pass at a node, its neighbours v(dx, dy, dz).
template <class C, class V>
__device__ __forceinline__ C smooth_sum(V&& v, int op, C alpha, C beta) {
  const C face = rn_add(rn_add(rn_add(rn_add(rn_add(v(-1, 0, 0), v(1, 0, 0)), v(0, -1, 0)), v(0, 1, 0)), v(0, 0, -1)),
                        v(0, 0, 1));
  if (op == 0) return rn_add(rn_mul(alpha, v(0, 0, 0)), rn_mul(beta, face));
  C edge = rn_add(v(-1, -1, 0), v(1, -1, 0));
  edge = rn_add(edge, v(-1, 1, 0)); edge = rn_add(edge, v(1, 1, 0));
  edge = rn_add(edge, v(-1, 0, -1)); edge = rn_add(edge, v(1, 0, -1));
  edge = rn_add(edge, v(-1, 0, 1)); edge = rn_add(edge, v(1, 0, 1));
  edge = rn_add(edge, v(0, -1, -1)); edge = rn_add(edge, v(0, 1, -1));
  edge = rn_add(edge, v(0, -1, 1)); edge = rn_add(edge, v(0, 1, 1));
  C corner = rn_add(v(-1, -1, -1), v(1, -1, -1));
  corner = rn_add(corner, v(-1, 1, -1)); corner = rn_add(corner, v(1, 1, -1));
  corner = rn_add(corner, v(-1, -1, 1)); corner = rn_add(corner, v(1, -1, 1));
  corner = rn_add(corner, v(-1, 1, 1)); corner = rn_add(corner, v(1, 1, 1));
  const C sum = rn_add(rn_add(rn_add(rn_mul(C(8), v(0, 0, 0)), rn_mul(C(4), face)), rn_mul(C(2), edge)), corner);
  return rn_mul(sum, C(1) / C(64));
}
// The pass at f[0]; sx, sy, sz are the neighbours' distances.
template <class C>
__device__ __forceinline__ C smooth_value(const C* f, int sx, int sy, int sz, int op, C alpha, C beta) {
  return smooth_sum<C>([&](int a, int b, int c) { return f[a * sx + b * sy + c * sz]; }, op, alpha, beta);
}

// A tile of unique nodes with `halo` more on each side. An axis of one cell is
// held once: its neighbours are the node itself (stride 0).
struct SmoothTile {
  int halo;
  int e[3];       // extents
  int h[3];       // the tile's first node (0 or halo)
  int s[3];       // strides (0 on an axis of one cell)
  int size;       // nodes held
  __host__ __device__ SmoothTile(int nx, int ny, int nz, int tx, int ty, int tz, int halo_) : halo(halo_) {
    const int n[3] = {nx, ny, nz}, t[3] = {tx, ty, tz};
    size = 1;
    for (int a = 0; a < 3; ++a) {
      h[a] = n[a] > 1 ? halo : 0;
      e[a] = n[a] > 1 ? t[a] + 2 * halo : 1;
      s[a] = n[a] > 1 ? size : 0;
      size *= e[a];
    }
  }
};

// `passes` passes over the components in a (component c at c * size),
// alternating with b, by `warps` warps of the CTA (warp: this warp's number,
// or any number from `warps` on to take no rows); pass m leaves the nodes at
// least m from the edge. A CTA barrier follows each pass. flag(x, y, z) is
// called for a nonfinite result. Returns the array of the last pass.
template <class C, class Flag>
__device__ __forceinline__ C* smooth_passes(const SmoothTile& t, int components, C* a, C* b, int passes, int op,
                                            double alpha_d, int warp, int warps, Flag&& flag) {
  const C alpha = C(alpha_d), beta = (C(1) - alpha) / C(6);
  const int lane = threadIdx.x & 31;
  for (int m = 1; m <= passes; ++m) {
    const int mx = t.s[0] ? m : 0, my = t.s[1] ? m : 0, mz = t.s[2] ? m : 0;
    const int ny = t.e[1] - 2 * my, rows = ny * (t.e[2] - 2 * mz);
    for (int r = warp; r < components * rows; r += warps) {
      const int c = r / rows, rest = r - c * rows, z = mz + rest / ny, y = my + rest % ny;
      const int at = c * t.size + y * t.e[0] + z * t.e[0] * t.e[1];
      for (int x = mx + lane; x < t.e[0] - mx; x += 32) {
        const C value = smooth_value<C>(a + at + x, t.s[0], t.s[1], t.s[2], op, alpha, beta);
        b[at + x] = value;
        if (!isfinite(value)) flag(x, y, z);
      }
    }
    __syncthreads();
    C* swap = a;
    a = b;
    b = swap;
  }
  return a;
}

}  // namespace tpicb200
