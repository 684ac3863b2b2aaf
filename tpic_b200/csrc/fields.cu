// Field kernels of the cycle: periodic node/cell ghost fills, cell-to-node
// B, the Maxwell right-hand side, the E/B advance and the energy reductions.
// All are HBM-streaming stencils, one thread per target sample.
#include "kernels.cuh"
#include "smoothing.cuh"
#include "stencils.cuh"

namespace tpicb200 {
namespace {

// Ghost nodes take their periodic images; component blockIdx.y. The shell
// index is decoded in 32-bit arithmetic (launch_node_ghosts checks that the
// shell holds fewer than 2^31 nodes): on a grid one cell thick the ghost
// planes hold three times the interior, and 64-bit division per node took
// 23 us per fill at 512 x 512 x 1.
template <class T>
__global__ void __launch_bounds__(256) node_fill_kernel(Geom g, T* __restrict__ f) {
  wait_for_predecessor();
  const uint32_t shell = uint32_t(shell_count(g));
  T* fc = f + (long long)blockIdx.y * g.nodes;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < shell; t += gridDim.x * blockDim.x) {
    int i, j, k;
    shell_coordinates32(g, t, i, j, k);
    fc[g.node(i, j, k)] = fc[g.node(wrap_index(i, g.nx), wrap_index(j, g.ny), wrap_index(k, g.nz))];
  }
}

// Ghost cells -1 and n per axis take cells n-1 and 0.
template <class T>
__global__ void __launch_bounds__(256) cell_fill_kernel(Geom g, T* __restrict__ f) {
  const long long zs = (long long)g.CX * g.CY, ys = (long long)g.CX * g.nz, xs = (long long)g.ny * g.nz;
  const long long shell = 2 * (zs + ys + xs), total = 3 * shell;
  for (long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; t0 < total;
       t0 += (long long)gridDim.x * blockDim.x) {
    const long long c = t0 / shell;
    long long t = t0 - c * shell;
    int i, j, k;
    if (t < 2 * zs) {
      const int p = int(t / zs);
      const long long r = t - p * zs;
      k = p == 0 ? -1 : g.nz;
      i = int(r % g.CX) - 1;
      j = int(r / g.CX) - 1;
    } else if ((t -= 2 * zs) < 2 * ys) {
      const int p = int(t / ys);
      const long long r = t - p * ys;
      j = p == 0 ? -1 : g.ny;
      i = int(r % g.CX) - 1;
      k = int(r / g.CX);
    } else {
      t -= 2 * ys;
      const int p = int(t / xs);
      const long long r = t - p * xs;
      i = p == 0 ? -1 : g.nx;
      j = int(r % g.ny);
      k = int(r / g.ny);
    }
    f[c * g.cells + g.cell(i, j, k)] =
        f[c * g.cells + g.cell(wrap_index(i, g.nx), wrap_index(j, g.ny), wrap_index(k, g.nz))];
  }
}

// cell_to_node_average in Compute::Magnetic (ecsim/fields/cell_to_node.hpp:19-32,
// ecsim/fields/cell_to_node_device.hpp:17-38) at every stored node, duplicates
// and ghosts as their unique node (no ghost fill behind it); component
// blockIdx.y.
template <class C, class T>
__global__ void __launch_bounds__(256) cell_to_node_kernel(Geom g, const T* __restrict__ cellf, T* __restrict__ node) {
  const T* f = cellf + blockIdx.y * g.cells;
  T* out = node + blockIdx.y * g.nodes;
  const uint32_t total = uint32_t(g.nodes), NX = uint32_t(g.NX), NY = uint32_t(g.NY);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const uint32_t row = t / NX;
    const int i = wrap_index(int(t - row * NX) - 1, g.nx), j = wrap_index(int(row % NY) - 1, g.ny),
              k = wrap_index(int(row / NY) - 1, g.nz);
    const C v = (C(f[g.cell(i - 1, j - 1, k - 1)]) + C(f[g.cell(i, j - 1, k - 1)]) +
                 C(f[g.cell(i - 1, j, k - 1)]) + C(f[g.cell(i, j, k - 1)]) +
                 C(f[g.cell(i - 1, j - 1, k)]) + C(f[g.cell(i, j - 1, k)]) +
                 C(f[g.cell(i - 1, j, k)]) + C(f[g.cell(i, j, k)])) * C(0.125);
    out[t] = T(v);
  }
}

// rhs = ((1*E + delta*curl_C2N(B)) + (-k)*J) in Compute::Electric
// (MaxwellOperator::complete_rhs, ecsim/maxwell/maxwell_device.hpp:152-172).
template <class C, class T, class TJ>
__global__ void __launch_bounds__(256) rhs_kernel(Geom g, C delta, C kfac, const T* __restrict__ e,
                                                  const T* __restrict__ bcell, const TJ* __restrict__ j,
                                                  double* __restrict__ rhs) {
  const C inv[3] = {C(g.inv[0]), C(g.inv[1]), C(g.inv[2])};
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < g.interior;
       t += (long long)gridDim.x * blockDim.x) {
    int i, jj, k;
    interior_node_coordinates(g, t, i, jj, k);
    C cb[3];
    curl_c2n_at<C>(g, bcell, i, jj, k, inv, cb);
    const long long at = g.node(i, jj, k);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long p = c * g.nodes + at;
      rhs[p] = double((C(1) * C(e[p]) + delta * cb[c]) + (-kfac) * C(j[p]));
    }
  }
}

// The field advance: the E update over the interior nodes
// (field_vector_linear_combination, two terms) and Faraday's
// next = 1*B + faraday*curl_N2C(theta) in Compute::Magnetic over all cells
// (faraday_update_kernel, ecsim/maxwell/field_update_device.hpp:25-44), each
// cell stored at its periodic copies too.
template <class C, class T>
__global__ void __launch_bounds__(256) advance_kernel(Geom g, C a, C b, bool copy, T* __restrict__ e, C faraday,
                                                      const T* __restrict__ bcell, const double* __restrict__ th,
                                                      T* __restrict__ next, uint32_t* invalid) {
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  for (long long t = first; t < g.interior; t += stride) {
    int i, j, k;
    interior_node_coordinates(g, t, i, j, k);
    const long long at = g.node(i, j, k);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long p = c * g.nodes + at;
      const T value = copy ? T(th[p]) : T(a * C(th[p]) + b * C(e[p]));
      e[p] = value;
      if (!isfinite(value)) atomicAdd(invalid, 1u);
    }
  }
  const C inv[3] = {C(g.inv[0]), C(g.inv[1]), C(g.inv[2])};
  const long long cells = (long long)g.nx * g.ny * g.nz;
  for (long long t = first; t < cells; t += stride) {
    const uint32_t u = uint32_t(t), nx = uint32_t(g.nx), row = u / nx;
    const int i = int(u - row * nx), j = int(row % uint32_t(g.ny)), k = int(row / uint32_t(g.ny));
    C cu[3];
    curl_n2c_at<C>(g, th, i, j, k, inv, cu);
    const long long at = g.cell(i, j, k);
    T value[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      value[c] = T(C(1) * C(bcell[c * g.cells + at]) + faraday * cu[c]);
      if (!isfinite(value[c])) atomicAdd(invalid, 1u);
    }
    // The copies of cell i on an axis of n: i + m n within -1 .. n.
    for (int kk = k - (k + 1) / g.nz * g.nz; kk <= g.nz; kk += g.nz)
      for (int jj = j - (j + 1) / g.ny * g.ny; jj <= g.ny; jj += g.ny)
        for (int ii = i - (i + 1) / g.nx * g.nx; ii <= g.nx; ii += g.nx)
#pragma unroll
          for (int c = 0; c < 3; ++c) next[c * g.cells + g.cell(ii, jj, kk)] = value[c];
  }
}

template <class T>
__global__ void __launch_bounds__(256) field_energy_kernel(Geom g, const T* __restrict__ e,
                                                           const T* __restrict__ b, double* partials) {
  __shared__ double scratch[2][8];
  const long long unique = (long long)g.nx * g.ny * g.nz;
  double we = 0, wb = 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < unique;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = int(t % g.nx), j = int((t / g.nx) % g.ny), k = int(t / ((long long)g.nx * g.ny));
    const long long n = g.node(i, j, k), c = g.cell(i, j, k);
    const double ex = e[n], ey = e[g.nodes + n], ez = e[2 * g.nodes + n];
    const double bx = b[c], by = b[g.cells + c], bz = b[2 * g.cells + c];
    we += ex * ex + ey * ey + ez * ez;
    wb += bx * bx + by * by + bz * bz;
  }
  we = block_sum<256>(we, scratch[0]);
  wb = block_sum<256>(wb, scratch[1]);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = we;
    partials[gridDim.x + blockIdx.x] = wb;
  }
}

template <class Vel>
__global__ void __launch_bounds__(256) species_kernel(const Vel* __restrict__ u, const Vel* __restrict__ v,
                                                      const Vel* __restrict__ w, const double* __restrict__ q,
                                                      uint32_t count, double inverse_qom, double* partials) {
  __shared__ double scratch[5][8];
  double s[5] = {0, 0, 0, 0, 0};
  for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < count; n += gridDim.x * blockDim.x) {
    const double weight = q[n], mass = weight * inverse_qom;
    const double vx = u[n], vy = v[n], vz = w[n];
    s[0] += 0.5 * mass * (vx * vx + vy * vy + vz * vz);
    s[1] += weight;
    s[2] += mass * vx;
    s[3] += mass * vy;
    s[4] += mass * vz;
  }
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    const double total = block_sum<256>(s[r], scratch[r]);
    if (threadIdx.x == 0) partials[r * gridDim.x + blockIdx.x] = total;
  }
}

// One block per row: out[row] = sum of the row's `count` partials; rows at or
// above `filled` store zero (reduce_block_partials_kernel,
// device/block_reduction_device.hpp:23-44).
__global__ void __launch_bounds__(256) reduce_rows_kernel(const double* __restrict__ partials, double* out,
                                                          int row_stride, int count, int filled) {
  wait_for_predecessor();
  __shared__ double scratch[8];
  const int row = blockIdx.x;
  if (row >= filled) {
    if (threadIdx.x == 0) out[row] = 0;
    return;
  }
  double sum = 0;
  for (int i = threadIdx.x; i < count; i += blockDim.x) sum += partials[(long long)row * row_stride + i];
  sum = block_sum<256>(sum, scratch);
  if (threadIdx.x == 0) out[row] = sum;
}

__global__ void __launch_bounds__(256) reduce_report_kernel(ReportRows rows, double* out) {
  __shared__ double scratch[8];
  const int row = blockIdx.x, sp = (row - 2) / 5;
  const double* from = row < 2 ? rows.fields + (long long)row * rows.blocks
                               : rows.movers + (long long)(row - 2) * kMoverPartials;
  const int count = row < 2 ? rows.blocks : rows.written[sp];
  double sum = 0;
  for (int i = threadIdx.x; i < count; i += blockDim.x) sum += from[i];
  sum = block_sum<256>(sum, scratch);
  if (threadIdx.x == 0) out[row] = sum;
}

template <class T>
__global__ void __launch_bounds__(256) copy_node_kernel(long long total, const T* __restrict__ in,
                                                        double* __restrict__ out) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x)
    out[t] = double(in[t]);
}

}  // namespace

cudaError_t launch_node_ghosts(const Geom& g, double* f, int components, cudaStream_t s, bool programmatic) {
  if (shell_count(g) >= (1LL << 31)) return cudaErrorInvalidValue;
  const dim3 blocks(grid_for(shell_count(g), 256), unsigned(components));
  count_launches(1);
  if (programmatic) return launch_programmatic(node_fill_kernel<double>, blocks, 256, 0, s, g, f);
  node_fill_kernel<double><<<blocks, 256, 0, s>>>(g, f);
  return cudaGetLastError();
}

cudaError_t launch_cell_ghosts(int precision, const Geom& g, void* f, cudaStream_t s) {
  const long long shell = 2 * ((long long)g.CX * g.CY + (long long)g.CX * g.nz + (long long)g.ny * g.nz);
  const unsigned blocks = grid_for(3 * shell, 256);
  if (precision == TPICB200_PRECISION_DOUBLE) cell_fill_kernel<double><<<blocks, 256, 0, s>>>(g, (double*)f);
  else cell_fill_kernel<float><<<blocks, 256, 0, s>>>(g, (float*)f);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_cell_to_node(int precision, const Geom& g, const void* cellf, void* node, cudaStream_t s) {
  if (g.nodes >= (1LL << 32)) return cudaErrorInvalidValue;
  const dim3 blocks(grid_for(g.nodes, 256), 3);
  if (precision == TPICB200_PRECISION_DOUBLE)
    cell_to_node_kernel<double, double><<<blocks, 256, 0, s>>>(g, (const double*)cellf, (double*)node);
  else
    cell_to_node_kernel<float, float><<<blocks, 256, 0, s>>>(g, (const float*)cellf, (float*)node);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_rhs(int precision, const Geom& g, double delta, double kfac, const void* e,
                       const void* bcell, const void* j, double* rhs, cudaStream_t s, bool j_double) {
  const unsigned blocks = grid_for(g.interior, 256);
  if (precision == TPICB200_PRECISION_DOUBLE)
    rhs_kernel<double, double, double><<<blocks, 256, 0, s>>>(g, delta, kfac, (const double*)e,
                                                             (const double*)bcell, (const double*)j, rhs);
  else if (j_double)
    rhs_kernel<float, float, double><<<blocks, 256, 0, s>>>(g, float(delta), float(kfac), (const float*)e,
                                                           (const float*)bcell, (const double*)j, rhs);
  else
    rhs_kernel<float, float, float><<<blocks, 256, 0, s>>>(g, float(delta), float(kfac), (const float*)e,
                                                          (const float*)bcell, (const float*)j, rhs);
  count_launches(1);
  return cudaGetLastError();
}

// `passes` smoothing passes of a double node field into another, the tile and
// its halo in shared memory (blockIdx.x a tile of unique nodes, blockIdx.y a
// component). Neighbours
// are read from the unique nodes by their periodic index, and every stored
// copy of a node is written, so no ghost fill is needed before, between or
// after. One launch per pass with a ghost fill behind it took 12 launches for
// the default six passes, some 55 us on 256 x 128 x 1, where the passes
// themselves are 1 us each; the halo costs (32 + 12)(8 + 12) / (32 x 8) = 3.4
// times the nodes there. Grids thicker than one cell
// on every axis take smooth_pass_kernel: halos all around cost more than a
// launch a pass (smoothed FP32 solve of 64^3 with three passes on 16 x 8 x 8
// tiles 7.0 ms, with one or two 9.1 and 7.2, with passes and ghost fills 4.4,
// now 3.9).
constexpr int kSmoothThreads = 256;

template <class C>
__global__ void __launch_bounds__(kSmoothThreads) smooth_tile_kernel(Geom g, SmoothTile t, int tx, int ty, int tz,
                                                                     int passes, int op, double alpha,
                                                                     const double* __restrict__ src,
                                                                     double* __restrict__ dst, uint32_t* invalid) {
  extern __shared__ __align__(16) uint8_t smooth_smem[];
  C* a = reinterpret_cast<C*>(smooth_smem);
  C* b = a + t.size;
  src += blockIdx.y * g.nodes;
  dst += blockIdx.y * g.nodes;
  const int tiles_x = (g.nx + tx - 1) / tx, tiles_y = (g.ny + ty - 1) / ty;
  const int row = blockIdx.x / tiles_x;
  const int i0 = (blockIdx.x - row * tiles_x) * tx, j0 = (row % tiles_y) * ty, k0 = (row / tiles_y) * tz;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = kSmoothThreads / 32;
  const int rows = t.e[1] * t.e[2];
  for (int r = warp; r < rows; r += warps) {
    const int z = r / t.e[1], y = r - z * t.e[1];
    const long long at = g.node(0, wrap_index(j0 - t.h[1] + y, g.ny), wrap_index(k0 - t.h[2] + z, g.nz));
    for (int x = lane; x < t.e[0]; x += 32) a[r * t.e[0] + x] = C(src[at + wrap_index(i0 - t.h[0] + x, g.nx)]);
  }
  __syncthreads();
  const int nx = min(tx, g.nx - i0), ny = min(ty, g.ny - j0), nz = min(tz, g.nz - k0);
  const C* out = smooth_passes<C>(t, 1, a, b, passes, op, alpha, warp, warps, [&](int x, int y, int z) {
    x -= t.h[0];
    y -= t.h[1];
    z -= t.h[2];
    if (invalid && x >= 0 && x < nx && y >= 0 && y < ny && z >= 0 && z < nz) atomicAdd(invalid, 1u);
  });
  for (int r = warp; r < ny * nz; r += warps) {
    const int z = r / ny, y = r - z * ny, j = j0 + y, k = k0 + z;
    for (int x = lane; x < nx; x += 32) {
      const int i = i0 + x;
      const double v = double(out[(x + t.h[0]) + t.e[0] * ((y + t.h[1]) + t.e[1] * (z + t.h[2]))]);
      // The copies of node i on an axis of n: i + m n within -1 .. n + 1.
      for (int kk = k - (k + 1) / g.nz * g.nz; kk <= g.nz + 1; kk += g.nz)
        for (int jj = j - (j + 1) / g.ny * g.ny; jj <= g.ny + 1; jj += g.ny)
          for (int ii = i - (i + 1) / g.nx * g.nx; ii <= g.nx + 1; ii += g.nx) dst[g.node(ii, jj, kk)] = v;
    }
  }
}

// One pass at every stored node, ghosts as their unique node (blockIdx.y a
// component), so no ghost fill follows.
template <class C>
__global__ void __launch_bounds__(kSmoothThreads) smooth_pass_kernel(Geom g, int op, C alpha, C beta,
                                                                     const double* __restrict__ src,
                                                                     double* __restrict__ dst, uint32_t* invalid) {
  src += blockIdx.y * g.nodes;
  dst += blockIdx.y * g.nodes;
  const uint32_t total = uint32_t(g.nodes), NX = uint32_t(g.NX), NY = uint32_t(g.NY);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const uint32_t row = t / NX;
    const int a = int(t - row * NX) - 1, b = int(row % NY) - 1, c = int(row / NY) - 1;
    const int i = wrap_index(a, g.nx), j = wrap_index(b, g.ny), k = wrap_index(c, g.nz);
    // The neighbours' unique indexes along each axis.
    const int x[3] = {i == 0 ? g.nx - 1 : i - 1, i, i + 1 == g.nx ? 0 : i + 1};
    const int y[3] = {j == 0 ? g.ny - 1 : j - 1, j, j + 1 == g.ny ? 0 : j + 1};
    const int z[3] = {k == 0 ? g.nz - 1 : k - 1, k, k + 1 == g.nz ? 0 : k + 1};
    const C value = smooth_sum<C>([&](int dx, int dy, int dz) { return C(src[g.node(x[dx + 1], y[dy + 1], z[dz + 1])]); },
                                  op, alpha, beta);
    dst[t] = double(value);
    if (invalid && a == i && b == j && c == k && !isfinite(value)) atomicAdd(invalid, 1u);
  }
}

template <class C>
cudaError_t launch_smooth_typed(const Geom& g, int niter, int op, double alpha, const double* src, double* out,
                                double* tmp, uint32_t* invalid, cudaStream_t s) {
  if (g.nx > 1 && g.ny > 1 && g.nz > 1) {
    if (g.nodes >= (1LL << 32)) return cudaErrorInvalidValue;
    const C a = C(alpha), beta = (C(1) - a) / C(6);
    for (int left = niter; left > 0; --left) {
      double* to = left % 2 == 1 ? out : tmp;
      smooth_pass_kernel<C><<<dim3(grid_for(g.nodes, kSmoothThreads), 3), kSmoothThreads, 0, s>>>(g, op, a, beta, src,
                                                                                                  to, invalid);
      count_launches(1);
      src = to;
    }
    return cudaGetLastError();
  }
  // Passes a launch: as many as a halo is worth, split evenly.
  // Two axes of the tile with eight passes' halo fit a kernel's default shared
  // memory (a raised limit would be one for all contexts).
  constexpr int most = 8;
  static_assert(2 * (32 + 2 * most) * (8 + 2 * most) * sizeof(C) <= 48 * 1024, "the tile and its copy");
  const int launches = (niter + most - 1) / most;
  const int tx = 32, ty = g.ny == 1 ? 1 : 8, tz = g.nz == 1 ? 1 : 8;
  const long long tiles = (long long)((g.nx + tx - 1) / tx) * ((g.ny + ty - 1) / ty) * ((g.nz + tz - 1) / tz);
  if (tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
  int done = 0;
  for (int l = 0; l < launches; ++l) {
    const int passes = (niter - done + launches - l - 1) / (launches - l);
    done += passes;
    const SmoothTile t(g.nx, g.ny, g.nz, tx, ty, tz, passes);
    const size_t bytes = size_t(2) * t.size * sizeof(C);
    double* to = (launches - l) % 2 == 1 ? out : tmp;
    smooth_tile_kernel<C><<<dim3(unsigned(tiles), 3), kSmoothThreads, bytes, s>>>(g, t, tx, ty, tz, passes, op, alpha, src, to,
                                                                         invalid);
    count_launches(1);
    src = to;
  }
  return cudaGetLastError();
}

// S^n(src) into out with its ghosts filled (complete_smoothing,
// ecsim/maxwell/maxwell_device.hpp:455-487 on a periodic domain); the launches
// alternate between out and tmp so that the last lands in out. Neither out
// nor tmp may alias src. double_arithmetic selects the pass arithmetic (the
// reference's Arithmetic / Compute::Electric). invalid (may be null) counts
// nonfinite smoothed values, as the reference's kernel flags them
// (node_smoothing_device.hpp:30-36).
cudaError_t launch_smooth(bool double_arithmetic, const Geom& g, int niter, int op, double alpha,
                          const double* src, double* out, double* tmp, uint32_t* invalid, cudaStream_t s) {
  if (niter <= 0 || src == out || src == tmp || out == tmp) return cudaErrorInvalidValue;
  return double_arithmetic ? launch_smooth_typed<double>(g, niter, op, alpha, src, out, tmp, invalid, s)
                           : launch_smooth_typed<float>(g, niter, op, alpha, src, out, tmp, invalid, s);
}

// A node field of float or double into double (every entry, ghosts included).
__global__ void __launch_bounds__(256) widen_kernel(const float* __restrict__ in, double* __restrict__ out,
                                                    long long n) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    out[t] = double(in[t]);
}
cudaError_t launch_widen(int precision, const Geom& g, const void* in, double* out, cudaStream_t s) {
  const long long n = 3 * g.nodes;
  if (precision == TPICB200_PRECISION_DOUBLE)
    return cudaMemcpyAsync(out, in, size_t(n) * 8, cudaMemcpyDeviceToDevice, s);
  widen_kernel<<<grid_for(n, 256), 256, 0, s>>>((const float*)in, out, n);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_field_advance(int precision, const Geom& g, double theta_value, double faraday,
                                 void* e, const void* bcell, const double* etheta, void* bnext,
                                 uint32_t* invalid, cudaStream_t s) {
  const bool copy = fabs(theta_value - 1.0) < 1e-10;
  const unsigned blocks = grid_for(g.interior, 256);
  if (precision == TPICB200_PRECISION_DOUBLE) {
    const double a = 1.0 / theta_value, b = -(1.0 - theta_value) / theta_value;
    advance_kernel<double, double><<<blocks, 256, 0, s>>>(g, a, b, copy, (double*)e, faraday, (const double*)bcell,
                                                         etheta, (double*)bnext, invalid);
  } else {
    const float th = float(theta_value);
    const float a = 1.0f / th, b = -(1.0f - th) / th;
    advance_kernel<float, float><<<blocks, 256, 0, s>>>(g, a, b, copy, (float*)e, float(faraday), (const float*)bcell,
                                                       etheta, (float*)bnext, invalid);
  }
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_field_energy(int precision, const Geom& g, const void* e, const void* bcell,
                                double* partials, int blocks, cudaStream_t s) {
  if (precision == TPICB200_PRECISION_DOUBLE)
    field_energy_kernel<double><<<blocks, 256, 0, s>>>(g, (const double*)e, (const double*)bcell, partials);
  else
    field_energy_kernel<float><<<blocks, 256, 0, s>>>(g, (const float*)e, (const float*)bcell, partials);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_species_scalars(int precision, const tpicb200_particles* p, double qom,
                                   double* partials, int blocks, cudaStream_t s) {
  if (precision == TPICB200_PRECISION_DOUBLE)
    species_kernel<double><<<blocks, 256, 0, s>>>((const double*)p->u, (const double*)p->v,
                                                  (const double*)p->w, p->q, p->count, 1.0 / qom, partials);
  else
    species_kernel<float><<<blocks, 256, 0, s>>>((const float*)p->u, (const float*)p->v,
                                                 (const float*)p->w, p->q, p->count, 1.0 / qom, partials);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_reduce_rows(const double* partials, double* out, int rows, int row_stride, int count,
                               int filled, cudaStream_t s, bool programmatic) {
  count_launches(1);
  if (programmatic)
    return launch_programmatic(reduce_rows_kernel, unsigned(rows), 256, 0, s, partials, out, row_stride, count,
                               filled);
  reduce_rows_kernel<<<rows, 256, 0, s>>>(partials, out, row_stride, count, filled);
  return cudaGetLastError();
}

cudaError_t launch_reduce_report(const ReportRows& rows, int ns, double* out, cudaStream_t s) {
  reduce_report_kernel<<<2 + 5 * ns, 256, 0, s>>>(rows, out);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_copy_node_field(const Geom& g, const void* in, int in_double, double* out, cudaStream_t s) {
  const long long total = 3 * g.nodes;
  if (in_double) copy_node_kernel<double><<<grid_for(total, 256), 256, 0, s>>>(total, (const double*)in, out);
  else copy_node_kernel<float><<<grid_for(total, 256), 256, 0, s>>>(total, (const float*)in, out);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace tpicb200
