// The GMRES restart cycle of a small grid as one resident kernel.
//
// On grids of up to some ten thousand nodes an Arnoldi step is short work
// behind nine launches: 36 us a step on a 1024 x 1 x 1 grid, 55 us on 256 x
// 128 x 1, where the mass matrix and the vectors stay in L2. Here every CTA
// owns the unique nodes of its tiles for the whole cycle, keeps its rows of the
// Krylov basis in shared memory where they fit, and the CTAs meet at two grid
// barriers a step:
//   A  the operator on the last vector (neighbours' rows read from one global
//      vector), and the dots of its image with the owned basis rows;
//      -- barrier: the dots of all CTAs --
//   B  Gram-Schmidt of the owned rows, the squared norm; the unnormalized
//      vector goes to the global vector;
//      -- barrier: the norm of all CTAs; each CTA scales what it reads --
// The Hessenberg column is rotated by one more warp while the others
// orthogonalize; every CTA does so from the same sums in the same order, so
// all take the same stopping decision. Vectors hold the unique nodes only; a
// row of node 0 on an axis stands for its duplicate at node n too, so it
// counts twice per such axis in the dots and norms, which are then those over
// the interior nodes. All sums run in a fixed order.
//
// A CTA has one tile, or several on grids of more tiles than CTAs fit. A tile of
// TN (32..256, a power of two) nodes has 256 / TN threads a node
// that share the 27 mass blocks: small grids take small tiles, so that every
// SM has one.
//
// With one CTA an SM, the rest of its shared memory keeps the mass blocks of its
// threads through the cycle, as many as fit, and the sums over columns run side
// by side: a step is bound by the latencies of its phases, and the 4 dependent
// block loads of a thread took a quarter of it. With two CTAs an SM, which hide
// each other's latencies and share L1, both made steps longer (40^3 mixed 528
// against 444 us a solve, 512 x 512 x 1 2.03 against 1.81 ms).
//
// With smoothing (grids one cell thick along z) a tile holds passes + 1 more
// nodes on each side and takes the passes in shared memory: the smoothed
// vector's mass response goes to a global vector, and after one more barrier
// the response is smoothed the same way.
//
// A grid of at most 16 tiles is launched as one cluster, whose hardware barrier
// takes the place of the grid barrier. Otherwise the launch is cooperative
// (all CTAs resident). A grid barrier that does not
// complete within its polls makes its CTA set ctl->failed and leave; the
// others then run out at theirs, and the solve fails. The cluster barrier is
// the hardware's: a cluster's CTAs start together, and one that has left is not
// waited for.
#pragma once

#include "common.cuh"
#include "grid_barrier.cuh"
#include "smoothing.cuh"
#include "stencils.cuh"

namespace tpicb200 {
namespace {

// Device-side state of one restart cycle's Arnoldi steps.
struct ArnoldiControl {
  int col;        // the step the step kernels take (0-based)
  int completed;  // steps completed in this cycle
  int columns;    // step limit of this cycle
  int stop;       // 0 running; 1 stopped (tolerance, breakdown or limit); 2 nonfinite estimate
  int breakdown;  // the last step's subdiagonal was zero
  int failed;     // a grid barrier of the resident kernel ran out of polls
  double tolerance;
};

constexpr int kResidentNodeThreads = 256;
constexpr int kResidentThreads = kResidentNodeThreads + 32;  // and the warp that rotates the Hessenberg column
constexpr int kResidentRestart = 32;                         // longest restart cycle (four columns a warp)

struct ResidentPlan {
  Geom g;
  int tx, ty, tz;          // tile, powers of two; tx*ty*tz = nodes
  int nodes, parts, shift; // nodes of a tile, threads per node, log2 nodes
  int tiles_x, tiles_y, tiles;
  int slots;               // tiles per CTA: tile blockIdx.x + slot * gridDim.x
  bool cluster;            // the grid is one cluster
  bool shared_basis;       // basis rows in shared memory, else in `basis`
  int kept;                // stencils of each thread whose mass blocks a cycle keeps in shared memory
  double delta, kfac, inv_volume;
  const void* mass;
  void* vector;            // [3][unique] S: the last unnormalized vector
  void* basis;             // owner-private rows, slots * 3 * nodes of each CTA per column
  double* x;               // [3][unique]
  double* b;
  double* r;
  double* values;          // |r|^2 and (start) |b|^2
  double* partials;        // kResidentRestart + 2 rows of gridDim.x
  ArnoldiControl* ctl;
  unsigned* barrier;       // kGridBarrierWords
  uint32_t polls;          // of its waits
  int restart, columns;
  double tolerance;        // of this cycle's residual estimate
  double accept;           // start: the relative tolerance; cycle: the absolute one
  const void* e;           // start: E, B and J, or the right-hand side itself with a zero guess
  const void* bcell;
  const void* j;
  const double* rhs;
  int smooth, smooth_op;   // smoothing passes (0: none), operator
  double smooth_alpha;
  double* response;        // [3][unique]: the smoothed vector's mass response
  uint32_t* invalid;       // counts nonfinite smoothed values
  double* etheta;          // the solution with its ghosts, written when the residual is accepted
};

// Shared memory of a plan with arithmetic up to double: bytes per array.
struct ResidentShared {
  int halo, cells;                 // nodes and cells a tile stages
  size_t vs, cs, part, h, hcol, rot, sums, basis, image, unode, mult, table, ctable, offsets, smooth, mass, total;
};
// The tile and halo of the smoothing passes (the mass product reads one more node).
inline __host__ __device__ SmoothTile resident_smooth_tile(const ResidentPlan& p) {
  return SmoothTile(p.g.nx, p.g.ny, p.g.nz, p.tx, p.ty, p.tz, p.smooth + 1);
}
inline __host__ __device__ ResidentShared resident_shared(const ResidentPlan& p, size_t scalar) {
  ResidentShared s;
  s.halo = (p.tx + 2) * (p.ty + 2) * (p.tz + 2);
  s.cells = (p.tx + 1) * (p.ty + 1) * (p.tz + 1);
  const int m = kResidentRestart;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += (bytes + 15) / 16 * 16;
    return here;
  };
  s.vs = take(size_t(3) * s.halo * 8);
  s.cs = take(size_t(3) * s.cells * 8);
  s.part = take(size_t(3) * kResidentNodeThreads * 8);
  s.h = take(size_t(m) * (m + 1) * 8);
  s.hcol = take(size_t(m + 1) * 8);
  s.rot = take(size_t(4) * (m + 1) * 8);  // cosines, sines, right-hand side, coefficients
  s.sums = take(size_t(kResidentThreads / 32 + 2) * 2 * 8);  // per warp, then the step's diagonal and decision
  s.basis = take(p.shared_basis ? size_t(p.restart + 1) * p.slots * 3 * p.nodes * scalar : 0);
  s.image = take(size_t(p.slots) * 3 * p.nodes * scalar);
  s.unode = take(size_t(p.slots) * p.nodes * 4);
  s.mult = take(size_t(p.slots) * p.nodes);
  s.table = take(size_t(s.halo) * 4);
  s.ctable = take(size_t(s.cells) * 4);
  s.offsets = take(size_t(14) * sizeof(int2));
  s.smooth = take(p.smooth ? size_t(6) * resident_smooth_tile(p).size * 8 : 0);
  s.mass = take(size_t(p.kept) * 18 * kResidentNodeThreads * scalar);  // [stencil][18 entries][thread]
  s.total = at;
  return s;
}

// stencil_offset, indexed at run time.
__constant__ int8_t kResidentOffsets[14][3] = {{0, 0, 0},  {1, 0, 0},  {0, 1, 0},  {0, 0, 1},  {1, 1, 0},
                                               {1, -1, 0}, {1, 0, 1},  {1, 0, -1}, {0, 1, 1},  {0, 1, -1},
                                               {1, -1, 1}, {1, 1, -1}, {-1, 1, 1}, {1, 1, 1}};

// kCtas: the CTAs an SM holds, which sets a thread's registers.
template <class S, class Mass, class Fld, bool kTranspose, bool kSmooth, int kCtas>
struct Resident {
  const ResidentPlan& p;
  uint8_t* smem;
  const ResidentShared L;
  GridBarrier<false> barrier;

  __device__ Resident(const ResidentPlan& plan, uint8_t* s)
      : p(plan), smem(s), L(resident_shared(plan, sizeof(S))), barrier(plan.barrier, GridWaits{plan.polls, 0}) {}

  template <class T> __device__ __forceinline__ T* at(size_t offset) const { return reinterpret_cast<T*>(smem + offset); }
  __device__ __forceinline__ long long unique() const { return (long long)p.g.nx * p.g.ny * p.g.nz; }
  __device__ __forceinline__ S* basis(int col) const {
    const int rows = p.slots * 3 * p.nodes;
    return p.shared_basis ? at<S>(L.basis) + col * rows
                          : static_cast<S*>(p.basis) + ((long long)col * gridDim.x + blockIdx.x) * rows;
  }
  __device__ __forceinline__ int tile_of(int slot) const { return int(blockIdx.x) + slot * int(gridDim.x); }
  __device__ __forceinline__ void origin(int slot, int& i0, int& j0, int& k0) const {
    const int tile = tile_of(slot), row = tile / p.tiles_x;
    i0 = (tile - row * p.tiles_x) * p.tx;
    k0 = row / p.tiles_y;
    j0 = (row - k0 * p.tiles_y) * p.ty;
    k0 *= p.tz;
  }

  // All CTAs of the grid. False when it gave up (for every thread of the CTA),
  // which then ends; the host, which reads ctl->failed, clears the words.
  __device__ bool grid_barrier() {
    if (p.cluster) {
      asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
      return true;
    }
    if (barrier.wait()) return true;
    if (threadIdx.x == 0) p.ctl->failed = 1;
    return false;
  }
  __device__ void leave() {
    if (!p.cluster && threadIdx.x == 0) barrier.depart();
  }

  // Table of a slot's tile: the unique index of every staged node (-1 beyond
  // the grid's halo).
  __device__ void tables(int slot) {
    const int vx = p.tx + 2, vy = p.ty + 2;
    int i0, j0, k0;
    origin(slot, i0, j0, k0);
    const Geom& g = p.g;
    int* table = at<int>(L.table);
    for (int n = threadIdx.x; n < L.halo; n += kResidentThreads) {
      const int row = n / vx, i = i0 - 1 + n - row * vx, j = j0 - 1 + row % vy, k = k0 - 1 + row / vy;
      int u = -1;
      if (i <= g.nx && j <= g.ny && k <= g.nz) {
        const int wi = i < 0 ? i + g.nx : (i >= g.nx ? i - g.nx : i), wj = j < 0 ? j + g.ny : (j >= g.ny ? j - g.ny : j),
                  wk = k < 0 ? k + g.nz : (k >= g.nz ? k - g.nz : k);
        u = wi + g.nx * (wj + g.ny * wk);
      }
      table[n] = u;
    }
  }
  // The tables that hold for every tile: the staged base node of a cell, the
  // stencils' distances.
  __device__ void fixed_tables() {
    const int vx = p.tx + 2, vy = p.ty + 2, cx = p.tx + 1, cy = p.ty + 1;
    const Geom& g = p.g;
    int* ctable = at<int>(L.ctable);
    if (threadIdx.x < 14) {
      // A stencil's distance in the array the mass product reads, and in the mass.
      const int ox = kResidentOffsets[threadIdx.x][0], oy = kResidentOffsets[threadIdx.x][1],
                oz = kResidentOffsets[threadIdx.x][2];
      // On an axis of one cell the fold's copies hold the node's own blocks.
      const SmoothTile t = resident_smooth_tile(p);
      at<int2>(L.offsets)[threadIdx.x] =
          make_int2(kSmooth ? ox * t.s[0] + oy * t.s[1] + oz * t.s[2] : ox + vx * (oy + vy * oz),
                    int(g.mass_offset(g.nx > 1 ? ox : 0, g.ny > 1 ? oy : 0, g.nz > 1 ? oz : 0) * g.mvs));
    }
    for (int n = threadIdx.x; n < L.cells; n += kResidentThreads) {
      const int row = n / cx;
      ctable[n] = (n - row * cx) + vx * (row % cy + vy * (row / cy));
    }
  }

  // Node n of a slot's tile: coordinates, and whether it is in the grid.
  __device__ __forceinline__ bool node_of(int slot, int n, int& i, int& j, int& k) const {
    origin(slot, i, j, k);
    i += n & (p.tx - 1);
    const int row = n / p.tx;
    j += row & (p.ty - 1);
    k += row / p.ty;
    return tile_of(slot) < p.tiles && i < p.g.nx && j < p.g.ny && k < p.g.nz;
  }

  // The operator in arithmetic C: stage() reads the vector load(component,
  // unique index) over the tile and its halo (the node threads; a CTA barrier
  // follows), image() forms its rows. The products and their order are those
  // of maxwell_apply_kernel where a node has one thread; with more, their
  // partial sums are added in order.
  template <class C, class Load>
  __device__ __forceinline__ void stage(Load&& load) {
    if (threadIdx.x >= kResidentNodeThreads) return;
    C* vs = at<C>(L.vs);
    const int* table = at<int>(L.table);
    const int VN = L.halo;
    // Two nodes' values at a time: the loads wait for L2 once for both.
    for (int n = threadIdx.x; n < VN; n += 2 * kResidentNodeThreads) {
      const int other = n + kResidentNodeThreads;
      const int u = table[n], w = other < VN ? table[other] : -1;
      C v[2][3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        v[0][c] = u >= 0 ? C(load(c, u)) : C(0);
        v[1][c] = w >= 0 ? C(load(c, w)) : C(0);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        vs[c * VN + n] = v[0][c];
        if (other < VN) vs[c * VN + other] = v[1][c];
      }
    }
    if constexpr (kSmooth) stage_region<C>(resident_smooth_tile(p), load);
  }
  // The cell curls of the staged vector.
  template <class C>
  __device__ __forceinline__ void cell_curls() {
    const C* vs = at<C>(L.vs);
    C* cs = at<C>(L.cs);
    const int* ctable = at<int>(L.ctable);
    const int vx = p.tx + 2, vxy = vx * (p.ty + 2), VN = L.halo, CN = L.cells;
    const C inv[3] = {C(p.g.inv[0]), C(p.g.inv[1]), C(p.g.inv[2])};
    for (int n = threadIdx.x; n < CN; n += kResidentThreads) {
      const C* v = vs + ctable[n];
      C q[3][8];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const C* f = v + c * VN;
        q[c][0] = f[0];       q[c][1] = f[1];       q[c][2] = f[vx];       q[c][3] = f[vxy];
        q[c][4] = f[vx + 1];  q[c][5] = f[vxy + 1]; q[c][6] = f[vxy + vx]; q[c][7] = f[vxy + vx + 1];
      }
      auto dx = [&](const C* w) { return C(0.25) * inv[0] * (w[1] - w[0] + (w[5] - w[3]) + (w[4] - w[2]) + (w[7] - w[6])); };
      auto dy = [&](const C* w) { return C(0.25) * inv[1] * (w[2] - w[0] + (w[6] - w[3]) + (w[4] - w[1]) + (w[7] - w[5])); };
      auto dz = [&](const C* w) { return C(0.25) * inv[2] * (w[3] - w[0] + (w[5] - w[1]) + (w[6] - w[2]) + (w[7] - w[4])); };
      cs[n] = dy(q[2]) - dz(q[1]);
      cs[CN + n] = dz(q[0]) - dx(q[2]);
      cs[2 * CN + n] = dx(q[1]) - dy(q[0]);
    }
  }
  // Keeps the mass blocks of the thread's first p.kept stencils for the steps
  // of a cycle (with one tile a CTA).
  int kept = 0;
  __device__ __forceinline__ void keep_mass() {
    kept = p.kept;
    int n, part, i, j, k;
    if (!kept || !my_node(0, n, part, i, j, k)) return;
    const Mass* mass = static_cast<const Mass*>(p.mass) + p.g.mass_vertex(i, j, k) * p.g.mvs;
    const int s0 = 14 * part / p.parts, s1 = min(s0 + kept, 14 * (part + 1) / p.parts);
    Mass* own = at<Mass>(L.mass) + threadIdx.x;
    for (int s = s0; s < s1; ++s, own += 18 * kResidentNodeThreads) {
      Mass m[18];
      load_blocks(mass, s, at<int2>(L.offsets)[s].y, m);
#pragma unroll
      for (int e = 0; e < 18; ++e)
        if (e < 9 || s > 0) own[e * kResidentNodeThreads] = m[e];
    }
  }
  // This thread's node of the tile and its part of the node's mass blocks.
  __device__ __forceinline__ bool my_node(int slot, int& n, int& part, int& i, int& j, int& k) const {
    n = threadIdx.x & (p.nodes - 1);
    part = threadIdx.x >> p.shift;
    return threadIdx.x < kResidentNodeThreads && node_of(slot, n, i, j, k);
  }
  __device__ __forceinline__ void local(int n, int& lx, int& ly, int& lz) const {
    lx = n & (p.tx - 1);
    ly = (n / p.tx) & (p.ty - 1);
    lz = n / (p.tx * p.ty);
  }
  // The mass product of node (i, j, k) from v (component stride vn), complete in the node's first thread. A CTA barrier
  // is in it.
  template <class C>
  __device__ __forceinline__ void mass(bool live, int n, int part, int i, int j, int k, const C* v, int vn, C out[3]) {
    const Geom& g = p.g;
    C x = C(0), y = C(0), z = C(0);
    if (live) {
      // Blocks in stencil order: part r of P takes stencils [14 r / P, 14 (r + 1) / P).
      const Mass* mass = static_cast<const Mass*>(p.mass) + g.mass_vertex(i, j, k) * g.mvs;
      const int2* offsets = at<int2>(L.offsets);
      const int s0 = 14 * part / p.parts, s1 = 14 * (part + 1) / p.parts;
      if constexpr (kCtas == 1) {
        // The stencils kept, then the others, each loaded while the last one
        // is applied.
        const int loaded = min(s0 + kept, s1);
        Mass next[18];
        if (loaded < s1) load_blocks(mass, loaded, offsets[loaded].y, next);
        const Mass* own = at<Mass>(L.mass) + threadIdx.x;
        for (int s = s0; s < loaded; ++s, own += 18 * kResidentNodeThreads) {
          const int o = offsets[s].x;
          product<C>([&](int e) { return own[e * kResidentNodeThreads]; }, v + o, vn, x, y, z);
          if (s > 0) product<C>([&](int e) { return own[(9 + e) * kResidentNodeThreads]; }, v - o, vn, x, y, z);
        }
        for (int s = loaded; s < s1; ++s) {
          const int o = offsets[s].x;
          Mass m[18];
#pragma unroll
          for (int e = 0; e < 18; ++e) m[e] = next[e];
          if (s + 1 < s1) load_blocks(mass, s + 1, offsets[s + 1].y, next);
          product<C>([&](int e) { return m[e]; }, v + o, vn, x, y, z);
          if (s > 0) product<C>([&](int e) { return m[9 + e]; }, v - o, vn, x, y, z);
        }
      } else {
        for (int s = s0; s < s1; ++s) {
          const int2 o = offsets[s];
          const Mass* b = mass + 9 * s * g.mes;
          if (p.slots > 1 && s + 1 < s1) {
            // Grids whose mass L2 does not hold: the next stencil's rows are
            // requested while this one's are applied, as in the step's apply.
            const Mass* next = b + 9 * g.mes;
            const int back = offsets[s + 1].y;
#pragma unroll
            for (int e = 0; e < 9; ++e) {
              prefetch_l2(next + e * g.mes);
              prefetch_l2(next + e * g.mes - back);
            }
          }
          product<C>([&](int e) { return __ldg(b + e * g.mes); }, v + o.x, vn, x, y, z);
          if (s > 0) product<C>([&](int e) { return __ldg(b - o.y + e * g.mes); }, v - o.x, vn, x, y, z);
        }
      }
      if (part > 0) {
        C* sum = at<C>(L.part);
        sum[threadIdx.x] = x;
        sum[kResidentNodeThreads + threadIdx.x] = y;
        sum[2 * kResidentNodeThreads + threadIdx.x] = z;
      }
    }
    __syncthreads();
    if (live && part == 0) {
      const C* sum = at<C>(L.part);
      for (int r = 1; r < p.parts; ++r) {
        const int t = r * p.nodes + n;
        x += sum[t];
        y += sum[kResidentNodeThreads + t];
        z += sum[2 * kResidentNodeThreads + t];
      }
    }
    const C iv = C(p.inv_volume);
    out[0] = x * iv;
    out[1] = y * iv;
    out[2] = z * iv;
  }
  // v + delta^2 curl curl v + k m at a node.
  template <class C>
  __device__ __forceinline__ void combine(int lx, int ly, int lz, const C m[3], C value[3]) const {
    const C* vs = at<C>(L.vs);
    const C* cs = at<C>(L.cs);
    const int vx = p.tx + 2, vxy = vx * (p.ty + 2), cx = p.tx + 1, cxy = cx * (p.ty + 1);
    const int VN = L.halo, CN = L.cells;
    const C inv[3] = {C(p.g.inv[0]), C(p.g.inv[1]), C(p.g.inv[2])};
    C w[3][8];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const C* f = cs + c * CN + (lx + 1) + cx * (ly + 1) + cxy * (lz + 1);
      w[c][0] = f[0];        w[c][1] = f[-1];       w[c][2] = f[-cx];       w[c][3] = f[-cxy];
      w[c][4] = f[-cx - 1];  w[c][5] = f[-cxy - 1]; w[c][6] = f[-cxy - cx]; w[c][7] = f[-cxy - cx - 1];
    }
    auto dx = [&](const C* q) { return C(0.25) * inv[0] * (q[0] - q[1] + (q[3] - q[5]) + (q[2] - q[4]) + (q[6] - q[7])); };
    auto dy = [&](const C* q) { return C(0.25) * inv[1] * (q[0] - q[2] + (q[3] - q[6]) + (q[1] - q[4]) + (q[5] - q[7])); };
    auto dz = [&](const C* q) { return C(0.25) * inv[2] * (q[0] - q[3] + (q[1] - q[5]) + (q[2] - q[6]) + (q[4] - q[7])); };
    const C curl[3] = {dy(w[2]) - dz(w[1]), dz(w[0]) - dx(w[2]), dx(w[1]) - dy(w[0])};
    const C d2 = C(p.delta * p.delta), kf = C(p.kfac);
    const int vi = (lx + 1) + vx * (ly + 1) + vxy * (lz + 1);
#pragma unroll
    for (int c = 0; c < 3; ++c) value[c] = (vs[c * VN + vi] + d2 * curl[c]) + kf * m[c];
  }

  // Smoothing: the region of the tile's passes filled from load(component,
  // unique index), and the passes over it (the passes have CTA barriers).
  template <class C, class Load>
  __device__ __forceinline__ void stage_region(const SmoothTile& t, Load&& load) {
    if (threadIdx.x >= kResidentNodeThreads) return;
    C* a = at<C>(L.smooth);
    int i0, j0, k0;
    origin(0, i0, j0, k0);
    const Geom& g = p.g;
    for (int y = threadIdx.x >> 5; y < t.e[1]; y += kResidentNodeThreads / 32) {
      const int row = g.nx * wrap_index(j0 - t.h[1] + y, g.ny);
      for (int x = threadIdx.x & 31; x < t.e[0]; x += 32) {
        const int u = wrap_index(i0 - t.h[0] + x, g.nx) + row;
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c * t.size + y * t.e[0] + x] = C(load(c, u));
      }
    }
  }
  template <class C>
  __device__ __forceinline__ const C* smoothed(const SmoothTile& t) {
    C* a = at<C>(L.smooth);
    int i0, j0, k0;
    origin(0, i0, j0, k0);
    return smooth_passes<C>(t, 3, a, a + 3 * t.size, p.smooth, p.smooth_op, p.smooth_alpha, threadIdx.x >> 5,
                            kResidentThreads / 32, [&](int x, int y, int) {
                              x -= t.h[0];
                              y -= t.h[1];
                              if (x >= 0 && x < p.tx && i0 + x < p.g.nx && y >= 0 && y < p.ty && j0 + y < p.g.ny)
                                atomicAdd(p.invalid, 1u);
                            });
  }

  // The operator on the tile's nodes, after stage() (and, with smoothing,
  // stage_region()) of the vector and a CTA barrier: store(node in tile, its
  // coordinates, the three values) from the first thread of each node in the
  // grid. False when a barrier gave up.
  template <class C, class Store>
  __device__ __forceinline__ bool image(int slot, Store&& store) {
    cell_curls<C>();
    int n, part, i = 0, j = 0, k = 0, lx, ly, lz;
    const bool live = my_node(slot, n, part, i, j, k);
    local(n, lx, ly, lz);
    C m[3];
    if constexpr (!kSmooth) {
      const int vx = p.tx + 2, vxy = vx * (p.ty + 2);
      mass<C>(live, n, part, i, j, k, at<C>(L.vs) + (lx + 1) + vx * (ly + 1) + vxy * (lz + 1), L.halo, m);
    } else {
      const SmoothTile t = resident_smooth_tile(p);
      const int own = (lx + t.h[0]) + t.e[0] * (ly + t.h[1]);
      const long long U = unique();
      const C* v = smoothed<C>(t);
      mass<C>(live, n, part, i, j, k, v + own, t.size, m);
      if (live && part == 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) p.response[c * U + i + p.g.nx * j] = double(m[c]);
      if (!grid_barrier()) return false;
      stage_region<C>(t, [&](int c, int u) { return __ldcg(p.response + c * U + u); });
      __syncthreads();
      v = smoothed<C>(t);
#pragma unroll
      for (int c = 0; c < 3; ++c) m[c] = live ? v[c * t.size + own] : C(0);
    }
    if (live && part == 0) {
      C value[3];
      combine<C>(lx, ly, lz, m, value);
      store(n, i, j, k, value);
    }
    return true;
  }

  // The blocks of stencil s at a node (m[0..8]) and at the node - s (m[9..17]).
  __device__ __forceinline__ void load_blocks(const Mass* __restrict__ mass, int s, int back, Mass (&m)[18]) const {
    const Mass* b = mass + 9 * s * p.g.mes;
#pragma unroll
    for (int e = 0; e < 9; ++e) m[e] = __ldg(b + e * p.g.mes);
    if (s > 0)
#pragma unroll
      for (int e = 0; e < 9; ++e) m[9 + e] = __ldg(b - back + e * p.g.mes);
  }
  template <class C, class Entry>
  __device__ __forceinline__ void product(Entry&& entry, const C* v, int VN, C& x, C& y, C& z) const {
    C m[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) m[e] = C(entry(e));
    const C v0 = v[0], v1 = v[VN], v2 = v[2 * VN];
    if constexpr (kTranspose) {
      x += v0 * m[0] + v1 * m[3] + v2 * m[6];
      y += v0 * m[1] + v1 * m[4] + v2 * m[7];
      z += v0 * m[2] + v1 * m[5] + v2 * m[8];
    } else {
      x += v0 * m[0] + v1 * m[1] + v2 * m[2];
      y += v0 * m[3] + v1 * m[4] + v2 * m[5];
      z += v0 * m[6] + v1 * m[7] + v2 * m[8];
    }
  }

  // Block totals of one or two sums, to rows `row` and `row + 1` of the partials.
  __device__ void publish(double a, double b, int row, bool two) {
    double* sums = at<double>(L.sums);
    const int warp = threadIdx.x >> 5;
    a = warp_sum(a);
    if (two) b = warp_sum(b);
    if ((threadIdx.x & 31) == 0) {
      sums[2 * warp] = a;
      sums[2 * warp + 1] = b;
    }
    __syncthreads();
    if (threadIdx.x < (two ? 2 : 1)) {
      double total = 0;
      for (int w = 0; w < kResidentThreads / 32; ++w) total += sums[2 * w + threadIdx.x];
      p.partials[(long long)(row + threadIdx.x) * gridDim.x + blockIdx.x] = total;
    }
  }
  // A row of the partials summed over the CTAs (every lane of a warp; fixed order).
  __device__ __forceinline__ double gathered(int row) const {
    const double* from = p.partials + (long long)row * gridDim.x;
    double total = 0;
    for (unsigned t = threadIdx.x & 31; t < gridDim.x; t += 32) total += __ldcg(from + t);
    return warp_sum(total);
  }
  // Sums over the lanes of a warp's columns first, first + step, ... <= last (at
  // most four), to sink(column, sum) in lane 0. The columns' terms and shuffles
  // run side by side: one after the other their latencies were a third of a
  // step on small grids.
  template <class Sink>
  __device__ __forceinline__ void column_sums(int first, int step, int last, double (&sum)[4], Sink&& sink) const {
    if (first + step <= last) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < 4; ++r) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
    } else {
      sum[0] = warp_sum(sum[0]);
    }
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (first + r * step <= last) sink(first + r * step, sum[r]);
  }

  // What the nodes keep: unique indexes, multiplicities and the tables.
  __device__ void prepare() {
    int* unode = at<int>(L.unode);
    uint8_t* mult = at<uint8_t>(L.mult);
    for (int t = threadIdx.x; t < p.slots * p.nodes; t += kResidentThreads) {
      int i, j, k;
      const bool live = node_of(t >> p.shift, t & (p.nodes - 1), i, j, k);
      unode[t] = live ? i + p.g.nx * (j + p.g.ny * k) : -1;
      mult[t] = live ? uint8_t((i == 0 ? 2 : 1) * (j == 0 ? 2 : 1) * (k == 0 ? 2 : 1)) : uint8_t(0);
    }
    S* last = at<S>(L.image);
    for (int t = threadIdx.x; t < p.slots * 3 * p.nodes; t += kResidentThreads) last[t] = S(0);
    fixed_tables();
    tables(0);
    __syncthreads();
  }
  // With several slots the table holds the slot in hand, whose centre blocks
  // are requested ahead.
  __device__ __forceinline__ void enter(int slot) {
    if (p.slots == 1) return;
    __syncthreads();
    tables(slot);
    int i, j, k;
    if (threadIdx.x < kResidentNodeThreads && node_of(slot, threadIdx.x & (p.nodes - 1), i, j, k)) {
      const Mass* b = static_cast<const Mass*>(p.mass) + p.g.mass_vertex(i, j, k) * p.g.mvs;
#pragma unroll
      for (int e = 0; e < 9; ++e) prefetch_l2(b + e * p.g.mes);
    }
    __syncthreads();
  }

  // r = b - A x over the owned nodes (x read through `load`), the sums of r^2
  // (and of b^2) published.
  template <class Load>
  __device__ bool residual(Load&& load, bool with_rhs) {
    double s0 = 0, s1 = 0;
    const long long U = unique();
    for (int slot = 0; slot < p.slots && tile_of(slot) < p.tiles; ++slot) {
      enter(slot);
      stage<double>(load);
      __syncthreads();
      const bool done = image<double>(slot, [&](int, int i, int j, int k, const double value[3]) {
        const int u = i + p.g.nx * (j + p.g.ny * k);
        const double m = (i == 0 ? 2.0 : 1.0) * (j == 0 ? 2.0 : 1.0) * (k == 0 ? 2.0 : 1.0);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double b = p.b[c * U + u], r = b - value[c];
          p.r[c * U + u] = r;
          s0 += m * (r * r);
          s1 += m * (b * b);
        }
      });
      if (!done) return false;
    }
    __syncthreads();
    publish(s0, s1, 0, with_rhs);
    return true;
  }

  // The solution x with its ghosts into etheta (node field).
  __device__ void write_solution() {
    const Geom& g = p.g;
    const long long U = unique();
    const uint32_t total = uint32_t(g.nodes), NX = uint32_t(g.NX), NY = uint32_t(g.NY);
    for (uint32_t t = blockIdx.x * kResidentThreads + threadIdx.x; t < total; t += gridDim.x * kResidentThreads) {
      const uint32_t row = t / NX;
      const int i = int(t - row * NX) - 1, j = int(row % NY) - 1, k = int(row / NY) - 1;
      const int u = wrap_index(i, g.nx) + g.nx * (wrap_index(j, g.ny) + g.ny * wrap_index(k, g.nz));
#pragma unroll
      for (int c = 0; c < 3; ++c) p.etheta[c * g.nodes + t] = __ldcg(p.x + c * U + u);
    }
  }
};

// The right-hand side, the guess and its residual (values[0] = |r|^2,
// values[1] = |b|^2).
template <class S, class Mass, class Fld, bool kTranspose, bool kSmooth, int kCtas>
__global__ void __launch_bounds__(kResidentThreads, kCtas) resident_start_kernel(const __grid_constant__ ResidentPlan p) {
  extern __shared__ __align__(16) uint8_t resident_smem[];
  using R = Resident<S, Mass, Fld, kTranspose, kSmooth, kCtas>;
  R r(p, resident_smem);
  r.prepare();
  const Geom& g = p.g;
  const long long U = r.unique();
  const Fld* e = static_cast<const Fld*>(p.e);
  const Fld inv[3] = {Fld(g.inv[0]), Fld(g.inv[1]), Fld(g.inv[2])};
  // With smoothing the right-hand side has S^n(J), in the field arithmetic.
  const Fld* smooth_j = nullptr;
  SmoothTile t = resident_smooth_tile(p);
  if constexpr (kSmooth) {
    r.template stage_region<Fld>(t, [&](int c, int u) {
      const int row = u / g.nx;
      return static_cast<const Fld*>(p.j)[c * g.nodes + g.node(u - row * g.nx, row, 0)];
    });
    __syncthreads();
    smooth_j = r.template smoothed<Fld>(t);
  }
  for (int slot = 0; slot < p.slots; ++slot) {
    int i, j, k;
    if (int(threadIdx.x) >= p.nodes || !r.node_of(slot, threadIdx.x, i, j, k)) continue;
    const int u = i + g.nx * (j + g.ny * k);
    const long long at = g.node(i, j, k);
    if (p.rhs) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        p.x[c * U + u] = 0.0;
        p.b[c * U + u] = p.rhs[c * g.nodes + at];
      }
    } else {
      Fld cb[3];
      curl_c2n_at<Fld>(g, static_cast<const Fld*>(p.bcell), i, j, k, inv, cb);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const Fld ev = e[c * g.nodes + at];
        Fld jv;
        if constexpr (kSmooth) {
          int lx, ly, lz;
          r.local(threadIdx.x, lx, ly, lz);
          jv = smooth_j[c * t.size + (lx + t.h[0]) + t.e[0] * (ly + t.h[1])];
        } else {
          jv = static_cast<const Fld*>(p.j)[c * g.nodes + at];
        }
        p.x[c * U + u] = double(ev);
        p.b[c * U + u] = double((ev + Fld(p.delta) * cb[c]) + (-Fld(p.kfac)) * jv);
      }
    }
  }
  __syncthreads();
  if (!r.residual([&](int c, int u) -> double {
        if (p.rhs) return 0.0;
        const int row = u / g.nx, k = row / g.ny;
        return double(e[c * g.nodes + g.node(u - row * g.nx, row - k * g.ny, k)]);
      }, true))
    return;
  if (!r.grid_barrier()) return;
  const double r2 = r.gathered(0), b2 = r.gathered(1);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    p.values[0] = r2;
    p.values[1] = b2;
  }
  const double norm = sqrt(b2);
  if (sqrt(r2) <= (norm == 0.0 ? 1.0 : norm) * p.accept) r.write_solution();
  r.leave();
}

// One restart cycle from the residual r (values[0] = |r|^2): at most
// `columns` Arnoldi steps, the update of x, its residual (values[0]).
template <class S, class Mass, class Fld, bool kTranspose, bool kSmooth, int kCtas>
__global__ void __launch_bounds__(kResidentThreads, kCtas) resident_cycle_kernel(const __grid_constant__ ResidentPlan p) {
  extern __shared__ __align__(16) uint8_t resident_smem[];
  using R = Resident<S, Mass, Fld, kTranspose, kSmooth, kCtas>;
  R r(p, resident_smem);
  constexpr int m = kResidentRestart, kWarps = kResidentThreads / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long U = r.unique();
  const int rows = p.slots * 3 * p.nodes;
  double* H = r.template at<double>(r.L.h);      // column c at c * (m + 1)
  double* hcol = r.template at<double>(r.L.hcol);
  double* cosine = r.template at<double>(r.L.rot);
  double* sine = cosine + m + 1;
  double* rhs = sine + m + 1;
  double* coefficient = rhs + m + 1;
  double* shared = r.template at<double>(r.L.sums) + 2 * kWarps;  // diagonal, decision, breakdown
  S* image = r.template at<S>(r.L.image);
  const int* unode = r.template at<int>(r.L.unode);
  const uint8_t* mult = r.template at<uint8_t>(r.L.mult);
  S* vector = static_cast<S*>(p.vector);
  constexpr bool kSideBySide = kCtas == 1;
  r.prepare();
  r.keep_mass();
  // Row t of the owned rows: its node and its place in a [3][unique] vector.
  auto place = [&](int t, int& n) -> long long {
    const int slot = p.slots == 1 ? 0 : t / (3 * p.nodes), rest = t - slot * 3 * p.nodes;
    n = slot * p.nodes + (rest & (p.nodes - 1));
    return (rest >> p.shift) * U + unode[n];
  };
  const double first = p.values[0];
  double scale = first > 0.0 ? 1.0 / sqrt(first) : 0.0;
  {
    S* v = r.basis(0);
    for (int t = threadIdx.x; t < rows; t += kResidentThreads) {
      int n;
      const long long at = place(t, n);
      v[t] = unode[n] >= 0 ? S(p.r[at] * scale) : S(0);
    }
  }
  if (threadIdx.x == kResidentNodeThreads) {
    rhs[0] = sqrt(first);
    shared[1] = 0.0;
  }
  int col = 0, stop = 0;
  while (true) {
    // A: image = A v_col; its dots with columns 0..col. The decision on the
    // last step is formed by the other warp while the vector is staged.
    for (int slot = 0; slot < p.slots && r.tile_of(slot) < p.tiles; ++slot) {
      r.enter(slot);
      if (col == 0) r.template stage<S>([&](int c, int u) { return S(__ldcg(p.r + c * U + u) * scale); });
      else r.template stage<S>([&](int c, int u) { return S(double(__ldcg(vector + c * U + u)) * scale); });
      __syncthreads();
      stop = int(shared[1]);
      if (stop) break;
      S* out = image + slot * 3 * p.nodes;
      if (!r.template image<S>(slot, [&](int n, int, int, int, const S value[3]) {
#pragma unroll
            for (int c = 0; c < 3; ++c) out[c * p.nodes + n] = value[c];
          }))
        return;
    }
    if (stop) break;
    __syncthreads();
    // A warp's columns one after the other with two CTAs an SM, which hide
    // each other's latency; else side by side.
    double dots[4] = {0.0, 0.0, 0.0, 0.0};
    if (kSideBySide && warp <= col) {
      const S* v = r.basis(warp);
      const long long next = r.basis(kWarps) - r.basis(0);
      const int columns = (col - warp) / kWarps + 1;
      for (int slot = 0, t0 = 0; slot < p.slots; ++slot, t0 += 3 * p.nodes)
#pragma unroll 2
        for (int t = lane; t < 3 * p.nodes; t += 32) {
          const double w = double(image[t0 + t]) * double(mult[slot * p.nodes + (t & (p.nodes - 1))]);
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (c < columns) dots[c] += double(v[c * next + t0 + t]) * w;
        }
    } else if (!kSideBySide) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (warp + c * kWarps > col) continue;
        const S* v = r.basis(warp + c * kWarps);
        for (int slot = 0, t0 = 0; slot < p.slots; ++slot, t0 += 3 * p.nodes)
          for (int t = lane; t < 3 * p.nodes; t += 32)
            dots[c] += double(v[t0 + t]) *
                       (double(image[t0 + t]) * double(mult[slot * p.nodes + (t & (p.nodes - 1))]));
      }
    }
    r.column_sums(warp, kWarps, col, dots,
                  [&](int c, double sum) { p.partials[(long long)c * gridDim.x + blockIdx.x] = sum; });
    if (!r.grid_barrier()) return;
    // B: Gram-Schmidt of the owned rows.
    double totals[4] = {0.0, 0.0, 0.0, 0.0};
    const double* from = p.partials + (long long)warp * gridDim.x;
    if (kSideBySide) {
#pragma unroll 2
      for (unsigned t = lane; t < gridDim.x; t += 32)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (warp + c * kWarps <= col) totals[c] += __ldcg(from + (long long)c * kWarps * gridDim.x + t);
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (warp + c * kWarps <= col)
          for (unsigned t = lane; t < gridDim.x; t += 32) totals[c] += __ldcg(from + (long long)c * kWarps * gridDim.x + t);
    }
    r.column_sums(warp, kWarps, col, totals, [&](int c, double sum) { hcol[c] = sum; });
    __syncthreads();
    double norm2 = 0;
    if (threadIdx.x < kResidentNodeThreads) {
      for (int t = threadIdx.x; t < rows; t += kResidentNodeThreads) {
        int n;
        const long long at = place(t, n);
        if (unode[n] < 0) continue;
        double value = double(image[t]);
        const S* v = r.basis(0) + t;
        const long long next = r.basis(1) - r.basis(0);
#pragma unroll 4
        for (int c = 0; c <= col; ++c) value -= hcol[c] * double(v[c * next]);
        const S stored = S(value);
        image[t] = stored;
        vector[at] = stored;
        norm2 += double(mult[n]) * (double(stored) * double(stored));
      }
    } else if (lane == 0) {
      // The column through the rotations so far.
      double* column = H + col * (m + 1);
      double upper = hcol[0];
      for (int row = 0; row < col; ++row) {
        const double lower = hcol[row + 1];
        column[row] = cosine[row] * upper + sine[row] * lower;
        upper = -sine[row] * upper + cosine[row] * lower;
      }
      shared[0] = upper;
    }
    r.publish(norm2, 0.0, m + 1, false);
    if (!r.grid_barrier()) return;
    const double n2 = r.gathered(m + 1);
    scale = n2 > 0.0 ? 1.0 / sqrt(n2) : 0.0;
    if (threadIdx.x == kResidentNodeThreads) {
      // ArnoldiLeastSquaresUpdate (gmres_device.hpp:62-98) and the stopping rule (:420-436).
      const double sub = sqrt(n2), diagonal = shared[0], den = hypot(diagonal, sub);
      const double c = den != 0.0 ? diagonal / den : 1.0, s = den != 0.0 ? sub / den : 0.0;
      cosine[col] = c;
      sine[col] = s;
      H[col * (m + 1) + col] = c * diagonal + s * sub;
      const double upper = rhs[col];
      rhs[col] = c * upper;
      rhs[col + 1] = -s * upper;
      const double estimate = fabs(rhs[col + 1]);
      const bool last = estimate <= p.tolerance || sub == 0.0 || col + 1 >= p.columns;
      shared[1] = !isfinite(estimate) ? 2.0 : last ? 1.0 : 0.0;
      shared[2] = sub == 0.0 ? 1.0 : 0.0;
    } else if (threadIdx.x < kResidentNodeThreads) {
      S* v = r.basis(col + 1);
      for (int t = threadIdx.x; t < rows; t += kResidentNodeThreads) v[t] = S(double(image[t]) * scale);
    }
    ++col;
  }
  const bool breakdown = shared[2] != 0.0;
  // Back substitution by columns (one warp), then x += V y.
  __syncthreads();
  if (warp == 0) {
    double s = lane < col ? rhs[lane] : 0.0;
    for (int row = col - 1; row >= 0; --row) {
      const double diagonal = H[row * (m + 1) + row];
      const double y = diagonal != 0.0 ? __shfl_sync(0xffffffffu, s, row) / diagonal : 0.0;
      if (lane < row) s -= H[row * (m + 1) + lane] * y;
      if (lane == 0) coefficient[row] = y;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < rows; t += kResidentThreads) {
    int n;
    const long long at = place(t, n);
    if (unode[n] < 0) continue;
    double value = p.x[at];
    const S* v = r.basis(0) + t;
    const long long next = r.basis(1) - r.basis(0);
    for (int c = 0; c < col; ++c) value += coefficient[c] * double(v[c * next]);
    p.x[at] = value;
  }
  if (!r.grid_barrier()) return;
  if (!r.residual([&](int c, int u) { return __ldcg(p.x + c * U + u); }, false)) return;
  if (!r.grid_barrier()) return;
  const double r2 = r.gathered(0);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    p.values[0] = r2;
    p.ctl->completed = col;
    p.ctl->stop = stop;
    p.ctl->breakdown = breakdown ? 1 : 0;
  }
  if (sqrt(r2) <= p.accept) r.write_solution();
  r.leave();
}

}  // namespace
}  // namespace tpicb200
