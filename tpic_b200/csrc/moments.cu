// The moments of the deposition off the tcgen05 forms: an FP32 form on the
// CUDA cores and an FP64 form on the FP64 tensor cores.
//
// Both form, per cell, G[t][e] = sum_p m_pt (s_p alpha_p[e]) and
// H[t][c] = sum_p m_pt j_p[c] over the records of up to two species, with m_pt
// the 27 pair-weight products (X_tx Y_ty) Z_tz, then the corner currents
// J_a[c] = sum_b H[t(a,b)][c], and store them as the moment records that
// launch_assemble_moments turns into J and the mass records without atomics.
// Per record this is 27 x 12 multiply-adds, where the reference's scalar and
// matrix-core kernels form the 64 corner-pair products of 9 entries
// (mass_matrix_scalar_device.hpp:25-97, mass_matrix_mma_device.hpp:58-150).
#include "kernels.cuh"
#include "moments.cuh"

#include <algorithm>

namespace tpicb200 {
namespace {

template <class Vel>
struct MomentSpecies {
  const double* rx;
  const double* ry;
  const double* rz;
  const Vel* u;
  const Vel* v;
  const Vel* w;
  const double* q;
  const int32_t* key;
  const uint32_t* counts;
  const uint32_t* offsets;
  double beta_over_c;
  const uint32_t* perm;  // sorted position -> record (null: records in sorted order)
  double* orx;           // sorted copy (null: none)
  double* ory;
  double* orz;
  Vel* ou;
  Vel* ov;
  Vel* ow;
  double* oq;
  int32_t* okey;
};

template <class Vel>
struct MomentParams {
  MomentSpecies<Vel> sp[kFuse];
  int ns;
  double inv_volume;
};

// A record of the cell `key`: its fractions, velocity and charge; false when
// it is not valid there. Copies it to its sorted position when asked.
template <class Vel>
struct MomentRecord {
  double f[3], q;
  Vel u, v, w;
  int32_t key;
  __device__ __forceinline__ void load(const MomentSpecies<Vel>& sp, uint32_t pos) {
    const uint32_t r = sp.perm ? sp.perm[pos] : pos;
    f[0] = sp.rx[r];
    f[1] = sp.ry[r];
    f[2] = sp.rz[r];
    u = sp.u[r];
    v = sp.v[r];
    w = sp.w[r];
    q = sp.q[r];
    key = sp.key[r];
    if (sp.orx) {
      sp.orx[pos] = f[0];
      sp.ory[pos] = f[1];
      sp.orz[pos] = f[2];
      sp.ou[pos] = u;
      sp.ov[pos] = v;
      sp.ow[pos] = w;
      sp.oq[pos] = q;
      sp.okey[pos] = key;
    }
  }
  __device__ __forceinline__ bool valid(int32_t cell) const {
    return key == cell && f[0] >= 0 && f[0] < 1 && f[1] >= 0 && f[1] < 1 && f[2] >= 0 && f[2] < 1;
  }
};

// The 12 values of a record, s alpha[9] and j[3], in arithmetic C (bc: B at the
// cell's corners, [c][a]) to value(e, v), and the 27 products to product(t, v);
// all zero, and false returned, for a record that is not there (`valid` false)
// or whose values are not finite.
// kSelect: by selects, for lanes that then all store; else `valid` holds and a
// nonfinite record is the exception, stored again as zeros.
template <class C, bool kSelect, class Vel, class Value, class Product>
__device__ __forceinline__ bool record_values(const MomentRecord<Vel>& r, bool valid, const C* bc, C beta_over_c,
                                              C inv_volume, Value&& value, Product&& product) {
  const bool take = !kSelect || valid;
  const C x = take ? C(r.f[0]) : C(0), y = take ? C(r.f[1]) : C(0), z = take ? C(r.f[2]) : C(0);
  C v[12];
  {
    C wt[8], b[3];
    cic_weights<C>(x, y, z, wt);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      C val = 0;
#pragma unroll
      for (int a = 0; a < 8; ++a) val += wt[a] * bc[c * 8 + a];
      b[c] = val;
    }
    const Response<C> resp(b[0], b[1], b[2], beta_over_c);
    const C scale = beta_over_c * C(r.q), qv = C(r.q) * inv_volume;
    C hx, hy, hz;
    resp.apply(C(r.u), C(r.v), C(r.w), hx, hy, hz);
#pragma unroll
    for (int e = 0; e < 9; ++e) v[e] = resp.a[e] * scale;
    v[9] = qv * hx;
    v[10] = qv * hy;
    v[11] = qv * hz;
  }
  bool ok = valid;
#pragma unroll
  for (int e = 0; e < 12; ++e) ok = ok && isfinite(v[e]);
#pragma unroll
  for (int e = 0; e < 12; ++e) value(e, !kSelect || ok ? v[e] : C(0));
  const C cx = C(1) - x, cy = C(1) - y, cz = C(1) - z;
  const bool keep = !kSelect || ok;
  const C px[3] = {keep ? cx * cx : C(0), keep ? cx * x : C(0), keep ? x * x : C(0)};
  const C py[3] = {cy * cy, cy * y, y * y}, pz[3] = {cz * cz, cz * z, z * z};
#pragma unroll
  for (int tz = 0; tz < 3; ++tz)
#pragma unroll
    for (int ty = 0; ty < 3; ++ty)
#pragma unroll
      for (int tx = 0; tx < 3; ++tx) product(tx + 3 * ty + 9 * tz, (px[tx] * py[ty]) * pz[tz]);
  return ok;
}

// A warp's walk over cells: the records of a cell's two species form one
// stream (species 0 first), so that a cell has at most one chunk that is not
// full.
struct MomentCell {
  int32_t key;
  uint32_t begin[kFuse], n[kFuse], total;
};
template <class Vel>
struct MomentWalk {
  const Geom& g;
  const MomentParams<Vel>& mp;
  uint32_t nx, ny, cells;
  __device__ __forceinline__ MomentWalk(const Geom& geom, const MomentParams<Vel>& params)
      : g(geom), mp(params), nx(geom.nx), ny(geom.ny), cells(uint32_t(geom.nx) * geom.ny * geom.nz) {}
  __device__ __forceinline__ void coordinates(uint32_t cell, int& i, int& j, int& k) const {
    const uint32_t row = cell / nx;
    i = int(cell - row * nx);
    j = int(row % ny);
    k = int(row / ny);
  }
  __device__ __forceinline__ MomentCell info(uint32_t cell) const {
    MomentCell c{};
    if (cell >= cells) return c;
    int i, j, k;
    coordinates(cell, i, j, k);
    c.key = g.encode(i, j, k);
#pragma unroll
    for (int s = 0; s < kFuse; ++s)
      if (s < mp.ns) {
        c.begin[s] = mp.sp[s].offsets[c.key];
        c.n[s] = mp.sp[s].counts[c.key];
      }
    c.total = c.n[0] + c.n[1];
    return c;
  }
  __device__ __forceinline__ int species(const MomentCell& c, uint32_t at) const { return at >= c.n[0] ? 1 : 0; }
  // Record o + lane of the cell.
  __device__ __forceinline__ void load(const MomentCell& c, uint32_t o, MomentRecord<Vel>& r) const {
    const uint32_t at = o + (threadIdx.x & 31u);
    if (at >= c.total) return;
    const int s = species(c, at);
    r.load(mp.sp[s], (s ? c.begin[1] - c.n[0] : c.begin[0]) + at);
  }
  // B at the corners of a cell, [c][a], by the first 24 lanes.
  template <class F, class C>
  __device__ __forceinline__ void corners(uint32_t cell, const F* __restrict__ bnode, C* bc) const {
    const int lane = threadIdx.x & 31;
    if (lane >= 24) return;
    int i, j, k;
    coordinates(cell, i, j, k);
    const int c = lane >> 3, a = lane & 7;
    bc[lane] = C(bnode[c * g.nodes + g.node(i + (a & 1), j + ((a >> 1) & 1), k + ((a >> 2) & 1))]);
  }
};

// A moment as it is stored: zero, and counted, when its sum is not finite.
template <class T>
__device__ __forceinline__ T checked(T value, uint32_t& bad) {
  if (isfinite(value)) return value;
  ++bad;
  return T(0);
}

// ---------------------------------------------------------------------------
// FP32 form (mixed precision, the SCALAR mass form): a warp per cell.
//
// The form this replaces shuffled every record's values to all lanes (12
// shuffles per 18 multiply-adds) and flushed 324 atomics per cell and species:
// 26 ms of the 128^3-cell workload's cycle. Here a lane forms one record's 27
// products and 12 values into shared memory; then the warp contracts the
// chunk, four records at a time: the 8 lanes of a quarter warp take one record
// and hold a 7 x 6 register tile each (four groups of 7 products by two of 6
// values), as packed FP32 pairs. The tile's shape is set by the shared-memory
// return path: 14 words per 42 multiply-adds keep it below the FP32 pipe's
// time, where a 4 x 3 tile over 28 lanes needed twice the words. The quarters
// are added at the cell's end. The next chunk's records are loaded before the
// contraction.
//
// A warp takes batches of four consecutive cells (one moment group) and stores
// the group's moments as contiguous 16-byte words; on grids with too few cells
// for that it takes single cells.
constexpr int kF32Warps = 4;
// Words of a record: the products in four groups of 7 (8 words each), the
// values in two groups of 6 (8 words each), padded so that the 8 lanes of a
// quarter storing 16 bytes each hit distinct banks (52 mod 32 = 20).
constexpr int kF32Pitch = 52;
// A cell's sums are staged in the order of the register tiles: tile (tg, eg)
// holds its 7 x 6 sums at 42 (2 tg + eg), so a lane stores at fixed distances.
__device__ __forceinline__ int f32_sum(int t, int entry) {
  const int tg = t / 7, eg = entry / 6;
  return 42 * (2 * tg + eg) + 6 * (t - 7 * tg) + (entry - 6 * eg);
}
struct __align__(16) F32Warp {
  float rec[32][kF32Pitch];
  float4 sums[8 * 42];  // of up to four cells
  float bc[24];         // B at the cell's corners, [c][a]
};

__global__ void __launch_bounds__(kF32Warps * 32, 4) moments_f32_kernel(Geom g, MomentParams<float> mp,
                                                                        const float* __restrict__ bnode,
                                                                        float* __restrict__ mom, int accumulate,
                                                                        int batch, uint32_t* invalid) {
  extern __shared__ __align__(16) uint8_t f32_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  F32Warp& S = reinterpret_cast<F32Warp*>(f32_smem)[warp];
  const MomentWalk<float> walk(g, mp);
  const uint32_t cells = walk.cells;
  const uint32_t warps = gridDim.x * kF32Warps;
  const int quarter = lane >> 3, tg = lane & 3, eg = (lane >> 2) & 1;
  uint32_t bad = 0;
  // The cell after `cell` in this warp's order (batches strided by the grid).
  auto following = [&](uint32_t cell) {
    const uint32_t next = cell + 1;
    return next % batch != 0 && next < cells ? next : (cell / batch + warps) * batch;
  };

  uint32_t cell = (blockIdx.x * kF32Warps + warp) * batch;
  MomentCell cur = walk.info(cell);
  MomentRecord<float> next;
  walk.load(cur, 0, next);
  while (cell < cells) {
    const uint32_t cell_next = following(cell);
    const MomentCell after = walk.info(cell_next);
    __syncwarp();
    walk.corners(cell, bnode, S.bc);
    __syncwarp();
    float2 acc[7][3];
#pragma unroll
    for (int i = 0; i < 7; ++i)
#pragma unroll
      for (int e = 0; e < 3; ++e) acc[i][e] = make_float2(0.0f, 0.0f);
    if (cur.total == 0) walk.load(after, 0, next);
    for (uint32_t o = 0; o < cur.total; o += 32) {
      const uint32_t m = min(cur.total - o, 32u);
      const MomentRecord<float> r = next;
      if (o + 32 < cur.total) walk.load(cur, o + 32, next);
      else walk.load(after, 0, next);
      const bool active = lane < int(m);
      const int sp = active ? walk.species(cur, o + lane) : 0;
      // Zeros from the lanes without a record fill the rows past m.
      float* row = S.rec[lane];
      float value[12], prod[28];
      prod[27] = 0.0f;
      __syncwarp();
      const bool ok = record_values<float, true>(
          r, active && r.valid(cur.key), S.bc, float(mp.sp[sp].beta_over_c), float(mp.inv_volume),
          [&](int e, float v) { value[e] = v; }, [&](int t, float v) { prod[t] = v; });
      if (active && !ok) ++bad;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int e = 6 * q;
        *reinterpret_cast<float4*>(row + 32 + 8 * q) = make_float4(value[e], value[e + 1], value[e + 2], value[e + 3]);
        *reinterpret_cast<float2*>(row + 36 + 8 * q) = make_float2(value[e + 4], value[e + 5]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int t = 7 * q;
        *reinterpret_cast<float4*>(row + 8 * q) = make_float4(prod[t], prod[t + 1], prod[t + 2], prod[t + 3]);
        *reinterpret_cast<float4*>(row + 8 * q + 4) = make_float4(prod[t + 4], prod[t + 5], prod[t + 6], 0.0f);
      }
      __syncwarp();
#pragma unroll 2
      for (uint32_t k = 0; k < m; k += 4) {
        const float* from = S.rec[k + quarter];
        const float4 a = *reinterpret_cast<const float4*>(from + 8 * tg);
        const float4 b = *reinterpret_cast<const float4*>(from + 8 * tg + 4);
        const float4 c = *reinterpret_cast<const float4*>(from + 32 + 8 * eg);
        const float2 d = *reinterpret_cast<const float2*>(from + 36 + 8 * eg);
        const float t[7] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z};
        const float2 v[3] = {make_float2(c.x, c.y), make_float2(c.z, c.w), d};
#pragma unroll
        for (int i = 0; i < 7; ++i)
#pragma unroll
          for (int e = 0; e < 3; ++e) acc[i][e] = __ffma2_rn(make_float2(t[i], t[i]), v[e], acc[i][e]);
      }
    }
    // The quarters' tiles are added: lanes 16 apart exchange halves of the 42
    // sums, then lanes 8 apart halves of those.
    float h[21];
    const bool upper = lane & 16, odd = lane & 8;
#pragma unroll
    for (int f = 0; f < 21; ++f) {
      auto at = [&](int n) { return (n & 1) ? acc[n / 6][(n % 6) / 2].y : acc[n / 6][(n % 6) / 2].x; };
      const float keep = upper ? at(f + 21) : at(f), send = upper ? at(f) : at(f + 21);
      h[f] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
    float sum[11];
#pragma unroll
    for (int f = 0; f < 10; ++f) {
      const float keep = odd ? h[f + 11] : h[f], send = odd ? h[f] : h[f + 11];
      sum[f] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    sum[10] = h[10] + __shfl_xor_sync(0xffffffffu, h[10], 8);
    const int slot = batch == 4 ? int(cell & 3) : 0;
    float* to = &S.sums[42 * (2 * tg + eg) + (upper ? 21 : 0) + (odd ? 11 : 0)].x + slot;
#pragma unroll
    for (int f = 0; f < 10; ++f) to[4 * f] = sum[f];
    if (!odd) to[40] = sum[10];
    __syncwarp();
    if (batch != 4 || slot == 3 || cell + 1 == cells) {
      // Entry q of the group's cells (of one cell without batches).
      for (int q = lane; q < kMoments; q += 32) {
        float4 v;
        if (q < kMassMoments) {
          const int t = q / 9;
          v = S.sums[f32_sum(t, q - 9 * t)];
        } else {
          const int a = (q - kMassMoments) / 3, c = (q - kMassMoments) % 3;
          v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const float4 h = S.sums[f32_sum(monomial_class(a, b), 9 + c)];
            v.x += h.x;
            v.y += h.y;
            v.z += h.z;
            v.w += h.w;
          }
        }
        v.x = checked(v.x, bad);
        if (batch != 4) {
          float* dst = mom + moment_index(cell, q);
          *dst = accumulate ? *dst + v.x : v.x;
          continue;
        }
        if (slot > 0) v.y = checked(v.y, bad);
        if (slot > 1) v.z = checked(v.z, bad);
        if (slot > 2) v.w = checked(v.w, bad);
        float4* dst = reinterpret_cast<float4*>(mom) + (long long)(cell >> 2) * kMoments + q;
        if (accumulate) {
          const float4 old = *dst;
          v = make_float4(v.x + old.x, v.y + old.y, v.z + old.z, v.w + old.w);
        }
        *dst = v;
      }
    }
    cell = cell_next;
    cur = after;
  }
  bad = warp_sum(bad);
  if (bad && lane == 0) atomicAdd(invalid, bad);
}

// ---------------------------------------------------------------------------
// FP64 form (MOMENTS_F64, the SCALAR forms in double precision and SCALAR_F64
// in mixed precision, which narrows a cell's sums once): a warp per cell. Per
// chunk of 32 records each lane forms one record's 27 products and 12 values
// in shared memory; then the warp contracts the chunk on the FP64 tensor cores
// (mma.sync m8n8k4: D[t][e] += sum_k m[k][t] src[k][e], t in four tiles of 8
// rows (27 used), e in two of 8 columns (12 used), four records per step). The
// contraction on the CUDA cores (a 3 x 4 register block per lane, 7 shared
// loads per 12 fused multiply-adds) was bound by the shared-memory pipe (93 %
// of its wavefronts at 64^3); the fragments need 6 shared loads per 4 records
// and lane (128^3-cell workload: the FP64 deposit stage 20.0 -> 16.1 ms).
constexpr int kF64Warps = 4;
// The products and values are stored by (t or entry, record), 36 records a
// row: a lane's stores of its record fall in consecutive words, and the 16
// lanes of a half-warp fragment load (4 rows x 4 records) hit 16 different
// bank pairs. With record-major rows of 29 and 13 words the fragment loads
// met 2-way conflicts (FP64 deposit stage of 268M records on 128^3: 16.2 ms,
// 15.7 ms with these rows).
constexpr int kF64Pitch = 36;
struct F64Warp {
  double bc[24];                 // B at the cell's corners, [c][a]
  double m[27][kF64Pitch];       // [t][record]: the 27 pair-weight products
  double src[12][kF64Pitch];     // [entry][record]: s alpha[9], j[3]
  double hs[27][3];              // H of the cell at the flush
};

template <class Vel, class Fld, class Mom>
__global__ void __launch_bounds__(kF64Warps * 32, 4) moments_f64_kernel(Geom g, MomentParams<Vel> mp,
                                                                     const Fld* __restrict__ bnode,
                                                                     Mom* __restrict__ mom, int accumulate,
                                                                     uint32_t* invalid) {
  __shared__ F64Warp shared[kF64Warps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  F64Warp& S = shared[warp];
  const MomentWalk<Vel> walk(g, mp);
  const uint32_t stride = gridDim.x * kF64Warps;
  const int kk = lane & 3, rr = lane >> 2;  // fragment coordinates
  uint32_t bad = 0;
  uint32_t cell = blockIdx.x * kF64Warps + warp;
  MomentCell cur = walk.info(cell);
  MomentRecord<Vel> next;
  walk.load(cur, 0, next);
  while (cell < walk.cells) {
    const uint32_t cell_next = cell + stride;
    const MomentCell after = walk.info(cell_next);
    walk.corners(cell, bnode, S.bc);
    __syncwarp();
    // D tiles (t: 4 x 8 rows, entry: 2 x 8 columns) of this lane.
    double acc[4][2][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) acc[i][e][0] = acc[i][e][1] = 0.0;
    if (cur.total == 0) walk.load(after, 0, next);
    for (uint32_t o = 0; o < cur.total; o += 32) {
      const uint32_t m = min(cur.total - o, 32u);
      const MomentRecord<Vel> r = next;
      if (o + 32 < cur.total) walk.load(cur, o + 32, next);
      else walk.load(after, 0, next);
      if (lane < int(m)) {
        bool ok = r.valid(cur.key);
        if (ok)
          ok = record_values<double, false>(r, true, S.bc, mp.sp[walk.species(cur, o + lane)].beta_over_c,
                                            mp.inv_volume, [&](int e, double v) { S.src[e][lane] = v; },
                                            [&](int t, double v) { S.m[t][lane] = v; });
        if (!ok) {
          ++bad;
#pragma unroll
          for (int e = 0; e < 12; ++e) S.src[e][lane] = 0.0;
#pragma unroll
          for (int t = 0; t < 27; ++t) S.m[t][lane] = 0.0;
        }
      }
      __syncwarp();
      for (uint32_t k0 = 0; k0 < m; k0 += 4) {
        const uint32_t k = k0 + kk;
        const bool in = k < m;
        double av[4], bv[2];
#pragma unroll
        for (int i = 0; i < 4; ++i) av[i] = in && 8 * i + rr < 27 ? S.m[8 * i + rr][k] : 0.0;
#pragma unroll
        for (int e = 0; e < 2; ++e) bv[e] = in && 8 * e + rr < 12 ? S.src[8 * e + rr][k] : 0.0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) dmma_884(acc[i][e], av[i], bv[e]);
      }
      __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int t = 8 * i + rr, entry = 8 * e + 2 * kk + h;
          if (t >= 27 || entry >= 12) continue;
          if (entry < 9) {
            Mom* dst = mom + moment_index(cell, t * 9 + entry);
            const Mom value = checked(Mom(acc[i][e][h]), bad);
            *dst = accumulate ? *dst + value : value;
          } else {
            S.hs[t][entry - 9] = acc[i][e][h];
          }
        }
    __syncwarp();
    if (lane < 24) {
      const int a = lane / 3, c = lane % 3;
      double sum = 0.0;
#pragma unroll
      for (int b = 0; b < 8; ++b) sum += S.hs[monomial_class(a, b)][c];
      Mom* dst = mom + moment_index(cell, kMassMoments + a * 3 + c);
      const Mom value = checked(Mom(sum), bad);
      *dst = accumulate ? *dst + value : value;
    }
    __syncwarp();
    cell = cell_next;
    cur = after;
  }
  bad = warp_sum(bad);
  if (bad && lane == 0) atomicAdd(invalid, bad);
}

template <class Vel>
MomentParams<Vel> moment_params(const Geom& g, int first, int ns, const double* qom, double dt, double c,
                                const tpicb200_particles* const* p, const uint32_t* const* counts,
                                const uint32_t* const* offsets, const SortedCopy* const* copies) {
  MomentParams<Vel> mp{};
  mp.ns = std::min(kFuse, ns - first);
  mp.inv_volume = g.inv_volume;
  for (int i = 0; i < mp.ns; ++i) {
    const tpicb200_particles* sp = p[first + i];
    const SortedCopy* cp = copies ? copies[first + i] : nullptr;
    const bool copy = cp && cp->perm && cp->out.rx;
    mp.sp[i] = MomentSpecies<Vel>{(const double*)sp->rx, (const double*)sp->ry, (const double*)sp->rz,
                                  (const Vel*)sp->u, (const Vel*)sp->v, (const Vel*)sp->w, sp->q, sp->cell,
                                  counts[first + i], offsets[first + i], qom[first + i] * dt / 2 / c,
                                  cp ? cp->perm : nullptr, copy ? (double*)cp->out.rx : nullptr,
                                  copy ? (double*)cp->out.ry : nullptr, copy ? (double*)cp->out.rz : nullptr,
                                  copy ? (Vel*)cp->out.u : nullptr, copy ? (Vel*)cp->out.v : nullptr,
                                  copy ? (Vel*)cp->out.w : nullptr, copy ? cp->out.q : nullptr,
                                  copy ? cp->out.cell : nullptr};
  }
  return mp;
}

}  // namespace

cudaError_t launch_deposit_moments(int precision, int mass_kind, const Geom& g, int ns, const double* qom, double dt,
                                   double c, const tpicb200_particles* const* p, const uint32_t* const* counts,
                                   const uint32_t* const* offsets, const void* bnode, void* moments, int accumulate,
                                   uint32_t* invalid, const SortedCopy* const* copies, cudaStream_t s) {
  if (!moments || ns < 1) return cudaErrorInvalidValue;
  const long long cells = (long long)g.nx * g.ny * g.nz;
  const bool dbl = precision == TPICB200_PRECISION_DOUBLE;
  const bool f32 = !dbl && mass_kind == TPICB200_MASS_SCALAR;
  constexpr size_t bytes = kF32Warps * sizeof(F32Warp);
  if (f32) {
    const cudaError_t e = cudaFuncSetAttribute(moments_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(bytes));
    if (e != cudaSuccess) return e;
  }
  const unsigned f64_blocks = unsigned(std::min<long long>((cells + kF64Warps - 1) / kF64Warps, 148LL * 4));
  // Batches of four cells once each resident warp has one.
  const int batch = cells >= 4LL * 148 * 4 * kF32Warps ? 4 : 1;
  const long long batches = (cells + batch - 1) / batch;
  const unsigned f32_blocks = unsigned(std::min<long long>((batches + kF32Warps - 1) / kF32Warps, 148LL * 4));
  for (int first = 0; first < ns; first += kFuse) {
    const int acc = (accumulate || first > 0) ? 1 : 0;
    if (dbl) {
      const auto mp = moment_params<double>(g, first, ns, qom, dt, c, p, counts, offsets, copies);
      moments_f64_kernel<double, double, double><<<f64_blocks, kF64Warps * 32, 0, s>>>(
          g, mp, (const double*)bnode, (double*)moments, acc, invalid);
    } else {
      const auto mp = moment_params<float>(g, first, ns, qom, dt, c, p, counts, offsets, copies);
      if (f32)
        moments_f32_kernel<<<f32_blocks, kF32Warps * 32, bytes, s>>>(g, mp, (const float*)bnode, (float*)moments, acc,
                                                                     batch, invalid);
      else
        moments_f64_kernel<float, float, float><<<f64_blocks, kF64Warps * 32, 0, s>>>(
            g, mp, (const float*)bnode, (float*)moments, acc, invalid);
    }
    count_launches(1);
    if (cudaError_t e = cudaGetLastError()) return e;
  }
  return cudaSuccess;
}

}  // namespace tpicb200
