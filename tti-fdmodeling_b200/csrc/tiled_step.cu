// Tiled half-step kernels: the velocity update (coord:614-672, tensor:617-666,
// bond:654-703) and the stress update (coord:804-845, tensor:799-851 with the
// sigma = R tau pass fused, bond:836-873), each in place.
//
// A CTA owns a tile of up to 120 rows and 8 columns. One elected thread loads
// the tile plus the stencil halo of every input field with a 2D TMA copy
// (cp.async.bulk.tensor, completion on an mbarrier, bounded wait); the box
// starts at row z0 - 8, so its innermost coordinate stays 16-byte aligned, and
// coordinates outside the array read zeros. The stencil sums come from the
// diagonal walks of walk.cuh (per four cells of the velocity update 51 shared
// loads, 24 stores of the sums and 6 16-byte reads of them, instead of 240 loads),
// then each lane updates four rows of one column with 128-bit accesses and packed
// arithmetic. The velocity kernel reads only stress
// and the stress kernel only velocity from the boxes, so in-place updates are
// race-free.
//
// What bounds them, 1126 x 7872 coordinate (9.48 M cells), B200: the stress
// update moves its compulsory bytes at 6.2 TB/s of DRAM traffic (82 us; 92 us
// with one cell per thread and ten shared reads per sum); its own inputs come
// by TMA too, with which four CTAs fit an SM and no load waits behind a
// barrier (91 us when loaded into registers after the walks). The velocity
// update (66 us; 94 us before) is bound by the copies' latency at four CTAs per
// SM (the registers' limit), 5.7 TB/s; TMA for its five inputs measured 71 us,
// a persistent grid with the next tile's copies in flight 98 us, sums in the
// boxes' place, which leaves more L1 but needs two barriers more, 74 us.
// Tiles of at most 120 rows need four warps of diagonals per field (128 rows
// need five): 200 x 400 took 11.5 against 13.9 us a step with 128.
//
// A small grid is bound by the latency of its two launches, each about 2.5 us in
// a graph of which 2 are copies' latency, walk, update and stores in series.
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "columns.cuh"
#include "walk.cuh"

namespace ttifd {
namespace tiled {

namespace {

// arguments of a batched half-step launch
struct BatchArgs {
  const HalfArgs *inst;  // each instance's arguments
  const void *maps;      // each instance's VelocityMaps or StressMaps
  const Work *work;      // the work table
  const int *step;       // the shared step counter
  int nwork, offset;     // offset: steps past the counter
  float nzero;           // -0.0f (see walk::coefs)
  unsigned wait_limit;   // polls of a box wait before it gives up
};

using walk::F4;
using walk::ld4;
using walk::ldg4;
using walk::st4;
using walk::WX;

// a tile's origin and a thread's cells: column x, rows z .. z + 3
struct Cells {
  int x0, z0, x, z;
  bool on;  // some of the rows are updated
};
__device__ __forceinline__ Cells cells_of(const HalfArgs &a, int z0, int x0)
{
  const int t = threadIdx.x;
  Cells c;
  c.z0 = z0;
  c.x0 = x0;
  c.x = x0 + (t >> 5);
  c.z = z0 + 4 * (t & 31);
  c.on = c.x < a.g.Nx - NH && 4 * (t & 31) < a.tile_rows && c.z + 3 >= a.g.izStart && c.z < a.g.Nz - NH;
  return c;
}

// Q (FMA mode, dx == dz): the coefficients carry h = 0.5 / dx, so a derivative
// is d1 + d2 or d1 - d2 without a product.
template <bool Q>
__device__ __forceinline__ walk::Coefs coefs(const HalfArgs &a, float nzero)
{
  return Q ? walk::coefs(a.hc[0], a.hc[1], a.hc[2], a.hc[3], a.hc[4], nzero)
           : walk::coefs(rsg(0), rsg(1), rsg(2), rsg(3), rsg(4), nzero);
}

// The velocity update reads its cells' inputs from global memory: while the
// boxes are in flight, each warp asks L2 for the lines of one of them
// (HalfArgs::ahead; the table's last two are coef1 and coef2, not read in
// undamped tiles).
__device__ __forceinline__ void prefetch_velocity(const HalfArgs &a, bool und, int z0, int x0)
{
  const int w = threadIdx.x >> 5;
  if (w < a.nahead - (und ? 2 : 0)) walk::prefetch_lines(a.ahead[w], a.g, x0, z0, a.tile_rows);
}
// Of the stress update's inputs only coef1 and coef2 come from there.
__device__ __forceinline__ void prefetch_stress(const HalfArgs &a, bool und, int z0, int x0)
{
  const int w = threadIdx.x >> 5;
  if (und || w == 0 || w > 2) return;
  walk::prefetch_lines(w == 1 ? a.p.coef1 : a.p.coef2, a.g, x0, z0, a.tile_rows);
}

// coef1, coef2 of a thread's rows
__device__ __forceinline__ void load_coefs(const HalfArgs &a, bool und, size_t gi, F4 &c1, F4 &c2)
{
  if (und) {
    c1.p[0] = c1.p[1] = walk::pack2(1.0f, 1.0f);
    c2.p[0] = c2.p[1] = walk::pack2(a.dt, a.dt);
  } else {
    c1 = ldg4(a.p.coef1 + gi);
    c2 = ldg4(a.p.coef2 + gi);
  }
}

// Shared memory of a velocity tile: the three boxes, the six sum arrays, the
// barrier. Stress tile: the two boxes, whose place the four sum arrays take
// once the walks have read them, the tile's own inputs (StressMaps::in),
// tile_rows x WX each, the barrier.
constexpr int V_SUMS = walk::LEAD + 3 * walk::BOX, V_BAR = V_SUMS + 6 * walk::SUM;
constexpr int V_STASH = V_BAR + 16, V_END = V_STASH + walk::NT / 32 * 11 * 4;  // (single shots: source_terms)
constexpr int S_IN = walk::LEAD + 2 * walk::BOX;
static_assert(4 * walk::SUM <= 2 * walk::BOX, "the sums fit in place of the boxes");
constexpr int s_inputs(int V) { return V == TTI_TENSOR ? 10 : 9; }
constexpr int s_bar(int V) { return S_IN + s_inputs(V) * walk::WZ * WX; }

// this launch's step, and the offset of its slot among the kept steps
__device__ __forceinline__ int step_of(const HalfArgs &a) { return a.clk ? a.clk[0] + a.n : a.n; }
__device__ __forceinline__ size_t kept_at(const HalfArgs &a, int n)
{
  return (size_t)(n - (a.clk ? a.clk[1] : a.k0)) * a.kstride;
}

// per-cell inputs of the velocity update, four rows
struct VCells {
  F4 vx, vz, c1, c2, ir, sv, cv;
};

template <int V>
__device__ __forceinline__ void load_vcells(const HalfArgs &a, bool und, size_t gi, VCells &o)
{
  o.vx = ld4(a.f.vx + gi);
  o.vz = ld4(a.f.vz + gi);
  load_coefs(a, und, gi, o.c1, o.c2);
  o.ir = ldg4(a.p.invrho + gi);
  if (V == TTI_COORDINATE) {
    o.sv = ldg4(a.p.snv + gi);
    o.cv = ldg4(a.p.csv + gi);
  }
}

// The velocity update of a thread's rows from their stencil sums d[f] = (d1,
// d2) of sxx, szz, sxz (coord:614-672, tensor:617-666, bond:654-703).
template <int V, bool X, bool Q, bool K>
__device__ __forceinline__ void velocity_rows(const HalfArgs &a, const Cells &c, size_t gi, const F4 (&d)[3][2],
                                              const VCells &p, walk::u64 nz, int n, F4 &vx, F4 &vz)
{
  typedef walk::Rows<X> A;
  typedef typename A::T T;
  const A r{nz};
  const T invdx = r.c(a.invdx), invdz = r.c(a.invdz), half = r.c(0.5f);
  F4 kd[4];
#pragma unroll
  for (int i = 0; i < A::N; ++i) {
    // x and z derivatives 0.5 (d1 +- d2) / dx, / dz (already scaled when Q)
    auto dx_ = [&](int f) {
      const T s = r.add(A::get(d[f][0], i), A::get(d[f][1], i));
      return Q ? s : r.mul(r.mul(half, s), invdx);
    };
    auto dz_ = [&](int f, T inv) {
      const T s = r.sub(A::get(d[f][0], i), A::get(d[f][1], i));
      return Q ? s : r.mul(r.mul(half, s), inv);
    };
    const T sxx_x = dx_(0);
    const T szz_z = dz_(1, invdz);
    const T sxz_x = dx_(2);
    const T sxz_z = dz_(2, invdz);
    const T br = r.mul(A::get(p.c2, i), A::get(p.ir, i));
    T fx, fz;
    if (V == TTI_COORDINATE) {
      const T sv = A::get(p.sv, i), cv = A::get(p.cv, i);
      const T sxx_z = dz_(0, invdx);  // invdx as coord:633
      const T szz_x = dx_(1);
      fx = r.add(r.add(r.sub(r.mul(cv, sxx_x), r.mul(sv, sxx_z)), r.mul(sv, sxz_x)), r.mul(cv, sxz_z));
      fz = r.add(r.add(r.sub(r.mul(cv, sxz_x), r.mul(sv, sxz_z)), r.mul(sv, szz_x)), r.mul(cv, szz_z));
      if (K) {
        A::set(kd[0], i, r.sub(sxz_x, sxx_z));
        A::set(kd[1], i, r.sub(szz_x, sxz_z));
        A::set(kd[2], i, r.add(sxx_x, sxz_z));
        A::set(kd[3], i, r.add(sxz_x, szz_z));
      }
    } else {
      fx = r.add(sxx_x, sxz_z);
      fz = r.add(sxz_x, szz_z);
    }
    const T c1 = A::get(p.c1, i);
    A::set(vx, i, r.add(r.mul(c1, A::get(p.vx, i)), r.mul(br, fx)));
    A::set(vz, i, r.add(r.mul(c1, A::get(p.vz, i)), r.mul(br, fz)));
  }
  if (K && V == TTI_COORDINATE) {
    const int lo = a.g.izStart, hi = min(a.g.Nz - NH, c.z0 + a.tile_rows);
    const size_t ki = kept_at(a, n) + gi;
#pragma unroll
    for (int k = 0; k < 4; ++k) st4(a.kd[k] + ki, kd[k], c.z, lo, hi);
  }
}

// the sums of N fields at a thread's rows
template <int N>
__device__ __forceinline__ void read_sums(const Cells &c, const float *sums, F4 (&d)[N][2])
{
  const int r1 = walk::d1_at(c.x - c.x0, c.z - c.z0), r2 = walk::d2_at(c.x - c.x0, c.z - c.z0);
#pragma unroll
  for (int f = 0; f < N; ++f) {
    d[f][0] = ld4(sums + 2 * f * walk::SUM + r1);
    d[f][1] = ld4(sums + (2 * f + 1) * walk::SUM + r2);
  }
}

// Column work in the tiles instead of a launch between the half-steps: us a
// step with and without, when it was moved (before it went off the critical
// path, column_work), 60 x 80 9.1 / 9.8, 200 x 400 11.6 / 14.3, 600 x 1200 19.2 /
// 20.2, 1126 x 7872 147.1 / 150.6.
// The rows whose column work a tile does: its own, the first and the last tile
// also those above and below all tiles.
__device__ __forceinline__ bool tile_work(const HalfArgs &a, int z0, int &r0, int &r1)
{
  r0 = z0 == a.z_base ? 0 : z0;
  r1 = z0 + a.tile_rows >= a.g.Nz - NH ? a.g.Nz : z0 + a.tile_rows;
  return r0 < a.work_z1 && r1 > a.work_z0;
}

__device__ __forceinline__ void st_shared4(float *p, const F4 &f)
{
  *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(f.p[0], f.p[1]);
}

// The velocity sources in the tile, one warp (all lanes) a column: as
// column_sources, but what they add is ready when the update is done
// (plan_sources before the wait for the previous kernel, source_terms while the
// copies are in flight) and the column's new rows take it in shared memory.
// Columns under several sources' windows go the general way. us a step, stype 4
// at 60 x 80 8.0 / 7.6, 200 x 400 8.6 / 7.9, 600 x 1200 19.5 / 18.65; stype 6 in
// the tensor rotation 401 x 857 13.3 / 12.8. A kernel of its own (W): where there
// are no velocity sources the plain one takes 60.5 against 61.1 us a step at
// 1126 x 3000.
struct SourcePlan {
  int src = -1, row = 0, mask = 0;  // the source; this lane's row; which of w there are
  float w[4];                       // weights: to vx, to vz, then to vx, to vz again (stype 4: 2, then 3)
  bool more = false;
};
__device__ __forceinline__ void plan_sources(const HalfArgs &a, int ix, int r0, int r1, SourcePlan &s)
{
  const Columns &p = *a.cols;
  const int lane = threadIdx.x & 31;
  const bool in = source_column(p, ix);
  const int4 e = __ldg(p.shead + (in ? ix - p.sx0 : 0));  // (not behind a branch: 12.59 against 12.73 us a step
                                                          // at 401 x 857, tensor rotation, stype 6)
  if (!in) return;
  s.more = e.w > 1;
  if (e.w != 1) return;
  s.src = e.x;
  const int dx = e.z, z = e.y, i = (dx + NH) * 11 + lane;
  s.row = z + lane - NH;
  if (p.stype == 8) {  // rows z and z - 1 of two columns
    s.row = z - lane;
    if (lane < 2 && (dx == 0 || dx == -1)) s.mask = 3;
    s.w[0] = lane ? p.t.q8 : -p.t.q8;
    s.w[1] = dx == 0 ? p.t.q8 : -p.t.q8;
  } else if (lane <= 2 * NH) {
    const int k = p.stype;
    s.mask = k == 4 ? 15 : k == 5 ? 1 : k == 6 ? 2 : 3;
    s.w[0] = k == 3 ? -p.t.kz[i] : k == 5 ? p.t.k5[i] : k == 7 ? p.t.k7[i] : p.t.kx[i];
    s.w[1] = k == 3 ? p.t.kx[i] : k == 6 ? p.t.k5[i] : k == 7 ? p.t.k7[i] : p.t.kz[i];
    s.w[2] = -p.t.kz[i];
    s.w[3] = p.t.kx[i];
  }
  if (s.row < max(r0, 0) || s.row >= min(r1, a.g.Nz)) s.mask = 0;
}

// Rows of the tile: the terms go to `stash` (four floats a lane), returned are
// the row and the mask. Rows that are not updated take them at once.
constexpr int SRC_ON = 1 << 16, SRC_MORE = 1 << 17;
__device__ __forceinline__ int source_terms(const HalfArgs &a, int ix, int z0, const SourcePlan &s, float *stash)
{
  if (s.more) return SRC_MORE;
  if (s.src < 0) return 0;
  const Columns &p = *a.cols;
  const float t = p.amp[(size_t)s.src * p.nt + time_index(p, step_of(a))];
  if (!s.mask) return SRC_ON;
  float u[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) u[k] = s.mask >> k & 1 ? __fmul_rn(s.w[k], t) : 0.0f;
  if (s.row >= a.g.izStart && s.row < a.g.Nz - NH) {
    *reinterpret_cast<float4 *>(stash) = make_float4(u[0], u[1], u[2], u[3]);
    return SRC_ON | s.mask << 8 | (s.row - z0);
  }
  const size_t i = (size_t)ix * a.g.ldz + s.row;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (s.mask >> k & 1) {
      float *v = (k & 1 ? a.f.vz : a.f.vx) + i;
      *v = __fadd_rn(*v, u[k]);
    }
  return SRC_ON;
}

// Velocity update of a tile whose boxes (sxx, szz, sxz) have arrived: one warp
// per field and 32 diagonals, then one per column.
template <int V, bool X, bool Q, bool K, bool W>
__device__ __forceinline__ void velocity_tile(const HalfArgs &a, const Cells &c, bool und, const walk::Coefs &k,
                                              float *sm, int n, bool early, int src)
{
  const int gr = walk::groups(a.tile_rows);
  float *sums = sm + V_SUMS;
  for (int t = threadIdx.x >> 5; t < 3 * gr; t += walk::NT / 32) {
    const int f = (t >= gr) + (t >= 2 * gr), d = (t - f * gr) * 32 + (threadIdx.x & 31);
    const float *box = sm + walk::LEAD + f * walk::BOX;
    if (d < a.tile_rows + WX - 1) {
      walk::u64 out[WX];
      walk::diagonals<0, X>(box, box, d, k, out);
      walk::put_sums(sums + 2 * f * walk::SUM, sums + (2 * f + 1) * walk::SUM, d, out);
    }
  }
  const size_t gi = (size_t)c.x * a.g.ldz + c.z;
  VCells p;
  if (c.on) load_vcells<V>(a, und, gi, p);
  __syncthreads();  // the sums are complete
  if (!early) pdl_trigger();
  const int lo = a.g.izStart, hi = min(a.g.Nz - NH, c.z0 + a.tile_rows);
  F4 vx, vz;
  if (c.on) {
    F4 ds[3][2];
    read_sums(c, sums, ds);
    velocity_rows<V, X, Q, K>(a, c, gi, ds, p, k.nz, n, vx, vz);
    if (!W || !(src & SRC_ON)) {
      st4(a.f.vx + gi, vx, c.z, lo, hi);
      st4(a.f.vz + gi, vz, c.z, lo, hi);
    }
  }
  if (!W) return;
  const int lane = threadIdx.x & 31;
  if (src & SRC_ON) {  // this warp's column
    float *S = sums + (c.x - c.x0) * walk::DP;
    const float *stash = sm + V_STASH + ((threadIdx.x >> 5) * 11 + lane) * 4;
    __syncwarp();  // every lane has read the column's sums
    if (c.on) {
      st_shared4(S + 4 * lane, vx);
      st_shared4(S + walk::SUM + 4 * lane, vz);
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (src >> (8 + k) & 1) {
        float *v = S + (k & 1) * walk::SUM + (src & 255);
        *v = __fadd_rn(*v, stash[k]);
      }
    __syncwarp();
    if (c.on) {
      st4(a.f.vx + gi, ld4(S + 4 * lane), c.z, lo, hi);
      st4(a.f.vz + gi, ld4(S + walk::SUM + 4 * lane), c.z, lo, hi);
    }
  }
  if (src & SRC_MORE) {
    int r0, r1;
    tile_work(a, c.z0, r0, r1);
    __syncwarp();
    column_sources(a.g, a.f, *a.cols, c.x, n, r0, r1);
  }
}

// per-cell inputs of the stress update, four rows
struct SCells {
  F4 o[3];  // sigma (coordinate, Bond) or tau (tensor)
  F4 c1, c2, c11, c13, c33, c55;
  F4 p, q, r;  // sin, cos theta; sin^2, cos^2, sin 2 theta; c15, c35
};

template <int V>
__device__ __forceinline__ void load_scells(const HalfArgs &a, bool und, const Cells &c, size_t gi, const float *sm,
                                            SCells &s)
{
  const float *in = sm + S_IN + (c.x - c.x0) * a.tile_rows + (c.z - c.z0);
  auto at = [&](int k) { return ld4(in + k * WX * a.tile_rows); };
#pragma unroll
  for (int k = 0; k < 3; ++k) s.o[k] = at(k);
  s.p = at(3);
  s.q = at(4);
  s.c11 = at(5);
  s.c13 = at(6);
  s.c33 = at(7);
  s.c55 = at(8);
  if (V == TTI_TENSOR) s.r = at(9);
  load_coefs(a, und, gi, s.c1, s.c2);
}

// The stress update of a thread's rows from their stencil sums d[f] = (d1, d2)
// of vx, vz (coord:804-845, tensor:799-851, bond:836-873): n the new sigma, t
// the new tau (tensor). What the gradient keeps of them goes to kd and kt.
template <int V, bool X, bool Q, bool K>
__device__ __forceinline__ void stress_rows(const HalfArgs &a, const Cells &c, size_t gi, const F4 (&d)[2][2],
                                            const SCells &s, walk::u64 nz, int step, F4 (&n)[3], F4 (&t)[3])
{
  typedef walk::Rows<X> A;
  typedef typename A::T T;
  const A r{nz};
  const T invdx = r.c(a.invdx), invdz = r.c(a.invdz), half = r.c(0.5f);
  const int lo = a.g.izStart, hi = min(a.g.Nz - NH, c.z0 + a.tile_rows);
  F4 e[4];  // vxx vxz vzx vzz
#pragma unroll
  for (int i = 0; i < A::N; ++i)
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      const T d1 = A::get(d[f][0], i), d2 = A::get(d[f][1], i), p = r.add(d1, d2), m = r.sub(d1, d2);
      A::set(e[2 * f], i, Q ? p : r.mul(r.mul(half, p), invdx));
      A::set(e[2 * f + 1], i, Q ? m : r.mul(r.mul(half, m), invdz));
    }
  if (K) {
    const size_t ki = kept_at(a, step) + gi;
#pragma unroll
    for (int k = 0; k < 4; ++k) st4(a.kd[k] + ki, e[k], c.z, lo, hi);
    if (V == TTI_TENSOR)
#pragma unroll
      for (int k = 0; k < 3; ++k) st4(a.kt[k] + ki, s.o[k], c.z, lo, hi);
  }
#pragma unroll
  for (int i = 0; i < A::N; ++i) {
    T vxx = A::get(e[0], i), vxz = A::get(e[1], i), vzx = A::get(e[2], i), vzz = A::get(e[3], i);
    const T c1 = A::get(s.c1, i), c2 = A::get(s.c2, i);
    const T o0 = A::get(s.o[0], i), o1 = A::get(s.o[1], i), o2 = A::get(s.o[2], i);
    const T c11 = A::get(s.c11, i), c13 = A::get(s.c13, i), c33 = A::get(s.c33, i), c55 = A::get(s.c55, i);
    if (V == TTI_COORDINATE) {
      const T sn = A::get(s.p, i), cs = A::get(s.q, i);
      T q = r.add(r.mul(sn, vxx), r.mul(cs, vxz));
      vxx = r.sub(r.mul(cs, vxx), r.mul(sn, vxz));
      vxz = q;
      q = r.add(r.mul(sn, vzx), r.mul(cs, vzz));
      vzx = r.sub(r.mul(cs, vzx), r.mul(sn, vzz));
      vzz = q;
      A::set(n[0], i, r.add(r.mul(c1, o0), r.mul(c2, r.add(r.mul(c11, vxx), r.mul(c13, vzz)))));
      A::set(n[1], i, r.add(r.mul(c1, o1), r.mul(c2, r.add(r.mul(c13, vxx), r.mul(c33, vzz)))));
      A::set(n[2], i, r.add(r.mul(c1, o2), r.mul(r.mul(c2, c55), r.add(vzx, vxz))));
    } else if (V == TTI_TENSOR) {
      const T s2 = A::get(s.p, i), cc2 = A::get(s.q, i), s2t = A::get(s.r, i);
      const T sh = r.add(vxz, vzx), hs = r.mul(half, s2t);
      const T exx = r.sub(r.add(r.mul(cc2, vxx), r.mul(s2, vzz)), r.mul(hs, sh));
      const T ezz = r.add(r.add(r.mul(s2, vxx), r.mul(cc2, vzz)), r.mul(hs, sh));
      const T exz = r.add(r.mul(s2t, r.sub(vxx, vzz)), r.mul(r.sub(cc2, s2), sh));
      const T ntx = r.add(r.mul(c1, o0), r.mul(c2, r.add(r.mul(c11, exx), r.mul(c13, ezz))));
      const T ntz = r.add(r.mul(c1, o1), r.mul(c2, r.add(r.mul(c13, exx), r.mul(c33, ezz))));
      const T ntq = r.add(r.mul(c1, o2), r.mul(r.mul(c2, c55), exz));
      A::set(t[0], i, ntx);
      A::set(t[1], i, ntz);
      A::set(t[2], i, ntq);
      A::set(n[0], i, r.add(r.add(r.mul(cc2, ntx), r.mul(s2, ntz)), r.mul(s2t, ntq)));
      A::set(n[1], i, r.sub(r.add(r.mul(s2, ntx), r.mul(cc2, ntz)), r.mul(s2t, ntq)));
      A::set(n[2], i, r.add(r.mul(r.mul(r.c(-0.5f), s2t), r.sub(ntx, ntz)), r.mul(r.sub(cc2, s2), ntq)));
    } else {
      const T c15 = A::get(s.p, i), c35 = A::get(s.q, i);
      const T sh = r.add(vzx, vxz);
      A::set(n[0], i,
             r.add(r.mul(c1, o0), r.mul(c2, r.add(r.add(r.mul(c11, vxx), r.mul(c13, vzz)), r.mul(c15, sh)))));
      A::set(n[1], i,
             r.add(r.mul(c1, o1), r.mul(c2, r.add(r.add(r.mul(c13, vxx), r.mul(c33, vzz)), r.mul(c35, sh)))));
      A::set(n[2], i,
             r.add(r.mul(c1, o2), r.mul(c2, r.add(r.add(r.mul(c15, vxx), r.mul(c35, vzz)), r.mul(c55, sh)))));
    }
  }
}

// The column work after the stress update in the tile, one warp (all lanes) a
// column: column_post's work on rows [r0, r1), arranged so that what it reads
// is there when it is needed. With every load after the update, as k_post does
// it, each dependent load cost an L2 latency at the end of the kernel: 5000
// cycles a stress launch at 60 x 80, of which 1600 for the source and 2000 for
// the receivers. us a step with the loads there / as below: coordinate 60 x 80
// 8.0 / 6.4, 200 x 400 10.8 / 9.2, 600 x 1200 19.0 / 18.9, 1126 x 3000 62.0 /
// 61.2; tensor 1126 x 3000 71.5 / 69.5.
//   plan_column     before the wait for the previous kernel: the geometry
//   sample_column   while the tile's copies are in flight: the velocity
//                   receivers, the first stress source's amplitudes
//   column_work     after the update: the rest, in shared memory
// The host folds the work in only where every row of it is updated or an image
// row (sync_columns).
struct ColumnPlan {
  int rz[3] = {-1, -1, -1}, rid[3];  // first 32 receivers of a component, one per lane
  int src = -1, sz = -1;             // first source whose window has the column; this lane's row in it
  bool more = false;                 // there may be further sources, receivers
  float ws = 0.0f;                   // what that source adds to the lane's row
};
// What is left of it after the update (held through the stencil walks, so few
// registers: whole plans spilled there). Rows are the tile's, + 8.
struct ColumnRest {
  static constexpr int NO_ROW = 255;
  int pr = NO_ROW, sr = NO_ROW;  // of the lane's pressure sample and of the first source
  bool more = false;
  float ws = 0.0f;
  float *rec = nullptr;  // where the pressure sample goes
};

__device__ __forceinline__ void plan_column(const HalfArgs &a, int ix, int r0, int r1, ColumnPlan &c)
{
  const Columns &p = *a.cols;
  const int lane = threadIdx.x & 31;
  if (p.rec_on) {
    int rb[3], re[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      rb[k] = re[k] = 0;
      if (p.colptr[k]) {
        rb[k] = p.colptr[k][ix];
        re[k] = p.colptr[k][ix + 1];
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (rb[k] + lane < re[k]) {
        c.rz[k] = p.rz[k][rb[k] + lane];
        c.rid[k] = p.rid[k][rb[k] + lane];
        if (c.rz[k] < r0 || c.rz[k] >= r1) c.rz[k] = -1;
      }
      c.more |= re[k] - rb[k] > 32;
    }
  }
  if (p.stype == 1 && source_column(p, ix)) {
    const int4 e = __ldg(p.shead + (ix - p.sx0));
    if (e.w == 0) return;
    c.more |= e.w > 1;
    c.src = e.x;
    c.sz = e.y + lane - NH;
    if (lane > 2 * NH || c.sz < r0 || c.sz >= r1) c.sz = -1;
    else c.ws = p.t.k1[(e.z + NH) * 11 + lane];
  }
}

__device__ __forceinline__ void put_sample(const Columns &p, float *rec, float v)
{
  *rec = v;
  if (!isfinite(v)) atomicOr(p.flag, 1);
}

template <int V>
__device__ __forceinline__ ColumnRest sample_column(const HalfArgs &a, int ix, int z0, const ColumnPlan &c)
{
  const Columns &p = *a.cols;
  const size_t col = (size_t)ix * a.g.ldz;
  const float vx = c.rz[0] >= 0 ? a.f.vx[col + c.rz[0]] : 0.0f, vz = c.rz[1] >= 0 ? a.f.vz[col + c.rz[1]] : 0.0f;
  const int it = time_index(p, step_of(a)), irec = record_index(p, it);
  ColumnRest w;
  w.more = c.more;
  if (c.src >= 0) w.ws = __fmul_rn(c.ws, p.amp[(size_t)c.src * p.nt + it]);
  if (c.sz >= 0) {
    w.sr = c.sz - z0 + 8;
    if (V == TTI_TENSOR && c.sz < max(z0, a.g.izStart)) {  // tau of the image rows changes nowhere else
      a.f.txx[col + c.sz] = __fadd_rn(a.f.txx[col + c.sz], w.ws);
      a.f.tzz[col + c.sz] = __fadd_rn(a.f.tzz[col + c.sz], w.ws);
    }
  }
  if (irec < 0) return w;
  if (c.rz[2] >= 0) {
    w.pr = c.rz[2] - z0 + 8;
    w.rec = p.rec[2] + (size_t)irec * p.nrec[2] + c.rid[2];
  }
  if (c.rz[0] >= 0) put_sample(p, p.rec[0] + (size_t)irec * p.nrec[0] + c.rid[0], vx);
  if (c.rz[1] >= 0) put_sample(p, p.rec[1] + (size_t)irec * p.nrec[1] + c.rid[1], vz);
  return w;
}

// Sources after the first of a column and receivers after 32 of a component;
// S: row 0 of the column's sigma.
template <typename F>
__device__ __forceinline__ void more_work(const HalfArgs &a, int ix, int r0, int r1, F source, const float *S)
{
  const Columns &p = *a.cols;
  const int lane = threadIdx.x & 31, it = time_index(p, step_of(a)), irec = record_index(p, it);
  if (p.stype == 1 && source_column(p, ix)) {
    const ColumnSources src(p, ix, it);
    for (int j = src.first + 1; j < src.last; ++j) {
      const int4 s = src.at(j);
      const int iz = s.y + lane - NH;
      if (lane <= 2 * NH && iz >= r0 && iz < r1)
        source(iz, __fmul_rn(__ldg(p.t.k1 + (s.z + NH) * 11 + lane), src.amp(s)), false);
      __syncwarp();
    }
  }
  if (irec < 0) return;
  for (int k = 0; k < 3; ++k) {
    if (!p.colptr[k]) continue;
    const int re = p.colptr[k][ix + 1];
    for (int j = p.colptr[k][ix] + lane + (k < 2 ? 32 : 0); j < re; j += 32) {
      const int rz = p.rz[k][j];
      if (rz < r0 || rz >= r1) continue;
      const size_t i = (size_t)ix * a.g.ldz + rz;
      const float v = k == TTI_REC_VX   ? a.f.vx[i]
                      : k == TTI_REC_VZ ? a.f.vz[i]
                                        : __fmul_rn(0.5f, __fadd_rn(S[rz], S[walk::SUM + rz]));
      put_sample(p, p.rec[k] + (size_t)irec * p.nrec[k] + p.rid[k][j], v);
    }
  }
}

// S: the column's sigma, rows -8 .. 119 of the tile, in place of its sums; tau
// (tensor) in place of its inputs.
template <int V>
__device__ __forceinline__ void column_work(const HalfArgs &a, const Cells &c, size_t gi, const F4 (&n)[3],
                                            const F4 (&t)[3], float *sm, const ColumnRest &w, int r0, int r1)
{
  const Grid &g = a.g;
  const int lane = threadIdx.x & 31;
  const int cx = c.x - c.x0, s = g.izStart - c.z0;
  float *S = sm + walk::LEAD + cx * walk::DP + 8, *U = sm + S_IN + cx * a.tile_rows;
  constexpr int F = walk::SUM;  // from one field of S to the next
  const int M = WX * a.tile_rows;
  const bool fs = a.freesurface && g.izStart >= r0 && g.izStart < r1;
  __syncwarp();  // every lane has read the column's sums and inputs
  if (c.on) {
#pragma unroll
    for (int k = 0; k < 3; ++k) st_shared4(S + k * F + 4 * lane, n[k]);
    if (V == TTI_TENSOR)
#pragma unroll
      for (int k = 0; k < 2; ++k) st_shared4(U + k * M + 4 * lane, t[k]);
  }
  __syncwarp();
  if (fs) {  // coord:847-863
    if (lane >= 1 && lane <= NH) {
      S[s - lane] = __fsub_rn(__fmul_rn(2.0f, S[s]), S[s + lane]);
      S[F + s - lane] = -S[F + s + lane];
      S[2 * F + s - lane] = -S[2 * F + s + lane];
    }
    __syncwarp();
    if (lane == 0) S[F + s] = S[2 * F + s] = 0.0f;
    __syncwarp();
  }
  auto source = [&](int iz, float ws, bool first) {
    const int r = iz - c.z0;
    S[r] = __fadd_rn(S[r], ws);
    S[F + r] = __fadd_rn(S[F + r], ws);
    if (V == TTI_TENSOR) {
      if (r >= 0 && iz >= g.izStart) {
        U[r] = __fadd_rn(U[r], ws);
        U[M + r] = __fadd_rn(U[M + r], ws);
      } else if (!first) {  // (the first source's: sample_column)
        const size_t i = (size_t)c.x * g.ldz + iz;
        a.f.txx[i] = __fadd_rn(a.f.txx[i], ws);
        a.f.tzz[i] = __fadd_rn(a.f.tzz[i], ws);
      }
    }
  };
  const int pr = w.pr, sr = w.sr;
  if (sr != ColumnRest::NO_ROW) source(c.z0 + sr - 8, w.ws, true);
  __syncwarp();
  if (w.more) more_work(a, c.x, r0, r1, source, S - c.z0);
  else if (pr != ColumnRest::NO_ROW) put_sample(*a.cols, w.rec, __fmul_rn(0.5f, __fadd_rn(S[pr - 8], S[F + pr - 8])));
  const int lo = fs ? g.izStart - NH : g.izStart, hi = min(g.Nz - NH, c.z0 + a.tile_rows);
  float *const f[3] = {a.f.sxx, a.f.szz, a.f.sxz};
  if (c.z + 3 >= lo && 4 * lane < a.tile_rows && c.z < hi)
#pragma unroll
    for (int k = 0; k < 3; ++k) st4(f[k] + gi, ld4(S + k * F + 4 * lane), c.z, lo, hi);
  const int above = c.z0 - 1 - lane;  // image rows above the tile
  if (fs && lane < 8 && above >= lo)
#pragma unroll
    for (int k = 0; k < 3; ++k) f[k][(size_t)c.x * g.ldz + above] = S[k * F - 1 - lane];
  if (V == TTI_TENSOR && c.on) {
    st4(a.f.txx + gi, ld4(U + 4 * lane), c.z, g.izStart, hi);
    st4(a.f.tzz + gi, ld4(U + M + 4 * lane), c.z, g.izStart, hi);
    st4(a.f.txz + gi, t[2], c.z, g.izStart, hi);
  }
}

// Stress update of a tile whose boxes (vx, vz) and inputs have arrived
template <int V, bool X, bool Q, bool K>
__device__ __forceinline__ void stress_tile(const HalfArgs &a, const Cells &c, bool und, const walk::Coefs &k,
                                            float *sm, int step, bool early, const ColumnRest *rest, bool work, int r0,
                                            int r1)
{
  const int gr = walk::groups(a.tile_rows), w = threadIdx.x >> 5, f = w >= gr;
  const int d = (w - f * gr) * 32 + (threadIdx.x & 31);
  const bool on = w < 2 * gr && d < a.tile_rows + WX - 1;  // one walk per warp: 2 gr <= 8
  walk::u64 out[WX];
  if (on) {
    const float *box = sm + walk::LEAD + f * walk::BOX;
    walk::diagonals<1, X>(box, box, d, k, out);
  }
  __syncthreads();  // the boxes have been read
  float *sums = sm + walk::LEAD;
  if (on) walk::put_sums(sums + 2 * f * walk::SUM, sums + (2 * f + 1) * walk::SUM, d, out);
  __syncthreads();  // the sums are complete
  if (!early) pdl_trigger();
  const size_t gi = (size_t)c.x * a.g.ldz + c.z;
  F4 n[3], t[3];
  if (c.on) {
    F4 ds[2][2];
    read_sums(c, sums, ds);
    SCells p;
    load_scells<V>(a, und, c, gi, sm, p);
    stress_rows<V, X, Q, K>(a, c, gi, ds, p, k.nz, step, n, t);
  }
  if (work) {
    if (c.x < a.g.Nx - NH) column_work<V>(a, c, gi, n, t, sm, *rest, r0, r1);  // this warp's column
  } else if (c.on) {
    const int lo = a.g.izStart, hi = min(a.g.Nz - NH, c.z0 + a.tile_rows);
    st4(a.f.sxx + gi, n[0], c.z, lo, hi);
    st4(a.f.szz + gi, n[1], c.z, lo, hi);
    st4(a.f.sxz + gi, n[2], c.z, lo, hi);
    if (V == TTI_TENSOR) {
      st4(a.f.txx + gi, t[0], c.z, lo, hi);
      st4(a.f.tzz + gi, t[1], c.z, lo, hi);
      st4(a.f.txz + gi, t[2], c.z, lo, hi);
    }
  }
}

// Single-shot launches, one tile per CTA.
template <int V, bool X, bool Q, bool K = false, bool W = false>
__global__ void __launch_bounds__(walk::NT, 4) k_velocity_tiled(const __grid_constant__ HalfArgs a,
                                                                const __grid_constant__ VelocityMaps m)
{
  extern __shared__ __align__(128) float sm[];
  unsigned long long *bar = reinterpret_cast<unsigned long long *>(sm + V_BAR);
  const int z0 = a.z_base + blockIdx.x * a.tile_rows, x0 = a.x_base + blockIdx.y * WX;
  walk::init_bar(bar);
  const int ix = x0 + (threadIdx.x >> 5);  // this warp's column
  int r0, r1;
  const bool work = W && tile_work(a, z0, r0, r1) && ix < a.g.Nx - NH;
  SourcePlan plan;
  if (work) plan_sources(a, ix, r0, r1, plan);
  pdl_wait();
  if (a.early) pdl_trigger();
  walk::issue_tile(m.box, 3, 4, nullptr, 0, 0, sm, 0, bar, z0, x0);
  const bool und = tile_undamped(a, z0, x0, WX);
  prefetch_velocity(a, und, z0, x0);
  const int n = step_of(a);
  const int src = work ? source_terms(a, ix, z0, plan, sm + V_STASH + ((threadIdx.x >> 5) * 11 + (threadIdx.x & 31)) * 4) : 0;
  const walk::Coefs k = coefs<Q>(a, a.nzero);
  if (!walk::wait_boxes(a.err, bar, a.wait_limit, 0)) return;
  // tiles without a source's window run the plain update: 61.4 against 62.5 us
  // a step at 1126 x 3000, 18.65 against 19.1 at 600 x 1200
  if (W && __syncthreads_or(src)) velocity_tile<V, X, Q, K, true>(a, cells_of(a, z0, x0), und, k, sm, n, a.early, src);
  else velocity_tile<V, X, Q, K, false>(a, cells_of(a, z0, x0), und, k, sm, n, a.early, 0);
}

// The stress update walks the tiles in the opposite order, so that it starts
// where the velocity update has just been and finds its last tens of megabytes
// in L2 (and the next velocity update starts where this one ended): 67.7
// against 70.3 us a step at 1126 x 3000, 160.3 against 162.7 at 1126 x 7872.
template <int V, bool X, bool Q, bool K = false>
__global__ void __launch_bounds__(walk::NT, K ? 3 : 4) k_stress_tiled(const __grid_constant__ HalfArgs a,
                                                                      const __grid_constant__ StressMaps m)
{
  extern __shared__ __align__(128) float sm[];
  unsigned long long *bar = reinterpret_cast<unsigned long long *>(sm + s_bar(V));
  const int z0 = a.z_base + (gridDim.x - 1 - blockIdx.x) * a.tile_rows;
  const int x0 = a.x_base + (gridDim.y - 1 - blockIdx.y) * WX;
  walk::init_bar(bar);
  const int ix = x0 + (threadIdx.x >> 5);  // this warp's column
  int r0, r1;
  const bool work = tile_work(a, z0, r0, r1);
  ColumnPlan plan;
  if (work && ix < a.g.Nx - NH) plan_column(a, ix, r0, r1, plan);
  pdl_wait();
  if (a.early) pdl_trigger();
  walk::issue_tile(m.box, 2, 5, m.in, s_inputs(V), a.tile_rows, sm, S_IN, bar, z0, x0);
  const bool und = tile_undamped(a, z0, x0, WX);
  prefetch_stress(a, und, z0, x0);
  const int n = step_of(a);
  ColumnRest rest;
  if (work && ix < a.g.Nx - NH) rest = sample_column<V>(a, ix, z0, plan);
  const walk::Coefs k = coefs<Q>(a, a.nzero);
  if (!walk::wait_boxes(a.err, bar, a.wait_limit, 0)) return;
  stress_tile<V, X, Q, K>(a, cells_of(a, z0, x0), und, k, sm, n, a.early, &rest, work, r0, r1);
}

// Batched launches copy the instance's arguments into shared memory: the fields
// are then uniform shared loads that the in-place global stores cannot alias.
// The copy runs while the boxes are in flight and is complete after the block
// barrier of wait_boxes.
static_assert(sizeof(HalfArgs) % 16 == 0, "HalfArgs must be whole 16-byte words");

__device__ __forceinline__ const HalfArgs &stage_args(const HalfArgs *src, void *dst)
{
  const int4 *s4 = reinterpret_cast<const int4 *>(src);
  int4 *d4 = static_cast<int4 *>(dst);
  for (int i = threadIdx.x; i < (int)(sizeof(HalfArgs) / 16); i += walk::NT) d4[i] = __ldg(s4 + i);
  return *static_cast<const HalfArgs *>(dst);
}

// A CTA's work item: item blockIdx.x of the table (from its end for the stress
// update, as in the single-shot kernels). The copies need only the item (its
// tile origin) and the instance's maps, so they are in flight before the
// arguments are staged. `bar` is followed by the staged arguments, 16-byte
// aligned.
template <typename I, typename F>
__device__ __forceinline__ void work_item(const BatchArgs &b, bool reverse, unsigned long long *bar, I issue, F f)
{
  walk::init_bar(bar);
  pdl_sync();
  const int n = *b.step + b.offset, i = reverse ? b.nwork - 1 - blockIdx.x : blockIdx.x;
  const int4 w = __ldg(reinterpret_cast<const int4 *>(b.work + i));  // inst, z0, x0 and the undamped bit, nt
  if (n >= w.w) return;  // uniform over the CTA
  const HalfArgs *src = b.inst + w.x;
  const int x0 = w.z & ~Work::UNDAMPED;
  const bool und = w.z & Work::UNDAMPED;
  issue(*src, w.x, und, w.y, x0);
  const HalfArgs &a = stage_args(src, bar + 2);
  if (!walk::wait_boxes(src->err, bar, b.wait_limit, 0)) return;
  f(a, cells_of(a, w.y, x0), und, n);
}

template <int V, bool X, bool Q>
__global__ void __launch_bounds__(walk::NT, 4) k_velocity_batch(const __grid_constant__ BatchArgs b)
{
  extern __shared__ __align__(128) float sm[];
  unsigned long long *bar = reinterpret_cast<unsigned long long *>(sm + V_BAR);
  work_item(
      b, false, bar,
      [&](const HalfArgs &a, int inst, bool und, int z0, int x0) {
        walk::issue_tile(static_cast<const VelocityMaps *>(b.maps)[inst].box, 3, 4, nullptr, 0, 0, sm, 0, bar, z0, x0);
        prefetch_velocity(a, und, z0, x0);
      },
      [&](const HalfArgs &a, const Cells &c, bool und, int n) {
        velocity_tile<V, X, Q, false, false>(a, c, und, coefs<Q>(a, b.nzero), sm, n, true, 0);
      });
}

template <int V, bool X, bool Q>
__global__ void __launch_bounds__(walk::NT, 4) k_stress_batch(const __grid_constant__ BatchArgs b)
{
  extern __shared__ __align__(128) float sm[];
  unsigned long long *bar = reinterpret_cast<unsigned long long *>(sm + s_bar(V));
  work_item(
      b, true, bar,
      [&](const HalfArgs &a, int inst, bool und, int z0, int x0) {
        const StressMaps &m = static_cast<const StressMaps *>(b.maps)[inst];
        walk::issue_tile(m.box, 2, 5, m.in, s_inputs(V), threadIdx.x ? 0 : a.tile_rows, sm, S_IN, bar, z0, x0);
        prefetch_stress(a, und, z0, x0);
      },
      [&](const HalfArgs &a, const Cells &c, bool und, int n) {
        stress_tile<V, X, Q, false>(a, c, und, coefs<Q>(a, b.nzero), sm, n, true, nullptr, false, 0, 0);
      });
}

// Sets a kernel's shared-memory attributes, once per device.
template <typename K>
cudaError_t prepare_kernel(K kernel, size_t bytes)
{
  static std::mutex mu;
  static std::vector<std::pair<const void *, int>> seen;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const std::pair<const void *, int> key{(const void *)kernel, dev};
  std::lock_guard<std::mutex> lock(mu);
  if (std::find(seen.begin(), seen.end(), key) != seen.end()) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) seen.push_back(key);
  return e;
}

template <typename M>
cudaError_t launch_k(void (*kernel)(HalfArgs, M), const HalfArgs &a, const M &m, size_t smem, cudaStream_t st)
{
  const cudaError_t e = prepare_kernel(kernel, smem);
  if (e != cudaSuccess) return e;
  int z_base, rows;
  const dim3 gr = tiles(a.g, a.g.izStart, &z_base, &rows);
  if (gr.x == 0 || gr.y == 0) return cudaSuccess;
  return launch_pdl(kernel, gr, dim3(walk::NT), smem, st, a, m);
}

}  // namespace


dim3 tiles(const Grid &g, int z_first, int *z_base, int *tile_rows)
{
  // from z_first rounded down to a 32-byte sector; tiles of equal height
  *z_base = z_first & ~7;
  const int nz = g.Nz - NH - *z_base, nx = g.Nx - 2 * NH;
  *tile_rows = walk::WZ;
  if (nz <= 0 || nx <= 0) return dim3(0, 0);
  const int nt = (nz + walk::WZ - 1) / walk::WZ;
  *tile_rows = ((nz + nt - 1) / nt + 7) & ~7;
  return dim3(nt, (nx + WX - 1) / WX);
}

static PFN_cuTensorMapEncodeTiled_v12000 encoder()
{
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    cudaDriverEntryPointQueryResult q;
    void *p = nullptr;
    const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
                    q == cudaDriverEntryPointSuccess;
    return ok ? reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p) : nullptr;
  }();
  return fn;
}

bool encode_map3(CUtensorMap *map, const Grid &g, float *fields, int count, int box_rows, int box_cols)
{
  const auto encode = encoder();
  if (!encode) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)g.ldz, (cuuint64_t)g.Nx, (cuuint64_t)count};
  const cuuint64_t strides[2] = {(cuuint64_t)g.ldz * sizeof(float), (cuuint64_t)g.n * sizeof(float)};
  const cuuint32_t box[3] = {(cuuint32_t)box_rows, (cuuint32_t)box_cols, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, fields, dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool encode_map(CUtensorMap *map, const Grid &g, float *field, int box_rows, int box_cols)
{
  const auto encode = encoder();
  if (!encode) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)g.ldz, (cuuint64_t)g.Nx};
  const cuuint64_t strides[1] = {(cuuint64_t)g.ldz * sizeof(float)};
  const cuuint32_t box[2] = {(cuuint32_t)box_rows, (cuuint32_t)box_cols};
  const cuuint32_t estr[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, field, dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool encode_maps(CUtensorMap *map, const Grid &g, int variant, const Fields &f, const Params &p)
{
  const bool t = variant == TTI_TENSOR, b = variant == TTI_BOND;
  float *const halo[HALO_MAPS] = {f.vx, f.vz, f.sxx, f.szz, f.sxz};
  const float *const in[IN_MAPS] = {t ? f.txx : f.sxx, t ? f.tzz : f.szz, t ? f.txz : f.sxz,
                                    t ? p.s2 : b ? p.c15 : p.sn, t ? p.c2 : b ? p.c35 : p.cs,
                                    p.c11, p.c13, p.c33, p.c55, t ? p.s2t : p.c55};
  int z_base, rows;
  tiles(g, g.izStart, &z_base, &rows);
  for (int k = 0; k < HALO_MAPS; ++k)
    if (!encode_map(map + k, g, halo[k], walk::WB, walk::WBX)) return false;
  for (int k = 0; k < IN_MAPS; ++k)
    if (!encode_map(map + HALO_MAPS + k, g, const_cast<float *>(in[k]), rows, WX)) return false;
  return true;
}

void fill_args(HalfArgs &ha, const tti_handle *h, const StepArgs &a)
{
  const tti_config &c = h->cfg;
  ha = HalfArgs{};
  ha.g = h->g;
  ha.f = a.f;
  ha.p = a.p;
  ha.invdx = h->invdx;
  ha.invdz = h->invdz;
  ha.dt = c.dt;
  const dim3 nt = tiles(h->g, h->g.izStart, &ha.z_base, &ha.tile_rows);
  ha.early = early_trigger((long long)nt.x * nt.y);
  ha.x_base = NH;
  ha.undamped_ok = h->undamped_ok;
  ha.freesurface = c.freesurface;
  set_square(ha, h->exact);
  ha.wait_limit = h->wait_limit;
  ha.err = h->d_flag;
  ha.cols = h->d_cols;
  for (const float *q : {(const float *)a.f.vx, (const float *)a.f.vz, a.p.invrho}) ha.ahead[ha.nahead++] = q;
  if (c.variant == TTI_COORDINATE)
    for (const float *q : {a.p.snv, a.p.csv}) ha.ahead[ha.nahead++] = q;
  for (const float *q : {a.p.coef1, a.p.coef2}) ha.ahead[ha.nahead++] = q;
}

void velocity_maps(VelocityMaps &m, const void *maps)
{
  std::copy_n(static_cast<const CUtensorMap *>(maps) + 2, 3, m.box);
}
void stress_maps(StressMaps &m, const void *maps)
{
  const CUtensorMap *t = static_cast<const CUtensorMap *>(maps);
  std::copy_n(t, 2, m.box);
  std::copy_n(t + HALO_MAPS, IN_MAPS, m.in);
}

template <bool X, bool Q>
cudaError_t velocity_xq(const HalfArgs &a, const VelocityMaps &m, int variant, cudaStream_t st)
{
  const bool kept = a.kd[0], work = a.work_z1 > a.work_z0;
  const size_t smem = (size_t)(work ? V_END : V_BAR + 16) * sizeof(float);
  auto go = [&](auto kernel, auto with_work) {
    return work ? launch_k(with_work, a, m, smem, st) : launch_k(kernel, a, m, smem, st);
  };
  constexpr int C = TTI_COORDINATE, T = TTI_TENSOR, B = TTI_BOND;
  if (variant == C && kept) return go(k_velocity_tiled<C, X, Q, true>, k_velocity_tiled<C, X, Q, true, true>);
  if (variant == C) return go(k_velocity_tiled<C, X, Q>, k_velocity_tiled<C, X, Q, false, true>);
  if (variant == T) return go(k_velocity_tiled<T, X, Q>, k_velocity_tiled<T, X, Q, false, true>);
  return go(k_velocity_tiled<B, X, Q>, k_velocity_tiled<B, X, Q, false, true>);
}

template <int V, bool X, bool Q>
cudaError_t stress_vxq(const HalfArgs &a, const StressMaps &m, cudaStream_t st)
{
  constexpr size_t smem = (size_t)(s_bar(V) + 16) * sizeof(float);
  return a.kd[0] ? launch_k(k_stress_tiled<V, X, Q, true>, a, m, smem, st)
                 : launch_k(k_stress_tiled<V, X, Q>, a, m, smem, st);
}
template <bool X, bool Q>
cudaError_t stress_xq(const HalfArgs &a, const StressMaps &m, int variant, cudaStream_t st)
{
  if (variant == TTI_COORDINATE) return stress_vxq<TTI_COORDINATE, X, Q>(a, m, st);
  return variant == TTI_TENSOR ? stress_vxq<TTI_TENSOR, X, Q>(a, m, st) : stress_vxq<TTI_BOND, X, Q>(a, m, st);
}

cudaError_t launch_velocity(const HalfArgs &a, const void *maps, int variant, bool exact, cudaStream_t st)
{
  VelocityMaps m;
  velocity_maps(m, maps);
  if (exact) return velocity_xq<true, false>(a, m, variant, st);
  return a.square ? velocity_xq<false, true>(a, m, variant, st) : velocity_xq<false, false>(a, m, variant, st);
}

cudaError_t launch_stress(const HalfArgs &a, const void *maps, int variant, bool exact, cudaStream_t st)
{
  StressMaps m;
  stress_maps(m, maps);
  if (exact) return stress_xq<true, false>(a, m, variant, st);
  return a.square ? stress_xq<false, true>(a, m, variant, st) : stress_xq<false, false>(a, m, variant, st);
}

// shared memory of a batched kernel whose barrier is at float `bar`
constexpr size_t batch_smem(int bar) { return (size_t)(bar + 4) * sizeof(float) + sizeof(HalfArgs); }

// One CTA per work item.
template <typename K>
cudaError_t launch_batch_k(K kernel, size_t smem, const BatchLaunch &l, cudaStream_t st)
{
  const cudaError_t e = prepare_kernel(kernel, smem);
  if (e != cudaSuccess || l.nwork == 0) return e;
  const BatchArgs b{l.inst, l.maps, l.work, l.step, l.nwork, l.offset, -0.0f, l.wait_limit};
  return launch_pdl(kernel, dim3(l.nwork), dim3(walk::NT), smem, st, b);
}

template <bool X, bool Q>
cudaError_t velocity_batch_x(const BatchLaunch &l, cudaStream_t st)
{
  constexpr size_t smem = batch_smem(V_BAR);
  if (l.variant == TTI_COORDINATE) return launch_batch_k(k_velocity_batch<TTI_COORDINATE, X, Q>, smem, l, st);
  if (l.variant == TTI_TENSOR) return launch_batch_k(k_velocity_batch<TTI_TENSOR, X, Q>, smem, l, st);
  return launch_batch_k(k_velocity_batch<TTI_BOND, X, Q>, smem, l, st);
}

template <bool X, bool Q>
cudaError_t stress_batch_x(const BatchLaunch &l, cudaStream_t st)
{
  constexpr int C = TTI_COORDINATE, T = TTI_TENSOR, B = TTI_BOND;
  if (l.variant == C) return launch_batch_k(k_stress_batch<C, X, Q>, batch_smem(s_bar(C)), l, st);
  if (l.variant == T) return launch_batch_k(k_stress_batch<T, X, Q>, batch_smem(s_bar(T)), l, st);
  return launch_batch_k(k_stress_batch<B, X, Q>, batch_smem(s_bar(B)), l, st);
}

cudaError_t launch_velocity_batch(const BatchLaunch &l, cudaStream_t st)
{
  if (l.exact) return velocity_batch_x<true, false>(l, st);
  return l.square ? velocity_batch_x<false, true>(l, st) : velocity_batch_x<false, false>(l, st);
}

cudaError_t launch_stress_batch(const BatchLaunch &l, cudaStream_t st)
{
  if (l.exact) return stress_batch_x<true, false>(l, st);
  return l.square ? stress_batch_x<false, true>(l, st) : stress_batch_x<false, false>(l, st);
}

cudaError_t prepare_batch(BatchLaunch l)
{
  // a launch over zero CTAs only sets the attributes
  l.nwork = 0;
  cudaError_t e = launch_velocity_batch(l, nullptr);
  if (e == cudaSuccess) e = launch_stress_batch(l, nullptr);
  return e;
}

}  // namespace tiled
}  // namespace ttifd
