// The column work of a time step: what happens to single padded-grid columns
// after each half-step. After the velocity update the velocity sources (stype
// 2-8, coord:674-802); after the stress update the free-surface image
// (coord:847-863), the stress source (stype 1, coord:865-886, tensor:871-895)
// and the receiver samples (isoelastic.c:103-144). Columns do not interact, so
// one warp does a column, in the reference's order: the single-shot tiled
// kernels in the tiles it falls in (after the stress update arranged as in
// tiled_step.cu), k_post and k_sources as launches of their own (batched shots,
// and columns outside the tiles).
#pragma once

#include "launch.cuh"

namespace ttifd {

__device__ __forceinline__ void acc(float *p, float k, float a) { *p = __fadd_rn(*p, __fmul_rn(k, a)); }
__device__ __forceinline__ void dec(float *p, float k, float a) { *p = __fsub_rn(*p, __fmul_rn(k, a)); }

// time index of step n, and its receiver sample (-1: none)
__device__ __forceinline__ int time_index(const Columns &p, int n) { return p.mode2 ? p.nt - 1 - n : n; }
__device__ __forceinline__ int record_index(const Columns &p, int it)
{
  return p.rec_on && it % p.mt == 0 ? it / p.mt : -1;
}

// whether column ix may have sources
__device__ __forceinline__ bool source_column(const Columns &p, int ix) { return ix >= p.sx0 && ix < p.sx1; }

// Such a column's sources at time index it.
struct ColumnSources {
  const Columns &p;
  int it, first, last;
  __device__ __forceinline__ ColumnSources(const Columns &q, int ix, int t)
      : p(q), it(t), first(q.scol[ix - q.sx0]), last(q.scol[ix - q.sx0 + 1])
  {
  }
  __device__ __forceinline__ int4 at(int j) const { return __ldg(p.sat + j); }
  __device__ __forceinline__ float amp(const int4 &s) const { return __ldg(p.amp + (size_t)s.x * p.nt + it); }
};

// Rows [r0, r1) of column ix after the stress update, one warp (all lanes).
// With `pdl` the column's receiver geometry (static since the receivers were
// set) is read before waiting for the previous kernel, so those loads overlap
// its tail.
__device__ __forceinline__ void column_post(const Grid &g, const Fields &f, const Columns &p, int ix, int n, int r0,
                                            int r1, bool pdl = false)
{
  const int lane = threadIdx.x & 31, it = time_index(p, n), irec = record_index(p, it);
  const size_t col = (size_t)ix * g.ldz;
  // the first 32 receivers of each component in this column, one per lane
  int rb[3] = {0, 0, 0}, re[3] = {0, 0, 0}, rzl[3] = {-1, -1, -1}, ridl[3] = {0, 0, 0};
  if (irec >= 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (p.colptr[k]) {
        rb[k] = p.colptr[k][ix];
        re[k] = p.colptr[k][ix + 1];
      }
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (rb[k] + lane < re[k]) {
        rzl[k] = p.rz[k][rb[k] + lane];
        ridl[k] = p.rid[k][rb[k] + lane];
      }
  }
  if (pdl) pdl_sync();
  if (p.freesurface && ix >= NH && ix < g.Nx - NH && g.izStart >= r0 && g.izStart < r1) {
    // lane k mirrors row izStart + k; the rows must be in [r0, r1)
    const size_t c = col + g.izStart;
    const float sxx0 = f.sxx[c];
    float xx = 0.0f, zz = 0.0f, xz = 0.0f;
    if (lane >= 1 && lane <= NH) {
      xx = f.sxx[c + lane];
      zz = f.szz[c + lane];
      xz = f.sxz[c + lane];
    }
    __syncwarp();
    if (lane >= 1 && lane <= NH) {
      f.sxx[c - lane] = __fsub_rn(__fmul_rn(2.0f, sxx0), xx);
      f.szz[c - lane] = -zz;
      f.sxz[c - lane] = -xz;
    } else if (lane == 0) {
      f.sxz[c] = 0.0f;
      f.szz[c] = 0.0f;
    }
    __syncwarp();
  }
  if (p.stype == 1 && source_column(p, ix)) {
    const ColumnSources src(p, ix, it);

#pragma unroll 1
    for (int j = src.first; j < src.last; ++j) {
      const int4 s = src.at(j);
      const int iz = s.y + lane - NH;
      if (lane <= 2 * NH && iz >= 0 && iz < g.Nz && iz >= r0 && iz < r1) {
        const float ws = __fmul_rn(__ldg(p.t.k1 + (s.z + NH) * 11 + lane), src.amp(s));
        const size_t c = col + iz;
        f.sxx[c] = __fadd_rn(f.sxx[c], ws);
        f.szz[c] = __fadd_rn(f.szz[c], ws);
        if (p.tensor) {
          f.txx[c] = __fadd_rn(f.txx[c], ws);
          f.tzz[c] = __fadd_rn(f.tzz[c], ws);
        }
      }
      __syncwarp();
    }
  }
  if (irec >= 0) {
    auto sample = [&](int k, int rz) {
      const size_t c = col + rz;
      return k == TTI_REC_VX ? f.vx[c] : k == TTI_REC_VZ ? f.vz[c] : __fmul_rn(0.5f, __fadd_rn(f.sxx[c], f.szz[c]));
    };
    // all three components' samples loaded before any is stored
    float v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = rzl[k] >= r0 && rzl[k] < r1 ? sample(k, rzl[k]) : 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (rzl[k] >= r0 && rzl[k] < r1) {
        p.rec[k][(size_t)irec * p.nrec[k] + ridl[k]] = v[k];
        if (!isfinite(v[k])) atomicOr(p.flag, 1);
      }
    // columns with more than 32 receivers of a component
    for (int k = 0; k < 3; ++k)
      for (int j = rb[k] + 32 + lane; j < re[k]; j += 32) {
        const int rz = p.rz[k][j];
        if (rz < r0 || rz >= r1) continue;
        const float w = sample(k, rz);
        p.rec[k][(size_t)irec * p.nrec[k] + p.rid[k][j]] = w;
        if (!isfinite(w)) atomicOr(p.flag, 1);
      }
  }
}

// The velocity sources on rows [r0, r1) of column ix after the velocity
// update, one warp: lanes over the window's rows, the sources one after
// another, so that overlapping windows accumulate in the reference's order.
__device__ __forceinline__ void column_sources(const Grid &g, const Fields &f, const Columns &p, int ix, int n, int r0,
                                               int r1)
{
  const int lane = threadIdx.x & 31, it = time_index(p, n);
  const size_t col = (size_t)ix * g.ldz;
  if (!source_column(p, ix)) return;
  const ColumnSources src(p, ix, it);
  if (p.stype == 8) {  // coord:782-801: four cells, one lane
    const float k = p.t.q8;
    for (int j = src.first; j < src.last && lane == 0; ++j) {
      const int4 s = src.at(j);
      const int dx = s.z, z = s.y;
      if (dx != 0 && dx != -1) continue;
      const float a = src.amp(s);
      if (z >= r0 && z < r1) {
        dec(f.vx + col + z, k, a);
        if (dx == 0) acc(f.vz + col + z, k, a);
        else dec(f.vz + col + z, k, a);
      }
      if (z - 1 >= r0 && z - 1 < r1) {
        acc(f.vx + col + z - 1, k, a);
        if (dx == 0) acc(f.vz + col + z - 1, k, a);
        else dec(f.vz + col + z - 1, k, a);
      }
    }
    return;
  }
  const int first = p.stype == 4 ? 2 : p.stype, last = p.stype == 4 ? 3 : p.stype;  // stype 4: 2, then 3
  for (int kind = first; kind <= last; ++kind)
#pragma unroll 1
    for (int j = src.first; j < src.last; ++j) {
      const int4 s = src.at(j);
      const int iz = s.y + lane - NH, w = (s.z + NH) * 11 + lane;
      if (lane <= 2 * NH && iz >= 0 && iz < g.Nz && iz >= r0 && iz < r1) {
        const float a = src.amp(s);
        float *vx = f.vx + col + iz, *vz = f.vz + col + iz;
        if (kind == 2) {
          acc(vx, __ldg(p.t.kx + w), a);
          acc(vz, __ldg(p.t.kz + w), a);
        } else if (kind == 3) {
          dec(vx, __ldg(p.t.kz + w), a);
          acc(vz, __ldg(p.t.kx + w), a);
        } else if (kind == 5) {
          acc(vx, __ldg(p.t.k5 + w), a);
        } else if (kind == 6) {
          acc(vz, __ldg(p.t.k5 + w), a);
        } else {
          acc(vx, __ldg(p.t.k7 + w), a);
          acc(vz, __ldg(p.t.k7 + w), a);
        }
      }
      __syncwarp();
    }
}

}  // namespace ttifd
