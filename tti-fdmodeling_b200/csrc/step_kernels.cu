// Per-step kernels of the RSG time loop: velocity and stress updates along
// the two grid diagonals, the column work, energy, snapshot packing.
#include <algorithm>

#include "columns.cuh"

namespace ttifd {

namespace {

// Velocity node (ix+1/2, iz+1/2) from a stress field, coord:621-630:
//   d1 = sum_k C_k (a[x+k][z+k]   - a[x-k+1][z-k+1])
//   d2 = sum_k C_k (a[x+k][z-k+1] - a[x-k+1][z+k])
template <bool X>
__device__ __forceinline__ void diag_v(const float *__restrict__ q, int L, float &d1, float &d2)
{
  using A = Ar<X>;
  float s1 = A::mul(rsg(0), A::sub(__ldg(q + L + 1), __ldg(q)));
  float s2 = A::mul(rsg(0), A::sub(__ldg(q + L), __ldg(q + 1)));
#pragma unroll
  for (int k = 2; k <= NH; ++k) {
    s1 = A::add(s1, A::mul(rsg(k - 1), A::sub(__ldg(q + k * (L + 1)), __ldg(q - (k - 1) * (L + 1)))));
    s2 = A::add(s2, A::mul(rsg(k - 1), A::sub(__ldg(q + k * L - (k - 1)), __ldg(q - (k - 1) * L + k))));
  }
  d1 = s1;
  d2 = s2;
}

// Stress node (ix, iz) from a velocity field, coord:811-816:
//   d1 = sum_k C_k (a[x+k-1][z+k-1] - a[x-k][z-k])
//   d2 = sum_k C_k (a[x+k-1][z-k]   - a[x-k][z+k-1])
template <bool X>
__device__ __forceinline__ void diag_s(const float *__restrict__ q, int L, float &d1, float &d2)
{
  using A = Ar<X>;
  float s1 = A::mul(rsg(0), A::sub(__ldg(q), __ldg(q - L - 1)));
  float s2 = A::mul(rsg(0), A::sub(__ldg(q - 1), __ldg(q - L)));
#pragma unroll
  for (int k = 2; k <= NH; ++k) {
    s1 = A::add(s1, A::mul(rsg(k - 1), A::sub(__ldg(q + (k - 1) * (L + 1)), __ldg(q - k * (L + 1)))));
    s2 = A::add(s2, A::mul(rsg(k - 1), A::sub(__ldg(q + (k - 1) * L - k), __ldg(q - k * L + (k - 1)))));
  }
  d1 = s1;
  d2 = s2;
}

constexpr int BZ = 32, BX = 8;

// coord:614-672, tensor:617-666, bond:654-703
template <int V, bool X>
__global__ void __launch_bounds__(BZ *BX) k_velocity(Grid g, Fields f, Params p, float invdx, float invdz)
{
  using A = Ar<X>;
  const int iz = g.izStart + blockIdx.x * BZ + threadIdx.x;
  const int ix = NH + blockIdx.y * BX + threadIdx.y;
  if (iz >= g.Nz - NH || ix >= g.Nx - NH) return;
  const int L = g.ldz;
  const size_t i = (size_t)ix * L + iz;
  float d1, d2;
  diag_v<X>(f.sxx + i, L, d1, d2);
  const float sxx_x = A::mul(A::mul(0.5f, A::add(d1, d2)), invdx);
  const float sxx_z = A::mul(A::mul(0.5f, A::sub(d1, d2)), invdx);  // invdx as in coord:633
  diag_v<X>(f.szz + i, L, d1, d2);
  const float szz_x = A::mul(A::mul(0.5f, A::add(d1, d2)), invdx);
  const float szz_z = A::mul(A::mul(0.5f, A::sub(d1, d2)), invdz);
  diag_v<X>(f.sxz + i, L, d1, d2);
  const float sxz_x = A::mul(A::mul(0.5f, A::add(d1, d2)), invdx);
  const float sxz_z = A::mul(A::mul(0.5f, A::sub(d1, d2)), invdz);
  const float a = p.coef1[i], br = A::mul(p.coef2[i], p.invrho[i]);
  float fx, fz;
  if (V == TTI_COORDINATE) {
    const float cv = p.csv[i], sv = p.snv[i];
    fx = A::add(A::add(A::sub(A::mul(cv, sxx_x), A::mul(sv, sxx_z)), A::mul(sv, sxz_x)), A::mul(cv, sxz_z));
    fz = A::add(A::add(A::sub(A::mul(cv, sxz_x), A::mul(sv, sxz_z)), A::mul(sv, szz_x)), A::mul(cv, szz_z));
  } else {
    fx = A::add(sxx_x, sxz_z);
    fz = A::add(sxz_x, szz_z);
  }
  f.vx[i] = A::add(A::mul(a, f.vx[i]), A::mul(br, fx));
  f.vz[i] = A::add(A::mul(a, f.vz[i]), A::mul(br, fz));
}

// coord:804-845, tensor:799-851 (tau update and sigma = R tau fused: the
// sigma pass reads only the same cell's tau), bond:836-873
template <int V, bool X>
__global__ void __launch_bounds__(BZ *BX) k_stress(Grid g, Fields f, Params p, float invdx, float invdz)
{
  using A = Ar<X>;
  const int iz = g.izStart + blockIdx.x * BZ + threadIdx.x;
  const int ix = NH + blockIdx.y * BX + threadIdx.y;
  if (iz >= g.Nz - NH || ix >= g.Nx - NH) return;
  const int L = g.ldz;
  const size_t i = (size_t)ix * L + iz;
  float d1, d2;
  diag_s<X>(f.vx + i, L, d1, d2);
  float vxx = A::mul(A::mul(0.5f, A::add(d1, d2)), invdx);
  float vxz = A::mul(A::mul(0.5f, A::sub(d1, d2)), invdz);
  diag_s<X>(f.vz + i, L, d1, d2);
  float vzx = A::mul(A::mul(0.5f, A::add(d1, d2)), invdx);
  float vzz = A::mul(A::mul(0.5f, A::sub(d1, d2)), invdz);
  const float a = p.coef1[i], b = p.coef2[i];
  const float c11 = p.c11[i], c13 = p.c13[i], c33 = p.c33[i], c55 = p.c55[i];
  if (V == TTI_COORDINATE) {
    const float s = p.sn[i], c = p.cs[i];
    float r = A::add(A::mul(s, vxx), A::mul(c, vxz));
    vxx = A::sub(A::mul(c, vxx), A::mul(s, vxz));
    vxz = r;
    r = A::add(A::mul(s, vzx), A::mul(c, vzz));
    vzx = A::sub(A::mul(c, vzx), A::mul(s, vzz));
    vzz = r;
    f.sxx[i] = A::add(A::mul(a, f.sxx[i]), A::mul(b, A::add(A::mul(c11, vxx), A::mul(c13, vzz))));
    f.szz[i] = A::add(A::mul(a, f.szz[i]), A::mul(b, A::add(A::mul(c13, vxx), A::mul(c33, vzz))));
    f.sxz[i] = A::add(A::mul(a, f.sxz[i]), A::mul(A::mul(b, c55), A::add(vzx, vxz)));
  } else if (V == TTI_TENSOR) {
    const float s2 = p.s2[i], c2 = p.c2[i], st = p.s2t[i];
    const float sh = A::add(vxz, vzx);
    const float exx = A::sub(A::add(A::mul(c2, vxx), A::mul(s2, vzz)), A::mul(A::mul(0.5f, st), sh));
    const float ezz = A::add(A::add(A::mul(s2, vxx), A::mul(c2, vzz)), A::mul(A::mul(0.5f, st), sh));
    const float exz = A::add(A::mul(st, A::sub(vxx, vzz)), A::mul(A::sub(c2, s2), sh));
    const float txx = A::add(A::mul(a, f.txx[i]), A::mul(b, A::add(A::mul(c11, exx), A::mul(c13, ezz))));
    const float tzz = A::add(A::mul(a, f.tzz[i]), A::mul(b, A::add(A::mul(c13, exx), A::mul(c33, ezz))));
    const float txz = A::add(A::mul(a, f.txz[i]), A::mul(A::mul(b, c55), exz));
    f.txx[i] = txx;
    f.tzz[i] = tzz;
    f.txz[i] = txz;
    f.sxx[i] = A::add(A::add(A::mul(c2, txx), A::mul(s2, tzz)), A::mul(st, txz));
    f.szz[i] = A::sub(A::add(A::mul(s2, txx), A::mul(c2, tzz)), A::mul(st, txz));
    f.sxz[i] = A::add(A::mul(A::mul(-0.5f, st), A::sub(txx, tzz)), A::mul(A::sub(c2, s2), txz));
  } else {
    const float c15 = p.c15[i], c35 = p.c35[i];
    const float sh = A::add(vzx, vxz);
    f.sxx[i] = A::add(A::mul(a, f.sxx[i]),
                      A::mul(b, A::add(A::add(A::mul(c11, vxx), A::mul(c13, vzz)), A::mul(c15, sh))));
    f.szz[i] = A::add(A::mul(a, f.szz[i]),
                      A::mul(b, A::add(A::add(A::mul(c13, vxx), A::mul(c33, vzz)), A::mul(c35, sh))));
    f.sxz[i] = A::add(A::mul(a, f.sxz[i]),
                      A::mul(b, A::add(A::add(A::mul(c15, vxx), A::mul(c35, vzz)), A::mul(c55, sh))));
  }
}

__global__ void k_advance(int *step, int n)
{
  pdl_sync();
  *step += n;
}

// coord:898-924, accumulated in double per step
__global__ void k_energy(Grid g, Fields f, Params p, int nz, int nx, double *out2)
{
  double ek = 0.0, ep = 0.0;
  const size_t n = (size_t)nz * nx;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
    const int ix = (int)(q / nz) + g.E, iz = (int)(q % nz) + g.E;
    const size_t i = (size_t)ix * g.ldz + iz;
    const float r = p.invrho[i], c11 = p.c11[i], c55 = p.c55[i];
    const float vx = f.vx[i], vz = f.vz[i], sx = f.sxx[i], sz = f.szz[i], sq = f.sxz[i];
    ek += (double)(__fdiv_rn(__fmul_rn(vx, vx), r) + __fdiv_rn(__fmul_rn(vz, vz), r));
    const float c1 = __fadd_rn(c11, __fmul_rn(2.0f, c55));
    const float num = __fadd_rn(__fmul_rn(__fsub_rn(__fmul_rn(c1, sx), __fmul_rn(c11, sz)), sx),
                                __fmul_rn(__fsub_rn(__fmul_rn(c11, sx), __fmul_rn(c1, sz)), sz));
    ep += (double)(__fdiv_rn(__fmul_rn(0.25f, num), __fmul_rn(c55, __fadd_rn(c11, c55))) +
                   __fdiv_rn(__fmul_rn(sq, sq), c55));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ek += __shfl_down_sync(0xffffffffu, ek, o);
    ep += __shfl_down_sync(0xffffffffu, ep, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(out2, ek);
    atomicAdd(out2 + 1, ep);
  }
}

__device__ __forceinline__ int warp_column(const ColumnShot &s)
{
  return s.x0 + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
}

__global__ void k_post(ColumnShot s, int n)
{
  const int ix = warp_column(s);
  if (ix < s.x1) column_post(s.g, s.f, *s.c, ix, n, 0, s.g.Nz, true);
  else pdl_sync();
}
__global__ void k_sources(ColumnShot s, int n)
{
  pdl_sync();
  const int ix = warp_column(s);
  if (ix < s.x1) column_sources(s.g, s.f, *s.c, ix, n, 0, s.g.Nz);
}
// Batched: blockIdx.y = shot.
__global__ void k_post_batch(const ColumnShot *d, const int *step, int n)
{
  const ColumnShot &s = d[blockIdx.y];
  pdl_sync();
  const int k = *step + n, ix = warp_column(s);
  if (k < s.c->nt && ix < s.x1) column_post(s.g, s.f, *s.c, ix, k, 0, s.g.Nz);
}
__global__ void k_sources_batch(const ColumnShot *d, const int *step, int n)
{
  const ColumnShot &s = d[blockIdx.y];
  pdl_sync();
  const int k = *step + n, ix = warp_column(s);
  if (k < s.c->nt && ix < s.x1) column_sources(s.g, s.f, *s.c, ix, k, 0, s.g.Nz);
}

__global__ void k_snapshot(Grid g, Fields f, int kind, int x0, int z0, int nzo, int nxo, float *dst)
{
  const int iz = blockIdx.x * blockDim.x + threadIdx.x;
  const int ix = blockIdx.y;
  if (iz >= nzo || ix >= nxo) return;
  const size_t c = (size_t)(ix + x0) * g.ldz + (iz + z0);
  float v;
  if (kind == 3) v = __fmul_rn(0.5f, __fadd_rn(f.sxx[c], f.szz[c]));
  else if (kind == 1 || kind == 4 || kind == 6) v = f.vx[c];
  else v = f.vz[c];
  dst[(size_t)ix * nzo + iz] = v;
}

}  // namespace

static dim3 interior_grid(const Grid &g)
{
  const int nz = g.Nz - NH - g.izStart, nx = g.Nx - 2 * NH;
  return dim3((nz + BZ - 1) / BZ, (nx + BX - 1) / BX);
}

#define TTI_DISPATCH(KERNEL, a, st)                                                                        \
  do {                                                                                                     \
    const dim3 grd = interior_grid(a.g), blk(BZ, BX);                                                       \
    if (grd.x == 0 || grd.y == 0) break;                                                                   \
    if (a.exact) {                                                                                         \
      if (a.variant == TTI_COORDINATE) KERNEL<TTI_COORDINATE, true><<<grd, blk, 0, st>>>(a.g, a.f, a.p, a.invdx, a.invdz); \
      else if (a.variant == TTI_TENSOR) KERNEL<TTI_TENSOR, true><<<grd, blk, 0, st>>>(a.g, a.f, a.p, a.invdx, a.invdz); \
      else KERNEL<TTI_BOND, true><<<grd, blk, 0, st>>>(a.g, a.f, a.p, a.invdx, a.invdz);                     \
    } else {                                                                                               \
      if (a.variant == TTI_COORDINATE) KERNEL<TTI_COORDINATE, false><<<grd, blk, 0, st>>>(a.g, a.f, a.p, a.invdx, a.invdz); \
      else if (a.variant == TTI_TENSOR) KERNEL<TTI_TENSOR, false><<<grd, blk, 0, st>>>(a.g, a.f, a.p, a.invdx, a.invdz); \
      else KERNEL<TTI_BOND, false><<<grd, blk, 0, st>>>(a.g, a.f, a.p, a.invdx, a.invdz);                    \
    }                                                                                                      \
  } while (0)

void launch_velocity(const StepArgs &a, cudaStream_t st) { TTI_DISPATCH(k_velocity, a, st); }
void launch_stress(const StepArgs &a, cudaStream_t st) { TTI_DISPATCH(k_stress, a, st); }

void launch_energy(const StepArgs &a, int nz, int nx, double *out2, cudaStream_t st)
{
  k_energy<<<296, 256, 0, st>>>(a.g, a.f, a.p, nz, nx, out2);
}

cudaError_t launch_post(const ColumnShot &s, int n, cudaStream_t st)
{
  return launch_pdl(k_post, dim3((s.x1 - s.x0 + 3) / 4), dim3(128), 0, st, s, n);  // 4 columns (warps) per block
}
cudaError_t launch_sources(const ColumnShot &s, int n, cudaStream_t st)
{
  return launch_pdl(k_sources, dim3((s.x1 - s.x0 + 3) / 4), dim3(128), 0, st, s, n);
}
cudaError_t launch_post_batch(const ColumnShot *d, int ns, int cols, const int *step, int n, cudaStream_t st)
{
  return launch_pdl(k_post_batch, dim3((cols + 3) / 4, ns), dim3(128), 0, st, d, step, n);
}
cudaError_t launch_sources_batch(const ColumnShot *d, int ns, int cols, const int *step, int n, cudaStream_t st)
{
  return launch_pdl(k_sources_batch, dim3((cols + 3) / 4, ns), dim3(128), 0, st, d, step, n);
}

// up to five state arrays copied in one launch (the gradient's kept states)
struct Copy5 {
  const float4 *src[5];
  float4 *dst[5];
  int nf;
};
__global__ void k_copy5(Copy5 c, size_t n4)
{
  pdl_sync();
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n4; q += (size_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int f = 0; f < 5; ++f)
      if (f < c.nf) c.dst[f][q] = c.src[f][q];
  }
}

void launch_copy5(float *const *src, float *const *dst, int nf, size_t n, cudaStream_t st)
{
  Copy5 c;
  c.nf = std::min(nf, 5);
  for (int f = 0; f < 5; ++f) {
    c.src[f] = f < c.nf ? reinterpret_cast<const float4 *>(src[f]) : nullptr;
    c.dst[f] = f < c.nf ? reinterpret_cast<float4 *>(dst[f]) : nullptr;
  }
  const size_t n4 = n / 4;
  launch_pdl(k_copy5, dim3((unsigned)std::min<size_t>((n4 + 255) / 256, 148 * 16)), dim3(256), 0, st, c, n4);
}

// Receivers r0 .. r0 + nr - 1 of the time-major [nts][n] block, transposed to
// [nr][nts] (the Receiver2D.recv layout), through 32 x 32 shared tiles.
__global__ void k_transpose(const float *in, float *out, int nts, int n, int r0, int nr)
{
  __shared__ float t[32][33];
  const int ra = blockIdx.x * 32, t0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int tt = t0 + k, r = ra + threadIdx.x;
    if (tt < nts && r < nr) t[k][threadIdx.x] = in[(size_t)tt * n + r0 + r];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int r = ra + k, tt = t0 + threadIdx.x;
    if (tt < nts && r < nr) out[(size_t)r * nts + tt] = t[threadIdx.x][k];
  }
}

void launch_transpose(const float *in, float *out, int nts, int n, int r0, int nr, cudaStream_t st)
{
  k_transpose<<<dim3((nr + 31) / 32, (nts + 31) / 32), dim3(32, 8), 0, st>>>(in, out, nts, n, r0, nr);
}

cudaError_t launch_advance(int *step, int n, cudaStream_t st)
{
  return launch_pdl(k_advance, dim3(1), dim3(1), 0, st, step, n);
}

void launch_snapshot(const StepArgs &a, int kind, int savew, float *dst, cudaStream_t st)
{
  const Grid &g = a.g;
  const int x0 = savew == 0 ? g.E : 0, z0 = savew == 0 ? g.E : 0;
  const int nxo = savew == 0 ? g.Nx - 2 * g.E : g.Nx, nzo = savew == 0 ? g.Nz - 2 * g.E : g.Nz;
  k_snapshot<<<dim3((nzo + 127) / 128, nxo), 128, 0, st>>>(g, a.f, kind, x0, z0, nzo, nxo, dst);
}

}  // namespace ttifd
