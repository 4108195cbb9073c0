// The diagonal walk: both diagonal sums of a halo box for every cell of a
// tile, from two shared-memory reads per box column and diagonal instead of
// ten per cell.
//
// The RSG stencil of a cell reads its field along the diagonal (x + m, z + m)
// (sum d1) and along the antidiagonal (d2), ten taps each. A thread walks one
// diagonal and one antidiagonal of the tile across its WX columns with the taps
// in registers: WX + 9 reads per sum and WX cells instead of 10 WX. It keeps
// (d1, d2) as one packed FP32 pair (sm_100 f32x2), so a stencil sum costs half
// the instructions of the scalar form. The sums go to shared memory skewed by
// their diagonal index, which makes every store a compile-time offset from the
// thread's own address (no bounds to test, no bank conflicts); after a barrier
// the cells' own threads read them back, four rows at a time.
#pragma once

#include "tiled.cuh"

namespace ttifd {
namespace walk {

constexpr int WX = 8;                        // tile columns: one warp each in the update
constexpr int WZ = 120;                      // most tile rows: four per lane in the update, four warps of diagonals
constexpr int WB = WZ + 16;                  // box rows (the box starts 8 rows above the tile)
static_assert((WB * 4) % 16 == 0, "TMA inner box extent must be a multiple of 16 bytes");
constexpr int WBX = WX + 9;                  // box columns
constexpr int DP = (WZ + WX + 2 + 3) / 4 * 4;  // column pitch of a sum array (see d1_row, d2_row)
constexpr int NT = 32 * WX;                  // threads per CTA
constexpr int BOX = (WBX * WB + 31) / 32 * 32;  // floats per box, 128-byte aligned
static_assert(BOX - WBX * WB >= 8, "walks of lanes below the tile read a few floats past the last box");
constexpr int LEAD = 32;                     // floats before the first box: a walk may start above it
constexpr int SUM = WX * DP;                 // floats per sum array
static_assert(SUM % 32 == 0, "sum arrays keep 128-byte alignment");
// Warps' worth of diagonals of a tile of `rows` rows.
__host__ __device__ __forceinline__ constexpr int groups(int rows) { return (rows + WX - 1 + 31) / 32; }

typedef unsigned long long u64;
__device__ __forceinline__ u64 pack2(float a, float b)
{
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(u64 v, float &a, float &b)
{
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c)
{
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b)
{
  u64 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b)
{
  u64 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Stencil coefficients as packed pairs held in registers (opaque to the
// compiler, which would otherwise rebuild each pair at every use).
struct Coefs {
  u64 c[5], nz;
};
// `nzero` is -0.0f at run time. An exact product is fma(c, d, -0.0): one
// rounding, signed zeros included. Written as a packed multiply, it would be
// fused with the packed add that follows into one rounding.
__device__ __forceinline__ Coefs coefs(float c0, float c1, float c2, float c3, float c4, float nzero)
{
  Coefs k;
  const float c[5] = {c0, c1, c2, c3, c4};
#pragma unroll
  for (int i = 0; i < 5; ++i) asm volatile("mov.b64 %0, {%1, %1};" : "=l"(k.c[i]) : "f"(c[i]));
  k.nz = pack2(nzero, nzero);
  return k;
}

// Place of a cell's sums in column c of a sum array: the diagonal index shifted
// so that rows 0, 4, 8, ... of every column fall on 16-byte boundaries.
__host__ __device__ __forceinline__ constexpr int d1_shift(int c) { return (c + 1) & 3; }
__host__ __device__ __forceinline__ constexpr int d2_shift(int c) { return -c & 3; }
// Offset of rows r .. r + 3 (r a multiple of 4) of column c
__device__ __forceinline__ int d1_at(int c, int r) { return c * DP + r + WX - 1 - c + d1_shift(c); }
__device__ __forceinline__ int d2_at(int c, int r) { return c * DP + r + c + d2_shift(c); }

// One thread's walk, diagonal index d: out[i] = (d1, d2), d1 of box `a` at cell
// (i, d - WX + 1 + i) and d2 of box `b` at cell (i, d - i), i < WX. O = 0:
// velocity-node stencil (box origin 4 columns left of the tile), O = 1:
// stress-node stencil (5 columns). EXACT rounds every product and sum
// separately in the reference's order; otherwise products are fused.
// Cells outside the tile's rows get sums nobody reads.
template <int O, bool EXACT>
__device__ __forceinline__ void diagonals(const float *a, const float *b, int d, const Coefs &k, u64 (&out)[WX])
{
  const float *pa = a + (d - WX + 5 - O), *pb = b + (d + 13 - O);
  u64 v[WBX];
#pragma unroll
  for (int c = 0; c < WBX; ++c) v[c] = pack2(pa[c * WB + c], pb[c * WB - c]);
#pragma unroll
  for (int i = 0; i < WX; ++i) {
    u64 s = fma2(k.c[0], sub2(v[i + 5], v[i + 4]), k.nz);
#pragma unroll
    for (int q = 2; q <= NH; ++q) {
      const u64 t = sub2(v[i + 4 + q], v[i + 5 - q]);
      s = EXACT ? add2(s, fma2(k.c[q - 1], t, k.nz)) : fma2(k.c[q - 1], t, s);
    }
    out[i] = s;
  }
}

// Stores a walk's sums into the sum arrays o1 (d1) and o2 (d2).
__device__ __forceinline__ void put_sums(float *o1, float *o2, int d, const u64 (&out)[WX])
{
#pragma unroll
  for (int i = 0; i < WX; ++i) {
    float s1, s2;
    unpack2(out[i], s1, s2);
    o1[i * DP + d + d1_shift(i)] = s1;
    o2[i * DP + d + d2_shift(i)] = s2;
  }
}

// Initialises a CTA's box barrier; one thread, before a __syncthreads that all
// threads reach ahead of their first wait.
__device__ __forceinline__ void init_bar(unsigned long long *bar)
{
  if (threadIdx.x == 0) {
    tiled::tma::mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}

// Issues the TMA copies of a tile: nb halo boxes (origin row z0 - 8, column x0 -
// xoff), then ni inputs of the tile's own cells (rows x WX) at `in_off`. One
// thread works, after every thread is done with what these replace. They
// complete the barrier's next phase.
__device__ __forceinline__ void issue_tile(const CUtensorMap *map, int nb, int xoff, const CUtensorMap *in, int ni,
                                           int rows, float *sm, int in_off, unsigned long long *bar, int z0, int x0)
{
  if (threadIdx.x != 0) return;
  tiled::tma::mbar_arrive_expect_tx(bar, (nb * WBX * WB + ni * rows * WX) * 4);
  for (int f = 0; f < nb; ++f) tiled::tma::tma_load_2d(sm + LEAD + f * BOX, map + f, z0 - 8, x0 - xoff, bar);
  for (int k = 0; k < ni; ++k) tiled::tma::tma_load_2d(sm + in_off + k * rows * WX, in + k, z0, x0, bar);
}

// Waits for the boxes: one warp polls, the others wait at the block barrier
// (where they take no issue slots). Returns false (all threads) after a
// timed-out wait.
__device__ __forceinline__ bool wait_boxes(int *err, unsigned long long *bar, unsigned limit, unsigned parity)
{
  const bool ok = threadIdx.x >= 32 || tiled::tma::mbar_wait(bar, parity, limit);
  if (__syncthreads_or(!ok)) {
    if (threadIdx.x == 0) {
      atomicOr(err, 4);
      tiled::tma::mbar_wait(bar, parity, 1u << 16);  // give the copies in flight a bounded time
    }
    return false;
  }
  tiled::tma::mbar_wait(bar, parity, 1);  // this thread's own view of the completed phase
  return true;
}

// One warp's L2 prefetch of a tile's rows of an array: lanes take four 128-byte
// lines of each of the WX columns. (A tile of 120 rows that begins 16 or 24 rows
// into a line reaches into a fifth, which is left to the loads.)
__device__ __forceinline__ void prefetch_lines(const float *base, const Grid &g, int x0, int z0, int rows)
{
  static_assert(WX == 8 && WZ <= 128, "four lines of eight columns");
  const int lane = threadIdx.x & 31, x = x0 + (lane >> 2), z = z0 + (lane & 3) * 32;
  if (x < g.Nx && z < min(g.ldz, z0 + rows))
    asm volatile("prefetch.global.L2 [%0];" ::"l"(base + (size_t)x * g.ldz + z));
}

// four consecutive rows of an array, as two packed pairs
struct F4 {
  u64 p[2];
};
__device__ __forceinline__ F4 ld4(const float *p)
{
  const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(p);
  return F4{{q.x, q.y}};
}
__device__ __forceinline__ F4 ldg4(const float *p)
{
  const ulonglong2 q = __ldg(reinterpret_cast<const ulonglong2 *>(p));
  return F4{{q.x, q.y}};
}
// stores rows z .. z + 3, those in [lo, hi) only
__device__ __forceinline__ void st4(float *p, const F4 &f, int z, int lo, int hi)
{
  if (z >= lo && z + 3 < hi) {
    *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(f.p[0], f.p[1]);
  } else {
    float v[4];
    unpack2(f.p[0], v[0], v[1]);
    unpack2(f.p[1], v[2], v[3]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (z + i >= lo && z + i < hi) p[i] = v[i];
  }
}

// Arithmetic of the update on a thread's four rows, N values of type T each.
// Exact: packed pairs, every product and sum rounded separately (a product is
// fma(a, b, -0.0), see Coefs), half the instructions of the scalar form.
// Otherwise scalar, so that the compiler may contract products into FMA.
template <bool EXACT>
struct Rows;
template <>
struct Rows<true> {
  typedef u64 T;
  static constexpr int N = 2;
  u64 nz;
  __device__ __forceinline__ T c(float a) const { return pack2(a, a); }
  __device__ __forceinline__ T mul(T a, T b) const { return fma2(a, b, nz); }
  __device__ __forceinline__ T add(T a, T b) const { return add2(a, b); }
  __device__ __forceinline__ T sub(T a, T b) const { return sub2(a, b); }
  static __device__ __forceinline__ T get(const F4 &f, int i) { return f.p[i]; }
  static __device__ __forceinline__ void set(F4 &f, int i, T v) { f.p[i] = v; }
};
template <>
struct Rows<false> {
  typedef float T;
  static constexpr int N = 4;
  u64 nz;
  __device__ __forceinline__ T c(float a) const { return a; }
  __device__ __forceinline__ T mul(T a, T b) const { return a * b; }
  __device__ __forceinline__ T add(T a, T b) const { return a + b; }
  __device__ __forceinline__ T sub(T a, T b) const { return a - b; }
  static __device__ __forceinline__ T get(const F4 &f, int i)
  {
    float a, b;
    unpack2(f.p[i >> 1], a, b);
    return i & 1 ? b : a;
  }
  static __device__ __forceinline__ void set(F4 &f, int i, T v)
  {
    float a, b;
    unpack2(f.p[i >> 1], a, b);
    f.p[i >> 1] = i & 1 ? pack2(a, v) : pack2(v, b);
  }
};

}  // namespace walk
}  // namespace ttifd
