// Tiled half-step kernels (tiled_step.cu): velocity and stress updates in
// place, each CTA loading its halo tile with TMA copies.
#pragma once

#include <cuda.h>

#include "launch.cuh"

namespace ttifd {
namespace tiled {

// A handle's tensor maps: the halo boxes of vx vz sxx szz sxz, then the tile
// inputs of the stress update: coordinate sxx szz sxz sin cos c11 c13 c33 c55;
// tensor txx tzz txz sin^2 cos^2 c11 c13 c33 c55 sin2theta; Bond sxx szz sxz
// c15 c35 c11 c13 c33 c55.
constexpr int HALO_MAPS = 5, IN_MAPS = 10, MAPS = HALO_MAPS + IN_MAPS;
struct alignas(64) VelocityMaps {
  CUtensorMap box[3];  // sxx szz sxz
};
struct alignas(64) StressMaps {
  CUtensorMap box[2];  // vx vz
  CUtensorMap in[IN_MAPS];
};
constexpr int AHEAD = 7;  // entries of HalfArgs::ahead

struct alignas(16) HalfArgs {
  Grid g;
  Fields f;
  Params p;
  float invdx, invdz, dt;
  int z_base;  // first tile row (multiple of 4, <= izStart)
  int x_base;  // first tile column (= 5)
  int tile_rows;  // rows of a tile (multiple of 8, at most walk::WZ)
  int undamped_ok;
  int freesurface;
  int *err;    // bit 4: a TMA wait timed out
  int square;  // FMA mode with dx == dz: stencil coefficients hc fold in h = 0.5 / dx
  unsigned wait_limit;  // polls of the first TMA wait before it gives up (tma::WAIT_LIMIT)
  float hc[5]; // h * C_k
  float nzero; // -0.0f (see walk::coefs)
  int early;   // trigger the next kernel at the start (early_trigger)
  // Gradient forward pass (null: nothing kept). Velocity update, coordinate
  // rotation: per cell the stress derivative combinations the adjoint's
  // theta_v terms need (sxz_x - sxx_z, szz_x - sxz_z, sxx_x + sxz_z,
  // sxz_x + szz_z). Stress update: the strain rates vxx vxz vzx vzz (not
  // rotated), and for the tensor rotation the tau it starts from (kt). Pointers
  // to the first slot.
  float *kd[4];
  float *kt[3];
  // the arrays the velocity update reads per cell, for the L2 prefetch: vx vz
  // invrho, coordinate also sin cos of theta_v, coef1, coef2
  const float *ahead[AHEAD];
  int nahead;
  // Column work in the tiles: rows [work_z0, work_z1) have some (none: empty).
  // After the velocity update the velocity sources, after the stress update the
  // rest (columns.cuh), of step n (batched launches: from the step counter).
  const Columns *cols;
  int work_z0, work_z1;
  // The step: n, or inside a graph clk[0] + n (StepClock). The gradient's kept
  // steps: the slot of step k0 (graph: clk[1]) is kd and kt, the next ones
  // kstride floats apart.
  const int *clk;
  int n, k0;
  size_t kstride;
};

// A handle's device step counters for graphs of several steps: the step, and
// the first step of the kept segment.
struct StepClock {
  int n, k0;
};

// Sets square / hc for FMA-mode launches on grids with dx == dz.
inline void set_square(HalfArgs &a, bool exact)
{
  a.square = !exact && a.invdx == a.invdz;
  for (int k = 0; k < 5; ++k) a.hc[k] = 0.5f * a.invdx * rsg(k);
  a.nzero = -0.0f;
}

// Encodes a handle's MAPS tensor maps.
bool encode_maps(CUtensorMap *map, const Grid &g, int variant, const Fields &f, const Params &p);
// Whether a single shot's half-step launch of so many tiles triggers its
// dependent as soon as it has waited for its own predecessor: only where the
// CTAs of two launches fit the device together (4 a SM on 148 SMs, as the plain
// half-steps run; the stress kernel that keeps fields for the gradient runs 3, so
// of 223 to 296 tiles two of its launches do not quite fit). The next launch's
// CTAs then wait in free slots. Where they do not fit, the part that finds a slot
// is spread unevenly, so the trigger comes when a tile's sums are complete. us a
// step early / late: 60 x 80 6.0 / 6.6, 300 x 600 (255 tiles) 7.95 / 9.1; 400 x
// 800 (440 tiles) 12.0 / 11.4, 500 x 1000 15.1 / 14.4, 600 x 1200 18.4 / 17.9,
// 1126 x 3000 61.0 / 60.4.
// The batched half-steps always trigger early; there it is close either way: 16
// shots of 1126 x 3000 911.5 / 907, 12 models of mixed sizes 265.8 / 264.8, 6 x 600
// x 1200 98.1 / 99.0, 24 x 200 x 400 69.4 / 70.1, 24 x 60 x 80 17.9 / 16.9.
inline int early_trigger(long long tiles) { return 2 * tiles <= 4 * 148; }
// The arguments of h's half-steps (a: handle_step_args), without column work.
void fill_args(HalfArgs &ha, const tti_handle *h, const StepArgs &a);
void velocity_maps(VelocityMaps &m, const void *maps);  // from a handle's maps
void stress_maps(StressMaps &m, const void *maps);
inline void set_work(HalfArgs &ha, const Extent &e)
{
  ha.work_z0 = e.x1 > 0 ? e.z0 : 0;
  ha.work_z1 = e.x1 > 0 ? e.z1 : 0;
}

// One item of a batched launch: instance, tile origin (x0 with the UNDAMPED
// bit: tile_undamped), the instance's time steps.
struct alignas(16) Work {
  static constexpr int UNDAMPED = 1 << 30;
  int inst, z0, x0, nt;
};

// true when every cell of the tile of WX columns lies where coef1 = 1 and coef2 = dt
__host__ __device__ __forceinline__ bool tile_undamped(const HalfArgs &a, int z0, int x0, int wx)
{
  const Grid &g = a.g;
  return a.undamped_ok && x0 >= g.E && x0 + wx <= g.Nx - g.E && z0 >= (a.freesurface ? 0 : g.E) &&
         z0 + a.tile_rows <= g.Nz - g.E;
}

// Encodes the 2D tensor map of one [Nx][ldz] field for boxes of box_rows x box_cols.
bool encode_map(CUtensorMap *map, const Grid &g, float *field, int box_rows, int box_cols);
// The same for `count` consecutive fields (3D; boxes of one field).
bool encode_map3(CUtensorMap *map, const Grid &g, float *fields, int count, int box_rows, int box_cols);
// Tile grid over rows z_first .. Nz - NH - 1: *z_base receives the first tile
// row, *tile_rows the height of a tile.
dim3 tiles(const Grid &g, int z_first, int *z_base, int *tile_rows);
// (maps: the handle's)
cudaError_t launch_velocity(const HalfArgs &a, const void *maps, int variant, bool exact, cudaStream_t st);
cudaError_t launch_stress(const HalfArgs &a, const void *maps, int variant, bool exact, cudaStream_t st);
// Batched: one launch over all instances' tiles (each instance's arguments
// with z_base set), driven by the work table.
struct BatchLaunch {
  const HalfArgs *inst;  // device: each instance's arguments
  const void *maps;      // device: each instance's VelocityMaps or StressMaps
  const Work *work;      // device: the CTA -> (instance, tile) table
  int nwork;
  const int *step;       // device: the shared step counter
  int offset;            // this launch's step: the counter plus offset
  int variant;
  bool exact, square;    // square: every instance has folded coefficients (set_square)
  unsigned wait_limit;   // polls of a box wait before it gives up
};
cudaError_t launch_velocity_batch(const BatchLaunch &l, cudaStream_t st);
cudaError_t launch_stress_batch(const BatchLaunch &l, cudaStream_t st);
// Sets the kernels' shared-memory attributes (call before a stream capture).
cudaError_t prepare_batch(BatchLaunch l);

// Device side of the TMA halo tiles, shared by the tiled forward and adjoint kernels.
namespace tma {

__device__ __forceinline__ unsigned smem_u32(const void *p)
{
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, unsigned bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// Polls of a bounded TMA wait (about a second): a copy that never lands cannot
// hang the GPU. A handle may lower it (TTIFD_WAIT_LIMIT at tti_create) to run
// the timeout path without a fault.
constexpr unsigned WAIT_LIMIT = 1u << 20;

__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity, unsigned limit = WAIT_LIMIT)
{
  const unsigned a = smem_u32(bar);
  for (unsigned n = 0; n < limit; ++n) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

__device__ __forceinline__ void tma_load_2d(float *dst, const CUtensorMap *map, int c_inner, int c_outer,
                                            unsigned long long *bar)
{
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(c_inner), "r"(c_outer), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(float *dst, const CUtensorMap *map, int c0, int c1, int c2,
                                            unsigned long long *bar)
{
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}

}  // namespace tma
}  // namespace tiled
}  // namespace ttifd
