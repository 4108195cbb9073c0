// Kernel launch wrappers shared by the C-ABI layer (api.cu).
#pragma once

#include "ttifd_internal.cuh"

namespace ttifd {

// ---------------- setup ----------------
struct SetupIn {
  const float *vp, *vs, *rho, *eps, *delta, *theta;  // padded raw model, [Nx][pitch]
  int pitch;                                         // floats per column (Nz: as uploaded)
};
struct SetupOut {
  float *D, *Beta, *coef1, *coef2, *vp, *vs, *rho, *invrho;
  float *c11, *c13, *c15, *c33, *c35, *c55;
  float *sn, *cs, *snv, *csv, *s2, *c2, *s2t;
};
// Scalars of the MEAL profile computed on the host with the host libm
// (exactly as meal.c evaluates them): w[l] = absorbWeight(alpha, l, E).
struct MealConst {
  const float *w;  // device, [E + 1]
  float logR;      // logf(Rcoef)
  float two_thx, two_thz;   // 2 * E * dx, 2 * E * dz
  float dx_fpeak, dz_fpeak; // dx * fpeak, dz * fpeak
  float sqrt3;              // sqrtf(3)
  float dt;
};
void launch_setup(const Grid &g, const SetupIn &in, const SetupOut &out, const MealConst &mc, int variant,
                  float scalar, int freesurface, cudaStream_t st);
// Expands `na` dense physical [nx][nz] arrays (nz * nx floats apart) into
// dense padded [Nx][Nz] arrays (Nz * Nx floats apart), the E-wide rims filled
// as padModel2d fills them on the host.
void launch_expand_physical(const float *phys, float *pad, int na, int nz, int nx, int E, cudaStream_t st);
// Counts cells of [E, Nx-E) x [zD, Nz-E) with coef1 != 1 or coef2 != dt; the
// tiled kernels skip those loads where there are none.
void launch_check_undamped(const Grid &g, const float *coef1, const float *coef2, float dt, int zD, int *count,
                           cudaStream_t st);

// ---------------- per-step ----------------
// Source weight tables over the 11 x 11 window (offset (a, b) at a*11+b,
// a = ix - isx + 5, b = iz - isz + 5), precomputed on the host in the
// reference's float expression order (coord:674-886).
struct SourceTables {
  float k1[121];  // 0.5 w          (stype 1, on sxx/szz)
  float kx[121];  // 2 alpha rx w   (stype 2/3)
  float kz[121];  // 2 alpha rz w
  float k5[121];  // w              (stype 5/6)
  float k7[121];  // 0.5 sqrt2 w    (stype 7)
  float q8;       // 0.125 sqrt2    (stype 8)
};

struct StepArgs {
  Grid g;
  Fields f;
  Params p;
  float invdx, invdz;
  int variant;
  bool exact;
};

void launch_velocity(const StepArgs &a, cudaStream_t st);
void launch_stress(const StepArgs &a, cudaStream_t st);
void launch_energy(const StepArgs &a, int nz, int nx, double *out2, cudaStream_t st);

// A shot's sources, receivers and the rest of its column work (columns.cuh),
// in device memory; rebuilt when its geometry changes.
struct Columns {
  int stype;  // 0: no sources
  int freesurface, tensor, nt, mode2, mt, rec_on;
  // sources by the columns [sx0, sx1) that their windows cover: column ix = sx0 + k
  // has the entries [scol[k], scol[k + 1]) of sat, in the sources' order: source,
  // row, column offset ix - x, and in a column's first one the number of its
  // entries. shead[k]: that first one (all 0: none), one load away.
  int sx0, sx1;
  const int *scol;
  const int4 *sat, *shead;
  const float *amp;  // [source][nt]
  SourceTables t;
  const int *colptr[3], *rz[3], *rid[3];  // receivers grouped by column (null: component off)
  float *rec[3];
  int nrec[3];
  int *flag;
};
// One shot's column work as launches of their own (batched shots, and where
// the tiles do not cover it): one warp per column of [x0, x1), step n (batched:
// *step + n, shots past their nt do nothing, at most `cols` columns each).
struct ColumnShot {
  Grid g;
  Fields f;
  const Columns *c;
  int x0, x1;
};
cudaError_t launch_post(const ColumnShot &s, int n, cudaStream_t st);
cudaError_t launch_sources(const ColumnShot &s, int n, cudaStream_t st);
cudaError_t launch_post_batch(const ColumnShot *d, int ns, int cols, const int *step, int n, cudaStream_t st);
cudaError_t launch_sources_batch(const ColumnShot *d, int ns, int cols, const int *step, int n, cudaStream_t st);
cudaError_t launch_advance(int *step, int n, cudaStream_t st);
// dst[f][0..n) = src[f][0..n), f < 5 (n a multiple of 4, 16-byte aligned arrays)
// the first nf (<= 5) of the arrays src[] into dst[], n floats each, one launch
void launch_copy5(float *const *src, float *const *dst, int nf, size_t n, cudaStream_t st);
// out[r - r0][t] = in[t][r] for t < nts, r0 <= r < r0 + nr (in has n columns)
void launch_transpose(const float *in, float *out, int nts, int n, int r0, int nr, cudaStream_t st);
// Pack a snapshot (kind 1..7) of the physical (savew = 0) or padded area
// into a dense [nx_out][nz_out] buffer.
void launch_snapshot(const StepArgs &a, int kind, int savew, float *dst, cudaStream_t st);

// C-ABI helpers shared by the entry points in other translation units
StepArgs handle_step_args(const tti_handle *h);
void handle_source_tables(const tti_handle *h, SourceTables *t);
int handle_check_flag(tti_handle *h);
// Steps [n0, n1) from the current state (the handle's step index is n0). With
// `keep` what the adjoint needs of them goes to slot n - n0 of the kept steps:
// keep[f] + slot * stride, f < keep_fields.
int handle_steps(tti_handle *h, int n1, float *const *keep, size_t stride);
// brings the handle's Columns on the device up to date with its geometry
int handle_columns(tti_handle *h);
Extent handle_post_extent(const tti_handle *h);  // the cells of its work after the stress update
// Fields of one kept step of the gradient (the arrays `keep` of handle_steps). Tiled kernels: the strain rates vxx vxz vzx vzz, then for the
// coordinate rotation the stress derivative combinations P Q R S (8 fields),
// for the tensor rotation txx tzz txz before the stress half (7), for Bond
// nothing more (4). Per-cell kernels: vx vz after the velocity half and the
// stresses (tensor: tau) before the stress half (5).
int keep_fields(const tti_handle *h);
// allocates what tti_grad_run_binomial of these numbers needs (adjoint.cu)
int grad_reserve(tti_handle *h, int snapshots, int keep_steps);
// frees the gradient's device memory of h (adjoint.cu)
void grad_release(tti_handle *h);
int create_handle(tti_handle **out, const tti_config *cfg, int device, const tti_handle *share, bool force_tiled);
int handle_error(tti_handle *h, int code, const char *msg);

}  // namespace ttifd
