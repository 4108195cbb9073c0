// C ABI of the B200 TTI RSG library (include/ttifd.h).
#include <cfloat>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <future>
#include <vector>

#include <algorithm>
#include <numeric>

#include "columns.cuh"
#include "walk.cuh"

using namespace ttifd;

namespace {

thread_local std::string g_create_error;

int set_err(tti_handle *h, int code, const char *fmt, ...)
{
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (h) h->err = buf;
  else g_create_error = buf;
  return code;
}

// On failure the runtime's last error is cleared too, so that a refused
// allocation is not found again by a later launch check.
#define CK(h, call)                                                                                     \
  do {                                                                                                  \
    cudaError_t e_ = (call);                                                                            \
    if (e_ != cudaSuccess) {                                                                            \
      cudaGetLastError();                                                                               \
      return set_err((h), e_ == cudaErrorMemoryAllocation ? TTI_ERR_NOMEM : TTI_ERR_CUDA, "%s: %s (%s:%d)", \
                     #call, cudaGetErrorString(e_), __FILE__, __LINE__);                                \
    }                                                                                                   \
  } while (0)

// Arrays each formulation needs on the device (beyond D/Beta/coef/vp/vs/rho
// which every formulation keeps for the setup dumps).
bool param_used(int variant, int p)
{
  switch (p) {
  case TTI_P_C15:
  case TTI_P_C35:
    return variant == TTI_BOND;
  case TTI_P_SIN:
  case TTI_P_COS:
  case TTI_P_SIN_V:
  case TTI_P_COS_V:
    return variant == TTI_COORDINATE;
  case TTI_P_SIN2:
  case TTI_P_COS2:
  case TTI_P_SIN_2T:
    return variant == TTI_TENSOR;
  default:
    return true;
  }
}

int nfields(int variant) { return variant == TTI_TENSOR ? 8 : 5; }

StepArgs step_args(const tti_handle *h)
{
  StepArgs a;
  a.g = h->g;
  a.f = Fields{h->fld[0], h->fld[1], h->fld[2], h->fld[3], h->fld[4], h->fld[5], h->fld[6], h->fld[7]};
  const float *const *P = h->par;
  a.p = Params{P[TTI_P_COEF1], P[TTI_P_COEF2], P[TTI_P_INVRHO], P[TTI_P_C11], P[TTI_P_C13], P[TTI_P_C15],
               P[TTI_P_C33],   P[TTI_P_C35],   P[TTI_P_C55],    P[TTI_P_SIN], P[TTI_P_COS], P[TTI_P_SIN_V],
               P[TTI_P_COS_V], P[TTI_P_SIN2],  P[TTI_P_COS2],   P[TTI_P_SIN_2T]};
  a.invdx = h->invdx;
  a.invdz = h->invdz;
  a.variant = h->cfg.variant;
  a.exact = h->exact;
  return a;
}

// Host precompute of the source weight tables in the reference's float
// expression order (coord:607, 684-691, 711-713, 733-734, 775-777, 880-882).
void source_tables(const tti_handle *h, SourceTables *t)
{
  const float dx = h->cfg.dx, dz = h->cfg.dz, dt = h->cfg.dt;
  const float alpha = logf(0.8f) / (dx * dx + dz * dz);
  for (int a = 0; a < 11; ++a)
    for (int b = 0; b < 11; ++b) {
      const float rx = (a - NH) * dx, rz = (b - NH) * dz;
      const float w = expf(alpha * (rx * rx + rz * rz)) * h->invdx * h->invdz * dt;
      const int k = a * 11 + b;
      t->k1[k] = 0.5f * w;
      t->kx[k] = 2.0f * alpha * rx * w;
      t->kz[k] = 2.0f * alpha * rz * w;
      t->k5[k] = w;
      t->k7[k] = 0.5f * sqrtf(2.0f) * w;
    }
  t->q8 = 0.125f * sqrtf(2.0f);
}

// A single shot's steps go out as replays of a graph of GRAPH_STEPS steps where
// the CTAs of two launches fit the device together (early_trigger): there the
// kernels are hardly longer than the host's launches, and the gaps between them
// show. us a step by replays / by launches: 60 x 80 6.25 / 6.7, 200 x 400 7.6 /
// 7.95, 300 x 600 (255 tiles) 8.2 / 8.3, the first run, which captures, 8.6 /
// 10.5. Above, a replay is not faster (400 x 800, 440 tiles, 12.0 / 11.65; 600 x
// 1200 18.5 / 18.5). The capture costs what replays save over 60 to 250 steps,
// so runs of fewer steps do without.
constexpr int GRAPH_TILES = 2 * 148, GRAPH_NT = 200;

int check_cfg(const tti_config *c)
{
  if (c->variant < 0 || c->variant > 2) return set_err(nullptr, TTI_ERR_ARG, "variant must be 0, 1 or 2");
  if (c->nz <= 0 || c->nx <= 0 || c->nt <= 0) return set_err(nullptr, TTI_ERR_ARG, "nz, nx, nt must be positive");
  if (!(c->dx > 0) || !(c->dz > 0) || !(c->dt > 0)) return set_err(nullptr, TTI_ERR_ARG, "dx, dz, dt must be positive");
  if (c->ealThick < 0) return set_err(nullptr, TTI_ERR_ARG, "ealThick must be >= 0");
  if (!(c->fpeak > 0)) return set_err(nullptr, TTI_ERR_ARG, "fpeak must be positive");
  if (c->freesurface != 0 && c->freesurface != 1) return set_err(nullptr, TTI_ERR_ARG, "freesurface must be 0 or 1");
  if (c->stype < 1 || c->stype > 8) return set_err(nullptr, TTI_ERR_ARG, "stype must be 1..8");
  if (c->seistype < 0 || c->seistype > 3) return set_err(nullptr, TTI_ERR_ARG, "seistype must be 0..3");
  if (c->mt < 1) return set_err(nullptr, TTI_ERR_ARG, "mt must be >= 1");
  if (c->wsave < 0 || c->wsave > 5) return set_err(nullptr, TTI_ERR_ARG, "wsave must be 0..5");
  if (c->savew != 0 && c->savew != 1) return set_err(nullptr, TTI_ERR_ARG, "savew must be 0 or 1");
  if (c->wsave > 0 && c->snap_sample < 1) return set_err(nullptr, TTI_ERR_ARG, "snap_sample must be >= 1");
  if (c->mode != 1 && c->mode != 2) return set_err(nullptr, TTI_ERR_ARG, "mode must be 1 or 2");
  return TTI_OK;
}

int current_it(const tti_handle *h) { return h->cfg.mode == 2 ? h->cfg.nt - 1 - h->step_index : h->step_index; }

// Fills h->d_cols from the geometry, and decides where the column work runs.
// The tiled kernels take it when every column it touches is in a tile
// ([NH, Nx - NH)) and its rows fall in at most two rows of tiles: each warp of
// such a tile then goes through its column's receivers once more, which for
// receivers spread over all depths costs more than the launch it saves.
int sync_columns(tti_handle *h)
{
  if (!h->cols_dirty) return TTI_OK;
  const tti_config &c = h->cfg;
  const Grid &g = h->g;
  Columns w;
  memset(&w, 0, sizeof w);
  w.stype = h->nsrc > 0 ? c.stype : 0;
  w.freesurface = c.freesurface == 1;
  w.tensor = c.variant == TTI_TENSOR;
  w.nt = c.nt;
  w.mode2 = c.mode == 2;
  w.mt = c.mt;
  w.sx0 = h->src_at.x0;
  w.sx1 = h->src_at.x1;
  w.scol = h->d_scol;
  w.sat = h->d_sat;
  w.shead = h->d_shead;
  w.amp = h->d_src;
  source_tables(h, &w.t);
  const bool want_v = c.seistype == 1 || c.seistype == 3, want_p = c.seistype == 2 || c.seistype == 3;
  h->rec_at = Extent();
  for (int k = 0; k < 3; ++k) {
    const bool on = (k < 2 ? want_v : want_p) && h->nrec[k] > 0;
    w.colptr[k] = on ? h->d_rcol[k] : nullptr;
    w.rz[k] = h->d_rzs[k];
    w.rid[k] = h->d_rid[k];
    w.rec[k] = h->d_rec[k];
    w.nrec[k] = h->nrec[k];
    if (on) h->rec_at.add(h->rec_of[k]);
  }
  w.rec_on = h->rec_at.x1 > 0;
  w.flag = h->d_flag;
  Extent post = h->rec_at;
  if (w.stype == 1) post.add(h->src_at);
  if (w.freesurface) post.add(NH, g.Nx - NH, g.izStart - NH, g.izStart + NH + 1);
  auto fold = [&](const Extent &e) {
    if (!h->use_tiled) return false;
    int z_base, rows;
    const int nt = (int)tiled::tiles(g, g.izStart, &z_base, &rows).x;
    auto tile = [&](int z) { return std::min(std::max((z - z_base) / rows, 0), nt - 1); };

    return nt > 0 && e.x1 > 0 && e.x0 >= NH && e.x1 <= g.Nx - NH && tile(e.z1 - 1) - tile(e.z0) < 2;
  };
  h->fold_src = w.stype >= 2 && fold(h->src_at);
  // after the stress update only rows that are updated or images of such
  // (column_work keeps them on chip)
  const int top = w.freesurface ? g.izStart - NH : g.izStart;
  int z_base, rows;
  tiled::tiles(g, g.izStart, &z_base, &rows);
  const bool images = !w.freesurface || g.izStart + NH < std::min(g.Nz - NH, z_base + rows);
  h->fold_post = fold(post) && post.z0 >= top && post.z1 <= g.Nz - NH && images;
  CK(h, cudaMemcpyAsync(h->d_cols, &w, sizeof w, cudaMemcpyHostToDevice, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));  // w goes out of scope
  h->cols_dirty = false;
  return TTI_OK;
}

// Rows of the column work after the stress update of a step that does or does
// not record.
Extent post_extent(const tti_handle *h, bool rec_now)
{
  const Grid &g = h->g;
  Extent e;
  if (rec_now) e = h->rec_at;
  if (h->nsrc > 0 && h->cfg.stype == 1) e.add(h->src_at);
  if (h->cfg.freesurface == 1) e.add(NH, g.Nx - NH, g.izStart - NH, g.izStart + NH + 1);
  return e;
}

// The arguments of one time step's tiled half-steps. What the gradient keeps
// of a step (keep_fields): the stress kernel writes the strain rates vxx vxz
// vzx vzz (keep[0..3]) and for the tensor rotation the tau it starts from
// (keep[4..6]); the coordinate velocity kernel writes the stress derivative
// combinations P Q R S (keep[4..7]).
struct TiledStep {
  tiled::HalfArgs v, s;
};
void tiled_step(const tti_handle *h, const Extent &post, float *const *keep, size_t stride, TiledStep &t)
{
  const int variant = h->cfg.variant;
  memset(&t, 0, sizeof t);
  tiled::fill_args(t.v, h, step_args(h));
  t.v.n = t.v.k0 = h->step_index;
  t.v.kstride = stride;
  t.s = t.v;
  if (h->fold_src) tiled::set_work(t.v, h->src_at);
  if (h->fold_post) tiled::set_work(t.s, post);
  if (!keep) return;
  if (variant == TTI_COORDINATE)
    for (int k = 0; k < 4; ++k) t.v.kd[k] = keep[4 + k];
  for (int k = 0; k < 4; ++k) t.s.kd[k] = keep[k];
  if (variant == TTI_TENSOR)
    for (int k = 0; k < 3; ++k) t.s.kt[k] = keep[4 + k];
}

// Launches one time step (coord:611-926 body). With `ev` (5 events) the
// phases are bracketed for tti_profile_steps: ev[0] | velocity | ev[1] |
// velocity sources | ev[2] | stress | ev[3] | the rest | ev[4] (the sources
// and the rest are empty where the half-step kernels do the column work). With
// `keep` the gradient's forward pass keeps what the adjoint needs of the step
// in slot step - k0; the per-cell kernels keep a copy of vx vz and sxx szz sxz
// (tensor: txx tzz txz) after the sources, from whose stencils the adjoint
// works.
int launch_one_step(tti_handle *h, cudaEvent_t *ev = nullptr, float *const *keep = nullptr, size_t stride = 0,
                    int k0 = 0)
{
  const tti_config &c = h->cfg;
  const int it = current_it(h), n = h->step_index;
  const StepArgs a = step_args(h);
  const Extent post = post_extent(h, it % c.mt == 0);
  ColumnShot cs{h->g, a.f, h->d_cols, h->src_at.x0, h->src_at.x1};
  TiledStep t;
  if (h->use_tiled) {
    tiled_step(h, post, keep, stride, t);
    t.v.k0 = t.s.k0 = k0;
  }
  if (ev) CK(h, cudaEventRecord(ev[0], h->stream));
  if (h->use_tiled) CK(h, tiled::launch_velocity(t.v, h->tmaps, c.variant, h->exact, h->stream));
  else launch_velocity(a, h->stream);
  h->launches++;
  if (ev) CK(h, cudaEventRecord(ev[1], h->stream));
  if (h->nsrc > 0 && c.stype >= 2 && !h->fold_src) {
    CK(h, launch_sources(cs, n, h->stream));
    h->launches++;
  }
  if (keep && !h->use_tiled) {  // v after the sources, and sigma or tau
    const bool ten = c.variant == TTI_TENSOR;
    float *const src[5] = {h->fld[0], h->fld[1], h->fld[ten ? 5 : 2], h->fld[ten ? 6 : 3], h->fld[ten ? 7 : 4]};
    float *dst[5];
    for (int f = 0; f < 5; ++f) dst[f] = keep[f] + (size_t)(n - k0) * stride;
    launch_copy5(src, dst, 5, h->g.n, h->stream);
    h->launches++;
  }
  if (ev) CK(h, cudaEventRecord(ev[2], h->stream));
  // after the stress update: free surface, stress source and receivers
  if (h->use_tiled) CK(h, tiled::launch_stress(t.s, h->tmaps, c.variant, h->exact, h->stream));
  else launch_stress(a, h->stream);
  h->launches++;
  if (ev) CK(h, cudaEventRecord(ev[3], h->stream));
  if (post.x1 > 0 && !h->fold_post) {
    cs.x0 = post.x0;
    cs.x1 = post.x1;
    CK(h, launch_post(cs, n, h->stream));
    h->launches++;
  }
  if (c.energy == 1) {
    launch_energy(a, c.nz, c.nx, h->d_energy + 2 * (size_t)it, h->stream);
    h->launches++;
  }
  if (ev) CK(h, cudaEventRecord(ev[4], h->stream));
  CK(h, cudaGetLastError());
  h->step_index++;
  return TTI_OK;
}

// Captures GRAPH_STEPS steps with the arguments t, whose step counters are on
// the device; false when no graph could be made.
bool capture_steps(tti_handle *h, StepGraph &g, TiledStep t)
{
  // relaxed for this thread: nothing here may spoil a capture that another
  // thread has under way
  struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  } relaxed;
  if (g.exec) cudaGraphExecDestroy(g.exec);
  g.exec = nullptr;
  g.key.assign(reinterpret_cast<unsigned char *>(&t), reinterpret_cast<unsigned char *>(&t + 1));
  if (cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < GRAPH_STEPS && e == cudaSuccess; ++k) {
    t.v.n = t.s.n = k;
    e = tiled::launch_velocity(t.v, h->tmaps, h->cfg.variant, h->exact, h->stream);
    if (e == cudaSuccess) e = tiled::launch_stress(t.s, h->tmaps, h->cfg.variant, h->exact, h->stream);
  }
  if (e == cudaSuccess) e = launch_advance(h->d_clk, GRAPH_STEPS, h->stream);
  cudaGraph_t graph = nullptr;
  const cudaError_t end = cudaStreamEndCapture(h->stream, &graph);
  if (e == cudaSuccess) e = end;
  if (e == cudaSuccess) e = cudaGraphInstantiate(&g.exec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (e == cudaSuccess) return true;
  cudaGetLastError();
  g.exec = nullptr;
  return false;
}

// As many whole graph replays as fit before step n1; the fields that are kept
// belong to the segment from step k0. Where no graph can be made the handle
// launches every step by itself from here on.
int replay_steps(tti_handle *h, int n1, float *const *keep, size_t stride, int k0)
{
  const int n = h->step_index, steps = (n1 - n) / GRAPH_STEPS * GRAPH_STEPS;
  if (steps == 0) return TTI_OK;
  TiledStep t;
  tiled_step(h, post_extent(h, true), keep, stride, t);
  for (tiled::HalfArgs *a : {&t.v, &t.s}) {
    a->clk = h->d_clk;
    a->n = a->k0 = 0;
  }
  StepGraph &g = h->graph[keep != nullptr];
  if (!g.exec || g.key.size() != sizeof t || memcmp(g.key.data(), &t, sizeof t) != 0)
    if (!capture_steps(h, g, t)) {
      h->use_graphs = false;
      return TTI_OK;
    }
  const tiled::StepClock clk{n, k0};
  CK(h, cudaMemcpyAsync(h->d_clk, &clk, sizeof clk, cudaMemcpyHostToDevice, h->stream));
  for (int k = 0; k < steps; k += GRAPH_STEPS) CK(h, cudaGraphLaunch(g.exec, h->stream));
  h->launches += 2 * steps + steps / GRAPH_STEPS;
  h->step_index += steps;
  return TTI_OK;
}

// Forward steps up to step n1 (see handle_steps): graph replays where the
// handle uses them and every launch of a step is a half-step, single launches
// for the rest. The first step of a run is never captured, so that its
// kernels' attributes are set outside a capture.
int run_forward(tti_handle *h, int n1, float *const *keep, size_t stride)
{
  const int k0 = h->step_index;
  const bool whole = h->cfg.energy == 0 && (h->fold_post || post_extent(h, true).x1 == 0) &&
                     (h->fold_src || h->nsrc == 0 || h->cfg.stype == 1);
  while (h->step_index < n1) {
    if (h->use_graphs && whole && h->step_index > k0)
      if (const int rc = replay_steps(h, n1, keep, stride, k0)) return rc;
    if (h->step_index < n1)
      if (const int rc = launch_one_step(h, nullptr, keep, stride, k0)) return rc;
  }
  return TTI_OK;
}

int snapshot_kinds(int wsave, int *kinds)
{
  switch (wsave) {
  case 1: kinds[0] = 1; kinds[1] = 2; return 2;
  case 2: kinds[0] = 3; return 1;
  case 3: kinds[0] = 1; kinds[1] = 2; kinds[2] = 3; return 3;
  case 4: kinds[0] = 4; kinds[1] = 5; return 2;
  case 5: kinds[0] = 6; kinds[1] = 7; return 2;
  default: return 0;
  }
}

// Copies `bytes` from device memory into a host buffer whose pages are
// resident, ordered after the work already on h's stream; returns once the
// data are in place. Above one chunk, through two page-locked chunks: the DMA
// of chunk c runs while host threads copy chunk c - 1 out (the driver's own
// staging of a pageable destination is slower); otherwise directly.
int download(tti_handle *h, void *dst, const void *src, size_t bytes)
{
  constexpr size_t CH = PIN_CHUNK * sizeof(float);
  float *pin[2] = {nullptr, nullptr};
  if (bytes > CH) {
    pin[0] = pinned_chunk();
    pin[1] = pinned_chunk();
  }
  for (int b = 0; b < 2 && pin[0] && pin[1]; ++b)
    if (!h->pev[5 + b] && cudaEventCreateWithFlags(&h->pev[5 + b], cudaEventDisableTiming) != cudaSuccess)
      pinned_release(pin[b]), pin[b] = nullptr;
  if (!pin[0] || !pin[1]) {
    pinned_release(pin[0]);
    pinned_release(pin[1]);
    CK(h, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    return TTI_OK;
  }
  const size_t nchunk = (bytes + CH - 1) / CH;
  cudaError_t e = cudaSuccess;
  for (size_t c = 0; c <= nchunk && e == cudaSuccess; ++c) {
    if (c < nchunk) {
      const size_t off = c * CH, nb = std::min(CH, bytes - off);
      e = cudaMemcpyAsync(pin[c & 1], static_cast<const char *>(src) + off, nb, cudaMemcpyDeviceToHost, h->stream);
      if (e == cudaSuccess) e = cudaEventRecord(h->pev[5 + (c & 1)], h->stream);
    }
    if (c > 0 && e == cudaSuccess) {
      const size_t p = c - 1, off = p * CH, nb = std::min(CH, bytes - off);
      e = cudaEventSynchronize(h->pev[5 + (p & 1)]);
      if (e == cudaSuccess) parallel_copy(static_cast<char *>(dst) + off, pin[p & 1], nb, 8);
    }
  }
  // wait on the error path too before the chunks go back to the shared list
  const cudaError_t es = cudaStreamSynchronize(h->stream);
  if (e == cudaSuccess) e = es;
  pinned_release(pin[0]);
  pinned_release(pin[1]);
  CK(h, e);
  return TTI_OK;
}

// Output size of one snapshot kind (savew = 0: the physical area).
void snapshot_dims(const tti_handle *h, int *nzo, int *nxo)
{
  const Grid &g = h->g;
  *nzo = h->cfg.savew == 0 ? g.Nz - 2 * g.E : g.Nz;
  *nxo = h->cfg.savew == 0 ? g.Nx - 2 * g.E : g.Nx;
}

// The snapshot of step h->snap_it whose copy into the caller's page-locked
// buffer is in flight on copy_stream: waits for the copy, then (deliver) runs
// the callbacks of its kinds in order. Error paths drop it once the copy is
// done, so that no transfer into the caller's buffer outlives tti_run.
int finish_snapshot(tti_handle *h, bool deliver)
{
  if (!h->snap_pending) return TTI_OK;
  h->snap_pending = false;
  const cudaError_t e = cudaEventSynchronize(h->snap_done);
  if (!deliver) return TTI_OK;
  CK(h, e);
  int nzo, nxo, kinds[3];
  snapshot_dims(h, &nzo, &nxo);
  const size_t n = (size_t)nzo * nxo;
  const int nk = snapshot_kinds(h->cfg.wsave, kinds);
  for (int q = 0; q < nk; ++q)
    if (h->snap_fn(h->snap_arg, h->snap_it, kinds[q], h->snap_user + q * n, nzo, nxo) != 0)
      return set_err(h, TTI_ERR_CALLBACK, "snapshot callback aborted the run at it=%d", h->snap_it);
  return TTI_OK;
}

int do_snapshot(tti_handle *h, tti_snapshot_fn fn, void *user, int it)
{
  int nzo, nxo, kinds[3];
  snapshot_dims(h, &nzo, &nxo);
  const size_t n = (size_t)nzo * nxo;
  const int nk = snapshot_kinds(h->cfg.wsave, kinds);
  // Into the caller's page-locked buffer: every kind packed on the device, one
  // copy on copy_stream that overlaps the next time steps on h->stream.
  const bool overlap = h->snap_user && h->snap_user_pinned;
  const size_t dev = overlap ? nk * n : n;
  if (overlap) {
    const int rc = finish_snapshot(h, true);  // the previous one, and d_snap is free again
    if (rc) return rc;
  }
  if (h->snap_cap < dev) {
    pool_free(h->d_snap, h->stream);
    h->d_snap = nullptr;
    h->snap_cap = 0;
    CK(h, pool_alloc(reinterpret_cast<void **>(&h->d_snap), dev * sizeof(float), h->stream));
    h->snap_cap = dev;
  }
  StepArgs a = step_args(h);
  if (overlap) {
    if (!h->copy_stream) CK(h, cudaStreamCreateWithFlags(&h->copy_stream, cudaStreamNonBlocking));
    if (!h->snap_packed) CK(h, cudaEventCreateWithFlags(&h->snap_packed, cudaEventDisableTiming));
    if (!h->snap_done) CK(h, cudaEventCreateWithFlags(&h->snap_done, cudaEventDisableTiming));
    for (int q = 0; q < nk; ++q) {
      launch_snapshot(a, kinds[q], h->cfg.savew, h->d_snap + q * n, h->stream);
      h->launches++;
    }
    CK(h, cudaEventRecord(h->snap_packed, h->stream));
    CK(h, cudaStreamWaitEvent(h->copy_stream, h->snap_packed, 0));
    CK(h, cudaMemcpyAsync(h->snap_user, h->d_snap, nk * n * sizeof(float), cudaMemcpyDeviceToHost, h->copy_stream));
    CK(h, cudaEventRecord(h->snap_done, h->copy_stream));
    h->snap_pending = true;
    h->snap_it = it;
    h->snap_fn = fn;
    h->snap_arg = user;
    return TTI_OK;
  }
  float *host = h->snap_user;  // a pageable caller's buffer: kind q at q * n
  if (!host && h->h_snap_cap < n) {
    free(h->h_snap);
    h->h_snap_cap = 0;
    h->h_snap = static_cast<float *>(malloc(n * sizeof(float)));
    if (!h->h_snap) return set_err(h, TTI_ERR_NOMEM, "host allocation of the snapshot buffer failed");
    prefault(h->h_snap, n * sizeof(float));
    h->h_snap_cap = n;
  }
  for (int q = 0; q < nk; ++q) {
    float *dst = host ? host + q * n : h->h_snap;
    launch_snapshot(a, kinds[q], h->cfg.savew, h->d_snap, h->stream);
    h->launches++;
    const int rc = download(h, dst, h->d_snap, n * sizeof(float));
    if (rc) return rc;
    if (fn(user, it, kinds[q], dst, nzo, nxo) != 0)
      return set_err(h, TTI_ERR_CALLBACK, "snapshot callback aborted the run at it=%d", it);
  }
  return TTI_OK;
}

// The time loop of tti_run after the reset; device time between events
// ev0 and ev1. A snapshot of the last snapshot step may still be in flight.
int run_steps(tti_handle *h, tti_snapshot_fn snap, void *user)
{
  const tti_config &c = h->cfg;
  CK(h, cudaEventRecord(h->ev0, h->stream));
  const bool snaps = snap && c.wsave > 0;
  while (h->step_index < c.nt) {
    // up to and with the next step that has a snapshot
    int n1 = snaps ? h->step_index : c.nt - 1;
    auto it_of = [&](int n) { return c.mode == 2 ? c.nt - 1 - n : n; };
    while (n1 < c.nt - 1 && it_of(n1) % c.snap_sample != 0) ++n1;
    int rc = run_forward(h, n1 + 1, nullptr, 0);
    if (rc == TTI_OK && snaps && it_of(n1) % c.snap_sample == 0) rc = do_snapshot(h, snap, user, it_of(n1));
    if (rc) return rc;
  }
  CK(h, cudaEventRecord(h->ev1, h->stream));
  CK(h, cudaEventSynchronize(h->ev1));
  CK(h, cudaEventElapsedTime(&h->last_ms, h->ev0, h->ev1));
  return TTI_OK;
}

int check_flag(tti_handle *h)
{
  int flag = 0;
  CK(h, cudaMemcpyAsync(&flag, h->d_flag, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  if (flag & 4) return set_err(h, TTI_ERR_CUDA, "a TMA tile wait timed out in a tiled half-step kernel");
  if (flag) return set_err(h, TTI_ERR_NONFINITE, "non-finite value recorded at a receiver (unstable run?)");
  return TTI_OK;
}

// Copies na host arrays [Nx][Nz] into dense device arrays [Nx][Nz] on h's
// stream (dense, not pitched: a contiguous host-to-device copy runs about 1.5x
// faster than a pitched one of the same bytes; the setup kernel re-pitches).
// From page-locked arrays (tti_host_alloc) one copy each, at the link's rate.
// Otherwise through two page-locked chunks, column blocks at a time: host threads copy
// block c into one chunk while the DMA engine moves block c - 1 from the other
// (TTIFD_UPLOAD=pageable: straight from the caller's pageable arrays, which
// the driver stages itself, about 10.5 GB/s on B200 hosts).
// `na` dense host arrays of `ncol` columns of `sl` floats each into dense
// device arrays (the padded model: Nx columns of Nz; the physical one: nx of nz).
int upload_arrays(tti_handle *h, const float *const *src, float *const *dst, int na, int sl, int ncol)
{
  const size_t col = (size_t)sl * sizeof(float);
  auto copy = [&](int k, int x0, const float *from, int nx) {
    return cudaMemcpyAsync(dst[k] + (size_t)x0 * sl, from, col * nx, cudaMemcpyHostToDevice, h->stream);
  };
  bool pinned = true;  // all from page-locked memory: straight to the device
  for (int k = 0; k < na; ++k) pinned = pinned && is_pinned(src[k]);
  if (pinned) {
    for (int k = 0; k < na; ++k) CK(h, copy(k, 0, src[k], ncol));
    return TTI_OK;
  }
  const char *mode = getenv("TTIFD_UPLOAD");
  const bool pageable = mode && strcmp(mode, "pageable") == 0;
  const int per = (int)std::min<size_t>(ncol, PIN_CHUNK / sl);  // columns per chunk
  float *pin[2] = {nullptr, nullptr};
  if (!pageable && per > 0) {
    pin[0] = pinned_chunk();
    pin[1] = pinned_chunk();
  }
  for (int b = 0; b < 2 && pin[0] && pin[1]; ++b)
    if (!h->pev[5 + b] && cudaEventCreateWithFlags(&h->pev[5 + b], cudaEventDisableTiming) != cudaSuccess)
      pinned_release(pin[b]), pin[b] = nullptr;
  if (!pin[0] || !pin[1]) {
    pinned_release(pin[0]);
    pinned_release(pin[1]);
    for (int k = 0; k < na; ++k) CK(h, copy(k, 0, src[k], ncol));
    return TTI_OK;
  }
  cudaError_t e = cudaSuccess;
  bool pending[2] = {false, false};
  int c = 0;
  for (int k = 0; k < na && e == cudaSuccess; ++k)
    for (int x0 = 0; x0 < ncol && e == cudaSuccess; x0 += per, ++c) {
      const int nx = std::min(per, ncol - x0), b = c & 1;
      if (pending[b]) e = cudaEventSynchronize(h->pev[5 + b]);  // chunk b's previous DMA has drained
      if (e != cudaSuccess) break;
      parallel_copy(pin[b], src[k] + (size_t)x0 * sl, col * nx, 8);
      e = copy(k, x0, pin[b], nx);
      if (e == cudaSuccess) e = cudaEventRecord(h->pev[5 + b], h->stream);
      pending[b] = true;
    }
  // the chunks go back to the shared free list only once their copies are done
  const cudaError_t es = cudaStreamSynchronize(h->stream);
  if (e == cudaSuccess) e = es;
  pinned_release(pin[0]);
  pinned_release(pin[1]);
  CK(h, e);
  return TTI_OK;
}

int copy_out_pitched(tti_handle *h, const float *src, float *out)
{
  const Grid &g = h->g;
  CK(h, cudaMemcpy2DAsync(out, (size_t)g.Nz * sizeof(float), src, (size_t)g.ldz * sizeof(float),
                          (size_t)g.Nz * sizeof(float), g.Nx, cudaMemcpyDeviceToHost, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  return TTI_OK;
}

}  // namespace

namespace ttifd {
int keep_fields(const tti_handle *h)
{
  if (!h->use_tiled) return 5;
  return h->cfg.variant == TTI_COORDINATE ? 8 : h->cfg.variant == TTI_TENSOR ? 7 : 4;
}
StepArgs handle_step_args(const tti_handle *h) { return step_args(h); }
void handle_source_tables(const tti_handle *h, SourceTables *t) { source_tables(h, t); }
int handle_steps(tti_handle *h, int n1, float *const *keep, size_t stride) { return run_forward(h, n1, keep, stride); }
int handle_columns(tti_handle *h) { return sync_columns(h); }
Extent handle_post_extent(const tti_handle *h) { return post_extent(h, true); }
int handle_check_flag(tti_handle *h) { return check_flag(h); }
int handle_error(tti_handle *h, int code, const char *msg) { return set_err(h, code, "%s", msg); }
}  // namespace ttifd

extern "C" {

const char *tti_last_error(const tti_handle *h) { return h ? h->err.c_str() : g_create_error.c_str(); }

int tti_create(tti_handle **out, const tti_config *cfg, int device)
{
  return ttifd::create_handle(out, cfg, device, nullptr, false);
}

}  // extern "C"

namespace ttifd {

// tti_create with two options for batched execution: `share` (its parameter
// arrays are used, not allocated; cfg must describe the same grid) and
// `force_tiled` (the tiled kernels whatever TTIFD_KERNEL says).
int create_handle(tti_handle **out, const tti_config *cfg, int device, const tti_handle *share, bool force_tiled)
{
  if (!out || !cfg) return set_err(nullptr, TTI_ERR_ARG, "null argument");
  *out = nullptr;
  int rc = check_cfg(cfg);
  if (rc) return rc;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return set_err(nullptr, TTI_ERR_CUDA, "no CUDA device available");
  if (device < 0 || device >= ndev) return set_err(nullptr, TTI_ERR_ARG, "device %d out of range", device);
  tti_handle *h = new tti_handle();
  h->cfg = *cfg;
  h->device = device;
  // Default arithmetic: every product and sum rounded separately in the
  // reference's expression order (the results of a -ffp-contract=off build of
  // the reference, bit for bit); TTIFD_EXACT=0 lets the compiler contract into
  // FMA (about 3 % faster on the full workload, within 1e-5 of it otherwise).
  const char *ex = getenv("TTIFD_EXACT");
  h->exact = !(ex && ex[0] == '0');
  // test hook: polls of the first TMA wait of the tiled kernels (the timeout path)
  const char *wl = getenv("TTIFD_WAIT_LIMIT");
  h->wait_limit = wl && *wl ? (unsigned)strtoul(wl, nullptr, 10) : tiled::tma::WAIT_LIMIT;
  Grid &g = h->g;
  g.E = cfg->ealThick + NH;
  g.Nz = cfg->nz + 2 * g.E;
  g.Nx = cfg->nx + 2 * g.E;
  g.ldz = (g.Nz + 31) / 32 * 32;
  g.izStart = cfg->freesurface == 0 ? NH : g.E;
  g.n = (size_t)g.ldz * g.Nx;
  h->invdx = (float)(1.0 / cfg->dx);
  h->invdz = (float)(1.0 / cfg->dz);
  h->nts = (cfg->nt - 1) / cfg->mt + 1;
  auto fail = [&](int code) {
    std::string msg = h->err;
    tti_destroy(h);
    set_err(nullptr, code, "%s", msg.c_str());
    return code;
  };
  if (cudaSetDevice(device) != cudaSuccess) {
    set_err(h, TTI_ERR_CUDA, "cudaSetDevice(%d) failed", device);
    return fail(TTI_ERR_CUDA);
  }
  auto alloc = [&](float **p) -> int {
    cudaError_t e = pool_alloc(reinterpret_cast<void **>(p), g.n * sizeof(float), h->stream);
    if (e != cudaSuccess)
      return set_err(h, TTI_ERR_NOMEM, "device allocation of %zu bytes failed: %s", g.n * sizeof(float),
                     cudaGetErrorString(e));
    e = cudaMemsetAsync(*p, 0, g.n * sizeof(float), h->stream);
    if (e != cudaSuccess) return set_err(h, TTI_ERR_CUDA, "cudaMemset failed: %s", cudaGetErrorString(e));
    return TTI_OK;
  };
  if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&h->ev0) != cudaSuccess || cudaEventCreate(&h->ev1) != cudaSuccess) {
    set_err(h, TTI_ERR_CUDA, "stream/event creation failed");
    return fail(TTI_ERR_CUDA);
  }
  {
    // default: the tiled half-step kernels; TTIFD_KERNEL=naive selects the
    // one-thread-per-cell kernels (the cross-check path)
    const char *kern = getenv("TTIFD_KERNEL");
    const bool naive = kern && strcmp(kern, "naive") == 0;
    h->use_tiled = force_tiled || !naive;
  }
  for (int f = 0; f < nfields(cfg->variant); ++f)
    if ((rc = alloc(&h->fld[f]))) return fail(rc);
  if (share) {
    h->owner = share;
    for (int p = 0; p < TTI_P_COUNT; ++p) h->par[p] = share->par[p];
  }
  for (int p = 0; p < TTI_P_COUNT && !share; ++p)
    if (param_used(cfg->variant, p) && (rc = alloc(&h->par[p]))) return fail(rc);
  if (h->use_tiled) {
    if (posix_memalign(&h->tmaps, 64, tiled::MAPS * sizeof(CUtensorMap)) != 0) {
      h->tmaps = nullptr;
      set_err(h, TTI_ERR_NOMEM, "host allocation failed");
      return fail(TTI_ERR_NOMEM);
    }
    const StepArgs a = step_args(h);
    int z_base, rows;
    const dim3 nt = tiled::tiles(g, g.izStart, &z_base, &rows);
    const char *gs = getenv("TTIFD_GRAPH_STEPS");  // 0: every step by its own launches
    h->use_graphs = (int)(nt.x * nt.y) <= GRAPH_TILES && cfg->nt >= GRAPH_NT && (!gs || atoi(gs) > 0);
    if (!tiled::encode_maps(static_cast<CUtensorMap *>(h->tmaps), g, cfg->variant, a.f, a.p)) {
      set_err(h, TTI_ERR_CUDA, "cuTensorMapEncodeTiled failed");
      return fail(TTI_ERR_CUDA);
    }
  }
  if (pool_alloc(reinterpret_cast<void **>(&h->d_clk), sizeof(tiled::StepClock), h->stream) != cudaSuccess ||
      pool_alloc(reinterpret_cast<void **>(&h->d_cols), sizeof(Columns), h->stream) != cudaSuccess ||
      pool_alloc(reinterpret_cast<void **>(&h->d_flag), sizeof(int), h->stream) != cudaSuccess ||
      pool_alloc(reinterpret_cast<void **>(&h->d_energy), sizeof(double) * 2 * (size_t)cfg->nt, h->stream) !=
          cudaSuccess) {
    set_err(h, TTI_ERR_NOMEM, "device allocation failed");
    return fail(TTI_ERR_NOMEM);
  }
  cudaMemsetAsync(h->d_flag, 0, sizeof(int), h->stream);
  cudaMemsetAsync(h->d_energy, 0, sizeof(double) * 2 * (size_t)cfg->nt, h->stream);
  if (cudaStreamSynchronize(h->stream) != cudaSuccess) {
    set_err(h, TTI_ERR_CUDA, "initialisation failed");
    return fail(TTI_ERR_CUDA);
  }
  *out = h;
  return TTI_OK;
}

}  // namespace ttifd

extern "C" {

int tti_destroy(tti_handle *h)
{
  if (!h) return TTI_OK;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (auto &g : h->graph)
    if (g.exec) cudaGraphExecDestroy(g.exec);
  cudaStream_t fs = h->stream;  // pool blocks are released in stream order
  for (auto &p : h->fld) pool_free(p, fs);
  if (!h->owner) {
    for (auto &p : h->par) pool_free(p, fs);
  }
  for (int k = 0; k < 3; ++k) {
    pool_free(h->d_rz[k], fs);  // with d_rzs, d_rid, d_rcol (one block)
    pool_free(h->d_rec[k], fs);
  }
  pool_free(h->d_sat, fs);  // with d_shead, d_sx, d_sz, d_scol
  pool_free(h->d_src, fs);
  pool_free(h->d_energy, fs);
  pool_free(h->d_flag, fs);
  if (!h->owner) {  // a batch instance borrows its model's copies
    pool_free(h->m_eps, fs);
    pool_free(h->m_delta, fs);
    pool_free(h->m_theta, fs);
  }
  pool_free(h->d_snap, fs);
  pool_free(h->d_stage, fs);
  pool_free(h->d_cols, fs);
  pool_free(h->d_clk, fs);
  if (fs) cudaStreamSynchronize(fs);
  grad_release(h);
  free(h->h_snap);
  if (h->ev0) cudaEventDestroy(h->ev0);
  if (h->ev1) cudaEventDestroy(h->ev1);
  free(h->tmaps);
  for (auto e : h->pev)
    if (e) cudaEventDestroy(e);
  if (h->snap_packed) cudaEventDestroy(h->snap_packed);
  if (h->snap_done) cudaEventDestroy(h->snap_done);
  if (h->copy_stream) cudaStreamDestroy(h->copy_stream);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
  return TTI_OK;
}

int tti_grid(const tti_handle *h, int *Nz, int *Nx, int *E)
{
  if (!h) return TTI_ERR_ARG;
  if (Nz) *Nz = h->g.Nz;
  if (Nx) *Nx = h->g.Nx;
  if (E) *E = h->g.E;
  return TTI_OK;
}

// tti_upload_model (padded arrays) and tti_upload_model_physical (physical
// arrays, the rims filled on the device) from here on are one path.
static int upload_model(tti_handle *h, const float *const *src, bool physical)
{
  for (int k = 0; k < 6; ++k)
    if (!src[k]) return set_err(h, TTI_ERR_ARG, "null model array");
  if (h->owner) return set_err(h, TTI_ERR_STATE, "this handle shares the parameters of another; upload through it");
  CK(h, cudaSetDevice(h->device));
  const tti_config &c = h->cfg;
  const Grid &g = h->g;
  const size_t np = (size_t)g.Nz * g.Nx;
  // Stability check on the unscaled padded vp (stable.c:217-246; the rims
  // repeat physical values, so the physical maximum is the padded one). Its
  // host maximum runs on other threads while the arrays travel to the
  // device; nothing is computed from them on the device before it has passed.
  const float *vp = src[0];
  const size_t nv = physical ? (size_t)c.nz * c.nx : np;
  auto vmax_f = std::async(std::launch::async, [vp, nv] { return host_max(vp, nv, FLT_MIN); });
  // raw model on the device (dense [Nx][Nz], one block of six arrays), freed
  // after the precompute; a physical model first lands densely after it (one
  // contiguous copy per array: a pitched copy into the padded layout ran
  // slower than the padded bytes it saves) and is expanded on the device
  float *raw[6] = {}, *phys[6] = {};
  float *d_w = nullptr, *raw_block = nullptr;
  int rc = TTI_OK;
  {
    const size_t extra = physical ? 6 * nv : 0;
    cudaError_t e = pool_alloc(reinterpret_cast<void **>(&raw_block), (6 * np + extra) * sizeof(float), h->stream);
    if (e != cudaSuccess) rc = set_err(h, TTI_ERR_NOMEM, "device allocation failed: %s", cudaGetErrorString(e));
  }
  for (int k = 0; k < 6; ++k) {
    raw[k] = raw_block + (size_t)k * np;
    phys[k] = raw_block + 6 * np + (size_t)k * nv;
  }
  if (rc == TTI_OK)
    rc = physical ? upload_arrays(h, src, phys, 6, c.nz, c.nx)
                  : upload_arrays(h, src, raw, 6, g.Nz, g.Nx);
  if (rc == TTI_OK && physical) {
    launch_expand_physical(phys[0], raw_block, 6, c.nz, c.nx, g.E, h->stream);
    if (cudaGetLastError() != cudaSuccess) rc = set_err(h, TTI_ERR_CUDA, "model expansion kernel failed to launch");
  }
  {
    const double vmax = vmax_f.get();
    const double csum = (double)rsg(0) + (double)rsg(2) + (double)rsg(4);
    const double dtmax = 1.0f / (vmax * sqrt((1.0 / (c.dx * c.dx) + 1.0 / (c.dz * c.dz)) * csum));
    if (rc == TTI_OK && c.dt > dtmax) {
      cudaStreamSynchronize(h->stream);
      pool_free(raw_block, h->stream);
      return set_err(h, TTI_ERR_UNSTABLE,
                     "the finite differenct scheme is unstable! the time step size must smaller than %5.5f!", dtmax);
    }
  }
  if (rc == TTI_OK) {
    // MEAL scalars evaluated with the host libm, as meal.c:23-29, 62-66 do
    const int nl = g.E;
    const float pd = 2;
    const float Rcoef = powf(10.0f, -1.0f * ((log10f((float)nl) - 1.0f) / (log10f(2.0f))) - 3.0f - 0.5f * pd);
    const float alpha = c.eal_alpha == -1.0f ? 2.5f : c.eal_alpha;
    std::vector<float> w(nl + 1, 0.0f);
    for (int l = 1; l <= nl; ++l) {
      const float d = (0.1f * l) / (0.1f * nl);
      w[l] = expf(logf(2.0f) * powf(d, alpha)) - 1.0f;
    }
    cudaError_t e = pool_alloc(reinterpret_cast<void **>(&d_w), sizeof(float) * (nl + 1), h->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(d_w, w.data(), sizeof(float) * (nl + 1), cudaMemcpyHostToDevice, h->stream);
    if (e != cudaSuccess) rc = set_err(h, TTI_ERR_CUDA, "MEAL table upload: %s", cudaGetErrorString(e));
    MealConst mc;
    mc.w = d_w;
    mc.logR = logf(Rcoef);
    const float thx = nl * c.dx, thz = nl * c.dz;
    mc.two_thx = 2.0f * thx;
    mc.two_thz = 2.0f * thz;
    mc.dx_fpeak = c.dx * c.fpeak;
    mc.dz_fpeak = c.dz * c.fpeak;
    mc.sqrt3 = sqrtf(3.0f);
    mc.dt = c.dt;
    float **P = h->par;
    SetupIn in{raw[0], raw[1], raw[2], raw[3], raw[4], raw[5], g.Nz};
    SetupOut o{P[TTI_P_D],   P[TTI_P_BETA],  P[TTI_P_COEF1], P[TTI_P_COEF2], P[TTI_P_VP],    P[TTI_P_VS],
               P[TTI_P_RHO], P[TTI_P_INVRHO], P[TTI_P_C11],  P[TTI_P_C13],   P[TTI_P_C15],   P[TTI_P_C33],
               P[TTI_P_C35], P[TTI_P_C55],   P[TTI_P_SIN],   P[TTI_P_COS],   P[TTI_P_SIN_V], P[TTI_P_COS_V],
               P[TTI_P_SIN2], P[TTI_P_COS2], P[TTI_P_SIN_2T]};
    if (rc == TTI_OK) {
      launch_setup(g, in, o, mc, c.variant, c.scalar, c.freesurface, h->stream);
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
      if (e != cudaSuccess) rc = set_err(h, TTI_ERR_CUDA, "setup kernels: %s", cudaGetErrorString(e));
    }
  }
  cudaStreamSynchronize(h->stream);
  // the gradient's chain rule needs epsilon and delta as given (and theta for Bond)
  if (rc == TTI_OK) {
    for (int k = 0; k < (c.variant == TTI_BOND ? 3 : 2); ++k) {
      float *&dst = k == 0 ? h->m_eps : k == 1 ? h->m_delta : h->m_theta;
      if (!dst && pool_alloc(reinterpret_cast<void **>(&dst), g.n * sizeof(float), h->stream) != cudaSuccess) {
        rc = set_err(h, TTI_ERR_NOMEM, "device allocation failed");
        break;
      }
      cudaMemsetAsync(dst, 0, g.n * sizeof(float), h->stream);
      cudaMemcpy2DAsync(dst, (size_t)g.ldz * sizeof(float), raw[3 + k], (size_t)g.Nz * sizeof(float),
                        (size_t)g.Nz * sizeof(float), g.Nx, cudaMemcpyDeviceToDevice, h->stream);
    }
    cudaStreamSynchronize(h->stream);
  }
  pool_free(raw_block, h->stream);
  pool_free(d_w, h->stream);
  if (rc == TTI_OK && h->use_tiled) {
    // the tiled kernels skip coef1/coef2 loads where they are exactly 1 and
    // dt; verify that on the device instead of assuming the MEAL rim geometry
    int *cnt = nullptr;
    int bad = -1;
    if (pool_alloc(reinterpret_cast<void **>(&cnt), sizeof(int), h->stream) == cudaSuccess) {
      cudaMemsetAsync(cnt, 0, sizeof(int), h->stream);
      launch_check_undamped(g, h->par[TTI_P_COEF1], h->par[TTI_P_COEF2], c.dt, c.freesurface ? 0 : g.E, cnt,
                                   h->stream);
      cudaMemcpyAsync(&bad, cnt, sizeof(int), cudaMemcpyDeviceToHost, h->stream);
      pool_free(cnt, h->stream);
      cudaStreamSynchronize(h->stream);
    }
    h->undamped_ok = bad == 0;
  }
  if (rc == TTI_OK) h->have_model = true;
  return rc;
}

int tti_upload_model(tti_handle *h, const float *vp, const float *vs, const float *rho, const float *epsilon,
                     const float *delta, const float *theta)
{
  if (!h) return set_err(h, TTI_ERR_ARG, "null handle");
  const float *src[6] = {vp, vs, rho, epsilon, delta, theta};
  return upload_model(h, src, false);
}

int tti_upload_model_physical(tti_handle *h, const float *vp, const float *vs, const float *rho,
                              const float *epsilon, const float *delta, const float *theta)
{
  if (!h) return set_err(h, TTI_ERR_ARG, "null handle");
  const float *src[6] = {vp, vs, rho, epsilon, delta, theta};
  return upload_model(h, src, true);
}

int tti_fetch_param(tti_handle *h, int which, float *out)
{
  if (!h || !out) return TTI_ERR_ARG;
  if (which < 0 || which >= TTI_P_COUNT || !h->par[which])
    return set_err(h, TTI_ERR_ARG, "parameter %d is not used by this formulation", which);
  if (!h->have_model) return set_err(h, TTI_ERR_STATE, "model not uploaded");
  CK(h, cudaSetDevice(h->device));
  return copy_out_pitched(h, h->par[which], out);
}

int tti_set_source(tti_handle *h, int ntrace, const int *posx, const int *posz, const float *src)
{
  if (!h || ntrace < 0 || (ntrace > 0 && (!posx || !posz || !src))) return set_err(h, TTI_ERR_ARG, "bad source");
  const tti_config &c = h->cfg;
  for (int i = 0; i < ntrace; ++i) {
    if (posz[i] < 0 || posz[i] > c.nz)
      return set_err(h, TTI_ERR_RANGE, "the position of source in 1st dimension (%d) must be between 0 and %d!",
                     posz[i], c.nz);
    if (posx[i] < 0 || posx[i] > c.nx)
      return set_err(h, TTI_ERR_RANGE, "the position of source in 2nd dimension (%d) must be between 0 and %d!",
                     posx[i], c.nx);
  }
  CK(h, cudaSetDevice(h->device));
  pool_free(h->d_sat, h->stream);
  pool_free(h->d_src, h->stream);
  h->d_sat = h->d_shead = nullptr;
  h->d_sx = h->d_sz = h->d_scol = nullptr;
  h->d_src = nullptr;
  h->nsrc = 0;
  h->cols_dirty = true;
  h->src_at = Extent();
  if (ntrace == 0) return TTI_OK;
  // One device block: the sources by column (Columns::sat), each column's first,
  // their positions, the column offsets. A warp of the column work reads what
  // its column has. Going through all sources instead, a load each, 300 along the
  // surface of 600 x 1200 cells took 82 us a step, where one takes 18 (now 21);
  // 750 at 1126 x 3000 228 (now 65).
  auto first_x = [&](int i) { return std::max(0, posx[i] + h->g.E - NH); };
  auto last_x = [&](int i) { return std::min(h->g.Nx, posx[i] + h->g.E + NH + 1); };
  for (int i = 0; i < ntrace; ++i) {
    const int z = posz[i] + h->g.E;
    h->src_at.add(first_x(i), last_x(i), std::max(0, z - NH), std::min(h->g.Nz, z + NH + 1));
  }
  const int x0 = h->src_at.x0, ncol = h->src_at.x1 - x0;
  std::vector<int> col(ncol + 1, 0);
  for (int i = 0; i < ntrace; ++i)
    for (int k = first_x(i); k < last_x(i); ++k) ++col[k - x0 + 1];
  for (int k = 0; k < ncol; ++k) col[k + 1] += col[k];
  const size_t m = (size_t)col[ncol];
  std::vector<int> blk(4 * (m + ncol) + 2 * (size_t)ntrace + ncol + 1, 0), next(col.begin(), col.end());
  int *head = blk.data() + 4 * m, *sx = head + 4 * (size_t)ncol, *sz = sx + ntrace;
  std::copy(col.begin(), col.end(), sz + ntrace);
  for (int i = 0; i < ntrace; ++i) {
    sx[i] = posx[i] + h->g.E;
    sz[i] = posz[i] + h->g.E;
    for (int k = first_x(i); k < last_x(i); ++k) {
      int *e = blk.data() + 4 * (size_t)next[k - x0]++;
      e[0] = i;
      e[1] = sz[i];
      e[2] = k - sx[i];
    }
  }
  for (int k = 0; k < ncol; ++k)
    if (col[k + 1] > col[k]) {
      int *e = blk.data() + 4 * (size_t)col[k];
      e[3] = col[k + 1] - col[k];
      std::copy_n(e, 4, head + 4 * (size_t)k);
    }
  CK(h, pool_alloc(reinterpret_cast<void **>(&h->d_sat), sizeof(int) * blk.size(), h->stream));
  h->d_shead = h->d_sat + m;
  h->d_sx = reinterpret_cast<int *>(h->d_shead + ncol);
  h->d_sz = h->d_sx + ntrace;
  h->d_scol = h->d_sz + ntrace;
  CK(h, pool_alloc(reinterpret_cast<void **>(&h->d_src), sizeof(float) * (size_t)ntrace * c.nt, h->stream));
  CK(h, cudaMemcpyAsync(h->d_sat, blk.data(), sizeof(int) * blk.size(), cudaMemcpyHostToDevice, h->stream));
  CK(h, cudaMemcpyAsync(h->d_src, src, sizeof(float) * (size_t)ntrace * c.nt, cudaMemcpyHostToDevice, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  h->nsrc = ntrace;
  return TTI_OK;
}

int tti_set_receivers(tti_handle *h, int kind, int ntrace, const int *posx, const int *posz)
{
  if (!h || kind < 0 || kind > 2 || ntrace < 0 || (ntrace > 0 && (!posx || !posz)))
    return set_err(h, TTI_ERR_ARG, "bad receiver arguments");
  const tti_config &c = h->cfg;
  for (int i = 0; i < ntrace; ++i) {
    if (posz[i] < 0 || posz[i] > c.nz)
      return set_err(h, TTI_ERR_RANGE, "the position of receiver in 1st dimension (%d) must be between 0 and %d!",
                     posz[i], c.nz);
    if (posx[i] < 0 || posx[i] > c.nx)
      return set_err(h, TTI_ERR_RANGE, "the position of receiver in 2nd dimension (%d) must be between 0 and %d!",
                     posx[i], c.nx);
  }
  CK(h, cudaSetDevice(h->device));
  // One device block per component holds its receiver rows in the caller's
  // order (d_rz, owner of the block), then, grouped by padded-grid column for
  // the column pass (k_post), the rows (d_rzs), the receiver ids (d_rid) and
  // the column offsets (d_rcol): one copy and one synchronisation per call.
  pool_free(h->d_rz[kind], h->stream);
  pool_free(h->d_rec[kind], h->stream);
  h->d_rz[kind] = h->d_rzs[kind] = h->d_rid[kind] = h->d_rcol[kind] = nullptr;
  h->d_rec[kind] = nullptr;
  h->nrec[kind] = 0;
  h->cols_dirty = true;
  h->rec_of[kind] = Extent();
  if (ntrace == 0) return TTI_OK;
  const int Nx = h->g.Nx;
  std::vector<int> blk(3 * (size_t)ntrace + Nx + 1, 0), x(ntrace), order(ntrace);
  int *z = blk.data(), *zs = z + ntrace, *ids = zs + ntrace, *colptr = ids + ntrace;
  for (int i = 0; i < ntrace; ++i) {
    x[i] = posx[i] + h->g.E;
    z[i] = posz[i] + h->g.E;
    h->rec_of[kind].add(x[i], x[i] + 1, z[i], z[i] + 1);
  }
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return x[a] < x[b]; });
  for (int i = 0; i < ntrace; ++i) colptr[x[i] + 1]++;
  for (int c = 0; c < Nx; ++c) colptr[c + 1] += colptr[c];
  for (int i = 0; i < ntrace; ++i) {
    zs[i] = z[order[i]];
    ids[i] = order[i];
  }
  int *d = nullptr;
  CK(h, pool_alloc(reinterpret_cast<void **>(&d), sizeof(int) * blk.size(), h->stream));
  h->d_rz[kind] = d;
  h->d_rzs[kind] = d + ntrace;
  h->d_rid[kind] = d + 2 * (size_t)ntrace;
  h->d_rcol[kind] = d + 3 * (size_t)ntrace;
  // the traces (ntrace x nts floats, the largest of these) from the handle's pool
  CK(h, pool_alloc(reinterpret_cast<void **>(&h->d_rec[kind]), sizeof(float) * (size_t)ntrace * h->nts, h->stream));
  CK(h, cudaMemcpyAsync(d, blk.data(), sizeof(int) * blk.size(), cudaMemcpyHostToDevice, h->stream));
  CK(h, cudaMemsetAsync(h->d_rec[kind], 0, sizeof(float) * (size_t)ntrace * h->nts, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));  // the host block goes out of scope
  h->nrec[kind] = ntrace;
  return TTI_OK;
}

int tti_reset(tti_handle *h)
{
  if (!h) return TTI_ERR_ARG;
  CK(h, cudaSetDevice(h->device));
  for (auto p : h->fld)
    if (p) CK(h, cudaMemsetAsync(p, 0, h->g.n * sizeof(float), h->stream));
  for (int k = 0; k < 3; ++k)
    if (h->d_rec[k]) CK(h, cudaMemsetAsync(h->d_rec[k], 0, sizeof(float) * (size_t)h->nrec[k] * h->nts, h->stream));
  CK(h, cudaMemsetAsync(h->d_energy, 0, sizeof(double) * 2 * (size_t)h->cfg.nt, h->stream));
  CK(h, cudaMemsetAsync(h->d_flag, 0, sizeof(int), h->stream));
  h->step_index = 0;
  return TTI_OK;
}

int tti_step(tti_handle *h, int nsteps)
{
  if (!h || nsteps < 0) return TTI_ERR_ARG;
  if (!h->have_model) return set_err(h, TTI_ERR_STATE, "model not uploaded");
  if (h->step_index + nsteps > h->cfg.nt) return set_err(h, TTI_ERR_STATE, "step past nt");
  CK(h, cudaSetDevice(h->device));
  if (int rc = sync_columns(h)) return rc;
  CK(h, cudaEventRecord(h->ev0, h->stream));
  if (const int rc = run_forward(h, h->step_index + nsteps, nullptr, 0)) return rc;
  CK(h, cudaEventRecord(h->ev1, h->stream));
  CK(h, cudaEventSynchronize(h->ev1));
  CK(h, cudaEventElapsedTime(&h->last_ms, h->ev0, h->ev1));
  return check_flag(h);
}

int tti_set_snapshot_buffer(tti_handle *h, float *host, size_t floats)
{
  if (!h) return TTI_ERR_ARG;
  if (host) {
    int nzo, nxo, kinds[3];
    snapshot_dims(h, &nzo, &nxo);
    const size_t need = (size_t)snapshot_kinds(h->cfg.wsave, kinds) * nzo * nxo;
    if (need == 0) return set_err(h, TTI_ERR_STATE, "wsave = %d writes no snapshots", h->cfg.wsave);
    if (floats < need)
      return set_err(h, TTI_ERR_ARG, "snapshot buffer of %zu floats, wsave = %d needs %zu", floats, h->cfg.wsave,
                     need);
  }
  h->snap_user = host;
  h->snap_user_pinned = host && is_pinned(host);
  return TTI_OK;
}

int tti_run(tti_handle *h, tti_snapshot_fn snap, void *user)
{
  if (!h) return TTI_ERR_ARG;
  if (!h->have_model) return set_err(h, TTI_ERR_STATE, "model not uploaded");
  int rc = tti_reset(h);
  if (rc) return rc;
  if ((rc = sync_columns(h))) return rc;
  rc = run_steps(h, snap, user);
  if (rc) {
    finish_snapshot(h, false);
    return rc;
  }
  if ((rc = finish_snapshot(h, true))) return rc;
  return check_flag(h);
}

int tti_profile_steps(tti_handle *h, int nsteps, float ms[3])
{
  if (!h || !ms || nsteps < 0) return TTI_ERR_ARG;
  if (!h->have_model) return set_err(h, TTI_ERR_STATE, "model not uploaded");
  if (h->step_index + nsteps > h->cfg.nt) return set_err(h, TTI_ERR_STATE, "step past nt");
  CK(h, cudaSetDevice(h->device));
  for (int k = 0; k < 5; ++k)
    if (!h->pev[k]) CK(h, cudaEventCreate(&h->pev[k]));
  if (int rc = sync_columns(h)) return rc;
  ms[0] = ms[1] = ms[2] = 0.0f;
  for (int n = 0; n < nsteps; ++n) {
    int rc = launch_one_step(h, h->pev);
    if (rc) return rc;
    CK(h, cudaEventSynchronize(h->pev[4]));
    float t01, t12, t23, t34;
    CK(h, cudaEventElapsedTime(&t01, h->pev[0], h->pev[1]));
    CK(h, cudaEventElapsedTime(&t12, h->pev[1], h->pev[2]));
    CK(h, cudaEventElapsedTime(&t23, h->pev[2], h->pev[3]));
    CK(h, cudaEventElapsedTime(&t34, h->pev[3], h->pev[4]));
    ms[0] += t01;
    ms[1] += t23;
    ms[2] += t12 + t34;
  }
  return check_flag(h);
}

int tti_kernel_launches(const tti_handle *h, long long *n)
{
  if (!h || !n) return TTI_ERR_ARG;
  *n = h->launches;
  return TTI_OK;
}

int tti_get_stream(const tti_handle *h, void **stream)
{
  if (!h || !stream) return TTI_ERR_ARG;
  *stream = static_cast<void *>(h->stream);
  return TTI_OK;
}

int tti_elapsed_ms(const tti_handle *h, float *ms)
{
  if (!h || !ms) return TTI_ERR_ARG;
  *ms = h->last_ms;
  return TTI_OK;
}

int tti_fetch_traces(tti_handle *h, int kind, float *out)
{
  if (!h || !out || kind < 0 || kind > 2) return TTI_ERR_ARG;
  if (!h->d_rec[kind]) return set_err(h, TTI_ERR_ARG, "no receivers of kind %d", kind);
  CK(h, cudaSetDevice(h->device));
  const int n = h->nrec[kind], nts = h->nts;
  // Chunks of receivers transposed on the device (time-major to the caller's
  // [ntrace][nts]) into a staging buffer, then to the caller's block.
  constexpr size_t STAGE = PIN_CHUNK;  // floats per chunk
  if (!h->d_stage) CK(h, pool_alloc(reinterpret_cast<void **>(&h->d_stage), STAGE * sizeof(float), h->stream));
  if ((size_t)nts > STAGE || nts > 65535 * 32)
    return set_err(h, TTI_ERR_ARG, "trace of %d samples is longer than the fetch supports", nts);
  const int per = (int)std::max<size_t>(1, STAGE / (size_t)nts);  // receivers per chunk
  const int nchunk = (n + per - 1) / per;
  if (is_pinned(out)) {
    // page-locked destination: each chunk's copy runs asynchronously, and the
    // next transpose into the staging buffer waits for it in stream order
    for (int r0 = 0; r0 < n; r0 += per) {
      const int nr = std::min(per, n - r0);
      launch_transpose(h->d_rec[kind], h->d_stage, nts, n, r0, nr, h->stream);
      h->launches++;
      CK(h, cudaMemcpyAsync(out + (size_t)r0 * nts, h->d_stage, sizeof(float) * (size_t)nr * nts,
                            cudaMemcpyDeviceToHost, h->stream));
    }
    CK(h, cudaStreamSynchronize(h->stream));
    return TTI_OK;
  }
  // A fetch of one chunk goes straight to the caller's block: staging would
  // not overlap anything, and the first staged fetch of a process pays for
  // page-locking the chunks (about 13 ms for two).
  float *pin[2] = {nullptr, nullptr};
  if (nchunk > 1) {
    pin[0] = pinned_chunk();
    pin[1] = pinned_chunk();
  }
  for (int b = 0; b < 2 && pin[0] && pin[1]; ++b)
    if (!h->pev[5 + b] && cudaEventCreateWithFlags(&h->pev[5 + b], cudaEventDisableTiming) != cudaSuccess)
      pinned_release(pin[b]), pin[b] = nullptr;
  if (pin[0] && pin[1]) {
    // Through two page-locked chunks: the copy of chunk c to the host runs
    // while the host threads copy chunk c - 1 into the caller's block (taking
    // its page faults in parallel).
    cudaError_t e = cudaSuccess;
    for (int c = 0; c <= nchunk && e == cudaSuccess; ++c) {
      if (c < nchunk) {
        const int r0 = c * per, nr = std::min(per, n - r0), b = c & 1;
        launch_transpose(h->d_rec[kind], h->d_stage, nts, n, r0, nr, h->stream);
        h->launches++;
        e = cudaMemcpyAsync(pin[b], h->d_stage, sizeof(float) * (size_t)nr * nts, cudaMemcpyDeviceToHost, h->stream);
        if (e == cudaSuccess) e = cudaEventRecord(h->pev[5 + b], h->stream);
      }
      if (c > 0 && e == cudaSuccess) {
        const int p = c - 1, r0 = p * per, nr = std::min(per, n - r0), b = p & 1;
        e = cudaEventSynchronize(h->pev[5 + b]);
        if (e == cudaSuccess) parallel_copy(out + (size_t)r0 * nts, pin[b], sizeof(float) * (size_t)nr * nts);
      }
    }
    // wait for the stream on the error path too: a device-to-host copy into a
    // chunk may still be in flight, and a released chunk can go to another
    // handle at once
    const cudaError_t es = cudaStreamSynchronize(h->stream);
    if (e == cudaSuccess) e = es;
    pinned_release(pin[0]);
    pinned_release(pin[1]);
    CK(h, e);
    return TTI_OK;
  }
  pinned_release(pin[0]);
  pinned_release(pin[1]);
  // no page-locked memory: straight into the caller's block, its pages
  // faulted in first from several host threads
  prefault(out, sizeof(float) * (size_t)n * nts);
  for (int r0 = 0; r0 < n; r0 += per) {
    const int nr = std::min(per, n - r0);
    launch_transpose(h->d_rec[kind], h->d_stage, nts, n, r0, nr, h->stream);
    h->launches++;
    // pageable destination: returns once the copy is complete, so the next
    // chunk may overwrite the staging buffer
    CK(h, cudaMemcpyAsync(out + (size_t)r0 * nts, h->d_stage, sizeof(float) * (size_t)nr * nts,
                          cudaMemcpyDeviceToHost, h->stream));
  }
  CK(h, cudaStreamSynchronize(h->stream));
  return TTI_OK;
}

int tti_fetch_field(tti_handle *h, int which, float *out)
{
  if (!h || !out || which < 0 || which >= 8) return TTI_ERR_ARG;
  if (!h->fld[which]) return set_err(h, TTI_ERR_ARG, "field %d is not used by this formulation", which);
  CK(h, cudaSetDevice(h->device));
  return copy_out_pitched(h, h->fld[which], out);
}

int tti_fetch_energy(tti_handle *h, float *ek, float *ep)
{
  if (!h || !ek || !ep) return TTI_ERR_ARG;
  CK(h, cudaSetDevice(h->device));
  const int nt = h->cfg.nt;
  std::vector<double> e(2 * (size_t)nt);
  CK(h, cudaMemcpyAsync(e.data(), h->d_energy, sizeof(double) * e.size(), cudaMemcpyDeviceToHost, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  for (int it = 0; it < nt; ++it) {
    ek[it] = 0.5f * (float)e[2 * (size_t)it] * h->cfg.dx * h->cfg.dz;
    ep[it] = 0.5f * (float)e[2 * (size_t)it + 1] * h->cfg.dx * h->cfg.dz;
  }
  return TTI_OK;
}

}  // extern "C"
