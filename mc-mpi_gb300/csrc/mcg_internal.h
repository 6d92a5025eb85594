/*
 * mcg_internal.h - context layout shared by the translation units of
 * libmcgb300 (not part of the public ABI).
 */
#ifndef MCG_INTERNAL_H
#define MCG_INTERNAL_H

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <vector>

#include "exact_libm.h"
#include "mcg_device.cuh"
#include "mcgb300.h"

/* Per-context state of the batched-slab unit (mcg_batch.cu). */
struct mcg_batch_state {
  int n_slabs = 0, total_cells = 0, max_cells = 0;
  int64_t total_histories = 0;
  std::vector<mcg_slab> slabs;
  std::vector<int32_t> cell_off;
  /* slabs that take a lane per history, strict and fast: 1 and 2 in the batch
   * (mcg_batch_lanes), 4 and 8 in a launch of their own (mcg_thick) */
  std::vector<uint8_t> slab_lanes;
  void *d_slabs = nullptr;  /* mcg_batch_slab_dev[] */
  void *d_items = nullptr;  /* mcg_batch_item[] */
  int n_items = 0, n_tiled = 0, items_cap = 0; /* the first n_tiled by tiles */
  int lane_cells = 0; /* of the longest slab of the others */
  float4 *d_cells_strict = nullptr, *d_cells_fast = nullptr;
  float4 *d_tab = nullptr; /* the tiles' per-cell parameters */
  unsigned long long *d_tally = nullptr;
  unsigned long long *d_item_next = nullptr;
  float min_w = 0.f;
  /* launch shape, chosen by mcg_batch_set_launch or the autotuner */
  int block = 1024, tally_mode = 1;
  int defer = 0; /* lanes that wait for the full step, 0: default (mcg_batch_set_deferral) */
  int64_t item_histories = 16384;
  /* history- or event-based; events per pass of the event engine */
  int algorithm = MCG_ALGO_HISTORY, event_steps = 8;
  unsigned long long *d_hist0 = nullptr; /* first history of each slab (event mode) */
  double hist0_fraction = -1.0;          /* fraction of the histories d_hist0 is for */
  /* CUDA graph of one run (memset of the item counter + the kernel) */
  cudaGraphExec_t graph = nullptr;
  bool graph_valid = false;
  cudaStream_t side = nullptr; /* the lane form's, between fork and join */
  cudaEvent_t fork = nullptr, join = nullptr;
  /* the context's settings that the graph's kernels hold by value */
  int graph_mode = -1, graph_scale = 0, graph_refill = 0;
  uint32_t graph_steps = 0;
  int64_t items_built_for = -1; /* item size, launch, arithmetic and share of the histories
                                   the list is for */
  int items_grid = 0;
  bool items_strict = false;
  double items_fraction = 1.0;
};

/* Per-context state of the adjoint unit (mcg_adjoint.cu). */
struct mcg_adj_state {
  float2 *d_aux = nullptr;               /* {w_c, 1/sig_s} per chain cell */
  unsigned long long *d_grad = nullptr;  /* grad_a[n], grad_s[n], loss */
  float2 *d_sum = nullptr;               /* `sums` histories' losses (forward -> replay) */
  int n = 0;
  int64_t sums = 0, histories = 0;
  int g_log2 = 36;
};

struct mcg_fit_state; /* mcg_fit.cu */

/* Device buffers of the workers' forms (mcg_worker.cu), kept between calls
 * and grown on demand, so a Worker called repeatedly allocates nothing. */
struct mcg_worker_state {
  void *dev = nullptr;
  size_t bytes = 0;
  cudaStream_t monitor = nullptr; /* progress reads and the abort word */
};

struct mcg_ext {
  mcg_batch_state batch;
  mcg_adj_state adj;
  mcg_fit_state *fit = nullptr;
  mcg_worker_state worker;
};

/* Structure-of-arrays particle buffer of the event-based tracker: per
 * particle the state, the cell index local to its chain or slab, the history
 * (chain) or slab (batched) it belongs to, and its step and scatter counts.
 * In the collision queue the seed is already advanced to the flight
 * sample's state, which determines the sample. */
struct mcg_soa {
  unsigned long long *seed;
  float *x, *mu, *wmc, *res; /* res: the fast weight's rounding residue */
  int32_t *idx, *hid, *nst, *nsc;
};

/* Counters of the event engine, on the device. */
struct mcg_ev_ctl {
  unsigned long long n_in, n_out, n_q;     /* particles in the bank, out, in the queue */
  unsigned long long next, total;          /* histories born so far, of the run */
  unsigned long long birth_base, birth_n;  /* this pass's newborns: slots, count */
  unsigned long long birth_first, passes;
};

/* One slab of the batched form (and of the event engine's slab mode). */
struct mcg_batch_slab_dev {
  int32_t cell_off, m;
  int64_t n_hist;
  mcg_source src;
};

/* Sums of a chain's optical widths, sig_a and sig_i: its optical depths. */
struct mcg_widths {
  double a = 0.0, i = 0.0;
  void add(const float4 &c)
  {
    const double len = (double)c.w - c.z;
    a += (c.x < 0.0f ? -c.x : c.x) * len;
    i += (c.y < 0.0f ? -c.y : c.y) * len;
  }
};

struct mcg_context {
  int device = 0, mode = MCG_MODE_STRICT;
  int sm_count = 0, smem_optin = 0, cc_major = 0, cc_minor = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  float last_ms = 0.f;
  int last_grid = 0, last_block = 0;
  long long launches = 0;

  /* chain of layers */
  int n_layers = 0, n_cells = 0, cell_lo = 0;
  float min_w = 0.f;
  std::vector<int32_t> layer_start, layer_m;
  std::vector<float> layer_dx;
  std::vector<float4> cells_strict;
  bool thin_step = false; /* mcg_strict_thin */
  bool thin = false;      /* every cell's sig_a width <= 2e-4 (strict THIN) */
  bool thin_fast = false; /* sig_a and sig_i widths <= 4e-4 (fast THIN) */
  bool thick = false, thick_fast = false; /* mcg_thick, strict and fast */
  float width_a = 0.f, width_i = 0.f; /* those largest widths */
  double depth_i = 0.0;               /* the chain's optical depth in sig_i, where it scatters */
  mcg_widths widths;
  float4 *d_cells_strict = nullptr, *d_cells_fast = nullptr;
  /* the tiles' per-cell parameters (mcg_tile_entry), MCG_TAB_PAD entries before
   * and after; of the thin form one such array per direction, for chains that may
   * take it */
  float4 *d_tab = nullptr;
  float2 *d_thin = nullptr;
  unsigned long long *d_tally = nullptr;
  int log2_scale = 40;
  unsigned long long *d_counters = nullptr, *d_next = nullptr;

  /* strict libm */
  bool libm_loaded = false;
  mcg_libm_dev libm = {};
  mcg_libm_tab *libm_tab = nullptr;
  float run_bounds[3] = {}; /* mcg_run_bounds of the table: b_thin, c_thin, b_mid */
  uint32_t libm_n_log = 0, libm_n_exp = 0;

  /* particle buffers of the host-pointer entry points */
  mcg_particle *d_part = nullptr;
  int32_t *d_res = nullptr;
  int64_t *d_steps = nullptr, *d_scat = nullptr;
  size_t scratch_cap = 0;

  /* launch shape */
  int block = 0, blocks_per_sm = 0, refill = 0; /* refill 0: chosen per kernel */
  uint32_t max_steps = 1u << 28; /* per-history step limit (MCG_ERR_LIMIT) */
  int tally_mode = 1;            /* MCG_TALLY_SMEM32 */

  /* algorithm: history-based (default) or event-based with K events per pass */
  int algorithm = MCG_ALGO_HISTORY, event_steps = 1, event_passes = 0;
  mcg_soa event_buf[3] = {}; /* bank in, bank out, collision queue */
  size_t event_cap = 0;
  std::vector<void *> event_owned;
  mcg_ev_ctl *event_ctl = nullptr;

  std::vector<void *> owned; /* device allocations freed at destroy */
  mcg_ext *ext = nullptr;
};

int mcg_fail(int code, const char *fmt, ...);
/* cudaMalloc of the set-up of a geometry or a fit (mcg_set_layers,
 * mcg_batch_set, mcg_fit_set) and of the histories' sums; a test can make one
 * of them report cudaErrorMemoryAllocation without attempting it
 * (mcg_testing_fail_allocation). */
cudaError_t mcg_dev_malloc(void **p, size_t bytes);
int mcg_cuda_fail(cudaError_t e, const char *what);
#define MCG_TAB_PAD 32 /* a tile reads past its chain's ends (mcg_tiles) */
bool mcg_thick(const mcg_widths &w, int n, bool strict);
cudaError_t mcg_read_tally(mcg_context *ctx, const unsigned long long *d, size_t n, int64_t *h_q,
                           double *h_f64);
/* The tiles' parameters of cell k of n consecutive ones (mcg_tiles): {sig_a, sig_i,
 * length of a flight that enters the cell by its left face, by its right face}, the
 * float differences of the faces that mcg_step_cross forms (entered at a neighbour's
 * face, which between layers of different spacing differs from the cell's own).
 * Lengths outside the range in which the cached-reciprocal division is exact, and
 * those of cells that would amplify the weight, are NaN: such steps take the full
 * form.  sig_i as in the cells: 0 when at most EPS in the fast ones. */
__host__ __device__ inline float4 mcg_tile_entry(const float4 *c, int n, int k)
{
  const float4 p = c[k];
  const float l = p.w - (k ? c[k - 1].w : p.z), r = (k + 1 < n ? c[k + 1].z : p.w) - p.z;
  return make_float4(p.x, p.y, l >= 0x1p-90f && l <= 0x1p90f && p.x >= 0.0f ? l : NAN,
                     r >= 0x1p-90f && r <= 0x1p90f && p.x >= 0.0f ? r : NAN);
}
void mcg_tile_table(const float4 *cells_fast, int n, float4 *tab);
void mcg_cell_params(float sig, float rate, int gi, float dx, float4 &strict, float4 &fast);
int mcg_track_launch(mcg_context *ctx, mcg_particle *d_particles, int64_t n, int32_t *d_results,
                     int64_t *d_steps, int64_t *d_scatters, const mcg_source *src, int64_t first);
int mcg_sync(mcg_context *ctx);
void mcg_ext_destroy(mcg_context *ctx);
int mcg_load_libm(mcg_context *ctx);
extern "C" int mcg_fit_release(mcg_context *ctx);
struct mcg_track_params;
/* Below this many live particles (once the source is exhausted) the event
 * engine finishes the run with one history-based launch. */
inline unsigned long long mcg_event_drain_below(const mcg_context *ctx)
{
  return (unsigned long long)ctx->sm_count * 1024;
}
/* The strict thin-cell step applies (mcg_step THIN, the workers' cycles): every
 * cell's sig_a width is at most 5e-4, so that a crossing has |sig_a d_edge| >=
 * MCG_EXP_SMALL_T only for |mu| < 0.093, under 1 % of the crossings, and
 * exception-table thresholds small enough for its test on |yl| (that test implies
 * the midpoint-distance test for thresholds below 0.4; the tables' are about
 * 0.002).  Not the tiles' line: each step tests its own argument. */
inline bool mcg_strict_thin(const mcg_context *ctx)
{
  return ctx->thin_step && ctx->libm.tau_exp_max < 0.25f;
}
int mcg_event_run(mcg_context *ctx, mcg_track_params &P);
int mcg_event_run_slabs(mcg_context *ctx, const float4 *cells, unsigned long long *tally,
                        const void *slabs, const unsigned long long *slab_hist0, int n_slabs,
                        unsigned long long total, float min_w, int steps_per_pass);

#endif
