/*
 * mcg_batch.cu - thousands of independent slabs of uneven size in one
 * persistent launch (the batched form of the tracker).
 *
 * Work is cut into items: up to `item_histories` consecutive histories of
 * one slab (fewer in small runs, build_items).  Items are sorted by expected
 * cost (histories x cells, largest first) and handed out through one global
 * counter.  A block works on one item at a time, its warps taking the item's
 * histories from a block-local counter and running them as the single-chain
 * tracker does (mcg_histories, mcg_track.cuh).  When the histories are handed
 * out, the block changes to the next item at once: if that is another slab's it
 * flushes its shared-memory tally to the slab's global tally and zeroes it
 * (at most max_cells 64-bit counters, 32 KB for 4096 cells), and the histories
 * its warps still hold go on in their lanes and add to the global tally.
 * Waiting for them instead, an item's end cost its block up to 3 ms (the
 * longest of its histories): 4096 slabs of up to 50,000 histories, strict,
 * took 285 ms with that, 278 without, 36 more of it per halving of the items.
 * Issue-bound (75 % of the slots; 4.65 warp instructions per step and lane, 40 %
 * in forming the steps, 20 % in the deposits, 16 % in full steps), then the
 * loads of the 136 MB step table through L2.  Whole run: 410 -> 206 ms strict,
 * 247 -> 155 ms fast.
 *
 * Short and thick slabs, whose histories take a few steps or end their flights
 * at every other one, go to a second kernel with a lane per history
 * (mcg_batch_lanes): 2000 slabs of 16 to 64 cells of width .5 (2000 histories each)
 * strict 6.8 ms by tiles, 3.2 so, fast 5.1 and 1.5; of width 1e-4 2.0 and .77.
 */
#include <algorithm>
#include <new>
#include <cmath>
#include <cstring>
#include <vector>

/* A warp whose lanes need both exp paths takes the general one for all: it
 * returns the small-argument path's bits wherever that applies.  Measured on
 * the batched kernels: about 0.5-1 % faster; on the single-chain tracker, whose
 * crossings almost all take the small path, 3 % slower, so it keeps the
 * per-lane choice. */
#define MCG_EXP_UNIFORM
#include "mcg_internal.h"
#include "mcg_batch.cuh"

template <bool STRICT, int TALLY>
__global__ void __launch_bounds__(1024) mcg_batch_kernel(mcg_batch_params P)
{
  mcg_batch_body<STRICT, TALLY, false>(P);
}

template <bool STRICT, int TALLY>
__global__ void __launch_bounds__(MCG_LANES_BLOCK, 4) mcg_batch_lanes_kernel(mcg_batch_params P)
{
  mcg_batch_lanes_body<STRICT, TALLY, false>(P);
}

/* ------------------------------------------------------------ host side */
static mcg_batch_state *batch_of(mcg_context *ctx)
{
  if (!ctx->ext)
    ctx->ext = new mcg_ext();
  return &ctx->ext->batch;
}

static void batch_free(mcg_batch_state *B)
{
  for (void *p : {B->d_slabs, B->d_items, (void *)B->d_cells_strict, (void *)B->d_cells_fast,
                  (void *)B->d_tab,
                  (void *)B->d_tally, (void *)B->d_item_next, (void *)B->d_hist0})
    if (p)
      cudaFree(p);
  if (B->graph)
    cudaGraphExecDestroy(B->graph);
  if (B->side)
    cudaStreamDestroy(B->side);
  for (cudaEvent_t ev : {B->fork, B->join})
    if (ev)
      cudaEventDestroy(ev);
  *B = mcg_batch_state();
}

void mcg_adjoint_release(mcg_adj_state *A);

void mcg_ext_destroy(mcg_context *ctx)
{
  if (!ctx->ext)
    return;
  batch_free(&ctx->ext->batch);
  mcg_adjoint_release(&ctx->ext->adj);
  if (ctx->ext->worker.dev)
    cudaFree(ctx->ext->worker.dev);
  if (ctx->ext->worker.monitor)
    cudaStreamDestroy(ctx->ext->worker.monitor);
  delete ctx->ext;
  ctx->ext = nullptr;
}

/* The fast arithmetic's cells (mcg_cell_params) and the tile table
 * (mcg_tile_entry: within a slab neighbours share their faces) from the strict
 * cells, on the GPU: uploading all three took 27 ms longer for 8.5e6 cells. */
__global__ void mcg_batch_tables(const float4 *strict, float4 *fast, float4 *tab, int64_t n)
{
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    const float4 c = strict[k];
    fast[k] = make_float4(c.x, c.y > 1e-4f ? c.y : 0.0f, c.z, c.w);
    tab[k] = mcg_tile_cell(fast[k]);
  }
}

/* Slabs whose histories take a lane each: up to 100 cells, and thick ones.  Batches
 * of up to 3000 slabs, tiles / lanes, strict: 20 cells of width .005 in both sections
 * 1.8 times, 40 1.2, 80 .8 (3000 histories each) to 2.4 (100,000), 160 .8, 320 .5; 80
 * cells of .1 and .01 3.3, 320 2.4; 320 of .05 1.2, of .02 .7; 200 to 800 of .03 .93.
 * Fast: 80 cells of .005 .8 to 3.1, 160 .7, 320 .5; 320 of .05 .7, of .1 1.0, of .01
 * and .5 2.4. */
bool mcg_batch_lanes(const mcg_widths &w, int n, bool strict)
{
  return n <= 100 || (strict ? w.a > 0.04 * n || w.i > 0.25 * n : w.a + w.i > 0.15 * n);
}

extern "C" int mcg_batch_set(mcg_context *ctx, int32_t n_slabs, const mcg_slab *h_slabs,
                             const float *h_sigs, const float *h_rates, float particle_min_weight)
{
  if (!ctx || n_slabs <= 0 || !h_slabs || !h_sigs || !h_rates)
    return mcg_fail(MCG_ERR_ARG, "mcg_batch_set: bad arguments");
  int64_t total = 0, hist = 0;
  int maxc = 0;
  for (int s = 0; s < n_slabs; ++s) {
    const mcg_slab &sl = h_slabs[s];
    if (sl.n_cells <= 0 || sl.n_histories < 0 || sl.seed_mode < 0 || sl.seed_mode > 1 ||
        sl.isotropic < 0 || sl.isotropic > 2)
      return mcg_fail(MCG_ERR_ARG, "mcg_batch_set: bad slab %d", s);
    total += sl.n_cells;
    hist += sl.n_histories;
    maxc = std::max(maxc, sl.n_cells);
  }
  /* the largest slab whose tally fits in a block's shared memory */
  const size_t smem_need = sizeof(mcg_libm_tab) + 16 * 8 + 4 * 8 + (size_t)maxc * 8;
  if (total > INT32_MAX || smem_need > (size_t)ctx->smem_optin)
    return mcg_fail(MCG_ERR_ARG, "mcg_batch_set: %lld cells / largest slab %d cells too large",
                    (long long)total, maxc);
  std::vector<float4> cs;
  std::vector<mcg_batch_slab_dev> sd;
  try {
    cs.resize(total);
    sd.resize(n_slabs);
  } catch (const std::bad_alloc &) {
    return mcg_fail(MCG_ERR_ARG, "mcg_batch_set: no host memory for %lld cells", (long long)total);
  }
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  mcg_batch_state *B = batch_of(ctx);
  const int keep_block = B->block, keep_tm = B->tally_mode;
  const int keep_defer = B->defer;
  const int64_t keep_item = B->item_histories;
  batch_free(B);
  B->block = keep_block;
  B->tally_mode = keep_tm;
  B->defer = keep_defer;
  B->item_histories = keep_item;
  B->n_slabs = n_slabs;
  B->total_cells = (int)total;
  B->max_cells = maxc;
  B->total_histories = hist;
  B->min_w = particle_min_weight;
  B->slabs.assign(h_slabs, h_slabs + n_slabs);
  B->cell_off.resize(n_slabs);
  B->slab_lanes.resize(n_slabs);
  int64_t off = 0;
  for (int s = 0; s < n_slabs; ++s) {
    const mcg_slab &sl = h_slabs[s];
    B->cell_off[s] = (int32_t)off;
    const float dx = (1.0f - 0.0f) / (float)sl.n_cells; /* Layer(0, 1, 0, m): src/layer.cpp:47 */
    float4 fast;
    mcg_widths widths;
    for (int j = 0; j < sl.n_cells; ++j) {
      mcg_cell_params(h_sigs[off + j], h_rates[off + j], j, dx, cs[off + j], fast);
      widths.add(cs[off + j]);
    }
    sd[s].cell_off = (int32_t)off;
    sd[s].m = sl.n_cells;
    sd[s].n_hist = sl.n_histories;
    sd[s].src.seed_mode = sl.seed_mode;
    sd[s].src.isotropic = sl.isotropic;
    sd[s].src.base_seed = sl.base_seed;
    sd[s].src.x0 = 0.0f;
    sd[s].src.mu0 = sl.mu0;
    sd[s].src.w0 = sl.w0;
    sd[s].src.cell0 = 0;
    B->slab_lanes[s] = (mcg_batch_lanes(widths, sl.n_cells, true) ? 1 : 0) |
                       (mcg_batch_lanes(widths, sl.n_cells, false) ? 2 : 0) |
                       (mcg_thick(widths, sl.n_cells, true) ? 4 : 0) |
                       (mcg_thick(widths, sl.n_cells, false) ? 8 : 0);
    off += sl.n_cells;
  }
  /* any failure from here on leaves no slabs set (launches return
   * MCG_ERR_STATE), with the launch shape kept */
  auto fail = [&](cudaError_t err, const char *what) {
    batch_free(B);
    B->block = keep_block;
    B->tally_mode = keep_tm;
    B->defer = keep_defer;
    B->item_histories = keep_item;
    return mcg_cuda_fail(err, what);
  };
  cudaError_t e;
  if ((e = mcg_dev_malloc((void **)&B->d_cells_strict, total * sizeof(float4))) != cudaSuccess ||
      (e = mcg_dev_malloc((void **)&B->d_cells_fast, total * sizeof(float4))) != cudaSuccess ||
      (e = mcg_dev_malloc((void **)&B->d_tab, (total + 2 * MCG_TAB_PAD) * sizeof(float4))) != cudaSuccess ||
      (e = mcg_dev_malloc((void **)&B->d_tally, total * sizeof(unsigned long long))) != cudaSuccess ||
      (e = mcg_dev_malloc(&B->d_slabs, n_slabs * sizeof(mcg_batch_slab_dev))) != cudaSuccess ||
      (e = mcg_dev_malloc((void **)&B->d_item_next, 64)) != cudaSuccess)
    return fail(e, "mcg_batch_set: cudaMalloc");
  if ((e = cudaMemcpy(B->d_cells_strict, cs.data(), total * sizeof(float4), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemset(B->d_tab, 0, (total + 2 * MCG_TAB_PAD) * sizeof(float4))) != cudaSuccess ||
      (e = cudaMemcpy(B->d_slabs, sd.data(), n_slabs * sizeof(mcg_batch_slab_dev), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemset(B->d_tally, 0, total * sizeof(unsigned long long))) != cudaSuccess)
    return fail(e, "mcg_batch_set: upload");
  mcg_batch_tables<<<(int)std::min<int64_t>((total + 255) / 256, 8LL * ctx->sm_count), 256>>>(
      B->d_cells_strict, B->d_cells_fast, B->d_tab + MCG_TAB_PAD, total);
  if ((e = cudaGetLastError()) != cudaSuccess || (e = cudaStreamSynchronize(0)) != cudaSuccess)
    return fail(e, "mcg_batch_set: tables");
  return mcg_tally_reset(ctx) == MCG_OK ? MCG_OK : MCG_ERR_CUDA;
}

/* Items of at most `item` histories, sorted by expected cost, optionally only
 * the first `fraction` of every slab's histories (autotuner samples).  An item
 * is also at most a sixteenth of a block's even share of the run (cost: histories
 * x cells), so a small run still has an item for every block and the last ones
 * are short: 37 slabs of up to 20,000 histories took 34 ms with the 40 items
 * that 16,384 histories make of them.  Not below 64 histories (512 for a lane
 * each, two rounds of a block): each item loads and adds its slab's tally.  The
 * items of the second kernel come last, and there are none unless they are a tenth
 * of the work: 37 slabs with three of them took 4 % longer in two launches. */
static int build_items(mcg_context *ctx, mcg_batch_state *B, int64_t item, double fraction, int grid)
{
  std::vector<mcg_batch_item> items;
  std::vector<double> cost;
  const bool strict = ctx->mode == MCG_MODE_STRICT;
  auto histories = [&](int s) {
    const int64_t n = B->slabs[s].n_histories;
    return fraction < 1.0 ? std::max<int64_t>(std::min<int64_t>(n, 32), (int64_t)std::ceil(n * fraction))
                          : n;
  };
  double total = 0.0, by_lanes = 0.0;
  for (int s = 0; s < B->n_slabs; ++s) {
    total += (double)histories(s) * B->slabs[s].n_cells;
    if (B->slab_lanes[s] & (strict ? 1 : 2))
      by_lanes += (double)histories(s) * B->slabs[s].n_cells;
  }
  const bool mixed = by_lanes > 0.1 * total;
  for (int s = 0; s < B->n_slabs; ++s) {
    const int64_t n = histories(s);
    const int64_t share = (int64_t)(total / (16.0 * grid) / B->slabs[s].n_cells);
    const bool lanes = mixed && (B->slab_lanes[s] & (strict ? 1 : 2));
    const int64_t step = std::min(item, std::max<int64_t>(lanes ? 512 : 64, share));
    for (int64_t f = 0; f < n; f += step) {
      mcg_batch_item it;
      it.slab = s;
      it.lanes = lanes;
      it.sum = 0;
      it.first = f;
      it.count = std::min(step, n - f);
      items.push_back(it);
      cost.push_back((double)it.count * (double)B->slabs[s].n_cells);
    }
  }
  std::vector<size_t> order(items.size());
  for (size_t i = 0; i < order.size(); ++i)
    order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) {
    return items[a].lanes != items[b].lanes ? items[a].lanes < items[b].lanes : cost[a] > cost[b];
  });
  std::vector<mcg_batch_item> sorted(items.size());
  for (size_t i = 0; i < order.size(); ++i)
    sorted[i] = items[order[i]];
  if ((int)sorted.size() > B->items_cap) {
    if (B->d_items)
      cudaFree(B->d_items);
    B->d_items = nullptr;
    cudaError_t e = cudaMalloc(&B->d_items, sorted.size() * sizeof(mcg_batch_item));
    if (e != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_batch: cudaMalloc(items)");
    B->items_cap = (int)sorted.size();
  }
  cudaError_t e = cudaMemcpy(B->d_items, sorted.data(), sorted.size() * sizeof(mcg_batch_item),
                             cudaMemcpyHostToDevice);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_batch: upload items");
  B->lane_cells = 0;
  for (int s = 0; s < B->n_slabs; ++s)
    if (B->slab_lanes[s] & (strict ? 1 : 2))
      B->lane_cells = std::max(B->lane_cells, B->slabs[s].n_cells);
  B->n_items = (int)sorted.size();
  B->n_tiled = (int)std::count_if(sorted.begin(), sorted.end(),
                                  [](const mcg_batch_item &it) { return !it.lanes; });
  B->items_built_for = item;
  B->items_strict = strict;
  B->items_grid = grid;
  B->items_fraction = fraction;
  B->graph_valid = false;
  return MCG_OK;
}

struct mcg_batch_launch {
  void (*kern)(mcg_batch_params);
  mcg_batch_params P;
  size_t smem;
  int grid, block;
  /* the items that take a lane per history, beside the others */
  void (*lanes_kern)(mcg_batch_params);
  mcg_batch_params lanes;
  size_t lanes_smem;
  int lanes_grid;
};

/* Lanes waiting for the full step that trigger it (mcg_batch_set_deferral 0):
 * 4 to 12 lie within 2 % on 4096 slabs of up to 4096 cells, 4 is 13 % faster
 * than 8 on 37 small ones. */
#define MCG_BATCH_POOL 4

/* Kernel choice, attributes, grid and items (of `fraction` of the histories):
 * done outside any stream capture. */
static int batch_configure(mcg_context *ctx, mcg_batch_state *B, int64_t item, double fraction,
                           mcg_batch_launch &L)
{
  const bool strict = ctx->mode == MCG_MODE_STRICT;
  mcg_batch_params &P = L.P;
  memset(&P, 0, sizeof(P));
  P.cells = strict ? B->d_cells_strict : B->d_cells_fast;
  P.tab = B->d_tab + MCG_TAB_PAD;
  P.slabs = static_cast<const mcg_batch_slab_dev *>(B->d_slabs);
  P.max_cells = B->max_cells;
  P.item_next = B->d_item_next;
  P.tally = B->d_tally;
  P.counters = ctx->d_counters;
  P.libm = ctx->libm;
  P.libm_tab = ctx->libm_tab;
  P.rules = mcg_rules_setup(ctx, B->min_w);
  P.rules.pool_lanes = B->defer ? B->defer : MCG_BATCH_POOL;
  /* the asked block, or a smaller one where the largest slab's tally and the
   * warps' tiles would not fit; the global tally where none does.  Both
   * shared-memory modes add 64 bits at once (mcg_shared_red_if). */
  int tm = B->tally_mode;
  if (mcg_batch_smem(B->max_cells, 256, true, false) > (size_t)ctx->smem_optin)
    tm = MCG_TALLY_GLOBAL;
  L.block = B->block;
  while (L.block > 256 && mcg_batch_smem(B->max_cells, L.block, tm != MCG_TALLY_GLOBAL, false) > (size_t)ctx->smem_optin)
    L.block /= 2;
  L.smem = mcg_batch_smem(B->max_cells, L.block, tm != MCG_TALLY_GLOBAL, false);
  if (strict)
    L.kern = tm == MCG_TALLY_GLOBAL ? mcg_batch_kernel<true, MCG_TALLY_GLOBAL>
                                    : mcg_batch_kernel<true, MCG_TALLY_SMEM64>;
  else
    L.kern = tm == MCG_TALLY_GLOBAL ? mcg_batch_kernel<false, MCG_TALLY_GLOBAL>
                                    : mcg_batch_kernel<false, MCG_TALLY_SMEM64>;
  /* the opt-in maximum on every call (mcg_track_launch) */
  cudaError_t e = cudaFuncSetAttribute(L.kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       ctx->smem_optin);
  int bps = 0;
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, L.kern, L.block, L.smem);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_batch: launch set-up");
  L.grid = ctx->sm_count * std::max(bps, 1);
  if (B->items_built_for != item || B->items_grid != L.grid || B->items_fraction != fraction ||
      B->items_strict != strict) {
    int rc = build_items(ctx, B, item, fraction, L.grid);
    if (rc != MCG_OK)
      return rc;
  }
  P.items = static_cast<const mcg_batch_item *>(B->d_items);
  P.n_items = B->n_tiled;
  L.lanes = P;
  L.lanes.items = P.items + B->n_tiled;
  L.lanes.n_items = B->n_items - B->n_tiled;
  L.lanes.item_next = P.item_next + 1;
  if (L.lanes.n_items == 0)
    return MCG_OK;
  const bool global = B->tally_mode == MCG_TALLY_GLOBAL ||
                      mcg_batch_lanes_smem(B->lane_cells, true) > (size_t)ctx->smem_optin;
  L.lanes_smem = mcg_batch_lanes_smem(B->lane_cells, !global);
  if (strict)
    L.lanes_kern = global ? mcg_batch_lanes_kernel<true, MCG_TALLY_GLOBAL>
                          : mcg_batch_lanes_kernel<true, MCG_TALLY_SMEM32>;
  else
    L.lanes_kern = global ? mcg_batch_lanes_kernel<false, MCG_TALLY_GLOBAL>
                          : mcg_batch_lanes_kernel<false, MCG_TALLY_SMEM32>;
  e = cudaFuncSetAttribute(L.lanes_kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, L.lanes_kern, MCG_LANES_BLOCK, L.lanes_smem);
  if (e == cudaSuccess && !B->side)
    e = cudaStreamCreateWithFlags(&B->side, cudaStreamNonBlocking);
  for (cudaEvent_t *ev : {&B->fork, &B->join})
    if (e == cudaSuccess && !*ev)
      e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_batch: launch set-up");
  L.lanes_grid = std::min(ctx->sm_count * std::max(bps, 1), L.lanes.n_items);
  return MCG_OK;
}

/* The two kernels side by side: the lane form's blocks come first, the others fill
 * the SMs that those leave. */
static int batch_enqueue(mcg_context *ctx, mcg_batch_state *B, const mcg_batch_launch &L)
{
  cudaError_t e = cudaMemsetAsync(B->d_item_next, 0, 16, ctx->stream);
  if (L.lanes.n_items) {
    const bool beside = L.P.n_items > 0;
    cudaStream_t st = beside ? B->side : ctx->stream;
    if (e == cudaSuccess && beside && (e = cudaEventRecord(B->fork, ctx->stream)) == cudaSuccess)
      e = cudaStreamWaitEvent(st, B->fork, 0);
    if (e == cudaSuccess) {
      L.lanes_kern<<<L.lanes_grid, MCG_LANES_BLOCK, L.lanes_smem, st>>>(L.lanes);
      e = cudaGetLastError();
      ctx->last_grid = L.lanes_grid;
      ctx->last_block = MCG_LANES_BLOCK;
      ctx->launches++;
    }
    if (e == cudaSuccess && beside)
      e = cudaEventRecord(B->join, st);
  }
  if (e == cudaSuccess && L.P.n_items) {
    L.kern<<<L.grid, L.block, L.smem, ctx->stream>>>(L.P);
    e = cudaGetLastError();
    ctx->last_grid = L.grid;
    ctx->last_block = L.block;
    ctx->launches++;
    if (e == cudaSuccess && L.lanes.n_items)
      e = cudaStreamWaitEvent(ctx->stream, B->join, 0);
  }
  return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(e, "mcg_batch_kernel launch");
}

/* First history of each slab for the event engine, with the same sampled
 * history counts as build_items at this fraction; returns the total. */
static int build_hist0(mcg_batch_state *B, double fraction, unsigned long long *total)
{
  std::vector<unsigned long long> h0(B->n_slabs);
  unsigned long long t = 0;
  for (int s = 0; s < B->n_slabs; ++s) {
    int64_t n = B->slabs[s].n_histories;
    if (fraction < 1.0)
      n = std::max<int64_t>(std::min<int64_t>(n, 32), (int64_t)std::ceil(n * fraction));
    h0[s] = t;
    t += (unsigned long long)n;
  }
  *total = t;
  if (B->hist0_fraction == fraction && B->d_hist0)
    return MCG_OK;
  cudaError_t e = cudaSuccess;
  if (!B->d_hist0)
    e = cudaMalloc(&B->d_hist0, (size_t)B->n_slabs * sizeof(unsigned long long));
  if (e == cudaSuccess)
    e = cudaMemcpy(B->d_hist0, h0.data(), h0.size() * sizeof(unsigned long long),
                   cudaMemcpyHostToDevice);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_batch: slab history offsets");
  B->hist0_fraction = fraction;
  return MCG_OK;
}

/* One batched run with the event engine (histories at this fraction). */
static int batch_run_event(mcg_context *ctx, mcg_batch_state *B, double fraction, int steps)
{
  unsigned long long total = 0;
  int rc = build_hist0(B, fraction, &total);
  if (rc != MCG_OK)
    return rc;
  const bool strict = ctx->mode == MCG_MODE_STRICT;
  return mcg_event_run_slabs(ctx, strict ? B->d_cells_strict : B->d_cells_fast, B->d_tally,
                             B->d_slabs, B->d_hist0, B->n_slabs, total, B->min_w, steps);
}

static int batch_prepare(mcg_context *ctx, mcg_batch_state **out)
{
  if (!ctx || !ctx->ext || ctx->ext->batch.n_slabs == 0)
    return mcg_fail(MCG_ERR_STATE, "mcg_batch: no slabs set (mcg_batch_set)");
  int rc = MCG_OK;
  if (ctx->mode == MCG_MODE_STRICT && !ctx->libm_loaded)
    rc = mcg_load_libm(ctx);
  cudaSetDevice(ctx->device);
  *out = &ctx->ext->batch;
  return rc;
}

extern "C" int mcg_batch_run(mcg_context *ctx)
{
  mcg_batch_state *B;
  int rc = batch_prepare(ctx, &B);
  if (rc != MCG_OK)
    return rc;
  if (B->algorithm == MCG_ALGO_EVENT) {
    if ((rc = batch_run_event(ctx, B, 1.0, B->event_steps)) != MCG_OK)
      return rc;
    return mcg_sync(ctx);
  }
  cudaError_t e;
  /* mcg_set_mode, _tally_scale, _launch and _step_limit leave the graph alone */
  if (!B->graph_valid || B->graph_mode != ctx->mode || B->graph_scale != ctx->log2_scale ||
      B->graph_refill != ctx->refill || B->graph_steps != ctx->max_steps) {
    B->graph_valid = false;
    if (B->graph) {
      cudaGraphExecDestroy(B->graph);
      B->graph = nullptr;
    }
    mcg_batch_launch L;
    if ((rc = batch_configure(ctx, B, B->item_histories, 1.0, L)) != MCG_OK)
      return rc;
    cudaGraph_t g;
    if ((e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_batch_run: begin capture");
    rc = batch_enqueue(ctx, B, L);
    e = cudaStreamEndCapture(ctx->stream, &g);
    if (rc != MCG_OK)
      return rc;
    if (e != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_batch_run: end capture");
    e = cudaGraphInstantiate(&B->graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_batch_run: instantiate");
    B->graph_mode = ctx->mode;
    B->graph_scale = ctx->log2_scale;
    B->graph_refill = ctx->refill;
    B->graph_steps = ctx->max_steps;
    B->graph_valid = true;
  }
  cudaEventRecord(ctx->ev0, ctx->stream);
  e = cudaGraphLaunch(B->graph, ctx->stream);
  cudaEventRecord(ctx->ev1, ctx->stream);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_batch_run: graph launch");
  return mcg_sync(ctx);
}

extern "C" int mcg_batch_run_per_slab(mcg_context *ctx)
{
  mcg_batch_state *B;
  int rc = batch_prepare(ctx, &B);
  if (rc != MCG_OK)
    return rc;
  const bool strict = ctx->mode == MCG_MODE_STRICT;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  cudaEventRecord(a, ctx->stream);
  for (int s = 0; s < B->n_slabs && rc == MCG_OK; ++s) {
    const mcg_slab &sl = B->slabs[s];
    if (sl.n_histories == 0)
      continue;
    mcg_track_params P;
    memset(&P, 0, sizeof(P));
    P.cells = (strict ? B->d_cells_strict : B->d_cells_fast) + B->cell_off[s];
    P.tab = {B->d_tab + MCG_TAB_PAD + B->cell_off[s], nullptr, 0};
    P.n_cells = sl.n_cells;
    P.cell_lo = 0;
    P.n = sl.n_histories;
    P.src.seed_mode = sl.seed_mode;
    P.src.isotropic = sl.isotropic;
    P.src.base_seed = sl.base_seed;
    P.src.mu0 = sl.mu0;
    P.src.w0 = sl.w0;
    P.next = ctx->d_next;
    P.tally = B->d_tally + B->cell_off[s];
    P.counters = ctx->d_counters;
    P.libm = ctx->libm;
    P.libm_tab = ctx->libm_tab;
    P.rules = mcg_rules_setup(ctx, B->min_w);
    const mcg_shape shape = mcg_track_shape(sl.n_cells, 0, false, false, (size_t)ctx->smem_optin);
    const int block = shape.block;
    const size_t smem = shape.smem;
    P.tally_copies = shape.copies;
    const bool lanes = B->slab_lanes[s] & (strict ? 4 : 8);
    void (*kern)(mcg_track_params);
    if (lanes)
      kern = strict ? (shape.global ? mcg_track_kernel<true, MCG_TALLY_GLOBAL, false, true>
                                    : mcg_track_kernel<true, MCG_TALLY_SMEM32, false, true>)
                    : (shape.global ? mcg_track_kernel<false, MCG_TALLY_GLOBAL, false, true>
                                    : mcg_track_kernel<false, MCG_TALLY_SMEM32, false, true>);
    else
      kern = strict ? (shape.global ? mcg_track_kernel<true, MCG_TALLY_GLOBAL, false>
                                    : mcg_track_kernel<true, MCG_TALLY_SMEM32, false>)
                    : (shape.global ? mcg_track_kernel<false, MCG_TALLY_GLOBAL, false>
                                    : mcg_track_kernel<false, MCG_TALLY_SMEM32, false>);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         ctx->smem_optin);
    int bps = 1;
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, block, smem);
    const int grid = mcg_track_grid(ctx->sm_count * std::max(bps, 1), block, sl.n_histories, lanes, P);
    if (e == cudaSuccess)
      e = cudaMemsetAsync(ctx->d_next, 0, 8, ctx->stream);
    if (e == cudaSuccess) {
      kern<<<grid, block, smem, ctx->stream>>>(P);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess)
      rc = mcg_cuda_fail(e, "mcg_batch_run_per_slab");
    ctx->launches++;
  }
  cudaEventRecord(b, ctx->stream);
  cudaError_t e = cudaStreamSynchronize(ctx->stream);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (rc != MCG_OK)
    return rc;
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_batch_run_per_slab: execution");
  rc = mcg_sync(ctx);
  ctx->last_ms = ms;
  return rc;
}

extern "C" int mcg_batch_tally_reset(mcg_context *ctx)
{
  mcg_batch_state *B;
  int rc = batch_prepare(ctx, &B);
  if (rc != MCG_OK)
    return rc;
  cudaError_t e = cudaMemsetAsync(B->d_tally, 0, B->total_cells * sizeof(unsigned long long),
                                  ctx->stream);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_batch_tally_reset");
  return mcg_tally_reset(ctx);
}

extern "C" int mcg_batch_tally_read(mcg_context *ctx, int64_t *h_q, double *h_f64)
{
  mcg_batch_state *B;
  int rc = batch_prepare(ctx, &B);
  if (rc != MCG_OK)
    return rc;
  cudaError_t e = mcg_read_tally(ctx, B->d_tally, (size_t)B->total_cells, h_q, h_f64);
  return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(e, "mcg_batch_tally_read");
}

extern "C" int mcg_batch_set_launch(mcg_context *ctx, int32_t block, int64_t item_histories,
                                    int32_t tally_mode)
{
  if (!ctx || (block && block != 256 && block != 512 && block != 1024) || item_histories < 0 ||
      tally_mode < -1 || tally_mode > 2)
    return mcg_fail(MCG_ERR_ARG, "mcg_batch_set_launch: bad arguments");
  mcg_batch_state *B = batch_of(ctx);
  if (block)
    B->block = block;
  if (item_histories)
    B->item_histories = item_histories;
  if (tally_mode >= 0)
    B->tally_mode = tally_mode;
  B->graph_valid = false;
  return MCG_OK;
}

extern "C" int mcg_batch_set_deferral(mcg_context *ctx, int32_t defer)
{
  if (!ctx || defer < 0 || defer > 32)
    return mcg_fail(MCG_ERR_ARG, "mcg_batch_set_deferral: bad arguments");
  mcg_batch_state *B = batch_of(ctx);
  B->defer = defer;
  B->graph_valid = false;
  return MCG_OK;
}

extern "C" int mcg_batch_set_algorithm(mcg_context *ctx, int32_t algorithm, int32_t steps_per_pass)
{
  if (!ctx || (algorithm != MCG_ALGO_HISTORY && algorithm != MCG_ALGO_EVENT) || steps_per_pass < 0)
    return mcg_fail(MCG_ERR_ARG, "mcg_batch_set_algorithm: bad arguments");
  mcg_batch_state *B = batch_of(ctx);
  B->algorithm = algorithm;
  B->event_steps = steps_per_pass ? steps_per_pass : 8;
  return MCG_OK;
}

extern "C" int mcg_batch_autotune(mcg_context *ctx, double sample_fraction, mcg_batch_tuning *out)
{
  mcg_batch_state *B;
  int rc = batch_prepare(ctx, &B);
  if (rc != MCG_OK)
    return rc;
  if (!(sample_fraction > 0.0 && sample_fraction <= 1.0))
    return mcg_fail(MCG_ERR_ARG, "mcg_batch_autotune: sample fraction must be in (0, 1]");
  const int blocks[] = {256, 512, 1024};
  const int64_t items[] = {4096, 16384, 65536};
  /* tally mode and lanes that wait for the full step */
  const int shapes[][2] = {{MCG_TALLY_SMEM32, 4}, {MCG_TALLY_SMEM32, 12}};
  /* every candidate runs the same sample, of at least four times the event
   * engine's drain size (below it the event-based form is a single drain
   * launch, and a persistent launch is dominated by its tail), or the whole
   * run; candidates compete on time per history */
  unsigned long long n_full = 0, n_hist = 0;
  if ((rc = build_hist0(B, 1.0, &n_full)) != MCG_OK)
    return rc;
  sample_fraction = std::min(
      1.0, std::max(sample_fraction, 4.0 * (double)mcg_event_drain_below(ctx) / (double)n_full));
  if ((rc = build_hist0(B, sample_fraction, &n_hist)) != MCG_OK)
    return rc;
  const double f_event = sample_fraction;
  const unsigned long long n_event = n_hist;
  double best = 1e30; /* ms per history */
  int nc = 0;
  mcg_batch_tuning pick = {B->block, B->tally_mode, B->item_histories, 0.f, 0, MCG_ALGO_HISTORY,
                           0, B->defer};
  bool warmed = false;
  for (int64_t it : items) {
    /* the sample keeps the full run's number of items per slab, so the
     * item-level tail the candidate would see is represented */
    const int64_t sample_item = std::max<int64_t>(32, (int64_t)std::llround(it * sample_fraction));
    for (int bl : blocks)
      for (const auto &sh : shapes) {
        const int tm = sh[0];
        B->block = bl;
        B->tally_mode = tm;
        B->defer = sh[1];
        mcg_batch_launch L;
        if ((rc = batch_configure(ctx, B, sample_item, sample_fraction, L)) != MCG_OK)
          return rc;
        for (int rep = warmed ? 1 : 0; rep < 2; ++rep) { /* the very first run warms up */
          cudaEventRecord(ctx->ev0, ctx->stream);
          if ((rc = batch_enqueue(ctx, B, L)) != MCG_OK)
            return rc;
          cudaEventRecord(ctx->ev1, ctx->stream);
          if ((rc = mcg_sync(ctx)) != MCG_OK)
            return rc;
        }
        warmed = true;
        ++nc;
        if (ctx->last_ms / (double)n_hist < best) {
          best = ctx->last_ms / (double)n_hist;
          pick = {bl, tm, it, ctx->last_ms, 0, MCG_ALGO_HISTORY, 0, sh[1]};
        }
      }
  }
  /* the event-based form */
  for (int k : {4, 16}) {
    for (int rep = 0; rep < 2; ++rep) /* the first run sizes the bank */
      if ((rc = batch_run_event(ctx, B, f_event, k)) != MCG_OK || (rc = mcg_sync(ctx)) != MCG_OK)
        return rc;
    ++nc;
    if (ctx->last_ms / (double)n_event < best) {
      best = ctx->last_ms / (double)n_event;
      pick = {B->block, B->tally_mode, B->item_histories, ctx->last_ms, 0, MCG_ALGO_EVENT, k, 0};
    }
  }
  B->algorithm = pick.algorithm;
  if (pick.algorithm == MCG_ALGO_EVENT)
    B->event_steps = pick.steps_per_pass;
  B->block = pick.block;
  B->tally_mode = pick.tally_mode;
  B->item_histories = pick.item_histories;
  B->defer = pick.defer;
  B->items_built_for = -1;
  B->graph_valid = false;
  pick.candidates = nc;
  if (out)
    *out = pick;
  return mcg_batch_tally_reset(ctx);
}
