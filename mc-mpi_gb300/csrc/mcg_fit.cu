/*
 * mcg_fit.cu - batched inverse fit of per-cell absorption cross sections.
 *
 * Many independent slabs (each a Layer(0, 1, 0, m)) with known scattering
 * cross sections and measured absorption tallies t_c (weight absorbed per
 * history); the fit minimises L = sum over all cells of (a_c - t_c)^2, a_c the
 * simulated tally, over every cell's sig_a by Adam.  One Adam step is:
 *   1. the batched forward pass (tally + G = sum w_c dep of every history) and
 *      the replay of every history from its seed accumulating dG/dsig_a (the
 *      pathwise derivative of mcg_adjoint.cu); the loss weights are
 *      w_c = 2 (a_c - t_c) from the previous step's tally (lagged by one
 *      step, so one set of histories per step suffices);
 *   2. a kernel forming the new weights and the loss from this step's tally;
 *   3. the Adam update of every sig_a, written straight into the step table.
 * The kernels are captured once in a CUDA graph and replayed for every
 * step; each step simulates fresh histories (source indices step * n + i).
 */
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "mcg_internal.h"
#include "mcg_batch.cuh"

struct mcg_fit_params {
  const float4 *cells;  /* fast step table; .x = sig_a, updated by the Adam kernel */
  const float2 *aux;    /* {w_c, unused} */
  const mcg_batch_slab_dev *slabs;
  const mcg_batch_item *items;
  int32_t n_items, max_cells;
  unsigned long long *item_next;
  const float2 *sum; /* the forward pass's losses (mcg_batch_params::loss) */
  double *grad;
  const long long *step;
  float min_w;
  int32_t q_log2, jumps; /* jumps: the seed chain's table fits in shared memory */
  uint32_t max_steps;
};

#define MCG_FIT_ITEM 8192   /* most histories of an item */
#define MCG_FIT_LANES 2048  /* ... of a slab whose histories take a lane each */
#define MCG_FIT_PART (1 << 24) /* most histories between a forward pass and its replay: 128 MB of losses */

/* Forward pass: the batched tracker with the losses.  64 slabs of up to 1024
 * cells, 1e5 histories each: 17.5 ms; 24 ms with a lane per history. */
__global__ void __launch_bounds__(1024) mcg_fit_forward(mcg_batch_params P)
{
  mcg_batch_body<false, MCG_TALLY_SMEM64, true>(P);
}

/* ... and its second kernel, for short and thick slabs (mcg_batch_lanes).  A gradient
 * of 64 slabs of 16 to 64 cells, 50,000 histories each, replay included: width .3
 * 10.1 ms by tiles, 5.6 so, .05 4.5 and 3.9; three such slabs 2.4 and 1.0. */
__global__ void __launch_bounds__(MCG_LANES_BLOCK, 4) mcg_fit_forward_lanes(mcg_batch_params P)
{
  mcg_batch_lanes_body<false, MCG_TALLY_SMEM32, true>(P);
}

/*
 * Replay of every history for dG/dsig_a: rounds, history starts and the reason
 * for a lane per history are those of the adjoint's replay.  Bound: instruction
 * issue, with the float atomics' compare-and-swap loops.  64 slabs of up to 1024
 * cells, 1e5 histories each: 25 ms.  Five Adam steps, with the forward pass that
 * starts them: 337 ms with forward pass and replay in one kernel of full steps,
 * 230 ms so.
 */
__global__ void __launch_bounds__(512, 2) mcg_fit_replay(mcg_fit_params P)
{
  extern __shared__ __align__(16) unsigned char smem[];
  long long *s_ctl = reinterpret_cast<long long *>(smem);
  float *s_g = reinterpret_cast<float *>(s_ctl + 4);
  mcg_chain_jumps *s_chain = reinterpret_cast<mcg_chain_jumps *>(s_g + ((P.max_cells + 1) & ~1));
  const int tid = threadIdx.x;
  const long long step = *P.step;
  int cur = -1, m = 0;
  const float4 *cells = nullptr;
  const float2 *aux = nullptr;
  double *ggrad = nullptr;
  const mcg_libm_dev no_libm = {};
  if (P.jumps)
    mcg_fill_chain_jumps(s_chain);
  auto flush = [&] {
    if (cur >= 0)
      for (int i = tid; i < m; i += blockDim.x)
        if (s_g[i] != 0.0f)
          atomicAdd(&ggrad[i], (double)s_g[i]);
  };
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      s_ctl[0] = (long long)atomicAdd(P.item_next, 1ull);
      s_ctl[1] = 0;
    }
    __syncthreads();
    const long long item = s_ctl[0];
    if (item >= P.n_items)
      break;
    const mcg_batch_item it = P.items[item];
    const mcg_batch_slab_dev &sd = P.slabs[it.slab];
    if (it.slab != cur) {
      flush();
      __syncthreads();
      cur = it.slab;
      m = sd.m;
      cells = P.cells + sd.cell_off;
      aux = P.aux + sd.cell_off;
      ggrad = P.grad + sd.cell_off;
      for (int i = tid; i < m; i += blockDim.x)
        s_g[i] = 0.0f;
      __syncthreads();
    }
    const int64_t src_base = step * sd.n_hist + it.first;
    const float2 *sum = P.sum + it.sum;

    uint64_t seed = 0;
    float x = 0.f, mu = 0.f, wmc = 0.f, inv_mu = 0.f;
    int idx = 0;
    uint32_t nst = 0, nsc = 0;
    float G_hi = 0.f, G_lo = 0.f, P_hi = 0.f, P_lo = 0.f;
    bool active = false, wait = false; /* wait: the lane's step needs the full form */
    mcg_pool pool;
    for (;;) {
      const unsigned need = __ballot_sync(0xffffffffu, !active);
      if (need) {
        const long long my = pool.take(need, reinterpret_cast<unsigned long long *>(&s_ctl[1]), it.count, 32);
        if (!active && my >= 0) {
          if (P.jumps)
            mcg_born(s_chain, sd.src, src_base + my, seed, x, mu, wmc, idx);
          else
            mcg_source_particle(sd.src, src_base + my, seed, x, mu, wmc, idx);
          inv_mu = mcg_flight_rcp(mu);
          nst = 0;
          const float2 g = sum[my];
          G_hi = g.x;
          G_lo = g.y;
          P_hi = P_lo = 0.f;
          active = true;
        }
      }
      if (!__any_sync(0xffffffffu, active))
        break;
      /* a round (the adjoint's replay, mcg_adjoint.cu) */
      auto account = [&](int c, float l, float dep) {
        const float wc = __ldg(&aux[c].x);
        mcg_ff_add(P_hi, P_lo, __fmul_rn(wc, dep));
        const float v_after = __fadd_rn(__fsub_rn(G_hi, P_hi), __fsub_rn(G_lo, P_lo));
        atomicAdd(&s_g[c], l * (wc * wmc - v_after));
        ++nst;
      };
      auto living = [&] {
        return active & (wmc >= P.min_w) & ((unsigned)idx < (unsigned)m) & (nst < P.max_steps);
      };
      auto cross = [&](int most) {
        bool go = living() & !wait;
        for (int j = 0; go & (j < most); ++j) {
          const int c = idx;
          float l, dep;
          if (!mcg_cross<false>(seed, x, mu, wmc, inv_mu, idx, __ldg(cells + c), 0.0f, l, dep)) {
            wait = true;
            go = false;
          } else {
            account(c, l, dep);
            go = living();
          }
        }
        return go;
      };
      auto full = [&] {
        if (wait) {
          const int c = idx;
          float l, dep;
          bool coll;
          mcg_full<false, MCG_TALLY_SMEM32>(seed, x, mu, wmc, inv_mu, idx, nsc, __ldg(cells + c), nullptr,
                                            P.q_log2, nullptr, no_libm, &l, &coll, &dep);
          account(c, l, dep);
          wait = false;
        }
      };
      for (;;) {
        const bool go = cross(MCG_GRAD_WINDOW);
        const unsigned wb = __ballot_sync(0xffffffffu, wait);
        const unsigned gb = __ballot_sync(0xffffffffu, go);
        if (wb && 32 * __popc(wb) >= MCG_GRAD_POOL * __popc(wb | gb)) {
          full();
        } else {
          const unsigned over = __ballot_sync(0xffffffffu, active ? !wait & !go : !pool.drained);
          if (!(wb | gb) || __popc(over) >= MCG_GRAD_REFILL)
            break;
        }
      }
      active &= wait | living();
    }
  }
  flush();
}

/* w_c = 2 (a_c - t_c) from this step's tally, the step's loss, and the
 * accumulators cleared for the next step. */
__global__ void mcg_fit_weights_kernel(int n_cells, const int32_t *cell_slab,
                                       const mcg_batch_slab_dev *slabs, const double *target,
                                       unsigned long long *tally, float2 *aux, double *loss_hist,
                                       const long long *step, int q_log2, int max_steps)
{
  const double inv_scale = ldexp(1.0, -q_log2);
  double part = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n_cells; c += gridDim.x * blockDim.x) {
    const double a = (double)(long long)tally[c] * inv_scale / (double)slabs[cell_slab[c]].n_hist;
    const double d = a - target[c];
    aux[c].x = (float)(2.0 * d);
    part += d * d;
    tally[c] = 0ull;
  }
  for (int o = 16; o > 0; o >>= 1)
    part += __shfl_down_sync(0xffffffffu, part, o);
  const long long s = *step;
  if ((threadIdx.x & 31) == 0 && s < max_steps)
    atomicAdd(&loss_hist[s], part);
}

/* Adam on every sig_a; the new value goes straight into the step table. */
__global__ void mcg_fit_adam_kernel(int n_cells, const int32_t *cell_slab,
                                    const mcg_batch_slab_dev *slabs, double *grad, float *sig_a,
                                    float4 *cells, float4 *tab, float *m1, float *m2, long long *step, float lr,
                                    float b1, float b2, float eps, float sig_min)
{
  const long long t = *step + 1;
  const float c1 = 1.0f - powf(b1, (float)t), c2 = 1.0f - powf(b2, (float)t);
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n_cells; c += gridDim.x * blockDim.x) {
    const float g = (float)(grad[c] / (double)slabs[cell_slab[c]].n_hist);
    grad[c] = 0.0;
    const float a = b1 * m1[c] + (1.0f - b1) * g;
    const float v = b2 * m2[c] + (1.0f - b2) * g * g;
    m1[c] = a;
    m2[c] = v;
    const float s = fmaxf(sig_a[c] - lr * (a / c1) / (sqrtf(v / c2) + eps), sig_min);
    sig_a[c] = s;
    cells[c].x = s;
    tab[c] = mcg_tile_cell(cells[c]);
  }
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x == 0)
    *step = t;
}

/* ------------------------------------------------------------ host side */
/* Items that go through a forward pass and its replay together, the first `tiled`
 * by tiles. */
struct mcg_fit_turn {
  int first, items, tiled;
};

struct mcg_fit_state {
  int n_slabs = 0, n_cells = 0, max_cells = 0, lane_cells = 0, max_steps = 0;
  std::vector<mcg_fit_turn> turns;
  std::vector<int32_t> cell_off;
  void *dev = nullptr; /* one allocation for everything below */
  void *dev_sum = nullptr; /* losses of a turn's histories, forward pass -> replay */
  float4 *cells = nullptr, *tab = nullptr; /* tab: mcg_tile_cell of cells */
  float2 *aux = nullptr;
  mcg_batch_slab_dev *slabs = nullptr;
  mcg_batch_item *items = nullptr;
  int32_t *cell_slab = nullptr;
  double *target = nullptr, *grad = nullptr, *loss_hist = nullptr;
  float *sig_a = nullptr, *m1 = nullptr, *m2 = nullptr;
  unsigned long long *tally = nullptr, *item_next = nullptr;
  long long *step = nullptr;
  float min_w = 0.f;
};

static mcg_fit_state *fit_of(mcg_context *ctx, bool create)
{
  if (!ctx->ext) {
    if (!create)
      return nullptr;
    ctx->ext = new mcg_ext();
  }
  if (!ctx->ext->fit && create)
    ctx->ext->fit = new mcg_fit_state();
  return ctx->ext->fit;
}

extern "C" int mcg_fit_release(mcg_context *ctx)
{
  if (!ctx || !ctx->ext || !ctx->ext->fit)
    return MCG_OK;
  if (ctx->ext->fit->dev)
    cudaFree(ctx->ext->fit->dev);
  if (ctx->ext->fit->dev_sum)
    cudaFree(ctx->ext->fit->dev_sum);
  delete ctx->ext->fit;
  ctx->ext->fit = nullptr;
  return MCG_OK;
}

extern "C" int mcg_fit_set(mcg_context *ctx, int32_t n_slabs, const mcg_slab *h_slabs,
                           const float *h_sig_a0, const float *h_sig_s, const double *h_target,
                           float particle_min_weight, int32_t max_steps)
{
  if (!ctx || n_slabs <= 0 || !h_slabs || !h_sig_a0 || !h_sig_s || !h_target || max_steps <= 0)
    return mcg_fail(MCG_ERR_ARG, "mcg_fit_set: bad arguments");
  cudaSetDevice(ctx->device);
  mcg_fit_release(ctx);
  int total = 0, maxc = 0;
  for (int s = 0; s < n_slabs; ++s) {
    if (h_slabs[s].n_cells <= 0 || h_slabs[s].n_histories <= 0)
      return mcg_fail(MCG_ERR_ARG, "mcg_fit_set: bad slab %d", s);
    total += h_slabs[s].n_cells;
    maxc = std::max(maxc, h_slabs[s].n_cells);
  }
  if (16 * 4 + (size_t)maxc * 12 > (size_t)ctx->smem_optin)
    return mcg_fail(MCG_ERR_ARG, "mcg_fit_set: slab of %d cells too large", maxc);
  /* items, largest first, those with a lane per history last */
  std::vector<mcg_batch_item> items;
  std::vector<uint8_t> lanes(n_slabs);
  double work = 0.0, by_lanes = 0.0;
  for (int s = 0, k = 0; s < n_slabs; ++s) {
    const int m = h_slabs[s].n_cells;
    mcg_widths w;
    for (int j = 0; j < m; ++j, ++k)
      w.add(make_float4(h_sig_a0[k], h_sig_s[k], 0.0f, 1.0f / (float)m));
    lanes[s] = mcg_batch_lanes(w, m, false);
    work += (double)h_slabs[s].n_histories * m;
    by_lanes += lanes[s] ? (double)h_slabs[s].n_histories * m : 0.0;
  }
  int lane_cells = 0;
  for (int s = 0; s < n_slabs; ++s) {
    if (!(by_lanes > 0.1 * work)) /* as in the batch (build_items) */
      lanes[s] = 0;
    lane_cells = std::max(lane_cells, lanes[s] ? h_slabs[s].n_cells : 0);
    const int64_t step = lanes[s] ? MCG_FIT_LANES : MCG_FIT_ITEM;
    for (int64_t f = 0; f < h_slabs[s].n_histories; f += step)
      items.push_back({s, lanes[s], f, std::min(step, h_slabs[s].n_histories - f), 0});
  }
  std::stable_sort(items.begin(), items.end(), [&](const mcg_batch_item &a, const mcg_batch_item &b) {
    return a.lanes != b.lanes ? a.lanes < b.lanes
                              : a.count * h_slabs[a.slab].n_cells > b.count * h_slabs[b.slab].n_cells;
  });
  /* carve one allocation */
  size_t off = 0;
  auto take = [&](size_t bytes) { size_t o = off; off += (bytes + 255) & ~(size_t)255; return o; };
  const size_t padded = total + 2 * (size_t)MCG_TAB_PAD; /* the tiles read past the ends */
  const size_t o_cells = take(total * sizeof(float4)), o_aux = take(padded * sizeof(float2));
  const size_t o_tab = take(padded * sizeof(float4));
  const size_t o_slabs = take(n_slabs * sizeof(mcg_batch_slab_dev));
  const size_t o_items = take(items.size() * sizeof(mcg_batch_item));
  const size_t o_cs = take(total * 4), o_t = take(total * 8), o_g = take(total * 8);
  const size_t o_lh = take(max_steps * 8), o_sa = take(total * 4), o_m1 = take(total * 4);
  const size_t o_m2 = take(total * 4), o_ta = take(total * 8), o_in = take(24), o_st = take(8);
  mcg_fit_state *F = fit_of(ctx, true);
  /* a failure from here on leaves no fit set and nothing allocated */
  auto fail = [&](cudaError_t err, const char *what) {
    mcg_fit_release(ctx);
    return mcg_cuda_fail(err, what);
  };
  cudaError_t e = mcg_dev_malloc(&F->dev, off);
  if (e != cudaSuccess)
    return fail(e, "mcg_fit_set: cudaMalloc");
  /* turns of as many histories as there is memory for, at least one item each */
  int64_t most = 0, all = 0;
  for (const mcg_batch_item &it : items) {
    most = std::max(most, it.count);
    all += it.count;
  }
  int64_t part = std::max<int64_t>(most, std::min<int64_t>(all, MCG_FIT_PART));
  while ((e = mcg_dev_malloc(&F->dev_sum, (size_t)part * sizeof(float2))) != cudaSuccess) {
    cudaGetLastError();
    F->dev_sum = nullptr;
    if (part == most)
      return fail(e, "mcg_fit_set: cudaMalloc");
    part = std::max(most, part / 2);
  }
  int64_t at = part;
  for (int i = 0; i < (int)items.size(); ++i) {
    if (at + items[i].count > part) {
      F->turns.push_back({i, 0, 0});
      at = 0;
    }
    items[i].sum = at;
    at += items[i].count;
    F->turns.back().items++;
    F->turns.back().tiled += !items[i].lanes;
  }
  char *b = static_cast<char *>(F->dev);
  F->cells = reinterpret_cast<float4 *>(b + o_cells);
  F->aux = reinterpret_cast<float2 *>(b + o_aux) + MCG_TAB_PAD;
  F->tab = reinterpret_cast<float4 *>(b + o_tab) + MCG_TAB_PAD;
  F->slabs = reinterpret_cast<mcg_batch_slab_dev *>(b + o_slabs);
  F->items = reinterpret_cast<mcg_batch_item *>(b + o_items);
  F->cell_slab = reinterpret_cast<int32_t *>(b + o_cs);
  F->target = reinterpret_cast<double *>(b + o_t);
  F->grad = reinterpret_cast<double *>(b + o_g);
  F->loss_hist = reinterpret_cast<double *>(b + o_lh);
  F->sig_a = reinterpret_cast<float *>(b + o_sa);
  F->m1 = reinterpret_cast<float *>(b + o_m1);
  F->m2 = reinterpret_cast<float *>(b + o_m2);
  F->tally = reinterpret_cast<unsigned long long *>(b + o_ta);
  F->item_next = reinterpret_cast<unsigned long long *>(b + o_in);
  F->step = reinterpret_cast<long long *>(b + o_st);
  cudaMemset(F->dev, 0, off);
  std::vector<float4> cf(total), ct(total);
  std::vector<mcg_batch_slab_dev> sd(n_slabs);
  std::vector<int32_t> cs(total);
  int k = 0;
  for (int s = 0; s < n_slabs; ++s) {
    const mcg_slab &sl = h_slabs[s];
    const float dx = 1.0f / (float)sl.n_cells;
    sd[s].cell_off = k;
    sd[s].m = sl.n_cells;
    sd[s].n_hist = sl.n_histories;
    sd[s].src = {sl.seed_mode, sl.isotropic, sl.base_seed, 0.0f, sl.mu0, sl.w0, 0};
    for (int j = 0; j < sl.n_cells; ++j, ++k) {
      const float sig_s = h_sig_s[k];
      cf[k] = make_float4(h_sig_a0[k], sig_s > 1e-4f ? sig_s : 0.0f,
                          (float)j * dx, (float)(j + 1) * dx);
      ct[k] = mcg_tile_cell(cf[k]);
      cs[k] = s;
    }
  }
  if ((e = cudaMemcpy(F->cells, cf.data(), total * sizeof(float4), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(F->tab, ct.data(), total * sizeof(float4), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(F->slabs, sd.data(), n_slabs * sizeof(mcg_batch_slab_dev), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(F->items, items.data(), items.size() * sizeof(mcg_batch_item), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(F->cell_slab, cs.data(), total * 4, cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(F->target, h_target, total * 8, cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(F->sig_a, h_sig_a0, total * 4, cudaMemcpyHostToDevice)) != cudaSuccess)
    return fail(e, "mcg_fit_set: upload");
  F->n_slabs = n_slabs;
  F->n_cells = total;
  F->max_cells = maxc;
  F->lane_cells = lane_cells;
  F->max_steps = max_steps;
  F->min_w = particle_min_weight;
  return MCG_OK;
}

/* The forward pass and (with_grad) the replay, in turns. */
static int fit_launch_track(mcg_context *ctx, mcg_fit_state *F, int with_grad)
{
  mcg_batch_params B;
  memset(&B, 0, sizeof(B));
  B.cells = F->cells;
  B.tab = F->tab;
  B.aux = F->aux;
  B.loss = with_grad ? static_cast<float2 *>(F->dev_sum) : nullptr;
  B.step = F->step;
  B.slabs = F->slabs;
  B.max_cells = F->max_cells;
  B.tally = F->tally;
  B.rules = mcg_rules_setup(ctx, F->min_w);
  mcg_fit_params P;
  memset(&P, 0, sizeof(P));
  P.cells = F->cells;
  P.aux = F->aux;
  P.slabs = F->slabs;
  P.max_cells = F->max_cells;
  P.item_next = F->item_next + 1;
  P.sum = static_cast<const float2 *>(F->dev_sum);
  P.grad = F->grad;
  P.step = F->step;
  P.min_w = F->min_w;
  P.q_log2 = ctx->log2_scale;
  P.max_steps = ctx->max_steps;
  int block = 1024, f_bps = 1, l_bps = 1, bps = 1;
  while (block > 128 && mcg_batch_smem(F->max_cells, block, true, true) > (size_t)ctx->smem_optin)
    block -= 128;
  const size_t f_smem = mcg_batch_smem(F->max_cells, block, true, true);
  size_t smem = 4 * 8 + (((size_t)F->max_cells + 1) & ~(size_t)1) * 4;
  cudaError_t e = cudaFuncSetAttribute(mcg_fit_forward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       ctx->smem_optin);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f_bps, mcg_fit_forward, block, f_smem);
  const size_t l_smem = mcg_batch_lanes_smem(F->lane_cells, true); /* fewer cells than mcg_fit_set's limit */
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(mcg_fit_forward_lanes, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&l_bps, mcg_fit_forward_lanes, MCG_LANES_BLOCK, l_smem);
  if (e == cudaSuccess)
    e = mcg_grad_shape(mcg_fit_replay, 512, ctx->smem_optin, &smem, &P.jumps, &bps);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_fit: launch set-up");
  /* two blocks: their accumulators take what they took before the forward
   * pass had its own kernel */
  bps = std::min(std::max(bps, 1), 2);
  for (const mcg_fit_turn &t : F->turns) {
    if ((e = cudaMemsetAsync(F->item_next, 0, 24, ctx->stream)) != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_fit: memset");
    P.items = F->items + t.first;
    P.n_items = t.items;
    B.items = P.items;
    B.n_items = t.tiled;
    B.item_next = F->item_next;
    if (t.tiled) {
      mcg_fit_forward<<<ctx->sm_count * std::max(f_bps, 1), block, f_smem, ctx->stream>>>(B);
      ctx->launches++;
    }
    B.items = P.items + t.tiled;
    B.n_items = t.items - t.tiled;
    B.item_next = F->item_next + 2;
    if (B.n_items) {
      mcg_fit_forward_lanes<<<std::min(ctx->sm_count * std::max(l_bps, 1), B.n_items), MCG_LANES_BLOCK, l_smem,
                              ctx->stream>>>(B);
      ctx->launches++;
    }
    if (with_grad) {
      mcg_fit_replay<<<ctx->sm_count * bps, 512, smem, ctx->stream>>>(P);
      ctx->launches++;
    }
    if ((e = cudaGetLastError()) != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_fit: launch");
  }
  return MCG_OK;
}

/* n_steps Adam steps (lr, beta1, beta2, eps; sig_a kept >= sig_min). */
extern "C" int mcg_fit_run(mcg_context *ctx, int32_t n_steps, float lr, float beta1, float beta2,
                           float eps, float sig_min)
{
  mcg_fit_state *F = ctx ? fit_of(ctx, false) : nullptr;
  if (!F || n_steps < 0)
    return mcg_fail(MCG_ERR_STATE, "mcg_fit_run: mcg_fit_set first");
  cudaSetDevice(ctx->device);
  long long step0 = 0;
  cudaMemcpy(&step0, F->step, 8, cudaMemcpyDeviceToHost);
  if (step0 + n_steps > F->max_steps)
    return mcg_fail(MCG_ERR_ARG, "mcg_fit_run: at most %d steps in total", F->max_steps);
  const int nb = std::min((F->n_cells + 255) / 256, ctx->sm_count * 4);
  int rc = MCG_OK;
  cudaError_t e;
  if (step0 == 0) {
    /* weights for the first step: a forward pass at the starting point */
    if ((rc = fit_launch_track(ctx, F, 0)) != MCG_OK)
      return rc;
    mcg_fit_weights_kernel<<<nb, 256, 0, ctx->stream>>>(F->n_cells, F->cell_slab, F->slabs, F->target,
                                                        F->tally, F->aux, F->loss_hist, F->step,
                                                        ctx->log2_scale, 0);
    cudaMemsetAsync(F->grad, 0, F->n_cells * 8, ctx->stream);
  }
  /* one step = fused forward+adjoint, weights + loss, Adam: a CUDA graph */
  cudaGraph_t g;
  cudaGraphExec_t ge = nullptr;
  if ((e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_fit_run: capture");
  rc = fit_launch_track(ctx, F, 1);
  mcg_fit_weights_kernel<<<nb, 256, 0, ctx->stream>>>(F->n_cells, F->cell_slab, F->slabs, F->target,
                                                      F->tally, F->aux, F->loss_hist, F->step,
                                                      ctx->log2_scale, F->max_steps);
  mcg_fit_adam_kernel<<<1, 1024, 0, ctx->stream>>>(F->n_cells, F->cell_slab, F->slabs, F->grad,
                                                   F->sig_a, F->cells, F->tab, F->m1, F->m2, F->step, lr,
                                                   beta1, beta2, eps, sig_min);
  e = cudaStreamEndCapture(ctx->stream, &g);
  if (rc != MCG_OK)
    return rc;
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_fit_run: end capture");
  e = cudaGraphInstantiate(&ge, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_fit_run: instantiate");
  cudaEventRecord(ctx->ev0, ctx->stream);
  for (int s = 0; s < n_steps && e == cudaSuccess; ++s)
    e = cudaGraphLaunch(ge, ctx->stream);
  cudaEventRecord(ctx->ev1, ctx->stream);
  cudaError_t e2 = cudaStreamSynchronize(ctx->stream);
  cudaGraphExecDestroy(ge);
  if (e != cudaSuccess || e2 != cudaSuccess)
    return mcg_cuda_fail(e != cudaSuccess ? e : e2, "mcg_fit_run");
  cudaEventElapsedTime(&ctx->last_ms, ctx->ev0, ctx->ev1);
  ctx->launches += (2LL * (long long)F->turns.size() + 2) * n_steps;
  return MCG_OK;
}

/* Current sig_a (all cells, slab order), the per-step loss history and the
 * number of steps done. */
extern "C" int mcg_fit_read(mcg_context *ctx, float *h_sig_a, double *h_loss_hist, int32_t *h_steps)
{
  mcg_fit_state *F = ctx ? fit_of(ctx, false) : nullptr;
  if (!F)
    return mcg_fail(MCG_ERR_STATE, "mcg_fit_read: mcg_fit_set first");
  cudaSetDevice(ctx->device);
  long long st = 0;
  cudaError_t e = cudaMemcpy(&st, F->step, 8, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && h_sig_a)
    e = cudaMemcpy(h_sig_a, F->sig_a, F->n_cells * 4, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && h_loss_hist)
    e = cudaMemcpy(h_loss_hist, F->loss_hist, F->max_steps * 8, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_fit_read");
  if (h_steps)
    *h_steps = (int32_t)st;
  return MCG_OK;
}

/* One batched forward + adjoint launch of the fit kernel at the current
 * sig_a with the given loss weights (testing aid): histories step * n + i of
 * every slab, as the next Adam step would run, with w_c = h_weights[c]
 * instead of 2 (a_c - t_c).  Returns per cell the weight absorbed per history
 * (h_tally) and dF/dsig_a per history (h_grad), F = sum_c w_c a_c, so the
 * fit's gradient can be compared with mcg_adjoint's on the same histories.
 * The fit's own loss weights and accumulators are left as they were. */
extern "C" int mcg_fit_gradient(mcg_context *ctx, const double *h_weights, double *h_tally,
                                double *h_grad)
{
  mcg_fit_state *F = ctx ? fit_of(ctx, false) : nullptr;
  if (!F)
    return mcg_fail(MCG_ERR_STATE, "mcg_fit_gradient: mcg_fit_set first");
  if (!h_weights || !h_tally || !h_grad)
    return mcg_fail(MCG_ERR_ARG, "mcg_fit_gradient: bad arguments");
  cudaSetDevice(ctx->device);
  const int n = F->n_cells;
  std::vector<float2> saved(n), ax(n);
  std::vector<double> keep_grad(n);
  std::vector<unsigned long long> keep_tally(n), q(n);
  std::vector<mcg_batch_slab_dev> sd(F->n_slabs);
  std::vector<int32_t> cs(n);
  for (int c = 0; c < n; ++c)
    ax[c] = make_float2((float)h_weights[c], 0.0f);
  cudaError_t e;
  if ((e = cudaMemcpy(saved.data(), F->aux, n * sizeof(float2), cudaMemcpyDeviceToHost)) != cudaSuccess ||
      (e = cudaMemcpy(keep_grad.data(), F->grad, n * 8, cudaMemcpyDeviceToHost)) != cudaSuccess ||
      (e = cudaMemcpy(keep_tally.data(), F->tally, n * 8, cudaMemcpyDeviceToHost)) != cudaSuccess ||
      (e = cudaMemcpy(sd.data(), F->slabs, F->n_slabs * sizeof(mcg_batch_slab_dev), cudaMemcpyDeviceToHost)) != cudaSuccess ||
      (e = cudaMemcpy(cs.data(), F->cell_slab, n * 4, cudaMemcpyDeviceToHost)) != cudaSuccess ||
      (e = cudaMemcpy(F->aux, ax.data(), n * sizeof(float2), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemset(F->grad, 0, n * 8)) != cudaSuccess ||
      (e = cudaMemset(F->tally, 0, n * 8)) != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_fit_gradient: set-up");
  int rc = fit_launch_track(ctx, F, 1);
  if (rc != MCG_OK)
    return rc;
  if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess ||
      (e = cudaMemcpy(q.data(), F->tally, n * 8, cudaMemcpyDeviceToHost)) != cudaSuccess ||
      (e = cudaMemcpy(h_grad, F->grad, n * 8, cudaMemcpyDeviceToHost)) != cudaSuccess ||
      (e = cudaMemcpy(F->aux, saved.data(), n * sizeof(float2), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(F->grad, keep_grad.data(), n * 8, cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(F->tally, keep_tally.data(), n * 8, cudaMemcpyHostToDevice)) != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_fit_gradient");
  const double inv_scale = std::ldexp(1.0, -ctx->log2_scale);
  for (int c = 0; c < n; ++c) {
    const double nh = (double)sd[cs[c]].n_hist;
    h_tally[c] = (double)(long long)q[c] * inv_scale / nh;
    h_grad[c] /= nh;
  }
  return MCG_OK;
}
