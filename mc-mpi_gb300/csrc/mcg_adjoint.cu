/*
 * mcg_adjoint.cu - forward tally plus adjoint gradients of a tally loss.
 *
 * Loss: F = sum_c w_c a_c, a_c = expected weight absorbed in chain cell c
 * per history.  Parameters: sig_a[c] = sigs*rates and sig_s[c] =
 * sigs*(1 - rates) of every chain cell (the two cross sections of
 * Layer::particle_step, src/layer.cpp:129-131).
 *
 * For one history with steps k (cell c_k, flight length l_k, weight W_k after
 * the step, deposit g_k = w_{c_k} (W_{k-1} - W_k)), G = sum_k g_k and
 * P_k = g_1 + ... + g_k:
 *  - sig_a enters only the weight attenuation exp(-sig_a l), never the flight
 *    sampling, so its derivative is pathwise:
 *        dG/dsig_a[c] = sum_{k: c_k = c} l_k (w_c W_k - (G - P_k));
 *    this is a deliberate deviation from a score-function (likelihood-ratio)
 *    estimator for sig_a: with implicit capture no sampled event depends on
 *    sig_a, so its score is zero and the pathwise derivative is the whole
 *    gradient (same expectation, far lower variance);
 *  - sig_s sets the flight distribution (exponential with rate sig_s): the
 *    log-density score of step k is 1/sig_s - l_k for a collision and -l_k
 *    for a crossing (no collision before the face), and it weights the loss
 *    deposited from step k on (earlier deposits do not depend on it):
 *        dG/dsig_s[c] = sum_{k: c_k = c} score_k (G - P_{k-1}).
 * A first pass runs the histories forward (accumulating G and the tally), a
 * second one replays them from the same source index and seed (the path is never
 * stored) accumulating the two gradients.  G and P are float-float sums, so G - P
 * keeps its accuracy at the end of long histories.  The tally and the loss
 * are 64-bit fixed point (exact, order-independent); the gradients, which are
 * statistical estimates, are accumulated with fp32 shared-memory atomics
 * (one instruction per deposit) and flushed to fp64 once per block.
 */
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

/* A warp whose lanes need both exp paths takes the general one for all: it
 * returns the small-argument path's bits wherever that applies.  Measured on
 * the adjoint kernels: about 0.5-1 % faster; on the single-chain tracker, whose
 * crossings almost all take the small path, 3 % slower, so it keeps the
 * per-lane choice. */
#define MCG_EXP_UNIFORM
#include "mcg_internal.h"
#include "mcg_track.cuh"

struct mcg_adj_params {
  const float4 *cells, *tab;
  const float2 *aux; /* {w_c, 1/sig_s or 0} */
  int32_t n_cells, cell_lo, g_log2;
  mcg_rules rules;
  mcg_source src;
  int64_t first, n;
  unsigned long long *next;
  unsigned long long *tally, *loss, *counters;
  float2 *sum; /* per history the loss G of the forward pass; null: not wanted */
  double *grad_a, *grad_s;
  mcg_libm_dev libm;
  const mcg_libm_tab *libm_tab;
  int32_t chunk, jumps; /* jumps: the seed chain's table fits in shared memory (replay) */
  float b_mid; /* mcg_run_consts */
  int32_t refill; /* fused: steps between two looks for new histories */
};

/* Shared memory of the forward kernel: the tracker's, with the tiles' loss
 * weights. */
#define MCG_ADJ_FORWARD_BLOCK 1024
#define MCG_ADJ_LANES_BLOCK 512
#define MCG_ADJ_SHORT 256 /* cells of the longest chain that mcg_adjoint_fused takes whatever their widths */
#define MCG_ADJ_FUSED_STEPS 8 /* its steps between two looks for new histories (mcg_set_launch 0) */
#define MCG_ADJ_PART (1 << 24) /* most histories between a forward pass and its replay */
static size_t adj_forward_smem(int n_cells, int block, bool lanes)
{
  if (lanes)
    return mcg_track_smem(n_cells, 0, false);
  return mcg_track_smem(n_cells, block, false) +
         (size_t)(block / 32) * (sizeof(mcg_loss_smem) - sizeof(mcg_tile_smem<false>));
}

/*
 * Forward pass: the tracker's tiles, with each history's loss as one more sum
 * of the serial phase.  Bound: instruction issue, as the tracker.  1000 cells, 2e6
 * histories, strict: 18.3 ms with a lane per history, 14.3 ms so.
 */
template <bool STRICT, bool LANES>
__global__ void __launch_bounds__(LANES ? MCG_ADJ_LANES_BLOCK : 1024, LANES ? 2 : 1)
mcg_adjoint_forward(mcg_adj_params P)
{
  extern __shared__ __align__(16) unsigned char smem[];
  mcg_libm_tab *T = reinterpret_cast<mcg_libm_tab *>(smem);
  unsigned long long *s_cnt = reinterpret_cast<unsigned long long *>(smem + sizeof(mcg_libm_tab));
  mcg_chain_jumps *s_chain = reinterpret_cast<mcg_chain_jumps *>(s_cnt + 16);
  mcg_real_jumps *s_real = reinterpret_cast<mcg_real_jumps *>(s_chain + 1);
  unsigned long long *s_tally = reinterpret_cast<unsigned long long *>(s_real + 1);
  const int tid = threadIdx.x, ncell = P.n_cells, lo = P.cell_lo, gs = P.g_log2;
  mcg_loss_smem *tile = reinterpret_cast<mcg_loss_smem *>(s_tally + ((ncell + 1) & ~1)) + (tid >> 5);
  mcg_fill_chain_jumps(s_chain);
  mcg_fill_real_jumps(s_real);
  if (STRICT) {
    const float *src = reinterpret_cast<const float *>(P.libm_tab);
    float *dst = reinterpret_cast<float *>(T);
    for (int i = tid; i < (int)(sizeof(mcg_libm_tab) / 4); i += blockDim.x)
      dst[i] = src[i];
  }
  if (tid < 16)
    s_cnt[tid] = 0ull;
  for (int i = tid; i < ncell; i += blockDim.x)
    s_tally[i] = 0ull;
  __syncthreads();
  unsigned long long tot_steps = 0, tot_scat = 0, loss = 0, hist = 0;
  auto birth = [&](long long my, uint64_t &seed, float &x, float &mu, float &wmc, int &idx) {
    mcg_born(s_chain, P.src, P.first + my, seed, x, mu, wmc, idx);
    idx -= lo;
    return my;
  };
  auto end = [&](long long hid, int r, const mcg_lane &p, int) {
    if (r == 2)
      atomicOr(&s_cnt[MCG_CNT_ERR], 1ull); /* the step limit */
    if (P.sum)
      P.sum[hid] = make_float2(p.G_hi, p.G_lo);
    loss += (unsigned long long)(mcg_to_fixed(p.G_hi, gs) + mcg_to_fixed(p.G_lo, gs));
    ++hist;
    tot_steps += p.nst;
    tot_scat += p.nsc;
  };
  if constexpr (LANES) {
    mcg_lane_histories<STRICT, MCG_TALLY_SMEM32, true>(ncell, P.cells, P.aux, s_tally, P.rules, T, P.libm,
                                                       P.next, P.n, P.chunk, birth, end);
  } else {
    const mcg_tile_warp<false> tiles(tile, s_real);
    mcg_geometry geo = {0, ncell};
    mcg_sink sink = {(uint32_t)__cvta_generic_to_shared(s_tally), P.tally};
    mcg_histories<STRICT, false, MCG_TALLY_SMEM32, false, true>(
        geo, sink, P.cells, {P.tab, nullptr, 0, P.aux}, s_tally, P.rules, tiles, s_real, T, P.libm,
        P.next, [&] { return (long long)P.n; }, P.chunk, birth, end, [] { return true; },
        [] { return false; });
  }
  for (int o = 16; o > 0; o >>= 1) {
    loss += __shfl_down_sync(0xffffffffu, loss, o);
    hist += __shfl_down_sync(0xffffffffu, hist, o);
    tot_steps += __shfl_down_sync(0xffffffffu, tot_steps, o);
    tot_scat += __shfl_down_sync(0xffffffffu, tot_scat, o);
  }
  if ((tid & 31) == 0) {
    atomicAdd(&s_cnt[MCG_CNT_WLEFT], loss);
    atomicAdd(&s_cnt[MCG_CNT_HIST], hist);
    atomicAdd(&s_cnt[MCG_CNT_STEPS], tot_steps);
    atomicAdd(&s_cnt[MCG_CNT_SCAT], tot_scat);
  }
  __syncthreads();
  for (int i = tid; i < ncell; i += blockDim.x)
    if (s_tally[i])
      atomicAdd(&P.tally[i], s_tally[i]);
  if (tid == 0) {
    atomicAdd(P.loss, s_cnt[MCG_CNT_WLEFT]);
    atomicAdd(&P.counters[MCG_CNT_HIST], s_cnt[MCG_CNT_HIST]);
    atomicAdd(&P.counters[MCG_CNT_STEPS], s_cnt[MCG_CNT_STEPS]);
    atomicAdd(&P.counters[MCG_CNT_SCAT], s_cnt[MCG_CNT_SCAT]);
    if (s_cnt[MCG_CNT_ERR])
      atomicOr(&P.counters[MCG_CNT_ERR], s_cnt[MCG_CNT_ERR]);
  }
}

/*
 * Replay: each history again from its birth, with its loss G known, for the
 * gradients.  Bound: instruction issue at 12 of 32 lanes, the histories of a warp
 * being at different places.  Almost every step is a crossing that the bounds of
 * mcg_cross decide without the logarithm, the exponential's table or the new
 * direction, so the few full steps are gathered (the rounds below) instead of
 * stopping the whole warp for one lane.  1000 cells, 2e6 histories, strict:
 * 19 ms; with the full step in every lane, forward pass and replay took 69.2 ms.
 * A history stays with a lane, and 512 lanes share one fp32 accumulator per
 * cell: tiles, as the forward pass has, add a cell's terms in another grouping,
 * which moved the gradients by more than two runs of this kernel differ (and
 * saved little: the two float atomics of a step are compare-and-swap loops).
 */
template <bool STRICT>
__global__ void __launch_bounds__(1024) mcg_adjoint_replay(mcg_adj_params P)
{
  extern __shared__ __align__(16) unsigned char smem[];
  mcg_libm_tab *T = reinterpret_cast<mcg_libm_tab *>(smem);
  float *s_ga = reinterpret_cast<float *>(smem + sizeof(mcg_libm_tab));
  float *s_gs = s_ga + P.n_cells;
  mcg_chain_jumps *s_chain = reinterpret_cast<mcg_chain_jumps *>(s_gs + P.n_cells);
  const int tid = threadIdx.x;
  const int ncell = P.n_cells, lo = P.cell_lo;
  if (P.jumps)
    mcg_fill_chain_jumps(s_chain);
  if (STRICT) {
    const float *src = reinterpret_cast<const float *>(P.libm_tab);
    float *dst = reinterpret_cast<float *>(T);
    for (int i = tid; i < (int)(sizeof(mcg_libm_tab) / 4); i += blockDim.x)
      dst[i] = src[i];
  }
  for (int i = tid; i < 2 * ncell; i += blockDim.x)
    s_ga[i] = 0.0f; /* both gradient arrays */
  __syncthreads();
  const float min_w = P.rules.min_w;
  const uint32_t max_steps = P.rules.max_steps;

  uint64_t seed = 0;
  float x = 0.f, mu = 0.f, wmc = 0.f, inv_mu = 0.f;
  int idx = 0;
  uint32_t nst = 0, nsc = 0;
  float G_hi = 0.f, G_lo = 0.f, P_hi = 0.f, P_lo = 0.f, v_before = 0.f;
  bool active = false, wait = false; /* wait: the lane's step needs the full form */
  mcg_pool pool;

  for (;;) {
    const unsigned need = __ballot_sync(0xffffffffu, !active);
    if (need) {
      const long long my = pool.take(need, P.next, P.n, P.chunk);
      if (!active && my >= 0) {
        if (P.jumps)
          mcg_born(s_chain, P.src, P.first + my, seed, x, mu, wmc, idx);
        else
          mcg_source_particle(P.src, P.first + my, seed, x, mu, wmc, idx);
        idx -= lo;
        inv_mu = mcg_flight_rcp(mu);
        nst = 0;
        const float2 g = P.sum[my];
        G_hi = g.x;
        G_lo = g.y;
        P_hi = P_lo = 0.f;
        v_before = __fadd_rn(G_hi, G_lo);
        active = true;
      }
    }
    if (!__any_sync(0xffffffffu, active))
      break;

    auto account = [&](int c, float l, bool coll, float dep) {
      const float2 ax = __ldg(P.aux + c);
      mcg_ff_add(P_hi, P_lo, __fmul_rn(ax.x, dep)); /* the loss so far */
      /* suffix before this step, then after it */
      const float v_after = __fadd_rn(__fsub_rn(G_hi, P_hi), __fsub_rn(G_lo, P_lo));
      const float ga = l * (ax.x * wmc - v_after);
      const float score = (coll ? ax.y : 0.0f) - l;
      const float gsc = score * v_before;
      atomicAdd(&s_ga[c], ga);
      atomicAdd(&s_gs[c], gsc);
      v_before = v_after;
      ++nst;
    };
    auto living = [&] {
      return active & (wmc >= min_w) & ((unsigned)idx < (unsigned)ncell) & (nst < max_steps);
    };
    /* crossings of the lanes that can, at most `most`; a lane that meets
     * another step waits; returns whether the lane could go on */
    auto cross = [&](int most) {
      bool go = living() & !wait;
      for (int j = 0; go & (j < most); ++j) {
        const int c = idx;
        float l, dep;
        if (!mcg_cross<STRICT>(seed, x, mu, wmc, inv_mu, idx, __ldg(P.cells + c), P.b_mid, l, dep)) {
          wait = true;
          go = false;
        } else {
          account(c, l, false, dep);
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
        mcg_full<STRICT, MCG_TALLY_SMEM32>(seed, x, mu, wmc, inv_mu, idx, nsc, __ldg(P.cells + c),
                                           nullptr, P.rules.q_log2, T, P.libm, &l, &coll, &dep);
        account(c, l, coll, dep);
        wait = false;
      }
    };
    /* a lane that waits does so while the others cross, MCG_GRAD_WINDOW steps
     * between two votes, until MCG_GRAD_POOL of 32 with a history wait, and as
     * many fewer as there are (a fixed number: 34.1 ms for 32.9, the last
     * histories waiting for one another); the round lasts until
     * MCG_GRAD_REFILL lanes have ended a history or want one.  Every pass
     * steps a lane, makes one wait or completes the waiting steps, and no lane
     * passes its step limit, so it ends. */
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
  __syncthreads();
  for (int i = tid; i < ncell; i += blockDim.x) {
    if (s_ga[i] != 0.0f)
      atomicAdd(&P.grad_a[i], (double)s_ga[i]);
    if (s_gs[i] != 0.0f)
      atomicAdd(&P.grad_s[i], (double)s_gs[i]);
  }
}

/*
 * Short chains, and those of thick cells (adj_thick): forward pass and replay in one
 * kernel, every lane through the whole step.  A short history is mostly its birth and its end, which the two
 * kernels pay twice (50 cells, 1e6 histories, strict: 4.8 ms here, 5.4 ms there;
 * 100 cells: 7.7 against 7.2), and where thousands of histories add to the same
 * few floats the order of the additions shows: rounds in which colliding
 * lanes fall behind the others moved dF/dsig_a of 50 cells by 2.6e-7, six times what
 * two runs differ by.  At 300 cells it is within that, and the two kernels
 * take 8.9 ms instead of 16.6 (1e6 histories).
 */
template <bool STRICT>
__global__ void __launch_bounds__(1024) mcg_adjoint_fused(mcg_adj_params P)
{
  extern __shared__ __align__(16) unsigned char smem[];
  mcg_libm_tab *T = reinterpret_cast<mcg_libm_tab *>(smem);
  unsigned long long *s_cnt = reinterpret_cast<unsigned long long *>(smem + sizeof(mcg_libm_tab));
  unsigned long long *s_tally = s_cnt + 16;
  float *s_ga = reinterpret_cast<float *>(s_tally + P.n_cells);
  float *s_gs = s_ga + P.n_cells;
  const int tid = threadIdx.x, lane = tid & 31;
  const int ncell = P.n_cells, lo = P.cell_lo;
  if (STRICT) {
    const float *src = reinterpret_cast<const float *>(P.libm_tab);
    float *dst = reinterpret_cast<float *>(T);
    for (int i = tid; i < (int)(sizeof(mcg_libm_tab) / 4); i += blockDim.x)
      dst[i] = src[i];
  }
  if (tid < 16)
    s_cnt[tid] = 0ull;
  for (int i = tid; i < 2 * ncell; i += blockDim.x)
    s_tally[i] = 0ull; /* the tally and both float gradient arrays */
  __syncthreads();
  const float min_w = P.rules.min_w;
  const int qs = P.rules.q_log2, gs = P.g_log2;

  uint64_t seed = 0;
  float x = 0.f, mu = 0.f, wmc = 0.f, inv_mu = 0.f;
  int idx = 0, phase = 0;
  int64_t hid = -1;
  uint32_t nst = 0, nsc = 0;
  float G_hi = 0.f, G_lo = 0.f, P_hi = 0.f, P_lo = 0.f;
  bool active = false;
  unsigned long long tot_steps = 0, tot_scat = 0;
  long long pool_next = 0, pool_end = 0;
  bool drained = false;

  for (;;) {
    unsigned need = __ballot_sync(0xffffffffu, !active);
    if (need) {
      int cnt = __popc(need), rank = __popc(need & lanemask_lt());
      long long avail = pool_end - pool_next, my = -1;
      if (rank < avail)
        my = pool_next + rank;
      if (cnt > avail && !drained) {
        unsigned long long base = 0;
        if (lane == 0)
          base = atomicAdd(P.next, (unsigned long long)P.chunk);
        base = __shfl_sync(0xffffffffu, base, 0);
        if ((long long)base >= P.n) {
          drained = true;
          pool_next = pool_end = 0;
        } else {
          long long end = min((long long)base + P.chunk, (long long)P.n);
          long long r2 = rank - avail;
          if (rank >= avail && r2 < end - (long long)base)
            my = (long long)base + r2;
          pool_next = min((long long)base + (cnt - avail), end);
          pool_end = end;
        }
      } else {
        pool_next += min((long long)cnt, avail);
      }
      if (!active && my >= 0) {
        hid = my;
        mcg_source_particle(P.src, P.first + hid, seed, x, mu, wmc, idx);
        idx -= lo;
        inv_mu = mcg_flight_rcp(mu);
        nst = nsc = 0;
        phase = 0;
        G_hi = G_lo = P_hi = P_lo = 0.f;
        active = true;
      }
    }
    if (!__any_sync(0xffffffffu, active))
      break;

    if (active) {
      /* up to P.refill steps, never past the step limit; idx is local
       * to the chain */
      const int kmax = (int)min((uint32_t)P.refill, P.rules.max_steps - nst);
      int k = 0;
      bool going = true;
      for (; k < kmax; ++k) {
        if (!((wmc >= min_w) & ((unsigned)idx < (unsigned)ncell))) {
          going = false;
          break;
        }
        const int c = idx;
        const float2 ax = __ldg(P.aux + c);
        float l, dep;
        bool coll;
        mcg_step<STRICT, MCG_TALLY_SMEM32>(seed, x, mu, wmc, inv_mu, idx, nsc, __ldg(P.cells + c),
                                           phase == 0 ? &s_tally[c] : nullptr, qs, T, P.libm, &l,
                                           &coll, &dep);
        const float g = __fmul_rn(ax.x, dep);
        if (phase == 0) {
          mcg_ff_add(G_hi, G_lo, g);
        } else {
          /* suffix before this step, then after it */
          const float v_before = __fadd_rn(__fsub_rn(G_hi, P_hi), __fsub_rn(G_lo, P_lo));
          mcg_ff_add(P_hi, P_lo, g);
          const float v_after = __fadd_rn(__fsub_rn(G_hi, P_hi), __fsub_rn(G_lo, P_lo));
          const float ga = l * (ax.x * wmc - v_after);
          const float score = (coll ? ax.y : 0.0f) - l;
          const float gsc = score * v_before;
          atomicAdd(&s_ga[c], ga);
          atomicAdd(&s_gs[c], gsc);
        }
      }
      nst += (uint32_t)k;
      if (!going || nst >= P.rules.max_steps) {
        if ((wmc >= min_w) && ((unsigned)idx < (unsigned)ncell))
          atomicOr(&s_cnt[MCG_CNT_ERR], 1ull); /* the step limit */
        if (phase == 0) {
          tot_steps += nst;
          tot_scat += nsc;
        }
        if (phase == 0) {
          /* replay the same history from its start */
          mcg_source_particle(P.src, P.first + hid, seed, x, mu, wmc, idx);
          idx -= lo;
          inv_mu = mcg_flight_rcp(mu);
          nst = nsc = 0;
          phase = 1;
        } else {
          atomicAdd(&s_cnt[MCG_CNT_HIST], 1ull);
          mcg_tally_add<MCG_TALLY_SMEM32>(&s_cnt[MCG_CNT_WLEFT],
                                           mcg_to_fixed(G_hi, gs) + mcg_to_fixed(G_lo, gs));
          active = false;
        }
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    tot_steps += __shfl_down_sync(0xffffffffu, tot_steps, o);
    tot_scat += __shfl_down_sync(0xffffffffu, tot_scat, o);
  }
  if (lane == 0) {
    atomicAdd(&s_cnt[MCG_CNT_STEPS], tot_steps);
    atomicAdd(&s_cnt[MCG_CNT_SCAT], tot_scat);
  }
  __syncthreads();
  for (int i = tid; i < ncell; i += blockDim.x) {
    if (s_tally[i])
      atomicAdd(&P.tally[i], s_tally[i]);
    if (s_ga[i] != 0.0f)
      atomicAdd(&P.grad_a[i], (double)s_ga[i]);
    if (s_gs[i] != 0.0f)
      atomicAdd(&P.grad_s[i], (double)s_gs[i]);
  }
  if (tid == 0) {
    atomicAdd(P.loss, s_cnt[MCG_CNT_WLEFT]);
    atomicAdd(&P.counters[MCG_CNT_HIST], s_cnt[MCG_CNT_HIST]);
    atomicAdd(&P.counters[MCG_CNT_STEPS], s_cnt[MCG_CNT_STEPS]);
    atomicAdd(&P.counters[MCG_CNT_SCAT], s_cnt[MCG_CNT_SCAT]);
    if (s_cnt[MCG_CNT_ERR])
      atomicOr(&P.counters[MCG_CNT_ERR], s_cnt[MCG_CNT_ERR]);
  }
}

/* ------------------------------------------------------------ host side */
static mcg_adj_state *adj_of(mcg_context *ctx)
{
  if (!ctx->ext)
    ctx->ext = new mcg_ext();
  return &ctx->ext->adj;
}

void mcg_adjoint_release(mcg_adj_state *A)
{
  if (A->d_aux)
    cudaFree(A->d_aux);
  if (A->d_grad)
    cudaFree(A->d_grad);
  if (A->d_sum)
    cudaFree(A->d_sum);
  *A = mcg_adj_state();
}

extern "C" int mcg_adjoint_set_weights(mcg_context *ctx, const float *h_w)
{
  if (!ctx || !h_w || !ctx->d_tally)
    return mcg_fail(MCG_ERR_ARG, "mcg_adjoint_set_weights: bad arguments or no layers");
  cudaSetDevice(ctx->device);
  mcg_adj_state *A = adj_of(ctx);
  const int n = ctx->n_cells;
  if (A->n != n) {
    if (A->d_aux)
      cudaFree(A->d_aux);
    if (A->d_grad)
      cudaFree(A->d_grad);
    A->d_aux = nullptr;
    A->d_grad = nullptr;
    cudaError_t e;
    if ((e = cudaMalloc(&A->d_aux, (n + 2 * (size_t)MCG_TAB_PAD) * sizeof(float2))) != cudaSuccess ||
        (e = cudaMalloc(&A->d_grad, (2 * (size_t)n + 1) * sizeof(unsigned long long))) != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_adjoint_set_weights: cudaMalloc");
    A->n = n;
  }
  std::vector<float2> aux(n + 2 * (size_t)MCG_TAB_PAD, make_float2(0.f, 0.f));
  for (int c = 0; c < n; ++c) {
    const float sig_i = ctx->cells_strict[c].y; /* the flight cross section of the step */
    aux[c + MCG_TAB_PAD] = make_float2(h_w[c], sig_i > 1e-4f ? 1.0f / sig_i : 0.0f);
  }
  cudaError_t e = cudaMemcpy(A->d_aux, aux.data(), aux.size() * sizeof(float2), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemset(A->d_grad, 0, (2 * (size_t)n + 1) * sizeof(unsigned long long));
  A->histories = 0;
  return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(e, "mcg_adjoint_set_weights");
}

extern "C" int mcg_adjoint_reset(mcg_context *ctx)
{
  if (!ctx)
    return mcg_fail(MCG_ERR_ARG, "mcg_adjoint_reset: null context");
  mcg_adj_state *A = adj_of(ctx);
  if (!A->d_grad)
    return mcg_fail(MCG_ERR_STATE, "mcg_adjoint_reset: no loss weights set");
  cudaSetDevice(ctx->device);
  cudaError_t e = cudaMemset(A->d_grad, 0, (2 * (size_t)A->n + 1) * sizeof(unsigned long long));
  A->histories = 0;
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_adjoint_reset");
  return mcg_tally_reset(ctx);
}

/* Chains of thick cells, on which most steps are full ones: with a gradient the one
 * kernel with every lane through the whole step (rounds gather too little there),
 * without one a forward pass with a lane per history.  Two kernels / one, widths
 * sig_a and sig_i, 300 to 1500 cells: strict .02, .02 .7, .03, .03 1.14, .05, .05 1.1, .1, .1 1.2,
 * .1, .01 1.3 to 1.7, .01, .1 .6; fast .05, .05 .8, .01, .1 .85, .1, .01 1.2, .1, .1
 * 1.2, .3, .3 1.5, .05, .3 1.7.  Forward pass, tiles / lanes, 40 and 300 cells: strict
 * .02, .02 1.0 and .6, .05, .05 1.9 and 1.2, .1, .01 4.5 and 3.7; fast .05, .05 1.0 and
 * .6, .1, .1 1.5 and .9, .3, .3 3.2 and 2.2, ten cells of .1, .1 1.7.  Below eight cells
 * lanes (two cells: 2.1). */
static bool adj_thick(const mcg_widths &w, int n, bool strict, bool gradient)
{
  if (n < 8)
    return true;
  if (strict)
    return w.a > 0.025 * n || w.i > 0.25 * n;
  return gradient ? w.a > 0.06 * n || w.a + w.i > 0.15 * n
                  : w.a + w.i > (n < 32 ? 0.1 : 0.25) * n;
}

extern "C" int mcg_adjoint_run(mcg_context *ctx, const mcg_source *src, int64_t first, int64_t n,
                               int32_t with_gradient)
{
  if (!ctx || !src || n < 0 || first < 0)
    return mcg_fail(MCG_ERR_ARG, "mcg_adjoint_run: bad arguments");
  mcg_adj_state *A = adj_of(ctx);
  if (!A->d_aux || A->n != ctx->n_cells)
    return mcg_fail(MCG_ERR_STATE, "mcg_adjoint_run: set the loss weights first");
  cudaSetDevice(ctx->device);
  const bool strict = ctx->mode == MCG_MODE_STRICT;
  if (strict && !ctx->libm_loaded) {
    int rc = mcg_load_libm(ctx);
    if (rc != MCG_OK)
      return rc;
  }
  if (n == 0)
    return MCG_OK;
  mcg_adj_params P;
  memset(&P, 0, sizeof(P));
  P.cells = strict ? ctx->d_cells_strict : ctx->d_cells_fast;
  P.tab = ctx->d_tab + MCG_TAB_PAD;
  P.aux = A->d_aux + MCG_TAB_PAD;
  P.n_cells = ctx->n_cells;
  P.cell_lo = ctx->cell_lo;
  P.g_log2 = A->g_log2;
  P.rules = mcg_rules_setup(ctx, ctx->min_w);
  P.src = *src;
  P.next = ctx->d_next;
  P.tally = ctx->d_tally;
  P.grad_a = reinterpret_cast<double *>(A->d_grad);
  P.grad_s = reinterpret_cast<double *>(A->d_grad) + A->n;
  P.loss = A->d_grad + 2 * A->n;
  P.counters = ctx->d_counters;
  P.libm = ctx->libm;
  P.libm_tab = ctx->libm_tab;
  P.b_mid = ctx->run_bounds[2];
  P.refill = ctx->refill ? ctx->refill : MCG_ADJ_FUSED_STEPS;
  /* the longest chain: that of the replay's arrays beside a tally */
  if (sizeof(mcg_libm_tab) + 16 * 8 + 2 * (size_t)ctx->n_cells * 8 > (size_t)ctx->smem_optin)
    return mcg_fail(MCG_ERR_ARG, "mcg_adjoint_run: chain of %d cells too long (max %d)",
                    ctx->n_cells, (int)((ctx->smem_optin - 2048 - 128) / 16));
  const bool thick = adj_thick(ctx->widths, ctx->n_cells, strict, with_gradient), lanes = thick && !with_gradient;
  auto forward = strict ? (lanes ? mcg_adjoint_forward<true, true> : mcg_adjoint_forward<true, false>)
                        : (lanes ? mcg_adjoint_forward<false, true> : mcg_adjoint_forward<false, false>);
  auto replay = strict ? mcg_adjoint_replay<true> : mcg_adjoint_replay<false>;
  auto short_chain = strict ? mcg_adjoint_fused<true> : mcg_adjoint_fused<false>;
  const bool fused = with_gradient && (ctx->n_cells <= MCG_ADJ_SHORT || thick);
  int f_block = lanes ? MCG_ADJ_LANES_BLOCK : MCG_ADJ_FORWARD_BLOCK, f_bps = 1, bps = 1;
  while (f_block > 128 && adj_forward_smem(ctx->n_cells, f_block, lanes) > (size_t)ctx->smem_optin)
    f_block -= 128;
  const size_t f_smem = adj_forward_smem(ctx->n_cells, f_block, lanes);
  const int block = ctx->block ? ctx->block : 512;
  size_t smem = sizeof(mcg_libm_tab) + (size_t)ctx->n_cells * 8;
  const size_t fused_smem = sizeof(mcg_libm_tab) + 16 * 8 + 2 * (size_t)ctx->n_cells * 8;
  cudaError_t e = cudaFuncSetAttribute(forward, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f_bps, forward, f_block, f_smem);
  if (e == cudaSuccess && fused)
    e = cudaFuncSetAttribute(short_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin);
  if (e == cudaSuccess)
    e = fused ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, short_chain, block, fused_smem)
              : mcg_grad_shape(replay, block, ctx->smem_optin, &smem, &P.jumps, &bps);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_adjoint_run: launch set-up");
  /* two blocks of 512: their accumulators take what they took before the
   * forward pass had its own kernel */
  bps = std::max(bps, 1);
  if (!fused)
    bps = std::min(bps, std::max(1024 / block, 1));
  /* the histories' sums: 8 bytes each, for up to MCG_ADJ_PART histories at a time */
  int64_t part = n;
  if (with_gradient && !fused) {
    part = std::min<int64_t>(n, MCG_ADJ_PART);
    while (A->sums < part) {
      if (A->d_sum)
        cudaFree(A->d_sum);
      A->d_sum = nullptr;
      A->sums = 0;
      if ((e = mcg_dev_malloc((void **)&A->d_sum, (size_t)part * sizeof(float2))) == cudaSuccess) {
        A->sums = part;
      } else {
        cudaGetLastError();
        if (part <= 4096)
          return mcg_cuda_fail(e, "mcg_adjoint_run: cudaMalloc");
        part /= 2;
      }
    }
    P.sum = A->d_sum;
  }
  cudaEventRecord(ctx->ev0, ctx->stream);
  if (fused) {
    P.first = first;
    P.n = n;
    P.chunk = 64;
    if ((e = cudaMemsetAsync(ctx->d_next, 0, 8, ctx->stream)) != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_adjoint_run: memset");
    short_chain<<<(int)std::min<int64_t>((int64_t)ctx->sm_count * bps, (n + block - 1) / block), block,
                  fused_smem, ctx->stream>>>(P);
    if ((e = cudaGetLastError()) != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_adjoint_run: launch");
    ctx->launches++;
  }
  for (int64_t at = 0; at < n && !fused; at += part) {
    P.first = first + at;
    P.n = std::min(part, n - at);
    const int64_t warps = (int64_t)ctx->sm_count * std::max(f_bps, 1) * (f_block / 32);
    P.chunk = lanes ? 32 : (int)std::min<int64_t>(32, (P.n + warps - 1) / warps);
    if ((e = cudaMemsetAsync(ctx->d_next, 0, 8, ctx->stream)) != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_adjoint_run: memset");
    forward<<<(int)std::min<int64_t>((int64_t)ctx->sm_count * std::max(f_bps, 1), P.n), f_block, f_smem,
              ctx->stream>>>(P);
    ctx->launches++;
    if (with_gradient) {
      P.chunk = 64;
      if ((e = cudaMemsetAsync(ctx->d_next, 0, 8, ctx->stream)) != cudaSuccess)
        return mcg_cuda_fail(e, "mcg_adjoint_run: memset");
      replay<<<(int)std::min<int64_t>((int64_t)ctx->sm_count * bps, (P.n + block - 1) / block), block, smem,
               ctx->stream>>>(P);
      ctx->launches++;
    }
    if ((e = cudaGetLastError()) != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_adjoint_run: launch");
  }
  cudaEventRecord(ctx->ev1, ctx->stream);
  A->histories += n;
  return mcg_sync(ctx);
}

extern "C" int mcg_adjoint_read(mcg_context *ctx, double *h_loss, double *h_grad_a, double *h_grad_s)
{
  if (!ctx)
    return mcg_fail(MCG_ERR_ARG, "mcg_adjoint_read: null context");
  mcg_adj_state *A = adj_of(ctx);
  if (!A->d_grad || A->histories == 0)
    return mcg_fail(MCG_ERR_STATE, "mcg_adjoint_read: nothing run");
  cudaSetDevice(ctx->device);
  std::vector<int64_t> q(2 * (size_t)A->n + 1);
  cudaError_t e = cudaMemcpy(q.data(), A->d_grad, q.size() * sizeof(int64_t), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_adjoint_read");
  const double inv = 1.0 / (double)A->histories;
  if (h_loss)
    *h_loss = (double)q[2 * A->n] * std::ldexp(1.0, -A->g_log2) * inv;
  for (int c = 0; c < A->n; ++c) {
    double ga, gs;
    memcpy(&ga, &q[c], 8);
    memcpy(&gs, &q[A->n + c], 8);
    if (h_grad_a)
      h_grad_a[c] = ga * inv;
    if (h_grad_s)
      h_grad_s[c] = gs * inv;
  }
  return MCG_OK;
}
