/*
 * mcg_track.cuh - the history-based tracker.
 *
 * One lane carries one particle history at a time through the whole chain of
 * layers (a sub-domain crossing is just the next cell's parameters, so the
 * hand-over between sub-domains costs nothing), and the warp advances its 32
 * histories together, a tile of certain crossings each (see "tiles" below).
 * The grid is persistent: every warp takes chunks of history indices from a
 * global counter and refills finished lanes from its chunk, so warps stay full
 * however uneven the history lengths are.  Deposits go to a shared-memory
 * fixed-point histogram (one copy per block, or one per warp when the chain is
 * short) and are added to the global tally once per block at the end; the sums
 * are exact, hence order-independent.
 *
 * The step follows Layer::particle_step (src/layer.cpp:123-190) and the loop
 * Layer::simulate_particle (src/layer.cpp:192-218).
 */
#ifndef MCG_TRACK_CUH
#define MCG_TRACK_CUH

#include <algorithm>
#include "mcg_device.cuh"
#include "mcgb300.h"
#include "mcg_internal.h"

/* Per-cell parameters of the tiles, readable MCG_TAB_PAD cells past both ends:
 * cell: {sig_a, sig_i, length of a flight entering by the left face, by the
 * right face}; thin (thin chains): {sig_a, that length} for flights to the
 * right and, `left` entries on, for flights to the left: half the bytes of the
 * other (the loads were a quarter of the L1's work on the 10,000-cell slab). */
struct mcg_tab {
  const float4 *cell;
  const float2 *thin;
  int32_t left;
  const float2 *aux; /* LOSS: {w_c, .}, readable as far */
};

inline mcg_tab mcg_chain_tab(const mcg_context *ctx)
{
  return {ctx->d_tab + MCG_TAB_PAD, ctx->d_thin ? ctx->d_thin + MCG_TAB_PAD : nullptr,
          ctx->n_cells + 2 * MCG_TAB_PAD};
}

/* How a warp runs its histories (mcg_histories). */
struct mcg_rules {
  float min_w;
  int32_t q_log2;
  uint32_t max_steps;
  int32_t window;       /* most steps of a tile (at most MCG_TW_MAX) */
  int32_t pool_lanes;   /* lanes waiting for the full step that trigger it */
  int32_t refill_lanes; /* lanes without a history that trigger a refill */
  mcg_run_consts run;
};

/* Per-cell step parameters.  strict: {sig_a, sig_i, edge_lo, edge_hi}
 * fast: {sig_a, sig_i (0 when sig_i <= EPS), edge_lo, edge_hi}
 * edge_lo = (float)i * dx_layer, edge_hi = (float)(i+1) * dx_layer with the
 * GLOBAL cell index i and the cell's own layer spacing (src/layer.cpp:146,150). */
struct mcg_track_params {
  const float4 *cells;
  mcg_tab tab;
  int32_t n_cells, cell_lo;
  mcg_particle *particles; /* NULL: source mode */
  int32_t *results;
  int64_t *steps, *scatters;
  int64_t n, first;
  mcg_source src;
  unsigned long long *next;  /* work counter, starts at 0 */
  unsigned long long *tally; /* [n_cells] fixed point */
  unsigned long long *counters; /* mcg_counters fields */
  mcg_libm_dev libm;
  const mcg_libm_tab *libm_tab;
  int32_t tally_copies; /* 1 or warps per block */
  int32_t chunk;        /* histories per warp grab */
  mcg_rules rules;
  /* null, or the largest |weight| of the particles (its bits): the launch does
   * nothing unless (*heaviest >= heavy_line) == heavy (mcg_heavy_weight) */
  const uint32_t *heaviest;
  uint32_t heavy_line;
  int32_t heavy;
};

/* Tally accumulation: shared-memory 64-bit atomics, shared-memory 32-bit
 * halves with an explicit carry, 64-bit atomics straight to the global tally,
 * or (thin chains) shared-memory low words with the carries going straight to
 * the global tally. */
enum { MCG_TALLY_SMEM64 = 0, MCG_TALLY_SMEM32 = 1, MCG_TALLY_GLOBAL = 2, MCG_TALLY_LO32 = 3 };

template <int TALLY>
__device__ __forceinline__ void mcg_tally_add(unsigned long long *t, long long q)
{
  if (TALLY == MCG_TALLY_SMEM32) {
    /* exact 64-bit sum from 32-bit atomics: a carry out of the low word is
     * detected by the adder that caused it and added to the high word */
    const uint64_t v = (uint64_t)q;
    const uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
    unsigned *w = reinterpret_cast<unsigned *>(t);
    const uint32_t old = atomicAdd(w, lo);
    const uint32_t add_hi = hi + (((uint32_t)(old + lo) < old) ? 1u : 0u);
    if (add_hi)
      atomicAdd(w + 1, add_hi);
  } else {
    atomicAdd(t, (unsigned long long)q);
  }
}

/* Adds the fixed-point deposit llrint(dw 2^S) (ties to even, the oracle's
 * quantisation) to a tally cell.  A deposit with 0 <= dw 2^S < 2^31 (all but
 * the largest, and the negative ones of particles started outside their
 * cell) converts with the 32-bit conversion and adds with one 32-bit atomic
 * and a carry into the high word; the others take the 64-bit conversion,
 * which issues on the FP64 pipe (about 6e11/s per GB300, the strict
 * tracker's binding resource while it ran on every step). */
template <int TALLY>
__device__ __forceinline__ void mcg_deposit_u31(unsigned long long *t, float v)
{
  /* v = dw 2^S with +0 <= v < 2^31: the 32-bit conversion is exact */
  const uint32_t q = __float2uint_rn(v);
  if (TALLY == MCG_TALLY_SMEM32) {
    unsigned *w = reinterpret_cast<unsigned *>(t);
    const uint32_t old = atomicAdd(w, q);
    if ((uint32_t)(old + q) < old)
      atomicAdd(w + 1, 1u);
  } else {
    atomicAdd(t, (unsigned long long)q);
  }
}

template <int TALLY>
__device__ __forceinline__ void mcg_deposit(unsigned long long *t, float dw, int S)
{
  const float v = __fmul_rn(dw, mcg_fixed_scale(S));
  if (__float_as_uint(v) < 0x4f000000u) /* +0 <= v < 2^31 */
    mcg_deposit_u31<TALLY>(t, v);
  else
    mcg_tally_add<TALLY>(t, mcg_to_fixed(dw, S));
}

enum { MCG_CNT_HIST = 0, MCG_CNT_STEPS, MCG_CNT_SCAT, MCG_CNT_LEFT, MCG_CNT_RIGHT, MCG_CNT_KILL,
       MCG_CNT_WLEFT, MCG_CNT_WRIGHT, MCG_CNT_WKILL, MCG_CNT_ERR, MCG_CNT_N };

/* Particle of a device-born source (see mcg_source in mcgb300.h) whose
 * seed-chain state s is known: particle k has s = the chain's (k+1)-th
 * state from base_seed (seed_mode 0) or base_seed + k (seed_mode 1). */
__device__ __forceinline__ void mcg_source_particle_at(const mcg_source &S, uint64_t s,
                                                       uint64_t &seed, float &x, float &mu,
                                                       float &wmc, int &idx)
{
  float m = S.mu0;
  if (S.isotropic == 1)
    m = __fsub_rn(__fmul_rn(2.0f, mcg_rnd_real(s)), 1.0f);
  else if (S.isotropic == 2)
    m = mcg_rnd_real(s);
  seed = s;
  x = S.x0;
  mu = m;
  wmc = S.w0;
  idx = S.cell0;
}

/* Particle k of a device-born source. */
__device__ __forceinline__ void mcg_source_particle(const mcg_source &S, int64_t k, uint64_t &seed,
                                                    float &x, float &mu, float &wmc, int &idx)
{
  const uint64_t s = S.seed_mode == 0 ? mcg_lcg_skip(S.base_seed, (uint64_t)k + 1, 1)
                                      : ((S.base_seed + (uint64_t)k) & MCG_MASK63);
  mcg_source_particle_at(S, s, seed, x, mu, wmc, idx);
}

__device__ __forceinline__ void mcg_load_particle(const mcg_track_params &P, int64_t i,
                                                  uint64_t &seed, float &x, float &mu, float &wmc,
                                                  int &idx)
{
  if (P.particles) {
    const unsigned long long *q = reinterpret_cast<const unsigned long long *>(P.particles + i);
    unsigned long long a = q[0], b = q[1], c = q[2];
    seed = a;
    x = __uint_as_float((uint32_t)b);
    mu = __uint_as_float((uint32_t)(b >> 32));
    wmc = __uint_as_float((uint32_t)c);
    idx = (int)(uint32_t)(c >> 32);
  } else {
    mcg_source_particle(P.src, P.first + i, seed, x, mu, wmc, idx);
  }
}

/* The fast arithmetic's weight update wmc <- RN(wmc - dep), with the exact
 * rounding residue (Fast2Sum: |dep| <= |wmc|) added to *wres when given: the
 * particle's weight is then the pair wmc + wres, so deposits plus final
 * weights conserve the born weight, while each deposit stays the rounded
 * product om wmc (no per-cell bias). */
__device__ __forceinline__ void mcg_fast_weight_update(float &wmc, float dep, float *wres)
{
  const float w = __fsub_rn(wmc, dep);
  if (wres)
    *wres = __fadd_rn(*wres, __fsub_rn(__fsub_rn(wmc, w), dep));
  wmc = w;
}

/* The fast step's flight: the crossing's absorption 1 - e^(-sig_a de) into
 * om_cross, and whether the flight ends in a collision before the face, the
 * event -ln(1 - u) / sig_i < de of the reference's test evaluated as
 * u < 1 - e^(-sig_i de) (no logarithm per step; the collision's distance is
 * computed only when it happens).  sig_i = 0 when it is at most EPS (never a
 * collision, as the reference's di = MAXREAL). */
__device__ __forceinline__ bool mcg_fast_flight(uint64_t seed, float sig_a, float sig_i, float de,
                                                float &om_cross)
{
  const float ta = -sig_a * de, ti = -sig_i * de;
  float p;
  if (fmaxf(fabsf(ta), fabsf(ti)) < 0x1p-7f) {
    om_cross = mcg_one_minus_exp_small(ta);
    p = mcg_one_minus_exp_small(ti);
  } else {
    om_cross = mcg_one_minus_exp_fast(ta);
    p = mcg_one_minus_exp_fast(ti);
  }
  return mcg_flight_u(seed) < p;
}

/* Distance of the fast step's collision: -ln(1 - u) / sig_i, at most de. */
__device__ __forceinline__ float mcg_fast_collision_distance(uint64_t seed, float sig_i, float de)
{
  return fminf(mcg_flight_log2(seed) * __fdividef(-0.6931472f, sig_i), de);
}

/* One Layer::particle_step (src/layer.cpp:123-190) on a lane's particle in
 * cell c = {sig_a, sig_i (fast: 0 when at most EPS), edge_lo, edge_hi}; deposits into
 * *tally_cell.  STRICT: the reference's float operations and host-libm
 * logf/expf; the crossing's absorption is computed before the logarithm and
 * a certified exponential bound settles most crossings without it (see
 * mcg_cross_threshold).  FAST: hardware log2/exp2.  THIN (strict; chains
 * whose crossings almost all have |sig_a de| < MCG_EXP_SMALL_T): the
 * certain-crossing path evaluates only the small-argument exp form and
 * leaves the rarer larger arguments to the full step. */
template <bool STRICT, int TALLY, bool THIN = false>
__device__ __forceinline__ void mcg_step(uint64_t &seed, float &x, float &mu, float &wmc,
                                         float &inv_mu, int &idx, uint32_t &nsc, const float4 c,
                                         unsigned long long *tally_cell, int qs,
                                         const mcg_libm_tab *T, const mcg_libm_dev &LM,
                                         float *l_out = nullptr,
                                         bool *coll_out = nullptr, float *dep_out = nullptr,
                                         float *wres = nullptr)
{
  const float sig_a = c.x;
  mcg_lcg_next(seed); /* the flight sample's state */
  const bool neg = mu < 0.0f;
  int inew = neg ? idx - 1 : idx + 1;
  const float edge = neg ? c.z : c.w;
  float om;
  if (STRICT) {
    /* The certain crossing, computed without branches: d_edge by the cached
     * reciprocal, the crossing's absorption by the exp evaluator, its
     * deposit, and the certified bound.  It is the reference's step exactly
     * when every condition in `easy` holds (division and exp arguments in the
     * range where those forms are exact, no exception-table candidate, a
     * deposit below 2^31 fixed-point units, a flight certainly past the
     * edge); almost every step of a fine mesh is such a crossing.  Any other
     * step takes the full step below with the same state. */
    const float a = __fsub_rn(edge, x), aa = fabsf(a);
    const float de_q = mcg_div_by_rcp(a, mu, inv_mu);
    const float t_q = __fmul_rn(-sig_a, de_q);
    /* no exception-table candidate: the midpoint distance 0.5 - |yl| 2^24
     * above the table's largest threshold tau; the thin form tests |yl|
     * against (0.5 - tau) 2^-24 (1 - 2^-21) instead, which implies it: the
     * bound's two roundings leave it below (0.5 - tau) 2^-24 (1 - 3.5e-7),
     * so 0.5 - |yl| 2^24 exceeds tau by more than 3.5e-8 for tau < 0.4,
     * more than the 2^-25 rounding of that subtraction (the host takes this
     * form only for tables with tau < 0.25, mcg_strict_thin); two
     * operations less per step */
    float d_q = 0.f, yl_q = 0.f;
    const float y_q = THIN ? mcg_exp_small_yl(t_q, &yl_q) : mcg_exp_ff_core(t_q, &d_q, T);
    const bool far_q =
        THIN ? (fabsf(yl_q) < __fmul_rn(__fsub_rn(0.5f, LM.tau_exp_max), 0x1.fffffp-25f))
             : (d_q > LM.tau_exp_max);
    const float dw_q = __fmul_rn(__fsub_rn(1.0f, y_q), wmc);
    const float v_q = __fmul_rn(dw_q, mcg_fixed_scale(qs));
    const bool t_ok = THIN ? (fabsf(t_q) < MCG_EXP_SMALL_T)
                           : ((t_q >= MCG_EXP_ONE_BOUND) & (t_q < 89.0f));
    const bool easy = (inv_mu != 0.0f) & (aa >= 0x1p-100f) & (aa <= 0x1p100f) & t_ok &
                      far_q & (__float_as_uint(v_q) < 0x4f000000u) &
                      (mcg_state_hi(seed) < mcg_cross_threshold(c.y, de_q));
    if (easy) {
      x = edge;
      wmc = __fsub_rn(wmc, dw_q);
      if (tally_cell)
        mcg_deposit_u31<TALLY>(tally_cell, v_q);
      if (l_out) {
        *l_out = de_q;
        *coll_out = false;
        *dep_out = dw_q;
      }
      idx = inew;
      return;
    }
    bool cross = true;
    float de, di = MCG_MAXREAL;
    {
      /* d_edge, and the crossing's absorption, do not depend on the flight
       * sample: start them before the logarithm */
      de = inv_mu == 0.0f ? MCG_MAXREAL
           : (aa >= 0x1p-100f && aa <= 0x1p100f) ? de_q
                                                  : __fdiv_rn(a, mu);
      const float om_cross = mcg_one_minus_expf_strict(__fmul_rn(-sig_a, de), T, LM);
      /* di = sig_i > EPS ? -log(h) / sig_i : MAXREAL; the exact value is
       * only needed when the flight may end inside the cell: the certified
       * test settles almost every crossing */
      if (c.y > MCG_EPS) {
        if (!(mcg_state_hi(seed) < mcg_cross_threshold(c.y, de))) {
          di = __fdiv_rn(-mcg_logf_strict(mcg_unit_of(seed), T, LM), c.y);
          cross = !(di < de);
        }
      } else {
        cross = !(di < de);
      }
      if (!cross) {
        inew = idx;
        x = __fadd_rn(x, __fmul_rn(di, mu));
        mu = __fsub_rn(__fmul_rn(2.0f, mcg_rnd_real(seed)), 1.0f);
        inv_mu = mcg_flight_rcp(mu);
        om = mcg_one_minus_expf_strict(__fmul_rn(-sig_a, di), T, LM);
        ++nsc;
      } else {
        x = edge;
        om = om_cross;
      }
    }
    const float dw = __fmul_rn(om, wmc);
    wmc = __fsub_rn(wmc, dw);
    if (tally_cell)
      mcg_deposit<TALLY>(tally_cell, dw, qs);
    if (l_out) {
      *l_out = cross ? de : di;
      *coll_out = !cross;
      *dep_out = dw;
    }
  } else {
    /* The common crossing without branches: a direction (|mu| > EPS), both
     * optical depths to the face below 2^-7 (the short series), no
     * collision and a deposit below 2^31 fixed-point units; it computes
     * exactly what the full step below computes for such a step. */
    const float de_q = (edge - x) * inv_mu;
    const float ta = -sig_a * de_q, ti = -c.y * de_q;
    const float dep_q = __fmul_rn(mcg_one_minus_exp_small(ta), wmc);
    const float v_q = __fmul_rn(dep_q, mcg_fixed_scale(qs));
    const bool easy = (inv_mu != 0.0f) & (fmaxf(fabsf(ta), fabsf(ti)) < 0x1p-7f) &
                      !(mcg_flight_u(seed) < mcg_one_minus_exp_small(ti)) &
                      (__float_as_uint(v_q) < 0x4f000000u);
    if (easy) {
      x = edge;
      mcg_fast_weight_update(wmc, dep_q, wres);
      if (tally_cell)
        mcg_deposit_u31<TALLY>(tally_cell, v_q);
      if (l_out) {
        *l_out = de_q;
        *coll_out = false;
        *dep_out = dep_q;
      }
      idx = inew;
      return;
    }
    const float de = inv_mu != 0.0f ? (edge - x) * inv_mu : MCG_MAXREAL;
    float om_cross;
    const bool coll = mcg_fast_flight(seed, sig_a, c.y, de, om_cross);
    const float di = coll ? mcg_fast_collision_distance(seed, c.y, de) : de;
    if (l_out) {
      *l_out = di;
      *coll_out = coll;
    }
    if (coll) {
      inew = idx;
      x = fmaf(di, mu, x);
      mu = fmaf(2.0f, mcg_rnd_real_fast(seed), -1.0f);
      inv_mu = mcg_flight_rcp(mu);
      om = mcg_one_minus_exp_fast(-sig_a * di);
      ++nsc;
    } else {
      x = edge;
      om = om_cross;
    }
    /* the deposit is the rounded product om wmc, as the reference's dw: a
     * deposit taken as the weight actually removed, wmc - RN(wmc - om wmc),
     * conserves the born weight exactly but carries the rounding of the
     * subtraction, up to half an ulp of wmc, which on a thin absorber
     * (om ~ 1e-5) is a 3e-3 relative error of the deposit, the same for
     * every uncollided particle of a cell: a systematic per-cell bias */
    const float dep = __fmul_rn(om, wmc);
    mcg_fast_weight_update(wmc, dep, wres);
    if (tally_cell)
      mcg_deposit<TALLY>(tally_cell, dep, qs);
    if (dep_out)
      *dep_out = dep;
  }
  idx = inew;
}

/* One Layer::particle_step (src/layer.cpp:123-190) on a lane's particle in
 * cell c = {sig_a, sig_i (fast: 0 when at most EPS), edge_lo, edge_hi}, in two parts, for
 * the event-based tracker: mcg_step_cross advances the state to the flight
 * sample's and completes the step when it is a certain crossing (STRICT: the
 * branch-free path of mcg_step; FAST: the flight ends past the edge),
 * returning true; otherwise it changes nothing but the seed and returns
 * false, and mcg_step_rest completes the step from the advanced state, which
 * determines the flight sample.  Together they perform exactly
 * mcg_step's operations (mcg_step, the one-piece form above, serves the
 * history-based kernels, where the split costs about 6 %).  STRICT: the reference's float operations and host-libm
 * logf/expf; the crossing's absorption is computed before the logarithm and
 * a certified exponential bound settles most crossings without it (see
 * MCG_CROSS_FACTOR).  FAST: hardware log2/exp2.  Deposits go into
 * *tally_cell; l_out/coll_out/dep_out (adjoint) receive the flight length,
 * whether it ended in a collision and the deposit. */
template <bool STRICT, int TALLY>
__device__ __forceinline__ bool mcg_step_cross(uint64_t &seed, float &x, float &mu, float &wmc,
                                               float &inv_mu, int &idx, const float4 c,
                                               unsigned long long *tally_cell, int qs,
                                               const mcg_libm_tab *T, const mcg_libm_dev &LM,
                                               float *l_out = nullptr,
                                               bool *coll_out = nullptr, float *dep_out = nullptr,
                                               float *wres = nullptr)
{
  const float sig_a = c.x;
  mcg_lcg_next(seed); /* the flight sample's state */
  const bool neg = mu < 0.0f;
  const float edge = neg ? c.z : c.w;
  if (STRICT) {
    /* The certain crossing, computed without branches: d_edge by the cached
     * reciprocal, the crossing's absorption by the exp evaluator, and the
     * certified bound.  It is the reference's step exactly when every
     * condition in `easy` holds (division and exp arguments in the range
     * where those forms are exact, no exception-table candidate, a flight
     * certainly past the edge); almost every step of a fine mesh is such a
     * crossing. */
    const float a = __fsub_rn(edge, x), aa = fabsf(a);
    const float de_q = mcg_div_by_rcp(a, mu, inv_mu);
    const float t_q = __fmul_rn(-sig_a, de_q);
    float d_q;
    const float y_q = mcg_exp_ff_core(t_q, &d_q, T);
    const bool easy = (inv_mu != 0.0f) & (aa >= 0x1p-100f) & (aa <= 0x1p100f) &
                      (t_q >= MCG_EXP_ONE_BOUND) & (t_q < 89.0f) & (d_q > LM.tau_exp_max) &
                      (mcg_state_hi(seed) < mcg_cross_threshold(c.y, de_q));
    if (!easy)
      return false;
    x = edge;
    const float dw = __fmul_rn(__fsub_rn(1.0f, y_q), wmc);
    wmc = __fsub_rn(wmc, dw);
    if (tally_cell)
      mcg_deposit<TALLY>(tally_cell, dw, qs);
    if (l_out) {
      *l_out = de_q;
      *coll_out = false;
      *dep_out = dw;
    }
  } else {
    const float de = inv_mu != 0.0f ? (edge - x) * inv_mu : MCG_MAXREAL;
    float om;
    if (mcg_fast_flight(seed, sig_a, c.y, de, om))
      return false;
    if (l_out) {
      *l_out = de;
      *coll_out = false;
    }
    x = edge;
    /* the deposit is the rounded product om wmc, as the reference's dw: a
     * deposit taken as the weight actually removed, wmc - RN(wmc - om wmc),
     * conserves the born weight exactly but carries the rounding of the
     * subtraction, up to half an ulp of wmc, which on a thin absorber
     * (om ~ 1e-5) is a 3e-3 relative error of the deposit, the same for
     * every uncollided particle of a cell: a systematic per-cell bias */
    const float dep = __fmul_rn(om, wmc);
    mcg_fast_weight_update(wmc, dep, wres);
    if (tally_cell)
      mcg_deposit<TALLY>(tally_cell, dep, qs);
    if (dep_out)
      *dep_out = dep;
  }
  idx = neg ? idx - 1 : idx + 1;
  return true;
}

template <bool STRICT, int TALLY>
__device__ __forceinline__ void mcg_step_rest(uint64_t &seed, float &x, float &mu,
                                              float &wmc, float &inv_mu, int &idx, uint32_t &nsc,
                                              const float4 c, unsigned long long *tally_cell,
                                              int qs, const mcg_libm_tab *T,
                                              const mcg_libm_dev &LM, float *l_out = nullptr,
                                              bool *coll_out = nullptr, float *dep_out = nullptr,
                                              float *wres = nullptr)
{
  const float sig_a = c.x;
  const bool neg = mu < 0.0f;
  int inew = neg ? idx - 1 : idx + 1;
  const float edge = neg ? c.z : c.w;
  float om;
  if (STRICT) {
    const float a = __fsub_rn(edge, x), aa = fabsf(a);
    const float de = inv_mu == 0.0f ? MCG_MAXREAL
                     : (aa >= 0x1p-100f && aa <= 0x1p100f) ? mcg_div_by_rcp(a, mu, inv_mu)
                                                            : __fdiv_rn(a, mu);
    /* di = sig_i > EPS ? -log(h) / sig_i : MAXREAL; the exact value is
     * only needed when the flight may end inside the cell: the certified
     * test settles almost every crossing */
    bool cross = true;
    float di = MCG_MAXREAL;
    if (c.y > MCG_EPS) {
      if (!(mcg_state_hi(seed) < mcg_cross_threshold(c.y, de))) {
        di = __fdiv_rn(-mcg_logf_strict(mcg_unit_of(seed), T, LM), c.y);
        cross = !(di < de);
      }
    } else {
      cross = !(di < de);
    }
    /* one exponential, of the length that the step takes */
    om = mcg_one_minus_expf_strict(__fmul_rn(-sig_a, cross ? de : di), T, LM);
    if (!cross) {
      inew = idx;
      x = __fadd_rn(x, __fmul_rn(di, mu));
      mu = __fsub_rn(__fmul_rn(2.0f, mcg_rnd_real(seed)), 1.0f);
      inv_mu = mcg_flight_rcp(mu);
      ++nsc;
    } else {
      x = edge;
    }
    const float dw = __fmul_rn(om, wmc);
    wmc = __fsub_rn(wmc, dw);
    if (tally_cell)
      mcg_deposit<TALLY>(tally_cell, dw, qs);
    if (l_out) {
      *l_out = cross ? de : di;
      *coll_out = !cross;
      *dep_out = dw;
    }
  } else {
    const float de = inv_mu != 0.0f ? (edge - x) * inv_mu : MCG_MAXREAL;
    float om_cross;
    const bool coll = mcg_fast_flight(seed, sig_a, c.y, de, om_cross);
    const float di = coll ? mcg_fast_collision_distance(seed, c.y, de) : de;
    if (l_out) {
      *l_out = di;
      *coll_out = coll;
    }
    if (coll) {
      inew = idx;
      x = fmaf(di, mu, x);
      mu = fmaf(2.0f, mcg_rnd_real_fast(seed), -1.0f);
      inv_mu = mcg_flight_rcp(mu);
      om = mcg_one_minus_exp_fast(-sig_a * di);
      ++nsc;
    } else {
      x = edge;
      om = om_cross;
    }
    const float dep = __fmul_rn(om, wmc);
    mcg_fast_weight_update(wmc, dep, wres);
    if (tally_cell)
      mcg_deposit<TALLY>(tally_cell, dep, qs);
    if (dep_out)
      *dep_out = dep;
  }
  idx = inew;
}

/* ---------------------------------------------------------------- tiles
 * A tile is up to TW consecutive certain crossings of one flight.  Along a
 * flight nothing but the weight is serial: the cells, the random numbers (the
 * LCG jumps ahead), the face-to-face lengths and the absorbed fractions of the
 * next TW cells are independent.  A warp holds 32 histories, one per lane,
 * and advances each by one tile per round:
 *   1. every lane with a history that can run puts its flight in shared memory;
 *   2. a few flights at a time, G lanes each: lane j forms the absorbed
 *      fractions of steps j and j + G, as pairs of the packed f32x2
 *      operations, and whether each is certainly a crossing;
 *   3. lane = history again: the weights in order, w <- w - RN(om w), up to the
 *      first step that is not certain, which gives the deposits;
 *   4. a few flights at a time, lane j adds the deposits of steps j and j + G
 *      to the tally.
 * Against one lane per history through the whole step this makes the cell
 * loads and the tally atomics runs of consecutive cells (with scattered lanes
 * the L1 was the bound: 18 of 19 cycles of a warp step on the 10,000-cell
 * slab), keeps the lanes busy whatever the histories do, and a single history
 * takes about 100 cycles per step (3200 per tile of 32) instead of 300 to 500, which
 * is what the end of a launch waits for.  Every step is exactly mcg_step_cross's. */
/* Lanes per flight in phases 2 and 4 (G) and steps of a tile (2 G).  Thin chains
 * take 16 and 32: fewer rounds and shared-memory rows per step; others 8 and
 * 16: their flights are short, and what a tile has after its flight's end is
 * lost. */
template <bool THIN> struct mcg_tile_shape {
  static constexpr int G = THIN ? 16 : 8, TW = 2 * G, F = 32 / G; /* F: flights at a time */
  static constexpr int PLANE = G * 33;
};
#define MCG_TW_MAX 32
#define MCG_THIN_BLOCK 768 /* most threads of a thin kernel: 85 registers */

/* A warp's shared memory: the flights, and one fraction (then deposit) per
 * step: step i of flight r at (i / G) PLANE + (r / F) 33 + (r % F) G + i % G,
 * consecutive over the lanes of phases 2 and 4 and free of bank conflicts down
 * the steps of 32 flights (phase 3). */
template <bool THIN> struct mcg_tile_smem {
  uint4 flight[32]; /* state << 1; THIN: the flight's bounds on g and |r| */
  float4 slant[32]; /* |mu| twice, -|RN(1 / mu)| twice */
  int4 place[32];   /* length to the first face (inf: the cell's), cell, direction, steps taken */
  float step[2 * mcg_tile_shape<THIN>::PLANE];
};

/* LOSS (not THIN): and the loss weight of each step's cell. */
struct mcg_loss_smem : mcg_tile_smem<false> {
  float weight[2 * mcg_tile_shape<false>::PLANE];
};

/* Jumps of the sample stream in the shifted representation (state << 1, so the
 * modulus is the word's): s -> A s + C after k steps. */
struct mcg_real_jumps {
  unsigned long long A[MCG_TW_MAX + 1], C[MCG_TW_MAX + 1];
};

__device__ __forceinline__ void mcg_fill_real_jumps(mcg_real_jumps *J)
{
  for (int k = threadIdx.x; k <= MCG_TW_MAX; k += blockDim.x) {
    const uint64_t c = mcg_lcg_skip(0ull, (uint64_t)k, 0);
    J->A[k] = (mcg_lcg_skip(1ull, (uint64_t)k, 0) - c) & MCG_MASK63;
    J->C[k] = c << 1;
  }
}

/* A warp's view: its shared memory, and its lanes' jumps of j + 1 and
 * G + j + 1 steps. */
template <bool THIN> struct mcg_tile_warp {
  mcg_tile_smem<THIN> *S;
  uint64_t A0, C0, A1, C1;

  __device__ __forceinline__ mcg_tile_warp(mcg_tile_smem<THIN> *s, const mcg_real_jumps *J)
  {
    constexpr int G = mcg_tile_shape<THIN>::G;
    const int lane = threadIdx.x & 31, j = lane & (G - 1);
    S = s;
    A0 = J->A[j + 1], C0 = J->C[j + 1], A1 = J->A[G + j + 1], C1 = J->C[G + j + 1];
    S->place[lane] = make_int4(0, 0, 0, 0); /* a row not yet used reads cell 0 */
  }
};

/* Pairs of floats in one 64-bit register: one instruction for two IEEE
 * operations (round to nearest, subnormals kept). */
typedef unsigned long long mcg_f2;
__device__ __forceinline__ mcg_f2 f2_make(float a, float b)
{
  mcg_f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ mcg_f2 f2_both(float a) { return f2_make(a, a); }
__device__ __forceinline__ void f2_get(mcg_f2 v, float &a, float &b)
{
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ mcg_f2 f2_mul(mcg_f2 a, mcg_f2 b)
{
  mcg_f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ mcg_f2 f2_add(mcg_f2 a, mcg_f2 b)
{
  mcg_f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ mcg_f2 f2_fma(mcg_f2 a, mcg_f2 b, mcg_f2 c)
{
  mcg_f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

/* Certain crossing by the linear bound: with g = 1 + floor(s / 2^40) 2^-23
 * (the state's top 23 bits as the float of [1, 2) below 1 + h),
 *     g < RN(K - sig_i de),  K = 2 - 2^-20,
 * gives h <= g - 1 + 2^-23 <= 1 - T - 2^-20 + 2^-23 + 2^-24, T = sig_i de
 * exactly (T <= 1, since g >= 1), hence -ln h >= 1 - h >= T + 2^-20.5 and
 * -logf(h) >= (T + 2^-20.5)(1 - 2^-22) > T: the reference's flight passes the
 * face (the reasoning of mcg_cross_threshold, with the tangent of e^-T
 * instead of a MUFU operation).  FAST: 1 - h exceeds the computed collision
 * probability, at most T (1 + 2^-20).  It fails on T + 1e-6 of the crossings
 * where the exponential one fails on 1 - e^-T + 6e-5. */
#define MCG_TILE_K (2.0f - 0x1p-20f)

/* One certain crossing of a lane's particle (the gradient kernels): completes
 * the step, with its length and deposit, when it is certainly a crossing that
 * the tiles' forms reproduce bit for bit; otherwise changes nothing and returns
 * false (the step is mcg_full's).  14 operations for the absorbed fraction
 * instead of the evaluator's 17 to 40, and 3 for the collision bound. */
template <bool STRICT>
__device__ __forceinline__ bool mcg_cross(uint64_t &seed, float &x, float mu, float &wmc, float inv_mu,
                                          int &idx, const float4 c, float b_mid, float &len, float &dep)
{
  const uint64_t s = MCG_RNG_G * seed + MCG_RNG_C;
  const float g = __uint_as_float(0x3f800000u | ((uint32_t)(s >> 40) & 0x007fffffu));
  const bool neg = mu < 0.0f;
  const float edge = neg ? c.z : c.w;
  const float a = __fsub_rn(edge, x), aa = fabsf(a);
  bool easy = inv_mu != 0.0f;
  float om;
  if (STRICT) {
    len = mcg_div_by_rcp(a, mu, inv_mu);
    const float u = __fmul_rn(c.x, len);
    float r;
    om = mcg_om_mid(u, __fmul_rn(u, u), &r);
    easy &= (aa >= 0x1p-100f) & (aa <= 0x1p100f) & (fabsf(r) < b_mid) &
            (__float_as_uint(u) < __float_as_uint(MCG_OM_MID_MAX)) &
            (g < __fmaf_rn(-c.y, len, MCG_TILE_K));
  } else {
    len = __fmul_rn(a, inv_mu);
    const float u = __fmul_rn(c.x, len), ti = __fmul_rn(c.y, len);
    om = fmaxf(u, ti) < 0x1p-7f ? mcg_one_minus_exp_small(-u) : mcg_one_minus_exp_fast(-u);
    easy &= (__float_as_uint(u) < 0x3e800000u) & (g < __fsub_rn(MCG_TILE_K, ti));
  }
  if (!easy)
    return false;
  seed = s & MCG_MASK63;
  x = edge;
  dep = __fmul_rn(om, wmc);
  wmc = __fsub_rn(wmc, dep);
  idx = neg ? idx - 1 : idx + 1;
  return true;
}

/* Rounds of the gradient kernels: certain crossings of a lane between two votes
 * of the warp, lanes (of 32 with a history) waiting for the full step that
 * trigger it, lanes that have ended a pass or want a history that end the round.  1000 cells, 2e6 histories:
 * windows of 1 to 8 and pools of 2 to 8 lie within 4 % of these, pools of 1 or 12
 * are 6 to 13 % slower.  Long windows with small pools let colliding histories fall
 * behind, and the gradients' float sums notice (mcg_adjoint_fused). */
#define MCG_GRAD_WINDOW 2
#define MCG_GRAD_POOL 4
#define MCG_GRAD_REFILL 1

/* float-float accumulation s += v (TwoSum) */
__device__ __forceinline__ void mcg_ff_add(float &hi, float &lo, float v)
{
  const float s = __fadd_rn(hi, v);
  const float bv = __fsub_rn(s, hi);
  const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bv)), __fsub_rn(v, bv));
  hi = s;
  lo = __fadd_rn(lo, e);
}

/* Two steps of a flight (packed): their absorbed fractions of the weight, NaN
 * where a step is not certainly a crossing that this form reproduces bit for
 * bit.  a: lengths to the faces along x; amu, ny: |mu| and -|RN(1 / mu)|, both
 * twice.  With the reciprocal's sign turned every quantity that the series
 * need negative comes out negative (roundings are symmetric): lengths and
 * fractions are returned negated.
 * THIN: the collision bound (thr) and the midpoint bound are the flight's,
 * taken at the chain's widest cell, and its largest u is below the thin
 * form's limit (mcg_thin_tests). */
template <bool STRICT, bool THIN>
__device__ __forceinline__ void mcg_tile_steps(mcg_f2 a, mcg_f2 amu, mcg_f2 ny, mcg_f2 sig_a,
                                               mcg_f2 sig_i, uint32_t s_hi0, uint32_t s_hi1,
                                               float thr, float bound, const mcg_run_consts &R,
                                               float &nom0, float &nom1, mcg_f2 &nde)
{
  const float g0 = __uint_as_float(__funnelshift_r(s_hi0, 0x7fu, 9));
  const float g1 = __uint_as_float(__funnelshift_r(s_hi1, 0x7fu, 9));
  bool ok0, ok1;
  mcg_f2 nom;
  if (STRICT) {
    /* mcg_div_by_rcp, mcg_om_thin / mcg_om_mid in pairs */
    const mcg_f2 nq = f2_mul(a, ny);
    nde = f2_fma(f2_fma(amu, nq, a), ny, nq);
    const mcg_f2 nu = f2_mul(sig_a, nde), uu = f2_mul(nu, nu);
    mcg_f2 r; /* of either sign */
    if (THIN) {
      const mcg_f2 w = f2_fma(nu, f2_both(1.0f / 6.0f), f2_both(0.5f));
      nom = f2_add(f2_add(f2_fma(uu, w, nu), f2_both(-0.75f)), f2_both(0.75f));
      r = f2_fma(uu, w, f2_fma(nom, f2_both(-1.0f), nu));
    } else {
      mcg_f2 p = f2_fma(nu, f2_both(1.0f / 720.0f), f2_both(1.0f / 120.0f));
      p = f2_fma(nu, p, f2_both(1.0f / 24.0f));
      p = f2_fma(nu, p, f2_both(1.0f / 6.0f));
      nom = f2_fma(uu, f2_fma(nu, p, f2_both(0.5f)), nu);
      nom = f2_add(f2_add(nom, f2_both(-0.75f)), f2_both(0.75f));
      const mcg_f2 ne = f2_fma(f2_mul(nu, f2_both(-1.0f)), nu, uu); /* uu - u^2 */
      mcg_f2 nd = f2_fma(f2_both(0.5f), uu, f2_fma(nom, f2_both(-1.0f), nu));
      nd = f2_fma(f2_both(-0.5f), ne, nd);
      r = f2_fma(f2_mul(uu, nu), p, nd);
    }
    float r0, r1;
    f2_get(r, r0, r1);
    if (THIN) {
      ok0 = (fabsf(r0) < bound) & (g0 < thr);
      ok1 = (fabsf(r1) < bound) & (g1 < thr);
    } else {
      float u0, u1, t0, t1;
      f2_get(nu, u0, u1);
      f2_get(f2_fma(sig_i, nde, f2_both(MCG_TILE_K)), t0, t1);
      ok0 = (fabsf(r0) < R.b_mid) & (fabsf(u0) < MCG_OM_MID_MAX) & (g0 < t0);
      ok1 = (fabsf(r1) < R.b_mid) & (fabsf(u1) < MCG_OM_MID_MAX) & (g1 < t1);
    }
  } else {
    /* mcg_one_minus_exp_small and, not THIN, mcg_one_minus_exp_fast of -u */
    nde = f2_mul(a, ny);
    const mcg_f2 nu = f2_mul(sig_a, nde);
    mcg_f2 p = f2_fma(nu, f2_both(1.0f / 6.0f), f2_both(0.5f));
    p = f2_fma(nu, p, f2_both(1.0f));
    nom = f2_mul(nu, p);
    if (THIN) {
      ok0 = g0 < thr;
      ok1 = g1 < thr;
    } else {
      float u0, u1, t0, t1, s0, s1, l0, l1;
      f2_get(nu, u0, u1);
      f2_get(f2_mul(sig_i, nde), t0, t1);
      p = f2_fma(nu, f2_both(1.0f / 5040.0f), f2_both(1.0f / 720.0f));
      p = f2_fma(nu, p, f2_both(1.0f / 120.0f));
      p = f2_fma(nu, p, f2_both(1.0f / 24.0f));
      p = f2_fma(nu, p, f2_both(1.0f / 6.0f));
      p = f2_fma(nu, p, f2_both(0.5f));
      p = f2_fma(nu, p, f2_both(1.0f));
      f2_get(f2_mul(nu, p), l0, l1);
      f2_get(nom, s0, s1);
      nom = f2_make(fminf(u0, t0) > -0x1p-7f ? s0 : l0, fminf(u1, t1) > -0x1p-7f ? s1 : l1);
      ok0 = (u0 > -0.25f) & (g0 < __fadd_rn(MCG_TILE_K, t0));
      ok1 = (u1 > -0.25f) & (g1 < __fadd_rn(MCG_TILE_K, t1));
    }
  }
  f2_get(nom, nom0, nom1);
  nom0 = ok0 ? nom0 : __int_as_float(0x7fc00000);
  nom1 = ok1 ? nom1 : __int_as_float(0x7fc00000);
}

/* The bounds of a flight on a thin chain from its widest cell (R.w_a, R.w_i:
 * the chain's largest sig_a and sig_i widths, over the lengths of the table): {thr, bound} of
 * mcg_tile_steps, which no step passes when the flight is so slanted that its
 * steps may leave the thin form's range or its first deposit 31 bits.  The
 * factor covers the roundings of the lengths and products. */
template <bool STRICT>
__device__ __forceinline__ float2 mcg_thin_tests(float inv_mu, float wmc, const mcg_run_consts &R)
{
  const float y = fabsf(inv_mu) * (1.0f + 0x1p-20f);
  const float u = __fmul_rn(R.w_a, y), ti = __fmul_rn(R.w_i, y);
  const bool ok = (STRICT ? u < MCG_OM_THIN_MAX : fmaxf(u, ti) < 0x1p-7f) &
                  (__fmul_rn(u, __fmul_rn(wmc, R.scale)) < 0x1p31f);
  return make_float2(ok ? __fsub_rn(MCG_TILE_K, ti) : -1.0f,
                     __fmaf_rn(__fmul_rn(u, u), -R.c_thin, R.b_thin));
}

/* Adds a deposit q to the 32-bit tally of a thin chain (MCG_TALLY_LO32): the
 * low words are in shared memory, and what passes them goes to the global
 * 64-bit tally at once.  A carry every 2^32 / q deposits (q about 2e6 at
 * scale 2^35, 6e7 at 2^40) costs less than shared memory for 64 bits per cell,
 * which takes it from the cell table's L1 and from more warps. */
__device__ __forceinline__ void mcg_lo32_add(unsigned *lo, unsigned long long *global, long long q)
{
  const uint32_t v = (uint32_t)q, old = atomicAdd(lo, v);
  const uint64_t hi = (uint64_t)(q >> 32) + ((uint32_t)(old + v) < old ? 1u : 0u);
  if (hi)
    atomicAdd(global, (unsigned long long)(hi << 32));
}

/* Shared-memory add under a predicate (no branch); the old value, or 0. */
__device__ __forceinline__ uint32_t mcg_shared_add_if(bool p, uint32_t addr, uint32_t v)
{
  uint32_t old;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\tmov.u32 %0, 0;\n\t"
               "@p atom.shared.add.u32 %0, [%1], %2;\n\t}"
               : "=r"(old)
               : "r"(addr), "r"(v), "r"((int)p)
               : "memory");
  return old;
}

/* The lesser of two floats, NaN if either is. */
__device__ __forceinline__ float mcg_min_nan(float a, float b)
{
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

/* Phase 2 for U passes of F flights from pass q0.  All loads come before the
 * first store, which the compiler could not tell apart from the next pass's
 * rows: 4 passes in flight instead of 1 took the 10,000-cell slab from 131 to
 * 110 ms per 5e6 histories (the table's L1 misses).  Rows past the last flight
 * are computed and never used.  The minimum keeps a cell's NaN length (a step for
 * the full form): on flights under way fminf made it inf, which the fast thin
 * form, testing the collision bound alone, accepted. */
template <bool STRICT, bool THIN, int U, bool LOSS>
__device__ __forceinline__ void mcg_tile_form(mcg_tile_smem<THIN> *S, int q0, const mcg_tab &tab,
                                              const mcg_tile_warp<THIN> &B,
                                              const mcg_run_consts &R)
{
  constexpr int G = mcg_tile_shape<THIN>::G, F = 32 / G, PLANE = mcg_tile_shape<THIN>::PLANE;
  const int lane = threadIdx.x & 31, sub = lane / G, j = lane & (G - 1);
  int4 pl[U];
  uint4 fl[U];
  ulonglong2 sl[U];
  float a[U], b[U], sa0[U], sa1[U], si0[U], si1[U], om0[U], om1[U], w0[U], w1[U];
#pragma unroll
  for (int v = 0; v < U; ++v)
    pl[v] = S->place[F * (q0 + v) + sub];
#pragma unroll
  for (int v = 0; v < U; ++v)
    if (THIN) {
      const float2 *p = tab.thin + (pl[v].y + j * pl[v].z);
      const float2 c = __ldg(p), d = __ldg(p + G * pl[v].z);
      sa0[v] = c.x, sa1[v] = d.x, a[v] = c.y, b[v] = d.y;
      si0[v] = si1[v] = 0.0f;
    } else {
      const float4 *p = tab.cell + (pl[v].y + j * pl[v].z);
      const float4 c = __ldg(p), d = __ldg(p + G * pl[v].z);
      sa0[v] = c.x, sa1[v] = d.x, si0[v] = c.y, si1[v] = d.y;
      a[v] = pl[v].z < 0 ? c.w : c.z, b[v] = pl[v].z < 0 ? d.w : d.z;
      if (LOSS) {
        const float2 *w = tab.aux + (pl[v].y + j * pl[v].z);
        w0[v] = __ldg(&w->x), w1[v] = __ldg(&(w + G * pl[v].z)->x);
      }
    }
#pragma unroll
  for (int v = 0; v < U; ++v) {
    fl[v] = S->flight[F * (q0 + v) + sub];
    sl[v] = *reinterpret_cast<const ulonglong2 *>(&S->slant[F * (q0 + v) + sub]);
  }
#pragma unroll
  for (int v = 0; v < U; ++v) {
    const uint64_t s = (uint64_t)fl[v].y << 32 | fl[v].x;
    const uint64_t n0 = B.A0 * s + B.C0, n1 = B.A1 * s + B.C1;
    mcg_f2 nde;
    mcg_tile_steps<STRICT, THIN>(
        f2_make(mcg_min_nan(a[v], __int_as_float(j ? 0x7f800000 : pl[v].x)), b[v]), sl[v].x, sl[v].y,
        f2_make(sa0[v], sa1[v]), f2_make(si0[v], si1[v]), (uint32_t)(n0 >> 32),
        (uint32_t)(n1 >> 32), __uint_as_float(fl[v].z), __uint_as_float(fl[v].w), R, om0[v], om1[v],
        nde);
  }
#pragma unroll
  for (int v = 0; v < U; ++v) {
    S->step[33 * (q0 + v) + lane] = om0[v];
    S->step[PLANE + 33 * (q0 + v) + lane] = om1[v];
    if (LOSS) {
      float *w = static_cast<mcg_loss_smem *>((mcg_tile_smem<false> *)S)->weight;
      w[33 * (q0 + v) + lane] = w0[v];
      w[PLANE + 33 * (q0 + v) + lane] = w1[v];
    }
  }
}

/* 64-bit shared-memory add under a predicate.  On batched slabs, whose
 * deposits often pass 32 bits, it is the cheaper form (4096 slabs, 3.1e7
 * histories, strict: 197 ms against 215 with 32-bit halves and a carry); on a
 * chain where a point source makes many lanes add to the same cells it is the
 * dearer one (1000 cells, 1e6 histories, fast: 2.34 ms against 2.02). */
__device__ __forceinline__ void mcg_shared_red_if(bool p, uint32_t addr, uint64_t v)
{
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p red.shared.add.u64 [%0], %1;\n\t}"
               :
               : "r"(addr), "l"(v), "r"((int)p)
               : "memory");
}

/* A deposit of scaled value v, 0 <= v < 2^63, as the 64-bit integer
 * llrint(v): from 2^31 on v is an integer, so it is its shifted significand
 * (the 64-bit conversion issues on the FP64 pipe). */
__device__ __forceinline__ uint64_t mcg_fixed_u63(float v)
{
  const uint32_t b = __float_as_uint(v);
  return v < 0x1p31f ? (uint64_t)__float2uint_rn(v)
                     : (uint64_t)((b & 0x007fffffu) | 0x00800000u) << (b >> 23) - 150u;
}

/* Where the deposits of a warp's tiles go: TALLY and its base, such that base
 * + 8 cell is a cell's word in shared memory (MCG_TALLY_GLOBAL: unused), and
 * the global tally for the rows marked so. */
struct mcg_sink {
  uint32_t shared;            /* shared-memory address of cell 0's word (THIN: of its low word) */
  unsigned long long *global; /* cell 0's word of the global tally */
};

/* Phase 4 for U passes from pass q0. */
template <bool THIN, int TALLY, bool MULTI, int U>
__device__ __forceinline__ void mcg_tile_add(mcg_tile_smem<THIN> *S, int q0, const mcg_sink &D)
{
  constexpr int G = mcg_tile_shape<THIN>::G, F = 32 / G, PLANE = mcg_tile_shape<THIN>::PLANE;
  const int lane = threadIdx.x & 31, sub = lane / G, j = lane & (G - 1);
  int4 pl[U];
  float v[2 * U];
  int at[2 * U];
  bool in[2 * U];
#pragma unroll
  for (int k = 0; k < U; ++k) {
    pl[k] = S->place[F * (q0 + k) + sub];
    v[2 * k] = S->step[33 * (q0 + k) + lane];
    v[2 * k + 1] = S->step[PLANE + 33 * (q0 + k) + lane];
    at[2 * k] = pl[k].y + j * pl[k].z;
    at[2 * k + 1] = at[2 * k] + G * pl[k].z;
    in[2 * k] = j < pl[k].w;
    in[2 * k + 1] = j + G < pl[k].w;
  }
  if (TALLY == MCG_TALLY_LO32) {
    bool carry[2 * U], any = false;
#pragma unroll
    for (int k = 0; k < 2 * U; ++k) {
      const uint32_t d = __float2uint_rn(v[k]);
      const uint32_t old = mcg_shared_add_if(in[k], D.shared + 4 * at[k], d);
      any |= carry[k] = (uint32_t)(old + d) < old;
    }
    if (__any_sync(0xffffffffu, any)) {
#pragma unroll
      for (int k = 0; k < 2 * U; ++k)
        if (carry[k])
          atomicAdd(D.global + at[k], 1ull << 32);
    }
  } else {
    bool far[2 * U], any_far = false, wide = false;
    uint64_t d[2 * U];
#pragma unroll
    for (int k = 0; k < 2 * U; ++k) {
      far[k] = in[k] && (TALLY == MCG_TALLY_GLOBAL || (MULTI && pl[k / 2].x));
      any_far |= far[k];
      d[k] = __float2uint_rn(v[k]);
      wide |= in[k] & !(v[k] < 0x1p31f);
    }
    if (__any_sync(0xffffffffu, wide)) {
#pragma unroll
      for (int k = 0; k < 2 * U; ++k)
        d[k] = mcg_fixed_u63(v[k]);
    }
    if (TALLY == MCG_TALLY_SMEM64) {
#pragma unroll
      for (int k = 0; k < 2 * U; ++k)
        mcg_shared_red_if(in[k] & !far[k], D.shared + 8 * at[k], d[k]);
    }
    if (TALLY == MCG_TALLY_SMEM32) {
      uint32_t hi[2 * U], more = 0u;
#pragma unroll
      for (int k = 0; k < 2 * U; ++k) {
        const bool here = in[k] & !far[k];
        const uint32_t lo = (uint32_t)d[k];
        const uint32_t old = mcg_shared_add_if(here, D.shared + 8 * at[k], lo);
        hi[k] = (here ? (uint32_t)(d[k] >> 32) : 0u) + ((uint32_t)(old + lo) < old ? 1u : 0u);
        more |= hi[k];
      }
      if (__any_sync(0xffffffffu, more != 0u)) {
#pragma unroll
        for (int k = 0; k < 2 * U; ++k)
          if (hi[k])
            mcg_shared_add_if(true, D.shared + 8 * at[k] + 4, hi[k]);
      }
    }
    if (TALLY == MCG_TALLY_GLOBAL || (MULTI && __any_sync(0xffffffffu, any_far))) {
#pragma unroll
      for (int k = 0; k < 2 * U; ++k)
        if (far[k])
          atomicAdd(D.global + at[k], (unsigned long long)d[k]);
    }
  }
}

/* The tile ends at the step that takes the weight below the minimum (scaled):
 * weights only fall, so the last one tells whether there is such a step. */
template <bool STRICT, bool THIN>
__device__ __forceinline__ void mcg_tile_cut(const float *st, int &n, float &W, float &res,
                                             float W0, float res0, float min_w)
{
  constexpr int G = mcg_tile_shape<THIN>::G, PLANE = mcg_tile_shape<THIN>::PLANE;
  if (W < min_w) {
    W = W0;
    res = res0;
    for (int i = 0; i < n; ++i) {
      const float dv = st[(i / G) * PLANE + i % G], w2 = __fsub_rn(W, dv);
      if (!STRICT)
        res = __fadd_rn(res, __fsub_rn(__fsub_rn(W, w2), dv));
      W = w2;
      if (W < min_w)
        n = i + 1; /* ends the loop */
    }
  }
}

/* One round over the warp (all lanes call): the lanes with `can` advance their
 * flights by up to nmax (1 .. TW) certain crossings and return their
 * number; a0: length to the first face when the flight starts inside the cell,
 * else infinity; W is the weight times the tally scale (or 1, mcg_run_consts), res
 * (fast) its residue, `down` the inverse of that scale; test: mcg_thin_tests
 * (THIN); far (MULTI): this flight's deposits go to the global tally.  idx indexes
 * tab, the tile table, and the tallies.  LOSS: adds w_c dep of every step to the
 * float-float sum (G_hi, G_lo), in order; res is left alone. */
template <bool STRICT, bool THIN, int TALLY, bool MULTI, bool LOSS>
__device__ __forceinline__ int mcg_tiles(bool can, uint64_t s2, float amu, float ainv, float a0,
                                         int dir, int idx, int nmax, float2 test, float &W,
                                         float &res, float &G_hi, float &G_lo, bool far, float down,
                                         const mcg_tab &tab, const mcg_sink &D, const mcg_tile_warp<THIN> &B,
                                         const mcg_run_consts &R)
{
  constexpr int G = mcg_tile_shape<THIN>::G, TW = 2 * G, F = 32 / G;
  constexpr int PLANE = mcg_tile_shape<THIN>::PLANE;
  mcg_tile_smem<THIN> *S = B.S;
  const int lane = threadIdx.x & 31;
  const unsigned mask = __ballot_sync(0xffffffffu, can);
  const int cnt = __popc(mask), rank = __popc(mask & lanemask_lt());
  S->place[lane].w = 0; /* rows past the last flight: no deposits */
  if (can) {
    S->flight[rank] = make_uint4((uint32_t)s2, (uint32_t)(s2 >> 32), __float_as_uint(test.x),
                                 __float_as_uint(test.y));
    S->slant[rank] = make_float4(amu, amu, -ainv, -ainv);
    S->place[rank] = make_int4(__float_as_int(a0), THIN && dir < 0 ? idx + tab.left : idx, dir, 0);
  }
  __syncwarp();
  /* An odd last pass goes alone, which is what the end of a launch waits for, a
   * history or two per warp at 3000 cycles per round: 100 cells, 1e5 histories,
   * strict 328 -> 295 us.  Not in batched slabs, which run at full warps (201 ms
   * against 206 with it), nor for the deposits of thin chains (the workers'
   * kernel 34.9 ms against 33.4). */
  int q = 0;
  if (THIN)
    for (; F * (q + 2) < cnt; q += 4)
      mcg_tile_form<STRICT, THIN, 4, LOSS>(S, q, tab, B, R);
  for (; F * (MULTI ? q : q + 1) < cnt; q += 2)
    mcg_tile_form<STRICT, THIN, 2, LOSS>(S, q, tab, B, R);
  if (!MULTI && F * q < cnt)
    mcg_tile_form<STRICT, THIN, 1, LOSS>(S, q, tab, B, R);
  __syncwarp();
  int n = 0;
  if (can) {
    const float W0 = W, res0 = res;
    float *st = S->step + 33 * (rank / F) + G * (rank % F);
    if (nmax < TW)
      st[(nmax / G) * PLANE + nmax % G] = __int_as_float(0x7fc00000);
    if (THIN) {
      /* unconditionally, with the last valid weight kept every eight steps
       * (from the first NaN on everything is NaN); the rest of an early end
       * again from there */
      float w = W, rs = res;
#pragma unroll
      for (int i = 0; i < TW; ++i) {
        float *si = st + (i / G) * PLANE + i % G;
        const float dv = __fmul_rn(-*si, w), w2 = __fsub_rn(w, dv);
        if (!STRICT)
          rs = __fadd_rn(rs, __fsub_rn(__fsub_rn(w, w2), dv));
        w = w2;
        *si = dv;
        if (i % 8 == 7 && w == w) {
          W = w;
          res = rs;
          n = i + 1;
        }
      }
      for (; n < TW; ++n) {
        const float dv = st[(n / G) * PLANE + n % G];
        if (dv != dv)
          break;
        const float w2 = __fsub_rn(W, dv);
        if (!STRICT)
          res = __fadd_rn(res, __fsub_rn(__fsub_rn(W, w2), dv));
        W = w2;
      }
      mcg_tile_cut<STRICT, THIN>(st, n, W, res, W0, res0, R.min_w);
      S->place[rank] = make_int4(0, idx, dir, n); /* phase 4: the cell, of either direction */
    } else {
      bool ok = true;
      const float *wt = nullptr;
      const float G0_hi = G_hi, G0_lo = G_lo;
      if (LOSS)
        wt = static_cast<mcg_loss_smem *>((mcg_tile_smem<false> *)S)->weight + (st - S->step);
#pragma unroll
      for (int i = 0; i < TW; ++i) {
        float *si = st + (i / G) * PLANE + i % G;
        const float dv = __fmul_rn(-*si, W);
        ok &= dv < 0x1p62f; /* false for NaN */
        if (ok) {
          const float w2 = __fsub_rn(W, dv);
          if (!STRICT && !LOSS)
            res = __fadd_rn(res, __fsub_rn(__fsub_rn(W, w2), dv));
          W = w2;
          *si = dv;
          n = i + 1;
          if (LOSS)
            mcg_ff_add(G_hi, G_lo,
                       __fmul_rn(wt[(i / G) * PLANE + i % G], __fmul_rn(dv, down)));
        }
      }
      const bool cut = W < R.min_w;
      mcg_tile_cut<STRICT, THIN>(st, n, W, res, W0, res0, R.min_w);
      if (LOSS && cut) {
        G_hi = G0_hi;
        G_lo = G0_lo;
        for (int i = 0; i < n; ++i) {
          const int at = (i / G) * PLANE + i % G;
          mcg_ff_add(G_hi, G_lo, __fmul_rn(wt[at], __fmul_rn(st[at], down)));
        }
      }
      S->place[rank] = make_int4(MULTI && far, idx, dir, n);
    }
  }
  __syncwarp();
  q = 0;
  if (THIN)
    for (; F * (q + 2) < cnt; q += 4)
      mcg_tile_add<THIN, TALLY, MULTI, 4>(S, q, D);
  for (; F * (MULTI || THIN ? q : q + 1) < cnt; q += 2)
    mcg_tile_add<THIN, TALLY, MULTI, 2>(S, q, D);
  if (!MULTI && !THIN && F * q < cnt)
    mcg_tile_add<THIN, TALLY, MULTI, 1>(S, q, D);
  __syncwarp();
  return n;
}

/* Length along x from x to the face ahead, for a flight that starts at x in a
 * cell; NaN (no tile) outside the range in which the tiles' division is exact,
 * without a direction, or beyond the cell's own length (x outside the cell, or
 * a cell without one). */
__device__ __forceinline__ float mcg_first_length(const float4 c, const float4 tab, float x,
                                                  float mu, float inv_mu, float wmc)
{
  const float a = fabsf(mu < 0.0f ? __fsub_rn(x, c.z) : __fsub_rn(c.w, x));
  const bool inside = mu < 0.0f ? x >= c.z : x <= c.w;
  return inside & (inv_mu != 0.0f) & (wmc <= 0x1p60f) & ((a == 0.0f) | (a >= 0x1p-100f)) &
                 (a <= (mu < 0.0f ? tab.w : tab.z))
             ? a
             : __int_as_float(0x7fc00000);
}

/* Most steps of a tile from cell idx of [lo, hi): to the end of the range; none
 * (the full step) below the weights that stay normal numbers, scaled or not,
 * through a tile (each step keeps more than 3/4), unless they are below `tiny`
 * (mcg_run_consts): with the full form from 2^-60 on, runs without a minimum weight
 * took 97 ms where a lane per history had taken 75 (5000 histories on 10,000 cells,
 * depth 60, strict); 15 ms so. */
__device__ __forceinline__ int mcg_tile_limit(int width, int idx, int lo, int hi, float mu,
                                              float wmc, uint32_t left, float tiny)
{
  const int n = min(width, mu < 0.0f ? idx - lo + 1 : hi - idx);
  return (wmc >= 0x1p-60f) | (fabsf(wmc) < tiny) ? (int)min((uint32_t)n, left) : 0;
}

/* The step that a tile left: the flight sample's state, then whatever the step
 * is (mcg_step_rest). */
template <bool STRICT, int TALLY>
__device__ __forceinline__ void mcg_full(uint64_t &seed, float &x, float &mu, float &wmc,
                                         float &inv_mu, int &idx, uint32_t &nsc, const float4 c,
                                         unsigned long long *tally_cell, int qs,
                                         const mcg_libm_tab *T, const mcg_libm_dev &LM,
                                         float *l_out = nullptr, bool *coll_out = nullptr,
                                         float *dep_out = nullptr, float *wres = nullptr)
{
  mcg_lcg_next(seed);
  mcg_step_rest<STRICT, TALLY>(seed, x, mu, wmc, inv_mu, idx, nsc, c, tally_cell, qs, T, LM, l_out,
                               coll_out, dep_out, wres);
}

/* Jumps of the seed chain by d 32^l steps, d < 32: A and C of s -> A s + C mod
 * 2^63 at l 32 + d.  A newborn's state is one multiply-add per base-32 digit of
 * its index (a jump-ahead by doubling takes about 500 instructions, run by the
 * one or two lanes that refill). */
#define MCG_JUMP_LEVELS 8
struct mcg_chain_jumps {
  unsigned long long A[32 * MCG_JUMP_LEVELS], C[32 * MCG_JUMP_LEVELS];
};

__device__ __forceinline__ void mcg_fill_chain_jumps(mcg_chain_jumps *J)
{
  for (int k = threadIdx.x; k < 32 * MCG_JUMP_LEVELS; k += blockDim.x) {
    const uint64_t steps = (uint64_t)(k & 31) << (5 * (k >> 5)), c = mcg_lcg_skip(0ull, steps, 1);
    J->A[k] = (mcg_lcg_skip(1ull, steps, 1) - c) & MCG_MASK63;
    J->C[k] = c;
  }
}

/* Shared memory and resident blocks of a gradient kernel: the table of the seed
 * chain (4 KB) goes after its arrays unless it does not fit or costs a block. */
template <typename K>
static cudaError_t mcg_grad_shape(K kern, int block, int limit, size_t *smem, int32_t *jumps, int *bps)
{
  const size_t more = (*smem + 7) / 8 * 8 + sizeof(mcg_chain_jumps);
  /* the opt-in maximum on every call (mcg_track_launch) */
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, kern, block, *smem);
  int with = 0;
  if (e == cudaSuccess && more <= (size_t)limit)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&with, kern, block, more);
  *jumps = with > 0 && with == *bps;
  if (*jumps)
    *smem = more;
  return e;
}

/* The seed chain's state n steps after s. */
__device__ __forceinline__ uint64_t mcg_chain_jump(const mcg_chain_jumps *J, uint64_t s, uint64_t n)
{
  for (int l = 0; l < MCG_JUMP_LEVELS && n; ++l, n >>= 5) {
    const int k = 32 * l + (int)(n & 31);
    s = J->A[k] * s + J->C[k];
  }
  if (n) /* indices from 2^40 on */
    s = mcg_lcg_skip(s & MCG_MASK63, n << (5 * MCG_JUMP_LEVELS), 1);
  return s & MCG_MASK63;
}

/* Particle k of a device-born source (see mcg_source). */
__device__ __forceinline__ void mcg_born(const mcg_chain_jumps *J, const mcg_source &S, int64_t k,
                                         uint64_t &seed, float &x, float &mu, float &wmc, int &idx)
{
  const uint64_t s = S.seed_mode == 0 ? mcg_chain_jump(J, S.base_seed, (uint64_t)k + 1)
                                      : ((S.base_seed + (uint64_t)k) & MCG_MASK63);
  mcg_source_particle_at(S, s, seed, x, mu, wmc, idx);
}

/* A warp's share of a launch's histories: a chunk taken from a counter, handed
 * to idle lanes in order. */
struct mcg_pool {
  long long next = 0, end = 0; /* what is left of the chunk */
  bool drained = false;

  /* The history of this lane (in `need`), or -1; chunk 0: no more than the
   * lanes ask for.  The whole warp calls. */
  __device__ __forceinline__ long long take(unsigned need, unsigned long long *counter, long long n,
                                            int chunk)
  {
    const int cnt = __popc(need), rank = __popc(need & lanemask_lt());
    const long long avail = end - next;
    long long my = -1;
    if (rank < avail)
      my = next + rank;
    if (cnt > avail && !drained) {
      const int grab = chunk ? chunk : cnt;
      unsigned long long b = 0;
      if ((threadIdx.x & 31) == 0)
        b = atomicAdd(counter, (unsigned long long)grab);
      b = __shfl_sync(0xffffffffu, b, 0);
      if ((long long)b >= n) {
        drained = true;
        next = end = 0;
      } else {
        end = min((long long)b + grab, n);
        const long long r2 = rank - avail;
        if (rank >= avail && r2 < end - (long long)b)
          my = (long long)b + r2;
        next = min((long long)b + (cnt - avail), end);
        drained = end == n; /* nothing more to ask for */
      }
    } else {
      next += min((long long)cnt, avail);
    }
    return my;
  }
};

/* Shared memory of mcg_track_kernel: libm tables, counters, jumps, the tally's
 * copies (an even number of words; thin: low words), the warps' tiles. */
inline size_t mcg_track_smem(size_t tally_words, int block, bool thin)
{
  if (thin)
    tally_words = (tally_words + 1) / 2; /* MCG_TALLY_LO32 */
  return sizeof(mcg_libm_tab) + 16 * 8 + sizeof(mcg_chain_jumps) + sizeof(mcg_real_jumps) +
         ((tally_words + 1) & ~(size_t)1) * 8 +
         (size_t)(block / 32) * (thin ? sizeof(mcg_tile_smem<true>) : sizeof(mcg_tile_smem<false>));
}

/* Launch shape of a chain: short ones keep one tally copy per warp in
 * 256-thread blocks; long ones share one copy per block of 1024 threads (thin
 * ones MCG_THIN_BLOCK), or of fewer where the copy and the warps' tiles would
 * not fit; a chain too long for any copy adds to the global tally.  block and
 * global as asked (0: automatic). */
struct mcg_shape {
  int block, copies;
  bool global, thin;
  size_t smem;
};

inline mcg_shape mcg_track_shape(int n_cells, int block, bool global, bool thin, size_t optin)
{
  mcg_shape s = {block, 1, global, thin, 0};
  auto fit = [&](int b) {
    s.copies = !s.thin && (size_t)n_cells * 8 * (b / 32) <= 24 * 1024 ? b / 32 : 1;
    s.smem = mcg_track_smem(s.global ? 0 : (size_t)n_cells * s.copies, b, s.thin);
    return s.smem <= optin;
  };
  if (!block) {
    s.block = thin ? MCG_THIN_BLOCK : ((size_t)n_cells * 8 * 8 <= 24 * 1024) ? 256 : 1024;
    while (!s.global && s.block > 256 && !fit(s.block))
      s.block -= 128;
  }
  if (!fit(s.block)) {
    s.global = true;
    s.thin = false;
    s.block = block ? block : 1024;
    fit(s.block);
  }
  return s;
}

/* Counters of a finished history: result r, final weight.  In 32-bit halves:
 * 64-bit shared-memory adds whose result is not used are compare-and-swap loops,
 * which all lanes of a block run on the same few words (short histories are little
 * else: 1e7 of one or two steps in 2-cell slabs 2.46 ms so, and half the
 * instructions waited for them). */
template <bool STRICT>
__device__ __forceinline__ void mcg_count_end(unsigned long long *s_cnt, int r, float wmc,
                                              float wres, int qs)
{
  long long wq = mcg_to_fixed(wmc, qs);
  if (!STRICT)
    wq += mcg_to_fixed(wres, qs); /* the weight's float-float remainder */
  mcg_tally_add<MCG_TALLY_SMEM32>(&s_cnt[MCG_CNT_HIST], 1);
  if (r == 2) {
    atomicOr(reinterpret_cast<unsigned *>(&s_cnt[MCG_CNT_ERR]), 1u);
    return;
  }
  const int side = r == -1 ? 0 : r == 1 ? 1 : 2; /* left, right, killed */
  mcg_tally_add<MCG_TALLY_SMEM32>(&s_cnt[MCG_CNT_LEFT + side], 1);
  mcg_tally_add<MCG_TALLY_SMEM32>(&s_cnt[MCG_CNT_WLEFT + side], wq);
}

/* The chain that a warp's newborns run in; with MULTI the slab, whose cells
 * start at `off` of the concatenated ones. */
struct mcg_geometry {
  int32_t off, ncell;
};

/* A lane's history. */
struct mcg_lane {
  uint64_t s2 = 0; /* the state, shifted left by one */
  float x = 0.f, mu = 0.f, wmc = 0.f, inv_mu = 0.f;
  float wres = 0.f; /* fast: the weight's rounding residue (mcg_fast_weight_update) */
  float2 test = {0.f, 0.f}; /* THIN: mcg_thin_tests */
  float a0 = 0.f;   /* mcg_first_length; inf: x is the face the cell was entered by */
  int idx = 0, off = 0, ncell = 0; /* its cell, of the range off .. off + ncell */
  uint32_t nst = 0, nsc = 0;
  float G_hi = 0.f, G_lo = 0.f; /* LOSS: sum of w_c dep */
  bool wait = false; /* its step needs the full form */

  __device__ __forceinline__ bool living(const mcg_rules &R) const
  {
    return (wmc >= R.min_w) & ((unsigned)(idx - off) < (unsigned)ncell) & (nst < R.max_steps);
  }
  /* Classification of simulate_particle for an ended history; one still alive
   * in the chain has reached the step limit (2). */
  __device__ __forceinline__ int outcome(const mcg_rules &R) const
  {
    const int c = idx - off;
    if ((wmc >= R.min_w) && ((unsigned)c < (unsigned)ncell))
      return 2;
    return c == -1 ? -1 : c == ncell ? 1 : wmc < R.min_w ? 0 : -1;
  }
  /* x, when it is only known as a face */
  __device__ __forceinline__ float place(const float4 *cells) const
  {
    return a0 != INFINITY ? x : mu < 0.0f ? __ldg(&cells[idx + 1].z) : __ldg(&cells[idx - 1].w);
  }
  /* A particle newly in the lane (state, x, mu, wmc, idx and range set). */
  template <bool STRICT, bool THIN>
  __device__ __forceinline__ void enter(const mcg_rules &R, const float4 *cells, const mcg_tab &tab)
  {
    a0 = 0.0f;
    inv_mu = mcg_flight_rcp(mu);
    wres = 0.f;
    nst = nsc = 0;
    G_hi = G_lo = 0.f;
    if (THIN)
      test = mcg_thin_tests<STRICT>(inv_mu, wmc, R.run);
    if (living(R))
      a0 = mcg_first_length(__ldg(cells + idx), __ldg(tab.cell + idx), x, mu, inv_mu, wmc);
  }
};

/* One tile for every lane with `alive` that can; the lanes whose step needs the
 * full form wait until pool_lanes of 32 alive ones do, and as many fewer as are
 * alive, and take it together: a fixed number made the last histories of a warp
 * wait for one another (10,000 cells, 1e5 histories, strict: 7.05 ms -> 5.85 ms).
 * MULTI, whose warps stay full, keeps the number until nothing else can step
 * (4096 slabs: 201 ms against 204).  Every call steps a lane, makes one wait or completes the
 * waiting steps, if any lane is alive, and no lane passes its step limit.
 * far (MULTI): the lane's deposits go to the global tally, the others' full
 * steps to word[idx - word_off].  The whole warp calls. */
template <bool STRICT, bool THIN, int TALLY, bool MULTI, bool LOSS = false>
__device__ __forceinline__ void mcg_advance(mcg_lane &p, bool alive, bool far, const float4 *cells,
                                            const mcg_tab &tab, const mcg_sink &D,
                                            unsigned long long *word, int word_off,
                                            const mcg_rules &R, const mcg_tile_warp<THIN> &tiles,
                                            const mcg_real_jumps *jumps, const mcg_libm_tab *T,
                                            const mcg_libm_dev &libm)
{
  bool can = alive & !p.wait;
  const int nmax = p.a0 == p.a0
                       ? mcg_tile_limit(min(R.window, mcg_tile_shape<THIN>::TW), p.idx, p.off,
                                        p.off + p.ncell, p.mu, p.wmc, R.max_steps - p.nst,
                                        THIN ? 0.0f : R.run.tiny)
                       : 0;
  p.wait |= can & (nmax == 0);
  can &= nmax != 0;
  if (__any_sync(0xffffffffu, can)) {
    const int dir = p.mu < 0.0f ? -1 : 1;
    const bool tiny = !THIN && fabsf(p.wmc) < R.run.tiny;
    const float up = tiny ? 1.0f : R.run.scale, down = tiny ? 1.0f : R.run.inv_scale;
    float W = __fmul_rn(p.wmc, up), res = __fmul_rn(p.wres, up);
    const int k = mcg_tiles<STRICT, THIN, TALLY, MULTI, LOSS>(
        can, p.s2, fabsf(p.mu), fabsf(p.inv_mu), p.a0, dir, p.idx, nmax, p.test, W, res, p.G_hi, p.G_lo,
        far, down, tab, D, tiles, R.run);
    if (k > 0) {
      p.s2 = jumps->A[k] * p.s2 + jumps->C[k];
      p.wmc = __fmul_rn(W, down);
      if (!STRICT)
        p.wres = __fmul_rn(res, down);
      p.idx += k * dir;
      p.nst += (uint32_t)k;
      p.a0 = INFINITY;
    }
    p.wait |= can & (k < nmax) & (p.wmc >= R.min_w);
  }
  const unsigned wb = __ballot_sync(0xffffffffu, p.wait);
  if (wb && (MULTI ? __popc(wb) >= R.pool_lanes || wb == __ballot_sync(0xffffffffu, alive)
                   : 32 * __popc(wb) >= R.pool_lanes * __popc(__ballot_sync(0xffffffffu, alive)))) {
    if (p.wait) {
      p.x = p.place(cells);
      uint64_t seed = p.s2 >> 1;
      const int cell = p.idx;
      float len, dep;
      bool coll;
      mcg_full<STRICT, TALLY>(seed, p.x, p.mu, p.wmc, p.inv_mu, p.idx, p.nsc, __ldg(cells + cell),
                              THIN ? nullptr
                                   : (TALLY == MCG_TALLY_GLOBAL || far ? D.global + cell
                                                                       : word + (cell - word_off)),
                              R.q_log2, T, libm, &len, &coll, &dep,
                              STRICT || LOSS ? nullptr : &p.wres);
      if (LOSS)
        mcg_ff_add(p.G_hi, p.G_lo, __fmul_rn(__ldg(&tab.aux[cell].x), dep));
      if (THIN) {
        mcg_lo32_add(reinterpret_cast<unsigned *>(word) + cell, D.global + cell,
                     mcg_to_fixed(dep, R.q_log2));
        p.test = mcg_thin_tests<STRICT>(p.inv_mu, p.wmc, R.run);
      }
      p.s2 = seed << 1;
      ++p.nst;
      p.wait = false;
      p.a0 = (unsigned)(p.idx - p.off) < (unsigned)p.ncell
                 ? mcg_first_length(__ldg(cells + p.idx), __ldg(tab.cell + p.idx), p.x, p.mu, p.inv_mu,
                                    p.wmc)
                 : 0.0f;
    }
  }
}

/* A warp's histories, to the end of the source: n() histories handed out by
 * *counter in chunks (mcg_pool::take).  birth(k, ...) makes history k's particle
 * with its cell index local to the chain and returns its number; end(number,
 * result, p, cell) sees its final state.  cells and tab are the chain's, word its shared-memory tally (base
 * of mcg_sink D) as a pointer.  The whole warp calls.
 *
 * MULTI: cells, tab and the global tally are those of all slabs; when a slab's
 * histories are handed out (exhausted()), the block changes to the next work
 * item together (more(), which returns false when there is none) while its
 * warps keep the histories they have: such a history stays in its lane, with
 * its own slab's cells, and its deposits go to the global tally.  So no warp
 * waits for another's longest history. */
template <bool STRICT, bool THIN, int TALLY, bool MULTI, bool LOSS, class N, class BIRTH, class END,
          class GONE, class MORE>
__device__ __forceinline__ void mcg_histories(mcg_geometry &geo, mcg_sink &D, const float4 *cells,
                                              const mcg_tab &tab, unsigned long long *word,
                                              const mcg_rules &R, const mcg_tile_warp<THIN> &tiles,
                                              const mcg_real_jumps *jumps, const mcg_libm_tab *T,
                                              const mcg_libm_dev &libm, unsigned long long *counter,
                                              const N &n, int chunk, const BIRTH &birth,
                                              const END &end, const GONE &exhausted, const MORE &more)
{
  mcg_lane p;
  int64_t hid = -1;
  bool active = false;
  mcg_pool pool;
  bool work = true; /* MULTI: more() has not yet returned false */

  for (;;) {
    bool alive = active & p.living(R);
    const unsigned ab = __ballot_sync(0xffffffffu, alive);
    /* ended histories leave and newborns come once refill_lanes lanes are
     * without a living history, or no lane has one */
    const bool gone = MULTI && work && exhausted();
    if (!ab || gone || (__popc(~ab) >= R.refill_lanes &&
                        (!pool.drained || __any_sync(0xffffffffu, active & !alive)))) {
      if (active & !alive) {
        p.x = p.place(cells);
        end(hid, p.outcome(R), p, p.idx - p.off);
        active = false;
      }
      unsigned need = __ballot_sync(0xffffffffu, !active);
      while (MULTI && work && exhausted()) {
        work = more();
        pool = mcg_pool();
      }
      if (MULTI && !work)
        pool.drained = true;
      const long long my = need ? pool.take(need, counter, n(), chunk) : -1;
      if (!active && my >= 0) {
        uint64_t seed;
        hid = birth(my, seed, p.x, p.mu, p.wmc, p.idx);
        p.s2 = seed << 1;
        p.off = MULTI ? geo.off : 0;
        p.ncell = geo.ncell;
        p.idx += p.off;
        p.enter<STRICT, THIN>(R, cells, tab);
        active = true;
        alive = p.living(R);
      }
      if (!__any_sync(0xffffffffu, active) && (!MULTI || !work))
        break;
    }
    /* each pass advances a living lane, ends a history or hands out work, so
     * this ends */
    mcg_advance<STRICT, THIN, TALLY, MULTI, LOSS>(p, alive, MULTI && p.off != geo.off, cells, tab, D, word,
                                            geo.off, R, tiles, jumps, T, libm);
  }
}

/* Histories of a chain of thick cells (mcg_thick): one lane each through every
 * step, MCG_LANES_STEPS of them between two looks for new ones.  Collisions and
 * steep absorptions leave the tiles a step or two each.  LOSS as in mcg_tiles. */
#define MCG_LANES_STEPS 8
template <bool STRICT, int TALLY, bool LOSS, class BIRTH, class END>
__device__ __forceinline__ void mcg_lane_histories(int ncell, const float4 *cells, const float2 *aux,
                                                   unsigned long long *tally, const mcg_rules &R,
                                                   const mcg_libm_tab *T, const mcg_libm_dev &libm,
                                                   unsigned long long *counter, long long n, int chunk,
                                                   const BIRTH &birth, const END &end)
{
  mcg_lane p;
  uint64_t seed = 0;
  int64_t hid = -1;
  bool active = false;
  mcg_pool pool;
  p.ncell = ncell;
  for (;;) {
    const unsigned need = __ballot_sync(0xffffffffu, !active);
    if (need) {
      const long long my = pool.take(need, counter, n, chunk);
      if (!active && my >= 0) {
        hid = birth(my, seed, p.x, p.mu, p.wmc, p.idx);
        p.inv_mu = mcg_flight_rcp(p.mu);
        p.wres = 0.f;
        p.nst = p.nsc = 0;
        p.G_hi = p.G_lo = 0.f;
        active = true;
      }
    }
    if (!__any_sync(0xffffffffu, active))
      break;
    if (active) {
      const int kmax = (int)min((uint32_t)MCG_LANES_STEPS, R.max_steps - p.nst);
      int k = 0;
#pragma unroll 1
      for (; k < kmax && (p.wmc >= R.min_w) & ((unsigned)p.idx < (unsigned)ncell); ++k) {
        const int cell = p.idx;
        float len, dep;
        bool coll;
        mcg_step<STRICT, TALLY, false>(seed, p.x, p.mu, p.wmc, p.inv_mu, p.idx, p.nsc,
                                       __ldg(cells + cell), tally + cell, R.q_log2, T, libm,
                                       LOSS ? &len : nullptr, LOSS ? &coll : nullptr,
                                       LOSS ? &dep : nullptr, STRICT || LOSS ? nullptr : &p.wres);
        if (LOSS)
          mcg_ff_add(p.G_hi, p.G_lo, __fmul_rn(__ldg(&aux[cell].x), dep));
      }
      p.nst += (uint32_t)k;
      if (!p.living(R)) {
        p.s2 = seed << 1;
        end(hid, p.outcome(R), p, p.idx);
        active = false;
      }
    }
  }
}

/* THIN: the chain is optically thin (see update_thin in mcg_api.cu) and the
 * tally is MCG_TALLY_LO32.  LANES: mcg_lane_histories instead of tiles. */
template <bool STRICT, int TALLY, bool THIN, bool LANES = false>
__global__ void __launch_bounds__(THIN ? MCG_THIN_BLOCK : 1024) mcg_track_kernel(mcg_track_params P)
{
  if (P.heaviest && (*P.heaviest >= P.heavy_line) != (P.heavy != 0))
    return;
  extern __shared__ __align__(16) unsigned char smem[];
  mcg_libm_tab *T = reinterpret_cast<mcg_libm_tab *>(smem);
  unsigned long long *s_cnt = reinterpret_cast<unsigned long long *>(smem + sizeof(mcg_libm_tab));
  mcg_chain_jumps *s_chain = reinterpret_cast<mcg_chain_jumps *>(s_cnt + 16);
  mcg_real_jumps *s_real = reinterpret_cast<mcg_real_jumps *>(s_chain + 1);
  unsigned long long *s_tally = reinterpret_cast<unsigned long long *>(s_real + 1);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ncell = P.n_cells, lo = P.cell_lo;
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
  /* the block's copy of the tally: 64-bit words, or low words (THIN) */
  const int words = TALLY == MCG_TALLY_GLOBAL ? 0 : THIN ? (ncell + 1) / 2 : ncell * P.tally_copies;
  for (int i = tid; i < words; i += blockDim.x)
    s_tally[i] = 0ull;
  mcg_tile_smem<THIN> *tile = reinterpret_cast<mcg_tile_smem<THIN> *>(
      s_tally + ((words + 1) & ~1)) + warp;
  __syncthreads();
  unsigned long long *my_tally = s_tally + (THIN ? 0 : (size_t)(warp % P.tally_copies) * ncell);

  const mcg_tile_warp<THIN> tiles(tile, s_real);
  mcg_geometry geo = {0, ncell};
  mcg_sink sink = {(uint32_t)__cvta_generic_to_shared(my_tally), P.tally};
  unsigned long long tot_steps = 0, tot_scat = 0;
  auto birth = [&](long long my, uint64_t &seed, float &x, float &mu, float &wmc, int &idx) {
    if (P.particles)
      mcg_load_particle(P, my, seed, x, mu, wmc, idx);
    else
      mcg_born(s_chain, P.src, P.first + my, seed, x, mu, wmc, idx);
    idx -= lo;
    return my;
  };
  auto end = [&](long long hid, int r, const mcg_lane &p, int idx) {
    if (P.particles && p.nst) { /* without a step the particle stays as it is */
      unsigned long long *q = reinterpret_cast<unsigned long long *>(P.particles + hid);
      q[0] = p.s2 >> 1;
      q[1] = (unsigned long long)__float_as_uint(p.x) |
             ((unsigned long long)__float_as_uint(p.mu) << 32);
      q[2] = (unsigned long long)__float_as_uint(p.wmc) |
             ((unsigned long long)(uint32_t)(idx + lo) << 32);
    }
    if (P.results)
      P.results[hid] = r;
    if (P.steps)
      P.steps[hid] = p.nst;
    if (P.scatters)
      P.scatters[hid] = p.nsc;
    mcg_count_end<STRICT>(s_cnt, r, p.wmc, p.wres, P.rules.q_log2);
    tot_steps += p.nst;
    tot_scat += p.nsc;
  };
  if constexpr (LANES)
    mcg_lane_histories<STRICT, TALLY, false>(ncell, P.cells, nullptr,
                                             TALLY == MCG_TALLY_GLOBAL ? P.tally : my_tally, P.rules, T,
                                             P.libm, P.next, P.n, P.chunk, birth, end);
  else
    mcg_histories<STRICT, THIN, TALLY, false, false>(
        geo, sink, P.cells, P.tab, my_tally, P.rules, tiles, s_real, T, P.libm, P.next,
        [&] { return (long long)P.n; }, P.chunk, birth, end, [] { return true; }, [] { return false; });

  /* per-thread counters -> block */
  for (int o = 16; o > 0; o >>= 1) {
    tot_steps += __shfl_down_sync(0xffffffffu, tot_steps, o);
    tot_scat += __shfl_down_sync(0xffffffffu, tot_scat, o);
  }
  if (lane == 0) {
    atomicAdd(&s_cnt[MCG_CNT_STEPS], tot_steps);
    atomicAdd(&s_cnt[MCG_CNT_SCAT], tot_scat);
  }
  __syncthreads();
  if (THIN) {
    const unsigned *lo32 = reinterpret_cast<const unsigned *>(s_tally);
    for (int i = tid; i < ncell; i += blockDim.x)
      if (lo32[i])
        atomicAdd(&P.tally[i], (unsigned long long)lo32[i]);
  } else if (TALLY != MCG_TALLY_GLOBAL)
    for (int i = tid; i < ncell; i += blockDim.x) {
      unsigned long long s = 0;
      for (int c = 0; c < P.tally_copies; ++c)
        s += s_tally[(size_t)c * ncell + i];
      if (s)
        atomicAdd(&P.tally[i], s);
    }
  if (tid < MCG_CNT_N) {
    if (tid == MCG_CNT_ERR) {
      if (s_cnt[tid])
        atomicOr(&P.counters[tid], s_cnt[tid]);
    } else if (s_cnt[tid]) {
      atomicAdd(&P.counters[tid], s_cnt[tid]);
    }
  }
}

/* The weight from which the thin form is no longer taken: its deposits have 31
 * bits (MCG_TALLY_LO32), and a flight whose deposits may pass them takes the full
 * form for every step.  20,000 histories of weight 1000 at scale 2^40 on 10,000
 * cells took 92 ms so, and 2.4 ms with weight 1.  At the line flights with |mu| <
 * 1/4 do.  Thin / other form by the |mu| below which they do, 50,000 histories on
 * 10,000 cells: strict .1 4.2 / 9.8 ms, .2 5.6 / 9.8, .4 9.0 / 9.8, all 111 / 10.3;
 * fast .1 4.2 / 6.3, .2 5.4 / 6.3, .4 9.0 / 6.5, all 111 / 6.7. */
inline float mcg_heavy_weight(const mcg_context *ctx)
{
  return 0x1p29f / (ctx->width_a * ldexpf(1.0f, ctx->log2_scale));
}

/* The rules of a launch.  Full steps are pooled for 4 lanes of 32 (thin chains
 * need them on 1 % of the tiles, others on a third of them) and ended histories
 * replaced for two; 2 to 16 and 1 to 8 were measured within 5 % of these on thin
 * chains and within 10 % on a 1000-cell one. */
#define MCG_WINDOW_LEAST 8 /* a caller's refill_steps below it: a tile's fixed costs (1000 cells, 3e5
                              histories, strict: 20 ms at 1, 5.5 at 4, 3.3 at 8, 2.1 at 32, where a lane
                              per history had taken 5.9, 4.6, 4.4 and 4.1) */
inline mcg_rules mcg_rules_setup(const mcg_context *ctx, float min_w)
{
  mcg_rules R;
  R.min_w = min_w;
  R.q_log2 = ctx->log2_scale;
  R.max_steps = ctx->max_steps;
  R.window = ctx->refill ? std::max(ctx->refill, MCG_WINDOW_LEAST) : MCG_TW_MAX;
  R.pool_lanes = 4;
  R.refill_lanes = 2;
  R.run = mcg_run_setup(ctx->log2_scale, min_w, ctx->run_bounds, ctx->width_a, ctx->width_i);
  return R;
}

/* Grid of at most `resident` blocks, and the chunk of histories a warp takes:
 * a warp advances its histories together, one tile of each per round, so few
 * histories are spread over as many warps as there are. */
inline int mcg_track_grid(int resident, int block, int64_t n, bool lanes, mcg_track_params &P)
{
  if (lanes) { /* a lane per history */
    P.chunk = 64;
    return (int)std::min<int64_t>(resident, (n + block - 1) / block);
  }
  const int64_t warps = (int64_t)resident * (block / 32);
  P.chunk = (int)std::min<int64_t>(32, (n + warps - 1) / warps);
  return (int)std::min<int64_t>(resident, n);
}

#endif
