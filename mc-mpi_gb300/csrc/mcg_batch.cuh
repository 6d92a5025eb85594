/*
 * mcg_batch.cuh - the batched tracker's device code: items of many slabs in one
 * persistent launch (mcg_batch.cu), and the forward pass of the inverse fit
 * (mcg_fit.cu).
 */
#ifndef MCG_BATCH_CUH
#define MCG_BATCH_CUH

#include <type_traits>

#include "mcg_track.cuh"

bool mcg_batch_lanes(const mcg_widths &w, int n, bool strict);

/* A cell's entry of the tile table from its fast-arithmetic parameters
 * (mcg_tile_entry: within a slab neighbours share their faces). */
__host__ __device__ inline float4 mcg_tile_cell(const float4 c)
{
  const float a = c.w - c.z;
  const float len = a >= 0x1p-90f && a <= 0x1p90f && c.x >= 0.0f ? a : NAN;
  return make_float4(c.x, c.y, len, len);
}

struct mcg_batch_item {
  int32_t slab, lanes; /* lanes: a lane per history (mcg_batch_lanes) */
  int64_t first, count;
  int64_t sum; /* LOSS: its first history's place in `loss` */
};

struct mcg_batch_params {
  const float4 *cells, *tab;
  const float2 *aux;      /* LOSS: loss weights, {w_c, .} */
  float2 *loss;           /* LOSS: the histories' sums; null: not wanted */
  const long long *step;  /* LOSS: histories of earlier steps precede this one's (null: none) */
  const mcg_batch_slab_dev *slabs;
  const mcg_batch_item *items;
  int32_t n_items;
  int32_t max_cells;
  unsigned long long *item_next;
  unsigned long long *tally;
  unsigned long long *counters;
  mcg_libm_dev libm;
  const mcg_libm_tab *libm_tab;
  mcg_rules rules;
};

/* The item that a block works on (shared memory). */
struct mcg_batch_work {
  unsigned long long taken; /* histories handed out */
  long long item, first, count, sum;
  int32_t off, m;
  mcg_source src;
};

/* Shared memory: libm tables, counters, the item, jumps, the tally of one slab,
 * the warps' tiles. */
inline size_t mcg_batch_smem(int max_cells, int block, bool tally, bool loss)
{
  return mcg_track_smem(tally ? max_cells : 0, block, false) + sizeof(mcg_batch_work) +
         (loss ? (size_t)(block / 32) * (sizeof(mcg_loss_smem) - sizeof(mcg_tile_smem<false>)) : 0);
}
static_assert(sizeof(mcg_batch_work) % 16 == 0, "the tally after it is read by 16 bytes");

/* LOSS: every history's sum of w_c dep is stored; nothing is counted. */
template <bool STRICT, int TALLY, bool LOSS>
__device__ __forceinline__ void mcg_batch_body(const mcg_batch_params &P)
{
  using tile_smem = std::conditional_t<LOSS, mcg_loss_smem, mcg_tile_smem<false>>;
  extern __shared__ __align__(16) unsigned char smem[];
  mcg_libm_tab *T = reinterpret_cast<mcg_libm_tab *>(smem);
  unsigned long long *s_cnt = reinterpret_cast<unsigned long long *>(smem + sizeof(mcg_libm_tab));
  mcg_batch_work *work = reinterpret_cast<mcg_batch_work *>(s_cnt + 16);
  mcg_chain_jumps *s_chain = reinterpret_cast<mcg_chain_jumps *>(work + 1);
  mcg_real_jumps *s_real = reinterpret_cast<mcg_real_jumps *>(s_chain + 1);
  unsigned long long *s_tally = reinterpret_cast<unsigned long long *>(s_real + 1);
  const int tid = threadIdx.x, lane = tid & 31;
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
  if (tid == 0)
    work->taken = work->count = 0; /* no item: exhausted at once */
  tile_smem *tile =
      reinterpret_cast<tile_smem *>(
          s_tally + (TALLY == MCG_TALLY_GLOBAL ? 0 : (P.max_cells + 1) & ~1)) + (tid >> 5);
  __syncthreads();
  const mcg_tile_warp<false> tiles(tile, s_real);
  mcg_geometry geo = {-1, 0};
  mcg_sink sink = {0u, P.tally};
  auto flush = [&] {
    if (TALLY != MCG_TALLY_GLOBAL)
      for (int i = tid; i < geo.ncell; i += blockDim.x)
        if (s_tally[i])
          atomicAdd(&P.tally[geo.off + i], s_tally[i]);
  };
  unsigned long long tot_steps = 0, tot_scat = 0;
  mcg_histories<STRICT, false, TALLY, true, LOSS>(
      geo, sink, P.cells, {P.tab, nullptr, 0, P.aux}, s_tally, P.rules, tiles, s_real, T, P.libm,
      &work->taken, [&] { return work->count; }, 0,
      [&](long long my, uint64_t &seed, float &x, float &mu, float &wmc, int &idx) {
        mcg_born(s_chain, work->src, work->first + my, seed, x, mu, wmc, idx);
        return LOSS ? work->sum + my : my;
      },
      [&](long long hid, int r, const mcg_lane &p, int) {
        if (LOSS) {
          if (P.loss)
            P.loss[hid] = make_float2(p.G_hi, p.G_lo);
          return;
        }
        mcg_count_end<STRICT>(s_cnt, r, p.wmc, p.wres, P.rules.q_log2);
        tot_steps += p.nst;
        tot_scat += p.nsc;
      },
      /* broadcast, so that the warp decides as one */
      [&] {
        return __shfl_sync(0xffffffffu, *(volatile unsigned long long *)&work->taken, 0) >=
               (unsigned long long)work->count;
      },
      [&] {
        /* every warp of the block comes here (each looks at the exhausted
         * item in every round), so nothing is being added to the tally */
        __syncthreads();
        if (tid == 0) {
          work->item = (long long)atomicAdd(P.item_next, 1ull);
          work->taken = 0;
          if (work->item < P.n_items) {
            const mcg_batch_item it = P.items[work->item];
            const mcg_batch_slab_dev sd = P.slabs[it.slab];
            work->first = it.first + (LOSS ? *P.step * sd.n_hist : 0);
            work->count = it.count;
            work->sum = it.sum;
            work->off = sd.cell_off;
            work->m = sd.m;
            work->src = sd.src;
          }
        }
        __syncthreads();
        if (work->item >= P.n_items)
          return false;
        if (work->off != geo.off) {
          flush();
          geo.off = work->off;
          geo.ncell = work->m;
          sink.shared = (uint32_t)__cvta_generic_to_shared(s_tally) - 8u * (uint32_t)geo.off;
          if (TALLY != MCG_TALLY_GLOBAL) {
            __syncthreads();
            for (int i = tid; i < geo.ncell; i += blockDim.x)
              s_tally[i] = 0ull;
            __syncthreads();
          }
        }
        return true;
      });
  __syncthreads();
  flush();
  if (LOSS)
    return;
  for (int o = 16; o > 0; o >>= 1) {
    tot_steps += __shfl_down_sync(0xffffffffu, tot_steps, o);
    tot_scat += __shfl_down_sync(0xffffffffu, tot_scat, o);
  }
  if (lane == 0) {
    atomicAdd(&s_cnt[MCG_CNT_STEPS], tot_steps);
    atomicAdd(&s_cnt[MCG_CNT_SCAT], tot_scat);
  }
  __syncthreads();
  if (tid < MCG_CNT_N && s_cnt[tid]) {
    if (tid == MCG_CNT_ERR)
      atomicOr(&P.counters[tid], s_cnt[tid]);
    else
      atomicAdd(&P.counters[tid], s_cnt[tid]);
  }
}

/* Shared memory of the lane form: libm tables, counters, the item and its history
 * counter, jumps, the tally of one slab. */
#define MCG_LANES_BLOCK 256
inline size_t mcg_batch_lanes_smem(int cells, bool tally)
{
  return sizeof(mcg_libm_tab) + 16 * 8 + 16 + sizeof(mcg_chain_jumps) + (tally ? (size_t)cells * 8 : 0);
}

/* The items of slabs on which a lane per history is faster (mcg_batch_lanes), each
 * by one block, to its end: such histories are short. */
template <bool STRICT, int TALLY, bool LOSS>
__device__ __forceinline__ void mcg_batch_lanes_body(const mcg_batch_params &P)
{
  extern __shared__ __align__(16) unsigned char smem[];
  mcg_libm_tab *T = reinterpret_cast<mcg_libm_tab *>(smem);
  unsigned long long *s_cnt = reinterpret_cast<unsigned long long *>(smem + sizeof(mcg_libm_tab));
  unsigned long long *s_ctl = s_cnt + 16; /* item, histories handed out */
  mcg_chain_jumps *s_chain = reinterpret_cast<mcg_chain_jumps *>(s_ctl + 2);
  unsigned long long *s_tally = reinterpret_cast<unsigned long long *>(s_chain + 1);
  const int tid = threadIdx.x, lane = tid & 31;
  mcg_fill_chain_jumps(s_chain);
  if (STRICT) {
    const float *src = reinterpret_cast<const float *>(P.libm_tab);
    float *dst = reinterpret_cast<float *>(T);
    for (int i = tid; i < (int)(sizeof(mcg_libm_tab) / 4); i += blockDim.x)
      dst[i] = src[i];
  }
  if (tid < 16)
    s_cnt[tid] = 0ull;
  int off = -1, m = 0;
  auto flush = [&] {
    if (TALLY != MCG_TALLY_GLOBAL)
      for (int i = tid; i < m; i += blockDim.x)
        if (s_tally[i])
          atomicAdd(&P.tally[off + i], s_tally[i]);
  };
  unsigned long long tot_steps = 0, tot_scat = 0;
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      s_ctl[0] = atomicAdd(P.item_next, 1ull);
      s_ctl[1] = 0;
    }
    __syncthreads();
    const long long item = (long long)s_ctl[0];
    if (item >= P.n_items)
      break;
    const mcg_batch_item it = P.items[item];
    const mcg_batch_slab_dev sd = P.slabs[it.slab];
    if (sd.cell_off != off) {
      flush(); /* and then zero, each thread its own words */
      off = sd.cell_off;
      m = sd.m;
      if (TALLY != MCG_TALLY_GLOBAL) {
        __syncthreads();
        for (int i = tid; i < m; i += blockDim.x)
          s_tally[i] = 0ull;
        __syncthreads();
      }
    }
    const int64_t first = it.first + (LOSS ? *P.step * sd.n_hist : 0);
    mcg_lane_histories<STRICT, TALLY, LOSS>(
        m, P.cells + off, LOSS ? P.aux + off : nullptr, TALLY == MCG_TALLY_GLOBAL ? P.tally + off : s_tally,
        P.rules, T, P.libm, &s_ctl[1], it.count, 0,
        [&](long long my, uint64_t &seed, float &x, float &mu, float &wmc, int &idx) {
          mcg_born(s_chain, sd.src, first + my, seed, x, mu, wmc, idx);
          return LOSS ? it.sum + my : my;
        },
        [&](long long hid, int r, const mcg_lane &p, int) {
          if (LOSS) {
            if (P.loss)
              P.loss[hid] = make_float2(p.G_hi, p.G_lo);
            return;
          }
          mcg_count_end<STRICT>(s_cnt, r, p.wmc, p.wres, P.rules.q_log2);
          tot_steps += p.nst;
          tot_scat += p.nsc;
        });
  }
  flush();
  if (LOSS)
    return;
  for (int o = 16; o > 0; o >>= 1) {
    tot_steps += __shfl_down_sync(0xffffffffu, tot_steps, o);
    tot_scat += __shfl_down_sync(0xffffffffu, tot_scat, o);
  }
  if (lane == 0) {
    atomicAdd(&s_cnt[MCG_CNT_STEPS], tot_steps);
    atomicAdd(&s_cnt[MCG_CNT_SCAT], tot_scat);
  }
  __syncthreads();
  if (tid < MCG_CNT_N && s_cnt[tid]) {
    if (tid == MCG_CNT_ERR)
      atomicOr(&P.counters[tid], s_cnt[tid]);
    else
      atomicAdd(&P.counters[tid], s_cnt[tid]);
  }
}

#endif
