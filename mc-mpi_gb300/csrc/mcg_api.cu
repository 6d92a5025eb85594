/*
 * mcg_api.cu - host side of libmcgb300: contexts, layer set-up, the strict
 * libm exception tables, kernel launches and the C ABI of include/mcgb300.h.
 */
#include <cuda_runtime.h>

#include <atomic>
#include <new>
#include <dlfcn.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "exact_libm.h"
#include "libm_file.h"
#include "mcg_internal.h"
#include "mcg_track.cuh"

static thread_local std::string g_last_error;

int mcg_fail(int code, const char *fmt, ...)
{
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_last_error = buf;
  return code;
}

int mcg_cuda_fail(cudaError_t e, const char *what)
{
  return mcg_fail(MCG_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

extern "C" const char *mcg_last_error(void) { return g_last_error.c_str(); }
extern "C" const char *mcg_version(void) { return "mcgb300 1.0 (sm_103a)"; }

/* ------------------------------------------------------------ libm tables */
static std::string library_dir()
{
  Dl_info info;
  if (dladdr((void *)&mcg_version, &info) && info.dli_fname) {
    std::string p(info.dli_fname);
    size_t s = p.find_last_of('/');
    return s == std::string::npos ? std::string(".") : p.substr(0, s);
  }
  return ".";
}

static int build_hash(const std::vector<uint32_t> &pairs, std::vector<uint2> &tab, uint32_t &mask,
                      int &probes)
{
  size_t n = pairs.size() / 2, cap = 64;
  while (cap < 2 * n + 1)
    cap <<= 1;
  tab.assign(cap, make_uint2(MCG_HASH_EMPTY, 0u));
  mask = (uint32_t)(cap - 1);
  probes = 1;
  for (size_t i = 0; i < n; ++i) {
    uint32_t key = pairs[2 * i], slot = (key * 0x9E3779B1u) & mask;
    int p = 1;
    while (tab[slot].x != MCG_HASH_EMPTY) {
      if (tab[slot].x == key)
        return mcg_fail(MCG_ERR_TABLES, "duplicate key in libm exception table");
      slot = (slot + 1) & mask;
      ++p;
    }
    tab[slot] = make_uint2(key, pairs[2 * i + 1]);
    probes = std::max(probes, p);
  }
  probes += 1; /* one more probe reaches the empty slot that ends a miss */
  return MCG_OK;
}

int mcg_load_libm(mcg_context *ctx)
{
  if (ctx->libm_loaded)
    return MCG_OK;
  const char *env = getenv("MCG_LIBM_TABLE");
  std::string path = env ? std::string(env) : library_dir() + "/libm_exceptions.bin";
  FILE *f = fopen(path.c_str(), "rb");
  if (!f)
    return mcg_fail(MCG_ERR_TABLES,
                    "strict mode needs the host-libm exception table %s (built by build())",
                    path.c_str());
  mcg_libm_file hdr;
  std::vector<uint32_t> lp, ep;
  bool ok = fread(&hdr, sizeof(hdr), 1, f) == 1 && memcmp(hdr.magic, MCG_LIBM_MAGIC, 8) == 0;
  if (ok) {
    lp.resize(2 * (size_t)hdr.n_log);
    ep.resize(2 * (size_t)hdr.n_exp);
    ok = (lp.empty() || fread(lp.data(), 4, lp.size(), f) == lp.size()) &&
         (ep.empty() || fread(ep.data(), 4, ep.size(), f) == ep.size());
  }
  fclose(f);
  if (!ok)
    return mcg_fail(MCG_ERR_TABLES, "malformed libm exception table %s", path.c_str());
  const mcg_libm_tab tab = MCG_LIBM_TAB_INIT;
  /* of this process's C library and forms: one for all contexts (1 ms) */
  static const uint64_t fingerprint = mcg_libm_fingerprint(&tab);
  if (hdr.fingerprint != fingerprint)
    return mcg_fail(MCG_ERR_TABLES,
                    "libm exception table %s was made against another C library (%s) or "
                    "another version of the evaluators; rebuild",
                    path.c_str(), hdr.libc_version);
  if (!(hdr.logf_relerr <= MCG_LOGF_RELERR_MAX))
    return mcg_fail(MCG_ERR_TABLES,
                    "host logf relative error %.3e exceeds the %.3e the strict tracker's "
                    "certain-crossing test assumes",
                    (double)hdr.logf_relerr, (double)MCG_LOGF_RELERR_MAX);
  std::vector<uint2> hl, he;
  int rc;
  if ((rc = build_hash(lp, hl, ctx->libm.mask_log, ctx->libm.probes_log)) != MCG_OK)
    return rc;
  if ((rc = build_hash(ep, he, ctx->libm.mask_exp, ctx->libm.probes_exp)) != MCG_OK)
    return rc;
  float tl = -1.f, te = -1.f;
  for (int b = 0; b < MCG_TAU_BUCKETS; ++b) {
    tl = std::max(tl, hdr.tau_log[b]);
    te = std::max(te, hdr.tau_exp[b]);
  }
  ctx->libm.tau_log_max = tl;
  ctx->libm.tau_exp_max = te;
  const mcg_run_bounds_t rb = mcg_run_bounds(hdr.tau_exp);
  ctx->run_bounds[0] = rb.b_thin;
  ctx->run_bounds[1] = rb.c_thin;
  ctx->run_bounds[2] = rb.b_mid;
  cudaError_t e;
  float *dtl = nullptr, *dte = nullptr;
  uint2 *dhl = nullptr, *dhe = nullptr;
  mcg_libm_tab *dtab = nullptr;
  /* each allocation joins the context's list as soon as it exists, so a
   * failure part-way leaves nothing behind at mcg_destroy */
  auto alloc = [ctx](void **p, size_t bytes) {
    cudaError_t r = cudaMalloc(p, bytes);
    if (r == cudaSuccess)
      ctx->owned.push_back(*p);
    return r;
  };
  if ((e = alloc((void **)&dtl, sizeof(hdr.tau_log))) != cudaSuccess ||
      (e = alloc((void **)&dte, sizeof(hdr.tau_exp))) != cudaSuccess ||
      (e = alloc((void **)&dhl, hl.size() * sizeof(uint2))) != cudaSuccess ||
      (e = alloc((void **)&dhe, he.size() * sizeof(uint2))) != cudaSuccess ||
      (e = alloc((void **)&dtab, sizeof(tab))) != cudaSuccess)
    return mcg_cuda_fail(e, "cudaMalloc(libm tables)");
  if ((e = cudaMemcpy(dtl, hdr.tau_log, sizeof(hdr.tau_log), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(dte, hdr.tau_exp, sizeof(hdr.tau_exp), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(dhl, hl.data(), hl.size() * sizeof(uint2), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(dhe, he.data(), he.size() * sizeof(uint2), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(dtab, &tab, sizeof(tab), cudaMemcpyHostToDevice)) != cudaSuccess)
    return mcg_cuda_fail(e, "cudaMemcpy(libm tables)");
  ctx->libm.tau_log = dtl;
  ctx->libm.tau_exp = dte;
  ctx->libm.hash_log = dhl;
  ctx->libm.hash_exp = dhe;
  ctx->libm_tab = dtab;
  ctx->libm_n_log = hdr.n_log;
  ctx->libm_n_exp = hdr.n_exp;
  ctx->libm_loaded = true;
  return MCG_OK;
}

/* ------------------------------------------------------------ context */
static int ensure_device(const mcg_context *ctx)
{
  cudaError_t e = cudaSetDevice(ctx->device);
  return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(e, "cudaSetDevice");
}

extern "C" int mcg_create(int device, int mode, mcg_context **out)
{
  if (!out || (mode != MCG_MODE_STRICT && mode != MCG_MODE_FAST))
    return mcg_fail(MCG_ERR_ARG, "mcg_create: bad arguments");
  *out = nullptr;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "cudaGetDeviceCount");
  if (device < 0 || device >= ndev)
    return mcg_fail(MCG_ERR_ARG, "mcg_create: device %d of %d", device, ndev);
  mcg_context *ctx = new mcg_context();
  ctx->device = device;
  ctx->mode = mode;
  int rc = ensure_device(ctx);
  if (rc == MCG_OK) {
    cudaDeviceProp prop;
    if ((e = cudaGetDeviceProperties(&prop, device)) != cudaSuccess)
      rc = mcg_cuda_fail(e, "cudaGetDeviceProperties");
    else {
      ctx->sm_count = prop.multiProcessorCount;
      ctx->smem_optin = (int)prop.sharedMemPerBlockOptin;
      ctx->cc_major = prop.major;
      ctx->cc_minor = prop.minor;
    }
  }
  if (rc == MCG_OK && ((e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking)) != cudaSuccess ||
                       (e = cudaEventCreate(&ctx->ev0)) != cudaSuccess ||
                       (e = cudaEventCreate(&ctx->ev1)) != cudaSuccess))
    rc = mcg_cuda_fail(e, "stream/event create");
  if (rc == MCG_OK) {
    if ((e = cudaMalloc(&ctx->d_counters, 16 * sizeof(unsigned long long))) == cudaSuccess)
      ctx->owned.push_back(ctx->d_counters);
    if (e == cudaSuccess &&
        (e = cudaMalloc(&ctx->d_next, 8 * sizeof(unsigned long long))) == cudaSuccess)
      ctx->owned.push_back(ctx->d_next);
    if (e != cudaSuccess)
      rc = mcg_cuda_fail(e, "cudaMalloc(counters)");
    else
      cudaMemset(ctx->d_counters, 0, 16 * sizeof(unsigned long long));
  }
  if (rc == MCG_OK && mode == MCG_MODE_STRICT)
    rc = mcg_load_libm(ctx);
  if (rc != MCG_OK) {
    std::string msg = g_last_error;
    mcg_destroy(ctx);
    g_last_error = msg;
    return rc;
  }
  *out = ctx;
  return MCG_OK;
}

/* Releases the chain's device buffers and leaves the context with no
 * geometry: launches and tally reads then return MCG_ERR_STATE. */
static void free_geometry(mcg_context *ctx)
{
  for (void *p : {(void *)ctx->d_cells_strict, (void *)ctx->d_cells_fast, (void *)ctx->d_tab,
                  (void *)ctx->d_thin, (void *)ctx->d_tally})
    if (p)
      cudaFree(p);
  ctx->d_cells_strict = ctx->d_cells_fast = ctx->d_tab = nullptr;
  ctx->d_thin = nullptr;
  ctx->d_tally = nullptr;
  ctx->n_layers = ctx->n_cells = ctx->cell_lo = 0;
  ctx->layer_start.clear();
  ctx->layer_m.clear();
  ctx->layer_dx.clear();
  ctx->cells_strict.clear();
  ctx->thin = ctx->thin_fast = ctx->thin_step = false;
}

/* Allocations still to succeed before one is made to fail (-1: none). */
static std::atomic<int> g_fail_alloc_in{-1};

cudaError_t mcg_dev_malloc(void **p, size_t bytes)
{
  int k = g_fail_alloc_in.load();
  while (k >= 0) {
    if (g_fail_alloc_in.compare_exchange_weak(k, k - 1)) {
      if (k == 0) {
        *p = nullptr;
        return cudaErrorMemoryAllocation;
      }
      break;
    }
  }
  return cudaMalloc(p, bytes);
}

extern "C" int mcg_testing_fail_allocation(int32_t after)
{
  g_fail_alloc_in.store(after < 0 ? -1 : after);
  return MCG_OK;
}

static void free_scratch(mcg_context *ctx)
{
  for (void *p : {(void *)ctx->d_part, (void *)ctx->d_res, (void *)ctx->d_steps, (void *)ctx->d_scat})
    if (p)
      cudaFree(p);
  ctx->d_part = nullptr;
  ctx->d_res = nullptr;
  ctx->d_steps = ctx->d_scat = nullptr;
  ctx->scratch_cap = 0;
}

extern "C" int mcg_destroy(mcg_context *ctx)
{
  if (!ctx)
    return MCG_OK;
  cudaSetDevice(ctx->device);
  if (ctx->stream)
    cudaStreamSynchronize(ctx->stream);
  free_geometry(ctx);
  free_scratch(ctx);
  mcg_fit_release(ctx);
  mcg_ext_destroy(ctx);
  for (void *p : ctx->owned)
    cudaFree(p);
  for (void *p : ctx->event_owned)
    cudaFree(p);
  if (ctx->ev0)
    cudaEventDestroy(ctx->ev0);
  if (ctx->ev1)
    cudaEventDestroy(ctx->ev1);
  if (ctx->stream)
    cudaStreamDestroy(ctx->stream);
  delete ctx;
  return MCG_OK;
}

extern "C" int mcg_set_mode(mcg_context *ctx, int mode)
{
  if (!ctx || (mode != MCG_MODE_STRICT && mode != MCG_MODE_FAST))
    return mcg_fail(MCG_ERR_ARG, "mcg_set_mode: bad arguments");
  int rc = ensure_device(ctx);
  if (rc == MCG_OK && mode == MCG_MODE_STRICT)
    rc = mcg_load_libm(ctx);
  if (rc == MCG_OK)
    ctx->mode = mode;
  return rc;
}

/* Per-cell step parameters exactly as Layer::particle_step forms them
 * (src/layer.cpp:129-131, 146, 150). */
void mcg_cell_params(float sig, float rate, int gi, float dx, float4 &strict, float4 &fast)
{
  const float interaction_rate = (float)(1.0 - (double)rate);
  const float sig_a = sig * rate;
  const float sig_i = sig * interaction_rate;
  const float elo = (float)gi * dx, ehi = (float)(gi + 1) * dx;
  strict = make_float4(sig_a, sig_i, elo, ehi);
  fast = make_float4(sig_a, sig_i > 1e-4f ? sig_i : 0.0f,
                     elo, ehi);
}

/* On the host (mcg_simulate_fast_noalloc). */
void mcg_tile_table(const float4 *c, int n, float4 *tab)
{
  for (int k = 0; k < n; ++k)
    tab[k] = mcg_tile_entry(c, n, k);
}

/* The fast arithmetic's cells (mcg_cell_params), the tile table and, where wanted, a
 * thin chain's two, from the strict cells and with zeros beyond the ends; the tally
 * and the counters cleared (mcg_tally_reset's two launches).  Made on the
 * host and uploaded they were 56 of the 72 bytes per cell (2e6 cells: 26 ms for
 * mcg_set_layers; 15 before there were tiles, 11 so). */
__global__ void mcg_chain_tables(const float4 *strict, int n, float4 *fast, float4 *tab, float2 *thin,
                                 unsigned long long *tally, unsigned long long *counters)
{
  const int row = n + 2 * MCG_TAB_PAD;
  if (blockIdx.x == 0 && threadIdx.x < 16)
    counters[threadIdx.x] = 0ull;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < row;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)i - MCG_TAB_PAD;
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if ((unsigned)k < (unsigned)n) {
      const float4 c = strict[k];
      t = mcg_tile_entry(strict, n, k);
      t.y = c.y > 1e-4f ? c.y : 0.0f;
      fast[k] = make_float4(c.x, t.y, c.z, c.w);
      tally[k] = 0ull;
    }
    tab[i] = t;
    if (thin) {
      thin[i] = make_float2(t.x, t.z);
      thin[row + i] = make_float2(t.x, t.w);
    }
  }
}

/* thin: every cell's absorption optical width, sig_a times the longer of its
 * tile lengths, is at most 2e-4, so that a crossing has u >= MCG_OM_THIN_MAX (2^-8)
 * only for |mu| < 0.05, 0.3 % of the crossings (their share of directions is about
 * mu^2), which go to the full step; thin_fast: both optical widths at most 4e-4 (the
 * short series, below 2^-7, again for |mu| > 0.05).  A transparent chain keeps its
 * slanted particles longer, so the strict line is lower there.  Thin form / other:
 * strict at depth 0.54 to 0.72, 3000 cells, widths (sig_a) 1.4e-4 1.01, 2e-4 1.12;
 * 10,000 cells at depth 1.2 1e-4 .92, 1.8 1.4e-4 .89, 2.4 2e-4 .73; fast, both widths,
 * 3000 and 10,000 cells: 2e-4 .79 and .59, 4e-4 .87 and .68, 6e-4 .92 and .85, 8e-4
 * 1.13 and 1.09.  Whether a run takes it: thin_pays. */
static void update_thin(mcg_context *ctx)
{
  const float4 *cells = ctx->cells_strict.data();
  const int n = (int)ctx->cells_strict.size();
  float wa = 0.0f, wi = 0.0f;
  float own = 0.0f; /* the widest cell between its own faces, in sig_a */
  mcg_widths sum;
  ctx->depth_i = 0.0;
  for (int k = 0; k < n; ++k) {
    const float4 c = cells[k];
    const float len = c.w - c.z;
    sum.add(c);
    ctx->depth_i += c.y > 1e-4f ? (double)c.y * len : 0.0;
    own = std::max(own, std::fabs(c.x) * len);
    /* the widths that bound a whole flight (mcg_thin_tests): of the lengths that
     * the tiles use, since a cell entered from another layer's face may be wider
     * than its own faces are apart (3.7 % at some sub-domains' ends of 10,000
     * cells in 64, without limit between layers of different spacing).  A NaN
     * length has no step in the tiles. */
    const float4 t = mcg_tile_entry(cells, n, k);
    const float entry = t.z > t.w ? t.z : t.w > 0.0f ? t.w : t.z > 0.0f ? t.z : 0.0f;
    wa = std::max(wa, std::fabs(c.x) * entry);
    wi = std::max(wi, std::fabs(c.y) * entry);
  }
  ctx->width_a = wa;
  ctx->width_i = wi;
  ctx->widths = sum;
  ctx->thin_step = n > 0 && own <= 5e-4f;
  ctx->thick = mcg_thick(sum, n, true);
  ctx->thick_fast = mcg_thick(sum, n, false);
  /* a chain of thick cells that hardly any flight may enter in the tiles is both:
   * it takes lanes, whose launch has no thin shape */
  ctx->thin = n > 0 && !ctx->thick && wa <= (sum.a + sum.i < 1.2 ? 7e-5f : 2e-4f);
  ctx->thin_fast = n > 0 && !ctx->thick_fast && std::max(wa, wi) <= 4e-4f;
}

/* Whether the thin form pays for n histories.  It halves the rounds of a history,
 * but its one block of 768 threads per SM holds fewer of them, which short chains
 * feel, and a flight with |mu| < `slant`, which leaves the short forms' range, takes
 * a full step and a round (1.2 to 1.5 us) per cell, `far` of them until it collides
 * or leaves, where the other tiles take 16 at a time: the end of a launch waits for
 * one, and all of them (4e-10 s per round over the GPU) add up.  Thin time / other:
 * without collisions .7 to .8 from 200 cells on, 1.0 at 100, 1.3 at 64, 1.85 at 32,
 * but .75 there for 1e6 cells times histories; widths 1e-4 in both sections, 6e8
 * cells times histories, strict: 1.06 at 300 cells, 1.3 at 1000, 1.7 at 2000, .76 at
 * 10,000; 1e7: 4.3, 5.1, 1.7 and .88; fast, as many: .94, 1.17, 1.12, .57; 3.3, 2.5,
 * 1.6, .73. */
static bool thin_pays(const mcg_context *ctx, bool strict, int64_t n, bool isotropic)
{
  const double m = ctx->n_cells;
  if (m < (n > 65536 ? 100.0 : 16.0))
    return false;
  const double slant = strict ? ctx->width_a / MCG_OM_THIN_MAX : std::max(ctx->width_a, ctx->width_i) * 128.0;
  /* histories with such a flight */
  const double slanted = (double)n * (ctx->depth_i + (isotropic ? 1.0 : 0.0)) * slant;
  if (slanted < 1.5)
    return true;
  const double far = std::min(0.5 * m, slant * m / ctx->depth_i);
  return 7e-13 * (double)n * m * (1.0 + ctx->depth_i) + 1e-7 * m > far * (1.2e-6 + 4e-10 * slanted);
}

/* Chains on which a lane per history is faster than tiles: of up to seven cells, on
 * which a tile is a few steps, and of thick cells, by their mean optical widths,
 * which end a tile's flights or (strict, u < 2^-4) its crossings after a step or
 * two; where absorption ends histories in a few cells, also long chains.  Tiles /
 * lanes, widths sig_a and sig_i: almost nothing 2.2 at one cell, 1.6 at four, 1.15 at
 * eight, .9 at twelve.  Strict .02 and .02 .65 to 1.0; .05, .05 1.5 to 1.7 from 8 to
 * 64 cells, 1.1 at 100, .8 at 200, .6 at 400; .3, .3 2.0 at 24, .86 at 100; .01, .5 1.3
 * at 24, .96 at 64; .1, .01 3.0 at 100, 2.1 at 200, 1.1 at 400.  Fast .05, .05 1.0 at
 * 24, .7 at 100; .1, .1 1.5 at 24, .8 at 100; .01, .1 1.2 at 16, .86 at 48; .05, .3
 * 1.4 at 100, 1.1 at 200; .3, .001 4.3 at 200, 1.7 at 400. */
bool mcg_thick(const mcg_widths &w, int n, bool strict)
{
  if (n < 8)
    return n > 0;
  if (n < 100)
    return strict ? w.a > 0.025 * n || (n < 80 && w.i > 0.25 * n) : w.a + w.i > 0.08 * n;
  return strict ? w.a > 0.05 * n && w.a > 3.0 * w.i : w.a + w.i > 0.25 * n;
}

/* The chain: layers checked, and its cells' two cross sections either from sigs and
 * rates (Layer, mcg_cell_params) or given (xs). */
static int set_geometry(mcg_context *ctx, const char *who, int n_layers, const int32_t *h_index_start,
                        const int32_t *h_m, const float *h_dx, const float *h_a, const float *h_b, bool xs,
                        float particle_min_weight)
{
  if (!ctx || n_layers <= 0 || !h_index_start || !h_m || !h_dx || !h_a || !h_b)
    return mcg_fail(MCG_ERR_ARG, "%s: bad arguments", who);
  int64_t total64 = 0;
  for (int l = 0; l < n_layers; ++l) {
    if (h_m[l] <= 0)
      return mcg_fail(MCG_ERR_ARG, "%s: layer %d has %d cells", who, l, h_m[l]);
    if (l > 0 && (int64_t)h_index_start[l] != (int64_t)h_index_start[l - 1] + h_m[l - 1])
      return mcg_fail(MCG_ERR_ARG, "%s: layer %d is not contiguous", who, l);
    total64 += h_m[l];
    if (total64 > INT32_MAX)
      return mcg_fail(MCG_ERR_ARG, "%s: more than 2^31 - 1 cells", who);
  }
  const int total = (int)total64;
  int rc = ensure_device(ctx);
  if (rc != MCG_OK)
    return rc;
  std::vector<float4> cells;
  std::vector<int32_t> start, m;
  std::vector<float> dx;
  try {
    cells.resize(total);
    start.assign(h_index_start, h_index_start + n_layers);
    m.assign(h_m, h_m + n_layers);
    dx.assign(h_dx, h_dx + n_layers);
  } catch (const std::bad_alloc &) {
    return mcg_fail(MCG_ERR_ARG, "%s: no host memory for %d cells", who, total);
  }
  int k = 0;
  float4 fast;
  for (int l = 0; l < n_layers; ++l)
    for (int j = 0; j < h_m[l]; ++j, ++k)
      if (xs) {
        const int gi = h_index_start[l] + j;
        cells[k] = make_float4(h_a[k], h_b[k], (float)gi * h_dx[l], (float)(gi + 1) * h_dx[l]);
      } else {
        mcg_cell_params(h_a[k], h_b[k], h_index_start[l] + j, h_dx[l], cells[k], fast);
      }
  cudaStreamSynchronize(ctx->stream);
  /* a chain of as many cells takes over the buffers (with the copies on the
   * stream and one synchronisation, a call of the reference's seam with 100
   * cells and 1000 particles takes 167 us instead of 204); otherwise the old
   * geometry goes first; any failure below leaves no geometry */
  cudaError_t e = cudaSuccess;
  if (!ctx->d_tally || ctx->n_cells != total) {
    free_geometry(ctx);
    if ((e = mcg_dev_malloc((void **)&ctx->d_cells_strict, total * sizeof(float4))) == cudaSuccess &&
        (e = mcg_dev_malloc((void **)&ctx->d_cells_fast, total * sizeof(float4))) == cudaSuccess &&
        (e = mcg_dev_malloc((void **)&ctx->d_tab, (total + 2 * (size_t)MCG_TAB_PAD) * sizeof(float4))) == cudaSuccess)
      e = mcg_dev_malloc((void **)&ctx->d_tally, total * sizeof(unsigned long long));
  }
  ctx->n_layers = n_layers;
  ctx->layer_start.swap(start);
  ctx->layer_m.swap(m);
  ctx->layer_dx.swap(dx);
  ctx->cells_strict.swap(cells);
  update_thin(ctx);
  /* the thin tables, for chains that the thin kernel can hold */
  const bool thin = (ctx->thin || ctx->thin_fast) &&
                    mcg_track_shape(total, 256, false, true, (size_t)ctx->smem_optin).thin;
  if (!thin)
    ctx->thin = ctx->thin_fast = false;
  else if (e == cudaSuccess && !ctx->d_thin)
    e = mcg_dev_malloc((void **)&ctx->d_thin, 2 * (total + 2 * (size_t)MCG_TAB_PAD) * sizeof(float2));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(ctx->d_cells_strict, ctx->cells_strict.data(), total * sizeof(float4),
                        cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) {
    mcg_chain_tables<<<(int)std::min<int64_t>(((int64_t)total + 2 * MCG_TAB_PAD + 255) / 256, 8LL * ctx->sm_count),
                       256, 0, ctx->stream>>>(ctx->d_cells_strict, total, ctx->d_cells_fast, ctx->d_tab,
                                              thin ? ctx->d_thin : nullptr, ctx->d_tally, ctx->d_counters);
    e = cudaGetLastError();
    const cudaError_t e2 = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess)
      e = e2;
  }
  if (e != cudaSuccess) {
    free_geometry(ctx);
    return mcg_fail(MCG_ERR_CUDA, "%s: cudaMalloc(layers) or upload: %s", who, cudaGetErrorString(e));
  }
  ctx->n_cells = total;
  ctx->cell_lo = h_index_start[0];
  ctx->min_w = particle_min_weight;
  return MCG_OK;
}

extern "C" int mcg_set_layers(mcg_context *ctx, int n_layers, const int32_t *h_index_start,
                              const int32_t *h_m, const float *h_dx, const float *h_sigs,
                              const float *h_rates, float particle_min_weight)
{
  return set_geometry(ctx, "mcg_set_layers", n_layers, h_index_start, h_m, h_dx, h_sigs, h_rates, false,
                      particle_min_weight);
}

/* Same as mcg_set_layers with the two cross sections of particle_step given
 * per cell directly: sig_a (absorption) and sig_s (flight sampling). */
extern "C" int mcg_set_layers_xs(mcg_context *ctx, int n_layers, const int32_t *h_index_start,
                                 const int32_t *h_m, const float *h_dx, const float *h_sig_a,
                                 const float *h_sig_s, float particle_min_weight)
{
  return set_geometry(ctx, "mcg_set_layers_xs", n_layers, h_index_start, h_m, h_dx, h_sig_a, h_sig_s, true,
                      particle_min_weight);
}

extern "C" int mcg_set_slab(mcg_context *ctx, float x_min, float x_max, int32_t nb_cells,
                            int32_t n_layers, const float *h_sigs, const float *h_rates,
                            float particle_min_weight)
{
  if (!ctx || nb_cells <= 0 || n_layers <= 0 || n_layers > nb_cells || !(x_max > x_min))
    return mcg_fail(MCG_ERR_ARG, "mcg_set_slab: bad arguments");
  std::vector<int32_t> st(n_layers), m(n_layers);
  std::vector<float> dx(n_layers), sigs(nb_cells), rates(nb_cells);
  /* decompose_domain (src/layer.cpp:17-42) and Layer::Layer (:44-69) */
  const int cpl = nb_cells / n_layers, extra = nb_cells % n_layers;
  const float gdx = (x_max - x_min) / ((float)nb_cells);
  for (int r = 0; r < n_layers; ++r) {
    m[r] = cpl + (r < extra);
    st[r] = r * cpl + std::min(r, extra);
    const float lx0 = x_min + (float)st[r] * gdx, lx1 = x_min + (float)(st[r] + m[r]) * gdx;
    dx[r] = (lx1 - lx0) / (float)m[r];
    for (int i = 0; i < m[r]; ++i) {
      const float x_mid = (float)((double)(lx0 + (float)i * dx[r]) + 0.5 * (double)dx[r]);
      sigs[st[r] + i] = h_sigs ? h_sigs[st[r] + i] : expf(-x_mid);
      rates[st[r] + i] = h_rates ? h_rates[st[r] + i] : 0.5f;
    }
  }
  return mcg_set_layers(ctx, n_layers, st.data(), m.data(), dx.data(), sigs.data(), rates.data(),
                        particle_min_weight);
}

extern "C" int mcg_set_tally_scale(mcg_context *ctx, int32_t log2_scale)
{
  if (!ctx || log2_scale < 0 || log2_scale > 62)
    return mcg_fail(MCG_ERR_ARG, "mcg_set_tally_scale: scale 2^%d out of [0, 62]", log2_scale);
  ctx->log2_scale = log2_scale;
  return mcg_tally_reset(ctx);
}

extern "C" int mcg_tally_reset(mcg_context *ctx)
{
  if (!ctx)
    return mcg_fail(MCG_ERR_ARG, "mcg_tally_reset: null context");
  int rc = ensure_device(ctx);
  if (rc != MCG_OK)
    return rc;
  cudaError_t e = cudaMemsetAsync(ctx->d_counters, 0, 16 * sizeof(unsigned long long), ctx->stream);
  if (e == cudaSuccess && ctx->d_tally)
    e = cudaMemsetAsync(ctx->d_tally, 0, ctx->n_cells * sizeof(unsigned long long), ctx->stream);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize(ctx->stream);
  return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(e, "mcg_tally_reset");
}

/* n words of a tally into either or both of the caller's arrays, without a
 * copy between (8.5e6 cells: 8.9 ms -> 3.0 ms). */
cudaError_t mcg_read_tally(mcg_context *ctx, const unsigned long long *d, size_t n, int64_t *h_q,
                           double *h_f64)
{
  static_assert(sizeof(int64_t) == sizeof(double), "a word is turned into a double in its place");
  void *dst = h_q ? (void *)h_q : (void *)h_f64;
  if (!dst)
    return cudaStreamSynchronize(ctx->stream);
  cudaError_t e = cudaMemcpyAsync(dst, d, n * sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess || !h_f64)
    return e;
  const double inv = std::ldexp(1.0, -ctx->log2_scale);
  for (size_t i = 0; i < n; ++i) {
    int64_t q;
    memcpy(&q, static_cast<const char *>(dst) + 8 * i, 8);
    h_f64[i] = (double)q * inv;
  }
  return cudaSuccess;
}

extern "C" int mcg_tally_read(mcg_context *ctx, int64_t *h_q, double *h_f64)
{
  if (!ctx || !ctx->d_tally)
    return mcg_fail(MCG_ERR_STATE, "mcg_tally_read: no layers set");
  int rc = ensure_device(ctx);
  if (rc != MCG_OK)
    return rc;
  cudaError_t e = mcg_read_tally(ctx, ctx->d_tally, ctx->n_cells, h_q, h_f64);
  return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(e, "mcg_tally_read");
}

extern "C" int mcg_counters_read(mcg_context *ctx, mcg_counters *out)
{
  if (!ctx || !out)
    return mcg_fail(MCG_ERR_ARG, "mcg_counters_read: bad arguments");
  int rc = ensure_device(ctx);
  if (rc != MCG_OK)
    return rc;
  unsigned long long c[16];
  cudaError_t e = cudaMemcpyAsync(c, ctx->d_counters, sizeof(c), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_counters_read");
  out->histories = (int64_t)c[MCG_CNT_HIST];
  out->steps = (int64_t)c[MCG_CNT_STEPS];
  out->scatters = (int64_t)c[MCG_CNT_SCAT];
  out->leaked_left = (int64_t)c[MCG_CNT_LEFT];
  out->leaked_right = (int64_t)c[MCG_CNT_RIGHT];
  out->killed = (int64_t)c[MCG_CNT_KILL];
  out->w_left_q = (int64_t)c[MCG_CNT_WLEFT];
  out->w_right_q = (int64_t)c[MCG_CNT_WRIGHT];
  out->w_killed_q = (int64_t)c[MCG_CNT_WKILL];
  out->error_flags = (int64_t)c[MCG_CNT_ERR];
  return MCG_OK;
}

extern "C" int mcg_last_kernel_ms(mcg_context *ctx, float *ms)
{
  if (!ctx || !ms)
    return mcg_fail(MCG_ERR_ARG, "mcg_last_kernel_ms: bad arguments");
  *ms = ctx->last_ms;
  return MCG_OK;
}

extern "C" int mcg_set_launch(mcg_context *ctx, int32_t block, int32_t blocks_per_sm,
                              int32_t refill_steps)
{
  if (!ctx || block < 0 || block > 1024 || (block % 32) || blocks_per_sm < 0 || refill_steps < 0)
    return mcg_fail(MCG_ERR_ARG, "mcg_set_launch: bad arguments");
  ctx->block = block; /* 0: chosen per launch from the chain length */
  ctx->blocks_per_sm = blocks_per_sm;
  ctx->refill = refill_steps; /* 0: chosen per kernel */
  return MCG_OK;
}

extern "C" int mcg_set_tally_mode(mcg_context *ctx, int32_t mode)
{
  if (!ctx || mode < 0 || mode > 2)
    return mcg_fail(MCG_ERR_ARG, "mcg_set_tally_mode: mode must be 0, 1 or 2");
  ctx->tally_mode = mode;
  return MCG_OK;
}

extern "C" int mcg_set_step_limit(mcg_context *ctx, int64_t max_steps)
{
  if (!ctx || max_steps < 1 || max_steps > 0xffffffffll)
    return mcg_fail(MCG_ERR_ARG, "mcg_set_step_limit: limit must be in [1, 2^32-1]");
  ctx->max_steps = (uint32_t)max_steps;
  return MCG_OK;
}

/* ------------------------------------------------------------ launches */
/* The largest |weight| of n particles, as its bits (a NaN is larger than any). */
__global__ void mcg_heaviest_kernel(const mcg_particle *p, int64_t n, uint32_t *out)
{
  uint32_t top = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    top = max(top, __float_as_uint(p[i].wmc) & 0x7fffffffu);
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0)
    atomicMax(out, top);
}

/* One launch of the tracker in the given shape. */
static int track_enqueue(mcg_context *ctx, mcg_track_params &P, const mcg_shape &shape)
{
  const bool strict = ctx->mode == MCG_MODE_STRICT, thin = shape.thin;
  const int block = shape.block;
  const size_t smem = shape.smem;
  P.tally_copies = shape.copies;
  const bool lanes = strict ? ctx->thick : ctx->thick_fast;
  void (*kern)(mcg_track_params);
  if (lanes && strict)
    kern = shape.global ? mcg_track_kernel<true, MCG_TALLY_GLOBAL, false, true>
           : ctx->tally_mode == MCG_TALLY_SMEM64 ? mcg_track_kernel<true, MCG_TALLY_SMEM64, false, true>
                                                 : mcg_track_kernel<true, MCG_TALLY_SMEM32, false, true>;
  else if (lanes)
    kern = shape.global ? mcg_track_kernel<false, MCG_TALLY_GLOBAL, false, true>
           : ctx->tally_mode == MCG_TALLY_SMEM64 ? mcg_track_kernel<false, MCG_TALLY_SMEM64, false, true>
                                                 : mcg_track_kernel<false, MCG_TALLY_SMEM32, false, true>;
  else if (strict)
    kern = thin ? mcg_track_kernel<true, MCG_TALLY_LO32, true>
           : shape.global ? mcg_track_kernel<true, MCG_TALLY_GLOBAL, false>
           : ctx->tally_mode == MCG_TALLY_SMEM64 ? mcg_track_kernel<true, MCG_TALLY_SMEM64, false>
                                                 : mcg_track_kernel<true, MCG_TALLY_SMEM32, false>;
  else
    kern = thin ? mcg_track_kernel<false, MCG_TALLY_LO32, true>
           : shape.global ? mcg_track_kernel<false, MCG_TALLY_GLOBAL, false>
           : ctx->tally_mode == MCG_TALLY_SMEM64 ? mcg_track_kernel<false, MCG_TALLY_SMEM64, false>
                                                 : mcg_track_kernel<false, MCG_TALLY_SMEM32, false>;
  /* the limit is raised to the device's opt-in maximum, the same value on
   * every call, so launches of the same kernel from other host threads (other
   * contexts, the no-allocation entry point) cannot lower it under this one */
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       ctx->smem_optin);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "cudaFuncSetAttribute");
  int bps = ctx->blocks_per_sm;
  if (bps <= 0) {
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, block, smem);
    if (e != cudaSuccess)
      return mcg_cuda_fail(e, "occupancy");
    bps = std::max(bps, 1);
  }
  const int grid = mcg_track_grid(ctx->sm_count * bps, block, P.n, lanes, P);
  if ((e = cudaMemsetAsync(ctx->d_next, 0, sizeof(unsigned long long), ctx->stream)) != cudaSuccess)
    return mcg_cuda_fail(e, "cudaMemsetAsync");
  if (!P.heaviest) /* else the run's time starts with the look at the weights */
    cudaEventRecord(ctx->ev0, ctx->stream);
  kern<<<grid, block, smem, ctx->stream>>>(P);
  e = cudaGetLastError();
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "mcg_track_kernel launch");
  ctx->last_grid = grid;
  ctx->last_block = block;
  ctx->launches++;
  return MCG_OK;
}

int mcg_track_launch(mcg_context *ctx, mcg_particle *d_particles, int64_t n, int32_t *d_results,
                     int64_t *d_steps, int64_t *d_scatters, const mcg_source *src, int64_t first)
{
  if (!ctx->d_tally)
    return mcg_fail(MCG_ERR_STATE, "no layers set (mcg_set_layers / mcg_set_slab)");
  if (n <= 0)
    return MCG_OK;
  const bool strict = ctx->mode == MCG_MODE_STRICT;
  if (strict && !ctx->libm_loaded) {
    int rc = mcg_load_libm(ctx);
    if (rc != MCG_OK)
      return rc;
  }
  mcg_track_params P;
  memset(&P, 0, sizeof(P));
  P.cells = strict ? ctx->d_cells_strict : ctx->d_cells_fast;
  P.tab = mcg_chain_tab(ctx);
  P.n_cells = ctx->n_cells;
  P.cell_lo = ctx->cell_lo;
  P.particles = d_particles;
  P.results = d_results;
  P.steps = d_steps;
  P.scatters = d_scatters;
  P.n = n;
  P.first = first;
  if (src)
    P.src = *src;
  P.next = ctx->d_next;
  P.tally = ctx->d_tally;
  P.counters = ctx->d_counters;
  P.libm = ctx->libm;
  P.libm_tab = ctx->libm_tab;
  P.rules = mcg_rules_setup(ctx, ctx->min_w);
  if (ctx->algorithm == MCG_ALGO_EVENT) {
    ctx->launches++;
    return mcg_event_run(ctx, P);
  }
  /* thin chains take the thin kernel with its tally unless it does not pay (with
   * a block size of the caller's it is taken all the same), the caller set the
   * global tally or a larger block, or the weights are too large for it */
  const bool global = ctx->tally_mode == MCG_TALLY_GLOBAL;
  const float heavy = mcg_heavy_weight(ctx);
  const bool try_thin = (strict ? ctx->thin : ctx->thin_fast) && !global &&
                        ctx->block <= MCG_THIN_BLOCK && !(src && std::fabs(src->w0) >= heavy) &&
                        (ctx->block || thin_pays(ctx, strict, n, src && src->isotropic));
  mcg_shape shape = mcg_track_shape(ctx->n_cells, ctx->block, global, try_thin, (size_t)ctx->smem_optin);
  if (shape.thin && d_particles) {
    /* which of the two forms runs is decided on the device, from the particles:
     * the other's launch returns at once */
    uint32_t *heaviest = reinterpret_cast<uint32_t *>(ctx->d_next + 1);
    cudaError_t e = cudaMemsetAsync(heaviest, 0, sizeof(uint32_t), ctx->stream);
    if (e != cudaSuccess)
      return mcg_cuda_fail(e, "cudaMemsetAsync");
    cudaEventRecord(ctx->ev0, ctx->stream);
    mcg_heaviest_kernel<<<(int)std::min<int64_t>((n + 255) / 256, 4LL * ctx->sm_count), 256, 0,
                          ctx->stream>>>(d_particles, n, heaviest);
    P.heaviest = heaviest;
    memcpy(&P.heavy_line, &heavy, 4);
    if ((e = cudaGetLastError()) != cudaSuccess)
      return mcg_cuda_fail(e, "mcg_heaviest_kernel launch");
    ctx->launches++;
    int rc = track_enqueue(ctx, P, shape);
    if (rc != MCG_OK)
      return rc;
    P.heavy = 1;
    shape = mcg_track_shape(ctx->n_cells, ctx->block, false, false, (size_t)ctx->smem_optin);
  }
  const int rc = track_enqueue(ctx, P, shape);
  cudaEventRecord(ctx->ev1, ctx->stream);
  return rc;
}

int mcg_sync(mcg_context *ctx)
{
  /* the error flags come with the same synchronisation */
  unsigned long long err = 0;
  cudaError_t e = cudaMemcpyAsync(&err, ctx->d_counters + MCG_CNT_ERR, sizeof(err),
                                  cudaMemcpyDeviceToHost, ctx->stream);
  const cudaError_t e2 = cudaStreamSynchronize(ctx->stream);
  if (e2 != cudaSuccess)
    return mcg_cuda_fail(e2, "kernel execution");
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "read error flags");
  cudaEventElapsedTime(&ctx->last_ms, ctx->ev0, ctx->ev1);
  if (err)
    return mcg_fail(MCG_ERR_LIMIT, "a history exceeded the step limit (error flags %llx)", err);
  return MCG_OK;
}

static int ensure_scratch(mcg_context *ctx, int64_t n)
{
  if ((size_t)n <= ctx->scratch_cap)
    return MCG_OK;
  free_scratch(ctx);
  cudaError_t e;
  if ((e = cudaMalloc(&ctx->d_part, n * sizeof(mcg_particle))) != cudaSuccess ||
      (e = cudaMalloc(&ctx->d_res, n * sizeof(int32_t))) != cudaSuccess ||
      (e = cudaMalloc(&ctx->d_steps, n * sizeof(int64_t))) != cudaSuccess ||
      (e = cudaMalloc(&ctx->d_scat, n * sizeof(int64_t))) != cudaSuccess) {
    free_scratch(ctx);
    return mcg_cuda_fail(e, "cudaMalloc(particle buffers)");
  }
  ctx->scratch_cap = (size_t)n;
  return MCG_OK;
}

/* Device address of a page-locked (pinned or registered) host buffer, or
 * nullptr for pageable memory.  Pinned memory is mapped into the device's
 * address space (unified addressing), so the tracker can read and write it
 * in place: over NVLink-C2C on Grace machines, over PCIe elsewhere. */
static void *pinned_device_ptr(const void *h)
{
  if (!h)
    return nullptr;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, h) != cudaSuccess) {
    cudaGetLastError(); /* clear the (non-sticky) error of an unknown pointer */
    return nullptr;
  }
  return a.type == cudaMemoryTypeHost ? a.devicePointer : nullptr;
}

extern "C" int mcg_simulate(mcg_context *ctx, mcg_particle *h_particles, int64_t n,
                            int32_t *h_results, int64_t *h_steps, int64_t *h_scatters)
{
  if (!ctx || n < 0 || (n > 0 && !h_particles))
    return mcg_fail(MCG_ERR_ARG, "mcg_simulate: bad arguments");
  if (n == 0)
    return MCG_OK;
  int rc = ensure_device(ctx);
  if (rc != MCG_OK)
    return rc;
  /* every buffer page-locked: one history reads and writes its 24-byte
   * particle once over ~1e2-1e4 steps, so the tracker works on the host
   * buffers in place instead of copying them through device memory */
  void *zp = pinned_device_ptr(h_particles);
  void *zr = pinned_device_ptr(h_results), *zs = pinned_device_ptr(h_steps);
  void *zc = pinned_device_ptr(h_scatters);
  if (zp && (!h_results || zr) && (!h_steps || zs) && (!h_scatters || zc)) {
    rc = mcg_track_launch(ctx, static_cast<mcg_particle *>(zp), n, static_cast<int32_t *>(zr),
                          static_cast<int64_t *>(zs), static_cast<int64_t *>(zc), nullptr, 0);
    return rc == MCG_OK ? mcg_sync(ctx) : rc;
  }
  rc = ensure_scratch(ctx, n);
  if (rc != MCG_OK)
    return rc;
  cudaError_t e = cudaMemcpyAsync(ctx->d_part, h_particles, n * sizeof(mcg_particle),
                                  cudaMemcpyHostToDevice, ctx->stream);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "cudaMemcpyAsync(particles)");
  rc = mcg_track_launch(ctx, ctx->d_part, n, ctx->d_res, h_steps ? ctx->d_steps : nullptr,
                        h_scatters ? ctx->d_scat : nullptr, nullptr, 0);
  if (rc != MCG_OK)
    return rc;
  e = cudaMemcpyAsync(h_particles, ctx->d_part, n * sizeof(mcg_particle), cudaMemcpyDeviceToHost,
                      ctx->stream);
  if (e == cudaSuccess && h_results)
    e = cudaMemcpyAsync(h_results, ctx->d_res, n * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess && h_steps)
    e = cudaMemcpyAsync(h_steps, ctx->d_steps, n * sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess && h_scatters)
    e = cudaMemcpyAsync(h_scatters, ctx->d_scat, n * sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream);
  if (e != cudaSuccess)
    return mcg_cuda_fail(e, "cudaMemcpyAsync(results)");
  return mcg_sync(ctx);
}

extern "C" int mcg_simulate_device(mcg_context *ctx, mcg_particle *d_particles, int64_t n,
                                   int32_t *d_results, int64_t *d_steps, int64_t *d_scatters)
{
  if (!ctx || n < 0 || (n > 0 && !d_particles))
    return mcg_fail(MCG_ERR_ARG, "mcg_simulate_device: bad arguments");
  int rc = ensure_device(ctx);
  if (rc == MCG_OK)
    rc = mcg_track_launch(ctx, d_particles, n, d_results, d_steps, d_scatters, nullptr, 0);
  return rc == MCG_OK ? mcg_sync(ctx) : rc;
}

extern "C" int mcg_simulate_source(mcg_context *ctx, const mcg_source *src, int64_t first, int64_t n)
{
  if (!ctx || !src || n < 0 || first < 0 || src->seed_mode < 0 || src->seed_mode > 1 ||
      src->isotropic < 0 || src->isotropic > 2)
    return mcg_fail(MCG_ERR_ARG, "mcg_simulate_source: bad arguments");
  int rc = ensure_device(ctx);
  if (rc == MCG_OK)
    rc = mcg_track_launch(ctx, nullptr, n, nullptr, nullptr, nullptr, src, first);
  return rc == MCG_OK ? mcg_sync(ctx) : rc;
}

/* ------------------------------------------------------------ particle source */
__global__ void mcg_make_particles_kernel(mcg_source S, int64_t first, int64_t n, mcg_particle *out)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    mcg_particle p;
    mcg_source_particle(S, first + i, p.seed, p.x, p.mu, p.wmc, p.index);
    out[i] = p;
  }
}

extern "C" int mcg_create_particles(mcg_context *ctx, const mcg_source *src, int64_t first,
                                    int64_t n, mcg_particle *h_out)
{
  if (!ctx || !src || n < 0 || first < 0 || (n > 0 && !h_out))
    return mcg_fail(MCG_ERR_ARG, "mcg_create_particles: bad arguments");
  if (n == 0)
    return MCG_OK;
  int rc = ensure_device(ctx);
  if (rc == MCG_OK)
    rc = ensure_scratch(ctx, n);
  if (rc != MCG_OK)
    return rc;
  int grid = (int)std::min<int64_t>((n + 255) / 256, (int64_t)ctx->sm_count * 8);
  mcg_make_particles_kernel<<<grid, 256, 0, ctx->stream>>>(*src, first, n, ctx->d_part);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h_out, ctx->d_part, n * sizeof(mcg_particle), cudaMemcpyDeviceToHost,
                        ctx->stream);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize(ctx->stream);
  return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(e, "mcg_create_particles");
}

/* ------------------------------------------------------------ cusimulate */
static thread_local mcg_context *g_cu_ctx = nullptr;

extern "C" int mcg_cusimulate(int n, mcg_particle *particles, const float *sigs,
                              const float *absorption_rates, float *weights_absorbed,
                              int min_index, int max_index, float dx)
{
  if (n < 0 || (n > 0 && !particles) || !sigs || !absorption_rates || !weights_absorbed ||
      max_index <= min_index)
    return mcg_fail(MCG_ERR_ARG, "cusimulate: bad arguments");
  int rc = MCG_OK;
  if (!g_cu_ctx) {
    int dev = 0;
    cudaGetDevice(&dev);
    rc = mcg_create(dev, MCG_MODE_STRICT, &g_cu_ctx);
    if (rc != MCG_OK)
      return rc;
  }
  const int m = max_index - min_index;
  /* the reference kernel has no weight cut: run until the particle leaves */
  rc = mcg_set_layers(g_cu_ctx, 1, &min_index, &m, &dx, sigs, absorption_rates, -INFINITY);
  if (rc == MCG_OK)
    rc = mcg_simulate(g_cu_ctx, particles, n, nullptr, nullptr, nullptr);
  if (rc != MCG_OK)
    return rc;
  std::vector<double> t(m);
  rc = mcg_tally_read(g_cu_ctx, nullptr, t.data());
  if (rc == MCG_OK)
    for (int j = 0; j < m; ++j)
      weights_absorbed[j] += (float)t[j];
  return rc;
}

extern "C" void cusimulate(int n, mcg_particle *particles, float const *const sigs,
                           float const *const absorption_rates, float *const weights_absorbed,
                           int min_index, int max_index, float dx)
{
  int rc = mcg_cusimulate(n, particles, sigs, absorption_rates, weights_absorbed, min_index,
                          max_index, dx);
  if (rc != MCG_OK) {
    fprintf(stderr, "cusimulate: %s\n", mcg_last_error());
    exit(rc);
  }
}
