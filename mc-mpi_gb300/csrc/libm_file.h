/*
 * libm_file.h - on-disk layout of the host-libm exception table written by
 * libm_tablegen and read by the library when a strict context is created.
 *
 *   mcg_libm_file header
 *   uint32_t log_pairs[2 * n_log]   (argument bits, host logf result bits)
 *   uint32_t exp_pairs[2 * n_exp]   (argument bits, host expf result bits)
 *
 * The fingerprint hashes the host library's logf/expf, the float-float
 * evaluators of exact_libm.h (value and midpoint distance) and its short forms
 * (value, residue, acceptance bounds), on a fixed set of arguments; the loader
 * recomputes it, so a table made against another C library (another machine) or
 * by another version of the forms is refused instead of silently used.
 * Host-only header; include exact_libm.h first.
 */
#ifndef MCG_LIBM_FILE_H
#define MCG_LIBM_FILE_H

#include <math.h>
#include <stdint.h>
#include <string.h>

#define MCG_LIBM_MAGIC "MCGLIBM3"
#ifndef MCG_TAU_BUCKETS
#define MCG_TAU_BUCKETS 8192
#endif

typedef struct mcg_libm_file {
  char magic[8];
  char libc_version[56];
  uint64_t fingerprint;
  uint32_t n_log, n_exp;
  float logf_relerr; /* max |logf(x) - ln x| / |ln x| over floats x in (0, 1) */
  uint32_t reserved;
  float tau_log[MCG_TAU_BUCKETS];
  float tau_exp[MCG_TAU_BUCKETS];
} mcg_libm_file;

/* Acceptance bounds of mcg_om_thin and mcg_om_mid (exact_libm.h), from the
 * exception table's per-bucket midpoint distances: |r| < b_mid, and
 * |r| < b_thin - c_thin u^2, imply that u is no exception and that the
 * form's error cannot have moved the result over a midpoint.  Near 0 the
 * host library's distances shrink with u^2 (its polynomial's error does), so
 * the thin bound follows them: c_thin is the largest tau / u^2 of the range's
 * buckets plus 16 for the form's own error of about u^2 grid units. */
typedef struct mcg_run_bounds_t {
  float b_thin, c_thin, b_mid;
} mcg_run_bounds_t;

static inline mcg_run_bounds_t mcg_run_bounds(const float *tau_exp)
{
  const double grid = 1.0 / 16777216.0;
  double c = 0.0, t = 0.0;
  for (uint32_t b = MCG_TAU_BUCKETS / 2; b < MCG_TAU_BUCKETS; ++b) {
    float lo; /* the bucket's smallest |argument| */
    uint32_t u = (b << 19) & 0x7fffffffu;
    memcpy(&lo, &u, 4);
    if (tau_exp[b] < 0.0f || !(lo < MCG_OM_MID_MAX))
      continue;
    t = tau_exp[b] > t ? tau_exp[b] : t;
    if (lo < MCG_OM_THIN_MAX) {
      const double v = lo > 0.0f ? tau_exp[b] / ((double)lo * lo) : 1e30;
      c = v > c ? v : c;
    }
  }
  mcg_run_bounds_t r;
  r.b_thin = (float)((0.5 - 1.0 / 262144.0) * grid);
  r.c_thin = (float)((c + 16.0) * grid);
  r.b_mid = (float)((0.5 - t - 1.0 / 2048.0) * grid);
  return r;
}

/* Whether the forms accept u, and their value (the tracker's own tests). */
static inline int mcg_om_thin_ok(float u, const mcg_run_bounds_t *B, float *om)
{
  float r;
  const float uu = u * u;
  *om = mcg_om_thin(u, uu, &r);
  return u < MCG_OM_THIN_MAX && fabsf(r) < fmaf(uu, -B->c_thin, B->b_thin);
}

static inline int mcg_om_mid_ok(float u, const mcg_run_bounds_t *B, float *om)
{
  float r;
  *om = mcg_om_mid(u, u * u, &r);
  return u < MCG_OM_MID_MAX && fabsf(r) < B->b_mid;
}

static inline uint64_t mcg_fnv_word(uint64_t h, float v)
{
  uint32_t u;
  memcpy(&u, &v, 4);
  for (int b = 0; b < 4; ++b) {
    h ^= (u >> (8 * b)) & 0xffu;
    h *= 1099511628211ull;
  }
  return h;
}

/* FNV-1a over the bits of logf/expf and of the evaluators at 8192
 * arguments spread over both domains by a 32-bit LCG (the exp arguments
 * cover both evaluator paths and both signs), and of the short forms with
 * their residues and acceptance bounds: a table is only good for the forms that
 * were checked when it was made. */
static inline uint64_t mcg_libm_fingerprint(const mcg_libm_tab *T)
{
  uint64_t h = 1469598103934665603ull;
  uint32_t s = 12345u;
  for (int i = 0; i < 8192; ++i) {
    s = s * 1664525u + 1013904223u;
    uint32_t ux = (s >> 2) % 0x3f800000u + 1u; /* (0, 1] */
    float x, d, t = 0.0f;
    memcpy(&x, &ux, 4);
    if (i & 1)
      t = (i & 2) ? -x * 17.0f : (i & 4) ? x * 0.005f : -x * 0.005f;
    h = mcg_fnv_word(h, (i & 1) ? expf(t) : logf(x));
    h = mcg_fnv_word(h, (i & 1) ? mcg_exp_ff(t, &d, T) : mcg_log_ff(x, &d, T));
    h = mcg_fnv_word(h, d);
  }
  float tau[MCG_TAU_BUCKETS]; /* some distances, growing with u^2: the bounds' formula counts */
  for (uint32_t b = 0; b < MCG_TAU_BUCKETS; ++b) {
    float lo;
    uint32_t ul = (b << 19) & 0x7fffffffu;
    memcpy(&lo, &ul, 4);
    tau[b] = lo >= 0x1p-14f && lo < MCG_OM_MID_MAX ? (float)(1 + b % 7) * (lo * lo) : -1.0f;
  }
  const mcg_run_bounds_t B = mcg_run_bounds(tau);
  h = mcg_fnv_word(mcg_fnv_word(mcg_fnv_word(h, B.b_thin), B.c_thin), B.b_mid);
  h = mcg_fnv_word(mcg_fnv_word(h, MCG_OM_THIN_MAX), MCG_OM_MID_MAX);
  for (int i = 0; i < 8192; ++i) {
    float u, r;
    s = s * 1664525u + 1013904223u;
    uint32_t ux = 0x33800000u + (s >> 2) % (0x3d800000u - 0x33800000u); /* [2^-24, 2^-4) */
    memcpy(&u, &ux, 4);
    h = mcg_fnv_word(h, mcg_om_mid(u, u * u, &r));
    h = mcg_fnv_word(h, r);
    if (u < MCG_OM_THIN_MAX) {
      h = mcg_fnv_word(h, mcg_om_thin(u, u * u, &r));
      h = mcg_fnv_word(h, r);
    }
  }
  return h;
}

#endif
