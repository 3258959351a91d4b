// liboqmc_b200: C ABI over the sm_100a kernels of the GTO-VMC hot path.
// Host code: validation, the device system tables, launch configuration.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cmath>
#include <string>
#include <map>
#include <vector>
#include <cuda_runtime.h>

#include "oqmc_launch.h"
#include "oqmc_rtc.h"
#include "oqmc_mlp_host.h"
#include "oqmc_mlp_sweep.cuh"
#include "../../include/oqmc_b200.h"

#include "oqmc_ctx.h"

static thread_local char g_create_err[512] = "";

static int set_err(oqmc_ctx* ctx, int code, const char* fmt, const char* extra = "") {
  char* dst = ctx ? ctx->err : g_create_err;
  snprintf(dst, 512, fmt, extra);
  return code;
}

#define OQ_CUDA(ctx, call)                                                    \
  do {                                                                        \
    cudaError_t _e = (call);                                                  \
    if (_e != cudaSuccess) return set_err(ctx, OQ_ERR_CUDA, "CUDA error: %s", \
                                          cudaGetErrorString(_e));            \
  } while (0)

// ---------------------------------------------------------------------------
// f and g harmonics as monomial tables (am = 3, 4), the polynomials of
// _angular_cartesian (OmegaQMC/psi/gto.py:607-671).
// ---------------------------------------------------------------------------
static void build_harm_table(OqHarmTable& t) {
  memset(&t, 0, sizeof(t));
  struct Term { double c; int i, j, k; };
  const double cf1 = sqrt(2.5) * 0.5, cf2 = 3.0 * cf1, cf3 = sqrt(15.0),
               cf4 = sqrt(1.5) * 0.5, cf5 = sqrt(6.0), cf6 = 1.5, cf7 = cf3 * 0.5;
  const double cg1 = 2.9580398915498085, cg2 = 6.2749501990055672,
               cg3 = 2.0916500663351894, cg4 = 1.1180339887498949,
               cg5 = 6.7082039324993694, cg6 = 2.3717082451262845,
               cg7 = 3.1622776601683795, cg8 = 0.55901699437494745,
               cg9 = 3.3541019662496847, cg10 = 0.73950997288745213,
               cg11 = 4.4370598373247132;
  std::vector<std::vector<Term>> f = {
      {{cf2, 2, 1, 0}, {-cf1, 0, 3, 0}},
      {{cf3, 1, 1, 1}},
      {{cf5, 0, 1, 2}, {-cf4, 2, 1, 0}, {-cf4, 0, 3, 0}},
      {{1.0, 0, 0, 3}, {-cf6, 2, 0, 1}, {-cf6, 0, 2, 1}},
      {{cf5, 1, 0, 2}, {-cf4, 3, 0, 0}, {-cf4, 1, 2, 0}},
      {{cf7, 2, 0, 1}, {-cf7, 0, 2, 1}},
      {{-cf2, 1, 2, 0}, {cf1, 3, 0, 0}}};
  std::vector<std::vector<Term>> g = {
      {{cg1, 3, 1, 0}, {-cg1, 1, 3, 0}},
      {{cg2, 2, 1, 1}, {-cg3, 0, 3, 1}},
      {{-cg4, 3, 1, 0}, {-cg4, 1, 3, 0}, {cg5, 1, 1, 2}},
      {{-cg6, 2, 1, 1}, {-cg6, 0, 3, 1}, {cg7, 0, 1, 3}},
      {{0.375, 4, 0, 0}, {0.375, 0, 4, 0}, {0.75, 2, 2, 0}, {1.0, 0, 0, 4},
       {-3.0, 2, 0, 2}, {-3.0, 0, 2, 2}},
      {{-cg6, 3, 0, 1}, {-cg6, 1, 2, 1}, {cg7, 1, 0, 3}},
      {{-cg8, 4, 0, 0}, {cg8, 0, 4, 0}, {cg9, 2, 0, 2}, {-cg9, 0, 2, 2}},
      {{-cg2, 1, 2, 1}, {cg3, 3, 0, 1}},
      {{cg10, 4, 0, 0}, {cg10, 0, 4, 0}, {-cg11, 2, 2, 0}}};
  int n = 0;
  const std::vector<std::vector<Term>>* tabs[2] = {&f, &g};
  for (int a = 0; a < 2; ++a) {
    const auto& tab = *tabs[a];
    for (size_t c = 0; c < tab.size(); ++c) {
      t.first[a][c] = n;
      for (const Term& x : tab[c]) {
        t.coef[n] = x.c;
        t.pow[n] = x.i | (x.j << 4) | (x.k << 8);
        ++n;
      }
    }
    t.first[a][tab.size()] = n;
  }
}

static bool nocc_supported(int n) {
  switch (n) {
    case 1: case 2: case 3: case 4: case 5: case 6: case 7: case 8:
    case 10: case 12: case 14: case 16: return true;
    default: return false;
  }
}

// Switch over the instantiated determinant sizes; EXPR uses N.
#define OQ_CASE(N, EXPR) \
  case N: {              \
    EXPR(N);             \
  } break;
#define OQ_SWITCH(nocc, EXPR)                                                       \
  switch (nocc) {                                                                   \
    OQ_CASE(1, EXPR) OQ_CASE(2, EXPR) OQ_CASE(3, EXPR) OQ_CASE(4, EXPR)             \
    OQ_CASE(5, EXPR) OQ_CASE(6, EXPR) OQ_CASE(7, EXPR) OQ_CASE(8, EXPR)             \
    OQ_CASE(10, EXPR) OQ_CASE(12, EXPR) OQ_CASE(14, EXPR) OQ_CASE(16, EXPR)         \
    default: err = cudaErrorInvalidValue;                                           \
  }

static OqLaunch make_launch(const oqmc_ctx* ctx, void* stream, size_t smem) {
  OqLaunch L;
  L.sys = ctx->d_sys; L.split = ctx->d_split; L.C64 = ctx->d_C64; L.C32 = ctx->d_C32;
  L.ao = ctx->d_ao; L.ao_bytes = ctx->ao_bytes; L.ext = ctx->ao_ext; L.Ct = ctx->d_Ct;
  L.flags = ctx->d_flags; L.stream = (cudaStream_t)stream; L.smem = smem;
  return L;
}

static void compute_split(oqmc_ctx* ctx) {
  OqSystem& S = ctx->hsys;
  for (int g = 0; g < OQ_MAX_GROUP; ++g) ctx->hsplit.r2[g] = 0.0;
  if (!(ctx->tight_alpha > 0.0)) return;
  for (int g = 0; g < S.ngroup; ++g) {
    double r2 = 0.0;
    for (int p = 0; p < S.g_n[g]; ++p) {
      const double a = S.alpha[S.g_off[g] + p];
      if (a > ctx->tight_alpha) r2 = fmax(r2, 25.0 / a);
    }
    ctx->hsplit.r2[g] = r2;
  }
}

// Record an error on a context (used by entry points in other files).

// Threads of a CTA of k_sweeps with `lanes` lanes per walker, and its shared
// memory: `most` threads, halved until the walkers' state fits.
static int sweep_cta(const oqmc_ctx* ctx, int mixed, int lanes, int most, size_t* smem) {
  const size_t real = mixed ? sizeof(float) : sizeof(double);
  const int cache = !mixed && lanes > 1 && ctx->hsys.has_j3;
  const int len = cache && ctx->j3_len <= 2048 ? ctx->j3_len : 0;
  const size_t head = sizeof(OqSystem) + sizeof(OqSplit) +
                      (((size_t)ctx->nbf * ctx->nocc * real + 15) & ~(size_t)15);
  for (int n = most;; n >>= 1) {
    *smem = head + oq_sweep_tile_bytes(ctx->nocc, ctx->natm, n / lanes, real, cache, len);
    if (*smem <= OQ_SMEM_OPTIN || n <= 32) return n;
  }
}

// Times that W walkers on `lanes` lanes each fill the GPU: the CTAs over those
// that are resident at once (registers: 512 threads per SM; shared memory:
// 228 KB with 1 KB of each CTA's for the system).
static int sweep_waves(const oqmc_ctx* ctx, int W, int mixed, int lanes) {
  size_t smem;
  const int n = sweep_cta(ctx, mixed, lanes, 128, &smem), wt = n / lanes;
  const int fit = (int)(228 * 1024 / (smem + 1024)), per_sm = fit < 512 / n ? fit : 512 / n;
  const int ctas = (W + wt - 1) / wt, room = 148 * (per_sm > 0 ? per_sm : 1);
  return (ctas + room - 1) / room;
}

// Lanes per walker of the sweeps: at most as many as there are electrons (all
// orbital rows of a sweep at once), and of these the number with the least
// waves(P) x P^-e: lanes shorten a walker's chain, but by less than they add
// threads, and what an SM holds at once is bounded by registers and, for larger
// molecules, by the walkers' state.  e = 1/2 in FP64 and 1/5 in FP32, where
// every lane sums all pair terms (one wave of H2O, four sweeps, FP64: 484, 340,
// 260 and 172 us on 1, 2, 4 and 8 lanes; mixed 187, 162 and 114).  Four sweeps,
// us, by threads alone (512 per SM) | by this: H2O FP64 30,000 walkers 557 | 485
// (one lane), table-driven 1,348 | 999; N2 FP64 24,000: 887 | 707 (four lanes),
// mixed 30,000: 437 | 332 (one); (H2O)2 mixed 16,384: 719 | 513 (two), FP64
// 30,000: 4,400 | 2,236 (eight).  Above 37,888 walkers (148 x 512 threads on two
// lanes) a walker has one lane.
//
// Three-body terms in FP64 fill 32 lanes, halved while the threads would exceed
// 512 per SM; they take the same time on any number of lanes once the SMs are
// full ((H2O)2, 37,888 walkers, two | eight lanes: 20.7 | 29.1 ms).
//
// Three-body terms in FP32: every lane sums all of them (the order of that sum
// decides moves), so lanes repeat that work and pay only while it hides in idle
// issue slots: all lanes up to a number of threads per SM, one lane beyond.
// Five sweeps, us, all lanes | one lane: H2O 2,048 walkers 3,316 | 3,459, 4,096:
// 3,933 | 3,459; orders (3, 3) 512 walkers 4,311 | 4,352, 4,096: 5,844 | 4,369;
// LiH 8,192: 451 | 520, 16,384: 553 | 520; (H2O)2 2,048: 7,643 | 11,000, 16 lanes
// at 4,096: 9,787 | 11,160.
static int sweep_lanes(const oqmc_ctx* ctx, int W, int mixed) {
  int P = 1;
  while (P < ctx->n_e && P < 32) P <<= 1;
  const OqSystem& S = ctx->hsys;
  if (S.has_j3 && mixed) {
    const int gammas = (S.j3_nI + 1) * (S.j3_nI + 1) * (S.j3_nE + 1);
    const long long cap = 148ll * (P == 2 || P == 32 ? 512 : gammas > 27 ? 128 : 256);
    if (P == 32 && (long long)W * P > cap) P = 16;
    return (long long)W * P > cap ? 1 : P;
  }
  if (2ll * W > 148ll * 512) return 1;
  if (S.has_j3) {
    P = 32;
    while ((long long)W * P > 148ll * 512) P >>= 1;
    return P;
  }
  const double e = mixed ? 0.87 : 0.7071;          // 2^-e
  double f = 1.0, best = 0.0;
  int lanes = 0;
  for (int q = 1; q <= P; q <<= 1, f *= e) {
    const double cost = sweep_waves(ctx, W, mixed, q) * f;
    if (!lanes || cost < 0.98 * best) {            // fewer lanes on a tie
      best = cost;
      lanes = q;
    }
  }
  return lanes;
}

// With one lane per walker, whether the moves run in k_moves instead of
// k_sweeps.  Without compiled-in orbitals, or with three-body terms, the local
// energy costs the fused kernel's moves registers and, at this size, nothing
// is left to share between lanes: 65,536 walkers, us per sweep, k_sweeps |
// k_moves and k_eloc: H2O table-driven 459 | 337 (mixed), 622 | 467 (FP64),
// H2O with three-body terms 2,200 | 1,761 and 3,132 | 1,869.  For few orbitals
// the launches cost more than that: LiH table-driven 85 | 112, with three-body
// terms mixed 155 | 169, but 246 | 237 in FP64, and mixed 16,384 walkers 123 |
// 104.
static bool moves_by_thread(const oqmc_ctx* ctx, int W, int mixed, int lanes) {
  if (lanes != 1 || ctx->nocc < 2) return false;
  if (ctx->nocc < 4) return ctx->spec && ctx->hsys.has_j3 && (!mixed || W <= 148 * 256);
  return !ctx->spec || ctx->hsys.has_j3;
}

// How the single-electron sweeps of W walkers run: lanes per walker, and
// whether the local energies are formed in the sweep kernel too (fused) or by
// k_eloc after each measured sweep.
struct SweepPlan {
  int lanes;
  bool fused;
};

// Lanes, and where the local energies are formed.  Several lanes: in the sweep
// kernel.  One lane: there too, except where k_moves makes the moves and in
// FP64, where a thread's local energy lives in local memory from eight
// orbitals on ((H2O)2, 65,536 walkers: 4,459 us per sweep fused, 2,699 with
// k_eloc; N2, seven orbitals: 658 and 700) and where a CTA size asked for by
// the caller leaves one thread per walker too few warps to hide it (H2O, 1,000
// walkers: 100 and 87 us; 65,536 in CTAs of 32: 332 and 314, of 128: 224 and
// 245).  wpb: walkers per CTA asked for (one lane then), or 0.
static SweepPlan sweep_plan(const oqmc_ctx* ctx, int W, int mixed, int wpb) {
  SweepPlan p;
  p.lanes = wpb ? 1 : sweep_lanes(ctx, W, mixed);
  const bool few = wpb && ctx->nocc >= 5 && (wpb < 128 || W < 148 * 128);
  p.fused = p.lanes > 1 ||
            (!moves_by_thread(ctx, W, mixed, 1) &&
             (mixed || !ctx->spec || (ctx->nocc < 8 && !few)));
  return p;
}

// Largest per-thread local memory (bytes) among the kernels that
// oqmc_refresh followed by oqmc_sweeps launch for W walkers of this context
// and precision (the same dispatch as those two entry points).  Returns OQ_OK
// or an error.
int oq_ctx_sweep_local_bytes(oqmc_ctx* ctx, int W, int precision, size_t* out) {
  const int mixed = precision == OQ_PREC_MIXED;
  size_t best = 0, v = 0;
  cudaError_t err = cudaSuccess;
  auto take = [&](int kind, int M) -> bool {
#define OQ_X(N) err = oq_local_bytes_##N(kind, mixed, ctx->ao_ext, M, &v)
    OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
    if (err != cudaSuccess) return false;
    best = v > best ? v : best;
    return true;
  };
  auto take_rtc = [&](void* fn) -> bool {
    const int b = fn ? oq_rtc_local_bytes(fn) : -1;
    if (b < 0) return false;
    best = (size_t)b > best ? (size_t)b : best;
    return true;
  };
  bool ok = true;
  if (ctx->md) {
    ok = take(4, ctx->md->M) && take(5, ctx->md->M) && take(6, ctx->md->M);
  } else {
    ok = take(0, 0);
    const bool alle = ctx->move_kind == 1, tc = mixed && ctx->use_tc;
    const SweepPlan plan = sweep_plan(ctx, W, mixed, 0);
    if (ok) {
      const int scaled = ctx->proposal == 1;
      if (alle) ok = take(7, 0);
      else if (ctx->mlp) ok = take_rtc(ctx->mlp_fn[ctx->mlp_groups == 4 ? 1 : 0]);
      else if (!moves_by_thread(ctx, W, mixed, plan.lanes))
        ok = ctx->spec ? take_rtc(oq_spec_function(ctx->spec, mixed)) : take(1, 0);
      else
        ok = ctx->spec ? take_rtc(oq_spec_function(ctx->spec, 4 + 2 * scaled + mixed))
                       : take(8 + scaled, 0);
    }
    // the fused sweeps and FP64 all-electron steps hold the local energy
    // themselves
    const bool own = alle ? mixed != 0 : ctx->mlp || tc || !plan.fused;
    if (ok && own) {
      if (tc) ok = take(3, 0);
      else if (ctx->spec) ok = take_rtc(oq_spec_function(ctx->spec, 2 + mixed));
      else ok = take(2, 0);
    }
  }
  if (!ok)
    return set_err(ctx, OQ_ERR_CUDA, "kernel attribute query failed: %s",
                   cudaGetErrorString(err != cudaSuccess ? err : cudaErrorInvalidValue));
  *out = best;
  return OQ_OK;
}

int oq_ctx_set_error(oqmc_ctx* ctx, int code, const char* msg) {
  return set_err(ctx, code, "%s", msg);
}

extern "C" {

const char* oqmc_version(void) { return "oqmc_b200 0.1.0 (sm_100a)"; }

const char* oqmc_last_error(const oqmc_ctx* ctx) { return ctx ? ctx->err : g_create_err; }

// Validate a descriptor and fill the device system tables (host side only).
static int fill_system(const oqmc_system_desc* d, OqSystem& S) {
  if (!d) return set_err(nullptr, OQ_ERR_ARG, "null argument%s");
  if (d->natm < 1 || d->natm > OQ_MAX_NUC)
    return set_err(nullptr, OQ_ERR_UNSUPPORTED, "natm out of range (1..16)%s");
  if (d->n_e != 2 * d->nocc)
    return set_err(nullptr, OQ_ERR_UNSUPPORTED, "only closed shells (n_e = 2 nocc)%s");
  if (!nocc_supported(d->nocc))
    return set_err(nullptr, OQ_ERR_UNSUPPORTED,
                   "nocc must be one of 1-8, 10, 12, 14, 16%s");
  if (d->nbf < d->nocc || d->nbf > OQ_MAX_BF)
    return set_err(nullptr, OQ_ERR_UNSUPPORTED, "nbf out of range%s");
  if (d->ngroup < 1 || d->ngroup > OQ_MAX_GROUP)
    return set_err(nullptr, OQ_ERR_UNSUPPORTED, "too many exponent groups%s");
  memset(&S, 0, sizeof(OqSystem));
  S.natm = d->natm; S.nbf = d->nbf; S.nocc = d->nocc; S.n_e = d->n_e;
  S.ngroup = d->ngroup; S.has_j1 = d->has_j1; S.has_j2 = d->has_j2; S.cusp = d->cusp;
  S.e_nn = d->e_nn;
  for (int i = 0; i < d->natm; ++i) {
    for (int c = 0; c < 3; ++c) S.nuc[i][c] = d->nuc[3 * i + c];
    S.Z[i] = d->Z[i];
    if (d->has_j1) { S.j1a[i] = d->j1[2 * i]; S.j1b[i] = d->j1[2 * i + 1]; }
    if (d->cusp) {
      S.rc[i] = d->cusp_rc[i]; S.q0[i] = d->cusp_q0[i];
      for (int k = 0; k < 8; ++k) S.cc[i][k] = d->cusp_coeff[8 * i + k];
    }
  }
  if (d->has_j2) for (int k = 0; k < 4; ++k) S.j2[k] = d->j2[k];
  int prim = 0, shell = 0, normo = 0, ao = 0;
  for (int g = 0; g < d->ngroup; ++g) {
    const int np = d->group_nprim[g], nc = d->group_ncol[g], am = d->group_am[g];
    const int ia = d->group_atom[g];
    if (np < 1 || nc < 1 || nc > OQ_MAX_COL || am < 0 || am > 4 || ia < 0 || ia >= d->natm ||
        prim + np > OQ_MAX_PRIM || shell + nc > OQ_MAX_SHELL || normo + np * nc > OQ_MAX_NORM)
      return set_err(nullptr, OQ_ERR_UNSUPPORTED, "basis group out of supported range%s");
    S.g_iat[g] = ia; S.g_off[g] = prim; S.g_n[g] = np; S.g_shell0[g] = shell;
    S.g_ncol[g] = nc; S.g_am[g] = am;
    for (int p = 0; p < np; ++p) S.alpha[prim + p] = d->alpha[prim + p];
    for (int k = 0; k < nc; ++k) {
      S.s_ao[shell + k] = ao;
      S.s_norm[shell + k] = normo;
      S.s_cusp[shell + k] = (d->cusp && am == 0) ? d->shell_cusp[shell + k] : 0;
      for (int p = 0; p < np; ++p) S.norm[normo + p] = d->norm[normo + p];
      normo += np;
      ao += 2 * am + 1;
    }
    prim += np;
    shell += nc;
  }
  S.nshell = shell;
  S.nprim_total = prim;
  if (ao != d->nbf) return set_err(nullptr, OQ_ERR_ARG, "group table does not add up to nbf AOs%s");
  if (d->has_bs2) {
    const int nl = d->bs2_ncoef_like, nu = d->bs2_ncoef_unlike;
    if (nl < 6 || nu < 6 || nl > OQ_MAX_BSC || nu > OQ_MAX_BSC || !(d->bs2_rcut > 0.0) ||
        !d->bs2_coef_like || !d->bs2_coef_unlike)
      return set_err(nullptr, OQ_ERR_ARG, "bad two-body B-spline table%s");
    S.has_bs2 = 1;
    S.bs2_n_like = nl - 4;
    S.bs2_n_unlike = nu - 4;
    S.bs2_rcut = d->bs2_rcut;
    S.bs2_dinv_like = (double)(nl - 3) / d->bs2_rcut;
    S.bs2_dinv_unlike = (double)(nu - 3) / d->bs2_rcut;
    for (int k = 0; k < nl; ++k) S.bs2_like[k] = d->bs2_coef_like[k];
    for (int k = 0; k < nu; ++k) S.bs2_unlike[k] = d->bs2_coef_unlike[k];
  }
  for (int i = 0; i < OQ_MAX_NUC; ++i) S.bs1_type[i] = -1;
  if (d->has_bs1) {
    if (d->bs1_ntype < 1 || d->bs1_ntype > OQ_MAX_BST || !d->bs1_type || !d->bs1_ncoef ||
        !d->bs1_rcut || !d->bs1_coef)
      return set_err(nullptr, OQ_ERR_ARG, "bad one-body B-spline table%s");
    S.has_bs1 = 1;
    int off = 0;
    for (int t = 0; t < d->bs1_ntype; ++t) {
      const int n = d->bs1_ncoef[t];
      if (n < 6 || n > OQ_MAX_BSC || !(d->bs1_rcut[t] > 0.0))
        return set_err(nullptr, OQ_ERR_ARG, "bad one-body B-spline table%s");
      S.bs1_n[t] = n - 4;
      S.bs1_rcut[t] = d->bs1_rcut[t];
      S.bs1_dinv[t] = (double)(n - 3) / d->bs1_rcut[t];
      for (int k = 0; k < n; ++k) S.bs1_c[t][k] = d->bs1_coef[off + k];
      off += n;
    }
    for (int i = 0; i < d->natm; ++i) {
      const int t = d->bs1_type[i];
      if (t < -1 || t >= d->bs1_ntype)
        return set_err(nullptr, OQ_ERR_ARG, "bad one-body B-spline atom type%s");
      S.bs1_type[i] = t;
    }
  }
  for (int i = 0; i < OQ_MAX_NUC; ++i) S.j3_type[i] = -1;
  if (d->has_j3) {
    if (d->j3_n_ei < 0 || d->j3_n_ei > 6 || d->j3_n_ee < 1 || d->j3_n_ee > 6 ||
        d->j3_ntype < 1 || d->j3_ntype > OQ_MAX_BST || !(d->j3_rcut > 0.0) || !d->j3_type ||
        !d->j3_on || !d->j3_gamma)
      return set_err(nullptr, OQ_ERR_ARG, "bad three-body Jastrow table%s");
    S.has_j3 = 1;
    S.j3_nI = d->j3_n_ei;
    S.j3_nE = d->j3_n_ee;
    S.j3_L = 0.5 * d->j3_rcut;
    S.j3_gamma = d->j3_gamma;     // host table; oqmc_create points it at a device copy
    for (int t = 0; t < d->j3_ntype; ++t)
      for (int b = 0; b < 2; ++b) S.j3_on[t][b] = d->j3_on[2 * t + b] ? 1 : 0;
    for (int i = 0; i < d->natm; ++i) {
      const int t = d->j3_type[i];
      if (t < -1 || t >= d->j3_ntype)
        return set_err(nullptr, OQ_ERR_ARG, "bad three-body Jastrow atom type%s");
      S.j3_type[i] = t;
    }
  }
  for (int i = 0; i < OQ_MAX_SHELL; ++i) S.s_spl[i] = -1;
  if (d->has_spl) {
    if (d->spl_npts < 3 || d->spl_ntab < 1 || !(d->spl_smin > 0.0) || !d->spl_shell ||
        !d->spl_knots || !d->spl_coef)
      return set_err(nullptr, OQ_ERR_ARG, "bad radial spline table%s");
    S.has_spl = 1;
    S.spl_npts = d->spl_npts;
    S.spl_smin = d->spl_smin;
    S.spl_knots = d->spl_knots;   // host tables; oqmc_create points them at device copies
    S.spl_coef = d->spl_coef;
    for (int i = 0; i < S.nshell; ++i) {
      const int t = d->spl_shell[i];
      if (t < -1 || t >= d->spl_ntab || (t >= 0 && S.s_cusp[i]))
        return set_err(nullptr, OQ_ERR_ARG, "bad radial spline shell table%s");
      S.s_spl[i] = t;
    }
  }
  build_harm_table(S.harm);
  return OQ_OK;
}

// Release a context's multi-determinant expansion.
static void md_free(oqmc_ctx* ctx) {
  OqMdHost* m = ctx->md;
  if (!m) return;
  cudaFree(m->d_C);
  cudaFree(m->d_coef);
  cudaFree(m->d_det);
  cudaFree(m->d_occ);
  cudaFree(m->d_scratch);
  delete m;
  ctx->md = nullptr;
}

// Doubles in the three-body Jastrow table of a descriptor.
static size_t j3_table_len(const oqmc_system_desc* d) {
  if (!d->has_j3) return 0;
  return (size_t)d->j3_ntype * 2 * (d->j3_n_ei + 1) * (d->j3_n_ei + 1) * (d->j3_n_ee + 1);
}

static_assert(sizeof(OqSystem) % 16 == 0, "OqSystem is copied in 16-byte chunks");

static void split_for(const OqSystem& S, double tight_alpha, OqSplit& sp) {
  for (int g = 0; g < OQ_MAX_GROUP; ++g) sp.r2[g] = 0.0;
  if (!(tight_alpha > 0.0)) return;
  for (int g = 0; g < S.ngroup; ++g) {
    double r2 = 0.0;
    for (int p = 0; p < S.g_n[g]; ++p) {
      const double a = S.alpha[S.g_off[g] + p];
      if (a > tight_alpha) r2 = fmax(r2, 25.0 / a);
    }
    sp.r2[g] = r2;
  }
}

}  // extern "C"

// Host-side system tables and split radii for a descriptor (used by the
// batch source generator); err receives the validation message.
int oq_fill_system_desc(const oqmc_system_desc* d, OqSystem* S, OqSplit* SP, int* nocc,
                        std::string* err) {
  const int rc = fill_system(d, *S);
  if (rc != OQ_OK) {
    *err = g_create_err;
    return rc;
  }
  split_for(*S, 50.0, *SP);
  *nocc = d->nocc;
  return OQ_OK;
}

extern "C" {

extern "C" int oqmc_spec_source_desc(const oqmc_system_desc* d, char* buf, size_t len) {
  OqSystem* S = new (std::nothrow) OqSystem();
  if (!S) return OQ_ERR_NOMEM;
  int rc = fill_system(d, *S);
  if (rc != OQ_OK) { delete S; return rc; }
  OqSplit sp;
  split_for(*S, 50.0, sp);
  const std::string src = oq_spec_source(*S, sp, d->C, d->nocc);
  delete S;
  if (buf && len) {
    const size_t n = src.size() < len - 1 ? src.size() : len - 1;
    memcpy(buf, src.data(), n);
    buf[n] = 0;
  }
  return (int)src.size();
}

// The packed tables of the FP64 evaluation (layout at OqAoHead): groups in
// atom order, groups of more than two contraction columns split into pairs.
static std::vector<unsigned char> pack_ao(const OqSystem& S, const double* C) {
  const int N = S.nocc, NP = (N + 1) / 2 * 2;
  std::vector<OqAoAtom> atoms(S.natm);
  std::vector<int4> groups;
  std::vector<double2> prim;
  bool ext = S.has_bs1 || S.has_bs2 || S.has_j3;
  for (int ia = 0; ia < S.natm; ++ia) {
    OqAoAtom& a = atoms[ia];
    memset(&a, 0, sizeof(a));
    a.x = S.nuc[ia][0]; a.y = S.nuc[ia][1]; a.z = S.nuc[ia][2];
    a.Z = S.Z[ia]; a.j1a = S.j1a[ia]; a.j1b = S.j1b[ia];
    a.g0 = (int)groups.size();
    for (int g = 0; g < S.ngroup; ++g) {
      if (S.g_iat[g] != ia) continue;
      for (int k = 0; k < S.g_ncol[g]; k += 2) {
        const int sh = S.g_shell0[g] + k, nc = S.g_ncol[g] - k >= 2 ? 2 : 1;
        int bits = 0;
        for (int c = 0; c < nc; ++c) {
          if (S.g_am[g] == 0 && S.s_cusp[sh + c]) bits |= 0x100 << c;
          if (S.has_spl && S.s_spl[sh + c] >= 0) bits |= 0x400 << c;
        }
        ext = ext || bits || S.g_am[g] > 2;
        groups.push_back(make_int4(S.g_am[g] | nc << 4 | bits | sh << 16, S.g_n[g],
                                   (int)prim.size(), S.s_ao[sh]));
        for (int p = 0; p < S.g_n[g]; ++p) {
          prim.push_back(make_double2(S.alpha[S.g_off[g] + p], S.norm[S.s_norm[sh] + p]));
          if (nc == 2) prim.push_back(make_double2(S.norm[S.s_norm[sh + 1] + p], 0.0));
        }
      }
    }
    a.g1 = (int)groups.size();
  }
  OqAoHead h;
  memset(&h, 0, sizeof(h));
  h.natm = S.natm; h.has_j1 = S.has_j1; h.has_j2 = S.has_j2; h.e_nn = S.e_nn;
  h.ext = ext;
  memcpy(h.j2, S.j2, sizeof(h.j2));
  h.off_group = (int)(sizeof(h) + atoms.size() * sizeof(OqAoAtom));
  h.off_prim = h.off_group + (int)(groups.size() * sizeof(int4));
  h.off_C = h.off_prim + (int)(prim.size() * sizeof(double2));
  h.bytes = h.off_C + (int)(sizeof(double) * S.nbf * NP);
  std::vector<unsigned char> b(h.bytes, 0);
  memcpy(b.data(), &h, sizeof(h));
  memcpy(b.data() + sizeof(h), atoms.data(), atoms.size() * sizeof(OqAoAtom));
  memcpy(b.data() + h.off_group, groups.data(), groups.size() * sizeof(int4));
  memcpy(b.data() + h.off_prim, prim.data(), prim.size() * sizeof(double2));
  double* c = reinterpret_cast<double*>(b.data() + h.off_C);
  for (int a = 0; a < S.nbf; ++a)
    for (int m = 0; m < N; ++m) c[(size_t)a * NP + m] = C[(size_t)a * N + m];
  return b;
}
static_assert(sizeof(OqAoHead) % 16 == 0 && sizeof(OqAoAtom) % 16 == 0,
              "the packed tables are copied in 16-byte chunks");

extern "C" int oqmc_create(oqmc_ctx** out, const oqmc_system_desc* d) {
  if (!out || !d) return set_err(nullptr, OQ_ERR_ARG, "null argument%s");
  *out = nullptr;
  oqmc_ctx* ctx = new (std::nothrow) oqmc_ctx();
  if (!ctx) return set_err(nullptr, OQ_ERR_NOMEM, "out of host memory%s");
  {
    const int rc = fill_system(d, ctx->hsys);
    if (rc != OQ_OK) { delete ctx; return rc; }
  }
  OqSystem& S = ctx->hsys;
  ctx->nocc = d->nocc; ctx->n_e = d->n_e; ctx->nbf = d->nbf; ctx->natm = d->natm;
  ctx->tight_alpha = 50.0;
  ctx->proposal = 0;
  ctx->spec = nullptr;
  ctx->use_tc = 0;
  ctx->d_Btc = nullptr;
  ctx->h_C = new double[(size_t)d->nbf * d->nocc];
  memcpy(ctx->h_C, d->C, sizeof(double) * (size_t)d->nbf * d->nocc);
  ctx->scale_r0 = 1.0;
  ctx->scale_fmin = 0.05;
  compute_split(ctx);
  cudaGetDevice(&ctx->device);
  std::vector<float> c32((size_t)d->nbf * d->nocc);
  for (size_t i = 0; i < c32.size(); ++i) c32[i] = (float)d->C[i];
  cudaError_t e = cudaSuccess;
  e = (e == cudaSuccess) ? cudaMalloc(&ctx->d_sys, sizeof(OqSystem)) : e;
  e = (e == cudaSuccess) ? cudaMalloc(&ctx->d_split, sizeof(OqSplit)) : e;
  e = (e == cudaSuccess) ? cudaMalloc(&ctx->d_C64, sizeof(double) * c32.size()) : e;
  e = (e == cudaSuccess) ? cudaMalloc(&ctx->d_C32, sizeof(float) * c32.size()) : e;
  e = (e == cudaSuccess) ? cudaMalloc(&ctx->d_flags, sizeof(unsigned)) : e;
  if (S.has_j3) {
    const size_t n3 = j3_table_len(d);
    e = (e == cudaSuccess) ? cudaMalloc(&ctx->d_j3, sizeof(double) * n3) : e;
    e = (e == cudaSuccess) ? cudaMemcpy(ctx->d_j3, d->j3_gamma, sizeof(double) * n3,
                                        cudaMemcpyHostToDevice) : e;
    S.j3_gamma = ctx->d_j3;
    ctx->j3_len = (int)n3;
  }
  if (S.has_spl) {
    const size_t nk = (size_t)d->spl_ntab * d->spl_npts;
    const size_t nc = (size_t)d->spl_ntab * (d->spl_npts - 1) * 6;
    e = (e == cudaSuccess) ? cudaMalloc(&ctx->d_spl_knots, sizeof(double) * nk) : e;
    e = (e == cudaSuccess) ? cudaMalloc(&ctx->d_spl_coef, sizeof(double) * nc) : e;
    e = (e == cudaSuccess) ? cudaMemcpy(ctx->d_spl_knots, d->spl_knots, sizeof(double) * nk,
                                        cudaMemcpyHostToDevice) : e;
    e = (e == cudaSuccess) ? cudaMemcpy(ctx->d_spl_coef, d->spl_coef, sizeof(double) * nc,
                                        cudaMemcpyHostToDevice) : e;
    S.spl_knots = ctx->d_spl_knots;
    S.spl_coef = ctx->d_spl_coef;
  }
  const std::vector<unsigned char> ao = pack_ao(S, d->C);
  ctx->ao_bytes = (int)ao.size();
  ctx->ao_ext = reinterpret_cast<const OqAoHead*>(ao.data())->ext;
  std::vector<double> Ct((size_t)d->nbf * d->nocc);
  for (int a = 0; a < d->nbf; ++a)
    for (int m = 0; m < d->nocc; ++m) Ct[(size_t)m * d->nbf + a] = d->C[(size_t)a * d->nocc + m];
  e = (e == cudaSuccess) ? cudaMalloc(&ctx->d_ao, ao.size() + sizeof(double) * Ct.size()) : e;
  e = (e == cudaSuccess) ? cudaMemcpy(ctx->d_ao, ao.data(), ao.size(), cudaMemcpyHostToDevice) : e;
  ctx->d_Ct = reinterpret_cast<double*>(ctx->d_ao + ao.size());
  e = (e == cudaSuccess) ? cudaMemcpy(ctx->d_Ct, Ct.data(), sizeof(double) * Ct.size(),
                                      cudaMemcpyHostToDevice) : e;
  e = (e == cudaSuccess) ? cudaMemcpy(ctx->d_sys, &S, sizeof(OqSystem), cudaMemcpyHostToDevice) : e;
  e = (e == cudaSuccess) ? cudaMemcpy(ctx->d_split, &ctx->hsplit, sizeof(OqSplit), cudaMemcpyHostToDevice) : e;
  e = (e == cudaSuccess) ? cudaMemcpy(ctx->d_C64, d->C, sizeof(double) * c32.size(), cudaMemcpyHostToDevice) : e;
  e = (e == cudaSuccess) ? cudaMemcpy(ctx->d_C32, c32.data(), sizeof(float) * c32.size(), cudaMemcpyHostToDevice) : e;
  e = (e == cudaSuccess) ? cudaMemset(ctx->d_flags, 0, sizeof(unsigned)) : e;
  if (e != cudaSuccess) {
    set_err(nullptr, OQ_ERR_CUDA, "CUDA error in create: %s", cudaGetErrorString(e));
    oqmc_destroy(ctx);
    return OQ_ERR_CUDA;
  }
  *out = ctx;
  return OQ_OK;
}

int oqmc_destroy(oqmc_ctx* ctx) {
  if (!ctx) return OQ_OK;
  oq_spec_destroy(ctx->spec);
  oq_rtc_unload(ctx->mlp_mod);
  cudaFree(ctx->d_Btc);
  delete[] ctx->h_C;
  cudaFree(ctx->d_sys);
  cudaFree(ctx->d_split);
  cudaFree(ctx->d_C64);
  cudaFree(ctx->d_C32);
  cudaFree(ctx->d_ao);
  cudaFree(ctx->d_flags);
  cudaFree(ctx->d_j3);
  cudaFree(ctx->d_spl_knots);
  cudaFree(ctx->d_spl_coef);
  md_free(ctx);
  delete ctx;
  return OQ_OK;
}

int oqmc_set_multidet(oqmc_ctx* ctx, int ndet, int ncol, const double* C, const double* coef,
                      const int* occ_up, const int* occ_dn) {
  if (!ctx) return OQ_ERR_ARG;
  md_free(ctx);
  if (ndet == 0) return OQ_OK;
  const int N = ctx->nocc, nbf = ctx->nbf;
  if (ndet < 0 || ncol < N || !C || !coef || !occ_up || !occ_dn)
    return set_err(ctx, OQ_ERR_ARG, "bad multi-determinant arguments%s");
  // the orbital columns the expansion uses, in increasing order
  std::vector<int> slot(ncol, -1);
  for (int d = 0; d < ndet; ++d)
    for (int sp = 0; sp < 2; ++sp) {
      const int* o = (sp ? occ_dn : occ_up) + (size_t)d * N;
      for (int k = 0; k < N; ++k) {
        if (o[k] < 0 || o[k] >= ncol)
          return set_err(ctx, OQ_ERR_ARG, "orbital index out of range%s");
        for (int q = 0; q < k; ++q)
          if (o[q] == o[k])
            return set_err(ctx, OQ_ERR_ARG, "orbital repeated within a determinant%s");
        slot[o[k]] = 0;
      }
      if (!std::isfinite(coef[d]))
        return set_err(ctx, OQ_ERR_ARG, "non-finite CI coefficient%s");
    }
  int nused = 0;
  for (int c = 0; c < ncol; ++c)
    if (slot[c] == 0) slot[c] = nused++;
  if (nused > 16)
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "multi-determinant expansions may use at most 16 orbitals%s");
  const int M = (nused <= 8 && N <= 8) ? 8 : 16;
  // unique spin determinants (orbital slots in the listed order)
  std::map<std::vector<int>, int> uniq[2];
  std::vector<std::vector<int>> lists[2];
  std::vector<int> det(2 * (size_t)ndet);
  for (int d = 0; d < ndet; ++d)
    for (int sp = 0; sp < 2; ++sp) {
      const int* o = (sp ? occ_dn : occ_up) + (size_t)d * N;
      std::vector<int> key(N);
      for (int k = 0; k < N; ++k) key[k] = slot[o[k]];
      auto it = uniq[sp].find(key);
      int idx;
      if (it == uniq[sp].end()) {
        idx = (int)lists[sp].size();
        uniq[sp][key] = idx;
        lists[sp].push_back(key);
      } else {
        idx = it->second;
      }
      det[2 * (size_t)d + sp] = idx;
    }
  const int nu0 = (int)lists[0].size(), nu1 = (int)lists[1].size();
  if (nu0 > OQ_MD_MAXU || nu1 > OQ_MD_MAXU)
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "at most 64 distinct determinants per spin%s");
  for (int d = 0; d < ndet; ++d) det[2 * (size_t)d + 1] += nu0;
  std::vector<int> occ((size_t)(nu0 + nu1) * N);
  for (int u = 0; u < nu0; ++u)
    for (int k = 0; k < N; ++k) occ[(size_t)u * N + k] = lists[0][u][k];
  for (int u = 0; u < nu1; ++u)
    for (int k = 0; k < N; ++k) occ[(size_t)(nu0 + u) * N + k] = lists[1][u][k];
  std::vector<double> Cp((size_t)nbf * M, 0.0);
  for (int a = 0; a < nbf; ++a)
    for (int c = 0; c < ncol; ++c)
      if (slot[c] >= 0) Cp[(size_t)a * M + slot[c]] = C[(size_t)a * ncol + c];
  OqMdHost* m = new (std::nothrow) OqMdHost();
  if (!m) return set_err(ctx, OQ_ERR_NOMEM, "out of host memory%s");
  m->ndet = ndet; m->nu0 = nu0; m->nu1 = nu1; m->M = M;
  ctx->md = m;
  cudaError_t e = cudaSuccess;
  e = (e == cudaSuccess) ? cudaMalloc(&m->d_C, sizeof(double) * Cp.size()) : e;
  e = (e == cudaSuccess) ? cudaMalloc(&m->d_coef, sizeof(double) * ndet) : e;
  e = (e == cudaSuccess) ? cudaMalloc(&m->d_det, sizeof(int) * det.size()) : e;
  e = (e == cudaSuccess) ? cudaMalloc(&m->d_occ, sizeof(int) * occ.size()) : e;
  e = (e == cudaSuccess) ? cudaMemcpy(m->d_C, Cp.data(), sizeof(double) * Cp.size(),
                                      cudaMemcpyHostToDevice) : e;
  e = (e == cudaSuccess) ? cudaMemcpy(m->d_coef, coef, sizeof(double) * ndet,
                                      cudaMemcpyHostToDevice) : e;
  e = (e == cudaSuccess) ? cudaMemcpy(m->d_det, det.data(), sizeof(int) * det.size(),
                                      cudaMemcpyHostToDevice) : e;
  e = (e == cudaSuccess) ? cudaMemcpy(m->d_occ, occ.data(), sizeof(int) * occ.size(),
                                      cudaMemcpyHostToDevice) : e;
  if (e != cudaSuccess) {
    md_free(ctx);
    return set_err(ctx, OQ_ERR_CUDA, "CUDA error in set_multidet: %s", cudaGetErrorString(e));
  }
  return OQ_OK;
}

int oqmc_multidet_info(const oqmc_ctx* ctx, int* ndet, int* nu_up, int* nu_dn, int* ncol) {
  if (!ctx) return OQ_ERR_ARG;
  const OqMdHost* m = ctx->md;
  if (ndet) *ndet = m ? m->ndet : 0;
  if (nu_up) *nu_up = m ? m->nu0 : 0;
  if (nu_dn) *nu_dn = m ? m->nu1 : 0;
  if (ncol) *ncol = m ? m->M : 0;
  return OQ_OK;
}

int oqmc_set_move_kind(oqmc_ctx* ctx, int kind) {
  if (!ctx) return OQ_ERR_ARG;
  if (kind != 0 && kind != 1) return set_err(ctx, OQ_ERR_ARG, "move kind must be 0 or 1%s");
  ctx->move_kind = kind;
  return OQ_OK;
}

int oqmc_set_proposal(oqmc_ctx* ctx, int kind, double r0, double fmin_frac) {
  if (!ctx) return OQ_ERR_ARG;
  if (kind < 0 || kind > 1 || (kind == 1 && (!(r0 > 0.0) || !(fmin_frac > 0.0) || fmin_frac > 1.0)))
    return set_err(ctx, OQ_ERR_ARG, "bad proposal parameters%s");
  ctx->proposal = kind;
  if (kind == 1) { ctx->scale_r0 = r0; ctx->scale_fmin = fmin_frac; }
  return OQ_OK;
}

int oqmc_set_mlp_proposal(oqmc_ctx* ctx, const oqmc_mlp* m) {
  if (!ctx) return OQ_ERR_ARG;
  if (!m) {
    ctx->mlp = nullptr;
    return OQ_OK;
  }
  if (!ctx->spec)
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "the learned proposal needs a specialised context (oqmc_specialize)%s");
  if (ctx->n_e > 32)
    return set_err(ctx, OQ_ERR_UNSUPPORTED, "the learned proposal handles up to 32 electrons%s");
  if (!ctx->mlp_fn[0]) {
    const std::string src = oq_spec_term_defines({&ctx->hsys}) +
                            "#include \"oqmc_mlp_sweep.cuh\"\n\n" +
                            oq_spec_basis_source(ctx->hsys, ctx->hsplit, ctx->h_C, ctx->nocc,
                                                 "OqSpecBasis");
    const std::string n = std::to_string(ctx->nocc);
    std::vector<void*> fns;
    std::string err;
    if (oq_rtc_build(src, {"k_moves_mlp<" + n + ", OqSpecBasis, 2>",
                           "k_moves_mlp<" + n + ", OqSpecBasis, 4>"},
                     &ctx->mlp_mod, &fns, &err) != 0)
      return set_err(ctx, OQ_ERR_UNSUPPORTED, "%s", err.c_str());
    ctx->mlp_fn[0] = fns[0];
    ctx->mlp_fn[1] = fns[1];
    if (ctx->mlp_groups != 4) ctx->mlp_groups = 2;
  }
  ctx->mlp = m;
  return OQ_OK;
}

int oqmc_set_mlp_groups(oqmc_ctx* ctx, int groups) {
  if (!ctx) return OQ_ERR_ARG;
  if (groups != 2 && groups != 4) return set_err(ctx, OQ_ERR_ARG, "groups must be 2 or 4%s");
  ctx->mlp_groups = groups;
  return OQ_OK;
}

// Jastrow-parameter derivatives, FP64: d ln|psi|/dp
// and dE_L/dp for p = (J2 like a, like b, unlike a, unlike b, J1 a_I, b_I per
// atom), from the positions and the full gradient G of ln|psi| (oqmc_eval).
// For u = a r/(1+b r): du/da = r/den, du/db = -a r^2/den^2; u' = a/den^2,
// u'' = -2ab/den^3; E_L changes only through -1/2 sum_e (lap_e + |G_e|^2).
__device__ __forceinline__ void oq_pade_dp(double a, double b, double r, double du[2],
                                           double dup[2], double dL[2]) {
  const double den = 1.0 + b * r, id = 1.0 / den, id2 = id * id, id3 = id2 * id;
  du[0] = r * id;
  du[1] = -a * r * r * id2;
  dup[0] = id2;
  dup[1] = -2.0 * a * r * id3;
  const double dupp0 = -2.0 * b * id3, dupp1 = -2.0 * a * id3 + 6.0 * a * b * r * id3 * id;
  dL[0] = dupp0 + 2.0 * dup[0] / r;
  dL[1] = dupp1 + 2.0 * dup[1] / r;
}

// One warp per walker.  Every parameter belongs to one lane (or is summed over
// the lanes by shuffles), so nothing is added to global memory: with one
// thread per walker each three-body term read and wrote the derivatives of
// all its gammas there (H2O with three-body orders 2 and 2, 2,048 walkers:
// 2,256 us, 58 with a warp each).  Many walkers of a few pairs each leave most
// lanes idle and go to k_param_derivs_thread instead, see launch_param_derivs.
#define OQ_PD_WARPS 4
// doubles of one listed three-body term: see oq_pd_j3
#define OQ_PD_GEO 16

__device__ __forceinline__ double oq_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Pair p = 0, 1, ... of the list (0,1), (0,2), (1,2), (0,3), ...: i < j.
__device__ __forceinline__ void oq_pair_of(int p, int& i, int& j) {
  j = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)p)) * 0.5f);
  while (j * (j - 1) / 2 > p) --j;
  while (j * (j + 1) / 2 <= p) ++j;
  i = p - j * (j - 1) / 2;
}

// Weight of coefficient k (value, first and second derivative) in the spline
// at r, see oq_bs_val; false when its knots do not reach r.
__device__ __forceinline__ bool oq_bs_weight(double r, double dinv, int n, int k, double& w,
                                             double& w1, double& w2) {
  double t;
  const int i = oq_bs_index<double>(r * dinv, n, t);
  const double t2 = t * t, t3 = t2 * t, s6 = 1.0 / 6.0, s61 = s6 * dinv, s62 = s61 * dinv;
  switch (k - i) {
    case 0:
      w = s6 * (-t3 + 3 * t2 - 3 * t + 1); w1 = s61 * (-3 * t2 + 6 * t - 3); w2 = s62 * (-6 * t + 6);
      break;
    case 1:
      w = s6 * (3 * t3 - 6 * t2 + 4); w1 = s61 * (9 * t2 - 12 * t); w2 = s62 * (18 * t - 12);
      break;
    case 2:
      w = s6 * (-3 * t3 + 3 * t2 + 3 * t + 1); w1 = s61 * (-9 * t2 + 6 * t + 3);
      w2 = s62 * (-18 * t + 6);
      break;
    case 3:
      w = s6 * t3; w1 = s61 * 3 * t2; w2 = s62 * 6 * t;
      break;
    default:
      return false;
  }
  return true;
}

// B-spline parameters of one block (n parameters, at dl, de): P_q is
// coefficient q + 1, and coefficient 0 is P_1 - 2 dr cusp, so it adds to P_1.
// Lane q sums its parameter over the cnt listed terms (r, gd) at list, in
// list order; half: the one-body form.
__device__ __forceinline__ void oq_pd_bspline(const double* list, int cnt, int n, double dinv,
                                              double rcut, bool half, int lane, double* dl,
                                              double* de) {
  for (int q = lane; q < n; q += 32) {
    double sl = 0.0, se = 0.0;
    for (int t = 0; t < cnt; ++t) {
      const double r = list[2 * t], gd = list[2 * t + 1];
      if (!(r < rcut)) continue;
      for (int idx = q + 1; idx >= 0; idx = (q == 1 && idx == 2) ? 0 : -1) {
        double w, w1, w2;
        if (!oq_bs_weight(r, dinv, n, idx, w, w1, w2)) continue;
        const double dL = w2 + 2.0 * w1 / r;
        sl += w;
        se -= half ? 0.5 * (dL + 2.0 * w1 * gd) : dL + w1 * gd;
      }
    }
    dl[q] = sl;
    de[q] = se;
  }
}

// Unique gammas of one three-body block: (l, m, n) with l >= m, ordered
// m, then l, then n (the constraint map's order).
__host__ __device__ static inline int j3_unique(const OqSystem& S) {
  return (S.j3_nI + 1) * (S.j3_nI + 2) / 2 * (S.j3_nE + 1);
}

// x^k and its first and second derivatives; x2, x1, x0 = x^(k-2), x^(k-1), x^k.
__device__ __forceinline__ void oq_pow_d(double x, int k, double& p0, double& p1, double& p2) {
  double x2 = 0.0, x1 = k >= 1 ? 1.0 : 0.0, x0 = 1.0;
  if (k >= 2) x2 = 1.0;
  for (int i = 2; i < k; ++i) x2 *= x;
  if (k >= 2) x1 = x2 * x;
  if (k >= 1) x0 = x1 * x;
  p0 = x0;
  p1 = k * x1;
  p2 = k * (k - 1) * x2;
}

// d log|psi| / d gamma and d E_L / d gamma of the three-body Jastrow for the
// unique gammas of every present block (types in order, like then unlike),
// starting at raw slot `base`.  J3 = -sum u is linear in the gammas, so each
// gamma's derivative is the J3 value, gradient and Laplacian with that
// gamma's monomial (r1^l r2^m + r1^m r2^l for l != m) r12^n in place of the
// polynomial.  For 32 pairs and one nucleus at a time the lanes form the
// geometry of a term each and list the terms inside the cutoff in shared
// memory; then every lane goes through the list with its own monomial.
__device__ void oq_pd_j3(const OqSystem& S, const double* x, const double* g, int n_e, int base,
                         int lane, double* geo, double* dl, double* de) {
  const int NG = j3_unique(S), np = n_e * (n_e - 1) / 2;
  const double L = S.j3_L;
  for (int ty = 0, off = base; ty < OQ_MAX_BST; ++ty) {
    if (!S.j3_on[ty][0] && !S.j3_on[ty][1]) continue;
    for (int u0 = 0; u0 < NG; u0 += 32) {
      // this lane's monomial
      int l = 0, m = 0, n = 0;
      {
        int u = u0 + lane < NG ? u0 + lane : 0;
        while (u >= (S.j3_nI + 1 - m) * (S.j3_nE + 1)) u -= (S.j3_nI + 1 - m++) * (S.j3_nE + 1);
        l = m + u / (S.j3_nE + 1);
        n = u % (S.j3_nE + 1);
      }
      double sl[2] = {0.0, 0.0}, se[2] = {0.0, 0.0};
      for (int I = 0; I < S.natm; ++I) {
        if (S.j3_type[I] != ty) continue;
        for (int p0 = 0; p0 < np; p0 += 32) {
          int i = 0, j = 1;
          bool in = p0 + lane < np;
          if (in) oq_pair_of(p0 + lane, i, j);
          const int blk = (i ^ j) & 1;
          double di[3], dj[3], dij[3];
          for (int c = 0; c < 3; ++c) {
            di[c] = x[3 * i + c] - S.nuc[I][c];
            dj[c] = x[3 * j + c] - S.nuc[I][c];
            dij[c] = x[3 * i + c] - x[3 * j + c];
          }
          const double ri = sqrt(di[0] * di[0] + di[1] * di[1] + di[2] * di[2]);
          const double rj = sqrt(dj[0] * dj[0] + dj[1] * dj[1] + dj[2] * dj[2]);
          in = in && S.j3_on[ty][blk] && ri < L && rj < L;
          const unsigned list = __ballot_sync(0xffffffffu, in);
          const unsigned likes = __ballot_sync(0xffffffffu, in && blk == 0);
          if (list == 0u) continue;
          if (in) {
            const double r12 = sqrt(dij[0] * dij[0] + dij[1] * dij[1] + dij[2] * dij[2]);
            // G_a . e_aI and G_a . e_ab for the two electrons, and the cosines
            double gi1 = 0, gie = 0, gj1 = 0, gje = 0, ci = 0, cj = 0;
            for (int c = 0; c < 3; ++c) {
              const double ei = di[c] / ri, ej = dj[c] / rj, e = dij[c] / r12;
              gi1 += g[3 * i + c] * ei;
              gie += g[3 * i + c] * e;
              gj1 += g[3 * j + c] * ej;
              gje -= g[3 * j + c] * e;
              ci += ei * e;
              cj -= ej * e;
            }
            const double si = ri - L, sj = rj - L;
            double* q = geo + lane * OQ_PD_GEO;
            q[0] = ri; q[1] = rj; q[2] = r12;
            // envelope (r_1I - L)^3 (r_2I - L)^3 and its derivatives over it
            q[3] = si * si * si * sj * sj * sj;
            q[4] = 3.0 * si * si * sj * sj * sj; q[5] = 6.0 * si * sj * sj * sj;
            q[6] = 3.0 * sj * sj * si * si * si; q[7] = 6.0 * sj * si * si * si;
            q[8] = gi1; q[9] = gj1; q[10] = gie + gje;
            q[11] = ci; q[12] = cj;
            q[13] = 2.0 / ri; q[14] = 2.0 / rj; q[15] = 2.0 / r12;
          }
          __syncwarp();
          for (unsigned todo = list; todo; todo &= todo - 1) {
            const int t = __ffs(todo) - 1;
            const double* q = geo + t * OQ_PD_GEO;
            const double a = q[0], b = q[1], r12 = q[2], E = q[3];
            double A, A1, A2, D, D1, D2, e0, e1, e2;
            oq_pow_d(a, l, A, A1, A2);
            oq_pow_d(b, m, D, D1, D2);
            oq_pow_d(r12, n, e0, e1, e2);
            double f = A * D, f1 = A1 * D, f11 = A2 * D, g1 = A * D1, g11 = A * D2;
            if (l != m) {
              oq_pow_d(a, m, A, A1, A2);
              oq_pow_d(b, l, D, D1, D2);
              f += A * D; f1 += A1 * D; f11 += A2 * D; g1 += A * D1; g11 += A * D2;
            }
            // partials of (monomial x envelope) with each electron as particle 1
            const double Ei1 = q[4], Ej1 = q[6];
            const double v = f * e0 * E, ae = f * e1 * E, aee = f * e2 * E;
            const double a1 = e0 * (f1 * E + f * Ei1), b1 = e0 * (g1 * E + f * Ej1);
            const double a11 = e0 * (f11 * E + 2.0 * f1 * Ei1 + f * q[5]);
            const double b11 = e0 * (g11 * E + 2.0 * g1 * Ej1 + f * q[7]);
            const double a1e = e1 * (f1 * E + f * Ei1), b1e = e1 * (g1 * E + f * Ej1);
            // J3 = -sum f: d lap and G . dG of both electrons
            const double lap = a11 + a1 * q[13] + b11 + b1 * q[14] + 2.0 * (aee + ae * q[15]) +
                               2.0 * (a1e * q[11] + b1e * q[12]);
            const double gdg = a1 * q[8] + b1 * q[9] + ae * q[10];
            const int blk_t = (likes >> t) & 1u ? 0 : 1;
            const double dE = 0.5 * lap + gdg;
            sl[0] -= blk_t ? 0.0 : v;
            sl[1] -= blk_t ? v : 0.0;
            se[0] += blk_t ? 0.0 : dE;
            se[1] += blk_t ? dE : 0.0;
          }
          __syncwarp();
        }
      }
      if (u0 + lane < NG) {
        int o = off + u0 + lane;
        if (S.j3_on[ty][0]) {
          dl[o] = sl[0];
          de[o] = se[0];
          o += NG;
        }
        if (S.j3_on[ty][1]) {
          dl[o] = sl[1];
          de[o] = se[1];
        }
      }
    }
    off += NG * (S.j3_on[ty][0] + S.j3_on[ty][1]);
  }
}

static int param_count_of(const OqSystem& S) {
  int n = 4 + 2 * S.natm;
  if (S.has_bs2) n += S.bs2_n_like + S.bs2_n_unlike;
  if (S.has_bs1)
    for (int t = 0; t < OQ_MAX_BST; ++t) n += S.bs1_n[t];
  if (S.has_j3)
    for (int t = 0; t < OQ_MAX_BST; ++t) n += j3_unique(S) * (S.j3_on[t][0] + S.j3_on[t][1]);
  return n;
}

// Shared memory of one warp: positions and gradient [3 n_e] each, the distance
// and gradient-projection list (r, gd) of the electron pairs or of one atom's
// electrons, the raw derivatives, and the listed three-body terms.
static size_t param_derivs_smem(const OqSystem& S) {
  const size_t np = (size_t)S.n_e * (S.n_e - 1) / 2;
  return sizeof(double) * (6 * (size_t)S.n_e + 2 * (np > (size_t)S.n_e ? np : S.n_e) +
                           2 * (size_t)param_count_of(S) + (S.has_j3 ? 32 * OQ_PD_GEO : 0));
}

// Where the derivatives go: the raw ones to dlog, del (W, n_raw) when map is
// null, else their products with map (n_raw, n_flat), zeros left out, to
// dlog, del (W, n_flat).  e_loc (W), when set, receives eparts[., 3].
struct OqPdOut {
  double *dlog, *del;
  const double* map;
  int n_flat, pad;
  const double* eparts;
  double* e_loc;
};

__global__ void __launch_bounds__(32 * OQ_PD_WARPS)
k_param_derivs(const OqSystem* __restrict__ gsys, const double* __restrict__ X,
               const double* __restrict__ G, int W, int n_e, int n_raw, int warp_bytes,
               OqPdOut out) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int w = blockIdx.x * OQ_PD_WARPS + warp;
  if (w >= W) return;
  const OqSystem& S = *gsys;
  const int np = n_e * (n_e - 1) / 2, natm = S.natm;
  double* x = reinterpret_cast<double*>(smem + (size_t)warp * warp_bytes);
  double* g = x + 3 * n_e;
  double* list = g + 3 * n_e;                    // pairs like first, then unlike
  double* dl = list + 2 * max(np, n_e);
  double* de = dl + n_raw;
  double* geo = de + n_raw;
  for (int k = lane; k < 3 * n_e; k += 32) {
    x[k] = X[(size_t)w * n_e * 3 + k];
    g[k] = G[(size_t)w * n_e * 3 + k];
  }
  __syncwarp();
  // electron pairs: two sets, like then unlike, in pair order
  const int h = n_e / 2, nlike = h * (h - 1);
  double al[4] = {0, 0, 0, 0}, ae[4] = {0, 0, 0, 0};
  int cl = 0, cu = 0;
  for (int p0 = 0; p0 < np; p0 += 32) {
    int i = 0, j = 1;
    const bool in = p0 + lane < np;
    if (in) oq_pair_of(p0 + lane, i, j);
    const double dx = x[3 * i] - x[3 * j], dy = x[3 * i + 1] - x[3 * j + 1],
                 dz = x[3 * i + 2] - x[3 * j + 2];
    const double r = sqrt(dx * dx + dy * dy + dz * dz);
    const double gd = ((g[3 * i] - g[3 * j]) * dx + (g[3 * i + 1] - g[3 * j + 1]) * dy +
                       (g[3 * i + 2] - g[3 * j + 2]) * dz) / r;
    const int blk = (i ^ j) & 1;
    if (S.has_j2 && in) {
      double du[2], dup[2], dL[2];
      oq_pade_dp(S.j2[2 * blk], S.j2[2 * blk + 1], r, du, dup, dL);
      for (int q = 0; q < 2; ++q) {
        const double e = dL[q] + dup[q] * gd;
        al[q] += blk ? 0.0 : du[q];
        al[2 + q] += blk ? du[q] : 0.0;
        ae[q] -= blk ? 0.0 : e;
        ae[2 + q] -= blk ? e : 0.0;
      }
    }
    const unsigned lk = __ballot_sync(0xffffffffu, in && !blk);
    const unsigned un = __ballot_sync(0xffffffffu, in && blk);
    const unsigned below = (1u << lane) - 1u;
    if (in) {
      const int at = blk ? nlike + cu + __popc(un & below) : cl + __popc(lk & below);
      list[2 * at] = r;
      list[2 * at + 1] = gd;
    }
    cl += __popc(lk);
    cu += __popc(un);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double sl = oq_warp_sum(al[k]), se = oq_warp_sum(ae[k]);
    if (lane == k) {
      dl[k] = sl;
      de[k] = se;
    }
  }
  __syncwarp();
  int base = 4 + 2 * natm;
  if (S.has_bs2) {
    oq_pd_bspline(list, cl, S.bs2_n_like, S.bs2_dinv_like, S.bs2_rcut, false, lane, dl + base,
                  de + base);
    base += S.bs2_n_like;
    oq_pd_bspline(list + 2 * nlike, cu, S.bs2_n_unlike, S.bs2_dinv_unlike, S.bs2_rcut, false,
                  lane, dl + base, de + base);
    base += S.bs2_n_unlike;
  }
  // electron-nucleus terms, one atom at a time; a B-spline block collects the
  // atoms of its element, so it is summed into place
  const int bs1_base = base;
  if (S.has_bs1) {
    for (int t = 0; t < OQ_MAX_BST; ++t) base += S.bs1_n[t];
    for (int k = bs1_base + lane; k < base; k += 32) dl[k] = de[k] = 0.0;
  }
  for (int I = 0; I < natm; ++I) {
    const int ty = S.has_bs1 ? S.bs1_type[I] : -1;
    double sl[2] = {0.0, 0.0}, se[2] = {0.0, 0.0};
    if (S.has_j1 || ty >= 0) {
      __syncwarp();
      if (lane < n_e) {
        const int e = lane;                       // n_e <= 32
        const double dx = x[3 * e] - S.nuc[I][0], dy = x[3 * e + 1] - S.nuc[I][1],
                     dz = x[3 * e + 2] - S.nuc[I][2];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        const double gd = (g[3 * e] * dx + g[3 * e + 1] * dy + g[3 * e + 2] * dz) / r;
        list[2 * e] = r;
        list[2 * e + 1] = gd;
        if (S.has_j1) {
          double du[2], dup[2], dL[2];
          oq_pade_dp(S.j1a[I], S.j1b[I], r, du, dup, dL);
          for (int q = 0; q < 2; ++q) {
            sl[q] = du[q];
            se[q] = -0.5 * (dL[q] + 2.0 * dup[q] * gd);
          }
        }
      }
      __syncwarp();
    }
    for (int q = 0; q < 2; ++q) {
      const double a = oq_warp_sum(sl[q]), b = oq_warp_sum(se[q]);
      if (lane == q) {
        dl[4 + 2 * I + q] = a;
        de[4 + 2 * I + q] = b;
      }
    }
    if (ty >= 0) {
      int off = bs1_base;
      for (int t = 0; t < ty; ++t) off += S.bs1_n[t];
      // lane q owns parameter q (at most OQ_MAX_BSC of them): adds its own sum
      double tl = 0.0, te = 0.0;
      const int n = S.bs1_n[ty];
      double* pl = dl + off;
      double* pe = de + off;
      if (lane < n) { tl = pl[lane]; te = pe[lane]; }
      oq_pd_bspline(list, n_e, n, S.bs1_dinv[ty], S.bs1_rcut[ty], true, lane, pl, pe);
      if (lane < n) { pl[lane] += tl; pe[lane] += te; }
    }
  }
  if (S.has_j3) oq_pd_j3(S, x, g, n_e, base, lane, geo, dl, de);
  __syncwarp();
  if (lane == 0 && out.e_loc) out.e_loc[w] = out.eparts[(size_t)w * 4 + 3];
  if (!out.map) {
    for (int k = lane; k < n_raw; k += 32) {
      out.dlog[(size_t)w * n_raw + k] = dl[k];
      out.del[(size_t)w * n_raw + k] = de[k];
    }
    return;
  }
  for (int p = lane; p < out.n_flat; p += 32) {
    double sl = 0.0, se = 0.0;
    for (int k = 0; k < n_raw; ++k) {
      const double m = out.map[(size_t)k * out.n_flat + p];
      if (m != 0.0) {
        sl += m * dl[k];
        se += m * de[k];
      }
    }
    out.dlog[(size_t)w * out.n_flat + p] = sl;
    out.del[(size_t)w * out.n_flat + p] = se;
  }
}

// All B-spline parameters that a term at distance r touches, see
// oq_pd_bspline: those of coefficients i..i+3 of its knot interval i, and P_1
// through coefficient 0.
__device__ __forceinline__ void oq_bs_param_add(int n, double dinv, double rcut, double r,
                                                double gd, bool half, double* dl, double* de) {
  if (!(r < rcut)) return;
  double t;
  const int i = oq_bs_index<double>(r * dinv, n, t);
  for (int k = 0; k < 4; ++k) {
    const int idx = i + k, q = idx == 0 ? 1 : idx - 1;
    double w, w1, w2;
    if (q < 0 || q >= n || !oq_bs_weight(r, dinv, n, idx, w, w1, w2)) continue;
    const double dL = w2 + 2.0 * w1 / r;
    dl[q] += w;
    de[q] -= half ? 0.5 * (dL + 2.0 * w1 * gd) : dL + w1 * gd;
  }
}

// The raw derivatives without three-body terms, one thread per walker.
__global__ void __launch_bounds__(128)
k_param_derivs_thread(const OqSystem* __restrict__ gsys, const double* __restrict__ X,
                      const double* __restrict__ G, int W, int n_e, int n_raw,
                      double* __restrict__ dlog, double* __restrict__ del) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= W) return;
  const OqSystem& S = *gsys;
  const int natm = S.natm, bs2 = 4 + 2 * natm;
  const int bs1 = bs2 + (S.has_bs2 ? S.bs2_n_like + S.bs2_n_unlike : 0);
  const double* x = X + (size_t)w * n_e * 3;
  const double* g = G + (size_t)w * n_e * 3;
  double* dl = dlog + (size_t)w * n_raw;
  double* de = del + (size_t)w * n_raw;
  for (int k = 0; k < n_raw; ++k) dl[k] = de[k] = 0.0;
  if (S.has_j2 || S.has_bs2) {
    double al[4] = {0, 0, 0, 0}, ae[4] = {0, 0, 0, 0};
    for (int i = 0; i < n_e; ++i)
      for (int j = i + 1; j < n_e; ++j) {
        const double dx = x[3 * i] - x[3 * j], dy = x[3 * i + 1] - x[3 * j + 1],
                     dz = x[3 * i + 2] - x[3 * j + 2];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        const double gd = ((g[3 * i] - g[3 * j]) * dx + (g[3 * i + 1] - g[3 * j + 1]) * dy +
                           (g[3 * i + 2] - g[3 * j + 2]) * dz) / r;
        const int blk = (i ^ j) & 1;
        if (S.has_j2) {
          double du[2], dup[2], dL[2];
          oq_pade_dp(S.j2[2 * blk], S.j2[2 * blk + 1], r, du, dup, dL);
          for (int q = 0; q < 2; ++q) {
            const double e = dL[q] + dup[q] * gd;
            al[q] += blk ? 0.0 : du[q];
            al[2 + q] += blk ? du[q] : 0.0;
            ae[q] -= blk ? 0.0 : e;
            ae[2 + q] -= blk ? e : 0.0;
          }
        }
        if (S.has_bs2) {
          const int o = bs2 + (blk ? S.bs2_n_like : 0);
          oq_bs_param_add(blk ? S.bs2_n_unlike : S.bs2_n_like,
                          blk ? S.bs2_dinv_unlike : S.bs2_dinv_like, S.bs2_rcut, r, gd, false,
                          dl + o, de + o);
        }
      }
    for (int k = 0; k < 4; ++k) {
      dl[k] = al[k];
      de[k] = ae[k];
    }
  }
  for (int I = 0; I < natm; ++I) {
    const int ty = S.has_bs1 ? S.bs1_type[I] : -1;
    if (!S.has_j1 && ty < 0) continue;
    int o = bs1;
    for (int t = 0; t < ty; ++t) o += S.bs1_n[t];
    double sl[2] = {0.0, 0.0}, se[2] = {0.0, 0.0};
    for (int e = 0; e < n_e; ++e) {
      const double dx = x[3 * e] - S.nuc[I][0], dy = x[3 * e + 1] - S.nuc[I][1],
                   dz = x[3 * e + 2] - S.nuc[I][2];
      const double r = sqrt(dx * dx + dy * dy + dz * dz);
      const double gd = (g[3 * e] * dx + g[3 * e + 1] * dy + g[3 * e + 2] * dz) / r;
      if (S.has_j1) {
        double du[2], dup[2], dL[2];
        oq_pade_dp(S.j1a[I], S.j1b[I], r, du, dup, dL);
        for (int q = 0; q < 2; ++q) {
          sl[q] += du[q];
          se[q] -= 0.5 * (dL[q] + 2.0 * dup[q] * gd);
        }
      }
      if (ty >= 0)
        oq_bs_param_add(S.bs1_n[ty], S.bs1_dinv[ty], S.bs1_rcut[ty], r, gd, true, dl + o, de + o);
    }
    for (int q = 0; q < 2; ++q) {
      dl[4 + 2 * I + q] = sl[q];
      de[4 + 2 * I + q] = se[q];
    }
  }
}

int oqmc_param_count(const oqmc_ctx* ctx) { return ctx ? param_count_of(ctx->hsys) : OQ_ERR_ARG; }

// A thread per walker pays from so many walkers per pair term on, and some
// thousands in all (raw derivatives, us, warp | thread: H2, 5 terms, 8,192
// walkers 27 | 17, 65,536: 116 | 26; LiH, 14 terms, 6,000: 25 | 26, 16,384: 40 |
// 26; H2O, 75 terms, 20,000: 60 | 71, 65,536: 160 | 89; N2, 119 terms, 131,072:
// 329 | 263; with B-splines, whose weights a warp forms again for each
// parameter, H2O 8,192: 177 | 210, 13,000: 258 | 134, H2 1,000: 18 | 25, 65,536:
// 207 | 50).  Beyond sixteen electrons it does not: its positions no longer
// stay in the cache ((H2O)2, 131,072 walkers: 648 | 728).
static int launch_param_derivs(oqmc_ctx* ctx, const double* X, int W, const double* grad,
                               const OqPdOut& out, void* stream) {
  const OqSystem& S = ctx->hsys;
  const int terms = S.n_e * (S.n_e - 1) / 2 + S.n_e * S.natm;
  if (!out.map && !S.has_j3 && S.n_e <= 16 && W > 4000 &&
      W > (S.has_bs1 || S.has_bs2 ? 140 : 400) * terms) {
    k_param_derivs_thread<<<(W + 127) / 128, 128, 0, (cudaStream_t)stream>>>(
        ctx->d_sys, X, grad, W, ctx->n_e, param_count_of(S), out.dlog, out.del);
    OQ_CUDA(ctx, cudaGetLastError());
    return OQ_OK;
  }
  const size_t wbytes = param_derivs_smem(ctx->hsys), sm = OQ_PD_WARPS * wbytes;
  if (sm > 48 * 1024)
    OQ_CUDA(ctx, cudaFuncSetAttribute(k_param_derivs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      OQ_SMEM_OPTIN));
  k_param_derivs<<<(W + OQ_PD_WARPS - 1) / OQ_PD_WARPS, 32 * OQ_PD_WARPS, sm,
                   (cudaStream_t)stream>>>(ctx->d_sys, X, grad, W, ctx->n_e,
                                           param_count_of(ctx->hsys), (int)wbytes, out);
  OQ_CUDA(ctx, cudaGetLastError());
  return OQ_OK;
}

int oqmc_param_derivs(oqmc_ctx* ctx, const double* X, int W, const double* grad, double* dlogpsi,
                      double* dEL, void* stream) {
  if (!ctx) return OQ_ERR_ARG;
  if (W < 0 || (W > 0 && (!X || !grad || !dlogpsi || !dEL)))
    return set_err(ctx, OQ_ERR_ARG, "bad arguments%s");
  if (W == 0) return OQ_OK;
  return launch_param_derivs(ctx, X, W, grad, OqPdOut{dlogpsi, dEL, nullptr, 0, 0, nullptr, nullptr},
                             stream);
}

int oqmc_param_derivs_mapped(oqmc_ctx* ctx, const double* X, int W, const double* grad,
                             const double* eparts, const double* map, int n_flat, double* e_loc,
                             double* dlogpsi, double* dEL, void* stream) {
  if (!ctx) return OQ_ERR_ARG;
  if (W < 0 || n_flat < 1 ||
      (W > 0 && (!X || !grad || !eparts || !map || !e_loc || !dlogpsi || !dEL)))
    return set_err(ctx, OQ_ERR_ARG, "bad arguments%s");
  if (W == 0) return OQ_OK;
  return launch_param_derivs(ctx, X, W, grad, OqPdOut{dlogpsi, dEL, map, n_flat, 0, eparts, e_loc},
                             stream);
}

// TF32 rounding as cvt.rna (nearest, ties away from zero) and BF16 (nearest even)
static float host_tf32(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  u = (u + 0x1000u) & 0xFFFFE000u;
  memcpy(&f, &u, 4);
  return f;
}
static uint16_t host_bf16(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  return (uint16_t)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16);
}

int oqmc_use_tensor_cores(oqmc_ctx* ctx, int enable) {
  if (ctx && enable && ctx->md)
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "the tensor-core local energy supports single determinants only%s");
  if (ctx && enable && ctx->hsys.has_spl)
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "the tensor-core local energy uses analytic radial functions only%s");
  if (ctx && enable && (ctx->hsys.has_bs1 || ctx->hsys.has_bs2 || ctx->hsys.has_j3))
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "the tensor-core local energy supports Pade Jastrow terms only%s");
  if (!ctx) return OQ_ERR_ARG;
  if (!enable) { ctx->use_tc = 0; return OQ_OK; }
  if (ctx->nocc > 16 || 128 / ctx->n_e < 1)
    return set_err(ctx, OQ_ERR_UNSUPPORTED, "tensor-core local energy needs n_occ <= 16%s");
  const OqTcPlan P = oq_tc_plan(ctx->nbf);
  if (P.total > 227u * 1024u)
    return set_err(ctx, OQ_ERR_UNSUPPORTED, "basis too large for the tensor-core tile%s");
  if (!ctx->d_Btc) {
    std::vector<unsigned char> h(P.b_end - P.b_hi, 0);
    const int KC4 = (int)(P.K4 >> 2), KC2 = (int)(P.K2 >> 3);
    for (int n = 0; n < 16; ++n)
      for (int k = 0; k < ctx->nbf; ++k) {
        const float c = n < ctx->nocc ? (float)ctx->h_C[(size_t)k * ctx->nocc + n] : 0.0f;
        const float hi = host_tf32(c), lo = c - hi;
        const uint32_t o4 = (uint32_t)(((n >> 3) * KC4 + (k >> 2)) << 7) + ((n & 7) << 4) + ((k & 3) << 2);
        const uint32_t o2 = (uint32_t)(((n >> 3) * KC2 + (k >> 3)) << 7) + ((n & 7) << 4) + ((k & 7) << 1);
        memcpy(&h[(P.b_hi - P.b_hi) + o4], &hi, 4);
        memcpy(&h[(P.b_lo - P.b_hi) + o4], &lo, 4);
        const uint16_t bf = host_bf16(hi);
        memcpy(&h[(P.b_bf - P.b_hi) + o2], &bf, 2);
      }
    OQ_CUDA(ctx, cudaMalloc(&ctx->d_Btc, h.size()));
    OQ_CUDA(ctx, cudaMemcpy(ctx->d_Btc, h.data(), h.size(), cudaMemcpyHostToDevice));
  }
  ctx->use_tc = 1;
  return OQ_OK;
}

int oqmc_specialize(oqmc_ctx* ctx, int enable) {
  if (!ctx) return OQ_ERR_ARG;
  oq_spec_destroy(ctx->spec);
  ctx->spec = nullptr;
  if (!enable) return OQ_OK;
  if (ctx->hsys.has_spl)
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "specialised kernels use analytic radial functions; the radial-spline "
                   "transform runs on the table-driven kernels%s");
  std::string err;
  OqSpecModule* m = nullptr;
  if (oq_spec_build(ctx->hsys, ctx->hsplit, ctx->h_C, ctx->nocc, &m, &err) != 0)
    return set_err(ctx, OQ_ERR_UNSUPPORTED, "specialisation unavailable: %s", err.c_str());
  ctx->spec = m;
  return OQ_OK;
}

int oqmc_spec_source(const oqmc_ctx* ctx, char* buf, size_t len) {
  if (!ctx) return OQ_ERR_ARG;
  const std::string s = oq_spec_source(ctx->hsys, ctx->hsplit, ctx->h_C, ctx->nocc);
  if (buf && len) {
    const size_t n = s.size() < len - 1 ? s.size() : len - 1;
    memcpy(buf, s.data(), n);
    buf[n] = 0;
  }
  return (int)s.size();
}

int oqmc_set_split(oqmc_ctx* ctx, double tight_alpha) {
  if (!ctx) return OQ_ERR_ARG;
  ctx->tight_alpha = tight_alpha;
  compute_split(ctx);
  if (ctx->spec) {   // the specialised kernels carry the split radii as literals
    const int rc = oqmc_specialize(ctx, 1);
    if (rc != OQ_OK) return rc;
  }
  if (ctx->mlp_mod) {   // so does the learned-proposal kernel: rebuild it
    oq_rtc_unload(ctx->mlp_mod);
    ctx->mlp_mod = ctx->mlp_fn[0] = ctx->mlp_fn[1] = nullptr;
    const oqmc_mlp* m = ctx->mlp;
    ctx->mlp = nullptr;
    if (m) {
      const int rc = oqmc_set_mlp_proposal(ctx, m);
      if (rc != OQ_OK) return rc;
    }
  }
  OQ_CUDA(ctx, cudaMemcpy(ctx->d_split, &ctx->hsplit, sizeof(OqSplit), cudaMemcpyHostToDevice));
  return OQ_OK;
}

static size_t real_size(int precision);

static cudaError_t to_soa(const oqmc_ctx* ctx, const double* X, double* pos, int W,
                          cudaStream_t s);

static int md_eval(oqmc_ctx* ctx, const double* X, int W, double* logpsi, double* grad,
                   double* lap, double* eparts, void* stream);

int oqmc_eval(oqmc_ctx* ctx, const double* X, int W, double* logpsi, double* grad,
              double* lap, double* eparts, void* stream) {
  if (!ctx) return OQ_ERR_ARG;
  if (W < 0 || (W > 0 && (!X || !logpsi))) return set_err(ctx, OQ_ERR_ARG, "bad arguments%s");
  if (W == 0) return OQ_OK;
  if (ctx->md) return md_eval(ctx, X, W, logpsi, grad, lap, eparts, stream);
  const OqLaunch L = make_launch(ctx, stream, 0);
  cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_eval_##N(L, X, W, logpsi, grad, lap, eparts)
  OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
  OQ_CUDA(ctx, err);
  return OQ_OK;
}

int oqmc_log_psi(oqmc_ctx* ctx, const double* X, int W, double* logpsi, void* stream) {
  if (!ctx) return OQ_ERR_ARG;
  if (W < 0 || (W > 0 && (!X || !logpsi))) return set_err(ctx, OQ_ERR_ARG, "bad arguments%s");
  if (W == 0) return OQ_OK;
  if (ctx->md) return md_eval(ctx, X, W, logpsi, nullptr, nullptr, nullptr, stream);
  const OqLaunch L = make_launch(ctx, stream, 0);
  cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_logpsi_##N(L, X, W, logpsi)
  OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
  OQ_CUDA(ctx, err);
  return OQ_OK;
}

int oqmc_mo_values(oqmc_ctx* ctx, const double* X, int W, double* out, void* stream) {
  if (!ctx) return OQ_ERR_ARG;
  if (W < 0 || (W > 0 && (!X || !out))) return set_err(ctx, OQ_ERR_ARG, "bad arguments%s");
  if (W == 0) return OQ_OK;
  const OqLaunch L = make_launch(ctx, stream, 0);
  cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_movals_##N(L, X, W, out)
  OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
  OQ_CUDA(ctx, err);
  return OQ_OK;
}

static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Sampler state: [pos SoA 3*n_e*W doubles][ainv 2*nocc^2*W Real][logdet W doubles]
struct OqStatePtrs {
  double* pos;
  void* ainv;
  double* logdet;
};

static size_t real_size(int precision) {
  return precision == OQ_PREC_MIXED ? sizeof(float) : sizeof(double);
}

// Multi-determinant sampler state: [pos SoA][inverses (nu0+nu1) nocc^2 W]
// [log|det| (nu0+nu1) W][signs (nu0+nu1) W], all FP64.
static size_t md_state_bytes(const oqmc_ctx* ctx, int W) {
  const size_t nu = (size_t)ctx->md->nu0 + ctx->md->nu1;
  return align256((size_t)3 * ctx->n_e * W * sizeof(double)) +
         align256(nu * ctx->nocc * ctx->nocc * W * sizeof(double)) +
         2 * align256(nu * W * sizeof(double));
}

static OqMdState md_state(const oqmc_ctx* ctx, void* state, int W) {
  const size_t nu = (size_t)ctx->md->nu0 + ctx->md->nu1;
  OqMdState st;
  char* b = static_cast<char*>(state);
  st.pos = reinterpret_cast<double*>(b);
  b += align256((size_t)3 * ctx->n_e * W * sizeof(double));
  st.ainv = reinterpret_cast<double*>(b);
  b += align256(nu * ctx->nocc * ctx->nocc * W * sizeof(double));
  st.ldet = reinterpret_cast<double*>(b);
  b += align256(nu * W * sizeof(double));
  st.sgn = reinterpret_cast<double*>(b);
  st.W = W;
  st.pad = 0;
  return st;
}

static OqMdTables md_tables(const oqmc_ctx* ctx) {
  const OqMdHost* m = ctx->md;
  OqMdTables T;
  T.C = m->d_C; T.coef = m->d_coef; T.det = m->d_det; T.occ = m->d_occ;
  T.ndet = m->ndet; T.nu0 = m->nu0; T.nu1 = m->nu1; T.pad = 0;
  return T;
}

// Multi-determinant evaluation from scratch: FP64 refresh of a scratch state,
// then the local-energy kernel with the per-walker outputs.
static int md_eval(oqmc_ctx* ctx, const double* X, int W, double* logpsi, double* grad,
                   double* lap, double* eparts, void* stream) {
  OqMdHost* m = ctx->md;
  cudaStream_t s = (cudaStream_t)stream;
  if (m->scratch_w < W) {
    OQ_CUDA(ctx, cudaStreamSynchronize(s));
    cudaFree(m->d_scratch);
    m->d_scratch = nullptr;
    m->scratch_w = 0;
    OQ_CUDA(ctx, cudaMalloc(&m->d_scratch, md_state_bytes(ctx, W)));
    m->scratch_w = W;
  }
  const OqMdState st = md_state(ctx, m->d_scratch, W);
  const OqMdTables T = md_tables(ctx);
  OQ_CUDA(ctx, to_soa(ctx, X, st.pos, W, s));
  const OqLaunch L = make_launch(ctx, stream, sizeof(OqSystem));
  OqElocArgs a;
  memset(&a, 0, sizeof(a));
  a.pos = st.pos; a.W = W; a.eparts = eparts; a.flags = ctx->d_flags;
  cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_md_refresh_##N(L, T, st, m->M)
  OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
  OQ_CUDA(ctx, err);
#define OQ_X(N) err = oq_md_local_##N(L, T, st, a, logpsi, grad, lap, m->M)
  OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
  OQ_CUDA(ctx, err);
  return OQ_OK;
}

size_t oqmc_state_bytes(const oqmc_ctx* ctx, int W, int precision) {
  if (!ctx || W < 0) return 0;
  if (ctx->md) return md_state_bytes(ctx, W);
  return align256((size_t)3 * ctx->n_e * W * sizeof(double)) +
         align256((size_t)2 * ctx->nocc * ctx->nocc * W * real_size(precision)) +
         align256((size_t)W * sizeof(double));
}

static OqStatePtrs state_ptrs(const oqmc_ctx* ctx, void* state, int W, int precision) {
  OqStatePtrs p;
  char* b = static_cast<char*>(state);
  p.pos = reinterpret_cast<double*>(b);
  b += align256((size_t)3 * ctx->n_e * W * sizeof(double));
  p.ainv = b;
  b += align256((size_t)2 * ctx->nocc * ctx->nocc * W * real_size(precision));
  p.logdet = reinterpret_cast<double*>(b);
  return p;
}

// (W, n3) row-major <-> [n3][W]
__global__ void k_aos_to_soa(const double* __restrict__ X, double* __restrict__ pos, int W,
                             int n3) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)W * n3) return;
  const int w = (int)(t / n3), k = (int)(t % n3);
  pos[(size_t)k * W + w] = X[t];
}

__global__ void k_soa_to_aos(const double* __restrict__ pos, double* __restrict__ X, int W,
                             int n3) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)W * n3) return;
  const int w = (int)(t / n3), k = (int)(t % n3);
  X[t] = pos[(size_t)k * W + w];
}

static cudaError_t to_soa(const oqmc_ctx* ctx, const double* X, double* pos, int W,
                          cudaStream_t s) {
  const long long n = (long long)W * 3 * ctx->n_e;
  k_aos_to_soa<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(X, pos, W, 3 * ctx->n_e);
  return cudaGetLastError();
}

static cudaError_t to_aos(const oqmc_ctx* ctx, const double* pos, double* X, int W,
                          cudaStream_t s) {
  const long long n = (long long)W * 3 * ctx->n_e;
  k_soa_to_aos<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(pos, X, W, 3 * ctx->n_e);
  return cudaGetLastError();
}

static bool valid_prec(int p) { return p == OQ_PREC_FP64 || p == OQ_PREC_MIXED; }

int oqmc_refresh(oqmc_ctx* ctx, const double* X, int W, void* state, int precision,
                 void* stream) {
  if (!ctx) return OQ_ERR_ARG;
  if (W < 0 || (W > 0 && (!X || !state)) || !valid_prec(precision))
    return set_err(ctx, OQ_ERR_ARG, "bad arguments%s");
  if (W == 0) return OQ_OK;
  cudaStream_t s = (cudaStream_t)stream;
  if (ctx->md) {
    if (precision != OQ_PREC_FP64)
      return set_err(ctx, OQ_ERR_UNSUPPORTED,
                     "multi-determinant trials are sampled in FP64 only%s");
    const OqMdState st = md_state(ctx, state, W);
    OQ_CUDA(ctx, to_soa(ctx, X, st.pos, W, s));
    const OqLaunch L = make_launch(ctx, stream, sizeof(OqSystem));
    const OqMdTables T = md_tables(ctx);
    cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_md_refresh_##N(L, T, st, ctx->md->M)
    OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
    OQ_CUDA(ctx, err);
    return OQ_OK;
  }
  const OqStatePtrs st = state_ptrs(ctx, state, W, precision);
  OQ_CUDA(ctx, to_soa(ctx, X, st.pos, W, s));
  const OqLaunch L = make_launch(ctx, stream, 0);
  const int mixed = precision == OQ_PREC_MIXED;
  cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_refresh_##N(L, st.pos, W, st.ainv, st.logdet, mixed)
  OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
  OQ_CUDA(ctx, err);
  return OQ_OK;
}

static size_t moves_smem(const oqmc_ctx* ctx, int wpb, int precision) {
  const size_t rs = real_size(precision);
  size_t b = sizeof(OqSystem) + sizeof(OqSplit);
  b += ((size_t)ctx->nbf * ctx->nocc * rs + 15) & ~(size_t)15;
  b += (size_t)3 * ctx->n_e * wpb * sizeof(double);
  b += (size_t)2 * ctx->nocc * ctx->nocc * wpb * rs;
  return b;
}

static size_t eloc_smem(const oqmc_ctx* ctx, int precision) {
  size_t b = sizeof(OqSystem) + sizeof(OqSplit);
  b += ((size_t)ctx->nbf * ctx->nocc * real_size(precision) + 15) & ~(size_t)15;
  b += (size_t)ctx->n_e * 4 * 32 * sizeof(double);
  return b;
}

static int pick_wpb(oqmc_ctx* ctx, int wpb, int precision, size_t* sm) {
  if (wpb == 0) wpb = 128;
  if (wpb != 32 && wpb != 64 && wpb != 128) return -1;
  *sm = moves_smem(ctx, wpb, precision);
  while (*sm > 227 * 1024 && wpb > 32) { wpb /= 2; *sm = moves_smem(ctx, wpb, precision); }
  if (*sm > 227 * 1024) return -2;
  return wpb;
}

// Launch the moves `m` describes with one thread per walker (the learned
// proposal: its tiles): sweeps (mode 0) or basin relocations (mode 1).
static int launch_moves(oqmc_ctx* ctx, const OqMoveArgs& m, int wpb, size_t sm, int precision,
                        void* stream) {
  const int mixed = precision == OQ_PREC_MIXED;
  const OqLaunch L = make_launch(ctx, stream, sm);
  if (ctx->mlp && m.mode == 0) {
    OqMoveArgs mm = m;
    const void* C = (const void*)ctx->d_C32;
    OqMlpWeights nw{ctx->mlp->wbf, ctx->mlp->theta};
    void* args[5] = {(void*)&L.sys, (void*)&L.split, (void*)&C, (void*)&mm, (void*)&nw};
    const int G = ctx->mlp_groups == 4 ? 4 : 2;
    if (oq_rtc_launch(ctx->mlp_fn[G == 4 ? 1 : 0], dim3((m.W + 128 * G - 1) / (128 * G)),
                      dim3(128 * G), oq_mlp_sweep_smem(G, ctx->n_e), L.stream, args) != 0)
      return set_err(ctx, OQ_ERR_CUDA, "learned-proposal move kernel launch failed%s");
    return OQ_OK;
  }
  if (ctx->spec && m.mode == 0) {
    OqMoveArgs mm = m;
    const void* C = mixed ? (const void*)ctx->d_C32 : (const void*)ctx->d_C64;
    void* args[4] = {(void*)&L.sys, (void*)&L.split, (void*)&C, (void*)&mm};
    if (oq_spec_launch(ctx->spec, (m.proposal == 1 ? 6 : 4) + mixed,
                       dim3((m.W + wpb - 1) / wpb), dim3(wpb), sm, L.stream, args) != 0)
      return set_err(ctx, OQ_ERR_CUDA, "specialised move kernel launch failed%s");
    return OQ_OK;
  }
  cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_moves_##N(L, m, wpb, mixed)
  OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
  OQ_CUDA(ctx, err);
  return OQ_OK;
}

// Launch the sweeps `a` describes with a.lanes lanes per walker; wpb1 is the
// CTA size that fits with one lane.
static int launch_sweeps(oqmc_ctx* ctx, OqSweepArgs a, int wpb1, int precision, void* stream) {
  const int mixed = precision == OQ_PREC_MIXED;
  size_t smem;
  const int nthr = sweep_cta(ctx, mixed, a.lanes, a.lanes == 1 ? wpb1 : 128, &smem);
  a.j3_cache = !mixed && a.lanes > 1 && ctx->hsys.has_j3;
  a.j3_len = a.j3_cache && ctx->j3_len <= 2048 ? ctx->j3_len : 0;
  const OqLaunch L = make_launch(ctx, stream, smem);
  if (ctx->spec) {
    const void* C = mixed ? (const void*)ctx->d_C32 : (const void*)ctx->d_C64;
    void* args[4] = {(void*)&L.sys, (void*)&L.split, (void*)&C, (void*)&a};
    const int wt = nthr / a.lanes;
    if (oq_spec_launch(ctx->spec, mixed, dim3((a.W + wt - 1) / wt), dim3(nthr), L.smem, L.stream,
                       args) != 0)
      return set_err(ctx, OQ_ERR_CUDA, "specialised sweep kernel launch failed%s");
    return OQ_OK;
  }
  cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_sweeps_##N(L, a, nthr, mixed)
  OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
  OQ_CUDA(ctx, err);
  return OQ_OK;
}

static OqSweepArgs sweep_args(const oqmc_ctx* ctx, double* X, int W, const OqStatePtrs& st) {
  OqSweepArgs a;
  memset(&a, 0, sizeof(a));
  a.X = X; a.pos = st.pos; a.ainv = st.ainv; a.logdet = st.logdet; a.W = W;
  a.proposal = ctx->proposal; a.scale_r0 = ctx->scale_r0; a.scale_fmin = ctx->scale_fmin;
  a.flags = ctx->d_flags;
  return a;
}

static int md_moves(oqmc_ctx* ctx, const OqMoveArgs& m, double* sgn, void* stream) {
  const OqLaunch L = make_launch(ctx, stream, sizeof(OqSystem));
  const OqMdTables T = md_tables(ctx);
  cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_md_moves_##N(L, T, m, sgn, ctx->md->M)
  OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
  OQ_CUDA(ctx, err);
  return OQ_OK;
}

// Sweeps with a multi-determinant Slater part (FP64; the same measurement
// layout as the single-determinant sweeps).
static int md_sweeps(oqmc_ctx* ctx, double* X, int W, void* state, int precision, int n_sweeps,
                     int measure_every, double step, uint64_t seed, uint64_t step_base,
                     double* sums, double* el_trace, double* eparts_last, void* stream) {
  if (precision != OQ_PREC_FP64)
    return set_err(ctx, OQ_ERR_UNSUPPORTED, "multi-determinant trials are sampled in FP64 only%s");
  if (ctx->mlp)
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "the learned proposal does not support multi-determinant trials%s");
  cudaStream_t s = (cudaStream_t)stream;
  const OqMdState st = md_state(ctx, state, W);
  const OqMdTables T = md_tables(ctx);
  OQ_CUDA(ctx, to_soa(ctx, X, st.pos, W, s));
  OqMoveArgs m;
  memset(&m, 0, sizeof(m));
  m.pos = st.pos; m.ainv = st.ainv; m.logdet = st.ldet; m.W = W; m.mode = 0;
  m.step = step; m.seed = seed; m.flags = ctx->d_flags;
  m.proposal = ctx->proposal; m.scale_r0 = ctx->scale_r0; m.scale_fmin = ctx->scale_fmin;
  OqElocArgs el;
  memset(&el, 0, sizeof(el));
  el.pos = st.pos; el.W = W; el.flags = ctx->d_flags;
  const OqLaunch Le = make_launch(ctx, stream, sizeof(OqSystem));
  const int n_meas = n_sweeps / measure_every;
  int done = 0;
  for (int k = 0; k < n_meas; ++k) {
    m.n_steps = measure_every;
    m.step_base = step_base + done;
    m.acc_sum = sums + (size_t)k * OQ_NSUM + 5;
    int rc = md_moves(ctx, m, st.sgn, stream);
    if (rc != OQ_OK) return rc;
    done += measure_every;
    el.sums = sums + (size_t)k * OQ_NSUM;
    el.el_trace = el_trace ? el_trace + (size_t)k * W : nullptr;
    el.eparts = (k == n_meas - 1) ? eparts_last : nullptr;
    cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_md_local_##N(Le, T, st, el, nullptr, nullptr, nullptr, ctx->md->M)
    OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
    OQ_CUDA(ctx, err);
  }
  if (done < n_sweeps) {
    m.n_steps = n_sweeps - done;
    m.step_base = step_base + done;
    m.acc_sum = nullptr;
    int rc = md_moves(ctx, m, st.sgn, stream);
    if (rc != OQ_OK) return rc;
  }
  OQ_CUDA(ctx, to_aos(ctx, st.pos, X, W, s));
  return OQ_OK;
}

int oqmc_sweeps(oqmc_ctx* ctx, double* X, int W, void* state, int precision, int n_sweeps,
                int measure_every, double step, uint64_t seed, uint64_t step_base,
                double* sums, double* el_trace, double* eparts_last, int wpb,
                void* stream) {
  if (!ctx) return OQ_ERR_ARG;
  if (W < 0 || n_sweeps < 0 || measure_every < 1 || !(step > 0.0) || !valid_prec(precision))
    return set_err(ctx, OQ_ERR_ARG, "bad arguments%s");
  if (W == 0 || n_sweeps == 0) return OQ_OK;
  if (!X || !state || (n_sweeps >= measure_every && !sums))
    return set_err(ctx, OQ_ERR_ARG, "null buffer%s");
  if (ctx->mlp && precision != OQ_PREC_MIXED)
    return set_err(ctx, OQ_ERR_UNSUPPORTED, "the learned proposal runs in mixed precision only%s");
  if (ctx->mlp && ctx->move_kind == 1)
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "the learned proposal moves one electron at a time%s");
  if (ctx->md && ctx->move_kind == 1)
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "all-electron steps are built for single determinants%s");
  if (ctx->md)
    return md_sweeps(ctx, X, W, state, precision, n_sweeps, measure_every, step, seed, step_base,
                     sums, el_trace, eparts_last, stream);
  size_t sm;
  const int wpb_asked = wpb;
  wpb = pick_wpb(ctx, wpb, precision, &sm);
  if (wpb == -1) return set_err(ctx, OQ_ERR_ARG, "walkers_per_block must be 32, 64 or 128%s");
  if (wpb < 0)
    return set_err(ctx, OQ_ERR_UNSUPPORTED, "system too large for the shared-memory move kernel%s");
  cudaStream_t s = (cudaStream_t)stream;
  const OqStatePtrs st = state_ptrs(ctx, state, W, precision);
  const int mixed = precision == OQ_PREC_MIXED;
  const bool tc = mixed && ctx->use_tc;
  OqSweepArgs sa = sweep_args(ctx, X, W, st);
  sa.step = step; sa.seed = seed; sa.step_base = step_base;
  const SweepPlan plan = sweep_plan(ctx, W, mixed, wpb_asked);
  sa.lanes = plan.lanes;
  if (ctx->move_kind == 0 && !ctx->mlp && !tc && plan.fused) {
    sa.n_sweeps = n_sweeps; sa.measure_every = n_sweeps >= measure_every ? measure_every : 0;
    sa.sums = sums; sa.el_trace = el_trace; sa.eparts_last = eparts_last;
    return launch_sweeps(ctx, sa, wpb, precision, stream);
  }
  OqAlleArgs aa;
  memset(&aa, 0, sizeof(aa));
  aa.X = X; aa.pos = st.pos; aa.ainv = st.ainv; aa.logdet = st.logdet; aa.W = W;
  aa.step = step; aa.seed = seed; aa.step_base = step_base; aa.flags = ctx->d_flags;
  auto alle = [&]() -> int {
    const OqLaunch La = make_launch(ctx, stream, 0);
    cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_alle_##N(La, aa, mixed)
    OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
    OQ_CUDA(ctx, err);
    return OQ_OK;
  };
  if (ctx->move_kind == 1 && !mixed) {
    aa.n_steps = n_sweeps; aa.measure_every = n_sweeps >= measure_every ? measure_every : 0;
    aa.sums = sums; aa.el_trace = el_trace; aa.eparts_last = eparts_last;
    return alle();
  }
  // mixed all-electron steps, the learned proposal, the tensor-core local
  // energy, sweeps that sweep_plan does not fuse: moves and local energies in
  // separate launches
  const bool threads =
      ctx->move_kind == 0 && (ctx->mlp || moves_by_thread(ctx, W, mixed, plan.lanes));
  if (threads) OQ_CUDA(ctx, to_soa(ctx, X, st.pos, W, s));
  OqMoveArgs m;
  memset(&m, 0, sizeof(m));
  m.pos = st.pos; m.ainv = st.ainv; m.logdet = st.logdet; m.W = W; m.mode = 0;
  m.step = step; m.seed = seed; m.flags = ctx->d_flags;
  m.proposal = ctx->proposal; m.scale_r0 = ctx->scale_r0; m.scale_fmin = ctx->scale_fmin;
  auto moves = [&](int n, int at, double* acc) -> int {
    m.n_steps = sa.n_sweeps = aa.n_steps = n;
    m.step_base = sa.step_base = aa.step_base = step_base + at;
    m.acc_sum = sa.acc_sum = aa.acc_sum = acc;
    if (ctx->move_kind == 1) return alle();
    return threads ? launch_moves(ctx, m, wpb, sm, precision, stream)
                   : launch_sweeps(ctx, sa, wpb, precision, stream);
  };
  OqElocArgs el;
  memset(&el, 0, sizeof(el));
  el.pos = st.pos; el.ainv = st.ainv; el.W = W; el.flags = ctx->d_flags;
  const OqLaunch Le = make_launch(ctx, stream, eloc_smem(ctx, precision));
  const int n_meas = n_sweeps / measure_every;
  int done = 0;
  for (int k = 0; k < n_meas; ++k) {
    int rc = moves(measure_every, done, sums + (size_t)k * OQ_NSUM + 5);
    if (rc != OQ_OK) return rc;
    done += measure_every;
    el.sums = sums + (size_t)k * OQ_NSUM;
    el.el_trace = el_trace ? el_trace + (size_t)k * W : nullptr;
    el.eparts = (k == n_meas - 1) ? eparts_last : nullptr;
    if (tc) {
      cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_eloc_tc_##N(Le, el, ctx->d_Btc, ctx->nbf)
      OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
      OQ_CUDA(ctx, err);
      continue;
    }
    if (ctx->spec) {
      OqElocArgs ee = el;
      const void* C = mixed ? (const void*)ctx->d_C32 : (const void*)ctx->d_C64;
      void* args[4] = {(void*)&Le.sys, (void*)&Le.split, (void*)&C, (void*)&ee};
      if (oq_spec_launch(ctx->spec, mixed ? 3 : 2, dim3((W + 31) / 32), dim3(32, ctx->n_e),
                         Le.smem, Le.stream, args) != 0)
        return set_err(ctx, OQ_ERR_CUDA, "specialised local-energy kernel launch failed%s");
      continue;
    }
    cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_eloc_##N(Le, el, mixed)
    OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
    OQ_CUDA(ctx, err);
  }
  if (done < n_sweeps) {
    int rc = moves(n_sweeps - done, done, nullptr);
    if (rc != OQ_OK) return rc;
  }
  if (threads) OQ_CUDA(ctx, to_aos(ctx, st.pos, X, W, s));
  return OQ_OK;
}

// One step of the reference's step-size rule (_adapt_step_size,
// OmegaQMC/vmc_gto.py:121-126) after a sweep of k_moves: with the acceptance
// ratio acc = (*accepted) * inv_moves of the sweep just made,
// log s <- log s + rate (acc - target).  Records the ratio in place of the
// count and the new width in step_trace (if set).  One thread.
__global__ void k_adapt_step(double* __restrict__ step, double* __restrict__ accepted,
                             double inv_moves, double rate, double target,
                             double* __restrict__ step_trace) {
  const double acc = *accepted * inv_moves;
  const double s = exp(log(*step) + rate * (acc - target));
  *step = s;
  *accepted = acc;
  if (step_trace) *step_trace = s;
}

int oqmc_equilibrate(oqmc_ctx* ctx, double* X, int W, void* state, int precision,
                     int n_steps, double* step, double target, double rate, uint64_t seed,
                     uint64_t step_base, int refresh_every, int since_refresh,
                     double* acc_trace, double* step_trace, void* stream) {
  if (!ctx) return OQ_ERR_ARG;
  if (W < 0 || n_steps < 0 || refresh_every < 1 || since_refresh < 0 || !valid_prec(precision))
    return set_err(ctx, OQ_ERR_ARG, "bad arguments%s");
  if (W == 0 || n_steps == 0) return OQ_OK;
  if (!X || !state || !step || !acc_trace) return set_err(ctx, OQ_ERR_ARG, "null buffer%s");
  if (ctx->md || ctx->mlp || ctx->move_kind != 0)
    return set_err(ctx, OQ_ERR_UNSUPPORTED,
                   "device-side equilibration runs single-determinant, single-electron "
                   "Gaussian sweeps only%s");
  size_t sm;
  const int wpb = pick_wpb(ctx, 0, precision, &sm);
  if (wpb < 0)
    return set_err(ctx, OQ_ERR_UNSUPPORTED, "system too large for the shared-memory move kernel%s");
  cudaStream_t s = (cudaStream_t)stream;
  const OqStatePtrs st = state_ptrs(ctx, state, W, precision);
  OQ_CUDA(ctx, cudaMemsetAsync(acc_trace, 0, sizeof(double) * (size_t)n_steps, s));
  OqSweepArgs a = sweep_args(ctx, X, W, st);
  a.n_sweeps = 1; a.seed = seed; a.step_dev = step; a.rate = rate; a.target = target;
  a.inv_moves = 1.0 / ((double)W * ctx->n_e);
  a.tick = 1.0;
  while (a.tick <= (double)W * ctx->n_e) a.tick *= 2.0;
  const OqLaunch Lr = make_launch(ctx, stream, 0);
  const int mixed = precision == OQ_PREC_MIXED;
  a.lanes = sweep_plan(ctx, W, mixed, 0).lanes;
  const bool threads = moves_by_thread(ctx, W, mixed, a.lanes);
  OqMoveArgs m;
  memset(&m, 0, sizeof(m));
  m.pos = st.pos; m.ainv = st.ainv; m.logdet = st.logdet; m.W = W; m.n_steps = 1;
  m.step_dev = step; m.seed = seed; m.flags = ctx->d_flags;
  m.proposal = ctx->proposal; m.scale_r0 = ctx->scale_r0; m.scale_fmin = ctx->scale_fmin;
  if (threads) OQ_CUDA(ctx, to_soa(ctx, X, st.pos, W, s));
  int since = since_refresh;
  for (int t = 0; t < n_steps; ++t) {
    const bool refresh = since + 1 >= refresh_every;
    a.step_base = m.step_base = step_base + t;
    a.acc_sum = m.acc_sum = acc_trace + t;
    a.step_trace = step_trace ? step_trace + t : nullptr;
    // the state's own positions are read by the refresh and after the call
    a.pos = refresh || t == n_steps - 1 ? st.pos : nullptr;
    const int rc = threads ? launch_moves(ctx, m, wpb, sm, precision, stream)
                           : launch_sweeps(ctx, a, wpb, precision, stream);
    if (rc != OQ_OK) return rc;
    if (threads) {
      k_adapt_step<<<1, 1, 0, s>>>(step, a.acc_sum, a.inv_moves, rate, target, a.step_trace);
      OQ_CUDA(ctx, cudaGetLastError());
    }
    ++since;
    if (refresh) {
      cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_refresh_##N(Lr, st.pos, W, st.ainv, st.logdet, mixed)
      OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
      OQ_CUDA(ctx, err);
      since = 0;
    }
  }
  if (threads) OQ_CUDA(ctx, to_aos(ctx, st.pos, X, W, s));
  return OQ_OK;
}

int oqmc_state_eval(oqmc_ctx* ctx, const void* state, int W, int precision, double* logpsi,
                    double* grad, double* lap, double* eparts, void* stream) {
  if (!ctx) return OQ_ERR_ARG;
  if (W < 0 || !valid_prec(precision)) return set_err(ctx, OQ_ERR_ARG, "bad arguments%s");
  if (W == 0) return OQ_OK;
  if (!state) return set_err(ctx, OQ_ERR_ARG, "null buffer%s");
  cudaStream_t s = (cudaStream_t)stream;
  if (ctx->md) {
    if (precision != OQ_PREC_FP64)
      return set_err(ctx, OQ_ERR_UNSUPPORTED,
                     "multi-determinant trials are sampled in FP64 only%s");
    // the expansion's local-energy kernel on the state's inverses
    const OqMdState st = md_state(ctx, const_cast<void*>(state), W);
    const OqMdTables T = md_tables(ctx);
    const OqLaunch L = make_launch(ctx, stream, sizeof(OqSystem));
    OqElocArgs a;
    memset(&a, 0, sizeof(a));
    a.pos = st.pos; a.W = W; a.eparts = eparts; a.flags = ctx->d_flags;
    cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_md_local_##N(L, T, st, a, logpsi, grad, lap, ctx->md->M)
    OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
    OQ_CUDA(ctx, err);
    return OQ_OK;
  }
  const OqStatePtrs st = state_ptrs(ctx, const_cast<void*>(state), W, precision);
  const int mixed = precision == OQ_PREC_MIXED;
  if (logpsi)
    OQ_CUDA(ctx, cudaMemcpyAsync(logpsi, st.logdet, sizeof(double) * (size_t)W,
                                 cudaMemcpyDeviceToDevice, s));
  OqElocArgs el;
  memset(&el, 0, sizeof(el));
  el.pos = st.pos; el.ainv = st.ainv; el.W = W; el.flags = ctx->d_flags;
  el.eparts = eparts; el.logpsi = logpsi; el.grad = grad; el.lap = lap;
  const OqLaunch Le = make_launch(ctx, stream, eloc_smem(ctx, precision));
  if (ctx->spec) {
    // the specialised kernel the sweeps use (the tensor-core form has no
    // per-electron outputs)
    const void* C = mixed ? (const void*)ctx->d_C32 : (const void*)ctx->d_C64;
    void* args[4] = {(void*)&Le.sys, (void*)&Le.split, (void*)&C, (void*)&el};
    if (oq_spec_launch(ctx->spec, mixed ? 3 : 2, dim3((W + 31) / 32), dim3(32, ctx->n_e),
                       Le.smem, Le.stream, args) != 0)
      return set_err(ctx, OQ_ERR_CUDA, "specialised local-energy kernel launch failed%s");
    return OQ_OK;
  }
  cudaError_t err = cudaSuccess;
#define OQ_X(N) err = oq_eloc_##N(Le, el, mixed)
  OQ_SWITCH(ctx->nocc, OQ_X)
#undef OQ_X
  OQ_CUDA(ctx, err);
  return OQ_OK;
}

int oqmc_basin(oqmc_ctx* ctx, double* X, int W, void* state, int precision, int n_steps,
               double sigma, uint64_t seed, uint64_t step_base, double* acc_sum,
               void* stream) {
  if (!ctx) return OQ_ERR_ARG;
  if (W < 0 || n_steps < 0 || !(sigma > 0.0) || !valid_prec(precision))
    return set_err(ctx, OQ_ERR_ARG, "bad arguments%s");
  if (W == 0 || n_steps == 0) return OQ_OK;
  if (!X || !state) return set_err(ctx, OQ_ERR_ARG, "null buffer%s");
  if (ctx->md) {
    if (precision != OQ_PREC_FP64)
      return set_err(ctx, OQ_ERR_UNSUPPORTED,
                     "multi-determinant trials are sampled in FP64 only%s");
    cudaStream_t s = (cudaStream_t)stream;
    const OqMdState st = md_state(ctx, state, W);
    OQ_CUDA(ctx, to_soa(ctx, X, st.pos, W, s));
    OqMoveArgs m;
    memset(&m, 0, sizeof(m));
    m.pos = st.pos; m.ainv = st.ainv; m.logdet = st.ldet; m.W = W; m.mode = 1;
    m.n_steps = n_steps; m.step = sigma; m.seed = seed; m.step_base = step_base;
    m.acc_sum = acc_sum; m.flags = ctx->d_flags;
    int rc = md_moves(ctx, m, st.sgn, stream);
    if (rc != OQ_OK) return rc;
    OQ_CUDA(ctx, to_aos(ctx, st.pos, X, W, s));
    return OQ_OK;
  }
  size_t sm;
  const int wpb = pick_wpb(ctx, 0, precision, &sm);
  if (wpb < 0)
    return set_err(ctx, OQ_ERR_UNSUPPORTED, "system too large for the shared-memory move kernel%s");
  cudaStream_t s = (cudaStream_t)stream;
  const OqStatePtrs st = state_ptrs(ctx, state, W, precision);
  OQ_CUDA(ctx, to_soa(ctx, X, st.pos, W, s));
  OqMoveArgs m;
  memset(&m, 0, sizeof(m));
  m.pos = st.pos; m.ainv = st.ainv; m.logdet = st.logdet; m.W = W; m.mode = 1;
  m.n_steps = n_steps; m.step = sigma; m.seed = seed; m.step_base = step_base;
  m.acc_sum = acc_sum; m.flags = ctx->d_flags;
  int rc = launch_moves(ctx, m, wpb, sm, precision, stream);
  if (rc != OQ_OK) return rc;
  OQ_CUDA(ctx, to_aos(ctx, st.pos, X, W, s));
  return OQ_OK;
}

int oqmc_get_flags(oqmc_ctx* ctx, unsigned* flags, int clear, void* stream) {
  if (!ctx || !flags) return OQ_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  unsigned h = 0;
  OQ_CUDA(ctx, cudaMemcpyAsync(&h, ctx->d_flags, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
  OQ_CUDA(ctx, cudaStreamSynchronize(s));
  if (clear) OQ_CUDA(ctx, cudaMemsetAsync(ctx->d_flags, 0, sizeof(unsigned), s));
  *flags = h;
  return OQ_OK;
}

}  // extern "C"
