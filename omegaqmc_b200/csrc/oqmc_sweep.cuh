// Single-electron Metropolis sweeps with Sherman-Morrison inverse updates.
//
// A CTA copies the system tables and its walkers' state (positions, the two
// inverse Slater matrices) into shared memory once, runs all sweeps of a call
// without touching HBM except to reduce the local energy of each measured
// sweep, and writes the state back at the end.  One to 32 threads of a warp
// share a walker (k_sweeps); a walker's state is contiguous, at an odd pitch.
//
// A sweep moves every electron once (Gaussian proposal of width `step`,
// exact Metropolis acceptance |R|^2 exp(2 dJ) with R the determinant ratio
// from the stored inverse) and then evaluates the local energy with the
// analytic Slater/Jastrow VGL, as the reference does after its move
// (OmegaQMC/vmc_gto.py:985-1034, psi/gto.py:2506-2579).  Proposals that
// land within MIN_DIST_THRESHOLD = 1e-4 bohr of a nucleus or another
// electron are rejected (vmc_gto.py:815-839, constants.py:23).
//
// Precision (template T/Real): T is the type of the AO/MO arithmetic and
// Real the storage type of the inverse.  FP64 build: T = Real = double.
// Mixed build: T = Real = float for moves and the MO VGL, with FP64 kept for
// positions, the periodic refresh of the inverses (k_team), the Coulomb terms and all
// energy accumulation.  Exponent groups whose tightest exponent exceeds
// `tight` are evaluated in FP64 for electrons within the group's split
// radius of their nucleus (the large-exponent Laplacian term
// (4a^2 r^2 - 6a) e^{-a r^2} loses FP32 precision there).
#pragma once
#include "oqmc_eval.cuh"

template <typename T> __device__ __forceinline__ T oq_exp(T v);
template <> __device__ __forceinline__ double oq_exp<double>(double v) { return exp(v); }
template <> __device__ __forceinline__ float oq_exp<float>(float v) { return __expf(v); }

// exp(-a r2) of a basis primitive in the generated code, given a and
// al2 = a log2(e) as literals: FP64 exp in the FP64 build; in FP32 the
// power of two 2^(-al2 r2) straight from the hardware approximation
// (ex2.approx, relative error ~2^-22), one multiply per primitive.
template <typename T> __device__ __forceinline__ T oq_exp_neg(T a, T al2, T r2);
template <> __device__ __forceinline__ double oq_exp_neg<double>(double a, double, double r2) {
  return exp(-a * r2);
}
template <> __device__ __forceinline__ float oq_exp_neg<float>(float, float al2, float r2) {
  float p;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p) : "f"(-al2 * r2));
  return p;
}

// exp(-a r2d) for a tight exponent a, the argument formed in FP64 (in FP32
// the rounding of a large argument would dominate the error), given a and
// al2 = a log2(e) as literals.  FP32 form: t = al2 r2d = k + f with k the
// nearest integer, taken by adding 1.5 * 2^52 (t < 2^51, so the sum is an
// integer whose low word is k: no conversion instruction) and f = t - k in
// [-1/2, 1/2] exactly; only 2^-f is evaluated in FP32 (ex2.approx), then
// scaled by 2^-k through the exponent field.  FP32 relative accuracy for
// every argument, without an FP64 exponential or a branch.
template <typename T> __device__ __forceinline__ T oq_exp_tight(double a, double al2, double r2d);
template <> __device__ __forceinline__ double oq_exp_tight<double>(double a, double, double r2d) {
  return exp(-(a * r2d));
}
template <> __device__ __forceinline__ float oq_exp_tight<float>(double, double al2, double r2d) {
  const double shift = 6755399441055744.0;                    // 1.5 * 2^52
  const double t = fmin(al2 * r2d, 125.0);                    // >= 0; 2^-125 is a normal float
  const double y = t + shift;
  const int k = __double2loint(y);                            // round(t), in [0, 125]
  const float f = (float)(t - (y - shift));                  // exact, in [-1/2, 1/2]
  float p;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p) : "f"(-f));
  return p * __int_as_float((127 - k) << 23);                // 2^-k
}

// per-group "tight" split radius squared (FP64 evaluation inside it);
// 0 disables.  Stored after the system struct in global memory.
struct OqSplit {
  double r2[OQ_MAX_GROUP];
};

// MO values at x in compute type T (accumulated in T).
template <int NOCC, typename T, typename TC>
__device__ __forceinline__ void oq_mo_val_t(const OqSystem& S, const OqSplit& SP,
                                            const TC* __restrict__ C, double x,
                                            double y, double z, T mv[NOCC]) {
#pragma unroll
  for (int m = 0; m < NOCC; ++m) mv[m] = (T)0;
  for (int g = 0; g < S.ngroup; ++g) {
    const int ia = S.g_iat[g];
    const double dxd = x - S.nuc[ia][0], dyd = y - S.nuc[ia][1], dzd = z - S.nuc[ia][2];
    const double r2d = dxd * dxd + dyd * dyd + dzd * dzd;
    const T dx = (T)dxd, dy = (T)dyd, dz = (T)dzd, r2 = (T)r2d;
    const int ncol = S.g_ncol[g], np = S.g_n[g], off = S.g_off[g], sh0 = S.g_shell0[g];
    T R[OQ_MAX_COL] = {0, 0, 0, 0};
    for (int p = 0; p < np; ++p) {
      const T e = oq_exp<T>(-(T)S.alpha[off + p] * r2);
#pragma unroll
      for (int k = 0; k < OQ_MAX_COL; ++k)
        if (k < ncol) R[k] += (T)S.norm[S.s_norm[sh0 + k] + p] * e;
    }
    if (S.has_spl) {
#pragma unroll
      for (int k = 0; k < OQ_MAX_COL; ++k)
        if (k < ncol && S.s_spl[sh0 + k] >= 0) {
          double gv, gp, gpp;
          oq_spline_gdd(S, S.s_spl[sh0 + k], r2d, gv, gp, gpp);
          R[k] = (T)gv;
        }
    }
    const int am = S.g_am[g];
#pragma unroll
    for (int k = 0; k < OQ_MAX_COL; ++k) {
      if (k >= ncol) break;
      const int sh = sh0 + k;
      const int ao = S.s_ao[sh];
      if (am == 0) {
        T v = R[k];
        if (S.s_cusp[sh]) v = (T)oq_cusp_val(S, ia, sqrt(r2d), (double)v);
#pragma unroll
        for (int m = 0; m < NOCC; ++m) mv[m] += (T)C[ao * NOCC + m] * v;
      } else if (am == 1) {
        const T v0 = R[k] * dx, v1 = R[k] * dy, v2 = R[k] * dz;
#pragma unroll
        for (int m = 0; m < NOCC; ++m)
          mv[m] += (T)C[ao * NOCC + m] * v0 + (T)C[(ao + 1) * NOCC + m] * v1 +
                   (T)C[(ao + 2) * NOCC + m] * v2;
      } else if (am == 2) {
        T Y[5], dY[5][3];
        oq_harm_d<T>(dx, dy, dz, Y, dY);
#pragma unroll
        for (int c = 0; c < 5; ++c) {
          const T v = R[k] * Y[c];
#pragma unroll
          for (int m = 0; m < NOCC; ++m) mv[m] += (T)C[(ao + c) * NOCC + m] * v;
        }
      } else {
        const int nc = 2 * am + 1;
        for (int c = 0; c < nc; ++c) {
          T Yc, dY[3];
          oq_harm_table<T>(S.harm, am, c, dx, dy, dz, Yc, dY);
          const T v = R[k] * Yc;
#pragma unroll
          for (int m = 0; m < NOCC; ++m) mv[m] += (T)C[(ao + c) * NOCC + m] * v;
        }
      }
    }
  }
}

// MO value/gradient/Laplacian at x in compute type T.  Groups flagged tight
// (SP.r2[g] > r^2) run their radial part in FP64.
template <int NOCC, typename T, typename TC>
__device__ __forceinline__ void oq_mo_vgl_t(const OqSystem& S, const OqSplit& SP,
                                            const TC* __restrict__ C, double x,
                                            double y, double z, T mv[NOCC],
                                            T mg[NOCC][3], T ml[NOCC]) {
#pragma unroll
  for (int m = 0; m < NOCC; ++m) {
    mv[m] = (T)0; mg[m][0] = mg[m][1] = mg[m][2] = (T)0; ml[m] = (T)0;
  }
  for (int g = 0; g < S.ngroup; ++g) {
    const int ia = S.g_iat[g];
    const double dxd = x - S.nuc[ia][0], dyd = y - S.nuc[ia][1], dzd = z - S.nuc[ia][2];
    const double r2d = dxd * dxd + dyd * dyd + dzd * dzd;
    const T dx = (T)dxd, dy = (T)dyd, dz = (T)dzd;
    const int ncol = S.g_ncol[g], np = S.g_n[g], off = S.g_off[g], sh0 = S.g_shell0[g];
    T R[OQ_MAX_COL], Rp[OQ_MAX_COL], Rl[OQ_MAX_COL];
    const bool fp64_radial = (sizeof(T) == 8) || (r2d < SP.r2[g]) || S.s_cusp[sh0];
    if (fp64_radial) {
      double Rd[OQ_MAX_COL] = {0, 0, 0, 0}, Rpd[OQ_MAX_COL] = {0, 0, 0, 0},
             Rld[OQ_MAX_COL] = {0, 0, 0, 0};
      for (int p = 0; p < np; ++p) {
        const double a = S.alpha[off + p];
        const double e = exp(-a * r2d);
        const double fp = -2.0 * a * e;
        const double fl = (4.0 * a * a * r2d - 6.0 * a) * e;
#pragma unroll
        for (int k = 0; k < OQ_MAX_COL; ++k)
          if (k < ncol) {
            const double n = S.norm[S.s_norm[sh0 + k] + p];
            Rd[k] += n * e; Rpd[k] += n * fp; Rld[k] += n * fl;
          }
      }
      if (S.g_am[g] == 0) {
#pragma unroll
        for (int k = 0; k < OQ_MAX_COL; ++k)
          if (k < ncol && S.s_cusp[sh0 + k]) oq_cusp_vgl(S, ia, sqrt(r2d), Rd[k], Rpd[k], Rld[k]);
      }
#pragma unroll
      for (int k = 0; k < OQ_MAX_COL; ++k) { R[k] = (T)Rd[k]; Rp[k] = (T)Rpd[k]; Rl[k] = (T)Rld[k]; }
    } else {
      const T r2 = (T)r2d;
#pragma unroll
      for (int k = 0; k < OQ_MAX_COL; ++k) { R[k] = Rp[k] = Rl[k] = (T)0; }
      for (int p = 0; p < np; ++p) {
        const T a = (T)S.alpha[off + p];
        const T e = oq_exp<T>(-a * r2);
        const T fp = (T)-2 * a * e;
        const T fl = ((T)4 * a * a * r2 - (T)6 * a) * e;
#pragma unroll
        for (int k = 0; k < OQ_MAX_COL; ++k)
          if (k < ncol) {
            const T n = (T)S.norm[S.s_norm[sh0 + k] + p];
            R[k] += n * e; Rp[k] += n * fp; Rl[k] += n * fl;
          }
      }
    }
    if (S.has_spl) {
#pragma unroll
      for (int k = 0; k < OQ_MAX_COL; ++k)
        if (k < ncol && S.s_spl[sh0 + k] >= 0) {
          double gv, gp, gpp;
          oq_spline_gdd(S, S.s_spl[sh0 + k], r2d, gv, gp, gpp);
          R[k] = (T)gv;
          Rp[k] = (T)(2.0 * gp);
          Rl[k] = (T)(6.0 * gp + 4.0 * r2d * gpp);
        }
    }
    const int am = S.g_am[g];
#pragma unroll
    for (int k = 0; k < OQ_MAX_COL; ++k) {
      if (k >= ncol) break;
      const int ao = S.s_ao[sh0 + k];
      if (am == 0) {
        const T v = R[k], l = Rl[k];
        const T gx = Rp[k] * dx, gy = Rp[k] * dy, gz = Rp[k] * dz;
#pragma unroll
        for (int m = 0; m < NOCC; ++m) {
          const T c = (T)C[ao * NOCC + m];
          mv[m] += c * v; mg[m][0] += c * gx; mg[m][1] += c * gy; mg[m][2] += c * gz;
          ml[m] += c * l;
        }
      } else {
        const int nc = 2 * am + 1;
        T Yd[5], dYd[5][3];
        if (am == 2) oq_harm_d<T>(dx, dy, dz, Yd, dYd);
        const T lfac = Rl[k] + (T)(2 * am) * Rp[k];
        for (int c = 0; c < nc; ++c) {
          T Y, dY[3];
          if (am == 1) {
            Y = (c == 0) ? dx : (c == 1) ? dy : dz;
            dY[0] = (T)(c == 0); dY[1] = (T)(c == 1); dY[2] = (T)(c == 2);
          } else if (am == 2) {
            Y = Yd[c]; dY[0] = dYd[c][0]; dY[1] = dYd[c][1]; dY[2] = dYd[c][2];
          } else {
            oq_harm_table<T>(S.harm, am, c, dx, dy, dz, Y, dY);
          }
          const T v = R[k] * Y;
          const T gx = Rp[k] * dx * Y + R[k] * dY[0];
          const T gy = Rp[k] * dy * Y + R[k] * dY[1];
          const T gz = Rp[k] * dz * Y + R[k] * dY[2];
          const T l = lfac * Y;
#pragma unroll
          for (int m = 0; m < NOCC; ++m) {
            const T cc = (T)C[(ao + c) * NOCC + m];
            mv[m] += cc * v; mg[m][0] += cc * gx; mg[m][1] += cc * gy;
            mg[m][2] += cc * gz; ml[m] += cc * l;
          }
        }
      }
    }
  }
}

// Basis policy: how a kernel evaluates the occupied MOs at one position.
// OqBasisTable reads the system tables (any molecule); a per-system policy
// generated at run time (oqmc_specialize) has the same two members with the
// exponents and coefficients compiled in.
// Generated policies also carry the molecule's charges and Padé constants
// (see OqJasOf); natm = 0 says that this one does not.
template <int NOCC>
struct OqBasisTable {
  static constexpr int natm = 0;
  template <typename T, typename TC>
  __device__ static __forceinline__ void mo_val(const OqSystem& S, const OqSplit& SP,
                                                const TC* __restrict__ C, double x, double y,
                                                double z, T* mv) {
    oq_mo_val_t<NOCC, T, TC>(S, SP, C, x, y, z, mv);
  }
  template <typename T, typename TC>
  __device__ static __forceinline__ void mo_vgl(const OqSystem& S, const OqSplit& SP,
                                                const TC* __restrict__ C, double x, double y,
                                                double z, T* mv, T (*mg)[3], T* ml) {
    oq_mo_vgl_t<NOCC, T, TC>(S, SP, C, x, y, z, mv, mg, ml);
  }
  // gradient and Laplacian of sum_m ac[m] phi_m
  template <typename T, typename TC>
  __device__ static __forceinline__ void mo_vgl_contract(const OqSystem& S, const OqSplit& SP,
                                                         const TC* __restrict__ C, double x,
                                                         double y, double z, const T* ac, T& gx,
                                                         T& gy, T& gz, T& lp) {
    T mv[NOCC], mg[NOCC][3], ml[NOCC];
    oq_mo_vgl_t<NOCC, T, TC>(S, SP, C, x, y, z, mv, mg, ml);
    gx = gy = gz = lp = (T)0;
#pragma unroll
    for (int m = 0; m < NOCC; ++m) {
      gx += ac[m] * mg[m][0]; gy += ac[m] * mg[m][1]; gz += ac[m] * mg[m][2];
      lp += ac[m] * ml[m];
    }
  }
};

// Nuclei and Jastrow constants of the molecule a generated policy B belongs to,
// in the form the move and local-energy code reads them.  What the generator
// knows is fixed at compile time: the loops over nuclei unroll, absent Padé
// terms leave no test behind, and the constants become literals of the working
// precision (an FP64 constant converted where it is used costs a slot of the
// conversion unit per pair).  The coordinates stay in memory, where an FP64
// operation can take them as an operand.
template <class B>
struct OqJasOf {
  static constexpr int natm = B::natm, has_j1 = B::has_j1, has_j2 = B::has_j2;
  struct Zs { __device__ constexpr double operator[](int i) const { return B::Z(i); } } Z;
  struct A1 { __device__ constexpr double operator[](int i) const { return B::j1a(i); } } j1a;
  struct B1 { __device__ constexpr double operator[](int i) const { return B::j1b(i); } } j1b;
  struct J2 { __device__ constexpr double operator[](int i) const { return B::j2(i); } } j2;
  const double (&nuc)[OQ_MAX_NUC][3];
  double e_nn;
  __device__ OqJasOf(const double (&n)[OQ_MAX_NUC][3], double e) : nuc(n), e_nn(e) {}
};
// The same for a table-driven policy: the system tables themselves.
template <class B, bool GENERATED = (B::natm > 0)>
struct OqJasSel {
  typedef OqJasOf<B> type;
  __device__ static type of(const OqSystem& S) { return type(S.nuc, S.e_nn); }
};
template <class B>
struct OqJasSel<B, false> {
  typedef const OqSystem& type;
  __device__ static type of(const OqSystem& S) { return S; }
};

// ---------------------------------------------------------------------------
// Sampler state in global memory, walker-minor so consecutive threads
// (walkers) touch consecutive words:
//   pos    [3*NE][W] double        positions, pos[(3e+c)*W + w]
//   ainv   [2*N*N][W] Real         ainv[((s*N + m)*N + j)*W + w] = (S_s^-1)[m][j]
//   logdet [W] double              log|det up| + log|det down|
// ---------------------------------------------------------------------------

// number of doubles reduced per measured sweep
#define OQ_NSUM 8   // ee, en, ke, eloc, eloc^2, accepted moves, finite walkers, pad

struct OqMoveArgs {
  double* pos;            // state positions (SoA)
  void* ainv;             // state inverses (Real, SoA)
  double* logdet;
  int W;
  int n_steps;            // sweeps (mode 0) or basin relocations (mode 1)
  int mode;               // 0: Gaussian single-electron sweeps; 1: basin relocation
  int proposal;           // mode 0: 0 = fixed width, 1 = nucleus-scaled width
  double step;            // Gaussian width (mode 0) or blob width sigma (mode 1)
  double scale_r0;        // nucleus-scaled width: sigma = step * clamp(r_near/r0, fmin, 1)
  double scale_fmin;
  uint64_t seed;
  uint64_t step_base;     // RNG counter of the first step
  double* acc_sum;        // += accepted moves (may be null)
  unsigned* flags;
  const double* step_dev; // when set, the Gaussian width is read here (device-side step
                          // adaptation, oqmc_equilibrate); else `step`
};

// The nucleus-scaled proposal's constants in FP32 (set once per launch or tile).
struct OqScaledF {
  float step, inv_r0, fmin;
};
__device__ __forceinline__ OqScaledF oq_scaled_f(double step, double r0, double fmn) {
  return {(float)step, 1.0f / (float)r0, (float)fmn};
}

// Proposal width at x for the nucleus-scaled Gaussian move,
// sigma(x) = step * clamp(r_near(x) / r0, fmin, 1): the nearest nucleus's
// squared distance in FP64, then sqrt.approx, the clamp and the product in
// FP32.  The width only has to be the same function of position on both
// sides of the ratio; the FP64 and the mixed samplers use this same
// function, so for the same random numbers they propose the same positions.
template <class SJ>
__device__ __forceinline__ float oq_scaled_width_f(const SJ& S, double x, double y, double z,
                                                   const OqScaledF& p) {
  double r2 = 1e300;
  for (int I = 0; I < S.natm; ++I) {
    const double dx = x - S.nuc[I][0], dy = y - S.nuc[I][1], dz = z - S.nuc[I][2];
    r2 = fmin(r2, dx * dx + dy * dy + dz * dz);
  }
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"((float)r2));
  return p.step * fminf(1.0f, fmaxf(p.fmin, r * p.inv_r0));
}

template <class SJ>
__device__ __forceinline__ double oq_scaled_width(const SJ& S, double x, double y,
                                                  double z, double step, double r0,
                                                  double fmn) {
  return (double)oq_scaled_width_f(S, x, y, z, oq_scaled_f(step, r0, fmn));
}

// Nucleus-scaled Gaussian proposal from (ox, oy, oz) with the FP32 standard
// normals nf: the new position (FP64) and the proposal-density ratio
// q(old | new) / q(new | old) = (so / sn)^3 exp(d^2 (1 / so^2 - 1 / sn^2) / 2),
// with d = so n: (so / sn)^3 exp(|n|^2 (1 - (so / sn)^2) / 2), returned as a
// factor mul and an exponent lx (no logarithm on the move path), in the
// working precision T (FP32 in the mixed build: its rounding, ~1e-7
// relative, is far below any statistical resolution).
template <typename T, class SJ>
__device__ __forceinline__ void oq_scaled_propose_t(const SJ& S, double ox, double oy, double oz,
                                                    const float nf[3], const OqScaledF& pf,
                                                    double& nx, double& ny, double& nz, T& mul,
                                                    T& lx) {
  const float so = oq_scaled_width_f(S, ox, oy, oz, pf);
  const double sod = (double)so;
  nx = ox + sod * (double)nf[0];
  ny = oy + sod * (double)nf[1];
  nz = oz + sod * (double)nf[2];
  const float sn = oq_scaled_width_f(S, nx, ny, nz, pf);
  if (sizeof(T) == 8) {
    const double q = sod / (double)sn;
    const double n2 = (double)nf[0] * (double)nf[0] + (double)nf[1] * (double)nf[1] +
                      (double)nf[2] * (double)nf[2];
    mul = (T)(q * q * q);
    lx = (T)(0.5 * n2 * (1.0 - q * q));
  } else {
    const float q = so * oq_rcp(sn);
    mul = (T)(q * q * q);
    lx = (T)(0.5f * (nf[0] * nf[0] + nf[1] * nf[1] + nf[2] * nf[2]) * (1.0f - q * q));
  }
}

// The Metropolis-Hastings test u < |R|^2 exp(2 dJ + log_extra) mul_extra in
// the working precision T (FP32 in the mixed build: the accurate expf, whose
// ~1e-7 relative error moves acceptance probabilities far below any
// statistical resolution), without logarithms.
template <typename T>
__device__ __forceinline__ bool oq_accept(T R, T dJ, T log_extra, T mul_extra, T u, bool valid) {
  const T ex = (sizeof(T) == 8) ? (T)exp((double)((T)2 * dJ + log_extra))
                                : (T)expf((float)((T)2 * dJ + log_extra));
  const T ratio = R * R * mul_extra * ex;
  return valid && (R != (T)0) && isfinite(R) && isfinite(dJ) && isfinite(log_extra) &&
         (u < ratio);
}

// Change of the Jastrow factor (arithmetic in T) when electron e moves from
// (ox, oy, oz) to (nx, ny, nz), and the MIN_DIST_THRESHOLD test of the new
// position (FP64; OmegaQMC/constants.py:23): valid is cleared when an
// electron-electron or electron-nucleus distance falls below 1e-4.  The
// other electrons' coordinate c is pos[(3 j + c) * ps].
template <int NE, typename T, class SJ>
__device__ __forceinline__ T oq_jastrow_delta(const SJ& J, const OqSystem& S, const double* pos,
                                              int ps, int e, double ox, double oy, double oz,
                                              double nx, double ny, double nz, bool& valid) {
  const double thr2 = 1e-4 * 1e-4;
  T dJ = (T)0;
  valid = true;
  for (int j = 0; j < NE; ++j) {
    if (j == e) continue;
    const double xj = pos[(3 * j) * ps], yj = pos[(3 * j + 1) * ps], zj = pos[(3 * j + 2) * ps];
    const double ax = nx - xj, ay = ny - yj, az = nz - zj;
    const double rn2 = ax * ax + ay * ay + az * az;
    valid = valid && (rn2 >= thr2);
    if (J.has_j2) {
      const double bx = ox - xj, by = oy - yj, bz = oz - zj;
      const T rn2t = (T)rn2, ro2t = (T)(bx * bx + by * by + bz * bz);
      const int o = ((e & 1) == (j & 1)) ? 0 : 2;
      const T pa = (T)J.j2[o], pb = (T)J.j2[o + 1];
      dJ += oq_pade_diff(pa, pb, rn2t * oq_rsqrt(rn2t), ro2t * oq_rsqrt(ro2t));
    }
    if (OQ_HAS_BS2(S)) {
      const double bx = ox - xj, by = oy - yj, bz = oz - zj;
      const T rn2t = (T)rn2, ro2t = (T)(bx * bx + by * by + bz * bz);
      const bool like = (e & 1) == (j & 1);
      const double* c = like ? S.bs2_like : S.bs2_unlike;
      const int n = like ? S.bs2_n_like : S.bs2_n_unlike;
      const T dinv = (T)(like ? S.bs2_dinv_like : S.bs2_dinv_unlike), rc = (T)S.bs2_rcut;
      dJ += oq_bs_val<T>(c, n, dinv, rc, rn2t * oq_rsqrt(rn2t)) -
            oq_bs_val<T>(c, n, dinv, rc, ro2t * oq_rsqrt(ro2t));
    }
  }
  for (int I = 0; I < J.natm; ++I) {
    const double ax = nx - J.nuc[I][0], ay = ny - J.nuc[I][1], az = nz - J.nuc[I][2];
    const double rn2 = ax * ax + ay * ay + az * az;
    valid = valid && (rn2 >= thr2);
    if (J.has_j1) {
      const double bx = ox - J.nuc[I][0], by = oy - J.nuc[I][1], bz = oz - J.nuc[I][2];
      const T rn2t = (T)rn2, ro2t = (T)(bx * bx + by * by + bz * bz);
      const T pa = (T)J.j1a[I], pb = (T)J.j1b[I];
      dJ += oq_pade_diff(pa, pb, rn2t * oq_rsqrt(rn2t), ro2t * oq_rsqrt(ro2t));
    }
    if (OQ_HAS_BS1(S) && S.bs1_type[I] >= 0) {
      const int ty = S.bs1_type[I];
      const double bx = ox - J.nuc[I][0], by = oy - J.nuc[I][1], bz = oz - J.nuc[I][2];
      const T rn2t = (T)rn2, ro2t = (T)(bx * bx + by * by + bz * bz);
      const T dinv = (T)S.bs1_dinv[ty], rc = (T)S.bs1_rcut[ty];
      dJ += oq_bs_val<T>(S.bs1_c[ty], S.bs1_n[ty], dinv, rc, rn2t * oq_rsqrt(rn2t)) -
            oq_bs_val<T>(S.bs1_c[ty], S.bs1_n[ty], dinv, rc, ro2t * oq_rsqrt(ro2t));
    }
  }
  if (OQ_HAS_J3(S))
    dJ -= oq_j3_electron<T>(S, pos, (size_t)ps, NE, e, 0, nx, ny, nz) -
          oq_j3_electron<T>(S, pos, (size_t)ps, NE, e, 0, ox, oy, oz);
  return dJ;
}

// One single-electron Metropolis move of electron e to (nx, ny, nz) against
// one walker's state: its positions pos[(3 j + c) ps] and its inverse
// matrices A[k as] (either in shared or in global memory); the
// proposal-density ratio q(old)/q(new) is
// mul_extra * exp(log_extra) (1 for symmetric proposals).  The move is
// accepted when u < |R|^2 exp(2 dJ) q(old)/q(new), the Metropolis-Hastings
// test of metropolis_move_1w (OmegaQMC/vmc_gto.py:841-905) without
// logarithms.  Returns acceptance.
// J supplies the nuclei and Jastrow constants (natm, nuc, has_j1, j1a, j1b,
// has_j2, j2): the system struct itself or a compact copy of those fields;
// S is handed to the basis policy.
template <int NOCC, typename T, typename Real, class B, class SJ>
__device__ __forceinline__ bool oq_try_move_s(const SJ& J, const OqSystem& S, const OqSplit& SP,
                                              const Real* __restrict__ C, double* pos, int ps,
                                              Real* A, int as, int e, double nx, double ny,
                                              double nz, T log_extra, T mul_extra, T u,
                                              double& logdet) {
  constexpr int NE = 2 * NOCC;
  constexpr int NN = NOCC * NOCC;
  const int s = e & 1, i = e >> 1;
  const double ox = pos[(3 * e) * ps], oy = pos[(3 * e + 1) * ps], oz = pos[(3 * e + 2) * ps];
  // Jastrow change (arithmetic in T) and the MIN_DIST_THRESHOLD test (FP64)
  bool valid;
  const T dJ = oq_jastrow_delta<NE, T>(J, S, pos, ps, e, ox, oy, oz, nx, ny, nz, valid);
  // new MO row and the ratio R = sum_m v_m A[m][i] (column i of the inverse)
  T v[NOCC];
  B::template mo_val<T, Real>(S, SP, C, nx, ny, nz, v);
  Real* As = A + (size_t)s * NN * as;
  T R = (T)0;
#pragma unroll
  for (int m = 0; m < NOCC; ++m) R += v[m] * (T)As[(m * NOCC + i) * as];
  const bool acc = oq_accept<T>(R, dJ, log_extra, mul_extra, u, valid);
  if (acc) {
    // Sherman-Morrison with the ratio vector w_j = sum_m v_m A[m][j]:
    // A[k][j] -= A[k][i] (w_j - delta_ij) / R, column i taken before the update
    const T rinv = oq_rcp(R);
    T coli[NOCC];
#pragma unroll
    for (int k = 0; k < NOCC; ++k) coli[k] = (T)As[(k * NOCC + i) * as];
#pragma unroll
    for (int j = 0; j < NOCC; ++j) {
      T w = (T)0;
#pragma unroll
      for (int m = 0; m < NOCC; ++m) w += v[m] * (T)As[(m * NOCC + j) * as];
      const T f = (w - (j == i ? (T)1 : (T)0)) * rinv;
#pragma unroll
      for (int k = 0; k < NOCC; ++k) {
        Real& ref = As[(k * NOCC + j) * as];
        ref = (Real)((T)ref - coli[k] * f);
      }
    }
    pos[(3 * e) * ps] = nx;
    pos[(3 * e + 1) * ps] = ny;
    pos[(3 * e + 2) * ps] = nz;
    logdet += log(fabs((double)R));
  }
  return acc;
}

// The same move with positions and inverses in one walker-minor layout of
// stride WPB (this walker at index tid).
template <int NOCC, typename T, typename Real, class B, class SJ>
__device__ __forceinline__ bool oq_try_move(const SJ& J, const OqSystem& S, const OqSplit& SP,
                                            const Real* __restrict__ C, double* pos,
                                            Real* Ai, int WPB, int tid, int e,
                                            double nx, double ny, double nz,
                                            T log_extra, T mul_extra, T u,
                                            double& logdet) {
  return oq_try_move_s<NOCC, T, Real, B>(J, S, SP, C, pos + tid, WPB, Ai + tid, WPB, e, nx, ny,
                                         nz, log_extra, mul_extra, u, logdet);
}

// Basin relocation proposal (basin_move_1w, OmegaQMC/vmc_gto.py:925-957):
// one random electron to N(R_J, sigma^2) around a random nucleus J.  Returns
// the electron; sets its proposed position, the log proposal ratio
// log q(old) - log q(new) with q(x) = sum_J exp(-|x - R_J|^2 / 2 sigma^2)
// (computed as a log-sum-exp) and the acceptance uniform u.
template <int NE>
__device__ __forceinline__ int oq_basin_propose(const OqSystem& S, const double* pos, int ps,
                                                uint64_t seed, uint32_t w, uint32_t gstep,
                                                double sg, double& nx, double& ny, double& nz,
                                                double& log_qratio, double& u) {
  double n3[3];
  oq_move_randoms(seed, w, gstep, 0xB0000000u, n3, u);
  const OqU4 c = {w, gstep, 0xB0000001u, 2u};
  const OqU4 r = oq_philox(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  const int e = (int)(((uint64_t)r.x * NE) >> 32);
  const int J = (int)(((uint64_t)r.y * S.natm) >> 32);
  const double inv2s2 = 1.0 / (2.0 * sg * sg);
  nx = S.nuc[J][0] + sg * n3[0];
  ny = S.nuc[J][1] + sg * n3[1];
  nz = S.nuc[J][2] + sg * n3[2];
  const double ox = pos[(3 * e) * ps], oy = pos[(3 * e + 1) * ps], oz = pos[(3 * e + 2) * ps];
  double mo = -INFINITY, mn = -INFINITY;
  for (int I = 0; I < S.natm; ++I) {
    const double dox = ox - S.nuc[I][0], doy = oy - S.nuc[I][1], doz = oz - S.nuc[I][2];
    const double dnx = nx - S.nuc[I][0], dny = ny - S.nuc[I][1], dnz = nz - S.nuc[I][2];
    mo = fmax(mo, -(dox * dox + doy * doy + doz * doz) * inv2s2);
    mn = fmax(mn, -(dnx * dnx + dny * dny + dnz * dnz) * inv2s2);
  }
  double so = 0.0, sn = 0.0;
  for (int I = 0; I < S.natm; ++I) {
    const double dox = ox - S.nuc[I][0], doy = oy - S.nuc[I][1], doz = oz - S.nuc[I][2];
    const double dnx = nx - S.nuc[I][0], dny = ny - S.nuc[I][1], dnz = nz - S.nuc[I][2];
    so += exp(-(dox * dox + doy * doy + doz * doz) * inv2s2 - mo);
    sn += exp(-(dnx * dnx + dny * dny + dnz * dnz) * inv2s2 - mn);
  }
  log_qratio = (mo + log(so)) - (mn + log(sn));
  return e;
}

// Metropolis moves alone, one thread per walker, state resident in shared
// memory for the whole launch: basin relocations, and the sweeps that
// moves_by_thread (oqmc.cu) keeps out of k_sweeps.  PROP (compile time) selects
// the proposal: 0 fixed-width Gaussian, 1 nucleus-scaled Gaussian, 2 basin
// relocation.  mode 0: n_steps sweeps over all electrons with Gaussian
// proposals (metropolis_move_1w, OmegaQMC/vmc_gto.py:841-905, as
// single-electron moves).  mode 1: n_steps basin relocations: one random
// electron proposed at N(R_J, sigma^2) around a random nucleus J, accepted
// with the exact proposal ratio q(old)/q(new), q(x) = sum_J
// exp(-|x-R_J|^2 / 2 sigma^2) (basin_move_1w, vmc_gto.py:925-957).
template <int NOCC, typename T, typename Real, int PROP, class B = OqBasisTable<NOCC>>
__global__ void __launch_bounds__(128, 4)
k_moves(const OqSystem* __restrict__ gsys, const OqSplit* __restrict__ gsplit,
        const void* __restrict__ gC, OqMoveArgs a) {
  constexpr int NE = 2 * NOCC;
  constexpr int NN = NOCC * NOCC;
  extern __shared__ __align__(16) unsigned char smem[];
  OqSystem& S = *reinterpret_cast<OqSystem*>(smem);
  OqSplit& SP = *reinterpret_cast<OqSplit*>(smem + sizeof(OqSystem));
  unsigned char* p = smem + sizeof(OqSystem) + sizeof(OqSplit);
  Real* C = reinterpret_cast<Real*>(p);
  const int nbf = gsys->nbf;
  p += ((size_t)nbf * NOCC * sizeof(Real) + 15) & ~(size_t)15;
  const int WPB = blockDim.x;
  double* pos = reinterpret_cast<double*>(p);          // [3*NE][WPB]
  p += (size_t)3 * NE * WPB * sizeof(double);
  Real* Ai = reinterpret_cast<Real*>(p);                // [2*NN][WPB]

  oq_load_system(&S, gsys);
  {
    const double* src = reinterpret_cast<const double*>(gsplit);
    double* dst = reinterpret_cast<double*>(&SP);
    for (int i = threadIdx.x; i < OQ_MAX_GROUP; i += blockDim.x) dst[i] = src[i];
    const Real* gc = reinterpret_cast<const Real*>(gC);
    for (int i = threadIdx.x; i < nbf * NOCC; i += blockDim.x) C[i] = gc[i];
  }
  const int tid = threadIdx.x;
  const int w = blockIdx.x * WPB + tid;
  const bool live = w < a.W;
  const int W = a.W;
  Real* gA = reinterpret_cast<Real*>(a.ainv);
  if (live) {
    for (int k = 0; k < 3 * NE; ++k) pos[k * WPB + tid] = a.pos[(size_t)k * W + w];
    for (int k = 0; k < 2 * NN; ++k) Ai[k * WPB + tid] = gA[(size_t)k * W + w];
  }
  __syncthreads();
  const double step = a.step_dev ? *a.step_dev : a.step;
  const OqScaledF pf = oq_scaled_f(step, a.scale_r0, a.scale_fmin);
  double logdet = live ? a.logdet[w] : 0.0;
  int nacc = 0;
  for (int t = 0; t < (live ? a.n_steps : 0); ++t) {
    const uint32_t gstep = (uint32_t)(a.step_base + t);
    if (PROP == 0) {
      for (int e = 0; e < NE; ++e) {
        float nf[3];
        uint32_t ub;
        oq_move_normals(a.seed, (uint32_t)w, gstep, (uint32_t)e, nf, ub);
        const double nx = pos[(3 * e) * WPB + tid] + step * (double)nf[0];
        const double ny = pos[(3 * e + 1) * WPB + tid] + step * (double)nf[1];
        const double nz = pos[(3 * e + 2) * WPB + tid] + step * (double)nf[2];
        nacc += oq_try_move<NOCC, T, Real, B>(S, S, SP, C, pos, Ai, WPB, tid, e, nx, ny, nz,
                                           (T)0, (T)1, oq_uniform<T>(ub), logdet);
      }
    } else if (PROP == 1) {
      // nucleus-scaled Gaussian: sigma(x) = step * clamp(r_near(x)/r0, fmin, 1);
      // exact MH with log q(x|x') - log q(x'|x) for the asymmetric proposal
      for (int e = 0; e < NE; ++e) {
        float nf[3];
        uint32_t ub;
        oq_move_normals(a.seed, (uint32_t)w, gstep, (uint32_t)e, nf, ub);
        const double ox = pos[(3 * e) * WPB + tid], oy = pos[(3 * e + 1) * WPB + tid],
                     oz = pos[(3 * e + 2) * WPB + tid];
        double nx, ny, nz;
        T mul, lx;
        oq_scaled_propose_t<T>(S, ox, oy, oz, nf, pf, nx, ny, nz, mul, lx);
        nacc += oq_try_move<NOCC, T, Real, B>(S, S, SP, C, pos, Ai, WPB, tid, e, nx, ny, nz, lx,
                                           mul, oq_uniform<T>(ub), logdet);
      }
    } else {
      double u, nx, ny, nz, log_qratio;
      const int e = oq_basin_propose<NE>(S, pos + tid, WPB, a.seed, (uint32_t)w, gstep, step,
                                         nx, ny, nz, log_qratio, u);
      nacc += oq_try_move<NOCC, T, Real, B>(S, S, SP, C, pos, Ai, WPB, tid, e, nx, ny, nz,
                                         (T)log_qratio, (T)1, (T)u, logdet);
    }
  }
  if (live) {
    for (int k = 0; k < 3 * NE; ++k) a.pos[(size_t)k * W + w] = pos[k * WPB + tid];
    for (int k = 0; k < 2 * NN; ++k) gA[(size_t)k * W + w] = Ai[k * WPB + tid];
    a.logdet[w] = logdet;
  }
  if (a.acc_sum) {
    double v = (double)nacc;   // every lane of the warp reaches here
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) atomicAdd(a.acc_sum, v);
  }
}

// Jastrow gradient and Laplacian of electron e at (xe, ye, ze) (Padé,
// B-spline and three-body terms; gto.py:1575-1649, 1657-1931, 2042-2196),
// accumulated into (jx, jy, jz, jl), and its Coulomb terms (e-e counted once,
// for partners j > e; e-n; gto.py:2406-2451) into ee, en.  The other
// electrons' coordinate c is pos[(3 j + c) * ps].
template <int NE, typename T, class SJ>
__device__ __forceinline__ void oq_jastrow_vgl_coulomb(const SJ& J, const OqSystem& S,
                                                       const double* pos, size_t ps, int e,
                                                       double xe, double ye, double ze, T& jx,
                                                       T& jy, T& jz, T& jl, double& ee,
                                                       double& en, bool j3 = true) {
  // The gradient sums run in FP64 on the FP64 displacements: in the mixed
  // build that converts one value per pair (u'(r)/r) to FP64 instead of
  // three displacement components to FP32.  The working-precision Coulomb
  // terms of one electron are summed in T and converted once.  In the FP64
  // build both forms are the same arithmetic in the same order.
  double gx = 0.0, gy = 0.0, gz = 0.0;
  T eet = (T)0, ent = (T)0;
  for (int j = 0; j < NE; ++j) {
    if (j == e) continue;
    const double dx = xe - pos[(size_t)(3 * j) * ps], dy = ye - pos[(size_t)(3 * j + 1) * ps],
                 dz = ze - pos[(size_t)(3 * j + 2) * ps];
    const double r2 = dx * dx + dy * dy + dz * dz;
    const T r2t = (T)r2, rinv = oq_rsqrt(r2t);
    // Coulomb: FP64 with the reference's eps in FP64 kernels; the working-
    // precision 1/r otherwise (eps is below FP32 resolution beyond the
    // 1e-4 bohr minimum distance)
    if (j > e) {
      if (sizeof(T) == 8)
        ee += rsqrt(r2 + OQ_EPS);
      else
        eet += rinv;
    }
    if (J.has_j2) {
      const int o = ((e & 1) == (j & 1)) ? 0 : 2;
      T upr, l;
      oq_pade_vgl_q((T)J.j2[o], (T)J.j2[o + 1], r2t * rinv, rinv, upr, l);
      const double u = (double)upr;
      gx += u * dx; gy += u * dy; gz += u * dz; jl += l;
    }
    if (OQ_HAS_BS2(S)) {
      const bool like = (e & 1) == (j & 1);
      T upr, l;
      oq_bs_vgl<T>(like ? S.bs2_like : S.bs2_unlike, like ? S.bs2_n_like : S.bs2_n_unlike,
                   (T)(like ? S.bs2_dinv_like : S.bs2_dinv_unlike), (T)S.bs2_rcut, r2t * rinv,
                   rinv, upr, l);
      const double u = (double)upr;
      gx += u * dx; gy += u * dy; gz += u * dz; jl += l;
    }
  }
  for (int I = 0; I < J.natm; ++I) {
    const double dx = xe - J.nuc[I][0], dy = ye - J.nuc[I][1], dz = ze - J.nuc[I][2];
    const double r2 = dx * dx + dy * dy + dz * dz;
    const T r2t = (T)r2, rinv = oq_rsqrt(r2t);
    if (sizeof(T) == 8)
      en -= J.Z[I] * rsqrt(r2 + OQ_EPS);
    else
      ent -= (T)J.Z[I] * rinv;
    if (J.has_j1) {
      T upr, l;
      oq_pade_vgl_q((T)J.j1a[I], (T)J.j1b[I], r2t * rinv, rinv, upr, l);
      const double u = (double)upr;
      gx += u * dx; gy += u * dy; gz += u * dz; jl += l;
    }
    if (OQ_HAS_BS1(S) && S.bs1_type[I] >= 0) {
      const int ty = S.bs1_type[I];
      T upr, l;
      oq_bs_vgl<T>(S.bs1_c[ty], S.bs1_n[ty], (T)S.bs1_dinv[ty], (T)S.bs1_rcut[ty], r2t * rinv,
                   rinv, upr, l);
      const double u = (double)upr;
      gx += u * dx; gy += u * dy; gz += u * dz; jl += l;
    }
  }
  if (sizeof(T) != 8) {
    ee += (double)eet;
    en += (double)ent;
  }
  jx += (T)gx; jy += (T)gy; jz += (T)gz;
  if (j3 && OQ_HAS_J3(S)) oq_j3_vgl_electron<T>(S, pos, ps, NE, e, xe, ye, ze, jx, jy, jz, jl);
}

// Local-energy contributions of electron e of one walker: its Coulomb terms
// (e-e counted once, for partners j > e; gto.py:2406-2451), the Laplacian
// term lap_e = sum_m A[m][i] L[i][m] - |Gamma_e|^2 + lap J_e and the squared
// total gradient |Gamma_e + grad J_e|^2 (_slater_det_assemble, gto.py:728-778;
// Padé VGL, gto.py:1575-1649).  pos points at the walker's x of electron 0
// with stride ps between coordinates; A at its inverse entry (0,0,0) with
// stride as between entries.  The four outputs are accumulated (+=).
// The _out form also returns electron e's gradient of log|psi| (Gx, Gy, Gz)
// and its Laplacian of log|psi| (lap_e).
template <int NOCC, typename T, typename Real, class B, class SJ>
__device__ __forceinline__ void oq_eloc_electron_out(const SJ& J, const OqSystem& S,
                                                     const OqSplit& SP,
                                                     const Real* __restrict__ C,
                                                     const double* pos, size_t ps,
                                                     const Real* A, size_t as, int e,
                                                     double& ee, double& en, double& lp_tot,
                                                     double& g2, double& gxo, double& gyo,
                                                     double& gzo, double& lape) {
  constexpr int NE = 2 * NOCC;
  const int s = e & 1, i = e >> 1;
  const double xe = pos[(size_t)(3 * e) * ps], ye = pos[(size_t)(3 * e + 1) * ps],
               ze = pos[(size_t)(3 * e + 2) * ps];
  // Gamma = sum_m A[m][i] grad phi_m, sum_m A[m][i] lap phi_m: the MO
  // coefficients contracted with column i of the inverse first
  T ac[NOCC];
#pragma unroll
  for (int m = 0; m < NOCC; ++m) ac[m] = (T)A[(size_t)((s * NOCC + m) * NOCC + i) * as];
  T gx, gy, gz, lp;
  B::template mo_vgl_contract<T, Real>(S, SP, C, xe, ye, ze, ac, gx, gy, gz, lp);
  T jx = (T)0, jy = (T)0, jz = (T)0, jl = (T)0;
  oq_jastrow_vgl_coulomb<NE, T>(J, S, pos, ps, e, xe, ye, ze, jx, jy, jz, jl, ee, en);
  const double sgx = (double)gx, sgy = (double)gy, sgz = (double)gz;
  const double Gx = sgx + (double)jx, Gy = sgy + (double)jy, Gz = sgz + (double)jz;
  lape = (double)lp - (sgx * sgx + sgy * sgy + sgz * sgz) + (double)jl;
  lp_tot += lape;
  g2 += Gx * Gx + Gy * Gy + Gz * Gz;
  gxo = Gx; gyo = Gy; gzo = Gz;
}

template <int NOCC, typename T, typename Real, class B, class SJ>
__device__ __forceinline__ void oq_eloc_electron(const SJ& J, const OqSystem& S,
                                                 const OqSplit& SP, const Real* __restrict__ C,
                                                 const double* pos, size_t ps, const Real* A,
                                                 size_t as, int e, double& ee, double& en,
                                                 double& lp_tot, double& g2) {
  double gx, gy, gz, le;
  oq_eloc_electron_out<NOCC, T, Real, B>(J, S, SP, C, pos, ps, A, as, e, ee, en, lp_tot, g2,
                                         gx, gy, gz, le);
}

// Electron e's share of the Jastrow value J (log_trial_wavefunction,
// gto.py:2220-2254): its pairs with the electrons j > e and its
// electron-nucleus terms, each term in working precision T, summed in FP64.
// Summed over all electrons this is J1 + J2 (+ B-spline, J3).
template <int NE, typename T>
__device__ __forceinline__ double oq_jastrow_value_electron(const OqSystem& S, const double* pos,
                                                           size_t ps, int e, double xe,
                                                           double ye, double ze) {
  double J = 0.0;
  for (int j = e + 1; j < NE; ++j) {
    const double dx = xe - pos[(size_t)(3 * j) * ps], dy = ye - pos[(size_t)(3 * j + 1) * ps],
                 dz = ze - pos[(size_t)(3 * j + 2) * ps];
    const T r = sqrt((T)(dx * dx + dy * dy + dz * dz));
    const bool like = (e & 1) == (j & 1);
    if (S.has_j2) {
      const int o = like ? 0 : 2;
      J += (double)oq_pade<T>((T)S.j2[o], (T)S.j2[o + 1], r);
    }
    if (OQ_HAS_BS2(S))
      J += (double)oq_bs_val<T>(like ? S.bs2_like : S.bs2_unlike,
                                like ? S.bs2_n_like : S.bs2_n_unlike,
                                (T)(like ? S.bs2_dinv_like : S.bs2_dinv_unlike),
                                (T)S.bs2_rcut, r);
  }
  for (int I = 0; I < S.natm; ++I) {
    const double dx = xe - S.nuc[I][0], dy = ye - S.nuc[I][1], dz = ze - S.nuc[I][2];
    const T r = sqrt((T)(dx * dx + dy * dy + dz * dz));
    if (S.has_j1) J += (double)oq_pade<T>((T)S.j1a[I], (T)S.j1b[I], r);
    if (OQ_HAS_BS1(S) && S.bs1_type[I] >= 0) {
      const int ty = S.bs1_type[I];
      J += (double)oq_bs_val<T>(S.bs1_c[ty], S.bs1_n[ty], (T)S.bs1_dinv[ty],
                                (T)S.bs1_rcut[ty], r);
    }
  }
  if (OQ_HAS_J3(S)) J -= (double)oq_j3_electron<T>(S, pos, ps, NE, e, e + 1, xe, ye, ze);
  return J;
}

struct OqElocArgs {
  const double* pos;
  const void* ainv;
  int W;
  int pad;
  double* sums;           // OQ_NSUM slot of this measurement (accumulated)
  double* el_trace;       // (W) local energies of this measurement, or null
  double* eparts;         // (W, 4) ee, en, ke, E_L, or null
  unsigned* flags;
  // per-walker outputs of oqmc_state_eval (null in the sampling kernels)
  double* logpsi;         // (W): holds log|det| on entry; each electron adds its J share
  double* grad;           // (W, NE, 3) gradient of log|psi|
  double* lap;            // (W, NE) Laplacian of log|psi|
};

// Local energy, one thread per (walker, electron): blockDim = (32, NE), lane
// x = walker, y = electron.  Each thread forms its electron's MO VGL, the
// Slater gradient/Laplacian against column i of the inverse
// (_slater_det_assemble, gto.py:728-778), the Padé Jastrow VGL
// (gto.py:1575-1649) and its Coulomb terms (gto.py:2406-2451); the CTA then
// reduces over electrons (local_energy_ke, gto.py:2506-2579) and over
// walkers (fused reduction of E, E^2 and the parts).
template <int NOCC, typename T, typename Real, class B = OqBasisTable<NOCC>>
__global__ void __launch_bounds__(64 * NOCC, (NOCC <= 6) ? 2 : 1)
k_eloc(const OqSystem* __restrict__ gsys, const OqSplit* __restrict__ gsplit,
       const void* __restrict__ gC, OqElocArgs a) {
  constexpr int NE = 2 * NOCC;
  extern __shared__ __align__(16) unsigned char smem[];
  OqSystem& S = *reinterpret_cast<OqSystem*>(smem);
  OqSplit& SP = *reinterpret_cast<OqSplit*>(smem + sizeof(OqSystem));
  unsigned char* p = smem + sizeof(OqSystem) + sizeof(OqSplit);
  Real* C = reinterpret_cast<Real*>(p);
  const int nbf = gsys->nbf;
  p += ((size_t)nbf * NOCC * sizeof(Real) + 15) & ~(size_t)15;
  double* red = reinterpret_cast<double*>(p);          // [NE][4][32]
  const int lane = threadIdx.x, e = threadIdx.y;
  const int flat = e * 32 + lane, nthr = 32 * NE;
  {
    const int4* s4 = reinterpret_cast<const int4*>(gsys);
    int4* d4 = reinterpret_cast<int4*>(&S);
    for (int i = flat; i < (int)(sizeof(OqSystem) / 16); i += nthr) d4[i] = s4[i];
    const double* src = reinterpret_cast<const double*>(gsplit);
    double* dst = reinterpret_cast<double*>(&SP);
    for (int i = flat; i < OQ_MAX_GROUP; i += nthr) dst[i] = src[i];
    const Real* gc = reinterpret_cast<const Real*>(gC);
    for (int i = flat; i < nbf * NOCC; i += nthr) C[i] = gc[i];
  }
  __syncthreads();
  const int W = a.W;
  const int w = blockIdx.x * 32 + lane;
  const bool live = w < W;
  double ee = 0.0, en = 0.0, lp_tot = 0.0, g2 = 0.0;
  if (live) {
    double gx, gy, gz, le;
    typename OqJasSel<B>::type J = OqJasSel<B>::of(S);
    oq_eloc_electron_out<NOCC, T, Real, B>(J, S, SP, C, a.pos + w, (size_t)W,
                                           reinterpret_cast<const Real*>(a.ainv) + w,
                                           (size_t)W, e, ee, en, lp_tot, g2, gx, gy, gz, le);
    if (a.grad) {
      double* g = a.grad + ((size_t)w * NE + e) * 3;
      g[0] = gx; g[1] = gy; g[2] = gz;
    }
    if (a.lap) a.lap[(size_t)w * NE + e] = le;
    if (a.logpsi) {
      const double* pw = a.pos + w;
      atomicAdd(a.logpsi + w,
                oq_jastrow_value_electron<NE, T>(S, pw, (size_t)W, e, pw[(size_t)(3 * e) * W],
                                                 pw[(size_t)(3 * e + 1) * W],
                                                 pw[(size_t)(3 * e + 2) * W]));
    }
  }
  red[(e * 4 + 0) * 32 + lane] = ee;
  red[(e * 4 + 1) * 32 + lane] = en;
  red[(e * 4 + 2) * 32 + lane] = lp_tot;
  red[(e * 4 + 3) * 32 + lane] = g2;
  __syncthreads();
  if (e != 0) return;
  double see = 0.0, sen = 0.0, slp = 0.0, sg2 = 0.0;
  for (int k = 0; k < NE; ++k) {
    see += red[(k * 4 + 0) * 32 + lane];
    sen += red[(k * 4 + 1) * 32 + lane];
    slp += red[(k * 4 + 2) * 32 + lane];
    sg2 += red[(k * 4 + 3) * 32 + lane];
  }
  const double ke = -0.5 * (slp + sg2);
  const double el = see + sen + ke + S.e_nn;
  const bool ok = live && isfinite(el);
  if (live) {
    if (a.el_trace) a.el_trace[w] = el;
    if (a.eparts) {
      double* ep = a.eparts + (size_t)w * 4;
      ep[0] = see; ep[1] = sen; ep[2] = ke; ep[3] = el;
    }
    if (!ok) atomicOr(a.flags, OQ_FLAG_NAN);
  }
  double vals[6] = {ok ? see : 0.0, ok ? sen : 0.0, ok ? ke : 0.0, ok ? el : 0.0,
                    ok ? el * el : 0.0, ok ? 1.0 : 0.0};
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    double v = vals[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    vals[k] = v;
  }
  if (lane == 0 && a.sums) {
#pragma unroll
    for (int k = 0; k < 5; ++k) atomicAdd(a.sums + k, vals[k]);
    atomicAdd(a.sums + 6, vals[5]);
  }
}

// ---------------------------------------------------------------------------
// Fused sweeps: moves and local energies of n_sweeps sweeps in one launch, with
// P lanes (threads of one warp) per walker, P a power of two chosen from the
// walker count (sweep_lanes, oqmc.cu).
//
// Why.  Separate move and local-energy launches per sweep with one thread per
// walker leave most of the chip idle below some ten thousand walkers: 1,000
// H2O walkers are 8 CTAs, each thread a serial chain of 10 orbital rows, 90
// pair terms and 10 updates per sweep, and every launch copies the tables and
// the state again.  The proposal of an electron and its orbital row depend on
// that electron alone, so the lanes of a walker form the rows of P electrons
// at once; the moves are then decided in order, every lane taking part (pair
// terms and columns of the update split over the lanes), and in the local
// energy each lane takes electrons of its own.
//
// In FP32 the Jastrow change is summed over all pairs on every lane, in the
// order of the one-lane form: a different order of summation would round
// differently and flip a decision in some 10^7.  In FP64 the pairs are split
// and added by shuffles (the rounding is below any decision's resolution).
// ---------------------------------------------------------------------------
struct OqSweepArgs {
  double* X;               // walkers (W, n_e, 3), updated in place
  double* pos;             // the state's positions (SoA), written at the end (may be null)
  void* ainv;
  double* logdet;
  int W;
  int n_sweeps;
  int measure_every;       // 0: no local energies
  int proposal;            // 0 fixed width, 1 nucleus-scaled width
  int lanes;               // P
  int j3_cache;            // three-body terms on several lanes: distances kept per walker
  int j3_len;              // doubles of the gamma table to copy to shared memory (0: none)
  int pad;
  double step, scale_r0, scale_fmin;
  uint64_t seed, step_base;
  double* sums;            // [n_meas][OQ_NSUM] or null
  double* el_trace;        // [n_meas][W] or null
  double* eparts_last;     // (W, 4) of the last measurement, or null
  unsigned* flags;
  double* acc_sum;         // += accepted moves outside measurements (may be null)
  // Equilibration (one sweep per launch): the width is read from step_dev and
  // the last CTA adapts it, see below.
  double* step_dev;
  double* step_trace;
  double tick, inv_moves, rate, target;
};

// Bytes of a tile of wt walkers after the system tables, split radii and
// coefficients: positions, inverses and, for three-body terms on several
// lanes, the nucleus-electron distances and the gamma table.
inline size_t oq_sweep_tile_bytes(int nocc, int natm, int wt, size_t real, int j3_cache,
                                  int j3_len) {
  return (size_t)(6 * nocc + 1) * wt * 8 +
         (((size_t)(2 * nocc * nocc + 1) * wt * real + 15) & ~(size_t)15) +
         (j3_cache ? (size_t)(2 * nocc * natm + 1) * wt * 8 + (size_t)j3_len * 8 : 0);
}

// This lane's share of the change of J3 when electron e moves to n (terms
// t = lane, lane + P, ... of the nucleus-electron list).  rI holds the
// walker's nucleus-electron distances [I][j].
template <int NE, typename T>
__device__ __forceinline__ T oq_j3_delta_lane(const OqSystem& S, const double* pos,
                                              const double* rI, int e, int lane, int P,
                                              double ox, double oy, double oz, double nx,
                                              double ny, double nz) {
  const int nI = S.j3_nI, nE = S.j3_nE, bsz = (nI + 1) * (nI + 1) * (nE + 1);
  const T L = (T)S.j3_L;
  T acc = (T)0;
  for (int t = lane; t < S.natm * NE; t += P) {
    const int I = t / NE, j = t - I * NE, ty = S.j3_type[I], blk = (e ^ j) & 1;
    if (j == e || ty < 0 || !S.j3_on[ty][blk]) continue;
    const T r2 = (T)rI[t];
    if (!(r2 < L)) continue;
    const T r1o = (T)rI[I * NE + e];
    const double ax = nx - S.nuc[I][0], ay = ny - S.nuc[I][1], az = nz - S.nuc[I][2];
    const T r1n = sqrt((T)(ax * ax + ay * ay + az * az));
    const double* g = S.j3_gamma + (size_t)(2 * ty + blk) * bsz;
    const double xj = pos[3 * j], yj = pos[3 * j + 1], zj = pos[3 * j + 2];
    if (r1n < L) {
      const double dx = nx - xj, dy = ny - yj, dz = nz - zj;
      acc += oq_j3_u_n<T>(g, nI, nE, L, sqrt((T)(dx * dx + dy * dy + dz * dz)), r1n, r2);
    }
    if (r1o < L) {
      const double dx = ox - xj, dy = oy - yj, dz = oz - zj;
      acc -= oq_j3_u_n<T>(g, nI, nE, L, sqrt((T)(dx * dx + dy * dy + dz * dz)), r1o, r2);
    }
  }
  return -acc;
}

// This lane's share of the Padé and B-spline change (pairs j and nuclei I
// congruent to lane modulo P; the terms of oq_jastrow_delta) and of the
// MIN_DIST_THRESHOLD test.
template <int NE, typename T, class SJ>
__device__ __forceinline__ T oq_jastrow_part(const SJ& J, const OqSystem& S, const double* pos,
                                             int e,
                                             int lane, int P, double ox, double oy, double oz,
                                             double nx, double ny, double nz, bool& valid) {
  const double thr2 = 1e-4 * 1e-4;
  T dJ = (T)0;
  valid = true;
  for (int j = lane; j < NE; j += P) {
    if (j == e) continue;
    const double xj = pos[3 * j], yj = pos[3 * j + 1], zj = pos[3 * j + 2];
    const double ax = nx - xj, ay = ny - yj, az = nz - zj;
    const double bx = ox - xj, by = oy - yj, bz = oz - zj;
    const double rn2 = ax * ax + ay * ay + az * az;
    valid = valid && (rn2 >= thr2);
    const T rn2t = (T)rn2, ro2t = (T)(bx * bx + by * by + bz * bz);
    const bool like = (e & 1) == (j & 1);
    if (J.has_j2) {
      const int o = like ? 0 : 2;
      dJ += oq_pade_diff((T)J.j2[o], (T)J.j2[o + 1], rn2t * oq_rsqrt(rn2t),
                         ro2t * oq_rsqrt(ro2t));
    }
    if (OQ_HAS_BS2(S)) {
      const double* c = like ? S.bs2_like : S.bs2_unlike;
      const int n = like ? S.bs2_n_like : S.bs2_n_unlike;
      const T dinv = (T)(like ? S.bs2_dinv_like : S.bs2_dinv_unlike), rc = (T)S.bs2_rcut;
      dJ += oq_bs_val<T>(c, n, dinv, rc, rn2t * oq_rsqrt(rn2t)) -
            oq_bs_val<T>(c, n, dinv, rc, ro2t * oq_rsqrt(ro2t));
    }
  }
  // the nuclei go to the lanes that the pairs load least
  for (int I = P - 1 - lane; I < J.natm; I += P) {
    const double ax = nx - J.nuc[I][0], ay = ny - J.nuc[I][1], az = nz - J.nuc[I][2];
    const double rn2 = ax * ax + ay * ay + az * az;
    valid = valid && (rn2 >= thr2);
    const double bx = ox - J.nuc[I][0], by = oy - J.nuc[I][1], bz = oz - J.nuc[I][2];
    const T rn2t = (T)rn2, ro2t = (T)(bx * bx + by * by + bz * bz);
    if (J.has_j1)
      dJ += oq_pade_diff((T)J.j1a[I], (T)J.j1b[I], rn2t * oq_rsqrt(rn2t), ro2t * oq_rsqrt(ro2t));
    if (OQ_HAS_BS1(S) && S.bs1_type[I] >= 0) {
      const int ty = S.bs1_type[I];
      const T dinv = (T)S.bs1_dinv[ty], rc = (T)S.bs1_rcut[ty];
      dJ += oq_bs_val<T>(S.bs1_c[ty], S.bs1_n[ty], dinv, rc, rn2t * oq_rsqrt(rn2t)) -
            oq_bs_val<T>(S.bs1_c[ty], S.bs1_n[ty], dinv, rc, ro2t * oq_rsqrt(ro2t));
    }
  }
  return dJ;
}

template <typename V>
__device__ __forceinline__ V oq_group_sum(V v, int P) {
  for (int o = P >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One sweep of a walker on its P lanes; returns the accepted moves (the same
// on every lane).  All lanes of the warp call it; walkers beyond the tile
// (live = false) never accept.
template <int NOCC, typename T, typename Real, class B, class SJ>
__device__ __forceinline__ int oq_sweep_lanes(const OqSweepArgs& a, const SJ& J, const OqSystem& S,
                                              const OqSplit& SP, const Real* C, double* pos,
                                              Real* Ai, double* rI, int lane, int P,
                                              bool live, uint32_t w, uint32_t gstep, double step,
                                              const OqScaledF& pf, double& logdet) {
  constexpr int NE = 2 * NOCC;
  constexpr int NN = NOCC * NOCC;
  double det = 1.0;         // product of the accepted |R|: one logarithm per sweep
  const unsigned gbits = P == 32 ? 0xffffffffu : (1u << P) - 1u;
  const int gshift = (threadIdx.x & 31) & ~(P - 1);
  int nacc = 0;
  for (int e0 = 0; e0 < NE; e0 += P) {
    // this lane's electron of the block: proposal and orbital row
    const int e = e0 + lane;
    double nx = 0.0, ny = 0.0, nz = 0.0;
    T u = (T)2, mul = (T)1, lx = (T)0;
    T v[NOCC];
#pragma unroll
    for (int m = 0; m < NOCC; ++m) v[m] = (T)0;
    if (live && e < NE) {
      float nf[3];
      uint32_t ub;
      oq_move_normals(a.seed, w, gstep, (uint32_t)e, nf, ub);
      u = oq_uniform<T>(ub);
      const double ox = pos[3 * e], oy = pos[3 * e + 1], oz = pos[3 * e + 2];
      if (a.proposal == 0) {
        nx = ox + step * (double)nf[0];
        ny = oy + step * (double)nf[1];
        nz = oz + step * (double)nf[2];
      } else {
        oq_scaled_propose_t<T>(J, ox, oy, oz, nf, pf, nx, ny, nz, mul, lx);
      }
      B::template mo_val<T, Real>(S, SP, C, nx, ny, nz, v);
    }
    // the block's moves in order
    const int nb = min(P, NE - e0);
    for (int q = 0; q < nb; ++q) {
      const int ee = e0 + q, s = ee & 1, i = ee >> 1;
      const double bx = __shfl_sync(0xffffffffu, nx, q, P);
      const double by = __shfl_sync(0xffffffffu, ny, q, P);
      const double bz = __shfl_sync(0xffffffffu, nz, q, P);
      const T bu = __shfl_sync(0xffffffffu, u, q, P);
      const T bmul = __shfl_sync(0xffffffffu, mul, q, P);
      const T blx = __shfl_sync(0xffffffffu, lx, q, P);
      T bv[NOCC];
#pragma unroll
      for (int m = 0; m < NOCC; ++m) bv[m] = __shfl_sync(0xffffffffu, v[m], q, P);
      const double ox = pos[3 * ee], oy = pos[3 * ee + 1],
                   oz = pos[3 * ee + 2];
      bool valid;
      T dJ;
      if (sizeof(T) == 8) {
        dJ = oq_jastrow_part<NE, T>(J, S, pos, ee, lane, P, ox, oy, oz, bx, by, bz, valid);
        if (OQ_HAS_J3(S))
          dJ += oq_j3_delta_lane<NE, T>(S, pos, rI, ee, lane, P, ox, oy, oz, bx, by, bz);
        dJ = oq_group_sum(dJ, P);
        valid = ((__ballot_sync(0xffffffffu, !valid) >> gshift) & gbits) == 0u;
      } else {
        dJ = oq_jastrow_delta<NE, T>(J, S, pos, 1, ee, ox, oy, oz, bx, by, bz, valid);
      }
      Real* As = Ai + s * NN;
      T R = (T)0;
      T coli[NOCC];
#pragma unroll
      for (int k = 0; k < NOCC; ++k) {
        coli[k] = (T)As[k * NOCC + i];
        R += bv[k] * coli[k];
      }
      const bool acc = live && oq_accept<T>(R, dJ, blx, bmul, bu, valid);
      // every lane has read column i before any lane updates it
      __syncwarp();
      if (acc) {
        const T rinv = oq_rcp(R);
        for (int j = lane; j < NOCC; j += P) {
          T wj = (T)0;
#pragma unroll
          for (int m = 0; m < NOCC; ++m) wj += bv[m] * (T)As[m * NOCC + j];
          const T f = (wj - (j == i ? (T)1 : (T)0)) * rinv;
#pragma unroll
          for (int k = 0; k < NOCC; ++k) {
            Real& ref = As[k * NOCC + j];
            ref = (Real)((T)ref - coli[k] * f);
          }
        }
        if (lane == 0) {
          pos[3 * ee] = bx;
          pos[3 * ee + 1] = by;
          pos[3 * ee + 2] = bz;
        }
        if (sizeof(T) == 8 && OQ_HAS_J3(S))
          for (int I = lane; I < S.natm; I += P) {
            const double ax = bx - S.nuc[I][0], ay = by - S.nuc[I][1], az = bz - S.nuc[I][2];
            rI[I * NE + ee] = sqrt(ax * ax + ay * ay + az * az);
          }
        ++nacc;
        det *= fabs((double)R);
        if (!(det > 1e-150 && det < 1e150)) {
          logdet += log(det);
          det = 1.0;
        }
      }
      // the move is visible to every lane before the next one
      __syncwarp();
    }
  }
  logdet += log(det);
  return nacc;
}

// Three-body part of the local energy of electron e: terms t = q, q + Q, ...
// of the nucleus-electron list (the terms of oq_j3_vgl_electron).
template <int NE, typename T>
__device__ __forceinline__ void oq_j3_vgl_part(const OqSystem& S, const double* pos,
                                               int e, int q, int Q, double x, double y, double z,
                                               T& gx, T& gy, T& gz, T& lp) {
  const int nI = S.j3_nI, nE = S.j3_nE, bsz = (nI + 1) * (nI + 1) * (nE + 1);
  const T L = (T)S.j3_L;
  for (int t = q; t < S.natm * NE; t += Q) {
    const int I = t / NE, j = t - I * NE, ty = S.j3_type[I], blk = (e ^ j) & 1;
    if (j == e || ty < 0 || !S.j3_on[ty][blk]) continue;
    const T ax = (T)(x - S.nuc[I][0]), ay = (T)(y - S.nuc[I][1]), az = (T)(z - S.nuc[I][2]);
    const T r1 = sqrt(ax * ax + ay * ay + az * az);
    if (!(r1 < L)) continue;
    const double xj = pos[3 * j], yj = pos[3 * j + 1], zj = pos[3 * j + 2];
    const T bx = (T)(xj - S.nuc[I][0]), by = (T)(yj - S.nuc[I][1]), bz = (T)(zj - S.nuc[I][2]);
    const T r2 = sqrt(bx * bx + by * by + bz * bz);
    if (!(r2 < L)) continue;
    const T dx = (T)(x - xj), dy = (T)(y - yj), dz = (T)(z - zj);
    const T r12 = sqrt(dx * dx + dy * dy + dz * dz);
    const T i1 = (T)1 / r1, i12 = (T)1 / r12;
    const T e1x = ax * i1, e1y = ay * i1, e1z = az * i1;
    const T ex = dx * i12, ey = dy * i12, ez = dz * i12;
    T u1, ue, u11, uee, u1e;
    oq_j3_partials_n<T>(S.j3_gamma + (size_t)(2 * ty + blk) * bsz, nI, nE, L, r12, r1, r2, u1, ue,
                        u11, uee, u1e);
    gx -= u1 * e1x + ue * ex;
    gy -= u1 * e1y + ue * ey;
    gz -= u1 * e1z + ue * ez;
    lp -= u11 + (T)2 * u1 * i1 + uee + (T)2 * ue * i12 +
          (T)2 * u1e * (e1x * ex + e1y * ey + e1z * ez);
  }
}

template <int NOCC, typename T, typename Real, class B = OqBasisTable<NOCC>>
__global__ void __launch_bounds__(128, 4)
k_sweeps(const OqSystem* __restrict__ gsys, const OqSplit* __restrict__ gsplit,
         const void* __restrict__ gC, OqSweepArgs a) {
  constexpr int NE = 2 * NOCC;
  constexpr int NN = NOCC * NOCC;
  extern __shared__ __align__(16) unsigned char smem[];
  OqSystem& S = *reinterpret_cast<OqSystem*>(smem);
  OqSplit& SP = *reinterpret_cast<OqSplit*>(smem + sizeof(OqSystem));
  unsigned char* p = smem + sizeof(OqSystem) + sizeof(OqSplit);
  Real* C = reinterpret_cast<Real*>(p);
  const int nbf = gsys->nbf, natm = gsys->natm;
  p += ((size_t)nbf * NOCC * sizeof(Real) + 15) & ~(size_t)15;
  const int P = a.lanes, WT = blockDim.x / P, tid = threadIdx.x;
  const int lane = tid & (P - 1), wl = tid / P, W = a.W;
  // a walker's state is contiguous (every index below is an immediate offset),
  // with odd pitches so that the walkers of a warp fall on different banks;
  // walker-minor, two thirds of the shared-memory wavefronts were conflicts
  constexpr int PP = 3 * NE + 1, AP = 2 * NN + 1;
  double* pos0 = reinterpret_cast<double*>(p);          // [WT][PP]
  p += (size_t)PP * WT * 8;
  Real* Ai0 = reinterpret_cast<Real*>(p);               // [WT][AP]
  p += ((size_t)AP * WT * sizeof(Real) + 15) & ~(size_t)15;
  double* rI0 = reinterpret_cast<double*>(p);           // [WT][natm NE + 1], three-body only
  const int RP = natm * NE + 1;
  double* gam = rI0 + (size_t)RP * WT;
  const int w0 = blockIdx.x * WT, cnt = min(WT, W - w0);
  oq_load_system(&S, gsys);
  {
    const double* src = reinterpret_cast<const double*>(gsplit);
    double* dst = reinterpret_cast<double*>(&SP);
    for (int i = tid; i < OQ_MAX_GROUP; i += blockDim.x) dst[i] = src[i];
    const Real* gc = reinterpret_cast<const Real*>(gC);
    for (int i = tid; i < nbf * NOCC; i += blockDim.x) C[i] = gc[i];
    const double* x = a.X + (size_t)w0 * 3 * NE;
    for (int q = tid; q < cnt * 3 * NE; q += blockDim.x) {
      const int j = q / (3 * NE), k = q - j * 3 * NE;
      pos0[j * PP + k] = x[q];
    }
    const Real* gA = reinterpret_cast<const Real*>(a.ainv);
    for (int q = tid; q < 2 * NN * WT; q += blockDim.x) {
      const int k = q / WT, j = q - k * WT;
      if (j < cnt) Ai0[j * AP + k] = gA[(size_t)k * W + w0 + j];
    }
    for (int i = tid; i < a.j3_len; i += blockDim.x) gam[i] = gsys->j3_gamma[i];
  }
  __syncthreads();
  if (a.j3_cache) {
    // the three-body code reads the table through S
    if (tid == 0 && a.j3_len) S.j3_gamma = gam;
    for (int q = tid; q < natm * NE * cnt; q += blockDim.x) {
      const int j = q % cnt, t = q / cnt, I = t / NE, e = t - I * NE;
      const double dx = pos0[j * PP + 3 * e] - S.nuc[I][0],
                   dy = pos0[j * PP + 3 * e + 1] - S.nuc[I][1],
                   dz = pos0[j * PP + 3 * e + 2] - S.nuc[I][2];
      rI0[j * RP + t] = sqrt(dx * dx + dy * dy + dz * dz);
    }
    __syncthreads();
  }
  const bool live = wl < cnt;
  const uint32_t w = (uint32_t)(w0 + wl);
  double* pos = pos0 + wl * PP;
  Real* Ai = Ai0 + wl * AP;
  double* rI = rI0 + wl * RP;
  typename OqJasSel<B>::type J = OqJasSel<B>::of(S);
  const double step = a.step_dev ? *a.step_dev : a.step;
  const OqScaledF pf = oq_scaled_f(step, a.scale_r0, a.scale_fmin);
  double logdet = live ? a.logdet[w] : 0.0;
  const int n_meas = a.measure_every > 0 ? a.n_sweeps / a.measure_every : 0;
  // local energy: PE electrons at a time, Q lanes share an electron's three-body terms
  const int PE = min(P, NE), Q = P / PE, le = lane % PE, lq = lane / PE;
  int nacc = 0, meas = 0;
  for (int t = 0; t < a.n_sweeps; ++t) {
    const uint32_t gstep = (uint32_t)(a.step_base + t);
    if (P > 1) {
      nacc += oq_sweep_lanes<NOCC, T, Real, B>(a, J, S, SP, C, pos, Ai, rI, lane, P, live, w,
                                               gstep, step, pf, logdet);
    } else if (live) {
      for (int e = 0; e < NE; ++e) {
        float nf[3];
        uint32_t ub;
        oq_move_normals(a.seed, w, gstep, (uint32_t)e, nf, ub);
        const T u = oq_uniform<T>(ub);
        const double ox = pos[3 * e], oy = pos[3 * e + 1],
                     oz = pos[3 * e + 2];
        double nx, ny, nz;
        T mul = (T)1, lx = (T)0;
        if (a.proposal == 0) {
          nx = ox + step * (double)nf[0];
          ny = oy + step * (double)nf[1];
          nz = oz + step * (double)nf[2];
        } else {
          oq_scaled_propose_t<T>(J, ox, oy, oz, nf, pf, nx, ny, nz, mul, lx);
        }
        nacc += oq_try_move_s<NOCC, T, Real, B>(J, S, SP, C, pos, 1, Ai, 1, e, nx, ny, nz, lx,
                                                mul, u, logdet);
      }
    }
    if (meas == n_meas || (t + 1) % a.measure_every != 0) continue;
    // a walker's state is read and written only by its own lanes, which
    // share one warp: the moves are complete for them after a warp barrier
    __syncwarp();
    double see = 0.0, sen = 0.0, slp = 0.0, sg2 = 0.0;
    if (sizeof(T) == 4) {
      if (live && lq == 0)
        for (int e = le; e < NE; e += PE)
          oq_eloc_electron<NOCC, T, Real, B>(J, S, SP, C, pos, 1, Ai, 1, e, see,
                                             sen, slp, sg2);
    } else {
      // one electron per lane; its three-body terms split over Q lanes
      for (int e0 = 0; e0 < NE; e0 += PE) {
        const bool mine_e = live && e0 + le < NE;
        const int e = mine_e ? e0 + le : 0, s = e & 1, i = e >> 1;
        const double xe = pos[3 * e], ye = pos[3 * e + 1],
                     ze = pos[3 * e + 2];
        T jx = (T)0, jy = (T)0, jz = (T)0, jl = (T)0;
        if (OQ_HAS_J3(S)) {
          T gx = (T)0, gy = (T)0, gz = (T)0, gl = (T)0;
          if (mine_e && lq < Q)
            oq_j3_vgl_part<NE, T>(S, pos, e, lq, Q, xe, ye, ze, gx, gy, gz, gl);
          for (int k = 0; k < Q; ++k) {
            jx += __shfl_sync(0xffffffffu, gx, le + k * PE, P);
            jy += __shfl_sync(0xffffffffu, gy, le + k * PE, P);
            jz += __shfl_sync(0xffffffffu, gz, le + k * PE, P);
            jl += __shfl_sync(0xffffffffu, gl, le + k * PE, P);
          }
        }
        if (mine_e && lq == 0) {
          T ac[NOCC];
#pragma unroll
          for (int m = 0; m < NOCC; ++m) ac[m] = (T)Ai[(s * NOCC + m) * NOCC + i];
          T gx, gy, gz, lp;
          B::template mo_vgl_contract<T, Real>(S, SP, C, xe, ye, ze, ac, gx, gy, gz, lp);
          oq_jastrow_vgl_coulomb<NE, T>(J, S, pos, 1, e, xe, ye, ze, jx, jy, jz, jl, see,
                                        sen, false);
          const double sx = (double)gx, sy = (double)gy, sz = (double)gz;
          const double Gx = sx + (double)jx, Gy = sy + (double)jy, Gz = sz + (double)jz;
          slp += (double)lp - (sx * sx + sy * sy + sz * sz) + (double)jl;
          sg2 += Gx * Gx + Gy * Gy + Gz * Gz;
        }
      }
    }
    see = oq_group_sum(see, P);
    sen = oq_group_sum(sen, P);
    slp = oq_group_sum(slp, P);
    sg2 = oq_group_sum(sg2, P);
    const double ke = -0.5 * (slp + sg2);
    const double el = see + sen + ke + S.e_nn;
    const bool mine = live && lane == 0;
    const bool ok = mine && isfinite(el);
    if (mine) {
      if (a.el_trace) a.el_trace[(size_t)meas * W + w] = el;
      if (a.eparts_last && meas == n_meas - 1) {
        double* ep = a.eparts_last + (size_t)w * 4;
        ep[0] = see; ep[1] = sen; ep[2] = ke; ep[3] = el;
      }
      if (!ok) atomicOr(a.flags, OQ_FLAG_NAN);
    }
    double vals[7] = {ok ? see : 0.0, ok ? sen : 0.0, ok ? ke : 0.0, ok ? el : 0.0,
                      ok ? el * el : 0.0, mine ? (double)nacc : 0.0, ok ? 1.0 : 0.0};
#pragma unroll
    for (int k = 0; k < 7; ++k) vals[k] = oq_group_sum(vals[k], 32);
    if ((tid & 31) == 0) {
      double* sm = a.sums + (size_t)meas * OQ_NSUM;
#pragma unroll
      for (int k = 0; k < 7; ++k) atomicAdd(sm + k, vals[k]);
    }
    // the next sweep's moves change state this measurement read
    __syncwarp();
    nacc = 0;
    ++meas;
  }
  __syncthreads();
  {
    double* x = a.X + (size_t)w0 * 3 * NE;
    for (int q = tid; q < cnt * 3 * NE; q += blockDim.x) {
      const int j = q / (3 * NE), k = q - j * 3 * NE;
      x[q] = pos0[j * PP + k];
    }
    Real* gA = reinterpret_cast<Real*>(a.ainv);
    for (int q = tid; q < 2 * NN * WT; q += blockDim.x) {
      const int k = q / WT, j = q - k * WT;
      if (j < cnt) gA[(size_t)k * W + w0 + j] = Ai0[j * AP + k];
    }
    if (a.pos)
      for (int q = tid; q < 3 * NE * WT; q += blockDim.x) {
        const int k = q / WT, j = q - k * WT;
        if (j < cnt) a.pos[(size_t)k * W + w0 + j] = pos0[j * PP + k];
      }
  }
  if (live && lane == 0) a.logdet[w] = logdet;
  if (!a.acc_sum) return;
  const int mine = (int)oq_group_sum(live && lane == 0 ? nacc : 0, 32);
  if (!a.step_dev) {
    if ((tid & 31) == 0) atomicAdd(a.acc_sum, (double)mine);
    return;
  }
  // Step adaptation (_adapt_step_size, OmegaQMC/vmc_gto.py:121-126): log s <-
  // log s + rate (acc - target).  Every CTA adds its accepted moves plus one
  // `tick`, a power of two above all moves of the sweep, to the sweep's slot;
  // the sum is exact, so the CTA that brings it to gridDim.x ticks is the last
  // one, knows the total, and every CTA has read the old width by then.  A
  // kernel of one thread for this cost a launch per equilibration step.
  int* part = reinterpret_cast<int*>(pos0);     // the walkers are written out
  __syncthreads();
  if ((tid & 31) == 0) part[tid >> 5] = mine;
  __syncthreads();
  if (tid != 0) return;
  int tot = 0;
  for (int k = 0; k < (int)blockDim.x / 32; ++k) tot += part[k];
  const double now = atomicAdd(a.acc_sum, (double)tot + a.tick) + (double)tot + a.tick;
  if (now >= a.tick * (double)gridDim.x) {
    const double acc = (now - a.tick * (double)gridDim.x) * a.inv_moves;
    const double sn = exp(log(step) + a.rate * (acc - a.target));
    *a.acc_sum = acc;
    *a.step_dev = sn;
    if (a.step_trace) *a.step_trace = sn;
  }
}
