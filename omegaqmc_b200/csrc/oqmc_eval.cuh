// FP64 pieces of a walker's wavefunction on one thread: the inverse of a
// Slater matrix and the Jastrow value (log_trial_wavefunction,
// OmegaQMC/psi/gto.py:2220-2254).
#pragma once
#include "oqmc_ao.cuh"

#define OQ_EPS 2.220446049250313e-16

// Gauss-Jordan inverse with partial pivoting of the N x N matrix a
// (destroyed); returns false if a pivot is exactly zero or not finite.
// logdet = log|det a|; *sign (when given) = the sign of det a.
template <int N>
__device__ bool oq_invert(double (&a)[N][N], double (&inv)[N][N], double& logdet,
                          double* sign = nullptr) {
  double sg = 1.0;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) inv[i][j] = (i == j) ? 1.0 : 0.0;
  logdet = 0.0;
  for (int k = 0; k < N; ++k) {
    int piv = k;
    double best = fabs(a[k][k]);
    for (int i = k + 1; i < N; ++i) {
      const double v = fabs(a[i][k]);
      if (v > best) { best = v; piv = i; }
    }
    if (!(best > 0.0) || !isfinite(best)) return false;
    if (piv != k) {
      sg = -sg;
      for (int j = 0; j < N; ++j) {
        double t = a[k][j]; a[k][j] = a[piv][j]; a[piv][j] = t;
        t = inv[k][j]; inv[k][j] = inv[piv][j]; inv[piv][j] = t;
      }
    }
    const double d = a[k][k];
    logdet += log(fabs(d));
    if (d < 0.0) sg = -sg;
    const double rd = 1.0 / d;
    for (int j = 0; j < N; ++j) { a[k][j] *= rd; inv[k][j] *= rd; }
    for (int i = 0; i < N; ++i) {
      if (i == k) continue;
      const double f = a[i][k];
      if (f != 0.0) {
        for (int j = 0; j < N; ++j) { a[i][j] -= f * a[k][j]; inv[i][j] -= f * inv[k][j]; }
      }
    }
  }
  if (sign) *sign = sg;
  return true;
}

// Jastrow value J1 + J2 (+ J3) for walker positions x[n_e][3] (in
// registers/local).
__device__ __forceinline__ double oq_jastrow_value(const OqSystem& S, const double* x,
                                                   int n_e) {
  double J = 0.0;
  if (S.has_j2) {
    for (int i = 0; i < n_e; ++i)
      for (int j = i + 1; j < n_e; ++j) {
        const double dx = x[3 * i] - x[3 * j], dy = x[3 * i + 1] - x[3 * j + 1],
                     dz = x[3 * i + 2] - x[3 * j + 2];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        const int o = ((i & 1) == (j & 1)) ? 0 : 2;
        J += oq_pade(S.j2[o], S.j2[o + 1], r);
      }
  }
  if (S.has_j1) {
    for (int i = 0; i < n_e; ++i)
      for (int I = 0; I < S.natm; ++I) {
        const double dx = x[3 * i] - S.nuc[I][0], dy = x[3 * i + 1] - S.nuc[I][1],
                     dz = x[3 * i + 2] - S.nuc[I][2];
        J += oq_pade(S.j1a[I], S.j1b[I], sqrt(dx * dx + dy * dy + dz * dz));
      }
  }
  if (S.has_bs2) {
    for (int i = 0; i < n_e; ++i)
      for (int j = i + 1; j < n_e; ++j) {
        const double dx = x[3 * i] - x[3 * j], dy = x[3 * i + 1] - x[3 * j + 1],
                     dz = x[3 * i + 2] - x[3 * j + 2];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        const bool like = (i & 1) == (j & 1);
        J += oq_bs_val<double>(like ? S.bs2_like : S.bs2_unlike,
                               like ? S.bs2_n_like : S.bs2_n_unlike,
                               like ? S.bs2_dinv_like : S.bs2_dinv_unlike, S.bs2_rcut, r);
      }
  }
  if (S.has_bs1) {
    for (int i = 0; i < n_e; ++i)
      for (int I = 0; I < S.natm; ++I) {
        const int ty = S.bs1_type[I];
        if (ty < 0) continue;
        const double dx = x[3 * i] - S.nuc[I][0], dy = x[3 * i + 1] - S.nuc[I][1],
                     dz = x[3 * i + 2] - S.nuc[I][2];
        J += oq_bs_val<double>(S.bs1_c[ty], S.bs1_n[ty], S.bs1_dinv[ty], S.bs1_rcut[ty],
                               sqrt(dx * dx + dy * dy + dz * dz));
      }
  }
  if (S.has_j3) {
    for (int i = 0; i < n_e; ++i)
      J -= oq_j3_electron<double>(S, x, 1, n_e, i, i + 1, x[3 * i], x[3 * i + 1], x[3 * i + 2]);
  }
  return J;
}
