// Kernel instantiations and launchers for one determinant size.
// Compile with -DOQ_N=<nocc>.
#include "oqmc_launch.h"

#ifndef OQ_N
#error "compile with -DOQ_N=<nocc>"
#endif

#define OQ_CAT2(a, b) a##_##b
#define OQ_CAT(a, b) OQ_CAT2(a, b)
#define OQ_FN(name) OQ_CAT(name, OQ_N)

// Dynamic shared memory above 48 KB needs an opt-in; every kernel also asks
// for the largest shared-memory carveout so several CTAs fit per SM.
template <typename K>
static cudaError_t oq_smem_attr(K kernel, size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  if (smem > 48 * 1024)
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                OQ_SMEM_OPTIN);
  return cudaSuccess;
}

// One tile kernel (oqmc_team.cuh); the tile's arrays follow the packed tables.
template <int MODE, typename Real, bool EXT>
static cudaError_t team_ext(const OqLaunch& L, OqTeamArgs a) {
  a.wb = oq_team_walkers<OQ_N>(a.W);
  a.flags = L.flags;
  a.Ct = L.Ct;
  // at least 128 threads, so that a small tile copies the system tables fast
  const int act = a.wb * 2 * OQ_N, tpb = act < 128 ? 128 : (act + 31) / 32 * 32;
  const size_t smem = L.ao_bytes + oq_team_tile_bytes(OQ_N, a.wb) +
                      (MODE == OQ_TEAM_EVAL ? sizeof(double) * 8 * OQ_N * OQ_N : 0);
  cudaError_t e = oq_smem_attr(k_team<OQ_N, MODE, Real, EXT>, smem);
  if (e != cudaSuccess) return e;
  k_team<OQ_N, MODE, Real, EXT><<<(a.W + a.wb - 1) / a.wb, tpb, smem, L.stream>>>(L.sys, L.ao,
                                                                            L.ao_bytes, a);
  return cudaGetLastError();
}

template <int MODE, typename Real>
static cudaError_t team(const OqLaunch& L, const OqTeamArgs& a) {
  return L.ext ? team_ext<MODE, Real, true>(L, a) : team_ext<MODE, Real, false>(L, a);
}

cudaError_t OQ_FN(oq_eval)(const OqLaunch& L, const double* X, int W, double* logpsi,
                           double* grad, double* lap, double* eparts) {
  OqTeamArgs a{};
  a.X = X; a.W = W; a.logpsi = logpsi; a.grad = grad; a.lap = lap; a.eparts = eparts;
  return team<OQ_TEAM_EVAL, double>(L, a);
}

cudaError_t OQ_FN(oq_logpsi)(const OqLaunch& L, const double* X, int W, double* logpsi) {
  OqTeamArgs a{};
  a.X = X; a.W = W; a.logpsi = logpsi;
  return team<OQ_TEAM_LOGPSI, double>(L, a);
}

template <bool EXT>
static cudaError_t movals(const OqLaunch& L, const double* X, int W, double* out) {
  const int tpb = 128;
  const long long n = (long long)W * 2 * OQ_N;
  const int nb = (int)((n + tpb - 1) / tpb);
  cudaError_t e = oq_smem_attr(k_mo_values<OQ_N, EXT>, L.ao_bytes);
  if (e != cudaSuccess) return e;
  k_mo_values<OQ_N, EXT><<<nb, tpb, L.ao_bytes, L.stream>>>(L.sys, L.ao, L.ao_bytes, X, W, out);
  return cudaGetLastError();
}

cudaError_t OQ_FN(oq_movals)(const OqLaunch& L, const double* X, int W, double* out) {
  return L.ext ? movals<true>(L, X, W, out) : movals<false>(L, X, W, out);
}

cudaError_t OQ_FN(oq_refresh)(const OqLaunch& L, const double* pos, int W, void* ainv,
                              double* logdet, int mixed) {
  OqTeamArgs a{};
  a.X = pos; a.W = W; a.ainv = ainv; a.logpsi = logdet;
  return mixed ? team<OQ_TEAM_REFRESH, float>(L, a) : team<OQ_TEAM_REFRESH, double>(L, a);
}

template <int PROP>
static cudaError_t moves_prop(const OqLaunch& L, const OqMoveArgs& a, int wpb, int mixed) {
  const int nb = (a.W + wpb - 1) / wpb;
  cudaError_t e;
  if (mixed) {
    e = oq_smem_attr(k_moves<OQ_N, float, float, PROP>, L.smem);
    if (e != cudaSuccess) return e;
    k_moves<OQ_N, float, float, PROP><<<nb, wpb, L.smem, L.stream>>>(L.sys, L.split, L.C32, a);
  } else {
    e = oq_smem_attr(k_moves<OQ_N, double, double, PROP>, L.smem);
    if (e != cudaSuccess) return e;
    k_moves<OQ_N, double, double, PROP><<<nb, wpb, L.smem, L.stream>>>(L.sys, L.split, L.C64, a);
  }
  return cudaGetLastError();
}

cudaError_t OQ_FN(oq_moves)(const OqLaunch& L, const OqMoveArgs& a, int wpb, int mixed) {
  if (a.mode == 1) return moves_prop<2>(L, a, wpb, mixed);
  // table-driven, fewer than four orbitals always sweep in k_sweeps (moves_by_thread)
#if OQ_N >= 4
  if (a.proposal == 1) return moves_prop<1>(L, a, wpb, mixed);
  return moves_prop<0>(L, a, wpb, mixed);
#else
  return cudaErrorInvalidValue;
#endif
}

cudaError_t OQ_FN(oq_sweeps)(const OqLaunch& L, const OqSweepArgs& a, int nthr, int mixed) {
  const int wt = nthr / a.lanes, nb = (a.W + wt - 1) / wt;
  cudaError_t e;
  if (mixed) {
    e = oq_smem_attr(k_sweeps<OQ_N, float, float>, L.smem);
    if (e != cudaSuccess) return e;
    k_sweeps<OQ_N, float, float><<<nb, nthr, L.smem, L.stream>>>(L.sys, L.split, L.C32, a);
  } else {
    e = oq_smem_attr(k_sweeps<OQ_N, double, double>, L.smem);
    if (e != cudaSuccess) return e;
    k_sweeps<OQ_N, double, double><<<nb, nthr, L.smem, L.stream>>>(L.sys, L.split, L.C64, a);
  }
  return cudaGetLastError();
}

cudaError_t OQ_FN(oq_eloc)(const OqLaunch& L, const OqElocArgs& a, int mixed) {
  const int nb = (a.W + 31) / 32;
  const dim3 block(32, 2 * OQ_N);
  cudaError_t e;
  if (mixed) {
    e = oq_smem_attr(k_eloc<OQ_N, float, float>, L.smem);
    if (e != cudaSuccess) return e;
    k_eloc<OQ_N, float, float><<<nb, block, L.smem, L.stream>>>(L.sys, L.split, L.C32, a);
  } else {
    e = oq_smem_attr(k_eloc<OQ_N, double, double>, L.smem);
    if (e != cudaSuccess) return e;
    k_eloc<OQ_N, double, double><<<nb, block, L.smem, L.stream>>>(L.sys, L.split, L.C64, a);
  }
  return cudaGetLastError();
}

cudaError_t OQ_FN(oq_eloc_tc)(const OqLaunch& L, const OqElocArgs& a, const void* Bpack, int nbf) {
  constexpr int WB = 128 / (2 * OQ_N);
  const int nb = (a.W + WB - 1) / WB;
  const size_t smem = oq_tc_plan(nbf).total;
  cudaError_t e = oq_smem_attr(k_eloc_tc<OQ_N>, smem);
  if (e != cudaSuccess) return e;
  k_eloc_tc<OQ_N><<<nb, 128, smem, L.stream>>>(L.sys, L.split,
                                                static_cast<const unsigned char*>(Bpack), a);
  return cudaGetLastError();
}

// Multi-determinant kernels: M = 8 or 16 orbital columns (M >= OQ_N).
template <int M>
static cudaError_t md_refresh_m(const OqLaunch& L, const OqMdTables& T, const OqMdState& st) {
  cudaError_t e = oq_smem_attr(k_md_refresh<OQ_N, M>, L.smem);
  if (e != cudaSuccess) return e;
  k_md_refresh<OQ_N, M><<<(st.W + 127) / 128, 128, L.smem, L.stream>>>(L.sys, T, st, L.flags);
  return cudaGetLastError();
}

template <int M>
static cudaError_t md_moves_m(const OqLaunch& L, const OqMdTables& T, const OqMoveArgs& a,
                              double* sgn) {
  cudaError_t e = oq_smem_attr(k_md_moves<OQ_N, M>, L.smem);
  if (e != cudaSuccess) return e;
  k_md_moves<OQ_N, M><<<(a.W + 127) / 128, 128, L.smem, L.stream>>>(L.sys, T, a, sgn);
  return cudaGetLastError();
}

template <int M>
static cudaError_t md_local_m(const OqLaunch& L, const OqMdTables& T, const OqMdState& st,
                              const OqElocArgs& a, double* logpsi, double* grad, double* lap) {
  cudaError_t e = oq_smem_attr(k_md_local<OQ_N, M>, L.smem);
  if (e != cudaSuccess) return e;
  k_md_local<OQ_N, M><<<(st.W + 127) / 128, 128, L.smem, L.stream>>>(L.sys, T, st, a, logpsi,
                                                                       grad, lap);
  return cudaGetLastError();
}

cudaError_t OQ_FN(oq_md_refresh)(const OqLaunch& L, const OqMdTables& T, const OqMdState& st,
                                 int M) {
  if constexpr (OQ_N <= 8) {
    if (M == 8) return md_refresh_m<8>(L, T, st);
  }
  return M == 16 ? md_refresh_m<16>(L, T, st) : cudaErrorInvalidValue;
}

cudaError_t OQ_FN(oq_md_moves)(const OqLaunch& L, const OqMdTables& T, const OqMoveArgs& a,
                               double* sgn, int M) {
  if constexpr (OQ_N <= 8) {
    if (M == 8) return md_moves_m<8>(L, T, a, sgn);
  }
  return M == 16 ? md_moves_m<16>(L, T, a, sgn) : cudaErrorInvalidValue;
}

cudaError_t OQ_FN(oq_md_local)(const OqLaunch& L, const OqMdTables& T, const OqMdState& st,
                               const OqElocArgs& a, double* logpsi, double* grad, double* lap,
                               int M) {
  if constexpr (OQ_N <= 8) {
    if (M == 8) return md_local_m<8>(L, T, st, a, logpsi, grad, lap);
  }
  return M == 16 ? md_local_m<16>(L, T, st, a, logpsi, grad, lap) : cudaErrorInvalidValue;
}

template <typename Real, bool EXT>
static cudaError_t alle(const OqLaunch& L, OqAlleArgs a) {
  a.wb = oq_team_walkers<OQ_N>(a.W);
  while (a.wb > 1 && L.ao_bytes + oq_alle_tile_bytes(OQ_N, a.wb) > 227 * 1024) a.wb >>= 1;
  a.flags = L.flags;
  const int act = a.wb * 2 * OQ_N, tpb = act < 128 ? 128 : (act + 31) / 32 * 32;
  const size_t smem = L.ao_bytes + oq_alle_tile_bytes(OQ_N, a.wb);
  cudaError_t e = oq_smem_attr(k_alle<OQ_N, Real, EXT>, smem);
  if (e != cudaSuccess) return e;
  k_alle<OQ_N, Real, EXT><<<(a.W + a.wb - 1) / a.wb, tpb, smem, L.stream>>>(L.sys, L.ao,
                                                                           L.ao_bytes, a);
  return cudaGetLastError();
}

cudaError_t OQ_FN(oq_alle)(const OqLaunch& L, const OqAlleArgs& a, int mixed) {
  if (mixed) return L.ext ? alle<float, true>(L, a) : alle<float, false>(L, a);
  return L.ext ? alle<double, true>(L, a) : alle<double, false>(L, a);
}

// Per-thread local memory (bytes) of one kernel this size launches: kind 0
// k_team (refresh), 1 k_sweeps, 2 k_eloc, 3 k_eloc_tc, 4 k_md_refresh,
// 5 k_md_moves, 6 k_md_local (M = 8 or 16 columns), 7 k_alle, 8 and 9 k_moves
// (fixed-width and nucleus-scaled proposal).  ext: OqLaunch::ext, for 0 and 7.
template <typename K>
static cudaError_t oq_lmem(K kernel, size_t* out) {
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
  if (e == cudaSuccess) *out = a.localSizeBytes;
  return e;
}

template <int M>
static cudaError_t md_lmem(int kind, size_t* out) {
  if (kind == 4) return oq_lmem(k_md_refresh<OQ_N, M>, out);
  if (kind == 5) return oq_lmem(k_md_moves<OQ_N, M>, out);
  return oq_lmem(k_md_local<OQ_N, M>, out);
}

template <bool EXT>
static cudaError_t tile_lmem(int kind, int mixed, size_t* out) {
  if (kind == 0)
    return mixed ? oq_lmem(k_team<OQ_N, OQ_TEAM_REFRESH, float, EXT>, out)
                 : oq_lmem(k_team<OQ_N, OQ_TEAM_REFRESH, double, EXT>, out);
  return mixed ? oq_lmem(k_alle<OQ_N, float, EXT>, out) : oq_lmem(k_alle<OQ_N, double, EXT>, out);
}

cudaError_t OQ_FN(oq_local_bytes)(int kind, int mixed, int ext, int M, size_t* out) {
  switch (kind) {
    case 0:
    case 7:
      return ext ? tile_lmem<true>(kind, mixed, out) : tile_lmem<false>(kind, mixed, out);
    case 1:
      return mixed ? oq_lmem(k_sweeps<OQ_N, float, float>, out)
                   : oq_lmem(k_sweeps<OQ_N, double, double>, out);
    case 2:
      return mixed ? oq_lmem(k_eloc<OQ_N, float, float>, out)
                   : oq_lmem(k_eloc<OQ_N, double, double>, out);
    case 3:
      return oq_lmem(k_eloc_tc<OQ_N>, out);
    case 4:
    case 5:
    case 6:
      if constexpr (OQ_N <= 8) {
        if (M == 8) return md_lmem<8>(kind, out);
      }
      return M == 16 ? md_lmem<16>(kind, out) : cudaErrorInvalidValue;
#if OQ_N >= 4
    case 8:
      return mixed ? oq_lmem(k_moves<OQ_N, float, float, 0>, out)
                   : oq_lmem(k_moves<OQ_N, double, double, 0>, out);
    case 9:
      return mixed ? oq_lmem(k_moves<OQ_N, float, float, 1>, out)
                   : oq_lmem(k_moves<OQ_N, double, double, 1>, out);
#endif
  }
  return cudaErrorInvalidValue;
}
