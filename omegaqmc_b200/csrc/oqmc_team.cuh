// FP64 evaluation with one thread per (walker, electron).
//
// A CTA takes a tile of WB walkers (a power of two) and gives every electron
// its own thread: thread t < WB * NE is walker t % WB, electron t / WB.  Each
// thread evaluates its electron's orbital row, the NE threads of a walker
// invert both Slater matrices together (one matrix column per thread) and
// each then forms its electron's gradient, Laplacian and pair terms.
//
// Why this split.  The work is FP64-pipe arithmetic (exponentials, the MO
// contraction, pair terms).  With one thread per walker the two inverses live
// in local memory and a walker is one serial chain of 2 N orbital
// evaluations: an H2O walker took 281 us alone, and 4,097 N2 walkers were 33
// CTAs on 148 SMs.  One electron per thread gives 2 N times the threads and
// an N-th of the chain, keeps one matrix column of N doubles in registers,
// and costs one barrier per elimination step.  Measured per call (thread per
// walker -> this): H2O, 1 walker 280 -> 25 us (launch and host time); N2,
// 4,097 walkers 855 -> 54 us, and 80 to 90 where walkers next to a node are
// done again (see k_team); (H2O)2, 16,384 walkers, 1,653 -> 243 us, 270 to 310
// with such walkers (FP64 pipe 38% busy, issue slots 54%); log|psi| of 65,536
// H2O walkers 181 -> 94 us.
#pragma once
#include "oqmc_sweep.cuh"

// Walkers per tile at most, and the CTA size that goes with it: 1024 threads
// would leave 64 registers, so larger determinants take fewer walkers.
template <int N>
struct OqTeam {
  static constexpr int NE = 2 * N;
  static constexpr int WB = N == 1 ? 64 : N <= 8 ? 32 : 16;
  static constexpr int T = WB * NE < 128 ? 128 : WB * NE;
  // 96 registers where that lets two or more CTAs share an SM
  static constexpr int MINB = 65536 / (96 * T) < 1 ? 1 : 65536 / (96 * T);
};

// Shared memory of a tile of wb walkers (beside the system tables and the MO
// coefficients): positions [3 NE][wb], Slater matrices [2][N][N][wb], the
// pivot columns of two elimination steps [2][2][N][wb], per-electron sums
// [NE][6][wb] and the pivot rows [2][2][wb].
constexpr size_t oq_team_tile_bytes(int n, int wb) {
  return sizeof(double) * (size_t)wb *
             ((size_t)6 * n + (size_t)2 * n * n + (size_t)4 * n + (size_t)12 * n) +
         sizeof(int) * (size_t)4 * wb;
}

// Walkers per tile for W walkers: the largest tile (whole warps of one
// electron, conflict-free shared memory) unless that leaves SMs idle; then
// halved until there are four tiles per SM, or, once a tile has no more than
// 128 threads (below that threads would idle), one per SM or a tile is a warp.
template <int N>
inline int oq_team_walkers(int W) {
  constexpr int NE = OqTeam<N>::NE;
  int wb = OqTeam<N>::WB;
  while (wb > 1 && wb * NE > 32 && (W + wb - 1) / wb < (wb * NE > 128 ? 4 * 148 : 148)) wb >>= 1;
  return wb;
}

// The tables a tile reads, packed by the host (pack_ao, oqmc.cu) into one block that
// every CTA copies into shared memory: what the FP64 evaluation of a molecule
// touches and nothing else (H2O: 2.5 KB against 14 KB of OqSystem and its MO
// coefficients), laid out as the loops read it.
//   OqAoHead
//   OqAoAtom [natm]       nuclei with their Jastrow constants and groups
//   int4     [ngroup]     x: am | columns << 4 | cusp bits << 8 | spline bits
//                         << 10 | first shell << 16; y: primitives; z: first
//                         double2 of the primitives; w: first AO
//   double2  [..]         per primitive (alpha, n0), or (alpha, n0), (n1, -)
//                         for two contraction columns
//   double   [nbf][NP]    MO coefficients, rows padded to whole double2s
// Groups with more than two columns are split, so a group has one or two.
struct OqAoHead {
  int natm, off_group, off_prim, off_C;      // byte offsets from the head
  int bytes, has_j1, has_j2, ext;            // ext: see k_team
  double e_nn, pad;
  double j2[4];
};
struct OqAoAtom {
  double x, y, z, Z, j1a, j1b;
  int g0, g1, pad0, pad1;
};

template <int N>
struct OqAo {
  static constexpr int NP = (N + 1) / 2 * 2;
  const OqAoHead* h;
  const OqAoAtom* atom;
  const int4* group;
  const double2* prim;
  const double* C;
  __device__ explicit OqAo(const unsigned char* b) {
    h = reinterpret_cast<const OqAoHead*>(b);
    atom = reinterpret_cast<const OqAoAtom*>(h + 1);
    group = reinterpret_cast<const int4*>(b + h->off_group);
    prim = reinterpret_cast<const double2*>(b + h->off_prim);
    C = reinterpret_cast<const double*>(b + h->off_C);
  }
};

template <int N>
__device__ __forceinline__ void oq_ao_add(const double* C, double v, double (&mv)[N]) {
  const double2* c2 = reinterpret_cast<const double2*>(C);
#pragma unroll
  for (int m = 0; m < N; m += 2) {
    const double2 c = c2[m / 2];
    mv[m] += c.x * v;
    if (m + 1 < N) mv[m + 1] += c.y * v;
  }
}

// The three AOs of a p function, added to each other first (the order of
// oq_mo_val).
template <int N>
__device__ __forceinline__ void oq_ao_add3(const double* C, double v0, double v1, double v2,
                                           double (&mv)[N]) {
  constexpr int NP = (N + 1) / 2 * 2;
  const double2* c2 = reinterpret_cast<const double2*>(C);
#pragma unroll
  for (int m = 0; m < N; m += 2) {
    const double2 a = c2[m / 2], b = c2[(NP + m) / 2], c = c2[(2 * NP + m) / 2];
    mv[m] += a.x * v0 + b.x * v1 + c.x * v2;
    if (m + 1 < N) mv[m + 1] += a.y * v0 + b.y * v1 + c.y * v2;
  }
}

template <int N>
__device__ __forceinline__ double oq_ao_dot(const double* C, const double (&ac)[N]) {
  const double2* c2 = reinterpret_cast<const double2*>(C);
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int m = 0; m < N; m += 2) {
    const double2 c = c2[m / 2];
    s0 += c.x * ac[m];
    if (m + 1 < N) s1 += c.y * ac[m + 1];
  }
  return s0 + s1;
}

// Radial factors of cusp-corrected and spline shells (bits as in the group
// word), out of line: few molecules have them, and inlined twice they cost
// every molecule registers.
static __device__ __noinline__ void oq_ao_special(const OqSystem* gS, int ia, int word, double r2,
                                                  double (&R)[2], double (&P)[2],
                                                  double (&L)[2]) {
  const int sh = word >> 16;
  for (int k = 0; k < 2; ++k) {
    if (word & (0x400 << k)) {
      double gv, gp, gpp;
      oq_spline_gdd(*gS, gS->s_spl[sh + k], r2, gv, gp, gpp);
      R[k] = gv;
      P[k] = 2.0 * gp;
      L[k] = 6.0 * gp + 4.0 * r2 * gpp;
    }
    if (word & (0x100 << k)) oq_cusp_vgl(*gS, ia, sqrt(r2), R[k], P[k], L[k]);
  }
}

static __device__ __noinline__ double oq_ao_special_value(const OqSystem* gS, int ia, int word,
                                                          int k, double r2, double R) {
  if (word & (0x400 << k)) {
    double gp, gpp;
    oq_spline_gdd(*gS, gS->s_spl[(word >> 16) + k], r2, R, gp, gpp);
  }
  return word & (0x100 << k) ? oq_cusp_val(*gS, ia, sqrt(r2), R) : R;
}

static __device__ __noinline__ void oq_ao_harm(const OqSystem* gS, int am, int q, double x,
                                               double y, double z, double (&Y)[4]) {
  double dY[3];
  oq_harm_table<double>(gS->harm, am, q, x, y, z, Y[0], dY);
  Y[1] = dY[0]; Y[2] = dY[1]; Y[3] = dY[2];
}

// The value alone: the gradient's powers, three more loops per monomial, are
// not formed (f and g shells, 65,536 walkers: mo_values 116 -> 90 us).
static __device__ __noinline__ double oq_ao_harm_value(const OqSystem* gS, int am, int q,
                                                       double x, double y, double z) {
  double Y, dY[3];
  oq_harm_table<double>(gS->harm, am, q, x, y, z, Y, dY);
  return Y;
}

// Occupied-orbital values at x (FP64).  gS: the full system tables, read only
// for cusp-corrected, spline and f or g shells.
template <int N, bool EXT>
__device__ __forceinline__ void oq_ao_value(const OqAo<N>& T, const OqSystem* __restrict__ gS,
                                            double x, double y, double z, double (&mv)[N]) {
  constexpr int NP = OqAo<N>::NP;
#pragma unroll
  for (int m = 0; m < N; ++m) mv[m] = 0.0;
#pragma unroll 1
  for (int ia = 0; ia < T.h->natm; ++ia) {
    const OqAoAtom& at = T.atom[ia];
    const double dx = x - at.x, dy = y - at.y, dz = z - at.z;
    const double r2 = dx * dx + dy * dy + dz * dz;
#pragma unroll 1
    for (int g = at.g0; g < at.g1; ++g) {
      const int4 G = T.group[g];
      const int am = G.x & 15, two = (G.x >> 4) & 2;
      const double2* pr = T.prim + G.z;
      double R0 = 0.0, R1 = 0.0;
      if (!two) {
#pragma unroll 2
        for (int p = 0; p < G.y; ++p) {
          const double2 t = pr[p];
          R0 += t.y * exp(-t.x * r2);
        }
      } else {
#pragma unroll 2
        for (int p = 0; p < G.y; ++p) {
          const double2 t = pr[2 * p];
          const double n1 = pr[2 * p + 1].x;
          const double e = exp(-t.x * r2);
          R0 += t.y * e;
          R1 += n1 * e;
        }
      }
      if (EXT && (G.x & 0xF00)) {
        R0 = oq_ao_special_value(gS, ia, G.x, 0, r2, R0);
        R1 = oq_ao_special_value(gS, ia, G.x, 1, r2, R1);
      }
      const double* C = T.C + G.w * NP;
#pragma unroll 1
      for (int k = 0;; ++k) {
        if (am == 0) {
          oq_ao_add<N>(C, R0, mv);
          C += NP;
        } else if (am == 1) {
          oq_ao_add3<N>(C, R0 * dx, R0 * dy, R0 * dz, mv);
          C += 3 * NP;
        } else if (!EXT || am == 2) {
          double Y[5], dY[5][3];
          oq_harm_d<double>(dx, dy, dz, Y, dY);
#pragma unroll
          for (int q = 0; q < 5; ++q) oq_ao_add<N>(C + q * NP, R0 * Y[q], mv);
          C += 5 * NP;
        } else {
          for (int q = 0; q < 2 * am + 1; ++q, C += NP) {
            oq_ao_add<N>(C, R0 * oq_ao_harm_value(gS, am, q, dx, dy, dz), mv);
          }
        }
        if (!two || k) break;
        R0 = R1;
      }
    }
  }
}

// Gradient and Laplacian of sum_m ac[m] phi_m at x (FP64): the MO coefficients
// of each AO are contracted with ac first, so an AO costs N multiply-adds
// instead of 5 N, and no orbital gradients are kept.
template <int N, bool EXT>
__device__ __forceinline__ void oq_ao_contract(const OqAo<N>& T, const OqSystem* __restrict__ gS,
                                               double x, double y, double z,
                                               const double (&ac)[N], double& gx, double& gy,
                                               double& gz, double& lp) {
  constexpr int NP = OqAo<N>::NP;
  gx = gy = gz = lp = 0.0;
#pragma unroll 1
  for (int ia = 0; ia < T.h->natm; ++ia) {
    const OqAoAtom& at = T.atom[ia];
    const double dx = x - at.x, dy = y - at.y, dz = z - at.z;
    const double r2 = dx * dx + dy * dy + dz * dz;
    double sd = 0.0;                     // the gradient's multiple of the displacement
#pragma unroll 1
    for (int g = at.g0; g < at.g1; ++g) {
      const int4 G = T.group[g];
      const int am = G.x & 15, two = (G.x >> 4) & 2;
      const double2* pr = T.prim + G.z;
      // R = sum n e, s = sum a n e, q = sum a^2 n e with e = exp(-a r^2):
      // R'/r = -2 s, R'' + 2 R'/r = 4 r^2 q - 6 s
      double R0 = 0.0, s0 = 0.0, q0 = 0.0, R1 = 0.0, s1 = 0.0, q1 = 0.0;
      if (!two) {
#pragma unroll 2
        for (int p = 0; p < G.y; ++p) {
          const double2 t = pr[p];
          const double e = t.y * exp(-t.x * r2), ae = t.x * e;
          R0 += e;
          s0 += ae;
          q0 += t.x * ae;
        }
      } else {
#pragma unroll 2
        for (int p = 0; p < G.y; ++p) {
          const double2 t = pr[2 * p];
          const double n1 = pr[2 * p + 1].x;
          const double e = exp(-t.x * r2), ae = t.x * e, aae = t.x * ae;
          R0 += t.y * e; s0 += t.y * ae; q0 += t.y * aae;
          R1 += n1 * e;  s1 += n1 * ae;  q1 += n1 * aae;
        }
      }
      double P0 = -2.0 * s0, L0 = 4.0 * r2 * q0 - 6.0 * s0;
      double P1 = -2.0 * s1, L1 = 4.0 * r2 * q1 - 6.0 * s1;
      if (EXT && (G.x & 0xF00)) {
        double R[2] = {R0, R1}, P[2] = {P0, P1}, L[2] = {L0, L1};
        oq_ao_special(gS, ia, G.x, r2, R, P, L);
        R0 = R[0]; P0 = P[0]; L0 = L[0];
        R1 = R[1]; P1 = P[1]; L1 = L[1];
      }
      const double* C = T.C + G.w * NP;
#pragma unroll 1
      for (int k = 0;; ++k) {
        if (am == 0) {
          const double c = oq_ao_dot<N>(C, ac);
          sd += c * P0;
          lp += c * L0;
          C += NP;
        } else {
          double A = 0.0, Gx = 0.0, Gy = 0.0, Gz = 0.0;
          if (am == 1) {
            Gx = oq_ao_dot<N>(C, ac);
            Gy = oq_ao_dot<N>(C + NP, ac);
            Gz = oq_ao_dot<N>(C + 2 * NP, ac);
            A = Gx * dx + Gy * dy + Gz * dz;
            C += 3 * NP;
          } else if (!EXT || am == 2) {
            double Y[5], dY[5][3];
            oq_harm_d<double>(dx, dy, dz, Y, dY);
#pragma unroll
            for (int q = 0; q < 5; ++q) {
              const double c = oq_ao_dot<N>(C + q * NP, ac);
              A += c * Y[q];
              Gx += c * dY[q][0]; Gy += c * dY[q][1]; Gz += c * dY[q][2];
            }
            C += 5 * NP;
          } else {
            for (int q = 0; q < 2 * am + 1; ++q, C += NP) {
              double Y[4];
              oq_ao_harm(gS, am, q, dx, dy, dz, Y);
              const double c = oq_ao_dot<N>(C, ac);
              A += c * Y[0];
              Gx += c * Y[1]; Gy += c * Y[2]; Gz += c * Y[3];
            }
          }
          sd += P0 * A;
          gx += R0 * Gx; gy += R0 * Gy; gz += R0 * Gz;
          lp += (L0 + 2.0 * am * P0) * A;
        }
        if (!two || k) break;
        R0 = R1; P0 = P1; L0 = L1;
      }
    }
    gx += sd * dx; gy += sd * dy; gz += sd * dz;
  }
}

// Shared-memory views of one tile.
template <int N>
struct OqTile {
  double *pos, *S, *f, *red;
  int* piv;
  __device__ OqTile(unsigned char* p, int wb) {
    pos = reinterpret_cast<double*>(p);
    S = pos + (size_t)6 * N * wb;
    f = S + (size_t)2 * N * N * wb;
    red = f + (size_t)4 * N * wb;
    piv = reinterpret_cast<int*>(red + (size_t)12 * N * wb);
  }
  // k_team's evaluation only: oq_walker_by_orbital's [2 N][N][4]
  __device__ double* orb(int wb) const { return reinterpret_cast<double*>(piv + 4 * wb); }
};

// Gauss-Jordan inversion of both N x N Slater matrices of every walker of
// the tile, in place, partial pivoting over rows (as oq_invert).  Thread
// (wl, s, c) holds column c of its spin's matrix in a[]; afterwards a[] is
// column `dst` of the inverse.  In step k the owner of column k searches the
// pivot in its own registers and publishes the column; one barrier later
// every thread eliminates its own column.  The published column alternates
// between two buffers, so one barrier per step is enough.  DET: only the
// determinant is wanted (rows below the pivot, columns right of it).  `det`
// receives the pivot of this thread's column; returns false (for all
// threads of the walker and spin) when a pivot is zero or not finite.  Every
// thread of the CTA has to call this.
template <int N, bool DET>
__device__ __forceinline__ bool oq_team_invert(double (&a)[N], const OqTile<N>& tl, int wb,
                                               int wl, int s, int c, bool active, double& det,
                                               int& dst) {
  bool ok = true;
  unsigned long long perm = 0ull;       // pivot row of each step, 4 bits each
  det = 1.0;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    double* f = tl.f + (size_t)((k & 1) * 2 + s) * N * wb + wl;
    int* pv = tl.piv + ((k & 1) * 2 + s) * wb + wl;
    if (active && c == k) {
      int piv = k;
      double best = fabs(a[k]);
#pragma unroll
      for (int i = k + 1; i < N; ++i) {
        const double v = fabs(a[i]);
        if (v > best) { best = v; piv = i; }
      }
      if (!(best > 0.0) || !isfinite(best)) piv = -1;
      double d = a[k];
#pragma unroll
      for (int i = k + 1; i < N; ++i)
        if (i == piv) { d = a[i]; a[i] = a[k]; }
      det = d;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (i != k && (!DET || i > k)) f[i * wb] = a[i];
      f[k * wb] = 1.0 / d;
      *pv = piv;
    }
    __syncthreads();
    if (active && ok) {
      const int piv = *pv;
      if (piv < 0) {
        ok = false;
      } else if (!DET || c > k) {
        perm |= (unsigned long long)piv << (4 * k);
        const double rd = f[k * wb];
        double ak = a[k];
        if (c != k) {
#pragma unroll
          for (int i = k + 1; i < N; ++i)
            if (i == piv) { const double t = a[i]; a[i] = ak; ak = t; }
        }
        const double t = c == k ? rd : ak * rd;
        if (!DET && c == k) {
#pragma unroll
          for (int i = 0; i < N; ++i) a[i] = 0.0;
        }
#pragma unroll
        for (int i = 0; i < N; ++i)
          if (i != k && (!DET || i > k)) a[i] -= f[i * wb] * t;
        a[k] = t;
      }
    }
  }
  // the row exchanges undone on the columns, last one first
  dst = c;
  if (!DET) {
#pragma unroll
    for (int k = N - 1; k >= 0; --k) {
      const int p = (int)((perm >> (4 * k)) & 15ull);
      dst = dst == k ? p : (dst == p ? k : dst);
    }
  }
  return ok;
}

// 1/sqrt(r^2 + eps) of the Coulomb terms from 1/r: to first order in eps/r^2
// (its square is below FP64 resolution) except within 1e-3 bohr.
__device__ __forceinline__ double oq_coulomb_inv(double r2, double rinv) {
  if (r2 < 1e-6) return rsqrt(r2 + OQ_EPS);
  return rinv - 0.5 * OQ_EPS * rinv * rinv * rinv;
}

// The B-spline and three-body terms of electron e (value over pairs j > e,
// gradient, Laplacian added to v), out of line as oq_ao_special.
template <int N, bool VGL>
static __device__ __noinline__ void oq_team_ext(const OqSystem* gS, const double* pos, int ps,
                                                int e, double xe, double ye, double ze,
                                                double (&v)[5]) {
  constexpr int NE = 2 * N;
  const OqSystem& S = *gS;
  double jv = 0.0, gx = 0.0, gy = 0.0, gz = 0.0, lp = 0.0;
  if (S.has_bs2)
    for (int j = VGL ? 0 : e + 1; j < NE; ++j) {
      if (j == e) continue;
      const double dx = xe - pos[(3 * j) * ps], dy = ye - pos[(3 * j + 1) * ps],
                   dz = ze - pos[(3 * j + 2) * ps];
      const double r = sqrt(dx * dx + dy * dy + dz * dz);
      const bool like = (e & 1) == (j & 1);
      const double* c = like ? S.bs2_like : S.bs2_unlike;
      const int n = like ? S.bs2_n_like : S.bs2_n_unlike;
      const double dinv = like ? S.bs2_dinv_like : S.bs2_dinv_unlike;
      if (j > e) jv += oq_bs_val<double>(c, n, dinv, S.bs2_rcut, r);
      if (VGL) {
        double up, l;
        oq_bs_vgl<double>(c, n, dinv, S.bs2_rcut, r, 1.0 / r, up, l);
        gx += up * dx; gy += up * dy; gz += up * dz; lp += l;
      }
    }
  if (S.has_bs1)
    for (int I = 0; I < S.natm; ++I) {
      const int ty = S.bs1_type[I];
      if (ty < 0) continue;
      const double dx = xe - S.nuc[I][0], dy = ye - S.nuc[I][1], dz = ze - S.nuc[I][2];
      const double r = sqrt(dx * dx + dy * dy + dz * dz);
      jv += oq_bs_val<double>(S.bs1_c[ty], S.bs1_n[ty], S.bs1_dinv[ty], S.bs1_rcut[ty], r);
      if (VGL) {
        double up, l;
        oq_bs_vgl<double>(S.bs1_c[ty], S.bs1_n[ty], S.bs1_dinv[ty], S.bs1_rcut[ty], r, 1.0 / r,
                          up, l);
        gx += up * dx; gy += up * dy; gz += up * dz; lp += l;
      }
    }
  if (S.has_j3) {
    const int nI = S.j3_nI, nE = S.j3_nE, bsz = (nI + 1) * (nI + 1) * (nE + 1);
    const double L = S.j3_L;
    for (int I = 0; I < S.natm; ++I) {
      const int ty = S.j3_type[I];
      if (ty < 0) continue;
      const double ax = xe - S.nuc[I][0], ay = ye - S.nuc[I][1], az = ze - S.nuc[I][2];
      const double r1 = sqrt(ax * ax + ay * ay + az * az);
      if (!(r1 < L)) continue;
      for (int j = VGL ? 0 : e + 1; j < NE; ++j) {
        const int blk = (e ^ j) & 1;
        if (j == e || !S.j3_on[ty][blk]) continue;
        const double xj = pos[(3 * j) * ps], yj = pos[(3 * j + 1) * ps], zj = pos[(3 * j + 2) * ps];
        const double bx = xj - S.nuc[I][0], by = yj - S.nuc[I][1], bz = zj - S.nuc[I][2];
        const double r2 = sqrt(bx * bx + by * by + bz * bz);
        if (!(r2 < L)) continue;
        const double dx = xe - xj, dy = ye - yj, dz = ze - zj;
        const double r12 = sqrt(dx * dx + dy * dy + dz * dz);
        const double* g = S.j3_gamma + (size_t)(2 * ty + blk) * bsz;
        if (!VGL) {
          jv -= oq_j3_u_n<double>(g, nI, nE, L, r12, r1, r2);
          continue;
        }
        double u1, ue, u11, uee, u1e, u;
        oq_j3_partials_n<double>(g, nI, nE, L, r12, r1, r2, u1, ue, u11, uee, u1e, &u);
        if (j > e) jv -= u;
        const double i1 = 1.0 / r1, i12 = 1.0 / r12;
        const double t1 = u1 * i1, te = ue * i12;
        gx -= t1 * ax + te * dx;
        gy -= t1 * ay + te * dy;
        gz -= t1 * az + te * dz;
        lp -= u11 + 2.0 * t1 + uee + 2.0 * te +
              2.0 * u1e * (ax * dx + ay * dy + az * dz) * (i1 * i12);
      }
    }
  }
  v[0] += jv; v[1] += gx; v[2] += gy; v[3] += gz; v[4] += lp;
}

// Jastrow value (pairs j > e), gradient and Laplacian of electron e and its
// Coulomb terms (e-e for j > e), FP64 (gto.py:1493-2254, 2406-2451).  VGL
// false: the value only.  pos is the walker's column, coordinate stride ps.
template <int N, bool VGL, bool EXT>
__device__ __forceinline__ void oq_team_pairs(const OqAo<N>& T, const OqSystem* __restrict__ gS,
                                              const double* pos, int ps, int e, double xe,
                                              double ye, double ze, double& jv, double& gx,
                                              double& gy, double& gz, double& lp, double& ee,
                                              double& en) {
  constexpr int NE = 2 * N;
  const bool has_j2 = T.h->has_j2, has_j1 = T.h->has_j1;
  if (VGL || has_j2)
    for (int j = VGL ? 0 : e + 1; j < NE; ++j) {
      if (j == e) continue;
      const double dx = xe - pos[(3 * j) * ps], dy = ye - pos[(3 * j + 1) * ps],
                   dz = ze - pos[(3 * j + 2) * ps];
      const double r2 = dx * dx + dy * dy + dz * dz;
      const double rinv = rsqrt(r2);
      if (VGL && j > e) ee += oq_coulomb_inv(r2, rinv);
      if (has_j2) {
        const double r = r2 > 0.0 ? r2 * rinv : r2;
        const double* ab = T.h->j2 + ((e ^ j) & 1) * 2;
        const double b = ab[1], q = oq_rcp(1.0 + b * r), aq = ab[0] * q;
        if (j > e) jv += aq * r;
        if (VGL) {
          const double aq2 = aq * q, up = aq2 * rinv;
          gx += up * dx; gy += up * dy; gz += up * dz;
          lp += 2.0 * up - 2.0 * b * aq2 * q;
        }
      }
    }
  if (VGL || has_j1)
    for (int I = 0; I < T.h->natm; ++I) {
      const OqAoAtom& at = T.atom[I];
      const double dx = xe - at.x, dy = ye - at.y, dz = ze - at.z;
      const double r2 = dx * dx + dy * dy + dz * dz;
      const double rinv = rsqrt(r2);
      if (VGL) en -= at.Z * oq_coulomb_inv(r2, rinv);
      if (has_j1) {
        const double r = r2 > 0.0 ? r2 * rinv : r2;
        const double b = at.j1b, q = oq_rcp(1.0 + b * r), aq = at.j1a * q;
        jv += aq * r;
        if (VGL) {
          const double aq2 = aq * q, up = aq2 * rinv;
          gx += up * dx; gy += up * dy; gz += up * dz;
          lp += 2.0 * up - 2.0 * b * aq2 * q;
        }
      }
    }
  if (EXT) {
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    oq_team_ext<N, VGL>(gS, pos, ps, e, xe, ye, ze, v);
    jv += v[0];
    gx += v[1]; gy += v[2]; gz += v[3]; lp += v[4];
  }
}

// Gradient and Laplacian at x of the orbital whose coefficients are C.
static __device__ __noinline__ void oq_orbital_vgl(const OqSystem* gS, const double* C, double x,
                                                   double y, double z, double* out) {
  double mv[1], mg[1][3], ml[1];
  oq_mo_vgl<1>(*gS, C, x, y, z, mv, mg, ml);
  out[0] = mg[0][0]; out[1] = mg[0][1]; out[2] = mg[0][2]; out[3] = ml[0];
}

// Gradient and Laplacian of log|psi| of every electron of one walker of the
// tile, orbital by orbital: a thread per (electron, orbital), then a thread
// per electron for the contraction with its inverse column and the pair
// terms, each sum in one fixed order.  See k_team for its use.  orb: [NE][N][4].
// Every thread of the CTA calls this.
template <int N, bool EXT>
static __device__ __noinline__ void oq_walker_by_orbital(const OqSystem* gS, const double* Ct,
                                                         const double* pos, const double* A,
                                                         int ps, double* orb, double* red,
                                                         double* grad, double* lap) {
  constexpr int NE = 2 * N;
  for (int t = threadIdx.x; t < NE * N; t += blockDim.x) {
    const int e = t / N, m = t - e * N;
    oq_orbital_vgl(gS, Ct + (size_t)m * gS->nbf, pos[(3 * e) * ps], pos[(3 * e + 1) * ps],
                   pos[(3 * e + 2) * ps], orb + t * 4);
  }
  __syncthreads();
  const int e = threadIdx.x;
  if (e < NE) {
    const OqSystem& S = *gS;
    const double x = pos[(3 * e) * ps], y = pos[(3 * e + 1) * ps], z = pos[(3 * e + 2) * ps];
    double gx = 0.0, gy = 0.0, gz = 0.0, lp = 0.0;
    for (int m = 0; m < N; ++m) {
      const double am = A[(size_t)(((e & 1) * N + (e >> 1)) * N + m) * ps];
      const double* o = orb + (e * N + m) * 4;
      gx += am * o[0]; gy += am * o[1]; gz += am * o[2];
      lp += am * o[3];
    }
    lp -= gx * gx + gy * gy + gz * gz;
    if (S.has_j2) {
      for (int j = 0; j < NE; ++j) {
        if (j == e) continue;
        const double dx = x - pos[(3 * j) * ps], dy = y - pos[(3 * j + 1) * ps],
                     dz = z - pos[(3 * j + 2) * ps];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        const int o = ((e & 1) == (j & 1)) ? 0 : 2;
        double upr, l;
        oq_pade_vgl(S.j2[o], S.j2[o + 1], r, upr, l);
        gx += upr * dx; gy += upr * dy; gz += upr * dz; lp += l;
      }
    }
    if (EXT && S.has_bs2) {
      for (int j = 0; j < NE; ++j) {
        if (j == e) continue;
        const double dx = x - pos[(3 * j) * ps], dy = y - pos[(3 * j + 1) * ps],
                     dz = z - pos[(3 * j + 2) * ps];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        const bool like = (e & 1) == (j & 1);
        double upr, l;
        oq_bs_vgl<double>(like ? S.bs2_like : S.bs2_unlike, like ? S.bs2_n_like : S.bs2_n_unlike,
                          like ? S.bs2_dinv_like : S.bs2_dinv_unlike, S.bs2_rcut, r, 1.0 / r,
                          upr, l);
        gx += upr * dx; gy += upr * dy; gz += upr * dz; lp += l;
      }
    }
    if (S.has_j1) {
      for (int I = 0; I < S.natm; ++I) {
        const double dx = x - S.nuc[I][0], dy = y - S.nuc[I][1], dz = z - S.nuc[I][2];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        double upr, l;
        oq_pade_vgl(S.j1a[I], S.j1b[I], r, upr, l);
        gx += upr * dx; gy += upr * dy; gz += upr * dz; lp += l;
      }
    }
    if (EXT && S.has_bs1) {
      for (int I = 0; I < S.natm; ++I) {
        const int ty = S.bs1_type[I];
        if (ty < 0) continue;
        const double dx = x - S.nuc[I][0], dy = y - S.nuc[I][1], dz = z - S.nuc[I][2];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        double upr, l;
        oq_bs_vgl<double>(S.bs1_c[ty], S.bs1_n[ty], S.bs1_dinv[ty], S.bs1_rcut[ty], r, 1.0 / r,
                          upr, l);
        gx += upr * dx; gy += upr * dy; gz += upr * dz; lp += l;
      }
    }
    if (EXT && S.has_j3)
      oq_j3_vgl_electron<double>(S, pos, (size_t)ps, NE, e, x, y, z, gx, gy, gz, lp);
    red[(size_t)(e * 6 + 4) * ps] = lp;
    orb[e * N * 4] = gx; orb[e * N * 4 + 1] = gy; orb[e * N * 4 + 2] = gz;
    if (grad) { grad[3 * e] = gx; grad[3 * e + 1] = gy; grad[3 * e + 2] = gz; }
    if (lap) lap[e] = lp;
  }
  __syncthreads();
  if (e < NE) {
    const double* o = orb + e * N * 4;
    red[(size_t)(e * 6 + 5) * ps] = o[0] * o[0] + o[1] * o[1] + o[2] * o[2];
  }
  __syncthreads();
}

// What the tile kernel computes.
enum { OQ_TEAM_EVAL = 0, OQ_TEAM_LOGPSI = 1, OQ_TEAM_REFRESH = 2 };

struct OqTeamArgs {
  const double* X;      // EVAL, LOGPSI: walkers (W, n_e, 3); REFRESH: [3 n_e][W]
  int W, wb;
  double* logpsi;       // REFRESH: log|det|
  double* grad;         // (W, n_e, 3) or null
  double* lap;          // (W, n_e) or null
  double* eparts;       // (W, 4) or null
  void* ainv;           // REFRESH: [2 N N][W] Real
  const double* Ct;     // EVAL: MO coefficients (N, nbf), for oq_walker_by_orbital
  unsigned* flags;
};

// EXT: the molecule has B-spline or three-body Jastrow terms, cusp-corrected,
// spline, f or g shells; without them that code, and the registers it takes,
// are compiled out.
//
// Full FP64 evaluation (log_trial_wavefunction, _slater_det_assemble,
// local_energy_ke; OmegaQMC/psi/gto.py:2220-2254, 728-778, 2506-2579), the
// value path, or the refresh of a sampler state's inverses.
template <int N, int MODE, typename Real, bool EXT>
__global__ void __launch_bounds__(OqTeam<N>::T, OqTeam<N>::MINB)
k_team(const OqSystem* __restrict__ gS, const unsigned char* __restrict__ ao, int ao_bytes,
       OqTeamArgs a) {
  constexpr int NE = 2 * N;
  extern __shared__ __align__(16) unsigned char smem[];
  const int wb = a.wb, W = a.W, tid = threadIdx.x;
  const OqTile<N> tl(smem + ao_bytes, wb);
  for (int i = tid; i < ao_bytes / 16; i += blockDim.x)
    reinterpret_cast<int4*>(smem)[i] = reinterpret_cast<const int4*>(ao)[i];
  const int w0 = blockIdx.x * wb;
  for (int q = tid; q < 3 * NE * wb; q += blockDim.x) {
    // positions beyond the last walker repeat it (computed, never stored)
    if (MODE == OQ_TEAM_REFRESH) {
      const int k = q / wb, j = q - k * wb;
      tl.pos[q] = a.X[(size_t)k * W + min(w0 + j, W - 1)];
    } else {
      const int j = q / (3 * NE), k = q - j * 3 * NE;
      tl.pos[k * wb + j] = a.X[(size_t)min(w0 + j, W - 1) * 3 * NE + k];
    }
  }
  __syncthreads();
  const OqAo<N> T(smem);
  const int wl = tid & (wb - 1), e = tid / wb, s = e & 1, i = e >> 1, w = w0 + wl;
  const bool active = e < NE;
  const bool live = active && w < W;
  const double* pos = tl.pos + wl;
  double* Sw = tl.S + (size_t)s * N * N * wb + wl;     // this spin's matrix of this walker
  double xe = 0.0, ye = 0.0, ze = 0.0;
  double col[N];
#pragma unroll
  for (int m = 0; m < N; ++m) col[m] = 0.0;
  if (active) {
    xe = pos[(3 * e) * wb]; ye = pos[(3 * e + 1) * wb]; ze = pos[(3 * e + 2) * wb];
    oq_ao_value<N, EXT>(T, gS, xe, ye, ze, col);
#pragma unroll
    for (int m = 0; m < N; ++m) Sw[(i * N + m) * wb] = col[m];
  }
  __syncthreads();
  if (active) {
#pragma unroll
    for (int r = 0; r < N; ++r) col[r] = Sw[(r * N + i) * wb];
  }
  double det;
  int dst;
  const bool ok = oq_team_invert<N, MODE == OQ_TEAM_LOGPSI>(col, tl, wb, wl, s, i, active, det,
                                                            dst);
  double jv = 0.0, ee = 0.0, en = 0.0, lap = 0.0, g2 = 0.0;
  if (MODE == OQ_TEAM_REFRESH) {
    if (live) {
      Real* A = reinterpret_cast<Real*>(a.ainv) + (size_t)s * N * N * W + w;
#pragma unroll
      for (int m = 0; m < N; ++m) A[(size_t)(m * N + dst) * W] = ok ? (Real)col[m] : (Real)0;
    }
  } else if (MODE == OQ_TEAM_LOGPSI) {
    double gx = 0.0, gy = 0.0, gz = 0.0;
    if (active)
      oq_team_pairs<N, false, EXT>(T, gS, pos, wb, e, xe, ye, ze, jv, gx, gy, gz, lap, ee, en);
  } else {
    // column i of the inverse to electron i's thread, through shared memory
    if (active) {
#pragma unroll
      for (int m = 0; m < N; ++m) Sw[(dst * N + m) * wb] = ok ? col[m] : 0.0;
    }
    __syncthreads();
    if (active) {
#pragma unroll
      for (int m = 0; m < N; ++m) col[m] = Sw[(i * N + m) * wb];
      double gx, gy, gz;
      oq_ao_contract<N, EXT>(T, gS, xe, ye, ze, col, gx, gy, gz, lap);
      lap -= gx * gx + gy * gy + gz * gz;
      oq_team_pairs<N, true, EXT>(T, gS, pos, wb, e, xe, ye, ze, jv, gx, gy, gz, lap, ee, en);
      g2 = gx * gx + gy * gy + gz * gz;
      if (live && a.grad) {
        double* gp = a.grad + ((size_t)w * NE + e) * 3;
        gp[0] = gx; gp[1] = gy; gp[2] = gz;
      }
      if (live && a.lap) a.lap[(size_t)w * NE + e] = lap;
    }
  }
  // sums over the electrons of a walker
  double* rd0 = tl.red + (size_t)e * 6 * wb + wl;
  if (active) {
    rd0[0] = ok ? log(fabs(det)) : -INFINITY;
    if (MODE != OQ_TEAM_REFRESH) rd0[wb] = jv;
    if (MODE == OQ_TEAM_EVAL) {
      rd0[2 * wb] = ee; rd0[3 * wb] = en; rd0[4 * wb] = lap; rd0[5 * wb] = g2;
    }
  }
  __syncthreads();
  double v[6] = {0, 0, 0, 0, 0, 0};
  constexpr int NV = MODE == OQ_TEAM_REFRESH ? 1 : (MODE == OQ_TEAM_LOGPSI ? 2 : 6);
  if (live && e == 0)
    for (int k = 0; k < NE; ++k) {
      const double* rd = tl.red + (size_t)k * 6 * wb + wl;
#pragma unroll
      for (int q = 0; q < NV; ++q) v[q] += rd[q * wb];
    }
  if (MODE == OQ_TEAM_EVAL) {
    // Next to a node of the determinant the sums of Laplacians and of squared
    // gradients, each of order 1/d^2 at distance d, cancel to the kinetic
    // energy, of order 1/d, whose last digits are then what rounding leaves:
    // FP64 determines it to some eps |grad|^2 only.  Such walkers are formed
    // again orbital by orbital, in the order of summation that this entry has
    // had since its first version, so that their energies keep reproducing what
    // it returned before; in the tile's order they move by up to 3e-9 of
    // themselves.  Neither order is the more accurate: against extended
    // precision, 720 such walkers, the mean error of the kinetic energy in eps
    // |grad|^2 is 0.70 here and 0.71 in the tile's order (H2O), 1.28 and 1.27
    // (N2), 0.99 and 0.98 ((H2O)2), most of it the inverse's.  All-electron
    // steps, whose energies were never formed in this order, go without.  A
    // tile does its walkers one after another: with one to three of them in
    // 4,097 N2 walkers 80 to 90 us, without any 54; 16,384 (H2O)2, 270 to 310
    // against 243.
    const bool close = live && e == 0 && v[5] > 2e5 * fabs(v[4] + v[5]);
    if (__syncthreads_or(close)) {
      if (active && e == 0) tl.piv[wl] = close;
      __syncthreads();
      for (int j = 0; j < wb; ++j)
        if (tl.piv[j])
          oq_walker_by_orbital<N, EXT>(
              gS, a.Ct, tl.pos + j, tl.S + j, wb, tl.orb(wb), tl.red + j,
              a.grad ? a.grad + (size_t)(w0 + j) * NE * 3 : nullptr,
              a.lap ? a.lap + (size_t)(w0 + j) * NE : nullptr);
      if (close) {
        v[4] = v[5] = 0.0;
        for (int k = 0; k < NE; ++k) {
          const double* rd = tl.red + (size_t)k * 6 * wb + wl;
          v[4] += rd[4 * wb];
          v[5] += rd[5 * wb];
        }
      }
    }
  }
  if (!live || e != 0) return;
  const bool good = v[0] > -INFINITY;
  const double lpsi = v[0] + v[1];
  a.logpsi[w] = good ? lpsi : -INFINITY;
  if (!good) atomicOr(a.flags, OQ_FLAG_SINGULAR);
  if (MODE == OQ_TEAM_EVAL) {
    const double ke = -0.5 * (v[4] + v[5]);
    if (a.eparts) {
      double* ep = a.eparts + (size_t)w * 4;
      ep[0] = v[2]; ep[1] = v[3]; ep[2] = ke; ep[3] = v[2] + v[3] + ke + T.h->e_nn;
    }
    if (good && (!isfinite(ke) || !isfinite(lpsi))) atomicOr(a.flags, OQ_FLAG_NAN);
  }
}

// ---------------------------------------------------------------------------
// All-electron Metropolis steps, the reference's move (metropolis_move_alle
// and metropolis_move_1w, OmegaQMC/vmc_gto.py:815-905): every electron is
// displaced by step * N(0, 1); a proposal with an electron-electron or
// electron-nucleus distance below 1e-4 bohr is rejected (ratio 0,
// constants.py:23); otherwise it is accepted when u < exp(2 (ln|psi'| -
// ln|psi|)), ln|psi| = log|det up| + log|det down| + J evaluated afresh in
// FP64 (inverses of the proposed Slater matrices, which become the state's
// inverses on acceptance).  Random numbers: electron e's normals from the
// Philox block (walker, step, e, 0), u from electron 0's block.
//
// The tile of k_team, kept for all steps of the launch: one thread per
// (walker, electron), the walker's state in shared memory.  A step is one
// orbital row, one share of the pair terms and one column of an inversion per
// thread instead of 2 N rows, all pairs and two inversions in local memory on
// one; the FP64 local energy of a measured step follows from what is already
// there (the mixed one has its own kernel).  Measured with a local energy
// every step, H2O, 16,384 walkers, FP64: 295 -> 69 us per step.
// ---------------------------------------------------------------------------
struct OqAlleArgs {
  double* X;               // walkers (W, n_e, 3), updated in place
  double* pos;             // the state's positions (SoA)
  void* ainv;
  double* logdet;
  int W, wb, n_steps;
  int measure_every;       // 0: no local energies
  double step;
  uint64_t seed, step_base;
  double* acc_sum;         // += accepted electron moves outside measurements, or null
  double* sums;            // as OqSweepArgs
  double* el_trace;
  double* eparts_last;
  unsigned* flags;
};

// Bytes of a tile: k_team's, the proposals and the accepted inverses, and the
// walkers' decisions.
constexpr size_t oq_alle_tile_bytes(int n, int wb) {
  return oq_team_tile_bytes(n, wb) + sizeof(double) * (size_t)wb * ((size_t)6 * n + 2 * n * n) +
         sizeof(int) * (size_t)wb;
}

template <int N, typename Real, bool EXT>
__global__ void __launch_bounds__(OqTeam<N>::T, OqTeam<N>::MINB)
k_alle(const OqSystem* __restrict__ gS, const unsigned char* __restrict__ ao, int ao_bytes,
       OqAlleArgs a) {
  constexpr int NE = 2 * N;
  extern __shared__ __align__(16) unsigned char smem[];
  const int wb = a.wb, W = a.W, tid = threadIdx.x;
  const OqTile<N> tl(smem + ao_bytes, wb);
  double* xnew = reinterpret_cast<double*>(smem + ao_bytes + oq_team_tile_bytes(N, wb));
  double* Acur = xnew + (size_t)6 * N * wb;
  int* decided = reinterpret_cast<int*>(Acur + (size_t)2 * N * N * wb);
  for (int i = tid; i < ao_bytes / 16; i += blockDim.x)
    reinterpret_cast<int4*>(smem)[i] = reinterpret_cast<const int4*>(ao)[i];
  const int w0 = blockIdx.x * wb;
  for (int q = tid; q < 3 * NE * wb; q += blockDim.x) {
    const int j = q / (3 * NE), k = q - j * 3 * NE;
    tl.pos[k * wb + j] = a.X[(size_t)min(w0 + j, W - 1) * 3 * NE + k];
  }
  Real* gA = reinterpret_cast<Real*>(a.ainv);
  for (int q = tid; q < 2 * N * N * wb; q += blockDim.x) {
    // state (s, m, j) -> tile (s, j, m): an electron's column contiguous
    const int j = q % wb, k = q / wb, s = k / (N * N), m = (k / N) % N, c = k % N;
    Acur[((s * N + c) * N + m) * wb + j] = (double)gA[(size_t)k * W + min(w0 + j, W - 1)];
  }
  __syncthreads();
  const OqAo<N> T(smem);
  const int wl = tid & (wb - 1), e = tid / wb, s = e & 1, i = e >> 1, w = w0 + wl;
  const bool active = e < NE;
  const bool live = active && w < W;
  double* pos = tl.pos + wl;
  double* pn = xnew + wl;
  double* Sw = tl.S + (size_t)s * N * N * wb + wl;
  double* Aw = Acur + (size_t)s * N * N * wb + wl;
  double* red = tl.red + (size_t)e * 6 * wb + wl;
  double x = 0.0, y = 0.0, z = 0.0;
  // the walker's ln|psi| and log|det|, held by its thread of electron 0
  double lpsi = 0.0, ld_cur = 0.0;
  int nacc = 0, meas = 0;
  double gx = 0.0, gy = 0.0, gz = 0.0, lap = 0.0, ee = 0.0, en = 0.0;
  if (active) {
    x = pos[(3 * e) * wb]; y = pos[(3 * e + 1) * wb]; z = pos[(3 * e + 2) * wb];
    double jv = 0.0;
    oq_team_pairs<N, false, EXT>(T, gS, pos, wb, e, x, y, z, jv, gx, gy, gz, lap, ee, en);
    red[0] = jv;
  }
  __syncthreads();
  if (live && e == 0) {
    ld_cur = a.logdet[w];
    double J = 0.0;
    for (int k = 0; k < NE; ++k) J += tl.red[(size_t)k * 6 * wb + wl];
    lpsi = ld_cur + J;
  }
  const int n_meas = a.measure_every > 0 ? a.n_steps / a.measure_every : 0;
  for (int t = 0; t < a.n_steps; ++t) {
    double nx = 0.0, ny = 0.0, nz = 0.0, u = 0.0;
    if (active) {
      double n3[3];
      oq_move_randoms(a.seed, (uint32_t)w, (uint32_t)(a.step_base + t), (uint32_t)e, n3, u);
      nx = x + a.step * n3[0];
      ny = y + a.step * n3[1];
      nz = z + a.step * n3[2];
      pn[(3 * e) * wb] = nx; pn[(3 * e + 1) * wb] = ny; pn[(3 * e + 2) * wb] = nz;
    }
    double col[N];
#pragma unroll
    for (int m = 0; m < N; ++m) col[m] = 0.0;
    if (active) {
      oq_ao_value<N, EXT>(T, gS, nx, ny, nz, col);
#pragma unroll
      for (int m = 0; m < N; ++m) Sw[(i * N + m) * wb] = col[m];
    }
    __syncthreads();
    if (active) {
#pragma unroll
      for (int r = 0; r < N; ++r) col[r] = Sw[(r * N + i) * wb];
    }
    double det;
    int dst;
    const bool ok = oq_team_invert<N, false>(col, tl, wb, wl, s, i, active, det, dst);
    if (active) {
      bool valid = true;
      for (int j = e + 1; j < NE; ++j) {
        const double dx = nx - pn[(3 * j) * wb], dy = ny - pn[(3 * j + 1) * wb],
                     dz = nz - pn[(3 * j + 2) * wb];
        valid = valid && (dx * dx + dy * dy + dz * dz >= 1e-8);
      }
      for (int I = 0; I < T.h->natm; ++I) {
        const double dx = nx - T.atom[I].x, dy = ny - T.atom[I].y, dz = nz - T.atom[I].z;
        valid = valid && (dx * dx + dy * dy + dz * dz >= 1e-8);
      }
      double jv = 0.0;
      oq_team_pairs<N, false, EXT>(T, gS, pn, wb, e, nx, ny, nz, jv, gx, gy, gz, lap, ee, en);
      red[0] = log(fabs(det));
      red[wb] = jv;
      red[2 * wb] = valid && ok ? 1.0 : 0.0;
    }
    __syncthreads();
    if (active && e == 0) {
      double ld = 0.0, J = 0.0, good = 1.0;
      for (int k = 0; k < NE; ++k) {
        const double* rd = tl.red + (size_t)k * 6 * wb + wl;
        ld += rd[0];
        J += rd[wb];
        good *= rd[2 * wb];
      }
      const double lpn = ld + J;
      bool acc = live && good != 0.0;
      if (acc && !isfinite(lpn)) {
        atomicOr(a.flags, OQ_FLAG_NAN);
        acc = false;
      }
      // an old state with psi = 0 (log -inf) accepts any finite proposal
      acc = acc && (!isfinite(lpsi) || log(u) < 2.0 * (lpn - lpsi));
      if (acc) {
        ++nacc;
        lpsi = lpn;
        ld_cur = ld;
      }
      decided[wl] = acc;
    }
    __syncthreads();
    if (active && decided[wl]) {
      x = nx; y = ny; z = nz;
      pos[(3 * e) * wb] = x; pos[(3 * e + 1) * wb] = y; pos[(3 * e + 2) * wb] = z;
#pragma unroll
      for (int m = 0; m < N; ++m) Aw[(dst * N + m) * wb] = col[m];
    }
    if (meas == n_meas || (t + 1) % a.measure_every != 0) continue;
    __syncthreads();
    if (active) {
#pragma unroll
      for (int m = 0; m < N; ++m) col[m] = Aw[(i * N + m) * wb];
      double jv = 0.0;
      ee = en = 0.0;
      oq_ao_contract<N, EXT>(T, gS, x, y, z, col, gx, gy, gz, lap);
      lap -= gx * gx + gy * gy + gz * gz;
      oq_team_pairs<N, true, EXT>(T, gS, pos, wb, e, x, y, z, jv, gx, gy, gz, lap, ee, en);
      red[0] = ee; red[wb] = en; red[2 * wb] = lap;
      red[3 * wb] = gx * gx + gy * gy + gz * gz;
    }
    __syncthreads();
    if (e == 0) {
      // whole warps reach this when wb is 32 or more; with smaller tiles the
      // walkers of electron 0 are the first wb threads of warp 0
      double v[4] = {0.0, 0.0, 0.0, 0.0};
      for (int k = 0; k < NE; ++k) {
        const double* rd = tl.red + (size_t)k * 6 * wb + wl;
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] += rd[q * wb];
      }
      const double ke = -0.5 * (v[2] + v[3]), el = v[0] + v[1] + ke + T.h->e_nn;
      const bool fine = live && isfinite(el);
      if (live) {
        if (a.el_trace) a.el_trace[(size_t)meas * W + w] = el;
        if (a.eparts_last && meas == n_meas - 1) {
          double* ep = a.eparts_last + (size_t)w * 4;
          ep[0] = v[0]; ep[1] = v[1]; ep[2] = ke; ep[3] = el;
        }
        if (!fine) atomicOr(a.flags, OQ_FLAG_NAN);
      }
      double vals[7] = {fine ? v[0] : 0.0, fine ? v[1] : 0.0, fine ? ke : 0.0, fine ? el : 0.0,
                        fine ? el * el : 0.0, live ? (double)(nacc * NE) : 0.0, fine ? 1.0 : 0.0};
      const int span = wb < 32 ? wb : 32;
      const unsigned mask = span == 32 ? 0xffffffffu : (1u << span) - 1u;
#pragma unroll
      for (int k = 0; k < 7; ++k)
        for (int o = span >> 1; o > 0; o >>= 1) vals[k] += __shfl_xor_sync(mask, vals[k], o);
      if ((wl & 31) == 0) {
        double* sm = a.sums + (size_t)meas * OQ_NSUM;
#pragma unroll
        for (int k = 0; k < 7; ++k) atomicAdd(sm + k, vals[k]);
      }
    }
    nacc = 0;
    ++meas;
    __syncthreads();         // the sums are read before the next step's are written
  }
  __syncthreads();
  for (int q = tid; q < 3 * NE * wb; q += blockDim.x) {
    const int j = q / (3 * NE), k = q - j * 3 * NE;
    if (w0 + j < W) a.X[(size_t)(w0 + j) * 3 * NE + k] = tl.pos[k * wb + j];
  }
  for (int q = tid; q < 3 * NE * wb; q += blockDim.x) {
    const int k = q / wb, j = q - k * wb;
    if (w0 + j < W) a.pos[(size_t)k * W + w0 + j] = tl.pos[q];
  }
  for (int q = tid; q < 2 * N * N * wb; q += blockDim.x) {
    const int j = q % wb, k = q / wb, sp = k / (N * N), m = (k / N) % N, c = k % N;
    if (w0 + j < W) gA[(size_t)k * W + w0 + j] = (Real)Acur[((sp * N + c) * N + m) * wb + j];
  }
  if (e == 0) {
    if (live) a.logdet[w] = ld_cur;
    if (a.acc_sum) {
      // one addition per warp: one per walker, all to one address, took most of
      // a mixed step of many small walkers (H2, 65,536: 137 us)
      const int span = wb < 32 ? wb : 32;
      const unsigned mask = span == 32 ? 0xffffffffu : (1u << span) - 1u;
      for (int o = span >> 1; o > 0; o >>= 1) nacc += __shfl_xor_sync(mask, nacc, o);
      if ((wl & 31) == 0 && nacc) atomicAdd(a.acc_sum, (double)(nacc * NE));
    }
  }
}

// Occupied MO values per (walker, electron): out[(w*n_e + e)*N + m]
// (get_psi_mo, OmegaQMC/psi/gto.py:1058-1070).  One thread per electron.
template <int N, bool EXT>
__global__ void __launch_bounds__(128)
k_mo_values(const OqSystem* __restrict__ gS, const unsigned char* __restrict__ ao, int ao_bytes,
            const double* __restrict__ X, int W, double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem[];
  for (int i = threadIdx.x; i < ao_bytes / 16; i += blockDim.x)
    reinterpret_cast<int4*>(smem)[i] = reinterpret_cast<const int4*>(ao)[i];
  __syncthreads();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)W * 2 * N) return;
  const double* xp = X + 3 * t;
  double mv[N];
  oq_ao_value<N, EXT>(OqAo<N>(smem), gS, xp[0], xp[1], xp[2], mv);
#pragma unroll
  for (int m = 0; m < N; ++m) out[t * N + m] = mv[m];
}
