// Drift-diffusion (generalized) Metropolis on the device, FP64, all steps of a
// call in one launch (generalized_metropolis.py:46-219).
//
// The reference's chain, kept as it is so that replayed draws give its chains:
// every proposal starts from the walkers' positions at the start of the call
// (move() clones walkers.pos, which is written back only after the last step)
// with one electron e moved by step * drift_i(e) + eta, eta ~ N(0, sqrt(step) I);
// the transition kernel is exp(-|x_f - x_i - step drift_i| / (2 step)) with the
// norm (not its square) of the whole walker vector; zero densities become
// 1e-16 after the drift is taken, so a proposal whose density is zero (or
// underflows) has a NaN drift there and is rejected; accept when
// min(1, T_if rho_f / (T_fi rho_i)) - u >= 0.
//
// Because each proposal differs from the start positions in one electron only,
// what the gradients need of the start positions is computed once per call; a
// step evaluates the moved electron's MO row, the determinants of its spin with
// that row replaced, and the Jastrow terms of its pairs. psi and its electron
// gradient at the proposal are the full Jacobi-formula values
// (slater_jastrow.py:346-447), not an approximation.
#include <cuda_runtime.h>
#include <stdint.h>

#include "qmc_grad.cuh"
#include "qmc_host.cuh"
#include "qmc_rng.cuh"

namespace qmc {

// A walker's nslot threads share its work: the AO groups of the moved electron
// (partial MO rows, partial gradients), the electrons' pairs and gradients.
// FP64 pipe bound, so counted in FP64 instructions (H2O cc-pVDZ
// single_double(4,4), about 1,700 per step instead of 14,000 of per-determinant
// factorisations and component-wise AO gradients). Excitation mode: with A^-1
// and X = A^-1 V of the start, a proposal of electron l is a rank-one change,
//   r = phi'^T A^-1 (det' / det = r_l),  X' = X + A^-1 e_l (phi'_virt - phi' X) / r_l,
// from the start each time, so nothing accumulates over the steps; and with
//   Z_i[l] = sum_k A^-1(k, l) grad MO_k(r_i),
//   m_i[v] = grad MO_virt,v(r_i) - sum_j X(j, v) grad MO_j(r_i)
// of the start the determinant gradient of every electron that did not move is
//   Sigma (Z_i[i] - q r_i Z_i[l]) + sum_v (m_i[v] - q t_v Z_i[l]) f_v(i),  q = 1 / r_l
// (without the l terms for the other spin), f_v(i) = sum_k A'^-1(k, i) F(k, v),
// F = d Sigma / d X (qmc_grad.cuh); the moved electron's comes from one pass over
// its AOs. Explicit mode (CAS), and a proposal with a large excitation ratio
// (kGradRatio), refactor the moved spin's determinants. A spin that has such a ratio at the
// start, or a ground determinant of zero, has no use of A^-1 and X there: its
// determinants are summed one by one at the start and at every proposal, whichever
// electron moves.
struct DriftShape {
  int nwb, nslot, nthreads, ncol;
  int64_t o_ecol, o_fix;  // W's column exponents (< 0: W is not in limbs), the threads' AO limbs
  int64_t smem, o_hot;  // o_hot < 0: the hot arrays too are in the scratch
  // per walker, in doubles. Hot (shared memory): start positions, the two drifts
  // (accepted and proposed), Jastrow gradient, the moved electron's MO row, its
  // partial rows, r, t, X', F of both spins, the proposal's determinants, G of
  // the moved electron, partial sums, scalars
  int xs, dr, gj, phi, part, r, t, xp, f, fs, dvf, g, red, val, hot;  // fs: a spin's F
  // cold (scratch): MO values and gradients, LU | X, Z | m, A^-1 by columns,
  // determinants, Jastrow of the start, pivots, work of the explicit sums, cofactors of the
  // start's determinants (of a spin that sums them, [determinant][row][column])
  int ma, mg, lx, zm, inv, dv0, jg0, ju, jen, piv, lu, ginv, gx, cof, cofs, cold;  // cofs: a spin's
};
// scalars: Sigma, q, det A of the start's spins (1 where the spin sums its determinants),
// whether the moved spin sums them, the accepted drift's half, the accepted electron and its
// position, the start's spins that sum their determinants, the moved electron
enum { DV_SIGMA = 0, DV_Q = 1, DV_DET = 2, DV_FLAG = 4, DV_CUR = 5, DV_EACC = 6, DV_XACC = 7,
       DV_START = 10, DV_MOVED = 12, DV_N = 13 };
constexpr int kDriftRed = 6;  // partial sums per slot: du, a1, a2, the moved electron's grad U

// Whether a spin's sums at a proposal that leaves its rows alone take the start's cofactors
// from the scratch (excitation mode, few enough for a warp's lanes).
__host__ __device__ inline bool drift_cofactors(const qmc_wf_desc& d, int s) {
  const int n = s ? d.ndown : d.nup;
  return d.det_mode == QMC_DET_EXCITATION && n <= kSumN && d.ndet[s] <= 32;
}

// fixed: W as limbs after the start rows, and slots for the AOs'; else W itself (the least
// shared memory)
static DriftShape drift_shape(const qmc_wf_desc& d, int nwb, int nslot, bool in_smem,
                              bool fixed = true) {
  DriftShape s;
  s.nwb = nwb;
  s.nslot = nslot;
  s.nthreads = ((nwb * nslot + 31) / 32) * 32;
  s.ncol = round_up(d.nmo_used, 8);
  const int ne = d.nelec, nmu = d.nmo_used, nmax = d.nup > d.ndown ? d.nup : d.ndown;
  const bool ex = d.det_mode == QMC_DET_EXPLICIT;
  const int v0 = ex ? 0 : d.max_orb[0] - d.nup, v1 = ex ? 0 : d.max_orb[1] - d.ndown;
  const int nv = v0 > v1 ? v0 : v1, nd = d.ndet[0] + d.ndet[1];
  int o = 0;
  auto take = [&](int n) {
    const int r = o;
    o += n;
    return r;
  };
  s.xs = take(3 * ne);
  s.dr = take(6 * ne);
  s.gj = take(3 * ne);
  s.phi = take(nmu);
  s.part = take(nslot * (nmu > 3 ? nmu : 3));
  s.r = take(nmax);
  s.t = take(nv);
  s.xp = take(nmax * nv);
  s.fs = nmax * nv;
  s.f = take(2 * s.fs);
  s.dvf = take(d.ndet[0] > d.ndet[1] ? d.ndet[0] : d.ndet[1]);
  s.g = take(nmu);
  s.red = take(nslot * kDriftRed);
  s.val = take(DV_N);
  s.hot = o;
  o = 0;
  s.ma = take(ne * nmu);
  s.mg = take(3 * ne * nmu);
  s.lx = take(ex ? 0 : ne * nmu);
  s.zm = take(ex ? 0 : 3 * ne * nmu);
  s.inv = take(ex ? 0 : ne * nmax);
  s.dv0 = take(nd);
  s.jg0 = take(3 * ne);
  s.ju = take(ne);
  s.jen = take(ne);
  s.piv = take(ne);
  s.lu = take(2 * nmax * nmax);
  s.ginv = take(2 * nmax * nmax);
  s.gx = take(ne * nmu);
  s.cofs = 0;
  for (int q = 0; q < 2; ++q) {
    const int n = q ? d.ndown : d.nup, m = drift_cofactors(d, q) ? d.ndet[q] * n * n : 0;
    s.cofs = m > s.cofs ? m : s.cofs;
  }
  s.cof = take(2 * s.cofs);
  s.cold = o;
  s.smem = (tables_smem_bytes<double>(d, s.ncol) + 15) & ~int64_t(15);
  s.o_ecol = -1;
  s.o_fix = s.smem;
  if (fixed) {
    s.o_ecol = s.smem;
    s.o_fix = s.o_ecol + align8((int64_t)s.ncol * 4);
    s.smem = (s.o_fix + (int64_t)s.nthreads * kFixAOs * 8 + 15) & ~int64_t(15);
  }
  s.o_hot = -1;
  if (in_smem) {
    s.o_hot = s.smem;
    s.smem += (int64_t)s.hot * nwb * 8;
  }
  return s;
}

struct DriftWork {  // one thread's walker: hot and cold arrays
  double* hp;
  int64_t hs;
  double* cp;
  int64_t cs;
  __device__ __forceinline__ double& H(int i) const { return hp[(int64_t)i * hs]; }
  __device__ __forceinline__ double& C(int i) const { return cp[(int64_t)i * cs]; }
};

// Electron-electron Pade pair at the difference dx: u = w0 r / (1 + w r), and
// returns the factor c of its gradient, c dx = w0 / (1 + w r)^2 dx / r.
__device__ __forceinline__ double pade_pair(double w0, double w, double dx, double dy, double dz,
                                            double& u) {
  const double r = psqrt(dx * dx + dy * dy + dz * dz);
  const double iu = prcp(fma(w, r, 1.0)), q = w0 * iu;
  u = q * r;
  return q * iu * prcp(r);
}

// One thread per (walker, spin): the explicit determinants of spin s from
// the start rows (electron er's row from `phi`; er < 0: none) to dst, and
// G(i, j) = sum_u coef_u det_u A_u^-T into the spin's rows of gx with coef_u
// from the other spin's determinants at oth (oth < 0: determinants only).
__device__ __noinline__ void drift_explicit(const qmc_wf_desc& d, const DriftShape& S,
                                      const DriftWork& k, int s, int er, double* dst, int64_t ds,
                                      const double* oth, int64_t os) {
  const int n = s ? d.ndown : d.nup, r0 = s ? d.nup : 0, nmu = d.nmo_used;
  const int nmax = d.nup > d.ndown ? d.nup : d.ndown;
  const MView<double> LU{k.cp + (int64_t)(S.lu + s * nmax * nmax) * k.cs, (int64_t)nmax * k.cs, k.cs};
  const MView<double> V{k.cp + (int64_t)(S.ginv + s * nmax * nmax) * k.cs, (int64_t)nmax * k.cs, k.cs};
  int piv[QMC_MAX_NSPIN], cols[QMC_MAX_NSPIN];
  if (oth)
    for (int i = 0; i < n * nmu; ++i) k.C(S.gx + r0 * nmu + i) = 0.0;
  for (int u = 0; u < d.ndet[s]; ++u) {
    if (n == 0) {
      dst[u * ds] = 1.0;
      continue;
    }
    det_columns(d, s, u, cols);
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j) {
        const int c = cols[j];
        LU(i, j) = r0 + i == er ? k.H(S.phi + c) : k.C(S.ma + (r0 + i) * nmu + c);
      }
    const double det = lu_factor<double>(LU, n, piv);
    dst[u * ds] = det;
    if (!oth) continue;
    double coef = 0.0;
    for (int c = 0; c < d.ncfg; ++c)
      if (__ldg(d.cfg_det[s] + c) == u)
        coef = fma(__ldg(d.ci_weight + c), oth[__ldg(d.cfg_det[1 - s] + c) * os], coef);
    if (coef == 0.0) continue;
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j) V(i, j) = i == j ? 1.0 : 0.0;
    lu_solve<double>(LU, n, piv, V.c(), V, n);
    for (int j = 0; j < n; ++j) {
      const int c = cols[j];
      for (int i = 0; i < n; ++i) {
        double& g = k.C(S.gx + (r0 + i) * nmu + c);
        g = fma(coef * det, V(j, i), g);
      }
    }
  }
}

// A lane's determinant for the sums of a few walkers' spins (start_sums and below). Rolled,
// in local memory, where sum_warp's is unrolled in registers: a walker in some hundred
// sums, so what counts here is what the code costs the others (registers around the call,
// instruction cache: H2O, 8192 walkers x 50 steps without any sum, 5.05 -> 4.71 ms), and the time of one
// sum is the same (it waits for the FP64 pipe, which the block's other warps and the SM's other block hold).
struct DetSum {
  double a[kSumN * kSumN], det;    // factors, 1 / U_kk on the diagonal
  int perm[kSumN], cols[kSumN];    // the row of A that row k of the factors came from

  // Factors the columns of unique determinant u of n electrons; row(i, c): MO c of the
  // spin's electron i.
  template <typename Row>
  __device__ __forceinline__ void factor(const qmc_wf_desc& d, int s, int n, int u, const Row& row) {
    det_columns(d, s, u, cols);
    double v[kSumN * kSumN];  // all loads in flight together
#pragma unroll
    for (int i = 0; i < kSumN; ++i)
#pragma unroll
      for (int j = 0; j < kSumN; ++j) v[i * kSumN + j] = i < n && j < n ? row(i, cols[j]) : 0.0;
#pragma unroll
    for (int i = 0; i < kSumN * kSumN; ++i) a[i] = v[i];
    det = 1.0;
#pragma unroll 1
    for (int k = 0; k < n; ++k) perm[k] = k;
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
      int p = k;
      double amax = fabs(a[k * kSumN + k]);
#pragma unroll 1
      for (int i = k + 1; i < n; ++i) {
        const double x = fabs(a[i * kSumN + k]);
        if (x > amax) {
          amax = x;
          p = i;
        }
      }
      if (p != k) {
        det = -det;
        const int q = perm[k];
        perm[k] = perm[p];
        perm[p] = q;
#pragma unroll 1
        for (int j = 0; j < n; ++j) {
          const double x = a[k * kSumN + j];
          a[k * kSumN + j] = a[p * kSumN + j];
          a[p * kSumN + j] = x;
        }
      }
      const double akk = a[k * kSumN + k];
      det *= akk;
      const double inv = akk != 0.0 ? prcp(akk) : 0.0;
      a[k * kSumN + k] = inv;
#pragma unroll 1
      for (int i = k + 1; i < n; ++i) {
        const double l = a[i * kSumN + k] * inv;
        a[i * kSumN + k] = l;
#pragma unroll 1
        for (int j = k + 1; j < n; ++j)
          a[i * kSumN + j] = fma(-l, a[k * kSumN + j], a[i * kSumN + j]);
      }
    }
  }
  // A x = b for b in the factors' row order
  __device__ __forceinline__ void solve(double* x, int n) const {
#pragma unroll 1
    for (int i = 1; i < n; ++i) {
      double v = x[i];
#pragma unroll 1
      for (int k = 0; k < i; ++k) v = fma(-a[i * kSumN + k], x[k], v);
      x[i] = v;
    }
#pragma unroll 1
    for (int i = n - 1; i >= 0; --i) {
      double v = x[i];
#pragma unroll 1
      for (int k = i + 1; k < n; ++k) v = fma(-a[i * kSumN + k], x[k], v);
      x[i] = v * a[i * kSumN + i];
    }
  }
  __device__ __forceinline__ void unit(int col, double* x, int n) const {  // column of A^-1
#pragma unroll 1
    for (int i = 0; i < n; ++i) x[i] = perm[i] == col ? 1.0 : 0.0;
    solve(x, n);
  }
};

// The same by a warp for a spin of n <= kSumN electrons (dst: null where the
// determinants are there already; ADJ: with G; cof: keeps det_u A_u^-T where the shape has
// room for it).
template <bool ADJ>
__device__ __noinline__ void drift_sum_warp(const qmc_wf_desc& d, const DriftShape& S,
                                            const DriftWork& k, int s, int n, int er, double* dst,
                                            int64_t ds, const double* oth, int64_t os, bool cof) {
  const int r0 = s ? d.nup : 0, nmu = d.nmo_used, nd = d.ndet[s];
  for (int u0 = 0; u0 < nd; u0 += 32) {
    const SumLanes l = sum_lanes(nd, n, u0);
    DetSum D;
    if (l.u < nd) {
      D.factor(d, s, n, l.u, [&](int i, int c) {
        return r0 + i == er ? k.H(S.phi + c) : k.C(S.ma + (r0 + i) * nmu + c);
      });
      if (dst && l.g == 0) dst[l.u * ds] = D.det;
    }
    if (!ADJ) continue;
    double coef = 0.0;
    sum_configs(d, s, l.u, [&](int v, double& a, double&) { a = oth[v * os]; },
                [&](double w, double a, double) { coef = fma(w, a, coef); });
    const bool on = l.u < nd && (cof || coef != 0.0);  // of weight zero: adds nothing
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += l.groups) {  // row i of A_u^-T: column i of A_u^-1
      const int i = i0 + l.g;
      double y[kSumN];
      if (on && i < n) {
        D.unit(i, y, n);
#pragma unroll 1
        for (int j = 0; j < n; ++j) {
          const double c = y[j] * D.det;
          if (cof) k.C(S.cof + s * S.cofs + (l.u * n + i) * n + j) = c;
          y[j] = coef * c;
        }
      }
      sum_columns<0>(l, D.cols, y, n, on && coef != 0.0, nd, i0, nmu, u0 == 0,
                     [&](int i, int c) -> double& { return k.C(S.gx + (r0 + i) * nmu + c); });
    }
  }
}

// G of a spin whose rows are the start's, from its cofactors there.
__device__ __noinline__ void drift_cof_warp(const qmc_wf_desc& d, const DriftShape& S,
                                            const DriftWork& k, int s, int n, const double* oth,
                                            int64_t os) {
  const int r0 = s ? d.nup : 0, nmu = d.nmo_used, nd = d.ndet[s];
  const SumLanes l = sum_lanes(nd, n, 0);
  int cols[kSumN];
  if (l.u < nd) det_columns(d, s, l.u, cols);
  double coef = 0.0;
  sum_configs(d, s, l.u, [&](int v, double& a, double&) { a = oth[v * os]; },
              [&](double w, double a, double) { coef = fma(w, a, coef); });
  const bool on = l.u < nd && coef != 0.0;
#pragma unroll 1
  for (int i0 = 0; i0 < n; i0 += l.groups) {
    const int i = i0 + l.g;
    double y[kSumN];
#pragma unroll
    for (int j = 0; j < kSumN; ++j)
      y[j] = on && i < n && j < n ? coef * k.C(S.cof + s * S.cofs + (l.u * n + i) * n + j) : 0.0;
    sum_columns<0>(l, cols, y, n, on, nd, i0, nmu, true,
                   [&](int i, int c) -> double& { return k.C(S.gx + (r0 + i) * nmu + c); });
  }
}

// Excitation mode: F(i, v) = d Sigma / d X of spin s at H(S.f + s nmax nv + i nv + v)
// from X and the other spin's relative determinants.
__device__ inline void drift_adjoint(const qmc_wf_desc& d, const DriftShape& S,
                                     const DriftWork& k, int s, CView<double> X, const double* oth,
                                     int64_t os) {
  const int n = s ? d.ndown : d.nup, nv = d.max_orb[s] - n;
  if (nv <= 0) return;
  const int f0 = S.f + s * S.fs;
  for (int i = 0; i < n * nv; ++i) k.H(f0 + i) = 0.0;
  for (int c = 0; c < d.ncfg; ++c) {
    const int* e = d.det_table[s] + 5 * __ldg(d.cfg_det[s] + c);
    const int ord = __ldg(e);
    if (ord == 0) continue;
    const double cd = __ldg(d.ci_weight + c) * oth[__ldg(d.cfg_det[1 - s] + c) * os];
    const int i0 = __ldg(e + 1);
    if (ord == 1) {
      k.H(f0 + i0) += cd;
    } else {  // x = X0 X3 - X1 X2
      const int i1 = __ldg(e + 2), i2 = __ldg(e + 3), i3 = __ldg(e + 4);
      const double x0 = X(i0 / nv, i0 % nv), x1 = X(i1 / nv, i1 % nv), x2 = X(i2 / nv, i2 % nv),
                   x3 = X(i3 / nv, i3 % nv);
      k.H(f0 + i0) = fma(cd, x3, k.H(f0 + i0));
      k.H(f0 + i3) = fma(cd, x0, k.H(f0 + i3));
      k.H(f0 + i1) = fma(-cd, x2, k.H(f0 + i1));
      k.H(f0 + i2) = fma(-cd, x1, k.H(f0 + i2));
    }
  }
}

// MO values and gradients of electron e at the start positions (eight columns
// at a time), and its Jastrow terms.
__device__ inline void drift_start_rows(const qmc_wf_desc& d, const Tables<double>& t,
                                        const DriftShape& S, const DriftWork& k, int e) {
  const int nmu = d.nmo_used, ne = d.nelec;
  const double x = k.H(S.xs + 3 * e), y = k.H(S.xs + 3 * e + 1), z = k.H(S.xs + 3 * e + 2);
  for (int j0 = 0; j0 < nmu; j0 += 8) {
    double m[4][8];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) m[q][jj] = 0.0;
    auto acc = [&](int a, const AOVal<double>& o) {
      double wv[8];
      load_w<8>(t.W + (int64_t)a * t.ncol + j0, wv);
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        m[0][jj] = fma(o.v, wv[jj], m[0][jj]);
        m[1][jj] = fma(o.gx, wv[jj], m[1][jj]);
        m[2][jj] = fma(o.gy, wv[jj], m[2][jj]);
        m[3][jj] = fma(o.gz, wv[jj], m[3][jj]);
      }
    };
    for_each_ao_ep<double, true, decltype(acc), false>(t, XP<double>{x, 0.0}, XP<double>{y, 0.0},
                                                       XP<double>{z, 0.0}, acc);
#pragma unroll
    for (int jj = 0; jj < 8; ++jj)
      if (j0 + jj < nmu) {
        k.C(S.ma + e * nmu + j0 + jj) = m[0][jj];
        for (int q = 0; q < 3; ++q) k.C(S.mg + (3 * e + q) * nmu + j0 + jj) = m[q + 1][jj];
      }
  }
  double u = 0.0, g[3] = {0.0, 0.0, 0.0}, uen = 0.0;
  if (d.use_jastrow_en) {
    const EnTerms en = en_terms(d, x, y, z);
    u = uen = en.u;
    for (int q = 0; q < 3; ++q) g[q] = en.g[q];
  }
  if (d.use_jastrow) {
    const double w = __ldg(d.jastrow_w);
    for (int j = 0; j < ne; ++j) {
      if (j == e) continue;
      const double dx = x - k.H(S.xs + 3 * j), dy = y - k.H(S.xs + 3 * j + 1),
                   dz = z - k.H(S.xs + 3 * j + 2);
      double uj;
      const double c = pade_pair(same_spin(d, e, j) ? 0.25 : 0.5, w, dx, dy, dz, uj);
      if (j > e) u += uj;
      g[0] = fma(c, dx, g[0]);
      g[1] = fma(c, dy, g[1]);
      g[2] = fma(c, dz, g[2]);
    }
  }
  k.C(S.ju + e) = u;
  k.C(S.jen + e) = uen;
  for (int q = 0; q < 3; ++q) k.C(S.jg0 + 3 * e + q) = g[q];
}

template <bool FIXED>
__global__ void __launch_bounds__(kGradThreads)
    drift_kernel(const __grid_constant__ qmc_wf_desc d, const __grid_constant__ qmc_drift_args a,
                 double* __restrict__ scr, int64_t ss, double sd,
                 const __grid_constant__ DriftShape S) {
  extern __shared__ __align__(16) unsigned char smem[];
  const Tables<double> t = load_tables<double>(d, d.nmo_used, S.ncol, smem);
  int* const ecol = FIXED ? reinterpret_cast<int*>(smem + S.o_ecol) : nullptr;
  int2* const fix = FIXED ? reinterpret_cast<int2*>(smem + S.o_fix) + threadIdx.x : nullptr;
  const int tid = threadIdx.x, slot = tid / S.nwb, wl = tid - slot * S.nwb, ns = S.nslot;
  const int64_t nw = a.nwalkers, w = (int64_t)blockIdx.x * S.nwb + wl;
  const bool on = slot < ns, live = on && w < nw;
  const int64_t ws = w < nw ? w : nw - 1;  // walkers past the last repeat it, storing nothing
  DriftWork k;
  if (S.o_hot >= 0) {
    k.hp = reinterpret_cast<double*>(smem + S.o_hot) + wl;
    k.hs = S.nwb;
  } else {
    k.hp = scr + (int64_t)S.cold * ss + w;
    k.hs = ss;
  }
  k.cp = scr + w;
  k.cs = ss;
  const int ne = d.nelec, nmu = d.nmo_used, nc = 3 * ne;
  const int nmax = d.nup > d.ndown ? d.nup : d.ndown;
  const bool ex = d.det_mode == QMC_DET_EXPLICIT;
  const double wj = d.use_jastrow ? __ldg(d.jastrow_w) : 0.0, step = a.step_size;
  const int spin = slot & 1;  // of the determinant phases (slots 0 and 1)
  auto nof = [&](int s) { return s ? d.ndown : d.nup; };
  auto r0of = [&](int s) { return s ? d.nup : 0; };
  auto nvof = [&](int s) { return ex ? 0 : d.max_orb[s] - nof(s); };
  auto f0of = [&](int s) { return S.f + s * S.fs; };
  auto dv0 = [&](int s) { return k.cp + (int64_t)(S.dv0 + (s ? d.ndet[0] : 0)) * k.cs; };
  // X of the start: the virtual columns beside the LU
  auto x0 = [&](int s) {
    return CView<double>{k.cp + ((int64_t)S.lx + r0of(s) * nmu + nof(s)) * k.cs,
                         (int64_t)nmu * k.cs, k.cs};
  };
  auto view = [&](int q) {  // of the block's walker q
    DriftWork kq = k;
    kq.hp += q - wl;
    kq.cp += q - wl;
    return kq;
  };
  // the start's spins that sum their determinants: f(view, spin)
  auto start_sums = [&](const auto& f) {
    sum_tasks(
        2 * S.nwb,
        [&](int ch) {
          const int s = ch / S.nwb;
          return nof(s) <= kSumN && view(ch - s * S.nwb).H(S.val + DV_START + s) != 0.0;
        },
        [&](int ch) {
          const int s = ch / S.nwb;
          f(view(ch - s * S.nwb), s);
        });
  };
  auto electron = [&](const DriftWork& kq) { return (int)kq.H(S.val + DV_MOVED); };  // moved
  auto dets = [&](const DriftWork& kq, int s) {  // the start's determinants of spin s
    return kq.cp + (int64_t)(S.dv0 + (s ? d.ndet[0] : 0)) * kq.cs;
  };
  double* const pos = a.pos + ws * nc;
  // this thread's AO groups of the moved electron: an even share of the AOs
  int glo = 0, ghi = 0;
  while (glo < t.ngroup && t.group_ao[glo] * ns < t.nao * slot) ++glo;
  ghi = glo;
  while (ghi < t.ngroup && t.group_ao[ghi] * ns < t.nao * (slot + 1)) ++ghi;

  // ---- start positions ----
  if (on)
    for (int e = slot; e < ne; e += ns)
      for (int q = 0; q < 3; ++q) k.H(S.xs + 3 * e + q) = pos[3 * e + q];
  __syncthreads();
  if (on)
    for (int e = slot; e < ne; e += ns) drift_start_rows(d, t, S, k, e);
  __syncthreads();
  if constexpr (FIXED) fix_table(const_cast<double*>(t.W), d.nao, S.ncol, ecol);
  bool start_sum = false;  // of this thread's walker and spin; then of any in the block
  if (slot < 2) {
    const int s = spin, n = nof(s);
    double det = 1.0;
    if (ex) {
      drift_explicit(d, S, k, s, -1, dv0(s), k.cs, nullptr, 0);
    } else if (n == 0) {
      for (int u = 0; u < d.ndet[s]; ++u) dv0(s)[u * k.cs] = 1.0;
    } else {
      int piv[QMC_MAX_NSPIN];
      const MView<double> M{k.cp + ((int64_t)S.lx + r0of(s) * nmu) * k.cs, (int64_t)nmu * k.cs, k.cs};
      for (int i = 0; i < n; ++i)
        for (int j = 0; j < d.max_orb[s]; ++j) M(i, j) = k.C(S.ma + (r0of(s) + i) * nmu + j);
      det = lu_factor<double>(M, n, piv);
      for (int i = 0; i < n; ++i) k.C(S.piv + r0of(s) + i) = (double)piv[i];
      const int nv = nvof(s);
      const MView<double> X{M.p + n * M.cs, M.rs, M.cs};
      if (nv > 0) lu_solve<double>(M, n, piv, X.c(), X, nv);
      excitation_values<double, double>(d, d.det_table[s], s, X.c(), nv > 0 ? nv : 1, dv0(s), k.cs);
      start_sum = det == 0.0;
      for (int u = 0; u < d.ndet[s]; ++u)
        start_sum |= __double2hiint(fabs(dv0(s)[u * k.cs])) > __double2hiint(kGradRatio);
      if (start_sum) {
        det = 1.0;
        if (n > kSumN) drift_explicit(d, S, k, s, -1, dv0(s), k.cs, nullptr, 0);
      }
    }
    k.H(S.val + DV_DET + s) = det;
    k.H(S.val + DV_START + s) = start_sum ? 1.0 : 0.0;
  }
  start_sum = __syncthreads_or(start_sum);
  if (start_sum) {
    start_sums([&](const DriftWork& kq, int s) {
      drift_sum_warp<false>(d, S, kq, s, nof(s), -1, dets(kq, s), kq.cs, nullptr, 0, false);
    });
    __syncthreads();
    start_sums([&](const DriftWork& kq, int s) {
      drift_sum_warp<true>(d, S, kq, s, nof(s), -1, nullptr, 0, dets(kq, 1 - s), kq.cs,
                           drift_cofactors(d, s));
    });
  }
  // A^-1 by columns; F, or G in explicit mode
  if (!ex && on)
    for (int e = slot; e < ne; e += ns) {
      const int s = e < d.nup ? 0 : 1, n = nof(s), r0 = r0of(s);
      const MView<double> LU{k.cp + ((int64_t)S.lx + r0 * nmu) * k.cs, (int64_t)nmu * k.cs, k.cs};
      const int y = S.inv + e * nmax;
      int at = e - r0;  // where the row interchanges move the one
      for (int r = 0; r < n; ++r) {
        const int p = (int)k.C(S.piv + r0 + r);
        at = at == r ? p : (at == p ? r : at);
      }
      for (int r = 0; r < n; ++r) {
        double v = r == at ? 1.0 : 0.0;
        for (int c = at; c < r; ++c) v = fma(-LU(r, c), k.C(y + c), v);
        k.C(y + r) = v;
      }
      for (int r = n - 1; r >= 0; --r) {
        double v = k.C(y + r);
        for (int c = r + 1; c < n; ++c) v = fma(-LU(r, c), k.C(y + c), v);
        k.C(y + r) = v * LU(r, r);
      }
    }
  if (slot < 2) {
    const bool sum = k.H(S.val + DV_START + spin) != 0.0;
    if (ex || (sum && nof(spin) > kSumN))
      drift_explicit(d, S, k, spin, -1, dv0(spin), k.cs, dv0(1 - spin), k.cs);
    else if (!sum)
      drift_adjoint(d, S, k, spin, x0(spin), dv0(1 - spin), k.cs);
    if (slot == 0) {
      double sigma = 0.0;
      for (int c = 0; c < d.ncfg; ++c)
        sigma = fma(__ldg(d.ci_weight + c), dv0(0)[__ldg(d.cfg_det[0] + c) * k.cs] *
                                                dv0(1)[__ldg(d.cfg_det[1] + c) * k.cs], sigma);
      k.H(S.val + DV_SIGMA) = sigma;
      k.H(S.val + DV_CUR) = 0.0;
      k.H(S.val + DV_EACC) = -1.0;
      k.H(S.val + DV_FLAG) = 0.0;
    }
  }
  __syncthreads();
  double rhoi = 0.0, logj0 = 0.0;
  const double dd0 = k.H(S.val + DV_DET) * k.H(S.val + DV_DET + 1);
  if (on) {
    // the walker's threads all hold the start's density and log J
    const double sigma = k.H(S.val + DV_SIGMA);
    for (int e = 0; e < ne; ++e) logj0 += k.C(S.ju + e);
    const double psi = jexp(logj0) * (dd0 * sigma);
    rhoi = psi * psi;
    // where rho is zero (underflow included) the reference's drift
    // grad(rho) / (2 rho) is undefined: every later transition kernel is NaN and
    // every move of this walker is rejected
    const bool zero = rhoi == 0.0;
    if (zero) rhoi = 1e-16;
    const double is = zero ? nan("") : 1.0 / sigma;
    for (int e = slot; e < ne; e += ns) {
      const int s = e < d.nup ? 0 : 1, n = nof(s), nv = nvof(s), i = e - r0of(s);
      double g[3] = {0.0, 0.0, 0.0};
      const int mg = S.mg + 3 * e * nmu;
      if (ex || k.H(S.val + DV_START + s) != 0.0) {
        for (int j = 0; j < nmu; ++j)
          for (int q = 0; q < 3; ++q)
            g[q] = fma(k.C(S.gx + e * nmu + j), k.C(mg + q * nmu + j), g[q]);
      } else {
        for (int q = 0; q < 3; ++q) {
          const int row = mg + q * nmu, zr = S.zm + (3 * e + q) * nmu;
          for (int v = 0; v < nv; ++v) {
            double m = k.C(row + n + v);
            for (int j = 0; j < n; ++j) m = fma(-x0(s)(j, v), k.C(row + j), m);
            k.C(zr + n + v) = m;
          }
          for (int l = 0; l < n; ++l) {
            double v = 0.0;
            for (int j = 0; j < n; ++j)
              v = fma(k.C(S.inv + (r0of(s) + l) * nmax + j), k.C(row + j), v);
            k.C(zr + l) = v;
          }
          g[q] = sigma * k.C(zr + i);
        }
        for (int v = 0; v < nv; ++v) {
          double f = 0.0;
          for (int j = 0; j < n; ++j)
            f = fma(k.C(S.inv + e * nmax + j), k.H(f0of(s) + j * nv + v), f);
          for (int q = 0; q < 3; ++q) g[q] = fma(f, k.C(S.zm + (3 * e + q) * nmu + n + v), g[q]);
        }
      }
      for (int q = 0; q < 3; ++q)
        k.H(S.dr + 3 * e + q) = fma(g[q], is, k.C(S.jg0 + 3 * e + q));
    }
  }
  __syncthreads();

  Rng rng{(uint32_t)a.seed, (uint32_t)(a.seed >> 32), (uint32_t)w, 0, 0};
  const bool replay = a.electron_index != nullptr;
  int nacc = 0, idecor = 0;
  int64_t isnap = 0;
  for (int istep = 0; istep < a.nstep; ++istep) {
    // ---- draws, by every thread of the walker: the moved electron, its noise, the
    // acceptance uniform ----
    int e;
    double eta[3], uacc;
    if (replay) {
      const int64_t o = (int64_t)istep * nw + ws;
      e = a.electron_index[o];
      for (int q = 0; q < 3; ++q) eta[q] = a.normals[o * 3 + q];
      uacc = a.uniforms[o];
    } else {
      rng.step = a.step_offset + istep;
      rng.call = 0;
      const U4 r0 = rng.next();
      e = (int)(((uint64_t)r0.x * (uint64_t)ne) >> 32);
      uacc = rng.uniform53(r0.y, r0.z);
      const U4 r1 = rng.next();
      double z3;
      rng.normal2(r1.x, r1.y, eta[0], eta[1]);
      rng.normal2(r1.z, r1.w, eta[2], z3);
      for (int q = 0; q < 3; ++q) eta[q] *= sd;
    }
    if (e < 0 || e >= ne) e = 0;  // replayed indices are checked by the host
    const int cur = k.H(S.val + DV_CUR) != 0.0 ? 3 * ne : 0;
    const int dri = S.dr + cur, drf = S.dr + 3 * ne - cur;
    // proposal: start positions with electron e at xs_e + (step drift_i(e) + eta)
    double pe[3], pe0[3];
    for (int q = 0; q < 3; ++q) {
      pe0[q] = k.H(S.xs + 3 * e + q);
      pe[q] = __dadd_rn(pe0[q], __dadd_rn(__dmul_rn(step, k.H(dri + 3 * e + q)), eta[q]));
    }
    const int sm = e < d.nup ? 0 : 1, n = nof(sm), r0 = r0of(sm), l = e - r0, nv = nvof(sm);

    // ---- this thread's AO groups of the moved electron (partial MO row) and its
    // electrons' pairs with it ----
    double du = 0.0, ge[3] = {0.0, 0.0, 0.0};
    if (on) {
      ep_rows<FIXED, false, false>(t, ecol, nmu, pe[0], pe[1], pe[2], 0.0, 0.0, 0.0, 0.0, fix,
                                   S.nthreads, &k.H(S.part + slot * nmu), nullptr, k.hs, glo, ghi);
      if (d.use_jastrow_en && slot == e % ns) {
        const EnTerms en = en_terms(d, pe[0], pe[1], pe[2]);
        du = en.u - k.C(S.jen + e);
        for (int q = 0; q < 3; ++q) ge[q] = en.g[q];
      }
      for (int j = slot; j < ne; j += ns) {
        if (j == e) continue;
        double gj[3];
        for (int q = 0; q < 3; ++q) gj[q] = k.C(S.jg0 + 3 * j + q);
        if (d.use_jastrow) {
          // pair (j, e) at the proposal and at the start
          const double w0 = same_spin(d, e, j) ? 0.25 : 0.5;
          double d1[3], d0[3], u1, u0;
          for (int q = 0; q < 3; ++q) {
            const double xj = k.H(S.xs + 3 * j + q);
            d1[q] = xj - pe[q];
            d0[q] = xj - pe0[q];
          }
          const double c1 = pade_pair(w0, wj, d1[0], d1[1], d1[2], u1);
          const double c0 = pade_pair(w0, wj, d0[0], d0[1], d0[2], u0);
          du += u1 - u0;
          for (int q = 0; q < 3; ++q) {
            const double g1 = c1 * d1[q];
            gj[q] += fma(-c0, d0[q], g1);
            ge[q] -= g1;  // grad_e of the pair is minus grad_j
          }
        }
        for (int q = 0; q < 3; ++q) k.H(S.gj + 3 * j + q) = gj[q];
      }
    }
    __syncthreads();
    if (on)
      for (int j = slot; j < nmu; j += ns) {
        double v = 0.0;
        for (int p = 0; p < ns; ++p) v += k.H(S.part + p * nmu + j);
        k.H(S.phi + j) = v;
      }
    __syncthreads();
    // ---- determinants at the proposal ----
    bool warp_sum = false;
    if (!ex) {
      if (on)
        for (int i = slot; i < n + nv; i += ns) {
          if (i < n) {  // r_i = phi' A^-1 e_i
            double v = 0.0;
            for (int j = 0; j < n; ++j) v = fma(k.H(S.phi + j), k.C(S.inv + (r0 + i) * nmax + j), v);
            k.H(S.r + i) = v;
          } else {  // t_v = phi'_virt - phi' X
            double v = k.H(S.phi + i);
            for (int j = 0; j < n; ++j) v = fma(-k.H(S.phi + j), x0(sm)(j, i - n), v);
            k.H(S.t + i - n) = v;
          }
        }
      __syncthreads();
      if (slot == 0) {
        bool sum = k.H(S.val + DV_START + sm) != 0.0;
        if (!sum) {
          const double q = 1.0 / k.H(S.r + l);
          for (int v = 0; v < nv; ++v) {
            const double tq = k.H(S.t + v) * q;
            k.H(S.t + v) = tq;
            for (int j = 0; j < n; ++j)
              k.H(S.xp + j * nv + v) = fma(k.C(S.inv + e * nmax + j), tq, x0(sm)(j, v));
          }
          k.H(S.val + DV_Q) = q;
          const CView<double> X{k.hp + (int64_t)S.xp * k.hs, (int64_t)nv * k.hs, k.hs};
          excitation_values<double, double>(d, d.det_table[sm], sm, X, nv > 0 ? nv : 1,
                                            k.hp + (int64_t)S.dvf * k.hs, k.hs);
          for (int u = 0; u < d.ndet[sm]; ++u)
            sum |= __double2hiint(fabs(k.H(S.dvf + u))) > __double2hiint(kGradRatio);
        }
        k.H(S.val + DV_FLAG) = sum ? 1.0 : 0.0;
        k.H(S.val + DV_MOVED) = (double)e;
        warp_sum = sum && n <= kSumN;
        if (sum && !warp_sum)
          drift_explicit(d, S, k, sm, e, k.hp + (int64_t)S.dvf * k.hs, k.hs, dv0(1 - sm), k.cs);
      }
    } else if (slot == 0) {
      drift_explicit(d, S, k, sm, e, k.hp + (int64_t)S.dvf * k.hs, k.hs, dv0(1 - sm), k.cs);
    }
    if (__syncthreads_or(warp_sum)) {
      sum_tasks(
          S.nwb,
          [&](int q) {
            const DriftWork kq = view(q);
            return kq.H(S.val + DV_FLAG) != 0.0 && nof(electron(kq) < d.nup ? 0 : 1) <= kSumN;
          },
          [&](int q) {
            const DriftWork kq = view(q);
            const int eq = electron(kq), s = eq < d.nup ? 0 : 1;
            drift_sum_warp<true>(d, S, kq, s, nof(s), eq, kq.hp + (int64_t)S.dvf * kq.hs, kq.hs,
                                 dets(kq, 1 - s), kq.cs, false);
          });
      __syncthreads();
    }
    if (start_sum)  // the other spin's G, with the moved spin's determinants
      sum_tasks(
          S.nwb,
          [&](int q) {
            const DriftWork kq = view(q);
            const int s = electron(kq) < d.nup ? 1 : 0;
            return nof(s) <= kSumN && kq.H(S.val + DV_START + s) != 0.0;
          },
          [&](int q) {
            const DriftWork kq = view(q);
            const int s = electron(kq) < d.nup ? 1 : 0;
            const double* const dvf = kq.hp + (int64_t)S.dvf * kq.hs;
            if (drift_cofactors(d, s))
              drift_cof_warp(d, S, kq, s, nof(s), dvf, kq.hs);
            else
              drift_sum_warp<true>(d, S, kq, s, nof(s), -1, nullptr, 0, dvf, kq.hs, false);
          });
    const double* const dvf = k.hp + (int64_t)S.dvf * k.hs;
    if (slot < 2) {
      const CView<double> X{k.hp + (int64_t)S.xp * k.hs, (int64_t)nv * k.hs, k.hs};
      if (!ex) {
        // slot 0: the moved spin (unless it has G already), slot 1: the other
        const int s = slot == 0 ? sm : 1 - sm;
        if (s == sm) {
          if (k.H(S.val + DV_FLAG) == 0.0) drift_adjoint(d, S, k, s, X, dv0(1 - s), k.cs);
        } else if (k.H(S.val + DV_START + s) == 0.0) {
          drift_adjoint(d, S, k, s, x0(s), dvf, k.hs);
        } else if (nof(s) > kSumN) {
          drift_explicit(d, S, k, s, -1, k.hp + (int64_t)S.part * k.hs, 0, dvf, k.hs);
        }
      } else if (slot == 1) {
        // the moved spin's G from the determinants phase; the other's now
        drift_explicit(d, S, k, 1 - sm, -1, k.hp + (int64_t)S.part * k.hs, 0, dvf, k.hs);
      }
      if (slot == (ex ? 0 : 1)) {
        double sigma = 0.0;
        for (int c = 0; c < d.ncfg; ++c)
          sigma = fma(__ldg(d.ci_weight + c), dvf[__ldg(d.cfg_det[sm] + c) * k.hs] *
                                                  dv0(1 - sm)[__ldg(d.cfg_det[1 - sm] + c) * k.cs],
                      sigma);
        k.H(S.val + DV_SIGMA) = sigma;
      }
    }
    __syncthreads();
    // ---- gradients: the moved electron's G row, this thread's electrons, then this
    // thread's AO groups of the moved electron ----
    const double sigma = k.H(S.val + DV_SIGMA), is = 1.0 / sigma;
    if (on) {
      // whether the moved spin's G, and the other's, is in gx
      const bool sum = ex || k.H(S.val + DV_FLAG) != 0.0;
      const bool osum = ex || k.H(S.val + DV_START + 1 - sm) != 0.0;
      const double q0 = ex ? 0.0 : k.H(S.val + DV_Q);
      double a1 = 0.0, a2 = 0.0;
      const int eacc = (int)k.H(S.val + DV_EACC);
      for (int i = slot; i < ne; i += ns) {
        if (i != e) {
          const int s = i < d.nup ? 0 : 1, mg = S.mg + 3 * i * nmu, ns_ = nof(s), nvs = nvof(s);
          double g[3] = {0.0, 0.0, 0.0};
          const bool moved = s == sm;
          if (moved ? sum : osum) {
            for (int j = 0; j < nmu; ++j)
              for (int q = 0; q < 3; ++q)
                g[q] = fma(k.C(S.gx + i * nmu + j), k.C(mg + q * nmu + j), g[q]);
          } else {
            const double ri = moved ? q0 * k.H(S.r + i - r0) : 0.0;
            const int zr = S.zm + 3 * i * nmu;
            double z[3];
            for (int q = 0; q < 3; ++q) {
              z[q] = moved ? k.C(zr + q * nmu + l) : 0.0;
              g[q] = sigma * fma(-ri, z[q], k.C(zr + q * nmu + i - r0of(s)));
            }
            for (int v = 0; v < nvs; ++v) {
              double f = 0.0;
              for (int j = 0; j < ns_; ++j) {
                const double yi = k.C(S.inv + i * nmax + j);
                f = fma(moved ? fma(-ri, k.C(S.inv + e * nmax + j), yi) : yi,
                        k.H(f0of(s) + j * nvs + v), f);
              }
              const double tv = moved ? k.H(S.t + v) : 0.0;
              for (int q = 0; q < 3; ++q)
                g[q] = fma(fma(-tv, z[q], k.C(zr + q * nmu + ns_ + v)), f, g[q]);
            }
          }
          for (int q = 0; q < 3; ++q) {
            const int c = 3 * i + q;
            const double df = fma(g[q], is, k.H(S.gj + c));
            k.H(drf + c) = df;
            // the proposal has the start's position here; the accepted one unless i moved
            double dx = 0.0;
            if (i == eacc) dx = __dsub_rn(k.H(S.val + DV_XACC + q), k.H(S.xs + c));
            const double t1 = __dsub_rn(dx, __dmul_rn(df, step));
            const double t2 = __dsub_rn(-dx, __dmul_rn(k.H(dri + c), step));
            a1 = fma(t1, t1, a1);
            a2 = fma(t2, t2, a2);
          }
        }
      }
      const int red = S.red + slot * kDriftRed;
      k.H(red) = du;
      k.H(red + 1) = a1;
      k.H(red + 2) = a2;
      for (int q = 0; q < 3; ++q) k.H(red + 3 + q) = ge[q];
      double ga[3] = {0.0, 0.0, 0.0};
      const int norb = ex ? nmu : d.max_orb[sm];
      for (int j0 = 0; j0 < norb; j0 += 8) {
        double G[8];
        if (sum) {
#pragma unroll
          for (int jj = 0; jj < 8; ++jj)
            G[jj] = j0 + jj < norb ? k.C(S.gx + e * nmu + j0 + jj) : 0.0;
        } else {
          // y' = A^-1 e_l / r_l; G_virt = y' F, G_occ = Sigma y' - G_virt X'^T
#pragma unroll
          for (int jj = 0; jj < 8; ++jj)
            G[jj] = j0 + jj < n ? sigma * (k.C(S.inv + e * nmax + j0 + jj) * q0) : 0.0;
          for (int v = 0; v < nv; ++v) {
            double f = 0.0;
            for (int j = 0; j < n; ++j)
              f = fma(k.C(S.inv + e * nmax + j) * q0, k.H(f0of(sm) + j * nv + v), f);
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
              if (j0 + jj < n) G[jj] = fma(-f, k.H(S.xp + (j0 + jj) * nv + v), G[jj]);
              if (j0 + jj == n + v) G[jj] = f;
            }
          }
        }
        RowG<8, FIXED> fg;
        fg.set(G, ecol + j0);
        auto h = [&](int ao) {
          return fg.dot(reinterpret_cast<const int2*>(t.W) + (int64_t)ao * t.ncol + j0);
        };
        grad_ao_backward(t, pe[0], pe[1], pe[2], h, ga, glo, ghi);
      }
      for (int q = 0; q < 3; ++q) k.H(S.part + slot * 3 + q) = ga[q];
    }
    __syncthreads();
    // ---- transition kernels and the decision ----
    if (slot == 0) {
      double logj = logj0, a1 = 0.0, a2 = 0.0, g[3] = {0.0, 0.0, 0.0}, gu[3] = {0.0, 0.0, 0.0};
      for (int p = 0; p < ns; ++p) {
        const int red = S.red + p * kDriftRed;
        logj += k.H(red);
        a1 += k.H(red + 1);
        a2 += k.H(red + 2);
        for (int q = 0; q < 3; ++q) {
          gu[q] += k.H(red + 3 + q);
          g[q] += k.H(S.part + p * 3 + q);
        }
      }
      const int eacc = (int)k.H(S.val + DV_EACC);
      for (int q = 0; q < 3; ++q) {
        const int c = 3 * e + q;
        const double df = fma(g[q], is, gu[q]);
        k.H(drf + c) = df;
        const double xi = e == eacc ? k.H(S.val + DV_XACC + q) : pe0[q];
        const double t1 = __dsub_rn(__dsub_rn(xi, pe[q]), __dmul_rn(df, step));
        const double t2 = __dsub_rn(__dsub_rn(pe[q], xi), __dmul_rn(k.H(dri + c), step));
        a1 = fma(t1, t1, a1);
        a2 = fma(t2, t2, a2);
      }
      // the determinants that Sigma is relative to
      const double det = ex ? 1.0
                            : (k.H(S.val + DV_FLAG) != 0.0 ? k.H(S.val + DV_DET + 1 - sm)
                                                           : dd0 * k.H(S.r + l));
      const double psif = jexp(logj) * (det * sigma);
      double rhof = psif * psif;
      const bool defined = rhof != 0.0;  // else the reference's drift is NaN: rejected
      if (rhof == 0.0) rhof = 1e-16;
      const double hs = 0.5 / step;
      const double tif = rexp(-hs * psqrt(a1)), tfi = rexp(-hs * psqrt(a2));
      double p = (tif * rhof) / (tfi * rhoi);
      if (p > 1.0) p = 1.0;
      if (defined && p - uacc >= 0.0) {
        ++nacc;
        rhoi = rhof;
        k.H(S.val + DV_CUR) = cur ? 0.0 : 1.0;
        k.H(S.val + DV_EACC) = (double)e;
        for (int q = 0; q < 3; ++q) k.H(S.val + DV_XACC + q) = pe[q];
      }
    }
    __syncthreads();
    if (istep >= a.ntherm) {
      if (idecor % a.ndecor == 0 && a.samples && isnap < a.nsnap) {
        if (live) {
          const int eacc = (int)k.H(S.val + DV_EACC);
          double* o = a.samples + (isnap * nw + w) * nc;
          for (int i = slot; i < ne; i += ns)
            for (int q = 0; q < 3; ++q)
              o[3 * i + q] = i == eacc ? k.H(S.val + DV_XACC + q) : k.H(S.xs + 3 * i + q);
        }
        ++isnap;
      }
      ++idecor;
    }
  }
  if (live && slot == 0) {
    const int eacc = (int)k.H(S.val + DV_EACC);
    if (eacc >= 0)
      for (int q = 0; q < 3; ++q) pos[3 * eacc + q] = k.H(S.val + DV_XACC + q);
    if (a.accepted) a.accepted[w] += nacc;
  }
}

// Launch plan, by the rule of grad_plan: the least warp work on the busiest SM
// (a walker's work is shared evenly by its threads, up to one per electron).
template <bool FIXED>
static DriftShape drift_plan(const qmc_wf_desc& d, int64_t nw) {
  const auto kernel = drift_kernel<FIXED>;
  int dev = 0, nsm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  DriftShape best = drift_shape(d, 1, 2, true, FIXED);
  const PlanKey key = plan_key((const void*)kernel, dev, nw, d, best.smem);
  PlanChoice got;
  if (plan_find(key, &got)) return drift_shape(d, got.nwb, got.nslot, got.in_smem, FIXED);
  best.smem = -1;
  double best_cost = 0.0;
  const int most = d.nelec > 16 ? 16 : (d.nelec < 2 ? 2 : d.nelec);
  for (int in_smem = 1; in_smem >= 0 && best.smem < 0; --in_smem)
    for (int nwb = 32; nwb >= 4; nwb /= 2)
      for (int nslot = 2; nslot <= most; ++nslot) {
        const DriftShape s = drift_shape(d, nwb, nslot, in_smem == 1, FIXED);
        if (s.nthreads > kGradThreads || s.smem > 227 * 1024) continue;
        if (prepare_smem(kernel, s.smem) != QMC_OK) continue;
        int occ = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, s.nthreads, s.smem) !=
                cudaSuccess ||
            occ < 1) {
          cudaGetLastError();
          continue;
        }
        const int64_t blocks = (nw + nwb - 1) / nwb, on_sm = (blocks + nsm - 1) / nsm;
        const int64_t rounds = (on_sm + occ - 1) / occ;
        const int64_t walkers = (rounds == 1 ? on_sm : rounds * occ) * nwb;
        const double warps = (double)(on_sm < occ ? on_sm : occ) * s.nthreads / 32.0;
        const int per = (d.nelec + nslot - 1) / nslot;
        double cost = (double)walkers * per * s.nthreads / ((double)nwb * d.nelec);
        if (warps < 12.0) cost *= sqrt(12.0 / warps);
        cost *= 1.0 + 0.1 * (nwb < 32 ? 32.0 / nwb : 1.0);
        if (best.smem < 0 || cost < 0.999 * best_cost) {
          best = s;
          best_cost = cost;
        }
      }
  if (best.smem >= 0) plan_keep(key, {best.nwb, best.nslot, best.o_hot >= 0, 0, false});
  return best;
}

template <bool FIXED>
static int launch_drift(const qmc_wf_desc& d, const qmc_drift_args& a, double* scr,
                        cudaStream_t s) {
  const DriftShape S = drift_plan<FIXED>(d, a.nwalkers);
  if (S.smem < 0) return QMC_ERR_SHAPE;
  const int st = prepare_smem(drift_kernel<FIXED>, S.smem);
  if (st) return st;
  const double sd = sqrt(sqrt(a.step_size));  // covariance sqrt(step) I
  drift_kernel<FIXED><<<(unsigned)((a.nwalkers + S.nwb - 1) / S.nwb), S.nthreads, S.smem, s>>>(
      d, a, scr, pad_walkers(a.nwalkers), sd, S);
  return launch_status();
}

}  // namespace qmc

using namespace qmc;

extern "C" {

int64_t qmc_drift_scratch_bytes(const qmc_wf_desc* d, int64_t nw) {
  if (check_desc(d) != QMC_OK || nw < 0) return -1;
  const DriftShape s = drift_shape(*d, 1, 16, false);  // the most threads per walker
  return (int64_t)(s.cold + s.hot) * pad_walkers(nw) * (int64_t)sizeof(double);
}

int qmc_drift_run(const qmc_wf_desc* d0, const qmc_drift_args* a, void* scratch,
                  int64_t scratch_bytes, void* stream) {
  int st = check_desc(d0);
  if (st) return st;
  if (!a) return QMC_ERR_ARG;
  qmc_wf_desc dd = *d0;
  dd.precision = QMC_PREC_FP64;  // the drift sampler is FP64
  const qmc_wf_desc* d = &dd;
  if (a->nwalkers < 0 || a->nstep < 0 || a->ntherm < 0 || a->ndecor < 1 || a->nsnap < 0 ||
      !(a->step_size > 0.0))
    return QMC_ERR_ARG;
  const int nrep = (a->electron_index != nullptr) + (a->normals != nullptr) +
                   (a->uniforms != nullptr);
  if (nrep != 0 && nrep != 3) return QMC_ERR_ARG;  // replay needs all three inputs
  if (a->nwalkers == 0 || a->nstep == 0) return QMC_OK;
  if (!a->pos || !scratch) return QMC_ERR_ARG;
  if (a->nsnap > 0 && !a->samples) return QMC_ERR_ARG;
  if (scratch_bytes < qmc_drift_scratch_bytes(d, a->nwalkers)) return QMC_ERR_SCRATCH;
  st = QMC_ERR_SHAPE;
  if (fix_applies(dd)) st = launch_drift<true>(dd, *a, (double*)scratch, (cudaStream_t)stream);
  // and without limbs where W and the AO slots do not fit (grad_plan)
  if (st == QMC_ERR_SHAPE) st = launch_drift<false>(dd, *a, (double*)scratch, (cudaStream_t)stream);
  return st;
}

}  // extern "C"
