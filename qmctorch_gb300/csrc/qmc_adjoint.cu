// Hand-written adjoints of psi and of the local energy with respect to the
// trainable parameters (ao.bas_exp, mo.mo_modifier through W = mo_scf *
// mo_modifier, the Pade weights, fc.weight), FP64, positions held fixed. Nothing
// is stored by the forward pass.
//
// A block takes tiles of nwb walkers, a thread per electron. Per tile: MO rows
// (for E_L also the kinetic rows B), one factorisation per (walker, spin), the
// adjoints of the MO values (G_A) and of B (G_B) from it, then one more pass
// over the AOs. The parameter gradients are contractions over all electrons of
// all walkers: dW = AO^T G, and d/d alpha_p = sum_a (weight of AO a) exp(-alpha_p
// r^2). Each thread puts its AO values, its weights and its exponentials of some
// AO groups into a shared-memory tile [row][electron], and the block's threads,
// an output each, sum the products over the electrons: one multiply-add per
// electron and gradient entry, no reduction across lanes. The sums go to the
// block's own row of the scratch; adj_reduce_kernel adds the rows in a fixed
// order, so the gradients are bitwise reproducible.
//
// E_L in excitation mode: with A the occupied block, V the virtual columns,
// X = A^-1 V, Y = A^-1 B and M = Y_virt - Y_occ X, every configuration's
// D T = D (x base + n), x(X) and n(X, M) of degree two at most, base = Tr Y_occ, so
//   KE = base_up + base_dn + Q / Sigma,
//   Sigma = sum c x x',  Q = sum c (n x' + x n').
// With F_X = (dQ/dX - Q/Sigma dSigma/dX) / Sigma, F_M = (dQ/dM) / Sigma,
// P = A^-T F_M and K = A^-T (F_X - Y_occ^T F_M):
//   G_B = [A^-T - P X^T | P],
//   G_A = [-(Y_occ A^-1)^T - P M^T - K X^T | K].
// Explicit mode (CAS), and a spin with a large excitation ratio (kAdjRatio), sum
//   dKE/dA_u = dD_u D_u X^T - dT_u (X B_u X)^T,  dKE/dB_u = dT_u X^T,  X = A_u^-1
// over the determinants. B = -1/2 (lap MO + 2 grad(U) . grad MO + (lap U +
// |grad U|^2) MO), U = log J (slater_jastrow.py:312-344, 449-482); V does not
// depend on the parameters.
//
// FP64 pipe bound (2 lanes per clock and SM), so counted in FP64 instructions:
// H2O cc-pVDZ single_double(4,4), about 29,000 per walker for E_L; 4000 walkers 4.3 -> 1.5 ms.
// Compiled twice: with limbs and the C entry points, and with -DQMC_INST_FIXED=0 for the
// instances without limbs.
#include <cuda_runtime.h>
#include <stdint.h>

#ifndef QMC_INST_FIXED
#define QMC_INST_FIXED 1
#endif

#include "qmc_grad.cuh"
#include "qmc_host.cuh"

namespace qmc {

constexpr int kAdjThreads = 256;
constexpr int kAdjBlocks = 608;  // most blocks (rows of partial sums): 4 per SM
// Rows of AO and exponential values in the tile: a group's AO rows (at most
// QMC_MAX_COMP components, five rows each for E_L, two for psi) and at least some
// of its exponentials.
__host__ __device__ constexpr int adj_tile_rows(bool el) { return el ? 40 : 24; }
__host__ __device__ constexpr int64_t adj_tile_doubles(bool el, int jc, int ts) {
  return (int64_t)(adj_tile_rows(el) + (el ? 2 : 1) * jc) * ts;
}
static_assert(adj_tile_rows(true) > 5 * QMC_MAX_COMP && adj_tile_rows(false) > 2 * QMC_MAX_COMP,
              "an AO group's rows fit the tile with room for its exponentials");

// gradient entries: W [nao][nmu], exponents [nweight] (one per basis entry), CI
// weights [ncfg], the e-e and the e-n Pade weight
__host__ __device__ inline int adj_params(const qmc_wf_desc& d) {
  return d.nao * d.nmo_used + d.nweight + d.ncfg + 2;
}
// Threads that share an output's electrons where a molecule has fewer outputs
// than a block has threads.
__host__ __device__ inline int adj_parts(const qmc_wf_desc& d) {
  const int n = d.nao * d.nmo_used;
  return n >= 128 ? 1 : (n >= 64 ? 2 : (n >= 32 ? 4 : 8));
}

// The E_L adjoint's line, by the same rule: parameter gradients of 2000 H2O walkers (2-norm,
// the largest of 25) differ from the explicit sums' by 3.2e-14 at 64 and below, which is
// their rounding, by 1.5e-13 at 256 and by 9e-12 at 1024. A step of 4000 walkers takes the
// same at 32 and at 256, 1.82 ms.
constexpr double kAdjRatio = 32.0;

struct AdjShape {
  GradShape g;  // per-walker arrays of the psi adjoint and the block's layout
  // E_L: kinetic rows (then Y_occ | M), F_M and F_X - Y_occ^T F_M, the n values,
  // Jastrow terms [8] per electron (grad U, lap U + |grad U|^2, their w derivatives)
  int bk, fm, fk, ov, jt, r, total;
  int64_t cold;  // per-walker doubles of the scratch: V, Z and G_B of the explicit sums
  int64_t o_tile, o_work, smem;  // o_tile < 0: the tile is in the scratch
  int ts, rows, parts, nparam, grid;
};

static AdjShape adj_shape(const qmc_wf_desc& d, bool el, int nwb, int nslot, int jc, bool in_smem,
                          bool fixed = true, bool tile_smem = true) {
  AdjShape s;
  s.g = grad_shape(d, nwb, nslot, jc, false, fixed);
  const int ne = d.nelec, nmu = d.nmo_used, nmax = d.nup > d.ndown ? d.nup : d.ndown;
  int o = s.g.total;
  auto take = [&](int n) {
    const int r = o;
    o += n;
    return r;
  };
  s.bk = take(el ? ne * nmu : 0);
  s.fm = take(el ? 2 * s.g.fs : 0);
  s.fk = take(el ? 2 * s.g.fs : 0);
  s.ov = take(el ? d.ndet[0] + d.ndet[1] : 0);
  s.jt = take(el ? 8 * ne : 0);
  s.r = take(4);  // R = Q / Sigma, the base traces, gout
  s.total = o;
  s.cold = el ? 4 * (int64_t)nmax * nmax + (int64_t)ne * nmu : 0;
  s.ts = (nwb * nslot) | 1;  // odd: lanes that read different rows hit different banks
  s.rows = adj_tile_rows(el);
  s.parts = adj_parts(d);
  s.nparam = adj_params(d);
  s.grid = 0;
  s.o_tile = -1;
  s.smem = s.g.smem;
  if (tile_smem) {
    s.o_tile = s.smem;
    s.smem += (adj_tile_doubles(el, jc, s.ts) * 8 + 15) & ~int64_t(15);
  }
  s.o_work = -1;
  if (in_smem) {
    s.o_work = s.smem;
    s.smem += (int64_t)s.total * nwb * 8;
  }
  return s;
}

// scratch: partial sums [grid * parts][nparam], the blocks' tiles (of the plan that has them
// there: one walker, two threads), then the cold arrays and, where they do not fit shared
// memory, the work arrays [item][walker]
__host__ __device__ inline int64_t adj_scratch_tiles(bool el) {
  return kAdjBlocks * adj_tile_doubles(el, 8, 3);
}
static int64_t adj_scratch_bytes(const qmc_wf_desc& d, bool el, int64_t nw) {
  const AdjShape s = adj_shape(d, el, 1, 2, 8, false);
  return 8 * ((int64_t)kAdjBlocks * s.parts * s.nparam + adj_scratch_tiles(el) +
              (s.cold + s.total) * pad_walkers(nw));
}

// Jastrow terms of electron e for the E_L adjoint: grad U, lap U + |grad U|^2 and
// the derivatives of grad U and lap U with respect to the e-e weight
// (K = w0 r / (1 + w r), K' = w0 / (1 + w r)^2, K'' = -2 w w0 / (1 + w r)^3).
__device__ inline void adj_jastrow(const qmc_wf_desc& d, const GradShape& S, const GradWork& k,
                                   int jt, int e) {
  const double x = k.at(S.pos + 3 * e), y = k.at(S.pos + 3 * e + 1), z = k.at(S.pos + 3 * e + 2);
  double g[3] = {0.0, 0.0, 0.0}, dg[3] = {0.0, 0.0, 0.0}, lap = 0.0, dlap = 0.0;
  if (d.use_jastrow) {
    const double w = __ldg(d.jastrow_w);
    for (int j = 0; j < d.nelec; ++j) {
      if (j == e) continue;
      const double dx[3] = {x - k.at(S.pos + 3 * j), y - k.at(S.pos + 3 * j + 1),
                            z - k.at(S.pos + 3 * j + 2)};
      const double r = psqrt(dx[0] * dx[0] + dx[1] * dx[1] + dx[2] * dx[2]), ir = prcp(r);
      const double w0 = same_spin(d, e, j) ? 0.25 : 0.5;
      const double u = prcp(fma(w, r, 1.0)), k1 = w0 * u * u, k1r = k1 * ir, ku = k1 * u;
      const double dk1 = -2.0 * ku * r;  // dK'/dw, and dK''/dw = -2 K' u + 6 w r K' u^2
      const double dk1r = -2.0 * ku;
      for (int q = 0; q < 3; ++q) {
        g[q] = fma(k1r, dx[q], g[q]);
        dg[q] = fma(dk1r, dx[q], dg[q]);
      }
      lap += 2.0 * fma(-w, ku, k1r);
      dlap += 2.0 * (dk1r - ku - 1.5 * w * dk1 * u);
    }
  }
  if (d.use_jastrow_en) {
    const EnTerms en = en_terms(d, x, y, z);
    for (int q = 0; q < 3; ++q) g[q] += en.g[q];
    lap += en.lap;
  }
  for (int q = 0; q < 3; ++q) {
    k.at(jt + 8 * e + q) = g[q];
    k.at(jt + 8 * e + 4 + q) = dg[q];
  }
  k.at(jt + 8 * e + 3) = lap + g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
  k.at(jt + 8 * e + 7) = dlap;
}

struct AdjCold {  // per-(walker, spin) scratch of the explicit sums
  double* p;
  int64_t ss;
};
__device__ __forceinline__ MView<double> adj_cold(const AdjCold& c, int64_t off, int64_t ld) {
  return MView<double>{c.p + off * c.ss, ld * c.ss, c.ss};
}

// D_u and n_u = D_u T_u of spin s from the explicit determinants.
__device__ __noinline__ inline void adj_sum_values(const qmc_wf_desc& d, const AdjShape& A,
                                            const GradWork& k, const AdjCold& cold, int s) {
  const GradShape& S = A.g;
  const int n = s ? d.ndown : d.nup, r0 = s ? d.nup : 0, nmu = d.nmo_used;
  const int nmax = d.nup > d.ndown ? d.nup : d.ndown;
  const int nd = d.ndet[s], o = s ? d.ndet[0] : 0;
  const MView<double> B = grad_view(k, A.bk, r0, nmu);
  int piv[QMC_MAX_NSPIN], cols[QMC_MAX_NSPIN];
  const MView<double> F{k.p + ((int64_t)S.y + r0 * nmax) * k.ws, (int64_t)nmax * k.ws, k.ws};
  const MView<double> V = adj_cold(cold, (int64_t)s * nmax * nmax, nmax);
  for (int u = 0; u < nd; ++u) {
    const double det = grad_factor(d, S, k, s, u, cols, piv);
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j) V(i, j) = B(i, cols[j]);
    lu_solve<double>(F, n, piv, V.c(), V, n);
    double tr = 0.0;
    for (int i = 0; i < n; ++i) tr += V(i, i);
    k.at(S.dv + o + u) = det;
    k.at(A.ov + o + u) = det * tr;
  }
}

// G_A (`lu`) and G_B (scratch) of spin s summed over the explicit determinants.
__device__ __noinline__ inline void adj_sum_adjoints(const qmc_wf_desc& d, const AdjShape& A,
                                              const GradWork& k, const AdjCold& cold, int s,
                                              double is, double R) {
  const GradShape& S = A.g;
  const int n = s ? d.ndown : d.nup, r0 = s ? d.nup : 0, nmu = d.nmo_used;
  const int nmax = d.nup > d.ndown ? d.nup : d.ndown;
  const int so = s ? d.ndet[0] : 0, oo = s ? 0 : d.ndet[0];
  const int* cu = d.cfg_det[s];
  const int* co = d.cfg_det[1 - s];
  const MView<double> L = grad_view(k, S.lu, r0, nmu), B = grad_view(k, A.bk, r0, nmu);
  const MView<double> F{k.p + ((int64_t)S.y + r0 * nmax) * k.ws, (int64_t)nmax * k.ws, k.ws};
  const MView<double> V = adj_cold(cold, (int64_t)s * nmax * nmax, nmax),
                      Z = adj_cold(cold, (int64_t)(2 + s) * nmax * nmax, nmax),
                      GB = adj_cold(cold, 4 * (int64_t)nmax * nmax + (int64_t)r0 * nmu, nmu);
  int piv[QMC_MAX_NSPIN], cols[QMC_MAX_NSPIN];
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < nmu; ++j) L(i, j) = GB(i, j) = 0.0;
  for (int u = 0; u < d.ndet[s]; ++u) {
    // d KE = dT D_u dT_u + (dD D_u + dT T_u D_u) d log D_u
    double dT = 0.0, dD = 0.0;
    for (int c = 0; c < d.ncfg; ++c) {
      if (__ldg(cu + c) != u) continue;
      const int v = oo + __ldg(co + c);
      const double w = __ldg(d.ci_weight + c) * is;
      dT = fma(w, k.at(S.dv + v), dT);
      dD = fma(w, k.at(A.ov + v) - R * k.at(S.dv + v), dD);
    }
    if (dT == 0.0 && dD == 0.0) continue;
    const double det = grad_factor(d, S, k, s, u, cols, piv);
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j) V(i, j) = i == j ? 1.0 : 0.0;
    lu_solve<double>(F, n, piv, V.c(), V, n);  // X = A_u^-1
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j) {  // Z = B_u X
        double z = 0.0;
        for (int c = 0; c < n; ++c) z = fma(B(i, cols[c]), V(c, j), z);
        Z(i, j) = z;
      }
    const double t = dT * det, sd = fma(dT, k.at(A.ov + so + u), dD * det);
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j) {
        double y = 0.0;  // (X B_u X)(j, i)
        for (int c = 0; c < n; ++c) y = fma(V(j, c), Z(c, i), y);
        L(i, cols[j]) += sd * V(j, i) - t * y;
        GB(i, cols[j]) += t * V(j, i);
      }
  }
}

// The two above by a warp, a lane per determinant, for a spin of n <= kSumN electrons.
__device__ __noinline__ inline void adj_sum_values_warp(const qmc_wf_desc& d, const AdjShape& A,
                                                 const GradWork& k, int s, int n_) {
  const GradShape& S = A.g;
  const int r0 = s ? d.nup : 0, nmu = d.nmo_used, o = s ? d.ndet[0] : 0;
  const MView<double> M = grad_view(k, S.mo, r0, nmu), B = grad_view(k, A.bk, r0, nmu);
  sum_traces(d, s, n_, [&](int i, int c) { return M(i, c); }, [&](int i, int c) { return B(i, c); },
             [&](int u, double det, double tr) {
               k.at(S.dv + o + u) = det;
               k.at(A.ov + o + u) = det * tr;
             });
}

__device__ __noinline__ inline void adj_sum_adjoints_warp(const qmc_wf_desc& d, const AdjShape& A,
                                                   const GradWork& k, const AdjCold& cold, int s,
                                                   int n_) {
  const GradShape& S = A.g;
  const int r0 = s ? d.nup : 0, nmu = d.nmo_used, nd = d.ndet[s];
  const int nmax = d.nup > d.ndown ? d.nup : d.ndown;
  const int so = s ? d.ndet[0] : 0, oo = s ? 0 : d.ndet[0];
  const double is = k.at(S.val + GV_INV), R = k.at(A.r);
  const MView<double> M = grad_view(k, S.mo, r0, nmu), L = grad_view(k, S.lu, r0, nmu),
                      B = grad_view(k, A.bk, r0, nmu);
  const MView<double> GB = adj_cold(cold, 4 * (int64_t)nmax * nmax + (int64_t)r0 * nmu, nmu);
  sum_dispatch(n_, [&](auto Nc) {
    constexpr int N = decltype(Nc)::value;
    for (int u0 = 0; u0 < nd; u0 += 32) {
      const SumLanes l = sum_lanes(nd, N, u0);
      // d KE = dT D_u dT_u + (dD D_u + dT T_u D_u) d log D_u
      double dT = 0.0, dD = 0.0, t = 0.0, sd = 0.0;
      sum_configs(
          d, s, l.u,
          [&](int v, double& a, double& b) {
            a = k.at(S.dv + oo + v);
            b = k.at(A.ov + oo + v) - R * a;
          },
          [&](double w, double a, double b) {
            dT = fma(w * is, a, dT);
            dD = fma(w * is, b, dD);
          });
      const bool on = l.u < nd && !(dT == 0.0 && dD == 0.0);
      DetRegs<N> D;
      double X[N][N];  // [column][row] of A_u^-1
      if (on) {
        D.factor(d, s, l.u, [&](int i, int c) { return M(i, c); });
#pragma unroll
        for (int i = 0; i < N; ++i) D.unit(i, X[i]);
        t = dT * D.det;
        sd = fma(dT, k.at(A.ov + so + l.u), dD * D.det);
      }
#pragma unroll 1
      for (int i0 = 0; i0 < N; i0 += l.groups) {
        const int i = i0 + l.g;
        double y[N], z1[N];  // rows of G_A and G_B, with column i of X B_u X
#pragma unroll
        for (int j = 0; j < N; ++j) y[j] = z1[j] = 0.0;
        if (on) {
          double xi[N], z[N];
#pragma unroll
          for (int c = 0; c < N; ++c) {
            xi[c] = X[0][c];
#pragma unroll
            for (int q = 1; q < N; ++q) xi[c] = q == i ? X[q][c] : xi[c];
          }
#pragma unroll
          for (int r = 0; r < N; ++r) {
            z[r] = 0.0;
#pragma unroll
            for (int c = 0; c < N; ++c) z[r] = fma(B(r, D.cols[c]), xi[c], z[r]);
          }
#pragma unroll
          for (int j = 0; j < N; ++j) {
            y[j] = 0.0;
#pragma unroll
            for (int c = 0; c < N; ++c) y[j] = fma(X[c][j], z[c], y[j]);
            y[j] = sd * xi[j] - t * y[j];
            z1[j] = t * xi[j];
          }
        }
        sum_columns<N>(l, D.cols, y, N, on, nd, i0, nmu, u0 == 0, L);
        sum_columns<N>(l, D.cols, z1, N, on, nd, i0, nmu, u0 == 0, GB);
      }
    }
  });
}

// E_L determinant phase, one thread per (walker, spin): the factors and X
// (`lu`), Y_occ | M over the kinetic rows, x and n of every unique determinant and
// the base trace. Returns whether the spin sums over explicit determinants instead.
__device__ inline bool adj_el_determinants(const qmc_wf_desc& d, const AdjShape& A,
                                           const GradWork& k, int s) {
  const GradShape& S = A.g;
  const int n = s ? d.ndown : d.nup, r0 = s ? d.nup : 0, nmu = d.nmo_used;
  const int nd = d.ndet[s], o = s ? d.ndet[0] : 0;
  const MView<double> M = grad_view(k, S.mo, r0, nmu), L = grad_view(k, S.lu, r0, nmu),
                      B = grad_view(k, A.bk, r0, nmu);
  int piv[QMC_MAX_NSPIN];
  double base = 0.0;
  bool sum = d.det_mode == QMC_DET_EXPLICIT;
  if (n == 0) {
    for (int u = 0; u < nd; ++u) {
      k.at(S.dv + o + u) = 1.0;
      k.at(A.ov + o + u) = 0.0;
    }
  } else if (!sum) {
    const int norb = d.max_orb[s], nv = norb - n;
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < norb; ++j) L(i, j) = M(i, j);
    sum = lu_factor<double>(L, n, piv) == 0.0;
    for (int i = 0; i < n; ++i) k.piv(S.piv, r0 + i) = piv[i];
    const MView<double> X{L.p + n * L.cs, L.rs, L.cs};
    if (nv > 0) lu_solve<double>(L, n, piv, X.c(), X, nv);
    excitation_values<double, double>(d, d.det_table[s], s, X.c(), nv > 0 ? nv : 1,
                                      k.p + (int64_t)(S.dv + o) * k.ws, k.ws);
    for (int u = 0; u < nd; ++u)
      sum |= __double2hiint(fabs(k.at(S.dv + o + u))) > __double2hiint(kAdjRatio);
    if (!sum) {
      lu_solve<double>(L, n, piv, B.c(), B, norb);  // Y
      for (int i = 0; i < n; ++i) base += B(i, i);
      for (int v = 0; v < nv; ++v)  // M = Y_virt - Y_occ X
        for (int i = 0; i < n; ++i) {
          double m = B(i, n + v);
          for (int j = 0; j < n; ++j) m = fma(-B(i, j), X(j, v), m);
          B(i, n + v) = m;
        }
      for (int u = 0; u < nd; ++u) {
        const int* e = d.det_table[s] + 5 * u;
        const int ord = __ldg(e);
        auto x = [&](int i) { return X(i / nv, i % nv); };
        auto m = [&](int i) { return B(i / nv, n + i % nv); };
        double v = 0.0;
        if (ord == 1) {
          v = m(__ldg(e + 1));
        } else if (ord >= 2) {
          const int i0 = __ldg(e + 1), i1 = __ldg(e + 2), i2 = __ldg(e + 3), i3 = __ldg(e + 4);
          v = x(i3) * m(i0) - x(i1) * m(i2) - x(i2) * m(i1) + x(i0) * m(i3);
        }
        k.at(A.ov + o + u) = v;
      }
    }
  }
  k.at(A.r + 1 + s) = base;
  k.at(S.val + GV_G + s) = sum ? 1.0 : 0.0;
  return sum;
}

// E_L adjoint phase, one thread per (walker, spin): the CI sums, F_M and F_X - Y_occ^T
// F_M, unless the spin sums over explicit determinants.
__device__ inline void adj_el_adjoints(const qmc_wf_desc& d, const AdjShape& A, const GradWork& k,
                                       int s) {
  const GradShape& S = A.g;
  const int n = s ? d.ndown : d.nup, r0 = s ? d.nup : 0, nmu = d.nmo_used;
  const int so = s ? d.ndet[0] : 0, oo = s ? 0 : d.ndet[0];
  const int* cu = d.cfg_det[s];
  const int* co = d.cfg_det[1 - s];
  double sigma = 0.0, num = 0.0;
  for (int c = 0; c < d.ncfg; ++c) {
    const int u = so + __ldg(cu + c), v = oo + __ldg(co + c);
    const double w = __ldg(d.ci_weight + c), xu = k.at(S.dv + u), xo = k.at(S.dv + v);
    sigma = fma(w, xu * xo, sigma);
    num = fma(w, k.at(A.ov + u) * xo + xu * k.at(A.ov + v), num);
  }
  const double is = 1.0 / sigma, R = num * is;
  if (s == 0) {
    k.at(S.val + GV_INV) = is;
    k.at(A.r) = R;
  }
  if (n == 0 || k.at(S.val + GV_G + s) != 0.0) return;
  const MView<double> L = grad_view(k, S.lu, r0, nmu), B = grad_view(k, A.bk, r0, nmu);
  const int nv = d.max_orb[s] - n, fm = A.fm + s * S.fs, fk = A.fk + s * S.fs;
  if (nv <= 0) return;
  for (int i = 0; i < n * nv; ++i) k.at(fm + i) = k.at(fk + i) = 0.0;
  auto x = [&](int i) { return L(i / nv, n + i % nv); };
  auto m = [&](int i) { return B(i / nv, n + i % nv); };
  for (int c = 0; c < d.ncfg; ++c) {
    const int* e = d.det_table[s] + 5 * __ldg(cu + c);
    const int ord = __ldg(e);
    if (ord == 0) continue;
    const int v = oo + __ldg(co + c);
    const double w = __ldg(d.ci_weight + c) * is, a = w * k.at(S.dv + v),
                 b = w * (k.at(A.ov + v) - R * k.at(S.dv + v));
    const int i0 = __ldg(e + 1);
    if (ord == 1) {  // x = X0, n = M0
      k.at(fk + i0) += b;
      k.at(fm + i0) += a;
    } else {  // x = X0 X3 - X1 X2, n = X3 M0 - X1 M2 - X2 M1 + X0 M3
      const int i1 = __ldg(e + 2), i2 = __ldg(e + 3), i3 = __ldg(e + 4);
      k.at(fk + i0) += fma(a, m(i3), b * x(i3));
      k.at(fk + i3) += fma(a, m(i0), b * x(i0));
      k.at(fk + i1) -= fma(a, m(i2), b * x(i2));
      k.at(fk + i2) -= fma(a, m(i1), b * x(i1));
      k.at(fm + i0) = fma(a, x(i3), k.at(fm + i0));
      k.at(fm + i3) = fma(a, x(i0), k.at(fm + i3));
      k.at(fm + i1) = fma(-a, x(i2), k.at(fm + i1));
      k.at(fm + i2) = fma(-a, x(i1), k.at(fm + i2));
    }
  }
  for (int i = 0; i < n; ++i)
    for (int v = 0; v < nv; ++v) {
      double f = k.at(fk + i * nv + v);
      for (int j = 0; j < n; ++j) f = fma(-B(j, i), k.at(fm + j * nv + v), f);
      k.at(fk + i * nv + v) = f;
    }
}

// Columns j0 .. j0 + JC - 1 of electron e's rows of G_A (with its part through B,
// dA = G_A - (lap U + |grad U|^2) G_B / 2) and G_B.
template <int JC>
__device__ inline void adj_el_g_rows(const qmc_wf_desc& d, const AdjShape& A, const GradWork& k,
                                     const AdjCold& cold, int e, int j0, double (&ga)[JC],
                                     double (&gb)[JC]) {
  const GradShape& S = A.g;
  const int s = e < d.nup ? 0 : 1, r0 = s ? d.nup : 0, n = s ? d.ndown : d.nup;
  const int nmu = d.nmo_used, nmax = d.nup > d.ndown ? d.nup : d.ndown, i = e - r0;
  const MView<double> L = grad_view(k, S.lu, r0, nmu), B = grad_view(k, A.bk, r0, nmu);
  const double lj = -0.5 * k.at(A.jt + 8 * e + 3);
  if (k.at(S.val + GV_G + s) != 0.0) {
    const MView<double> GB = adj_cold(cold, 4 * (int64_t)nmax * nmax + (int64_t)r0 * nmu, nmu);
#pragma unroll
    for (int jj = 0; jj < JC; ++jj) {
      gb[jj] = j0 + jj < nmu ? GB(i, j0 + jj) : 0.0;
      ga[jj] = j0 + jj < nmu ? fma(lj, gb[jj], L(i, j0 + jj)) : 0.0;
    }
    return;
  }
  const int y = S.y + e * nmax, nv = d.max_orb[s] - n, fm = A.fm + s * S.fs, fk = A.fk + s * S.fs;
#pragma unroll
  for (int jj = 0; jj < JC; ++jj) {
    ga[jj] = 0.0;
    gb[jj] = j0 + jj < n ? k.at(y + j0 + jj) : 0.0;
  }
  for (int c = 0; c < n; ++c) {  // -(Y_occ A^-1)^T
    const double yc = k.at(y + c);
#pragma unroll
    for (int jj = 0; jj < JC; ++jj)
      if (j0 + jj < n) ga[jj] = fma(-B(j0 + jj, c), yc, ga[jj]);
  }
  for (int v = 0; v < nv; ++v) {
    double pv = 0.0, kv = 0.0;
    for (int c = 0; c < n; ++c) {
      pv = fma(k.at(y + c), k.at(fm + c * nv + v), pv);
      kv = fma(k.at(y + c), k.at(fk + c * nv + v), kv);
    }
#pragma unroll
    for (int jj = 0; jj < JC; ++jj) {
      if (j0 + jj < n) {
        const double xv = L(j0 + jj, n + v);
        gb[jj] = fma(-pv, xv, gb[jj]);
        ga[jj] = fma(-pv, B(j0 + jj, n + v), fma(-kv, xv, ga[jj]));
      }
      if (j0 + jj == n + v) {
        gb[jj] = pv;
        ga[jj] = kv;
      }
    }
  }
#pragma unroll
  for (int jj = 0; jj < JC; ++jj) ga[jj] = fma(lj, gb[jj], ga[jj]);
}

// One electron's position, Jastrow gradient and G columns in the AO pass.
template <int JC>
struct AdjElectron {
  double x[3], gu[3], ga[JC], gb[JC];
};

// Gradients of the W columns j0 .. j0 + nj - 1 and of the exponents from the
// block's electrons (thread t < ncols holds one, with zero G where it has none):
// the AO groups go through the tile a few at a time. dg[3] (E_L) gets
// -sum_a hb_a grad AO_a, the adjoint of grad U. Every thread of the block calls it.
template <bool EL, int JC, bool FIXED>
__device__ inline void adj_ao_pass(const qmc_wf_desc& d, const GradTables& tb,
                                   const AdjShape& A, double* tile, int ncols,
                                   const AdjElectron<JC>& el, int j0, int nj,
                                   const int* __restrict__ w_entry, double* __restrict__ sums,
                                   double (&dg)[3]) {
  const Tables<double>& t = tb.t;
  const int tid = threadIdx.x, ts = A.ts, nmu = d.nmo_used;
  const bool on = tid < ncols;
  // rows per AO: its value and, without own exponents per component, the weights
  // of the exponentials; E_L: also its part through B
  constexpr int kG = EL ? 2 * JC : JC, kT = EL ? 2 : 1, kQ = EL ? 3 : 1;
  double* const gt = tile;
  double* const rt = tile + kG * ts;
  RowG<JC, FIXED> fa, fb;
  if (on) {
#pragma unroll
    for (int jj = 0; jj < JC; ++jj) {
      gt[jj * ts + tid] = el.ga[jj];
      if (EL) gt[(JC + jj) * ts + tid] = -el.gb[jj];
    }
    fa.set(el.ga, tb.ecol + j0);
    if (EL) fb.set(el.gb, tb.ecol + j0);
  }
  auto ncomp = [&](int g) { return t.group_ao[g + 1] - t.group_ao[g]; };
  auto nprim = [&](int g) { return t.group_prim[g + 1] - t.group_prim[g]; };
  // exponents of their own per component, Slater type or uncontracted: the
  // derivative of every weight takes a row
  auto own_rows = [&](int g) {
    return t.radial != QMC_RADIAL_GTO || t.group_split[g] || t.vscale != nullptr;
  };
  auto ao_rows = [&](int g) { return ncomp(g) * (kT + (own_rows(g) ? 0 : kQ)); };
  auto ex_rows = [&](int g) { return own_rows(g) ? ncomp(g) * nprim(g) : nprim(g); };
  int g = 0, x0 = 0;  // next group, and its next exponential row
  while (g < t.ngroup) {
    // as many whole groups as fit, or part of one group's exponential rows
    int g1 = g, used = 0, xn;
    while (g1 < t.ngroup && used + ao_rows(g1) + ex_rows(g1) <= A.rows) {
      used += ao_rows(g1) + ex_rows(g1);
      ++g1;
    }
    const bool part = g1 == g || x0 > 0;
    if (part) {
      g1 = g + 1;
      xn = ex_rows(g) - x0;
      const int room = A.rows - ao_rows(g);
      if (xn > room) xn = room;
    } else {
      xn = 0;
    }
    if (on) {
      int row = 0, last = -1;
      double dx = 0.0, dy = 0.0, dz = 0.0, r2 = 0.0, gur = 0.0;
      for (int gi = g; gi < g1; ++gi) {
        const int at = t.group_atom[gi], np = nprim(gi), nc = ncomp(gi), a0 = t.group_ao[gi];
        const int kind = t.group_kind[gi];
        if (at != last) {
          dx = el.x[0] - t.atom_xyz[3 * at];
          dy = el.x[1] - t.atom_xyz[3 * at + 1];
          dz = el.x[2] - t.atom_xyz[3 * at + 2];
          r2 = dx * dx + dy * dy + dz * dz;
          if (EL) gur = el.gu[0] * dx + el.gu[1] * dy + el.gu[2] * dz;
          last = at;
        }
        const bool own = own_rows(gi), sto = t.radial != QMC_RADIAL_GTO;
        const int e0 = part ? x0 : 0, en = part ? xn : ex_rows(gi);  // this pass's rows
        double* const er = rt + (row + ao_rows(gi)) * ts + tid;      // the first of them
        auto prim = [&](int p) {  // exponential of group primitive p
          const double ar = t.alpha[t.group_prim[gi] + p] * r2;
          return above_zero(ar) ? 0.0 : rexp(-ar);
        };
        if (!own)
          for (int p = e0; p < e0 + en; ++p) er[(p - e0) * ts] = prim(p);
        double sh[2][3];  // radial sums that components share
        for (int c = 0; c < nc; ++c) {
          const int a = a0 + c, wo = t.ao_wofs[a];
          const int kx = t.ao_k[3 * a], ky = t.ao_k[3 * a + 1], kz = t.ao_k[3 * a + 2];
          const int l = kx + ky + kz;
          const double px = pk0(dx, kx), py = pk0(dy, ky), pz = pk0(dz, kz), P = px * py * pz;
          double qx = 0.0, qy = 0.0, qz = 0.0, lapP = 0.0;
          if (EL) {
            qx = pk1(dx, kx) * py * pz;
            qy = px * pk1(dy, ky) * pz;
            qz = px * py * pk1(dz, kz);
            if (l > 1)
              lapP = pk2(dx, kx) * py * pz + px * pk2(dy, ky) * pz + px * py * pk2(dz, kz);
          }
          const double vs = t.vscale ? t.vscale[a] : 1.0;
          // weights of the AO and of its part through B
          const int2* const wl = reinterpret_cast<const int2*>(t.W) + (int64_t)a * t.ncol + j0;
          const double ha = fa.dot(wl), hb = EL ? fb.dot(wl) : 0.0;
          AOVal<double> o{};
          if (sto) {
            for (int p = 0; p < np; ++p) {
              const double wg = t.wd[wo + p];
              const AOVal<double> q = sto_from<double, EL>(P, qx, qy, qz, lapP, l, dx, dy, dz, r2,
                                                           t.ao_kr(a), t.walpha[wo + p], vs * wg, wg);
              o.v += q.v;
              if (EL) {
                o.gx += q.gx;
                o.gy += q.gy;
                o.gz += q.gz;
                o.lap += q.lap;
              }
            }
          } else {
            const int share = kind == GK_P ? 0 : (kind == GK_D ? (c == 0 || c == 3 || c == 5 ? 0 : 1) : -1);
            double s0 = 0.0, s1 = 0.0, s2 = 0.0;
            if (share >= 0 && c > share) {
              s0 = sh[share][0];
              s1 = sh[share][1];
              s2 = sh[share][2];
            } else {
              for (int p = 0; p < np; ++p) {
                const double al = own ? t.walpha[wo + p] : t.alpha[t.group_prim[gi] + p];
                double ev;
                if (own) {
                  const double ar = al * r2;
                  ev = above_zero(ar) ? 0.0 : rexp(-ar);
                } else {
                  ev = (p >= e0 && p < e0 + en) ? er[(p - e0) * ts] : prim(p);
                }
                const double we = t.wd[wo + p] * ev;
                s0 += we;
                if (EL) {
                  const double w1 = al * we;
                  s1 += w1;
                  s2 = fma(al, w1, s2);
                }
              }
              if (share >= 0) {
                sh[share][0] = s0;
                sh[share][1] = s1;
                sh[share][2] = s2;
              }
            }
            o = ao_from<double, EL>(P, qx, qy, qz, lapP, l, dx, dy, dz, r2, s0, s1, s2, vs);
          }
          double* const r = rt + row * ts + tid;
          r[0] = o.v;
          if (EL) {
            r[ts] = 0.5 * o.lap + el.gu[0] * o.gx + el.gu[1] * o.gy + el.gu[2] * o.gz;
            if (x0 == 0) {
              dg[0] = fma(-hb, o.gx, dg[0]);
              dg[1] = fma(-hb, o.gy, dg[1]);
              dg[2] = fma(-hb, o.gz, dg[2]);
            }
          }
          row += kT;
          // d/d alpha: value -P r^2 e, and through B with z = alpha r^2
          //   e (-r^2 c0 + hb P [A (1 - z) - 4 z + 2 z^2]),  A = 2 gradU . r + 3 + 2 l
          const double c0 = EL ? ha * P - hb * (el.gu[0] * qx + el.gu[1] * qy + el.gu[2] * qz + 0.5 * lapP)
                               : ha * P;
          const double q2 = EL ? hb * P : 0.0, ca = EL ? fma(2.0, gur, (double)(3 + 2 * l)) : 0.0;
          if (!own) {
            double* const q = rt + row * ts + tid;
            q[0] = EL ? fma(q2, ca, -r2 * c0) : -r2 * c0;
            if (EL) {
              const double rq = q2 * r2;
              q[ts] = -(ca + 4.0) * rq;
              q[2 * ts] = 2.0 * r2 * rq;
            }
            row += kQ;
          } else {
            for (int p = 0; p < np; ++p) {
              const int i = c * np + p;
              if (i < e0 || i >= e0 + en) continue;
              const double al = t.walpha[wo + p];
              double v;
              if (sto) {
                const StoDAlpha sd = sto_dalpha(P, qx, qy, qz, lapP, l, dx, dy, dz, r2, t.ao_kr(a), al);
                v = ha * vs * sd.v;
                if (EL)
                  v -= hb * (0.5 * vs * sd.lap + el.gu[0] * sd.gx + el.gu[1] * sd.gy + el.gu[2] * sd.gz);
              } else {
                const double z = al * r2, ev = above_zero(z) ? 0.0 : rexp(-z);
                // the value and Laplacian carry vs, the gradient does not
                v = -vs * ha * P * r2;
                if (EL) {
                  const double qq = 1.0 - z;
                  const double dlap = -r2 * lapP + P * (8.0 * z - 4.0 * z * z - (double)(6 + 4 * l) * qq);
                  const double dgr = -r2 * (el.gu[0] * qx + el.gu[1] * qy + el.gu[2] * qz) -
                                     2.0 * gur * P * qq;
                  v -= hb * (0.5 * vs * dlap + dgr);
                }
                v *= ev;
              }
              er[(i - e0) * ts] = v;
            }
          }
        }
        row += part ? xn : ex_rows(gi);
      }
    }
    __syncthreads();
    // outputs of these groups: W entries, then exponents; `parts` threads share one
    {
      int row = 0;
      const int parts = A.parts, share = (ncols + parts - 1) / parts;
      int first = 0;  // outputs so far, dealt to the threads in order
      for (int gi = g; gi < g1; ++gi) {
        const int nc = ncomp(gi), np = nprim(gi), a0 = t.group_ao[gi];
        const bool own = own_rows(gi);
        const int ka = kT + (own ? 0 : kQ);
        const int e0 = part ? x0 : 0, en = part ? xn : ex_rows(gi);
        const int nW = x0 == 0 ? nc * nj : 0, nE = own ? en : nc * en, nout = (nW + nE) * parts;
        const double* const er = rt + (row + nc * ka) * ts;
        int o = tid - first % (int)blockDim.x;
        if (o < 0) o += blockDim.x;
        for (; o < nout; o += blockDim.x) {
          const int pt = o % parts, i = o / parts;
          const int c0 = pt * share, c1 = c0 + share < ncols ? c0 + share : ncols;
          if (i < nW) {
            const int c = i / nj, jj = i - c * nj;
            const double* const r = rt + (row + c * ka) * ts;
            const double* const gr = gt + jj * ts;
            double v = 0.0;
#pragma unroll 4
            for (int q = c0; q < c1; ++q) {
              v = fma(r[q], gr[q], v);
              if (EL) v = fma(r[ts + q], gr[JC * ts + q], v);
            }
            sums[(int64_t)pt * A.nparam + (a0 + c) * nmu + j0 + jj] += v;
          } else {
            const int m = i - nW;
            int c, p;
            double v = 0.0;
            if (own) {
              c = (e0 + m) / np;
              p = e0 + m - c * np;
              for (int q = c0; q < c1; ++q) v += er[m * ts + q];
            } else {
              c = m / en;
              p = m - c * en;
              const double* const r = rt + (row + c * ka + kT) * ts;
              const double* const ev = er + p * ts;
              p += e0;
              double v1 = 0.0, v2 = 0.0;
#pragma unroll 4
              for (int q = c0; q < c1; ++q) {
                v = fma(r[q], ev[q], v);
                if (EL) {
                  v1 = fma(r[ts + q], ev[q], v1);
                  v2 = fma(r[2 * ts + q], ev[q], v2);
                }
              }
              if (EL) {
                const double al = t.alpha[t.group_prim[gi] + p];
                v = fma(al, fma(al, v2, v1), v);
              }
            }
            const int wi = t.ao_wofs[a0 + c] + p;
            sums[(int64_t)pt * A.nparam + d.nao * nmu + __ldg(w_entry + wi)] += t.wd[wi] * v;
          }
        }
        first += nout;
        row += nc * ka + en;
      }
    }
    __syncthreads();
    if (part) {
      x0 += xn;
      if (x0 >= ex_rows(g)) {
        x0 = 0;
        ++g;
      }
    } else {
      g = g1;
    }
  }
}

template <bool EL, int JC, bool FIXED>
__global__ void __launch_bounds__(kAdjThreads, 1)
    adjoint_kernel(const __grid_constant__ qmc_wf_desc d, const double* __restrict__ pos,
                   int64_t nw, const double* __restrict__ gout, const int* __restrict__ w_entry,
                   double* __restrict__ scr, int64_t ss, const __grid_constant__ AdjShape A) {
  extern __shared__ __align__(16) unsigned char smem[];
  const GradShape& S = A.g;
  const GradTables tb = grad_tables<FIXED>(d, S, smem);
  const Tables<double>& t = tb.t;
  const int tid = threadIdx.x, ne = d.nelec, nmu = d.nmo_used, nwb = S.nwb;
  const int ncols = nwb * S.nslot, nmax = d.nup > d.ndown ? d.nup : d.ndown;
  const int slot = tid / nwb, wl = tid - slot * nwb;
  const bool on = slot < S.nslot;
  double* const sums = scr + (int64_t)blockIdx.x * A.parts * A.nparam;
  double* const tiles = scr + (int64_t)kAdjBlocks * A.parts * A.nparam;
  double* const cold0 = tiles + adj_scratch_tiles(EL);
  double* tile = reinterpret_cast<double*>(smem + A.o_tile);
  if constexpr (!FIXED) {
    if (A.o_tile < 0) tile = tiles + blockIdx.x * adj_tile_doubles(EL, JC, A.ts);
  }
  for (int i = tid; i < A.parts * A.nparam; i += blockDim.x) sums[i] = 0.0;
  const int64_t ntile = (nw + nwb - 1) / nwb;
  for (int64_t tl = blockIdx.x; tl < ntile; tl += gridDim.x) {
    const int64_t w = tl * nwb + wl, wc = w < nw ? w : nw - 1;  // past the last: repeated, gout 0
    GradWork k;
    if (A.o_work >= 0) {
      k.p0 = reinterpret_cast<double*>(smem + A.o_work);
      k.ws = nwb;
      k.wl = wl;
    } else {
      k.p0 = cold0 + A.cold * ss;
      k.ws = ss;
      k.wl = w;
    }
    k.p = k.p0 + k.wl;
    const AdjCold cold{cold0 + w, ss};
    if (on)
      for (int e = slot; e < ne; e += S.nslot)
        for (int q = 0; q < 3; ++q) k.at(S.pos + 3 * e + q) = pos[wc * 3 * ne + 3 * e + q];
    __syncthreads();
    if constexpr (EL) {
      if (on)
        for (int e = slot; e < ne; e += S.nslot) {
          adj_jastrow(d, S, k, A.jt, e);
          const int j = A.jt + 8 * e;
          ep_rows<FIXED, true, false>(t, tb.ecol, nmu, k.at(S.pos + 3 * e), k.at(S.pos + 3 * e + 1),
                                     k.at(S.pos + 3 * e + 2), k.at(j), k.at(j + 1), k.at(j + 2),
                                     k.at(j + 3), tb.fix, S.nthreads, &k.at(S.mo + e * nmu),
                                     &k.at(A.bk + e * nmu), k.ws, 0, t.ngroup);
        }
      __syncthreads();
      bool sum = false;
      if (tid < 2 * nwb) sum = adj_el_determinants(d, A, k, slot);
      sum = __syncthreads_or(sum);
      auto at = [&](int q) { return AdjCold{cold.p + (q - wl), ss}; };
      if (sum) {
        sum_channels(d, S, k, wl, slot, [&](int s) { adj_sum_values(d, A, k, cold, s); },
                     [&](const GradWork& kq, int, int s, int n) { adj_sum_values_warp(d, A, kq, s, n); });
        __syncthreads();
      }
      if (tid < 2 * nwb) adj_el_adjoints(d, A, k, slot);
      if (sum) {
        __syncthreads();
        sum_channels(d, S, k, wl, slot,
                     [&](int s) { adj_sum_adjoints(d, A, k, cold, s, k.at(S.val + GV_INV), k.at(A.r)); },
                     [&](const GradWork& kq, int q, int s, int n) {
                       adj_sum_adjoints_warp(d, A, kq, at(q), s, n);
                     });
      }
      if (tid < nwb) k.at(A.r + 3) = w < nw ? gout[w] : 0.0;
      __syncthreads();
    } else {
      if (on)
        for (int e = slot; e < ne; e += S.nslot) {
          // log J, and its derivatives with respect to the weights (in `mom`)
          grad_jastrow<true>(d, S, k, e);
          ep_rows<FIXED, false, false>(t, tb.ecol, nmu, k.at(S.pos + 3 * e), k.at(S.pos + 3 * e + 1),
                                      k.at(S.pos + 3 * e + 2), 0.0, 0.0, 0.0, 0.0, tb.fix, S.nthreads,
                                      &k.at(S.mo + e * nmu), nullptr, k.ws, 0, t.ngroup);
        }
      __syncthreads();
      grad_determinant_phases(d, S, k, wl, slot);
      __syncthreads();
      if (tid < nwb) {
        double logj = 0.0, dw = 0.0, dn = 0.0;
        for (int e = 0; e < ne; ++e) {
          logj += k.at(S.ju + e);
          dw += k.at(S.mom + e);
          dn += k.at(S.mom + ne + e);
        }
        // gout J dd: what the CI sum is multiplied with
        const double dd = k.at(S.val + GV_DET) * k.at(S.val + GV_DET + 1);
        k.at(A.r) = (w < nw ? gout[w] : 0.0) * jexp(logj) * dd;
        k.at(A.r + 1) = dw;
        k.at(A.r + 2) = dn;
      }
      __syncthreads();
    }
    // CI weights: an output per thread, summed over the block's walkers
    {
      const GradWork k0{k.p0, k.ws, k.p0, 0};
      const int64_t wb = k.wl - wl;  // the tile's first walker in the arrays
      for (int c = tid; c < d.ncfg; c += blockDim.x) {
        const int u = __ldg(d.cfg_det[0] + c), v = d.ndet[0] + __ldg(d.cfg_det[1] + c);
        double acc = 0.0;
        for (int q = 0; q < nwb; ++q) {
          auto at = [&](int item) { return k0.p0[(int64_t)item * k.ws + wb + q]; };
          const double xu = at(S.dv + u), xv = at(S.dv + v);
          if (EL) {
            const double nn = at(A.ov + u) * xv + xu * at(A.ov + v);
            acc = fma(at(A.r + 3) * at(S.val + GV_INV), fma(-at(A.r), xu * xv, nn), acc);
          } else {
            acc = fma(at(A.r), xu * xv, acc);
          }
        }
        sums[d.nao * nmu + d.nweight + c] += acc;
      }
    }
    // the AO pass, a round of electrons at a time
    double dwj = 0.0, dwn = 0.0;
    for (int b = 0; b < ne; b += S.nslot) {
      const int e = on && b + slot < ne ? b + slot : 0;
      const bool has = on && b + slot < ne;
      const int s = e < d.nup ? 0 : 1;
      AdjElectron<JC> el;
      const double scale = has ? k.at(EL ? A.r + 3 : A.r) : 0.0;
      if (has && k.at(S.val + GV_G + s) == 0.0)
        grad_inverse_column(d, S, k, s, e - (s ? d.nup : 0), S.y + e * nmax);
      if (on)
        for (int q = 0; q < 3; ++q) {
          el.x[q] = k.at(S.pos + 3 * e + q);
          el.gu[q] = EL ? k.at(A.jt + 8 * e + q) : 0.0;
        }
      double dg[3] = {0.0, 0.0, 0.0}, dl = 0.0;
      for (int j0 = 0; j0 < nmu; j0 += JC) {
        if (has) {
          if constexpr (EL)
            adj_el_g_rows<JC>(d, A, k, cold, e, j0, el.ga, el.gb);
          else
            grad_g_row<JC>(d, S, k, e, j0, el.ga);
        }
#pragma unroll
        for (int jj = 0; jj < JC; ++jj) {
          el.ga[jj] = has ? scale * el.ga[jj] : 0.0;
          el.gb[jj] = EL && has ? scale * el.gb[jj] : 0.0;
          if (EL && has && j0 + jj < nmu) dl = fma(-0.5 * el.gb[jj], k.at(S.mo + e * nmu + j0 + jj), dl);
        }
        adj_ao_pass<EL, JC, FIXED>(d, tb, A, tile, ncols, el, j0, nmu - j0 < JC ? nmu - j0 : JC, w_entry,
                            sums, dg);
      }
      if (EL && has) {
        // Pade weights, through grad U and lap U + |grad U|^2
        if (d.use_jastrow) {
          double gdg = 0.0;
          for (int q = 0; q < 3; ++q) {
            const double dgw = k.at(A.jt + 8 * e + 4 + q);
            dwj = fma(dg[q], dgw, dwj);
            gdg = fma(el.gu[q], dgw, gdg);
          }
          dwj = fma(dl, k.at(A.jt + 8 * e + 7) + 2.0 * gdg, dwj);
        }
        if (d.use_jastrow_en) {
          const EnTerms en = en_terms(d, el.x[0], el.x[1], el.x[2]);
          double gdg = 0.0;
          for (int q = 0; q < 3; ++q) {
            dwn = fma(dg[q], en.dg[q], dwn);
            gdg = fma(el.gu[q], en.dg[q], gdg);
          }
          dwn = fma(dl, en.dlap + 2.0 * gdg, dwn);
        }
      }
    }
    // the Pade weights' sums over the block (through the tile)
    if (on) {
      if (EL) {
        tile[tid] = dwj;
        tile[A.ts + tid] = dwn;
      } else {
        const double v = slot == 0 ? k.at(A.r) * k.at(S.val + GV_SIGMA) : 0.0;
        tile[tid] = v * (slot == 0 ? k.at(A.r + 1) : 0.0);
        tile[A.ts + tid] = v * (slot == 0 ? k.at(A.r + 2) : 0.0);
      }
    }
    __syncthreads();
    if (tid < 2) {
      double v = 0.0;
      for (int q = 0; q < (EL ? ncols : nwb); ++q) v += tile[tid * A.ts + q];
      sums[d.nao * nmu + d.nweight + d.ncfg + tid] += v;
    }
    __syncthreads();
  }
}

// Sum of parameter i over the blocks' rows in a fixed order (per-thread strided
// partial sums, then a fixed tree), added to its output: W (row stride ldw),
// exponents, CI weights, Pade weights. One block per parameter.
constexpr int kRedTPB = 128;
static __global__ void __launch_bounds__(kRedTPB) adj_reduce_kernel(
    const double* __restrict__ sums, int nrow, int nparam, int nao, int nmu, int nweight,
    int nent, int ncfg, double* __restrict__ g_W, int ldw, double* __restrict__ g_exp,
    double* __restrict__ g_ci, double* __restrict__ g_jw, double* __restrict__ g_jwn) {
  __shared__ double sh[kRedTPB];
  const int i = blockIdx.x;
  double s = 0.0;
  for (int r = threadIdx.x; r < nrow; r += kRedTPB) s += sums[(int64_t)r * nparam + i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int h = kRedTPB / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  const double v = sh[0];
  const int nw_ = nao * nmu;
  if (i < nw_) {
    g_W[(int64_t)(i / nmu) * ldw + i % nmu] += v;
  } else if (i < nw_ + nweight) {
    if (i - nw_ < nent) g_exp[i - nw_] += v;
  } else if (i < nw_ + nweight + ncfg) {
    g_ci[i - nw_ - nweight] += v;
  } else if (i == nw_ + nweight + ncfg) {
    if (g_jw) g_jw[0] += v;
  } else if (g_jwn) {
    g_jwn[0] += v;
  }
}

// Launch plan, by the rule of grad_plan; the blocks take their tiles in turn, so the
// busiest SM's work is its resident blocks times their tiles.
template <typename K>
static AdjShape adj_plan(const qmc_wf_desc& d, bool el, int jc, K kernel, int64_t nw, bool fixed) {
  int dev = 0, nsm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  AdjShape best = adj_shape(d, el, 1, 2, jc, true, fixed);
  const PlanKey key = plan_key((const void*)kernel, dev, nw, d, best.smem);
  PlanChoice got;
  if (plan_find(key, &got)) {
    best = adj_shape(d, el, got.nwb, got.nslot, jc, got.in_smem, fixed, got.tile);
    best.grid = got.grid;
    return best;
  }
  best.smem = -1;
  double best_cost = 0.0;
  for (int in_smem = 1; in_smem >= 0 && best.smem < 0; --in_smem)
    for (int nwb = 32; nwb >= 1; nwb /= 2)
      for (int per = 1; per <= 8; ++per) {
        const int nslot = (d.nelec + per - 1) / per;
        if (per > 1 && nslot == (d.nelec + per - 2) / (per - 1)) continue;
        AdjShape s = adj_shape(d, el, nwb, nslot, jc, in_smem == 1, fixed);
        if (s.g.nthreads > kAdjThreads || s.smem > 227 * 1024) continue;
        if (prepare_smem(kernel, s.smem) != QMC_OK) continue;
        int occ = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, s.g.nthreads, s.smem) !=
                cudaSuccess ||
            occ < 1) {
          cudaGetLastError();
          continue;
        }
        const int64_t tiles = (nw + nwb - 1) / nwb;
        int64_t grid = tiles < (int64_t)occ * nsm ? tiles : (int64_t)occ * nsm;
        if (grid > kAdjBlocks) grid = kAdjBlocks;
        const int64_t each = (tiles + grid - 1) / grid, on_sm = (grid + nsm - 1) / nsm;
        const double warps = (double)on_sm * s.g.nthreads / 32.0;
        double cost = (double)(each * on_sm * nwb) * per * s.g.nthreads / ((double)nwb * d.nelec);
        if (warps < 12.0) cost *= sqrt(12.0 / warps);
        cost *= 1.0 + 0.05 * (nwb < 16 ? 16.0 / nwb : 1.0);
        if (best.smem < 0 || cost < 0.999 * best_cost) {
          s.grid = (int)((tiles + each - 1) / each);  // even shares
          best = s;
          best_cost = cost;
        }
      }
  if (best.smem < 0 && !fixed) {  // the tables alone
    AdjShape s = adj_shape(d, el, 1, 2, jc, false, fixed, false);
    if (s.smem <= 227 * 1024 && prepare_smem(kernel, s.smem) == QMC_OK) {
      s.grid = (int)(nw < nsm ? nw : nsm);
      best = s;
    }
  }
  if (best.smem >= 0)
    plan_keep(key, {best.g.nwb, best.g.nslot, best.o_work >= 0, best.grid, best.o_tile >= 0});
  return best;
}

struct AdjArgs {
  const double *pos, *gout;
  int64_t nw;
  const int* w_entry;
  int nentries, ldw;
  double *g_exp, *g_W, *g_jw, *g_ci, *scr;
};

template <bool EL, int JC, bool FIXED>
int launch_adjoint(const qmc_wf_desc& d, const AdjArgs& a, cudaStream_t s) {
  const AdjShape A = adj_plan(d, EL, JC, adjoint_kernel<EL, JC, FIXED>, a.nw, FIXED);
  if (A.smem < 0) return QMC_ERR_SHAPE;
  const int st = prepare_smem(adjoint_kernel<EL, JC, FIXED>, A.smem);
  if (st) return st;
  adjoint_kernel<EL, JC, FIXED><<<(unsigned)A.grid, A.g.nthreads, A.smem, s>>>(
      d, a.pos, a.nw, a.gout, a.w_entry, a.scr, pad_walkers(a.nw), A);
  adj_reduce_kernel<<<(unsigned)A.nparam, kRedTPB, 0, s>>>(
      a.scr, A.grid * A.parts, A.nparam, d.nao, d.nmo_used, d.nweight, a.nentries, d.ncfg, a.g_W,
      a.ldw, a.g_exp, a.g_ci, d.use_jastrow ? a.g_jw : nullptr,
      d.use_jastrow_en ? a.g_jw + 1 : nullptr);
  return launch_status();
}

#if !QMC_INST_FIXED
template int launch_adjoint<false, 8, false>(const qmc_wf_desc&, const AdjArgs&, cudaStream_t);
template int launch_adjoint<true, 8, false>(const qmc_wf_desc&, const AdjArgs&, cudaStream_t);
}  // namespace qmc
#else
extern template int launch_adjoint<false, 8, false>(const qmc_wf_desc&, const AdjArgs&,
                                                    cudaStream_t);
extern template int launch_adjoint<true, 8, false>(const qmc_wf_desc&, const AdjArgs&,
                                                   cudaStream_t);

// The checks and the dispatch of both entry points.
template <bool EL>
static int run_adjoint(const qmc_wf_desc* d0, const double* pos, int64_t nw, const double* gout,
                       const int32_t* weight_entry, int32_t nentries, double* grad_exp,
                       double* grad_W, int32_t ldw, double* grad_jastrow_w, double* grad_ci,
                       void* scratch, int64_t scratch_bytes, void* stream) {
  int st = check_desc(d0);
  if (st) return st;
  qmc_wf_desc dd = *d0;
  dd.precision = QMC_PREC_FP64;  // the adjoints are FP64
  if (nw < 0 || nentries < 0 || ldw < dd.nmo_used) return QMC_ERR_ARG;
  if (nw > 0 && (!pos || !gout || !weight_entry || !grad_exp || !grad_W || !grad_ci || !scratch))
    return QMC_ERR_ARG;
  if (nw == 0) return QMC_OK;
  if (scratch_bytes < adj_scratch_bytes(dd, EL, nw)) return QMC_ERR_SCRATCH;
  if (nentries > dd.nweight) return QMC_ERR_ARG;
  const AdjArgs a{pos, gout, nw, weight_entry, nentries, ldw, grad_exp, grad_W, grad_jastrow_w,
                  grad_ci, (double*)scratch};
  // wider columns would not leave registers for the AO pass
  st = QMC_ERR_SHAPE;
  if (fix_applies(dd)) st = launch_adjoint<EL, 8, true>(dd, a, (cudaStream_t)stream);
  if (st == QMC_ERR_SHAPE) st = launch_adjoint<EL, 8, false>(dd, a, (cudaStream_t)stream);
  return st;
}

}  // namespace qmc

using namespace qmc;

extern "C" {

int64_t qmc_adjoint_scratch_bytes(const qmc_wf_desc* d, int64_t nw) {
  if (check_desc(d) != QMC_OK || nw < 0) return -1;
  return adj_scratch_bytes(*d, false, nw);
}

int qmc_wf_psi_adjoint(const qmc_wf_desc* d, const double* pos, int64_t nw, const double* gout,
                       const int32_t* weight_entry, int32_t nentries, double* grad_exp,
                       double* grad_W, int32_t ldw, double* grad_jastrow_w, double* grad_ci,
                       void* scratch, int64_t scratch_bytes, void* stream) {
  return run_adjoint<false>(d, pos, nw, gout, weight_entry, nentries, grad_exp, grad_W, ldw,
                            grad_jastrow_w, grad_ci, scratch, scratch_bytes, stream);
}

int64_t qmc_eloc_adjoint_scratch_bytes(const qmc_wf_desc* d, int64_t nw) {
  if (check_desc(d) != QMC_OK || nw < 0) return -1;
  return adj_scratch_bytes(*d, true, nw);
}

int qmc_wf_local_energy_adjoint(const qmc_wf_desc* d, const double* pos, int64_t nw,
                                const double* gout, const int32_t* weight_entry, int32_t nentries,
                                double* grad_exp, double* grad_W, int32_t ldw,
                                double* grad_jastrow_w, double* grad_ci, void* scratch,
                                int64_t scratch_bytes, void* stream) {
  return run_adjoint<true>(d, pos, nw, gout, weight_entry, nentries, grad_exp, grad_W, ldw,
                           grad_jastrow_w, grad_ci, scratch, scratch_bytes, stream);
}

}  // extern "C"
#endif  // QMC_INST_FIXED
