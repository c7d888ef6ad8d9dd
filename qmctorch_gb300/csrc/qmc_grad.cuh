// Electron-position gradients of log psi for a block of walkers, FP64 (the
// gradient entry point and the Hamiltonian sampler).
//
// grad_i log psi = sum_j G_ij grad MO_j(r_i) / Sigma + grad_i U, where Sigma is
// the CI sum and G = d Sigma / d MO the adjoint of the MO values. G comes from
// one factorisation per spin: with A the occupied block, V the virtual columns
// and X = A^-1 V, every determinant of the excitation expansion is det(A) times
// a polynomial x(X) of degree two at most, so that with F = d Sigma / d X
//   G_virt = A^-T F,   G_occ = Sigma A^-T - G_virt X^T
// (all relative to det A of both spins, which cancel in the logarithmic
// gradient). An explicit configuration set (CAS) sums coef det_u A_u^-T over
// its determinants. The gradient then takes one more pass over the AOs with
// the weights h_a = sum_j G_ij W_aj, instead of contracting every component of
// the AO gradients with W.
//
// What bounds it is the FP64 pipe (2 lanes per clock and SM), so the work is
// counted in FP64 instructions: H2O cc-pVDZ single_double(4,4), about 8,700 per
// walker, against about four times as many with per-determinant inverses and
// AO gradients contracted component by component; the exponentials of the
// second pass are recomputed, on the integer pipe. A block holds nwb walkers
// with nslot threads each (thread t: walker t % nwb, electrons t / nwb,
// + nslot, ...); the per-walker arrays live in shared memory
// ([item][walker]), or in the caller's scratch when they do not fit.
#pragma once

#include <algorithm>
#include <math.h>

#include "qmc_detsum.cuh"
#include "qmc_host.cuh"

namespace qmc {

constexpr int kGradThreads = 512;  // 128 registers
constexpr int kGradSlots = 2 * kFixElAOs > kFixAOs ? 2 * kFixElAOs : kFixAOs;  // AO limbs per thread

struct GradShape {
  int nwb, nslot, nthreads, ncol;
  int64_t smem, o_work;  // o_work < 0: the work arrays are in the scratch
  int64_t o_ecol, o_fix;  // W's column exponents (< 0: W is not in limbs), the threads' AO limbs
  // per-walker arrays, offsets in doubles
  int fs;  // stride of the spins' F
  int pos, mom, mo, lu, f, y, dv, jg, ju, val, piv, total;
};
// entries of `val`: Sigma relative to dd = det A_up det A_down, 1 / Sigma (NaN
// where psi is zero), dd, the determinants, the walker's decision, and whether
// the rows of a spin in `lu` are G itself (1) or the factors and X (0)
enum { GV_SIGMA = 0, GV_INV = 1, GV_DD = 2, GV_DET = 3, GV_ACC = 5, GV_G = 6, GV_N = 8 };
// An excitation ratio above this takes the walker's spin to the sum over explicit
// determinants: where the ground determinant is that much smaller than an excited
// one, the double excitations' 2 x 2 minors of X cancel by about its square. The line lies
// where that stays within the rounding that the explicit sums have as well. Position
// gradients of 10,000 H2O walkers, difference from the explicit sums (their own error: 99.9 %
// below 9e-15, largest 1.4e-14): at 32, where one walker in 22 has such a spin, 99.9 % below
// 4.7e-15 and largest 1.2e-14; at 64 8.4e-15 and 3.7e-14; at 4096 7e-13 and 1e-11. H2O,
// 8192 walkers: two HMC trajectories take 4.22 ms at 32, 4.05 at 4096, 50 drift steps 8.21, 5.73
// and without any sum 4.78.
constexpr double kGradRatio = 32.0;

// fixed: W as limbs (in the tables' place) and slots for the AOs'; else W itself, the least
// shared memory.
inline GradShape grad_shape(const qmc_wf_desc& d, int nwb, int nslot, int jc, bool in_smem,
                            bool fixed = true) {
  GradShape s;
  s.nwb = nwb;
  s.nslot = nslot;
  const int nt = nwb * (nslot > 2 ? nslot : 2);
  s.nthreads = ((nt + 31) / 32) * 32;
  s.ncol = round_up(d.nmo_used, jc);
  const int ne = d.nelec, nmu = d.nmo_used, nmax = d.nup > d.ndown ? d.nup : d.ndown;
  const bool ex = d.det_mode == QMC_DET_EXPLICIT;
  const int v0 = ex ? 0 : d.max_orb[0] - d.nup, v1 = ex ? 0 : d.max_orb[1] - d.ndown;
  const int nv = v0 > v1 ? v0 : v1;
  int o = 0;
  auto take = [&](int n) {
    const int r = o;
    o += n;
    return r;
  };
  s.pos = take(3 * ne);
  s.mom = take(3 * ne);
  s.mo = take(ne * nmu);
  s.lu = take(ne * nmu);
  s.fs = nmax * nv;
  s.f = take(2 * s.fs);
  s.y = take(ne * nmax);
  s.dv = take(d.ndet[0] + d.ndet[1]);
  s.jg = take(3 * ne);
  s.ju = take(ne);
  s.val = take(GV_N);
  s.piv = take((ne + 1) / 2);
  s.total = o;
  s.smem = (tables_smem_bytes<double>(d, s.ncol) + 15) & ~int64_t(15);
  s.o_ecol = -1;
  s.o_fix = s.smem;
  if (fixed) {
    s.o_ecol = s.smem;
    s.o_fix = s.o_ecol + align8((int64_t)s.ncol * 4);
    s.smem = (s.o_fix + (int64_t)s.nthreads * kGradSlots * 8 + 15) & ~int64_t(15);
  }
  s.o_work = -1;
  if (in_smem) {
    s.o_work = s.smem;
    s.smem += (int64_t)s.total * nwb * 8;
  }
  return s;
}

// One thread's view of its walker's arrays.
struct GradWork {
  double* p;
  int64_t ws;
  __device__ __forceinline__ double& at(int item) const { return p[(int64_t)item * ws]; }
  __device__ __forceinline__ int& piv(int base, int e) const {
    // an int array in the doubles' storage: entry e of walker wl at e * ws + wl
    return reinterpret_cast<int*>(p0 + (int64_t)base * ws)[(int64_t)e * ws + wl];
  }
  double* p0;  // walker 0 of the block (or of the scratch)
  int64_t wl;
};

// Jastrow terms of electron e: log J contributions (pairs above e, all nuclei)
// and grad_e log J or, with DW, the derivatives of the former with respect to the
// e-e and e-n weights (in `mom`).
template <bool DW = false>
__device__ inline void grad_jastrow(const qmc_wf_desc& d, const GradShape& S, const GradWork& k,
                                    int e) {
  const double x = k.at(S.pos + 3 * e), y = k.at(S.pos + 3 * e + 1), z = k.at(S.pos + 3 * e + 2);
  double u = 0.0, gx = 0.0, gy = 0.0, gz = 0.0, dw = 0.0, dn = 0.0;
  if (d.use_jastrow_en) {
    const EnTerms en = en_terms(d, x, y, z);
    u = en.u;
    dn = en.du;
    gx = en.g[0];
    gy = en.g[1];
    gz = en.g[2];
  }
  if (d.use_jastrow) {
    const double w = __ldg(d.jastrow_w);
    for (int j = DW ? e + 1 : 0; j < d.nelec; ++j) {
      if (j == e) continue;
      const double dx = x - k.at(S.pos + 3 * j), dy = y - k.at(S.pos + 3 * j + 1),
                   dz = z - k.at(S.pos + 3 * j + 2);
      const double r = psqrt(dx * dx + dy * dy + dz * dz);
      const double iu = prcp(fma(w, r, 1.0));
      const double q = (same_spin(d, e, j) ? 0.25 : 0.5) * iu;
      if (j > e) u = fma(q, r, u);
      if (DW) {
        dw = fma(-q * r, iu * r, dw);
        continue;
      }
      const double c = q * iu * prcp(r);
      gx = fma(c, dx, gx);
      gy = fma(c, dy, gy);
      gz = fma(c, dz, gz);
    }
  }
  k.at(S.ju + e) = u;
  if (DW) {
    k.at(S.mom + e) = dw;
    k.at(S.mom + d.nelec + e) = dn;
    return;
  }
  k.at(S.jg + 3 * e) = gx;
  k.at(S.jg + 3 * e + 1) = gy;
  k.at(S.jg + 3 * e + 2) = gz;
}

// The block's tables (FIXED: W as limbs).
struct GradTables {
  Tables<double> t;
  const int* ecol;
  int2* fix;  // this thread's AO limb slots, stride nthreads
};
template <bool FIXED>
__device__ inline GradTables grad_tables(const qmc_wf_desc& d, const GradShape& S,
                                         unsigned char* smem) {
  GradTables g;
  g.t = load_tables<double>(d, d.nmo_used, S.ncol, smem);
  g.ecol = nullptr;
  g.fix = nullptr;
  if constexpr (FIXED) {
    int* const ecol = reinterpret_cast<int*>(smem + S.o_ecol);
    fix_table(const_cast<double*>(g.t.W), d.nao, S.ncol, ecol);
    g.ecol = ecol;
    g.fix = reinterpret_cast<int2*>(smem + S.o_fix) + threadIdx.x;
  }
  return g;
}

// g += sum_a h(a) grad AO_a at the electron-atom difference (dx, dy, dz), and
// gc += sum_a h(a) P_a G1_a: with grad AO = dP G0 - 2 r P G1 the second part
// is -2 gc times the difference, added once per atom.
template <typename H>
__device__ __forceinline__ void grad_group(const Tables<double>& t, int gi, double dx, double dy,
                                           double dz, double r2, const H& h, double (&g)[3],
                                           double& gc) {
  const int a0 = t.group_ao[gi], nc = t.group_ao[gi + 1] - a0;
  const int kind = t.group_kind[gi];
  if (kind == GK_S && nc == 1) {
    double G0[1], G1[1], G2[1];
    group_radial<double, true, 1>(t, gi, r2, G0, G1, G2);
    gc = fma(h(a0), G1[0], gc);
  } else if (kind == GK_S && nc == 2) {
    double G0[2], G1[2], G2[2];
    group_radial<double, true, 2>(t, gi, r2, G0, G1, G2);
    gc = fma(h(a0), G1[0], gc);
    gc = fma(h(a0 + 1), G1[1], gc);
  } else if (kind == GK_P) {
    double G0[1], G1[1], G2[1];
    group_radial<double, true, 1>(t, gi, r2, G0, G1, G2);
    const double hx = h(a0), hy = h(a0 + 1), hz = h(a0 + 2);
    g[0] = fma(hx, G0[0], g[0]);
    g[1] = fma(hy, G0[0], g[1]);
    g[2] = fma(hz, G0[0], g[2]);
    gc = fma(hx * dx + hy * dy + hz * dz, G1[0], gc);
  } else if (kind == GK_D) {
    double G0[2], G1[2], G2[2];
    group_radial<double, true, 2>(t, gi, r2, G0, G1, G2);
    const double xx = h(a0), xy = h(a0 + 1), xz = h(a0 + 2), yy = h(a0 + 3), yz = h(a0 + 4),
                 zz = h(a0 + 5);
    // P = xx x^2 + ...: its gradient is 2 S r (squares) and M r (mixed products)
    const double sx = xx * dx, sy = yy * dy, sz = zz * dz;
    const double mx = xy * dy + xz * dz, my = xy * dx + yz * dz, mz = xz * dx + yz * dy;
    const double s2 = 2.0 * G0[0];
    g[0] = fma(s2, sx, fma(G0[1], mx, g[0]));
    g[1] = fma(s2, sy, fma(G0[1], my, g[1]));
    g[2] = fma(s2, sz, fma(G0[1], mz, g[2]));
    gc = fma(G1[0], sx * dx + sy * dy + sz * dz, gc);
    gc = fma(0.5 * G1[1], mx * dx + my * dy + mz * dz, gc);
  } else {
    for (int c = 0; c < nc; ++c) {
      // one component at a time, with its own exponents
      const int a = a0 + c, wi0 = t.ao_wofs[a], np = t.group_prim[gi + 1] - t.group_prim[gi];
      double s0 = 0.0, s1 = 0.0;
      for (int p = 0; p < np; ++p) {
        const double al = t.walpha[wi0 + p], ar = al * r2;
        if (above_zero(ar)) continue;
        const double e0 = t.wd[wi0 + p] * rexp(-ar);
        s0 += e0;
        s1 = fma(al, e0, s1);
      }
      const int kx = t.ao_k[3 * a], ky = t.ao_k[3 * a + 1], kz = t.ao_k[3 * a + 2];
      const double px = pk0(dx, kx), py = pk0(dy, ky), pz = pk0(dz, kz), ha = h(a);
      s0 *= ha;
      g[0] = fma(s0, pk1(dx, kx) * py * pz, g[0]);
      g[1] = fma(s0, px * pk1(dy, ky) * pz, g[1]);
      g[2] = fma(s0, px * py * pk1(dz, kz), g[2]);
      gc = fma(ha * s1, px * py * pz, gc);
    }
  }
}

// g += sum_a h(a) grad AO_a of one electron at (x, y, z), over the AO groups
// g0 .. g1 - 1
template <typename H>
__device__ inline void grad_ao_backward(const Tables<double>& t, double x, double y, double z,
                                        const H& h, double (&g)[3], int g0, int g1) {
  if (t.radial != QMC_RADIAL_GTO) {
    auto acc = [&](int a, const AOVal<double>& o) {
      const double ha = h(a);
      g[0] = fma(ha, o.gx, g[0]);
      g[1] = fma(ha, o.gy, g[1]);
      g[2] = fma(ha, o.gz, g[2]);
    };
    for (int gi = g0; gi < g1; ++gi) {
      const int A = t.group_atom[gi];
      const double dx = x - t.atom_xyz[3 * A], dy = y - t.atom_xyz[3 * A + 1],
                   dz = z - t.atom_xyz[3 * A + 2];
      group_sto<double, true>(t, gi, dx, dy, dz, dx * dx + dy * dy + dz * dz, acc);
    }
    return;
  }
  int last = -1;
  double dx = 0.0, dy = 0.0, dz = 0.0, r2 = 0.0, gc = 0.0;
  auto flush = [&]() {
    const double c = -2.0 * gc;
    g[0] = fma(c, dx, g[0]);
    g[1] = fma(c, dy, g[1]);
    g[2] = fma(c, dz, g[2]);
    gc = 0.0;
  };
  for (int gi = g0; gi < g1; ++gi) {
    const int A = t.group_atom[gi];
    if (A != last) {
      if (last >= 0) flush();
      dx = x - t.atom_xyz[3 * A];
      dy = y - t.atom_xyz[3 * A + 1];
      dz = z - t.atom_xyz[3 * A + 2];
      r2 = dx * dx + dy * dy + dz * dz;
      last = A;
    }
    grad_group(t, gi, dx, dy, dz, r2, h, g, gc);
  }
  if (last >= 0) flush();
}

// The spin channels' rows of a walker in the work arrays.
__device__ __forceinline__ MView<double> grad_view(const GradWork& k, int off, int row0, int nmu) {
  return MView<double>{k.p + ((int64_t)off + (int64_t)row0 * nmu) * k.ws, (int64_t)nmu * k.ws, k.ws};
}

// A warp: the determinants of spin s to dst(u), and with ADJ g(i, c) = the sum of coef_u
// det_u A_u^-T over them, coef_u = sum_c c_c D(other spin's).
template <int N, bool ADJ, typename Row, typename Dst, typename Other, typename G>
__device__ __forceinline__ void sum_warp(const qmc_wf_desc& d, int s, const Row& row,
                                         const Dst& dst, const Other& other, const G& g) {
  const int nd = d.ndet[s];
  for (int u0 = 0; u0 < nd; u0 += 32) {
    const SumLanes l = sum_lanes(nd, N, u0);
    DetRegs<N> D;
    if (l.u < nd) {
      D.factor(d, s, l.u, row);
      if (l.g == 0) dst(l.u, D.det);
    }
    if (!ADJ) continue;
    double coef = 0.0;
    sum_configs(d, s, l.u, [&](int v, double& a, double&) { a = other(v); },
                [&](double w, double a, double) { coef = fma(w, a, coef); });
    const bool on = l.u < nd && coef != 0.0;  // a determinant of weight zero adds nothing
    const double scale = on ? coef * D.det : 0.0;
#pragma unroll 1
    for (int i0 = 0; i0 < N; i0 += l.groups) {  // row i of A_u^-T: column i of A_u^-1
      double y[N];
#pragma unroll
      for (int j = 0; j < N; ++j) y[j] = 0.0;
      if (on) {
        D.unit(i0 + l.g, y);
#pragma unroll
        for (int j = 0; j < N; ++j) y[j] *= scale;
      }
      sum_columns<N>(l, D.cols, y, N, on, nd, i0, d.nmo_used, u0 == 0, g);
    }
  }
}

// The matrix of unique determinant u of spin s from the MO rows, factored in the
// spin's part of `y`; returns the determinant.
__device__ __noinline__ inline double grad_factor(const qmc_wf_desc& d, const GradShape& S, const GradWork& k,
                                     int s, int u, int* cols, int* piv) {
  const int n = s ? d.ndown : d.nup, r0 = s ? d.nup : 0, nmu = d.nmo_used;
  const int nmax = d.nup > d.ndown ? d.nup : d.ndown;
  const MView<double> M = grad_view(k, S.mo, r0, nmu);
  const MView<double> A{k.p + ((int64_t)S.y + r0 * nmax) * k.ws, (int64_t)nmax * k.ws, k.ws};
  det_columns(d, s, u, cols);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) A(i, j) = M(i, cols[j]);
  return lu_factor<double>(A, n, piv);
}

__device__ __noinline__ inline void grad_sum_values(const qmc_wf_desc& d, const GradShape& S,
                                             const GradWork& k, int s) {
  int piv[QMC_MAX_NSPIN], cols[QMC_MAX_NSPIN];
  const int dv = S.dv + (s ? d.ndet[0] : 0);
  for (int u = 0; u < d.ndet[s]; ++u) k.at(dv + u) = grad_factor(d, S, k, s, u, cols, piv);
}

// G of spin s summed over the explicit determinants, into its rows of `lu`.
__device__ __noinline__ inline void grad_sum_adjoints(const qmc_wf_desc& d, const GradShape& S,
                                               const GradWork& k, int s) {
  const int n = s ? d.ndown : d.nup, r0 = s ? d.nup : 0, nmu = d.nmo_used;
  const int nmax = d.nup > d.ndown ? d.nup : d.ndown, oth = S.dv + (s ? 0 : d.ndet[0]);
  const MView<double> L = grad_view(k, S.lu, r0, nmu);
  const MView<double> A{k.p + ((int64_t)S.y + r0 * nmax) * k.ws, (int64_t)nmax * k.ws, k.ws};
  int piv[QMC_MAX_NSPIN], cols[QMC_MAX_NSPIN];
  double col[QMC_MAX_NSPIN];
  const MView<double> V{col, 1, 1};
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < nmu; ++j) L(i, j) = 0.0;
  for (int u = 0; u < d.ndet[s]; ++u) {
    double coef = 0.0;
    for (int c = 0; c < d.ncfg; ++c)
      if (__ldg(d.cfg_det[s] + c) == u)
        coef = fma(__ldg(d.ci_weight + c), k.at(oth + __ldg(d.cfg_det[1 - s] + c)), coef);
    if (coef == 0.0) continue;
    const double scale = coef * grad_factor(d, S, k, s, u, cols, piv);
    for (int i = 0; i < n; ++i) {  // row i of A_u^-T: column i of A_u^-1
      for (int j = 0; j < n; ++j) col[j] = i == j ? 1.0 : 0.0;
      lu_solve<double>(A, n, piv, V.c(), V, 1);
      for (int j = 0; j < n; ++j) L(i, cols[j]) = fma(scale, col[j], L(i, cols[j]));
    }
  }
}

// A warp's version of the two above, for a spin of n <= kSumN.
template <bool ADJ>
__device__ __noinline__ inline void grad_sum_warp(const qmc_wf_desc& d, const GradShape& S,
                                                  const GradWork& k, int s, int n) {
  const int r0 = s ? d.nup : 0, dv = S.dv + (s ? d.ndet[0] : 0), oth = S.dv + (s ? 0 : d.ndet[0]);
  const MView<double> M = grad_view(k, S.mo, r0, d.nmo_used), L = grad_view(k, S.lu, r0, d.nmo_used);
  sum_dispatch(n, [&](auto N) {
    sum_warp<decltype(N)::value, ADJ>(
        d, s, [&](int i, int c) { return M(i, c); },
        [&](int u, double det) { if (!ADJ) k.at(dv + u) = det; },
        [&](int u) { return k.at(oth + u); }, [&](int i, int c) -> double& { return L(i, c); });
  });
}

// The block's (walker, spin) channels that sum over explicit determinants: chain(s) for
// this thread's own of more than kSumN electrons, warp(k, wl, s, n) for the others. The flags
// are behind a barrier. k, wl, slot: this thread's.
template <typename Chain, typename Warp>
__device__ __forceinline__ void sum_channels(const qmc_wf_desc& d, const GradShape& S,
                                             const GradWork& k, int wl, int slot,
                                             const Chain& chain, const Warp& warp) {
  const int tid = threadIdx.x, nwb = S.nwb;
  if (tid < 2 * nwb && (slot ? d.ndown : d.nup) > kSumN && k.at(S.val + GV_G + slot) != 0.0)
    chain(slot);
  auto view = [&](int q) {
    GradWork kq = k;
    kq.wl += q - wl;
    kq.p = kq.p0 + kq.wl;
    return kq;
  };
  sum_tasks(
      2 * nwb,
      [&](int ch) {
        const int s = ch / nwb, n = s ? d.ndown : d.nup;
        return n > 0 && n <= kSumN && view(ch - s * nwb).at(S.val + GV_G + s) != 0.0;
      },
      [&](int ch) {
        const int s = ch / nwb, q = ch - s * nwb;
        warp(view(q), q, s, s ? d.ndown : d.nup);
      });
}

// Determinant phase, one thread per (walker, spin): excitation mode factors a
// copy of the MO rows (occupied columns: the LU, virtual columns: X) and writes
// the determinants relative to det A; explicit mode (and a walker with a large
// ratio) leaves the determinants themselves to the sums and returns true.
__device__ inline bool grad_determinants(const qmc_wf_desc& d, const GradShape& S,
                                         const GradWork& k, int s) {
  const int n = s ? d.ndown : d.nup, r0 = s ? d.nup : 0, nmu = d.nmo_used;
  const int nd = d.ndet[s], dv = S.dv + (s ? d.ndet[0] : 0);
  const MView<double> M = grad_view(k, S.mo, r0, nmu), L = grad_view(k, S.lu, r0, nmu);
  int piv[QMC_MAX_NSPIN];
  double det = 1.0;
  bool sum = d.det_mode == QMC_DET_EXPLICIT;
  if (n == 0) {
    for (int u = 0; u < nd; ++u) k.at(dv + u) = 1.0;
  } else if (!sum) {
    const int norb = d.max_orb[s], nv = norb - n;
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < norb; ++j) L(i, j) = M(i, j);
    det = lu_factor<double>(L, n, piv);
    for (int i = 0; i < n; ++i) k.piv(S.piv, r0 + i) = piv[i];
    const MView<double> X{L.p + n * L.cs, L.rs, L.cs};
    if (nv > 0) lu_solve<double>(L, n, piv, X.c(), X, nv);
    excitation_values<double, double>(d, d.det_table[s], s, X.c(), nv > 0 ? nv : 1,
                                      k.p + (int64_t)dv * k.ws, k.ws);
    sum = det == 0.0;
    for (int u = 0; u < nd; ++u)
      sum |= __double2hiint(fabs(k.at(dv + u))) > __double2hiint(kGradRatio);
  }
  if (sum) det = 1.0;
  k.at(S.val + GV_DET + s) = det;
  k.at(S.val + GV_G + s) = sum ? 1.0 : 0.0;
  return sum;
}

// Adjoint phase, one thread per (walker, spin), after both spins'
// determinants: the CI sum, and F unless the spin sums over explicit determinants
// (their G: grad_sums).
__device__ inline void grad_adjoints(const qmc_wf_desc& d, const GradShape& S, const GradWork& k,
                                     int s) {
  const int n = s ? d.ndown : d.nup, r0 = s ? d.nup : 0, nmu = d.nmo_used;
  const int own = S.dv + (s ? d.ndet[0] : 0), oth = S.dv + (s ? 0 : d.ndet[0]);
  const MView<double> L = grad_view(k, S.lu, r0, nmu);
  const int* cu = d.cfg_det[s];
  const int* co = d.cfg_det[1 - s];
  double sigma = 0.0;
  for (int c = 0; c < d.ncfg; ++c)
    sigma = fma(__ldg(d.ci_weight + c),
                k.at(own + __ldg(cu + c)) * k.at(oth + __ldg(co + c)), sigma);
  const double dd = k.at(S.val + GV_DET) * k.at(S.val + GV_DET + 1);
  if (s == 0) {
    k.at(S.val + GV_SIGMA) = sigma;
    k.at(S.val + GV_DD) = dd;
    k.at(S.val + GV_INV) = dd * sigma == 0.0 ? nan("") : 1.0 / sigma;
  }
  if (n == 0 || k.at(S.val + GV_G + s) != 0.0) return;
  const int nv = d.max_orb[s] - n;
  const MView<double> X{L.p + n * L.cs, L.rs, L.cs};
  const int f0 = S.f + s * S.fs;
  for (int i = 0; i < n * nv; ++i) k.at(f0 + i) = 0.0;
  const int* tab = d.det_table[s];
  for (int c = 0; c < d.ncfg; ++c) {
    const int* e = tab + 5 * __ldg(cu + c);
    const int ord = __ldg(e);
    if (ord == 0) continue;
    const double cd = __ldg(d.ci_weight + c) * k.at(oth + __ldg(co + c));
    const int i0 = __ldg(e + 1);
    if (ord == 1) {
      k.at(f0 + i0) += cd;
    } else {  // x = X0 X3 - X1 X2
      const int i1 = __ldg(e + 2), i2 = __ldg(e + 3), i3 = __ldg(e + 4);
      const double x0 = X(i0 / nv, i0 % nv), x1 = X(i1 / nv, i1 % nv), x2 = X(i2 / nv, i2 % nv),
                   x3 = X(i3 / nv, i3 % nv);
      k.at(f0 + i0) = fma(cd, x3, k.at(f0 + i0));
      k.at(f0 + i3) = fma(cd, x0, k.at(f0 + i3));
      k.at(f0 + i1) = fma(-cd, x2, k.at(f0 + i1));
      k.at(f0 + i2) = fma(-cd, x1, k.at(f0 + i2));
    }
  }
}

// Both determinant phases and the sums. Every thread of the block calls it; what it
// writes is behind the caller's next barrier.
__device__ inline void grad_determinant_phases(const qmc_wf_desc& d, const GradShape& S,
                                               const GradWork& k, int wl, int slot) {
  bool sum = false;
  if (threadIdx.x < 2 * S.nwb) sum = grad_determinants(d, S, k, slot);
  sum = __syncthreads_or(sum);
  if (sum) {
    sum_channels(d, S, k, wl, slot, [&](int s) { grad_sum_values(d, S, k, s); },
                 [&](const GradWork& kq, int, int s, int n) { grad_sum_warp<false>(d, S, kq, s, n); });
    __syncthreads();
  }
  if (threadIdx.x < 2 * S.nwb) grad_adjoints(d, S, k, slot);
  if (sum)  // own arrays: nothing of grad_adjoints is read or written
    sum_channels(d, S, k, wl, slot, [&](int s) { grad_sum_adjoints(d, S, k, s); },
                 [&](const GradWork& kq, int, int s, int n) { grad_sum_warp<true>(d, S, kq, s, n); });
}

// Column i of A^-1 of spin s (A y = e_i with the factors in `lu`):
// y[k] = A^-1(k, i) to k.at(dst + k).
__device__ inline void grad_inverse_column(const qmc_wf_desc& d, const GradShape& S,
                                           const GradWork& k, int s, int i, int dst) {
  const int n = s ? d.ndown : d.nup, r0 = s ? d.nup : 0;
  const MView<double> LU = grad_view(k, S.lu, r0, d.nmo_used);
  int at = i;  // where the row interchanges move the one
  for (int r = 0; r < n; ++r) {
    const int p = k.piv(S.piv, r0 + r);
    at = at == r ? p : (at == p ? r : at);
  }
  for (int r = 0; r < n; ++r) {
    double v = r == at ? 1.0 : 0.0;
    for (int c = at; c < r; ++c) v = fma(-LU(r, c), k.at(dst + c), v);
    k.at(dst + r) = v;
  }
  for (int r = n - 1; r >= 0; --r) {
    double v = k.at(dst + r);
    for (int c = r + 1; c < n; ++c) v = fma(-LU(r, c), k.at(dst + c), v);
    k.at(dst + r) = v * LU(r, r);
  }
}

// Columns j0 .. j0 + JC - 1 of G's row of electron e; y_e, column e of A^-1, is
// in `y` where the spin has factors.
template <int JC>
__device__ __forceinline__ void grad_g_row(const qmc_wf_desc& d, const GradShape& S,
                                           const GradWork& k, int e, int j0, double (&G)[JC]) {
  const int s = e < d.nup ? 0 : 1, r0 = s ? d.nup : 0, n = s ? d.ndown : d.nup;
  const int nmu = d.nmo_used, nmax = d.nup > d.ndown ? d.nup : d.ndown;
  const MView<double> L = grad_view(k, S.lu, r0, nmu);
  if (k.at(S.val + GV_G + s) != 0.0) {
#pragma unroll
    for (int jj = 0; jj < JC; ++jj) G[jj] = j0 + jj < nmu ? L(e - r0, j0 + jj) : 0.0;
    return;
  }
  const int y = S.y + e * nmax, norb = d.max_orb[s], nv = norb - n, f0 = S.f + s * S.fs;
  const double sg = k.at(S.val + GV_SIGMA);
#pragma unroll
  for (int jj = 0; jj < JC; ++jj) G[jj] = j0 + jj < n ? sg * k.at(y + j0 + jj) : 0.0;
  for (int v = 0; v < nv; ++v) {  // G_virt = A^-T F, and its part of G_occ
    double f = 0.0;
    for (int c = 0; c < n; ++c) f = fma(k.at(y + c), k.at(f0 + c * nv + v), f);
#pragma unroll
    for (int jj = 0; jj < JC; ++jj) {
      if (j0 + jj < n) G[jj] = fma(-f, L(j0 + jj, n + v), G[jj]);
      if (j0 + jj == n + v) G[jj] = f;
    }
  }
}

// g = sum_j G_ej grad MO_j(r_e): the determinant part of electron e's
// gradient times Sigma (relative to dd).
template <int JC, bool FIXED>
__device__ inline void grad_backward(const qmc_wf_desc& d, const GradTables& t,
                                     const GradShape& S, const GradWork& k, int e, double (&g)[3]) {
  const int s = e < d.nup ? 0 : 1, nmax = d.nup > d.ndown ? d.nup : d.ndown;
  if (k.at(S.val + GV_G + s) == 0.0)
    grad_inverse_column(d, S, k, s, e - (s ? d.nup : 0), S.y + e * nmax);
  g[0] = g[1] = g[2] = 0.0;
  for (int j0 = 0; j0 < d.nmo_used; j0 += JC) {
    double G[JC];
    grad_g_row<JC>(d, S, k, e, j0, G);
    RowG<JC, FIXED> fg;
    fg.set(G, t.ecol + j0);
    auto h = [&](int a) {
      return fg.dot(reinterpret_cast<const int2*>(t.t.W) + (int64_t)a * t.t.ncol + j0);
    };
    grad_ao_backward(t.t, k.at(S.pos + 3 * e), k.at(S.pos + 3 * e + 1), k.at(S.pos + 3 * e + 2), h,
                     g, 0, t.t.ngroup);
  }
}

// Thread roles and work views of a block.
struct GradBlock {
  int slot, wl;
  int64_t w;
  bool on, live;  // an electron slot; of a walker below nw
  GradWork k;
  __device__ GradBlock(const GradShape& S, unsigned char* smem, double* scr, int64_t ss,
                       int64_t nw) {
    const int tid = threadIdx.x;
    slot = tid / S.nwb;
    wl = tid - slot * S.nwb;
    const int64_t w0 = (int64_t)blockIdx.x * S.nwb;
    w = w0 + wl;
    on = slot < S.nslot;
    live = on && w < nw;
    if (S.o_work >= 0) {
      k.p0 = reinterpret_cast<double*>(smem + S.o_work);
      k.ws = S.nwb;
      k.wl = wl;
    } else {
      k.p0 = scr;
      k.ws = ss;
      k.wl = w;
    }
    k.p = k.p0 + k.wl;
  }
};

// Forward, determinant and adjoint phases at the positions in S.pos, which a
// barrier has made visible: afterwards every thread of the walker may call
// grad_backward and read val, jg and ju. Every thread of the block calls it.
template <bool FIXED>
__device__ inline void grad_evaluate(const qmc_wf_desc& d, const GradTables& t,
                                     const GradShape& S, const GradBlock& b) {
  if (b.on)
    for (int e = b.slot; e < d.nelec; e += S.nslot) {
      grad_jastrow(d, S, b.k, e);
      ep_rows<FIXED, false, false>(t.t, t.ecol, d.nmo_used, b.k.at(S.pos + 3 * e),
                                   b.k.at(S.pos + 3 * e + 1), b.k.at(S.pos + 3 * e + 2), 0.0, 0.0,
                                   0.0, 0.0, t.fix, S.nthreads, &b.k.at(S.mo + e * d.nmo_used),
                                   nullptr, b.k.ws, 0, t.t.ngroup);
    }
  __syncthreads();
  grad_determinant_phases(d, S, b.k, b.wl, b.slot);
  __syncthreads();
}

// The launch plans' choices, kept per kernel, device, walker count and the sizes that the
// shapes depend on (a search asks the occupancy calculator some 40 times, 0.1 ms).
struct PlanKey {
  const void* kernel;
  int64_t v[16];
  bool operator==(const PlanKey& o) const {
    return kernel == o.kernel && std::equal(v, v + 16, o.v);
  }
};
struct PlanChoice {
  int nwb, nslot;
  bool in_smem;
  int grid;
  bool tile;
};
inline PlanKey plan_key(const void* kernel, int dev, int64_t nw, const qmc_wf_desc& d,
                        int64_t smem) {
  return PlanKey{kernel, {dev, nw, smem, d.nelec, d.nup, d.ndown, d.nao, d.nmo_used, d.nweight,
                          d.det_mode, d.ncfg, d.max_orb[0], d.max_orb[1], d.ndet[0], d.ndet[1],
                          d.ngroup}};
}
inline std::mutex plan_mutex;
inline std::vector<std::pair<PlanKey, PlanChoice>> plan_choices;  // at most 256
inline bool plan_find(const PlanKey& key, PlanChoice* c) {
  std::lock_guard<std::mutex> g(plan_mutex);
  for (const auto& kv : plan_choices)
    if (kv.first == key) {
      *c = kv.second;
      return true;
    }
  return false;
}
inline void plan_keep(const PlanKey& key, const PlanChoice& c) {
  std::lock_guard<std::mutex> g(plan_mutex);
  if (plan_choices.size() >= 256) plan_choices.clear();
  plan_choices.emplace_back(key, c);
}

// Launch plan. The kernels are FP64 bound (the pipe was 100 % busy on an SM with
// 15 warps), and a warp instruction costs the same with idle lanes, so of the
// block sizes that fit the one with the least warp work on the busiest SM is
// taken: its walkers (whole rounds of resident blocks), times the threads per
// electron of a walker (idle lanes and slots), weighted by too few warps to
// keep the pipe full and by the half-empty warps of the determinant phases;
// ties go to the larger block. 8192 H2O walkers: 32 x 5 threads (2 blocks per
// SM, one round) against 8 x 10 in two rounds, 4.75 -> 3.5 ms for the HMC kernel.
// fixed: of the instance with limbs. Refused (smem < 0) where no block fits; the callers then
// take the instance with eight columns (W's rows are padded to the instance's), and after
// that the one without limbs, which needs no more than the tables.
template <typename K>
inline GradShape grad_plan(const qmc_wf_desc& d, int jc, K kernel, int64_t nw, bool fixed) {
  int dev = 0, nsm = 1;
  cudaGetDevice(&dev);
  GradShape best = grad_shape(d, 1, 2, jc, true, fixed);
  const PlanKey key = plan_key((const void*)kernel, dev, nw, d, best.smem);
  PlanChoice got;
  if (plan_find(key, &got)) return grad_shape(d, got.nwb, got.nslot, jc, got.in_smem, fixed);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  best.smem = -1;
  double best_cost = 0.0;
  for (int in_smem = 1; in_smem >= 0 && best.smem < 0; --in_smem)
    for (int nwb = 32; nwb >= 1; nwb /= 2)
      for (int per = 1; per <= 8; ++per) {
        const int nslot = (d.nelec + per - 1) / per;
        if (per > 1 && nslot == (d.nelec + per - 2) / (per - 1)) continue;
        const GradShape s = grad_shape(d, nwb, nslot, jc, in_smem == 1, fixed);
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
        // walkers of the busiest SM: blocks beyond the resident ones start when a whole
        // round has ended
        const int64_t rounds = (on_sm + occ - 1) / occ;
        const int64_t walkers = (rounds == 1 ? on_sm : rounds * occ) * nwb;
        const double warps = (double)(on_sm < occ ? on_sm : occ) * s.nthreads / 32.0;
        double cost = (double)walkers * per * s.nthreads / ((double)nwb * d.nelec);
        if (warps < 12.0) cost *= sqrt(12.0 / warps);
        cost *= 1.0 + 0.05 * (nwb < 16 ? 16.0 / nwb : 1.0);
        if (best.smem < 0 || cost < 0.999 * best_cost) {
          best = s;
          best_cost = cost;
        }
      }
  if (best.smem >= 0) plan_keep(key, {best.nwb, best.nslot, best.o_work >= 0, 0, false});
  return best;
}

}  // namespace qmc
