// Staged kernels behind the module-level API (AO, MO, Jastrow, Slater pooling).
#include <cuda_runtime.h>
#include <stdint.h>

#include "qmc_host.cuh"

namespace qmc {

// ---------------------------------------------------------------------------
// staged kernels of the module-level API
// ---------------------------------------------------------------------------
// AO values and derivatives, a thread per (walker, electron). Blocks stay for
// several items, so that a call loads the basis tables a few times per SM and not
// once per 128 electrons. FP64 pipe bound (exponentials on the integer pipe, one
// radial sum per p shell): H2O cc-pVDZ, 16384 walkers: 201 -> 90 us.
constexpr int kAoBlocks = 152 * 8;
__global__ void __launch_bounds__(128) ao_kernel(const __grid_constant__ qmc_wf_desc d,
                                                 const double* __restrict__ pos, int64_t nw,
                                                 int mode, double* __restrict__ ao,
                                                 double* __restrict__ dao,
                                                 double* __restrict__ d2ao) {
  extern __shared__ __align__(16) unsigned char smem[];
  const Tables<double> t = load_tables<double>(d, 0, 0, smem);
  const int64_t nitem = nw * d.nelec, step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t item = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; item < nitem; item += step) {
    const double* pe = pos + item * 3;  // pos[w][3*ne] row-major == [(w*ne+e)*3]
    const XP<double> ex{pe[0], 0.0}, ey{pe[1], 0.0}, ez{pe[2], 0.0};
    const int64_t row = item * d.nao;
    if (mode == 0) {
      auto put = [&](int a, const AOVal<double>& o) { ao[row + a] = o.v; };
      for_each_ao_ep<double, false, decltype(put), false>(t, ex, ey, ez, put);
    } else {
      auto put = [&](int a, const AOVal<double>& o) {
        if (mode == 1 || mode == 4) {
          dao[(row + a) * 3] = o.gx;
          dao[(row + a) * 3 + 1] = o.gy;
          dao[(row + a) * 3 + 2] = o.gz;
        }
        if (mode == 2 || mode == 4) d2ao[row + a] = o.lap;
        if (mode == 4) ao[row + a] = o.v;
        if (mode == 3) {
          // sum of the gradient: value-path coefficient convention
          // (_sum_gradient_kernel, atomic_orbitals.py:290-307)
          const double vs = t.vscale ? t.vscale[a] : 1.0;
          ao[row + a] = vs * (o.gx + o.gy + o.gz);
        }
      };
      for_each_ao_ep<double, true, decltype(put), false>(t, ex, ey, ez, put);
    }
  }
}

// MO = AO @ W in fixed point (qmc_fixdot.cuh), a thread per row: the row's values
// as limbs in the thread's shared-memory slots, nc columns of W as limbs beside
// them, blockIdx.y counting the column blocks (W's slice is kept to 48 KB so that
// several blocks stay resident). The FP64 kernel was FP64 pipe bound; H2O cc-pVDZ,
// 163840 rows x 25 AOs x 24 MOs: 190 -> 111 us, and 143 with the entries formed again (below).
//
// The limbs' error is relative to the largest AO value and the column's largest entry, but
// each entry here is a result: one below 2^-12 of their product (an electron close to the
// orbital's node or far from its atoms), and one that is not finite, is formed again by
// multiply-adds, on the FP64 pipe, which the limbs leave idle. Relative errors of the entries
// of H2O against a 64-bit mantissa, 40,000 rows: mean 1.3e-15, 99 % below 3.6e-15, 99.9 % below
// 9.0e-14, largest 2.5e-10 (next to a node), by multiply-adds alone 1.5e-15, 8.5e-15, 9.9e-14
// and 2.5e-10. Limbs alone have the same quantiles but fail next to a nodal plane: 7e-12
// where the AOs that the orbital has are 1e-6 of the others.
constexpr int kMoBlocks = 152 * 8;
constexpr int kMoSmall = 12;
__device__ __noinline__ double mo_entry(const double* ao, const double* scf, const double* mod,
                                        int nao, int64_t nmo) {
  double s = 0.0;
  for (int a = 0; a < nao; ++a) s = fma(ao[a], scf[a * nmo] * mod[a * nmo], s);
  return s;
}
__global__ void __launch_bounds__(128) mo_kernel(const __grid_constant__ qmc_wf_desc d,
                                                 const double* __restrict__ ao, int64_t nrows,
                                                 int nc, double* __restrict__ mo) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int nao = d.nao, nt = blockDim.x, tid = threadIdx.x;
  double* const W = reinterpret_cast<double*>(smem);
  int2* const v = reinterpret_cast<int2*>(W + (int64_t)nao * nc) + tid;
  int* const ecol = reinterpret_cast<int*>(reinterpret_cast<int2*>(W + (int64_t)nao * nc) + nt * nao);
  int* const ech = ecol + nc + tid;  // exponent of the row's chunk c at ech[c * nt]
  const int c0 = blockIdx.y * nc, ncol = d.nmo - c0 < nc ? d.nmo - c0 : nc;
  for (int i = tid; i < nao * nc; i += nt) {
    const int a = i / nc, j = i - a * nc;
    const int64_t k = (int64_t)a * d.nmo + c0 + j;
    W[i] = j < ncol ? d.mo_scf[k] * d.mo_modifier[k] : 0.0;
  }
  __syncthreads();
  fix_table(W, nao, nc, ecol);
  const int64_t step = (int64_t)gridDim.x * nt;
  for (int64_t r = (int64_t)blockIdx.x * nt + tid; r < nrows; r += step) {
    const double* ar = ao + r * nao;
    int most = 0;
    for (int a0 = 0, c = 0; a0 < nao; a0 += kFixAOs, ++c) {
      const int na = nao - a0 < kFixAOs ? nao - a0 : kFixAOs;
      int E = 0;
      for (int i = 0; i < na; ++i) {
        const double x = ar[a0 + i];
        const int e = (__double2hiint(x) >> 20) & 0x7FF;
        E = e > E ? e : E;
        v[(a0 + i) * nt] = make_int2(__double2hiint(x), __double2loint(x));
      }
      for (int i = a0; i < a0 + na; ++i) {
        const int2 q = v[i * nt];
        v[i * nt] = fix_limbs(__hiloint2double(q.x, q.y), E);
      }
      ech[c * nt] = E;
      most = E > most ? E : most;
    }
    uint64_t again = 0;  // entries of the last 64 columns
    for (int j0 = 0; j0 < ncol; j0 += 8) {
      double s[8];
      for (int a0 = 0, c = 0; a0 < nao; a0 += kFixAOs, ++c) {
        const int na = nao - a0 < kFixAOs ? nao - a0 : kFixAOs;
        int64_t hh[8], mid[8], ll[8];
        fix_products(v + a0 * nt, nt, na, reinterpret_cast<const int2*>(W) + a0 * nc + j0, nc, hh,
                     mid, ll);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const double x = fix_entry(hh[j], mid[j], ll[j], ech[c * nt], ecol[j0 + j]);
          s[j] = a0 == 0 ? x : s[j] + x;
        }
      }
      double* const out = mo + r * d.nmo + c0;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j0 + j < ncol) {
          const int e = (__double2hiint(s[j]) >> 20) & 0x7FF;
          if (e == 0x7FF || e <= most + ecol[j0 + j] - kMoSmall)
            again |= (uint64_t)1 << ((j0 + j) & 63);
          out[j0 + j] = s[j];
        }
      if ((j0 & 56) != 56 && j0 + 8 < ncol) continue;
      for (; again; again &= again - 1) {
        const int j = (j0 & ~63) + __ffsll((long long)again) - 1;
        out[j] = mo_entry(ar, d.mo_scf + c0 + j, d.mo_modifier + c0 + j, nao, d.nmo);
      }
    }
  }
}
// threads, columns per block and shared memory of mo_kernel
static void mo_shape(const qmc_wf_desc& d, int* nt, int* nc, int64_t* smem) {
  const int64_t all = round_up(d.nmo, 8);
  int64_t c = 49152 / (8 * (int64_t)d.nao) / 8 * 8;
  *nc = (int)(c < 8 ? 8 : (c < all ? c : all));
  const int chunks = (d.nao + kFixAOs - 1) / kFixAOs;
  for (*nt = 128; *nt >= 32; *nt /= 2) {
    *smem = (int64_t)d.nao * *nc * 8 + (int64_t)*nt * d.nao * 8 + 4 * (*nc + (int64_t)chunks * *nt);
    if (*smem <= 112 * 1024 || *nt == 32) break;
  }
}

// Jastrow factor and derivatives per walker, each pair visited from both
// electrons so that no per-electron accumulator is needed.
__global__ void __launch_bounds__(128) jastrow_kernel(const qmc_wf_desc d, const double* __restrict__ pos,
                                                      int64_t nw, double* __restrict__ jast,
                                                      double* __restrict__ djast,
                                                      double* __restrict__ d2jast, int sum_grad) {
  const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nw) return;
  const int ne = d.nelec;
  PosView P{pos + w * 3 * ne, 1};
  const double wj = __ldg(d.jastrow_w);
  const double J = jexp(jastrow_log<double>(d, P, wj));
  if (jast) jast[w] = J;
  if (!djast && !d2jast) return;
  for (int i = 0; i < ne; ++i) {
    double gx = 0, gy = 0, gz = 0, lp = 0;
    const double xi = P(3 * i), yi = P(3 * i + 1), zi = P(3 * i + 2);
    for (int j = 0; j < ne; ++j) {
      if (j == i) continue;
      const double dx = xi - P(3 * j), dy = yi - P(3 * j + 1), dz = zi - P(3 * j + 2);
      const double r = psqrt(dx * dx + dy * dy + dz * dz);
      const double ir = prcp(r);
      const double iu = prcp(1.0 + wj * r);
      const double k1 = (same_spin(d, i, j) ? 0.25 : 0.5) * iu * iu;
      gx += k1 * dx * ir;
      gy += k1 * dy * ir;
      gz += k1 * dz * ir;
      lp += 2.0 * k1 * ir - 2.0 * wj * k1 * iu;
    }
    if (djast) {
      if (sum_grad) {
        djast[w * ne + i] = J * (gx + gy + gz);
      } else {
        djast[(w * 3 + 0) * ne + i] = J * gx;
        djast[(w * 3 + 1) * ne + i] = J * gy;
        djast[(w * 3 + 2) * ne + i] = J * gz;
      }
    }
    if (d2jast) d2jast[w * ne + i] = J * (lp + gx * gx + gy * gy + gz * gz);
  }
}

// Electron-nucleus Pade factor alone and its derivatives per walker
// (JastrowFactorElectronNuclei.forward, jastrow_factor_electron_nuclei.py:66-161):
// J = exp(sum_{i,A} K(r_iA)), grad_i J = J grad_i U, lap_i J = J (lap_i U + |grad_i U|^2).
__global__ void __launch_bounds__(128) jastrow_en_kernel(const qmc_wf_desc d,
                                                         const double* __restrict__ pos, int64_t nw,
                                                         double* __restrict__ jast,
                                                         double* __restrict__ djast,
                                                         double* __restrict__ d2jast, int sum_grad) {
  const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nw) return;
  const int ne = d.nelec;
  PosView P{pos + w * 3 * ne, 1};
  double u = 0.0;
  for (int i = 0; i < ne; ++i) u += en_terms(d, P(3 * i), P(3 * i + 1), P(3 * i + 2)).u;
  const double J = jexp(u);
  if (jast) jast[w] = J;
  if (!djast && !d2jast) return;
  for (int i = 0; i < ne; ++i) {
    const EnTerms en = en_terms(d, P(3 * i), P(3 * i + 1), P(3 * i + 2));
    const double gx = en.g[0], gy = en.g[1], gz = en.g[2];
    if (djast) {
      if (sum_grad) {
        djast[w * ne + i] = J * (gx + gy + gz);
      } else {
        djast[(w * 3 + 0) * ne + i] = J * gx;
        djast[(w * 3 + 1) * ne + i] = J * gy;
        djast[(w * 3 + 2) * ne + i] = J * gz;
      }
    }
    if (d2jast) d2jast[w * ne + i] = J * (en.lap + gx * gx + gy * gy + gz * gz);
  }
}

// A thread per (walker, spin): kTPB walkers and two warps per block, one spin each;
// then the block's threads share the configurations' products.
template <bool OP>
__global__ void __launch_bounds__(2 * kTPB) slater_kernel(const __grid_constant__ qmc_wf_desc d,
                                                          const double* __restrict__ mo,
                                                          const double* __restrict__ bop, int ld,
                                                          int64_t nw, double* __restrict__ dets,
                                                          double* __restrict__ op,
                                                          unsigned char* __restrict__ scr,
                                                          int64_t ss) {
  __shared__ double dref[2][kTPB];
  const int spin = threadIdx.x / kTPB, wl = threadIdx.x - spin * kTPB;
  const int64_t w0 = (int64_t)blockIdx.x * kTPB, w = w0 + wl;
  const Layout L = scratch_layout(d);
  const int ne = d.nelec;
  double* const dv0 = rptr<double>(scr, L.dv, ss, 0);
  double* const ov0 = rptr<double>(scr, L.ov, ss, 0);
  if (w < nw) {
    const int64_t r0 = spin ? d.nup : 0;
    const CView<double> m{mo + (w * ne + r0) * ld, ld, 1};
    const CView<double> b = OP ? CView<double>{bop + (w * ne + r0) * ld, ld, 1} : m;
    const int64_t vm = L.vmax > 0 ? L.vmax : 1;
    auto at = [&](const Region& r, int64_t n) {
      return rptr<double>(scr, r, ss, w) + (spin ? n * ss : 0);
    };
    SpinWork<double> wk;
    wk.LU = MView<double>{at(L.lu, (int64_t)L.nmax * L.nmax), (int64_t)L.nmax * ss, ss};
    wk.X = MView<double>{at(L.x, (int64_t)L.nmax * L.vmax), vm * ss, ss};
    wk.Y = MView<double>{at(L.y, (int64_t)L.nmax * L.omax), (int64_t)L.omax * ss, ss};
    wk.rc = wk.LU;  // unused: FP64 needs no refinement
    wk.X64 = wk.X;
    wk.Y64 = wk.Y;
    const int64_t o = spin ? d.ndet[0] * ss : 0;
    spin_channel<double, OP>(d, spin, m, b, wk,
                             SpinOut<double>{dv0 + w + o, ov0 + w + o, ss, &dref[spin][wl]});
  }
  __syncthreads();  // both spins' values (written by this block) and dref
  const int64_t nb = nw - w0 < kTPB ? nw - w0 : kTPB;
  for (int64_t i = threadIdx.x; i < nb * d.ncfg; i += blockDim.x) {
    const int q = (int)(i / d.ncfg), k = (int)(i - (int64_t)q * d.ncfg);
    const int64_t wq = w0 + q;
    const int iu = __ldg(d.cfg_det[0] + k), idn = __ldg(d.cfg_det[1] + k) + d.ndet[0];
    dets[wq * d.ncfg + k] = (dref[0][q] * dv0[iu * ss + wq]) * (dref[1][q] * dv0[idn * ss + wq]);
    if (OP) op[wq * d.ncfg + k] = ov0[iu * ss + wq] + ov0[idn * ss + wq];
  }
}

__global__ void __launch_bounds__(128) potentials_kernel(const qmc_wf_desc d, const double* __restrict__ pos,
                                                         int64_t nw, double* __restrict__ v_en,
                                                         double* __restrict__ v_ee) {
  const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nw) return;
  const int ne = d.nelec;
  PosView P{pos + w * 3 * ne, 1};
  if (v_en) {
    double v = 0.0;
    for (int e = 0; e < ne; ++e)
      for (int A = 0; A < d.natom; ++A) {
        const double dx = P(3 * e) - __ldg(d.atom_coords + 3 * A),
                     dy = P(3 * e + 1) - __ldg(d.atom_coords + 3 * A + 1),
                     dz = P(3 * e + 2) - __ldg(d.atom_coords + 3 * A + 2);
        v -= pdiv(__ldg(d.atom_charge + A), psqrt(dx * dx + dy * dy + dz * dz));
      }
    v_en[w] = v;
  }
  if (v_ee) {
    double v = 0.0;
    for (int i = 0; i < ne - 1; ++i)
      for (int j = i + 1; j < ne; ++j) {
        const double dx = P(3 * i) - P(3 * j), dy = P(3 * i + 1) - P(3 * j + 1),
                     dz = P(3 * i + 2) - P(3 * j + 2);
        v += prcp(psqrt(dx * dx + dy * dy + dz * dz));
      }
    v_ee[w] = v;
  }
}

}  // namespace qmc

using namespace qmc;

extern "C" {

int qmc_ao_eval(const qmc_wf_desc* d, const double* pos, int64_t nw, int32_t mode, double* ao,
                double* dao, double* d2ao, void* stream) {
  int st = check_desc(d);
  if (st) return st;
  if (nw < 0 || mode < 0 || mode > 4 || (nw > 0 && !pos)) return QMC_ERR_ARG;
  if ((mode == 0 || mode == 3 || mode == 4) && !ao) return QMC_ERR_ARG;
  if ((mode == 1 || mode == 4) && !dao) return QMC_ERR_ARG;
  if ((mode == 2 || mode == 4) && !d2ao) return QMC_ERR_ARG;
  if (nw == 0) return QMC_OK;
  const int64_t smem = tables_smem_bytes<double>(*d, 0);
  if ((st = prepare_smem(ao_kernel, smem))) return st;
  const int64_t blocks = (nw * d->nelec + 127) / 128;
  ao_kernel<<<(unsigned)(blocks < kAoBlocks ? blocks : kAoBlocks), 128, smem,
              (cudaStream_t)stream>>>(*d, pos, nw, mode, ao, dao, d2ao);
  return launch_status();
}

int qmc_mo_eval(const qmc_wf_desc* d, const double* ao, int64_t nrows, double* mo, void* stream) {
  int st = check_desc(d);
  if (st) return st;
  if (nrows < 0 || (nrows > 0 && (!ao || !mo))) return QMC_ERR_ARG;
  if (nrows == 0) return QMC_OK;
  int nt, nc;
  int64_t smem;
  mo_shape(*d, &nt, &nc, &smem);
  if ((st = prepare_smem(mo_kernel, smem))) return st;
  const int64_t blocks = (nrows + nt - 1) / nt;
  const dim3 grid((unsigned)(blocks < kMoBlocks ? blocks : kMoBlocks), (unsigned)((d->nmo + nc - 1) / nc));
  mo_kernel<<<grid, nt, smem, (cudaStream_t)stream>>>(*d, ao, nrows, nc, mo);
  return launch_status();
}

int qmc_jastrow_ee(const qmc_wf_desc* d, const double* pos, int64_t nw, double* jast, double* djast,
                   double* d2jast, int32_t sum_grad, void* stream) {
  int st = check_desc(d);
  if (st) return st;
  if (!d->jastrow_w || nw < 0 || (nw > 0 && !pos)) return QMC_ERR_ARG;
  if (nw == 0) return QMC_OK;
  jastrow_kernel<<<(unsigned)((nw + 127) / 128), 128, 0, (cudaStream_t)stream>>>(*d, pos, nw, jast,
                                                                                 djast, d2jast,
                                                                                 sum_grad);
  return launch_status();
}

int qmc_jastrow_en(const qmc_wf_desc* d, const double* pos, int64_t nw, double* jast,
                   double* djast, double* d2jast, int32_t sum_grad, void* stream) {
  int st = check_desc(d);
  if (st) return st;
  if (!d->use_jastrow_en || nw < 0 || (nw > 0 && !pos)) return QMC_ERR_ARG;
  if (nw == 0) return QMC_OK;
  jastrow_en_kernel<<<(unsigned)((nw + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
      *d, pos, nw, jast, djast, d2jast, sum_grad);
  return launch_status();
}

int qmc_slater(const qmc_wf_desc* d0, const double* mo, const double* bop, int32_t ld, int64_t nw,
               double* dets, double* op, void* scratch, int64_t scratch_bytes, void* stream) {
  int st = check_desc(d0);
  if (st) return st;
  qmc_wf_desc dd = *d0;
  dd.precision = QMC_PREC_FP64;  // the staged pooling kernel is FP64
  const qmc_wf_desc* d = &dd;
  if (nw < 0 || ld < d->nmo_used || (nw > 0 && (!mo || !dets || !scratch))) return QMC_ERR_ARG;
  if (bop && !op) return QMC_ERR_ARG;
  if (nw == 0) return QMC_OK;
  if (scratch_bytes < qmc_scratch_bytes(d, nw, 1)) return QMC_ERR_SCRATCH;
  const int64_t ss = pad_walkers(nw);
  const dim3 grid((unsigned)((nw + kTPB - 1) / kTPB));
  unsigned char* scr = (unsigned char*)scratch;
  if (bop)
    slater_kernel<true><<<grid, 2 * kTPB, 0, (cudaStream_t)stream>>>(dd, mo, bop, ld, nw, dets, op, scr,
                                                                 ss);
  else
    slater_kernel<false><<<grid, 2 * kTPB, 0, (cudaStream_t)stream>>>(dd, mo, nullptr, ld, nw, dets,
                                                                  nullptr, scr, ss);
  return launch_status();
}

int qmc_potentials(const qmc_wf_desc* d, const double* pos, int64_t nw, double* v_en, double* v_ee,
                   void* stream) {
  int st = check_desc(d);
  if (st) return st;
  if (nw < 0 || (nw > 0 && !pos)) return QMC_ERR_ARG;
  if (nw == 0 || (!v_en && !v_ee)) return QMC_OK;
  potentials_kernel<<<(unsigned)((nw + 127) / 128), 128, 0, (cudaStream_t)stream>>>(*d, pos, nw, v_en,
                                                                                    v_ee);
  return launch_status();
}

}  // extern "C"
