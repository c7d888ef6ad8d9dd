// Hamiltonian Monte Carlo on the device, FP64 (hamiltonian.py:75-201): all
// trajectories of a call in one launch, blocks of walkers with a thread per
// electron (qmc_grad.cuh). One translation unit per MO column chunk: compiled
// with -DQMC_INST_JC=<8|16|24> and, for the instance without limbs, 8 and
// -DQMC_INST_FIXED=0; the instance 8 with limbs holds the C entry points.
#include <cuda_runtime.h>
#include <stdint.h>

#ifndef QMC_INST_FIXED
#define QMC_INST_FIXED 1
#endif

#include "qmc_grad.cuh"
#include "qmc_host.cuh"
#include "qmc_rng.cuh"

namespace qmc {

// ---------------------------------------------------------------------------
// Hamiltonian Monte Carlo (hamiltonian.py:75-201)
// ---------------------------------------------------------------------------
// Per step and walker: momenta p ~ N(0, I) over all 3 Ne coordinates,
// H_start = U(q) + |p|^2 / 2 with U = -log psi^2, a leapfrog trajectory of L
// steps of size eps (half momentum step, L - 1 full position + momentum steps,
// a last position step and half momentum step) with the force
// -grad U = 2 grad psi / psi from the full Jacobi evaluation at each point,
// p negated, and the end point rejected when exp(H_start - H_end) < u. The
// trajectory's positions, momenta and forces live in the walker's work
// arrays (xi, dri, drf); pos holds the chain's current positions.
template <int JC, bool FIXED>
__global__ void __launch_bounds__(kGradThreads) hmc_kernel(const __grid_constant__ qmc_wf_desc d,
                                                           const __grid_constant__ qmc_hmc_args a,
                                                           double* __restrict__ scr, int64_t ss,
                                                           const __grid_constant__ GradShape S) {
  extern __shared__ __align__(16) unsigned char smem[];
  const GradTables t = grad_tables<FIXED>(d, S, smem);
  const GradBlock b(S, smem, scr, ss, a.nwalkers);
  const GradWork& k = b.k;
  const int ne = d.nelec, nc = 3 * ne, tid = threadIdx.x;
  // walkers past the last repeat its positions; they store nothing
  double* const x0 = a.pos + (b.w < a.nwalkers ? b.w : a.nwalkers - 1) * nc;
  const double eps = a.step_size, heps = 0.5 * a.step_size;
  const bool replay = a.momenta != nullptr;
  Rng rng{(uint32_t)a.seed, (uint32_t)(a.seed >> 32), (uint32_t)b.w, 0, 0};
  int nacc = 0, idecor = 0;
  int64_t isnap = 0;
  double h0 = 0.0;  // thread tid < nwb: the walker's starting energy
  // U + |p|^2 / 2 from the electrons' shares in `ju` and in `ekin`
  auto energy = [&](double psq) {
    double logj = 0.0;
    for (int e = 0; e < ne; ++e) logj += k.at(S.ju + e);
    return -2.0 * (logj + log(fabs(k.at(S.val + GV_DD) * k.at(S.val + GV_SIGMA)))) + 0.5 * psq;
  };
  auto momentum_sq = [&]() {
    double psq = 0.0;
    for (int c = 0; c < nc; ++c) psq = fma(k.at(S.mom + c), k.at(S.mom + c), psq);
    return psq;
  };
  for (int istep = 0; istep < a.nstep; ++istep) {
    rng.step = a.step_offset + istep;
    // momenta: replayed, or four to a counter of the step's Philox stream
    // (coordinate c: counter c / 4), drawn by the electron's thread
    if (b.on)
      for (int e = b.slot; e < ne; e += S.nslot) {
        double z[4];
        int have = -1;
        for (int q = 0; q < 3; ++q) {
          const int c = 3 * e + q;
          double p;
          if (replay) {
            p = b.live ? a.momenta[((int64_t)istep * a.nwalkers + b.w) * nc + c] : 0.0;
          } else {
            if (have != c >> 2) {
              have = c >> 2;
              rng.call = (uint32_t)have;
              const U4 r = rng.next();
              rng.normal2(r.x, r.y, z[0], z[1]);
              rng.normal2(r.z, r.w, z[2], z[3]);
            }
            const int i = c & 3;
            p = i == 0 ? z[0] : (i == 1 ? z[1] : (i == 2 ? z[2] : z[3]));
          }
          k.at(S.mom + c) = p;
          k.at(S.pos + c) = x0[c];
        }
      }
    __syncthreads();
    const double psq0 = tid < S.nwb ? momentum_sq() : 0.0;
    // l = 0: the half momentum step from the start and the first position step;
    // then a full step of each, the last momentum step a half one again:
    // p -= f grad U with grad U = -2 grad log psi
    for (int l = 0; l <= a.traj_length; ++l) {
      grad_evaluate<FIXED>(d, t, S, b);
      if (l == 0 && tid < S.nwb) h0 = energy(psq0);
      const double f = (l == 0 || l == a.traj_length) ? heps : eps;
      if (b.on)
        for (int e = b.slot; e < ne; e += S.nslot) {
          double g[3];
          grad_backward<JC, FIXED>(d, t, S, k, e, g);
          const double is = k.at(S.val + GV_INV);
          for (int q = 0; q < 3; ++q) {
            const double gl = fma(g[q], is, k.at(S.jg + 3 * e + q));
            const double p = __dsub_rn(k.at(S.mom + 3 * e + q), __dmul_rn(f, -2.0 * gl));
            k.at(S.mom + 3 * e + q) = p;
            if (l < a.traj_length)
              k.at(S.pos + 3 * e + q) = __dadd_rn(k.at(S.pos + 3 * e + q), __dmul_rn(eps, p));
          }
        }
      __syncthreads();
    }
    // p is negated before the kinetic energy, which its sign does not change
    if (tid < S.nwb) {
      const double h1 = energy(momentum_sq());
      double u;
      if (replay) {
        u = b.w < a.nwalkers ? a.uniforms[(int64_t)istep * a.nwalkers + b.w] : 0.0;
      } else {
        rng.call = (uint32_t)((nc + 3) / 4);
        const U4 r = rng.next();
        u = rng.uniform53(r.x, r.y);
      }
      const bool acc = !(exp(h0 - h1) < u);
      nacc += acc;
      k.at(S.val + GV_ACC) = acc ? 1.0 : 0.0;
    }
    __syncthreads();
    const bool acc = b.on && k.at(S.val + GV_ACC) != 0.0;
    const bool keep = istep >= a.ntherm && idecor % a.ndecor == 0 && a.samples && isnap < a.nsnap;
    if (b.live)
      for (int e = b.slot; e < ne; e += S.nslot)
        for (int q = 0; q < 3; ++q) {
          const int c = 3 * e + q;
          const double x = acc ? k.at(S.pos + c) : x0[c];
          if (acc) x0[c] = x;
          if (keep) a.samples[(isnap * a.nwalkers + b.w) * nc + c] = x;
        }
    if (istep >= a.ntherm) {
      isnap += idecor % a.ndecor == 0;
      ++idecor;
    }
    __syncthreads();  // the decisions and the moments are read
  }
  if (tid < S.nwb && b.w < a.nwalkers && a.accepted) a.accepted[b.w] += nacc;
}

template <int JC, bool FIXED>
int launch_hmc(const qmc_wf_desc& d, const qmc_hmc_args& a, double* scr, cudaStream_t s) {
  const GradShape S = grad_plan(d, JC, hmc_kernel<JC, FIXED>, a.nwalkers, FIXED);
  if (S.smem < 0) return QMC_ERR_SHAPE;
  const int st = prepare_smem(hmc_kernel<JC, FIXED>, S.smem);
  if (st) return st;
  hmc_kernel<JC, FIXED><<<(unsigned)((a.nwalkers + S.nwb - 1) / S.nwb), S.nthreads, S.smem, s>>>(
      d, a, scr, pad_walkers(a.nwalkers), S);
  return launch_status();
}

template int launch_hmc<QMC_INST_JC, QMC_INST_FIXED != 0>(const qmc_wf_desc&, const qmc_hmc_args&,
                                                          double*, cudaStream_t);
}  // namespace qmc

#if QMC_INST_JC == 8 && QMC_INST_FIXED
namespace qmc {
#define QMC_HMC_EXTERN(JC, FIXED)                                                      \
  extern template int launch_hmc<JC, FIXED>(const qmc_wf_desc&, const qmc_hmc_args&, \
                                            double*, cudaStream_t);
QMC_HMC_EXTERN(16, true)
QMC_HMC_EXTERN(24, true)
QMC_HMC_EXTERN(8, false)
#undef QMC_HMC_EXTERN
}  // namespace qmc

using namespace qmc;

extern "C" {

int64_t qmc_hmc_scratch_bytes(const qmc_wf_desc* d, int64_t nw) {
  return qmc_drift_scratch_bytes(d, nw);
}

int qmc_hmc_run(const qmc_wf_desc* d0, const qmc_hmc_args* a, void* scratch,
                int64_t scratch_bytes, void* stream) {
  int st = check_desc(d0);
  if (st) return st;
  if (!a) return QMC_ERR_ARG;
  qmc_wf_desc dd = *d0;
  dd.precision = QMC_PREC_FP64;  // the HMC sampler is FP64
  const qmc_wf_desc* d = &dd;
  if (a->nwalkers < 0 || a->nstep < 0 || a->ntherm < 0 || a->ndecor < 1 || a->nsnap < 0 ||
      a->traj_length < 1 || !(a->step_size > 0.0))
    return QMC_ERR_ARG;
  if ((a->momenta != nullptr) != (a->uniforms != nullptr)) return QMC_ERR_ARG;
  if (a->nwalkers == 0 || a->nstep == 0) return QMC_OK;
  if (!a->pos || !scratch) return QMC_ERR_ARG;
  if (a->nsnap > 0 && !a->samples) return QMC_ERR_ARG;
  if (scratch_bytes < qmc_hmc_scratch_bytes(d, a->nwalkers)) return QMC_ERR_SCRATCH;
  cudaStream_t cs = (cudaStream_t)stream;
  double* const scr = (double*)scratch;
  st = QMC_ERR_SHAPE;
  if (!fix_applies(dd)) return qmc::launch_hmc<8, false>(dd, *a, scr, cs);
  if (d->nmo_used > 16) st = qmc::launch_hmc<24, true>(dd, *a, scr, cs);
  else if (d->nmo_used > 8) st = qmc::launch_hmc<16, true>(dd, *a, scr, cs);
  if (st == QMC_ERR_SHAPE) st = qmc::launch_hmc<8, true>(dd, *a, scr, cs);
  if (st == QMC_ERR_SHAPE) st = qmc::launch_hmc<8, false>(dd, *a, scr, cs);
  return st;
}

}  // extern "C"
#endif
