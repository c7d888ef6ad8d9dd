// Electron-position gradients of psi and psi^2 (qmc_wf_gradients), FP64:
// grad_i psi = J dd (sum_j G_ij grad MO_j(r_i) + Sigma grad_i U), the Jacobi
// formula of slater_jastrow.py:346-447 with one adjoint matrix per spin
// (qmc_grad.cuh).
#include <cuda_runtime.h>
#include <stdint.h>

#include "qmc_grad.cuh"
#include "qmc_host.cuh"

namespace qmc {

template <int JC, bool FIXED>
__global__ void __launch_bounds__(kGradThreads)
    gradients_kernel(const __grid_constant__ qmc_wf_desc d, const double* __restrict__ pos,
                     int64_t nw, int pdf, double* __restrict__ out, double* __restrict__ scr,
                     int64_t ss, const __grid_constant__ GradShape S) {
  extern __shared__ __align__(16) unsigned char smem[];
  const GradTables t = grad_tables<FIXED>(d, S, smem);
  const GradBlock b(S, smem, scr, ss, nw);
  const GradWork& k = b.k;
  const int ne = d.nelec;
  const double* x = pos + (b.w < nw ? b.w : nw - 1) * 3 * ne;
  if (b.on)
    for (int e = b.slot; e < ne; e += S.nslot)
      for (int q = 0; q < 3; ++q) k.at(S.pos + 3 * e + q) = x[3 * e + q];
  __syncthreads();
  grad_evaluate<FIXED>(d, t, S, b);
  if (!b.live) return;
  double logj = 0.0;
  for (int e = 0; e < ne; ++e) logj += k.at(S.ju + e);
  const double J = jexp(logj), sigma = k.at(S.val + GV_SIGMA), dd = k.at(S.val + GV_DD);
  const double scale = pdf ? 2.0 * J * J * (dd * sigma) * dd : J * dd;
  for (int e = b.slot; e < ne; e += S.nslot) {
    double g[3];
    grad_backward<JC, FIXED>(d, t, S, k, e, g);
    for (int q = 0; q < 3; ++q)
      out[b.w * 3 * ne + 3 * e + q] = scale * fma(sigma, k.at(S.jg + 3 * e + q), g[q]);
  }
}

template <int JC, bool FIXED = true>
static int launch_gradients(const qmc_wf_desc& d, const double* pos, int64_t nw, int pdf,
                            double* out, double* scr, cudaStream_t s) {
  const GradShape S = grad_plan(d, JC, gradients_kernel<JC, FIXED>, nw, FIXED);
  if (S.smem < 0) return QMC_ERR_SHAPE;
  const int st = prepare_smem(gradients_kernel<JC, FIXED>, S.smem);
  if (st) return st;
  gradients_kernel<JC, FIXED><<<(unsigned)((nw + S.nwb - 1) / S.nwb), S.nthreads, S.smem, s>>>(
      d, pos, nw, pdf, out, scr, pad_walkers(nw), S);
  return launch_status();
}

}  // namespace qmc

using namespace qmc;

extern "C" {

// per-walker arrays of the gradient kernel, used when they do not fit shared memory
int64_t qmc_grad_scratch_bytes(const qmc_wf_desc* d, int64_t nw) {
  if (check_desc(d) != QMC_OK || nw < 0) return -1;
  return (int64_t)grad_shape(*d, 1, 2, 8, false).total * pad_walkers(nw) * (int64_t)sizeof(double);
}

int qmc_wf_gradients(const qmc_wf_desc* d0, const double* pos, int64_t nw, int32_t pdf,
                     double* grad, void* scratch, int64_t scratch_bytes, void* stream) {
  int st = check_desc(d0);
  if (st) return st;
  qmc_wf_desc dd = *d0;
  dd.precision = QMC_PREC_FP64;
  const qmc_wf_desc* d = &dd;
  if (nw < 0) return QMC_ERR_ARG;
  if (nw == 0) return QMC_OK;
  if (!pos || !grad || !scratch) return QMC_ERR_ARG;
  if (scratch_bytes < qmc_grad_scratch_bytes(d, nw)) return QMC_ERR_SCRATCH;
  cudaStream_t cs = (cudaStream_t)stream;
  double* scr = (double*)scratch;
  const int p = pdf ? 1 : 0;
  st = QMC_ERR_SHAPE;
  if (!fix_applies(dd)) return launch_gradients<8, false>(dd, pos, nw, p, grad, scr, cs);
  if (d->nmo_used > 16) st = launch_gradients<24>(dd, pos, nw, p, grad, scr, cs);
  else if (d->nmo_used > 8) st = launch_gradients<16>(dd, pos, nw, p, grad, scr, cs);
  if (st == QMC_ERR_SHAPE) st = launch_gradients<8>(dd, pos, nw, p, grad, scr, cs);
  if (st == QMC_ERR_SHAPE) st = launch_gradients<8, false>(dd, pos, nw, p, grad, scr, cs);
  return st;
}

}  // extern "C"
