// Sums over explicit determinants by a warp, a determinant per lane in registers.
#pragma once

#include <type_traits>

#include "qmc_device.cuh"

namespace qmc {

// The sums over explicit determinants (explicit mode, large ratios). A spin of up to
// kSumN electrons has a warp: a lane factors a determinant in registers (the steps of
// lu_factor and lu_solve in their order) and the lanes add their terms one after the
// other, in the determinants' order. As one thread's chain over the determinants,
// with its matrices in memory, the block waited some 190 us for one such walker (H2O:
// HMC 4.19 -> 3.42 ms, E_L adjoint step 2.56 -> 1.89 ms). Larger spins do not fit the
// registers and keep the chain: in explicit mode every thread has one.
constexpr int kSumN = 5;

template <int N>
struct DetRegs {
  double a[N][N], det;     // factors, 1 / U_kk on the diagonal
  int perm[N], cols[N];    // the row of A that row k of the factors came from

  // Factors the columns of unique determinant u; row(i, c): MO c of the spin's electron i.
  template <typename Row>
  __device__ __forceinline__ void factor(const qmc_wf_desc& d, int s, int u, const Row& row) {
    int c[QMC_MAX_NSPIN];
    det_columns(d, s, u, c);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      cols[j] = c[j];
      perm[j] = j;
#pragma unroll
      for (int i = 0; i < N; ++i) a[i][j] = row(i, c[j]);
    }
    det = 1.0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      int p = k;
      double amax = fabs(a[k][k]);
#pragma unroll
      for (int i = k + 1; i < N; ++i) {
        const double v = fabs(a[i][k]);
        if (v > amax) {
          amax = v;
          p = i;
        }
      }
#pragma unroll
      for (int i = k + 1; i < N; ++i) {
        const bool sw = i == p;
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const double x = a[k][j], y = a[i][j];
          a[k][j] = sw ? y : x;
          a[i][j] = sw ? x : y;
        }
        const int x = perm[k], y = perm[i];
        perm[k] = sw ? y : x;
        perm[i] = sw ? x : y;
      }
      if (p != k) det = -det;
      const double akk = a[k][k];
      det *= akk;
      const double inv = akk != 0.0 ? prcp(akk) : 0.0;
      a[k][k] = inv;
#pragma unroll
      for (int i = k + 1; i < N; ++i) {
        const double l = a[i][k] * inv;
        a[i][k] = l;
#pragma unroll
        for (int j = k + 1; j < N; ++j) a[i][j] = fma(-l, a[k][j], a[i][j]);
      }
    }
  }
  // A x = b for b in the factors' row order
  __device__ __forceinline__ void solve(double (&x)[N]) const {
#pragma unroll
    for (int i = 1; i < N; ++i)
#pragma unroll
      for (int k = 0; k < i; ++k) x[i] = fma(-a[i][k], x[k], x[i]);
#pragma unroll
    for (int i = N - 1; i >= 0; --i) {
#pragma unroll
      for (int k = i + 1; k < N; ++k) x[i] = fma(-a[i][k], x[k], x[i]);
      x[i] *= a[i][i];
    }
  }
  __device__ __forceinline__ void unit(int col, double (&x)[N]) const {  // column of A^-1
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = perm[i] == col ? 1.0 : 0.0;
    solve(x);
  }
};

// Calls f with the spin's electron count as a constant; n is 1 .. kSumN.
template <typename F>
__device__ __forceinline__ void sum_dispatch(int n, const F& f) {
  static_assert(kSumN == 5, "the cases below");
  switch (n) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
  }
}

// The determinants of spin s (n electrons) and the traces Tr(A_u^-1 B_u) by a warp:
// mo(i, c), b(i, c) the rows of the spin's electron i; put(u, det, trace).
template <typename M, typename B, typename P>
__device__ __forceinline__ void sum_traces(const qmc_wf_desc& d, int s, int n_, const M& mo,
                                           const B& b, const P& put) {
  sum_dispatch(n_, [&](auto Nc) {
    constexpr int N = decltype(Nc)::value;
    for (int u = threadIdx.x & 31; u < d.ndet[s]; u += 32) {
      DetRegs<N> D;
      D.factor(d, s, u, mo);
      double tr = 0.0;
#pragma unroll
      for (int j = 0; j < N; ++j) {
        double y[N];
#pragma unroll
        for (int i = 0; i < N; ++i) y[i] = b(D.perm[i], D.cols[j]);
        D.solve(y);
        tr += y[j];
      }
      put(u, D.det, tr);
    }
  });
}

}  // namespace qmc
