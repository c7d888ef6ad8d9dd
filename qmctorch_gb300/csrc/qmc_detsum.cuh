// Sums over explicit determinants by a warp, a determinant per lane in registers.
#pragma once

#include <type_traits>

#include "qmc_device.cuh"

namespace qmc {

// The sums over explicit determinants (explicit mode, large ratios). A spin of up to
// kSumN electrons has a warp: a lane factors a determinant (the steps of lu_factor and
// lu_solve in their order). An FP64 instruction takes 64 cycles of the warp's scheduler with
// one lane as with 32, so where the determinants leave lanes over, several lanes have the
// same one and share its rows (sum_lanes), and the sums over the determinants are a lane's
// per row and orbital, the terms handed round by shuffles in the determinants' order: 9
// determinants of 5 electrons take some 150 FP64 instructions instead of 400 with a lane per
// determinant that adds its columns in memory. Larger spins keep a thread's chain over the
// determinants, as explicit mode has it for each of its threads.
constexpr int kSumN = 5;

template <int N>
struct DetRegs {
  double a[N][N], det;     // factors, 1 / U_kk on the diagonal
  int perm[N], cols[N];    // the row of A that row k of the factors came from

  // det_columns' with constant indices
  __device__ __forceinline__ void columns(const qmc_wf_desc& d, int s, int u) {
    const int* const tab = d.det_table[s];
    if (d.det_mode == QMC_DET_EXPLICIT) {
#pragma unroll
      for (int j = 0; j < N; ++j) cols[j] = __ldg(tab + (int64_t)u * N + j);
      return;
    }
    const int nv = d.max_orb[s] - N, ord = __ldg(tab + 5 * u);
    int p0 = -1, c0 = 0, p1 = -1, c1 = 0;  // positions replaced, and by which orbital
    if (ord >= 1) {
      const int i0 = __ldg(tab + 5 * u + 1);
      p0 = i0 / nv;
      c0 = N + i0 % nv;
    }
    if (ord == 2) {
      const int i2 = __ldg(tab + 5 * u + 3);
      p1 = i2 / nv;
      c1 = N + __ldg(tab + 5 * u + 2) % nv;
    }
#pragma unroll
    for (int j = 0; j < N; ++j) cols[j] = j == p1 ? c1 : (j == p0 ? c0 : j);
  }

  // Factors the columns of unique determinant u; row(i, c): MO c of the spin's electron i.
  template <typename Row>
  __device__ __forceinline__ void factor(const qmc_wf_desc& d, int s, int u, const Row& row) {
    columns(d, s, u);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      perm[j] = j;
#pragma unroll
      for (int i = 0; i < N; ++i) a[i][j] = row(i, cols[j]);
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

// This lane's determinant u (none: nd) and its share g of the rows, of `groups`.
struct SumLanes {
  int u, g, groups;
};
__device__ __forceinline__ SumLanes sum_lanes(int nd, int n, int u0) {
  const int lane = threadIdx.x & 31;
  int groups = nd <= 16 ? 32 / nd : 1;
  if (groups > n) groups = n;
  if (groups <= 1) return SumLanes{u0 + lane < nd ? u0 + lane : nd, 0, 1};
  const int g = lane / nd;
  return SumLanes{g < groups ? lane - g * nd : nd, g < groups ? g : 0, groups};
}

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

// Row i0 + g of the sum for every share g: out(i, c) += sum_u x_u[j] over the lanes of that
// share (cols: their orbitals) with cols_u[j] = c, in the determinants' order. on: whether this
// lane holds one. first: out is set. N: the number of columns n as a constant, or 0 (rolled).
template <int N, typename Out>
__device__ __forceinline__ void sum_columns(const SumLanes& l, const int* cols, const double* x,
                                            int n, bool on, int nd, int i0, int nmu, bool first,
                                            const Out& out) {
  const int lane = threadIdx.x & 31, width = 32 / l.groups;
  const int g = lane / width, i = i0 + g, m = nd < 32 ? nd : 32;
  for (int c0 = 0; c0 < nmu; c0 += width) {
    const int c = c0 + lane - g * width;
    const bool live = g < l.groups && i < n && c < nmu;
    double acc = first || !live ? 0.0 : out(i, c);
    for (int q = 0; q < m; ++q) {
      const int src = (g < l.groups ? g * nd : 0) + q;
      double v = 0.0;
      bool hit = false;
      auto take = [&](int j) {
        const int cq = __shfl_sync(0xffffffffu, on ? cols[j] : -1, src);
        const double xq = __shfl_sync(0xffffffffu, x[j], src);
        v = cq == c ? xq : v;
        hit |= cq == c;
      };
      if constexpr (N > 0) {
#pragma unroll
        for (int j = 0; j < N; ++j) take(j);
      } else {
#pragma unroll 1
        for (int j = 0; j < n; ++j) take(j);
      }
      if (hit) acc += v;
    }
    if (live) out(i, c) = acc;
  }
}

// f(ch) for the block's channels ch < nch with flag(ch), a warp each. Every thread of the block
// calls it, with the flags behind a barrier.
template <typename Flag, typename F>
__device__ __forceinline__ void sum_tasks(int nch, const Flag& flag, const F& f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  int t = 0;
  for (int c0 = 0; c0 < nch; c0 += 32) {
    unsigned left = __ballot_sync(0xffffffffu, c0 + lane < nch && flag(c0 + lane));
    for (; left; left &= left - 1, ++t)
      if (t % nwarp == warp) f(c0 + __ffs(left) - 1);
  }
}

// What the configurations with the lane's determinant u of spin s add: f(c_c, a, b) for each
// of them in their order, load(v, a, b) having read what belongs to the other spin's
// determinant v. The configurations are read a lane each.
template <typename Load, typename F>
__device__ __forceinline__ void sum_configs(const qmc_wf_desc& d, int s, int u, const Load& load,
                                            const F& f) {
  const int lane = threadIdx.x & 31;
  for (int c0 = 0; c0 < d.ncfg; c0 += 32) {
    const int c = c0 + lane;
    int uc = -1;
    double w = 0.0, a = 0.0, b = 0.0;
    if (c < d.ncfg) {
      uc = __ldg(d.cfg_det[s] + c);
      w = __ldg(d.ci_weight + c);
      load(__ldg(d.cfg_det[1 - s] + c), a, b);
    }
    unsigned mine = 0;  // the lanes with configurations of this lane's u
    for (int q = 0; q < 32; ++q) mine |= (__shfl_sync(0xffffffffu, uc, q) == u ? 1u : 0u) << q;
    while (__any_sync(0xffffffffu, mine != 0)) {
      const int q = mine ? __ffs(mine) - 1 : 0;
      const double wq = __shfl_sync(0xffffffffu, w, q), aq = __shfl_sync(0xffffffffu, a, q),
                   bq = __shfl_sync(0xffffffffu, b, q);
      if (mine) f(wq, aq, bq);
      mine &= mine - 1;
    }
  }
}

// The determinants of spin s (n electrons) and the traces Tr(A_u^-1 B_u) by a warp:
// mo(i, c), b(i, c) the rows of the spin's electron i; put(u, det, trace).
template <typename M, typename B, typename P>
__device__ __forceinline__ void sum_traces(const qmc_wf_desc& d, int s, int n_, const M& mo,
                                           const B& b, const P& put) {
  sum_dispatch(n_, [&](auto Nc) {
    constexpr int N = decltype(Nc)::value;
    const int nd = d.ndet[s];
    for (int u0 = 0; u0 < nd; u0 += 32) {
      const SumLanes l = sum_lanes(nd, N, u0);
      DetRegs<N> D;
      double tr = 0.0;
      if (l.u < nd) {
        D.factor(d, s, l.u, mo);
#pragma unroll 1
        for (int j = l.g; j < N; j += l.groups) {  // column j of A_u^-1 B_u, its element j
          double y[N];
          int c = 0;
#pragma unroll
          for (int q = 0; q < N; ++q) c = q == j ? D.cols[q] : c;
#pragma unroll
          for (int i = 0; i < N; ++i) y[i] = b(D.perm[i], c);
          D.solve(y);
#pragma unroll
          for (int i = 0; i < N; ++i) tr += i == j ? y[i] : 0.0;
        }
      }
      double all = 0.0;  // the shares' parts, to the first's lane
      for (int g = 0; g < l.groups; ++g)
        all += __shfl_sync(0xffffffffu, tr, (g * nd + (threadIdx.x & 31)) & 31);
      if (l.u < nd && l.g == 0) put(l.u, D.det, l.groups > 1 ? all : tr);
    }
  });
}

}  // namespace qmc
