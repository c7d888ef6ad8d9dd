// AO -> MO contraction of the FP64 kernels in fixed point on the integer pipe.
//
// An FP64 multiply-add takes as long as 64 integer instructions on this GPU; a
// 60 x 60 bit product takes four 32 x 32 -> 64 bit multiply-adds. So the sums
// sum_a v_a W_aj of an electron's MO row are formed from integers: W_aj scaled by a
// power of two per column (its largest entry below 2^59), the AO values of up to
// kFixAOs AOs by one per electron and chunk, both as two signed 30-bit limbs, the
// products of equal weight summed in 64 bits (no overflow for 15 AOs), and the
// total rounded to FP64 once per chunk. The limbs hold six bits more than FP64's
// mantissa at the largest entry: measured against 80-bit arithmetic on 400 walkers
// each, the determinants of H2O (cc-pVDZ), H8 and H24 (sto-3g) come out with 0.4,
// 0.4 and 0.3 of the median error of FP64 multiply-adds, and 0.5, 0.4 and 0.3 of the
// mean. H24, 2048 walkers x 50 steps: 5.82 -> 5.05 ms; H2O, 50003 local energies:
// 1.68 -> 1.48 ms, 5001 walkers x 25 steps: 1.73 -> 1.67 ms.
#pragma once

#include "qmc_device.cuh"

namespace qmc {

// The error is relative to the largest AO value of a chunk times the column's largest entry,
// not to the sum: where an electron lies close to a column's nodal plane, so that the AOs
// that the column has are small against others, multiply-adds keep the entry's own relative
// error and limbs do not (six bits in hand, then a bit lost for every halving). In a
// determinant of several electrons the column's other entries carry the value; the
// determinant of a single electron is that entry. So molecules with one electron of a spin
// take the sums of multiply-adds (ep_plain_rows, PlainG); the AO -> MO layer, whose entries
// are the result, forms such an entry again (mo_kernel).
__host__ __device__ inline bool fix_applies(const qmc_wf_desc& d) {
  return d.nup != 1 && d.ndown != 1;
}

constexpr int kFixAOs = 15;  // AOs per chunk: 15 x 2 x 2^58 < 2^63

// x 2^(59 - e) (e: |x| < 2^e; biased exponent of the bound E = e + 1022) as limbs
// (hi, lo), x = hi 2^30 + lo.
__device__ __forceinline__ int2 fix_limbs(double x, int E) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7FFu), s = E - e;
  uint64_t m = (((uint64_t)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo) << 6;
  m = (e == 0 || s > 60) ? 0 : (m + ((1ull << s) >> 1)) >> s;  // zero and subnormal: 0
  const int64_t v = (hi & 0x80000000u) ? -(int64_t)m : (int64_t)m;
  const int l = (int)((unsigned)v << 2) >> 2;
  return make_int2((int)((v - l) >> 30), l);
}

// hh 2^60 + mid 2^30 + ll in units of 2^(u - 118) as FP64 (rounded once).
__device__ __forceinline__ double fix_value(int64_t hh, int64_t mid, int64_t ll, int u) {
  const __int128 t = ((__int128)hh << 60) + ((__int128)mid << 30) + ll;
  const bool neg = t < 0;
  const unsigned __int128 m = neg ? (unsigned __int128)(-t) : (unsigned __int128)t;
  const uint64_t mh = (uint64_t)(m >> 64), ml = (uint64_t)m;
  if ((mh | ml) == 0) return 0.0;
  const int z = mh ? __clzll((long long)mh) : 64 + __clzll((long long)ml);
  const uint64_t top = (uint64_t)((m << z) >> 64);
  const int ex = 1022 + 127 - z + u - 118;  // exponent field less the implicit bit
  if ((unsigned)ex >= 2046u)  // below FP64's normal range, or beyond it
    return ex < 0 ? 0.0 : (neg ? -INFINITY : INFINITY);
  return __longlong_as_double(
      (long long)(((uint64_t)neg << 63) | (((uint64_t)ex << 52) + (top >> 11) + ((top >> 10) & 1))));
}

// Replaces the block's FP64 W table by limbs in place; ecol[j] = exponent e of
// column j (|W_aj| < 2^e), or kFixNaN for a column with an infinity or NaN. Every
// thread of the block calls it, after a barrier; ends with one.
constexpr int kFixNaN = 1 << 20;
__device__ inline void fix_table(double* W, int nao, int ncol, int* ecol) {
  for (int j = threadIdx.x; j < ncol; j += blockDim.x) {
    int e = 0;
    for (int a = 0; a < nao; ++a) {
      const int x = (__double2hiint(W[a * ncol + j]) >> 20) & 0x7FF;
      e = x > e ? x : e;
    }
    ecol[j] = e == 0x7FF ? kFixNaN : e - 1022;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nao * ncol; i += blockDim.x) {
    const int e = ecol[i % ncol];
    const int2 q = e == kFixNaN ? make_int2(0, 0) : fix_limbs(W[i], e + 1022);
    reinterpret_cast<int2*>(W)[i] = q;
  }
  __syncthreads();
}

// The chunk's products of eight columns. v: the thread's AO values as limbs at
// v[i * vs], i < na; Wl: limbs of the first AO's row of W at the first column (rows of
// ncol).
__device__ __forceinline__ void fix_products(const int2* v, int vs, int na, const int2* Wl,
                                             int ncol, int64_t (&hh)[8], int64_t (&mid)[8],
                                             int64_t (&ll)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) hh[j] = mid[j] = ll[j] = 0;
  for (int i = 0; i < na; ++i) {
    const int2 a = v[i * vs];
    if ((a.x | a.y) == 0) continue;
    const int4* w = reinterpret_cast<const int4*>(Wl + i * ncol);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const int4 q = w[j >> 1];
      hh[j] += (int64_t)a.x * q.x;
      mid[j] += (int64_t)a.x * q.y;
      mid[j] += (int64_t)a.y * q.x;
      ll[j] += (int64_t)a.y * q.y;
      hh[j + 1] += (int64_t)a.x * q.z;
      mid[j + 1] += (int64_t)a.x * q.w;
      mid[j + 1] += (int64_t)a.y * q.z;
      ll[j + 1] += (int64_t)a.y * q.w;
    }
  }
}
// An entry's value from its products; E: biased exponent bound of the AO values, e:
// the column's exponent. An AO or a coefficient that is not finite makes it NaN.
__device__ __forceinline__ double fix_entry(int64_t hh, int64_t mid, int64_t ll, int E, int e) {
  return (E >= 0x7FF || e == kFixNaN) ? nan("") : fix_value(hh, mid, ll, E - 1022 + e);
}
// Adds the chunk's products of n columns to row[j * rs] (first: sets).
__device__ __forceinline__ void fix_rows(const int2* v, int vs, int na, int E, const int2* Wl,
                                         int ncol, const int* ecol, int n, double* row,
                                         int64_t rs, bool first) {
  for (int j0 = 0; j0 < n; j0 += 8) {
    int64_t hh[8], mid[8], ll[8];
    fix_products(v, vs, na, Wl + j0, ncol, hh, mid, ll);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j0 + j < n) {
        const double x = fix_entry(hh[j], mid[j], ll[j], E, ecol[j0 + j]);
        double& r = row[(j0 + j) * rs];
        r = first ? x : r + x;
      }
  }
}

// Weights of an electron's AOs, h_a = sum_j G_j W_aj over N columns, N a multiple of
// eight: G in limbs relative to the largest G_j 2^ecol[j], each eight products as in
// fix_rows.
template <int N>
struct FixG {
  int2 g[N];
  int u;  // h's units are 2^(u - 118); kFixNaN: not finite
  __device__ __forceinline__ void set(const double (&G)[N], const int* ecol) {
    int E = 0;
    bool bad = false;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int e = (__double2hiint(G[j]) >> 20) & 0x7FF, c = ecol[j];
      bad |= e == 0x7FF || (c == kFixNaN && e > 0);
      if (e > 0 && c != kFixNaN) E = e + c > E ? e + c : E;
    }
#pragma unroll
    for (int j = 0; j < N; ++j)
      g[j] = bad || ecol[j] == kFixNaN ? make_int2(0, 0) : fix_limbs(G[j], E - ecol[j]);
    u = bad ? kFixNaN : E - 1022;
  }
  __device__ __forceinline__ double dot(const int2* w) const {
    double h = 0.0;
#pragma unroll
    for (int j0 = 0; j0 < N; j0 += 8) {
      int64_t hh = 0, mid = 0, ll = 0;
#pragma unroll
      for (int j = j0; j < j0 + 8; j += 2) {
        const int4 q = reinterpret_cast<const int4*>(w)[j >> 1];
        hh += (int64_t)g[j].x * q.x + (int64_t)g[j + 1].x * q.z;
        mid += (int64_t)g[j].x * q.y;
        mid += (int64_t)g[j].y * q.x;
        mid += (int64_t)g[j + 1].x * q.w;
        mid += (int64_t)g[j + 1].y * q.z;
        ll += (int64_t)g[j].y * q.y + (int64_t)g[j + 1].y * q.w;
      }
      const double v = fix_value(hh, mid, ll, u);
      h = j0 == 0 ? v : h + v;
    }
    return u == kFixNaN ? nan("") : h;
  }
};

// The same weights with W itself, by FP64 multiply-adds.
template <int N>
struct PlainG {
  double g[N];
  __device__ __forceinline__ void set(const double (&G)[N], const int*) {
#pragma unroll
    for (int j = 0; j < N; ++j) g[j] = G[j];
  }
  __device__ __forceinline__ double dot(const int2* w) const {
    double h = 0.0;
#pragma unroll
    for (int j = 0; j < N; j += 2) {
      const double2 q = reinterpret_cast<const double2*>(w)[j >> 1];
      h = fma(g[j], q.x, h);
      h = fma(g[j + 1], q.y, h);
    }
    return h;
  }
};
template <int N, bool FIXED>
using RowG = typename std::conditional<FIXED, FixG<N>, PlainG<N>>::type;

}  // namespace qmc
