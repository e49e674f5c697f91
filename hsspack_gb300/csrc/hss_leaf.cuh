// hss_leaf.cuh -- what the leaf kernels (tridiagonal QL, bidiagonal SVD) share.
#pragma once
#include "hss_common.cuh"

namespace hss {

// |r| <= eps (|a| + |b|).  Exponents decide all but the close cases: with 2^k the
// power of two of max(|a|, |b|), the bound is below 2^(k - 51), so a normal r of at
// least that is not negligible (integer instructions instead of three FP64 ones).
__device__ __forceinline__ bool negligible(double r, double a, double b) {
  const int kr = (__double2hiint(r) & 0x7fffffff) >> 20;
  const int k = max(__double2hiint(a) & 0x7fffffff, __double2hiint(b) & 0x7fffffff) >> 20;
  if (kr > 0 && kr >= k - 51) return false;
  return fabs(r) <= HSS_EPS * (fabs(a) + fabs(b));
}

// integer that orders as the double does (-0 as +0; not for NaN)
__device__ __forceinline__ long long order_key(double v) {
  const long long b = __double_as_longlong(v + 0.0);
  return b < 0 ? b ^ 0x7fffffffffffffffLL : b;
}

// Ranks of the m values D[c * 32] of a G-lane group, each lane (g0 of G) those of
// its own columns, into rk[c * 64]; true on the group's first lane when some are
// equal or unordered (leaf_ranks_ties then).  Called by the whole warp.
template <int G>
__device__ __forceinline__ bool leaf_ranks(int m, const double *D, int *rk, int g0) {
  __syncwarp();
  bool tie = false;
  for (int c = g0; c < m; c += G) {
    const double v = D[c * 32];
    const long long kv = order_key(v);
    int rank = 0;
    tie |= v != v;
    for (int j = 0; j < m; ++j) {
      const long long ku = order_key(D[j * 32]);
      rank += ku < kv;
      tie |= ku == kv && j != c;
    }
    rk[c * 64] = rank;
  }
  const unsigned ties = __ballot_sync(HSS_FULL, tie);
  __syncwarp();
  return g0 == 0 && ((ties >> (threadIdx.x & 31)) & (0xffffffffu >> (32 - G)));
}

// The same with equal (or unordered) values, by one lane: selection sort's own
// order, on the indices.
__device__ __forceinline__ void leaf_ranks_ties(int m, const double *D, int *rk) {
  for (int c = 0; c < m; ++c) rk[c * 64 + 1] = c;
  for (int c = 0; c < m - 1; ++c) {
    int k = c;
    double pmin = D[rk[c * 64 + 1] * 32];
    for (int j = c + 1; j < m; ++j) {
      const double u = D[rk[j * 64 + 1] * 32];
      if (u < pmin) { k = j; pmin = u; }
    }
    const int t = rk[c * 64 + 1];
    rk[c * 64 + 1] = rk[k * 64 + 1];
    rk[k * 64 + 1] = t;
  }
  for (int c = 0; c < m; ++c) rk[rk[c * 64 + 1] * 64] = c;
}

// Lanes per leaf for nleaf leaves of at most mmax rows.  An FP64 warp instruction
// takes 64 cycles of its SM quarter whatever lanes are active and nothing hides
// behind it (measured: a dependent chain and eight independent ones, 1 to 4
// warps per SM, all 64.2 cycles per instruction, 8 warps 128).  So few leaves
// get a warp each, and the group halves once there are more than two warps per
// quarter of the SMs.  Leaf stage of tridiagonal batches, the rule's choice (*) and its
// neighbours, ms:
//   128 leaves of 16 rows   G = 32 0.47   16* 0.50    8 0.62    4 0.79
//   512 of 25               G = 32* 1.15  16 1.35     8 1.71    4 2.48
//   1024 of 16              G = 32 0.76   16* 0.57    8 0.66    4 0.82
//   3800 of 8 to 16         G = 16 1.30    8* 0.92    4 0.83    2 1.11
//   15000 of 8 to 16        G = 4 2.32     2* 2.17    1 2.90
//   61000 of 8 to 16        G = 4 7.85     2* 6.21    1 7.38
//   61000 of 4 to 8         G = 4 2.22     2 1.34     1* 0.97
// Above 12 rows one lane per leaf leaves shared memory for three CTAs on an SM, two lanes
// for five.  Many leaves of 24 to 32 rows would want more lanes for the same reason (15000
// of them: 2* 36.7, 8 16.2).
inline int leaf_lanes(int nleaf, int mmax) {
  int G = 32;
  while (G > 1 && (long long)nleaf * G / 32 > 8 * HSS_SMS) G /= 2;
  while (G > 8 && G / 2 >= mmax) G /= 2;
  if (G == 1 && mmax > 12) G = 2;
  while (G < 32 && (mmax + G - 1) / G > 16) G *= 2;
  return G;
}

}  // namespace hss
