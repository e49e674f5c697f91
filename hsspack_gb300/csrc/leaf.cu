// leaf.cu -- batched eigensolver for the DC leaves (the DSTEQR('I') calls of
// SRC/mdlaed0.f90:262-266).
//
// G lanes per leaf of size m <= 32, 32 / G leaves per one-warp CTA.  Every lane
// of a group runs the implicit QL iteration with a Wilkinson shift (Golub & Van
// Loan, Matrix Computations, sec. 8.3) on its own copy of (D, E), so a group
// needs no exchange, and rotates its own rows of the eigenvector block.  The
// eigenpairs are then sorted ascending (in selection sort's order, as DSTEQR
// ends).  The rank-one cuts of the divide step (mdlaed0.f90:213-219) are applied
// on load: d(first) -= |e(left cut)|, d(last) -= |e(right cut)|.
//
// What bounds it: the serial chain of rotations (each needs the one before),
// and per SM the FP64 pipe, which a warp instruction holds for as long with one
// active lane as with 32.  Hence
//  * one flat loop: a pass of it is one rotation for every lane, whatever
//    column and sweep its leaf is at; sweeps start together once a quarter of
//    the working lanes wait for one.  With nested loops the lanes of a warp
//    take turns (their sweeps differ), so a warp costs the sum over its leaves.
//  * the split test of the next sweep is made as the sweep goes (a bit per
//    off-diagonal), so no scan over E precedes a sweep;
//  * column i + 1 of the eigenvector block stays in registers from one rotation
//    to the next; r and 1 / r of a rotation come from one estimate, each rounded
//    to nearest (but for a divisor in 2^52).
// The arithmetic is the plain loop's to the last bit (the fused multiply-adds are
// written out; tests/test_gpu_bits.py).  A merge takes the signs of its vectors from z, which holds entries
// down to 8 eps: with a shift or rotations an ulp off, leaves of 20 rows and more turned
// a vector's sign in one solve of ten.
// Shared memory is interleaved by lane, so lanes at different columns never
// share a bank.  Leaf stage, one thread per leaf with nested loops before -> now:
// n = 257 (16 leaves of 16 rows) 2.33 -> 0.50 ms, n = 2048 2.10 -> 0.51 ms, 512
// problems (61000 leaves of 8 to 16) 6.37 -> 3.97 ms, n = 32768 (4096 of 8)
// 0.41 -> 0.27 ms.
#include "hss_common.cuh"
#include "hss_kernels.h"
#include "hss_leaf.cuh"

#include <algorithm>

namespace hss {

constexpr int LEAF_MAX = 32;

// bytes of shared memory of one CTA: D, E and R rows of Z per lane
static size_t leaf_smem(int mmax, int R) {
  return (size_t)mmax * 32 * (2 + R) * sizeof(double);
}

template <int G, int R>
__global__ void __launch_bounds__(32)
k_leaf_ql(int nleaf, const int *__restrict__ lstart, const int *__restrict__ lsize, int mmax,
          int nblk, const double *__restrict__ d, const double *__restrict__ e,
          double *__restrict__ Q, long long ldq, double *__restrict__ Dp,
          int *__restrict__ perm, int *__restrict__ status, int2 *__restrict__ sup) {
  extern __shared__ double sm[];
  constexpr int LPW = 32 / G;  // leaves per CTA
  const int lane = threadIdx.x, q = lane / G, g0 = lane % G;
  const int leaf = blockIdx.x * LPW + q;
  double *D = sm + lane;                 // D[i * 32]
  double *E = D + mmax * 32;             // E[i * 32]
  double *Z = E + mmax * 32;             // Z[(c * R + t) * 32]: row g0 + G t, column c
  // once the iteration is done, the E entries of a group's first lane hold two
  // integers per column: rk[c * 64] its rank, rk[c * 64 + 1] scratch
  int *rk = (int *)(sm + (size_t)mmax * 32 + q * G);
  int s = 0, m = 0;
  if (leaf < nleaf) {
    s = lstart[leaf];
    m = lsize[leaf];
  }
  // bit i: E(i) is negligible (the last index always is)
  auto split_mask = [&]() {
    unsigned b = 1u << (m - 1);
    for (int i = 0; i < m - 1; ++i)
      if (negligible(E[i * 32], D[i * 32], D[(i + 1) * 32])) b |= 1u << i;
    return b;
  };
  unsigned mask = 0;
  if (m > 0) {
    for (int i = 0; i < m; ++i) {
      double dv = d[s + i];
      if (i == 0 && s > 0) dv -= fabs(e[s - 1]);
      if (i == m - 1 && s + m < nblk) dv -= fabs(e[s + m - 1]);
      D[i * 32] = dv;
      E[i * 32] = (i < m - 1) ? e[s + i] : 0.0;
#pragma unroll
      for (int t = 0; t < R; ++t) Z[(i * R + t) * 32] = (g0 + G * t == i) ? 1.0 : 0.0;
    }
    mask = split_mask();
  }
  int rows = m;  // rows of the CTA's largest leaf
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rows = max(rows, __shfl_xor_sync(HSS_FULL, rows, o));
  rows = (rows + G - 1) / G;
  int bad = 0, l = 0, mm = 0, i = 0, iter = 0;
  bool done = m == 0, sweeping = false;
  double sn = 1.0, cs = 1.0, p = 0.0, g = 0.0, d1 = 0.0, dprev = 0.0;
  double zc[R];  // this lane's rows of column i + 1
  while (true) {
    const unsigned work = __ballot_sync(HSS_FULL, !done), idle = __ballot_sync(HSS_FULL, !done && !sweeping);
    if (!work) break;
    if (4 * __popc(idle) >= __popc(work) && !done && !sweeping) {
      const unsigned open = ~mask & (0xffffffffu >> (32 - m)) & (0xffffffffu << l);
      if (!open) {
        done = true;
      } else {
        const int nl = __ffs(open) - 1;
        if (nl != l) { l = nl; iter = 0; }
        mm = __ffs(mask & (0xffffffffu << l)) - 1;
        if (++iter > 30 * m) {
          bad = 1;
          done = true;
        } else {
          // Wilkinson's shift; operands are O(||T||) after the block scaling, so a plain
          // sqrt is safe
          const double el = E[l * 32], dl = D[l * 32];
          g = quot_rn(D[(l + 1) * 32] - dl, 2.0 * el);
          const double x0 = fma(g, g, 1.0);
          double r0, ri0;
          if (__double2hiint(x0) < 0x7bf00000) sqrt_rcp_rn(x0, r0, ri0);  // below 2^960
          else r0 = sqrt(x0);
          d1 = D[mm * 32];
          g = d1 - dl + quot_rn(el, g + copysign(r0, g));
          sn = 1.0; cs = 1.0; p = 0.0;
          i = mm - 1;
          dprev = 0.0;
#pragma unroll
          for (int t = 0; t < R; ++t) zc[t] = Z[(mm * R + t) * 32];
          sweeping = true;
        }
      }
    }
    if (sweeping) {  // one rotation of columns i, i + 1
      const double ei = E[i * 32], di = D[i * 32];
      const double f = sn * ei, b = cs * ei;
      const double x = fma(f, f, g * g);
      double r, rinv;
      const int hx = __double2hiint(x);
      if (hx >= 0x03f00000 && hx < 0x7bf00000) {  // 2^-960 <= x < 2^960
        // (sqrt_rcp_rn but for its last bit where r's mantissa is all ones: the test of that
        // in this chain costs 4 % of the stage)
        double y;
        r = sqrt_rn(x, y);
        rinv = fma(y, fma(-r, y, 1.0), y);
        sn = f * rinv;
        cs = g * rinv;
      } else {
        r = hypot(f, g);
        sn = f / r;
        cs = g / r;
      }
      // r = 0 only off the fast path
      if (hx < 0x03f00000 && r == 0.0) {
        D[(i + 1) * 32] = d1 - p;
        if (i + 1 < mm) E[(i + 1) * 32] = 0.0;
        E[mm * 32] = 0.0;
#pragma unroll
        for (int t = 0; t < R; ++t) Z[((i + 1) * R + t) * 32] = zc[t];
        mask = split_mask();
        sweeping = false;
      } else {
        g = d1 - p;
        // 2 cs by its exponent (b = cs E(i) is zero or NaN where that is not 2 cs)
        const double cs2 = __hiloint2double(__double2hiint(cs) + (1 << 20), __double2loint(cs));
        const double w = fma(cs2, b, (di - g) * sn);
        p = sn * w;
        d1 = g + p;
        D[(i + 1) * 32] = d1;
        g = cs * w - b;
        if (i + 1 < mm) {
          E[(i + 1) * 32] = r;
          const unsigned bit = 2u << i;
          mask = negligible(r, d1, dprev) ? mask | bit : mask & ~bit;
        }
        dprev = d1;
        d1 = di;
#pragma unroll
        for (int t = 0; t < R; ++t) {
          if (R > 4 && t >= rows) break;
          const double zi = Z[(i * R + t) * 32];
          Z[((i + 1) * R + t) * 32] = fma(sn, zi, cs * zc[t]);
          zc[t] = fma(cs, zi, -(sn * zc[t]));
        }
        if (i == l) {  // end of the sweep
          d1 = __dsub_rn(d1, p);
          D[l * 32] = d1;
          E[l * 32] = g;
          E[mm * 32] = 0.0;
          const unsigned bit = 1u << l;
          mask = negligible(g, d1, dprev) ? mask | bit : mask & ~bit;
#pragma unroll
          for (int t = 0; t < R; ++t) Z[(l * R + t) * 32] = zc[t];
          sweeping = false;
        }
        --i;
      }
    }
  }
  if (leaf_ranks<G>(m, D, rk, g0)) leaf_ranks_ties(m, D, rk);
  __syncwarp();
  for (int c = g0; c < m; c += G) {
    Dp[s + rk[c * 64]] = D[c * 32];
    perm[s + c] = s + c;
    if (sup) sup[s + c] = make_int2(s, s + m);  // rows the column is written on
  }
  if (bad) atomicMax(status, HSS_LEAF_NOCONV);
  // write the blocks: lanes over the entries, one leaf at a time (coalesced)
  const double *Zw = sm + (size_t)mmax * 64;
  const int *rw = (const int *)(sm + (size_t)mmax * 32);
  for (int k = 0; k < LPW; ++k) {
    const int s2 = __shfl_sync(HSS_FULL, s, k * G), m2 = __shfl_sync(HSS_FULL, m, k * G);
    for (int x = lane; x < m2 * m2; x += 32) {
      const int c = x / m2, r = x - c * m2;
      Q[(long long)(s2 + rw[c * 64 + 2 * k * G]) * ldq + s2 + r] =
          Zw[(c * R + r / G) * 32 + k * G + r % G];
    }
  }
}

template <int G, int R>
static void leaf_launch(int nleaf, const int *lstart, const int *lsize, int mmax, int nblk,
                        const double *d, const double *e, double *Q, long long ldq, double *Dp,
                        int *perm, int *status, int2 *sup, cudaStream_t st) {
  const size_t smem = leaf_smem(mmax, R);
  static size_t attr = 48 * 1024;
  if (smem > attr) {
    cudaFuncSetAttribute(k_leaf_ql<G, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr = smem;
  }
  k_leaf_ql<G, R><<<(nleaf * G + 31) / 32, 32, smem, st>>>(nleaf, lstart, lsize, mmax, nblk, d, e,
                                                           Q, ldq, Dp, perm, status, sup);
}

void launch_leaf(int nleaf, const int *lstart, const int *lsize, int mmax, int nblk,
                 const double *d, const double *e, double *Q, long long ldq, double *Dp, int *perm,
                 int *status, cudaStream_t st, int2 *sup) {
  if (nleaf <= 0) return;
  mmax = std::max(1, std::min(mmax, LEAF_MAX));
  const int G = leaf_lanes(nleaf, mmax);
  const int R = (mmax + G - 1) / G;
#define LEAF_ARGS nleaf, lstart, lsize, mmax, nblk, d, e, Q, ldq, Dp, perm, status, sup, st
#define LEAF_TRY(g, r) if (G == g && R <= r) return leaf_launch<g, r>(LEAF_ARGS)
  LEAF_TRY(1, 8);
  LEAF_TRY(1, 12);
  LEAF_TRY(2, 4);
  LEAF_TRY(2, 6);
  LEAF_TRY(2, 8);
  LEAF_TRY(2, 16);
  LEAF_TRY(4, 4);
  LEAF_TRY(4, 8);
  LEAF_TRY(8, 1);
  LEAF_TRY(8, 2);
  LEAF_TRY(8, 4);
  LEAF_TRY(16, 1);
  LEAF_TRY(16, 2);
  leaf_launch<32, 1>(LEAF_ARGS);  // mmax <= 32 rows
#undef LEAF_TRY
#undef LEAF_ARGS
}

}  // namespace hss
