// svd.cu -- bidiagonal SVD divide and conquer (MDBDSDC, SRC/mdbdsdc.f90:1;
// MDLASD0-3/8, SRC/mdlasd1.f90, SRC/mdlasd2.f90, SRC/mdlasd8.f90).
//
// Storage ("physical slots", as the eigensolver): U (n x n) and V (m x m,
// V = VT^T, right singular vectors as columns) never move their columns.  Slot
// p holds U(:, p), V(:, p) and sigma_p = Dp[p]; a node covering rows
// [s, s + N) has its N triples in slots s .. s + N - 1 and, when it has an extra
// column (sqre = 1), its null vector in V slot s + N.  The center row c = s + nl
// of a merge starts as U(:, c) = e_c, paired with V slot c = the left child's
// null vector (the d_1 = 0 entry of DLASD2).
//
// A merge is the SVD of the K x K "broken arrow" M = e_1 z^T + diag(d),
// d_1 = 0 (after deflation).  Since M^T M = diag(d^2) + z z^T, its right
// singular vectors are the Cauchy-like columns z_i / (d_i^2 - sigma_j^2) and
// U = M V Sigma^-1 gives u_1j = -1, u_ij = d_i z_i / (d_i^2 - sigma_j^2) up to
// column norms (DLASD3).  The secular equation, the Loewner rebuild of z and
// the column norms therefore run through the eigensolver's kernels in their
// squared mode; this file holds the leaf SVDs, the deflation (MDLASD2) and the
// construction of the two K x K vector blocks.
#include "hss_block.cuh"
#include "hss_common.cuh"
#include "hss_kernels.h"
#include "hss_leaf.cuh"
#include "hss_svdprep.cuh"

#include <climits>

namespace hss {

constexpr int SVD_LEAF_MAX = 32;

// ------------------------------------------------------------- leaves -----
// G lanes per leaf: the r x (r + sqre) upper bidiagonal rows a .. a + r - 1
// (diag d[a + i], superdiag e[a + i]; with sqre the extra entry e[a + r - 1] sits
// in column a + r) by the Golub-Kahan implicit-shift QR SVD (Golub & Kahan
// 1965; Golub & Van Loan, Alg. 8.6.2), U and V accumulated as products of
// rotations (the role of DLASDQ at SRC/mdlasd0.f90).  The extra column is first
// chased out by column rotations, leaving its null vector in V(:, r).  Results
// sorted ascending into slots a .. a + r - 1 (U, V, Dp, perm) and V slot a + r.
//
// Bound and layout as the tridiagonal leaves (leaf.cu): a serial chain of
// rotations at one FP64 warp instruction per 64 cycles.  Each lane carries its
// own copy of the bidiagonal and its rows of U and V, one pass of the flat
// loop is one pair of rotations for every lane, and the zero tests run as the
// sweep goes: bit i of `ez` says E(i) = 0, of `dz` D(i) = 0.  The rotations are hypot
// and the correctly rounded quotients (div_rn), for the signs' sake as there: half an
// ulp either way turned a pair of vectors in a third of the solves with leaves of 20
// rows.  Leaf stage, one
// thread per leaf before -> now: n = 1001 (64 leaves of 15 rows) 5.12 -> 0.94 ms,
// n = 16384 (1024 of 15) 5.52 -> 1.52 ms.

// Rotation taking (y, z) to (t, 0): t = hypot(y, z), cs = y / t, sn = z / t (the divides
// from one reciprocal estimate where all three are within 2^+-480)
__device__ __forceinline__ void plane_rotation(double y, double z, double &t, double &cs,
                                               double &sn) {
  t = hypot(y, z);
  const unsigned hy = __double2hiint(y) & 0x7fffffff, hz = __double2hiint(z) & 0x7fffffff;
  constexpr unsigned lo = 0x21f00000, w = 0x5df00000 - lo;
  if (hy - lo < w && hz - lo < w) {
    const double ri = rcp_nr(t);
    cs = div_rn(y, t, ri);
    sn = div_rn(z, t, ri);
  } else {
    cs = t == 0.0 ? 1.0 : y / t;
    sn = t == 0.0 ? 0.0 : z / t;
  }
}

static size_t svd_leaf_smem(int rmax, int R) {
  return (size_t)(2 * rmax + (2 * rmax + 1) * R) * 32 * sizeof(double);
}

// A rotation's two results with their fused multiply-adds written out: left to the compiler,
// instances for different G and R fuse different products, and the vectors of leaves of
// 3 to 7 and of 32 rows differed in the last bit from the plain loop's.
__device__ __forceinline__ double turn0(double cs, double sn, double x, double y) {
  return fma(cs, x, sn * y);
}
__device__ __forceinline__ double turn1(double cs, double sn, double x, double y) {
  return fma(cs, y, -(sn * x));
}

template <int G, int R>
__global__ void __launch_bounds__(32)
k_svd_leaf(int nleaf, const int *__restrict__ lstart, const int *__restrict__ lsize,
           const int *__restrict__ lsqre, int rmax, const double *__restrict__ d,
           const double *__restrict__ e, double *__restrict__ U, long long ldu,
           double *__restrict__ V, long long ldv, double *__restrict__ Dp, int *__restrict__ perm,
           int *__restrict__ status, int2 *__restrict__ supU, int2 *__restrict__ supV) {
  extern __shared__ double lsm[];
  constexpr int LPW = 32 / G;
  const int lane = threadIdx.x, q = lane / G, g0 = lane % G;
  const int leaf = blockIdx.x * LPW + q;
  double *D = lsm + lane;           // D[i * 32]
  double *E = D + rmax * 32;        // E[i * 32]
  double *Us = E + rmax * 32;       // Us[(c * R + t) * 32]: row g0 + G t, column c
  double *Vs = Us + rmax * R * 32;  // likewise, rmax + 1 columns
  // after the iteration: rk[c * 64] rank of column c, rk[c * 64 + 1] scratch
  int *rk = (int *)(lsm + rmax * 32 + q * G);
  int a = 0, r = 0, sq = 0;
  if (leaf < nleaf) {
    a = lstart[leaf];
    r = lsize[leaf];
    sq = lsqre[leaf];
  }
  const int c = r + sq;
  int rows = c;  // rows per lane of the CTA's largest leaf
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rows = max(rows, __shfl_xor_sync(HSS_FULL, rows, o));
  rows = (rows + G - 1) / G;
  // columns i, j of X <- (cs x_i + sn x_j, cs x_j - sn x_i)
  auto rotate = [&](double *X, int i, int j, double cs, double sn) {
    for (int t = 0; t < rows; ++t) {
      const double xi = X[(i * R + t) * 32], xj = X[(j * R + t) * 32];
      X[(i * R + t) * 32] = turn0(cs, sn, xi, xj);
      X[(j * R + t) * 32] = turn1(cs, sn, xi, xj);
    }
  };
  unsigned ez = 0, dz = 0;
  auto scan = [&]() {  // negligible E to zero, both masks
    ez = r > 0 ? 1u << (r - 1) : 0u;
    dz = 0;
    for (int i = 0; i < r; ++i) {
      if (i + 1 < r) {
        const double ei = E[i * 32];
        if (ei == 0.0 || negligible(ei, D[i * 32], D[(i + 1) * 32])) {
          E[i * 32] = 0.0;
          ez |= 1u << i;
        }
      }
      if (D[i * 32] == 0.0) dz |= 1u << i;
    }
  };
  for (int i = 0; i < r; ++i) {
    D[i * 32] = d[a + i];
    E[i * 32] = (i < r - 1 + sq) ? e[a + i] : 0.0;
#pragma unroll
    for (int t = 0; t < R; ++t) Us[(i * R + t) * 32] = (g0 + G * t == i) ? 1.0 : 0.0;
  }
  for (int i = 0; i < c; ++i)
#pragma unroll
    for (int t = 0; t < R; ++t) Vs[(i * R + t) * 32] = (g0 + G * t == i) ? 1.0 : 0.0;
  if (sq && r > 0) {  // chase the extra column's entry up and out: column r becomes zero
    double f = E[(r - 1) * 32];
    E[(r - 1) * 32] = 0.0;
    for (int i = r - 1; i >= 0; --i) {
      double t, cs, sn;
      plane_rotation(D[i * 32], f, t, cs, sn);
      D[i * 32] = t;
      rotate(Vs, i, r, cs, sn);
      if (i > 0) {
        const double ei = E[(i - 1) * 32];
        f = -sn * ei;
        E[(i - 1) * 32] = cs * ei;
      }
    }
  }
  scan();
  int iter = 0, bad = 0, lo = 0, hi = 0, k = 0;
  bool done = r == 0, sweeping = false;
  double y = 0.0, z = 0.0, dk = 0.0, ek = 0.0, dprev = 0.0;
  double uc[R], vc[R];  // this lane's rows of column k
  while (true) {
    const unsigned work = __ballot_sync(HSS_FULL, !done), idle = __ballot_sync(HSS_FULL, !done && !sweeping);
    if (!work) break;
    if (4 * __popc(idle) >= __popc(work) && !done && !sweeping) {
      const unsigned open = ~ez & ((1u << (r - 1)) - 1u);
      if (!open) {
        done = true;
      } else {
        hi = 32 - __clz(open);  // E(hi - 1) is the last nonzero one
        const unsigned zb = ez & ((1u << (hi - 1)) - 1u);
        lo = zb ? 32 - __clz(zb) : 0;
        const unsigned dzb = dz & (0xffffffffu << lo) & ((1u << hi) - 1u);
        if (++iter > 30 * r * r) {
          bad = 1;
          done = true;
        } else if (dzb) {  // zero inside: chase row zi's superdiagonal out by rows
          const int zi = __ffs(dzb) - 1;
          double f = E[zi * 32];
          E[zi * 32] = 0.0;
          for (int j = zi + 1; j <= hi; ++j) {
            double t, cs, sn;
            plane_rotation(D[j * 32], f, t, cs, sn);
            D[j * 32] = t;
            rotate(Us, j, zi, cs, sn);
            if (j < hi) {
              const double ej = E[j * 32];
              f = -sn * ej;
              E[j * 32] = cs * ej;
            }
          }
          scan();
        } else if (dz >> hi & 1u) {  // zero at the bottom: chase E(hi-1) out by columns
          double f = E[(hi - 1) * 32];
          E[(hi - 1) * 32] = 0.0;
          for (int j = hi - 1; j >= lo; --j) {
            double t, cs, sn;
            plane_rotation(D[j * 32], f, t, cs, sn);
            D[j * 32] = t;
            rotate(Vs, j, hi, cs, sn);
            if (j > lo) {
              const double ej = E[(j - 1) * 32];
              f = -sn * ej;
              E[(j - 1) * 32] = cs * ej;
            }
          }
          scan();
        } else {
          // Wilkinson shift from the trailing 2 x 2 of B^T B of the block
          const double d1 = D[(hi - 1) * 32], d2 = D[hi * 32], e1 = E[(hi - 1) * 32];
          const double e0 = hi - 1 > lo ? E[(hi - 2) * 32] : 0.0, t11 = fma(d1, d1, e0 * e0);
          const double t12 = d1 * e1, t22 = fma(d2, d2, e1 * e1), dd = 0.5 * (t11 - t22);
          double mu;
          if (dd == 0.0 && t12 == 0.0) mu = t22;
          else mu = t22 - t12 * t12 / (dd + copysign(hypot(dd, t12), dd != 0.0 ? dd : 1.0));
          dk = D[lo * 32];
          ek = E[lo * 32];
          y = fma(dk, dk, -mu);
          z = dk * ek;
          k = lo;
          dprev = 0.0;
#pragma unroll
          for (int t = 0; t < R; ++t) {
            uc[t] = Us[(lo * R + t) * 32];
            vc[t] = Vs[(lo * R + t) * 32];
          }
          sweeping = true;
        }
      }
    }
    if (sweeping) {  // columns k, k + 1 by the right, then rows k, k + 1 by the left
      double d1 = D[(k + 1) * 32];
      double t, cs, sn;
      plane_rotation(y, z, t, cs, sn);
      const double eprev = t;  // E(k - 1)
      const double d0 = turn0(cs, sn, dk, ek), e0 = turn1(cs, sn, dk, ek);
      const double bl = sn * d1;
      d1 *= cs;
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (R > 4 && j >= rows) break;
        const double x = Vs[((k + 1) * R + j) * 32];
        Vs[(k * R + j) * 32] = turn0(cs, sn, vc[j], x);
        vc[j] = turn1(cs, sn, vc[j], x);
      }
      plane_rotation(d0, bl, t, cs, sn);
      D[k * 32] = t;
      dz = t == 0.0 ? dz | 1u << k : dz & ~(1u << k);
      if (k > lo) {
        const bool ng = negligible(eprev, dprev, t);
        E[(k - 1) * 32] = ng ? 0.0 : eprev;
        ez = ng ? ez | 1u << (k - 1) : ez;
      }
      dprev = t;
      const double ekn = turn0(cs, sn, e0, d1), d1n = turn1(cs, sn, e0, d1);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (R > 4 && j >= rows) break;
        const double x = Us[((k + 1) * R + j) * 32];
        Us[(k * R + j) * 32] = turn0(cs, sn, uc[j], x);
        uc[j] = turn1(cs, sn, uc[j], x);
      }
      if (k + 1 < hi) {
        ek = E[(k + 1) * 32];
        y = ekn;
        z = sn * ek;
        ek *= cs;
        dk = d1n;
        ++k;
      } else {  // end of the sweep
        D[hi * 32] = d1n;
        dz = d1n == 0.0 ? dz | 1u << hi : dz & ~(1u << hi);
        const bool ng = ekn == 0.0 || negligible(ekn, t, d1n);
        E[k * 32] = ng ? 0.0 : ekn;
        ez = ng ? ez | 1u << k : ez;
#pragma unroll
        for (int j = 0; j < R; ++j) {
          Us[(hi * R + j) * 32] = uc[j];
          Vs[(hi * R + j) * 32] = vc[j];
        }
        sweeping = false;
      }
    }
  }
  // ascending by |D| (a negative one turns its column of V): ranks, each lane
  // those of its own columns
  __syncwarp();
  unsigned neg = 0;
  for (int i = 0; i < r; ++i)
    if (D[i * 32] < 0.0) {
      neg |= 1u << i;
      D[i * 32] = -D[i * 32];
    }
  if (leaf_ranks<G>(r, D, rk, g0)) leaf_ranks_ties(r, D, rk);
  __syncwarp();
  for (int i = g0; i < r; i += G) {
    Dp[a + rk[i * 64]] = D[i * 32];
    perm[a + i] = a + i;
    supU[a + i] = make_int2(a, a + r);  // rows the columns are written on
    supV[a + i] = make_int2(a, a + c);
  }
  if (sq && g0 == 0) supV[a + r] = make_int2(a, a + c);
  if (bad) atomicMax(status, HSS_LEAF_NOCONV);
  // write the blocks: lanes over the entries, one leaf at a time (coalesced)
  const double *Uw = lsm + (size_t)rmax * 64, *Vw = Uw + (size_t)rmax * R * 32;
  const int *rw = (const int *)(lsm + (size_t)rmax * 32);
  for (int l = 0; l < LPW; ++l) {
    const int a2 = __shfl_sync(HSS_FULL, a, l * G), r2 = __shfl_sync(HSS_FULL, r, l * G),
              c2 = __shfl_sync(HSS_FULL, c, l * G);
    const unsigned n2 = __shfl_sync(HSS_FULL, neg, l * G);
    for (int x = lane; x < r2 * r2; x += 32) {
      const int j = x / r2, i = x - j * r2;
      U[(long long)(a2 + rw[j * 64 + 2 * l * G]) * ldu + a2 + i] =
          Uw[(j * R + i / G) * 32 + l * G + i % G];
    }
    for (int x = lane; x < c2 * c2; x += 32) {
      const int j = x / c2, i = x - j * c2;
      const int to = j < r2 ? rw[j * 64 + 2 * l * G] : j;
      const double v = Vw[(j * R + i / G) * 32 + l * G + i % G];
      V[(long long)(a2 + to) * ldv + a2 + i] = j < r2 && (n2 >> j & 1u) ? -v : v;
    }
  }
}

// ------------------------------------------------------------ deflation ---
// One CTA per merge (MDLASD2, SRC/mdlasd2.f90).  Merge m: rows s .. s + N - 1
// with N = nl + 1 + nr, center c = s + nl, alpha = d[c], beta = e[c], extra
// column if sqre.  Outputs as the eigensolver's prepare: the non-deflated list
// (position 0 = the center, pole 0) in dl / zw / ndslot, the deflated slots in
// ascending order in dfval / dfslot, Givens pairs, out[5m] = {K, #rotations,
// #left-only, #right-only, #mixed}, and the scale onrm[m] of the merge
// (MDLASD1 divides by max(|alpha|, |beta|, |d_i|), SRC/mdlasd1.f90).
template <int MT>
__global__ void __launch_bounds__(MT)
k_svd_prepare(int P, const int *__restrict__ ms, const int *__restrict__ mnl,
              const int *__restrict__ mnr, const int *__restrict__ msq,
              const double *__restrict__ dB, const double *__restrict__ eB, double *__restrict__ U,
              long long ldu, double *__restrict__ V, long long ldv, const double *__restrict__ Dp,
              const int *__restrict__ perm, LevelScratch w, int *__restrict__ out,
              double *__restrict__ onrm, int2 *__restrict__ supU, int2 *__restrict__ supV,
              int2 *__restrict__ winU, int2 *__restrict__ winV) {
  const int m = blockIdx.x;
  if (m >= P) return;
  const int s = ms[m], nl = mnl[m], nr = mnr[m], sqre = msq[m];
  const int N = nl + 1 + nr, c = s + nl;
  const int tid = threadIdx.x;
  const double alpha = dB[c], beta = eB[c];
  if (tid == 0) {  // the center row's left vector e_c
    U[(long long)c * ldu + c] = 1.0;
    supU[c] = make_int2(c, c + 1);
  }
  // V(row, slot): zero outside the rows the column holds data on
  auto vat = [&](int slot, int row) -> double {
    const int2 r = supV[slot];
    return row >= r.x && row < r.y ? V[(long long)slot * ldv + row] : 0.0;
  };
  // ---- scale (MDLASD1) and merge the children's ascending lists (DLAMRG) into
  //      positions 1 .. N-1; position 0 is the center
  double dm = fmax(fabs(alpha), fabs(beta));
  for (int i = tid; i < N - 1; i += MT) {
    const int slot = i < nl ? perm[s + i] : perm[c + 1 + (i - nl)];
    const double v = Dp[slot];
    w.zs[s + i] = v;
    dm = fmax(dm, fabs(v));
  }
  const double nrm0 = block_max<MT>(dm);
  const double nrm = nrm0 > 0.0 ? nrm0 : 1.0;
  __syncthreads();
  const double *hv = w.zs + s;
  for (int i = tid; i < nl; i += MT) {
    const double a = hv[i];
    int lo = 0, hi = nr;
    while (lo < hi) { const int md = (lo + hi) >> 1; if (hv[nl + md] < a) lo = md + 1; else hi = md; }
    w.srt[s + 1 + i + lo] = perm[s + i];
    w.ds[s + 1 + i + lo] = a / nrm;
  }
  for (int j = tid; j < nr; j += MT) {
    const double b = hv[nl + j];
    int lo = 0, hi = nl;
    while (lo < hi) { const int md = (lo + hi) >> 1; if (hv[md] <= b) lo = md + 1; else hi = md; }
    w.srt[s + 1 + j + lo] = perm[c + 1 + j];
    w.ds[s + 1 + j + lo] = b / nrm;
  }
  __syncthreads();
  // ---- z (mdlasd2.f90: alpha * VT(i, NL+1) for the left, beta * VT(i, NL+2)
  //      for the right) in merged order
  const double an = alpha / nrm, bn = beta / nrm;
  for (int i = tid + 1; i < N; i += MT) {
    const int slot = w.srt[s + i];
    const bool left = slot < c;
    w.zs[s + i] = left ? an * vat(slot, c) : bn * vat(slot, c + 1);
    w.typ[s + i] = left ? 1 : 2;
  }
  if (tid == 0) { w.srt[s] = c; w.ds[s] = 0.0; w.typ[s] = 0; }
  const double z1 = an * vat(c, c);
  const double zM = sqre ? bn * vat(s + N, c + 1) : 0.0;
  __syncthreads();
  const double dmaxn = N > 1 ? w.ds[s + N - 1] : 0.0;
  const double tol = 8.0 * HSS_EPS * fmax(dmaxn, fmax(fabs(an), fabs(bn)));
  // ---- small z deflates (mdlasd2.f90 loop 80/100); equal singular values
  //      within tol are rotated together
  const int ng = svd_prep_chain<MT>(s, N, tol, w);
  // ---- the center's z (with the right null vector rotated in when sqre)
  double zz1, cg1 = 1.0, sg1 = 0.0;
  if (sqre) {
    zz1 = hypot(z1, zM);
    if (zz1 <= tol) zz1 = tol;
    else { cg1 = z1 / zz1; sg1 = zM / zz1; }
    // V(:, c) <- cg V(:, c) + sg V(:, s+N);  V(:, s+N) <- -sg V(:, c) + cg V(:, s+N)
    // on the union of their rows
    const int2 rc = supV[c], rn = supV[s + N];
    const int2 u = make_int2(min(rc.x, rn.x), max(rc.y, rn.y));
    __syncthreads();
    for (int rr = u.x + tid; rr < u.y; rr += MT) {
      const double vc = rr >= rc.x && rr < rc.y ? V[(long long)c * ldv + rr] : 0.0;
      const double vn = rr >= rn.x && rr < rn.y ? V[(long long)(s + N) * ldv + rr] : 0.0;
      V[(long long)c * ldv + rr] = cg1 * vc + sg1 * vn;
      V[(long long)(s + N) * ldv + rr] = -sg1 * vc + cg1 * vn;
    }
    if (tid == 0) { supV[c] = u; supV[s + N] = u; }
  } else {
    zz1 = fabs(z1) <= tol ? tol : z1;
  }
  if (tid == 0) w.zs[s] = zz1;
  __syncthreads();
  // ---- compact: non-deflated (position 0 first) and the two deflated lists
  svd_prep_compact<MT>(s, N, tol, ng, Dp, w, out + 5 * m);
  if (tid == 0) onrm[m] = nrm;
  // ---- row windows: the union of the supports of the columns taken up or rotated
  __shared__ int s_win[4];
  if (tid < 4) s_win[tid] = tid & 1 ? 0 : INT_MAX;
  __syncthreads();
  int2 wu = make_int2(INT_MAX, 0), wv = wu;
  for (int i = tid; i < N; i += MT) {
    if (w.typ[s + i] == 4) continue;
    const int slot = w.srt[s + i];
    const int2 a = supU[slot], b = supV[slot];
    wu = make_int2(min(wu.x, a.x), max(wu.y, a.y));
    wv = make_int2(min(wv.x, b.x), max(wv.y, b.y));
  }
  if (wu.y > 0) {
    atomicMin(&s_win[0], wu.x); atomicMax(&s_win[1], wu.y);
    atomicMin(&s_win[2], wv.x); atomicMax(&s_win[3], wv.y);
  }
  __syncthreads();
  if (tid == 0) {
    winU[m] = make_int2(s_win[0], s_win[1]);
    winV[m] = make_int2(s_win[2], s_win[3]);
  }
}

// ------------------------------------------------------- vector blocks ----
// Warp per column j of merge m: V block v_ij = zhat_i / (d_i^2 - sigma_j^2),
// U block u_0j = -1, u_ij = d_i zhat_i / (d_i^2 - sigma_j^2), each column scaled
// to unit length (DLASD3).  Column-major K x K blocks at Vb / Ub + boff[m].
__global__ void k_svd_vectors(LevelView lv, const double *__restrict__ dl,
                              const double *__restrict__ difl, const double *__restrict__ difr,
                              const double *__restrict__ zhat, const long long *__restrict__ boff,
                              double *__restrict__ Ub, double *__restrict__ Vb, NewRows nu,
                              NewRows nv) {
  const int lane = threadIdx.x & 31;
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (r >= __ldg(lv.rootoff + lv.P)) return;
  const int m = find_merge(lv.rootoff, lv.P, r);
  const int j = r - __ldg(lv.rootoff + m);
  const int s = __ldg(lv.s + m);
  const int K = __ldg(lv.K + m);
  if (nu.sup && lane == 0) nu.set(m, s + j);
  if (nv.sup && lane == 0) nv.set(m, s + j);
  PoleDiff P{dl + s, difl + s, difr + s, true};
  double *vc = Vb + boff[m] + (long long)j * K, *uc = Ub + boff[m] + (long long)j * K;
  // each entry is formed once (FP64 issue slots are the scarce resource): the
  // unnormalised V column goes out first and is rescaled from L2 by the same
  // lanes; the divide through the one-ulp reciprocal
  double sv = 0.0, su = 0.0;
  for (int i = lane; i < K; i += HSS_WARP) {
    const double v = qdiv(__ldg(zhat + s + i), P.fd(i, j));
    vc[i] = v;
    sv += v * v;
    if (i > 0) { const double u = __ldg(dl + s + i) * v; su += u * u; }
  }
  sv = warp_sum(sv);
  su = warp_sum(su);
  const double av = 1.0 / sqrt(sv), au = 1.0 / sqrt(1.0 + su);
  for (int i = lane; i < K; i += HSS_WARP) {
    const double v = vc[i];
    vc[i] = v * av;
    uc[i] = i == 0 ? -au : __ldg(dl + s + i) * v * au;
  }
}

// One merge's column norms for the HSS path: alpha_j (V block), beta_j (U
// block, including the -1 of row 0) and the U generator ud_i = d_i zhat_i
// (arrays already offset to the merge; warp per column).
__global__ void k_svd_norms(int K, const double *__restrict__ dl, const double *__restrict__ difl,
                            const double *__restrict__ difr, const double *__restrict__ zhat,
                            double *__restrict__ alpha, double *__restrict__ beta,
                            double *__restrict__ ud) {
  const int lane = threadIdx.x & 31;
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (j >= K) return;
  PoleDiff P{dl, difl, difr, true};
  double sv = 0.0, su = 0.0;
  for (int i = lane; i < K; i += HSS_WARP) {
    const double v = __ldg(zhat + i) / P.fd(i, j);
    sv += v * v;
    if (i > 0) { const double u = __ldg(dl + i) * v; su += u * u; }
  }
  sv = warp_sum(sv);
  su = warp_sum(su);
  if (lane == 0) {
    alpha[j] = 1.0 / sqrt(sv);
    beta[j] = 1.0 / sqrt(1.0 + su);
    ud[j] = __ldg(dl + j) * __ldg(zhat + j);
  }
}

// T(:, j) -= beta_j X(:, 0): the row-0 entries -beta_j of the U block.
__global__ void k_svd_rank1(int nrows, int K, const double *__restrict__ X, long long ldx,
                            const double *__restrict__ beta, double *__restrict__ T,
                            long long ldt) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)nrows * K) return;
  const int i = (int)(idx % nrows), j = (int)(idx / nrows);
  T[(long long)j * ldt + i] -= beta[j] * X[i];
}

void launch_svd_norms(int K, const double *dl, const double *difl, const double *difr,
                      const double *zhat, double *alpha, double *beta, double *ud,
                      cudaStream_t st) {
  if (K > 0)
    k_svd_norms<<<(unsigned)(((long long)K * 32 + 255) / 256), 256, 0, st>>>(K, dl, difl, difr,
                                                                             zhat, alpha, beta, ud);
}
void launch_svd_rank1(int nrows, int K, const double *X, long long ldx, const double *beta,
                      double *T, long long ldt, cudaStream_t st) {
  const long long tot = (long long)nrows * K;
  if (tot > 0)
    k_svd_rank1<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(nrows, K, X, ldx, beta, T, ldt);
}

// sigma of every root back to the merge's scale (lam *= onrm[m]).
__global__ void k_svd_unscale(LevelView lv, const double *__restrict__ onrm,
                              double *__restrict__ lam) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= __ldg(lv.rootoff + lv.P)) return;
  const int m = find_merge(lv.rootoff, lv.P, r);
  lam[__ldg(lv.s + m) + r - __ldg(lv.rootoff + m)] *= onrm[m];
}

// VT(i, :) = V(:, perm(n-1-i))^T (descending singular values): 32 x 32 tiles
// through shared memory so both the reads of V and the writes of VT coalesce.
// sup (optional): rows each column holds data on (zero elsewhere).
__global__ void k_svd_vt(int n, const int *__restrict__ perm, const double *__restrict__ V,
                         long long ldv, double *__restrict__ VT, long long ldvt,
                         const int2 *__restrict__ sup) {
  __shared__ double tile[32][33];
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;  // rows i of VT, columns j
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int i = i0 + k, j = j0 + threadIdx.x;
    if (i < n && j < n) {
      const int p = perm[n - 1 - i];
      const int2 r = sup ? sup[p] : make_int2(0, n);
      tile[k][threadIdx.x] = j >= r.x && j < r.y ? V[(long long)p * ldv + j] : 0.0;
    }
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int j = j0 + k, i = i0 + threadIdx.x;
    if (i < n && j < n) VT[(long long)j * ldvt + i] = tile[threadIdx.x][k];
  }
}

// U(:, i) = Uq(:, perm(n-1-i)), w(i) = Dp(perm(n-1-i)) (descending).
__global__ void k_svd_u(int n, const int *__restrict__ perm, const double *__restrict__ Dp,
                        const double *__restrict__ Uq, long long ldq, double *__restrict__ Uo,
                        long long ldu, double *__restrict__ w, const int2 *__restrict__ sup) {
  const int col = blockIdx.x;
  if (col >= n) return;
  const long long p = perm[n - 1 - col];
  const int2 r = sup ? sup[p] : make_int2(0, n);
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    Uo[(long long)col * ldu + i] = i >= r.x && i < r.y ? Uq[p * ldq + i] : 0.0;
  if (threadIdx.x == 0) w[col] = Dp[p];
}

__global__ void k_svd_w(int n, const int *__restrict__ perm, const double *__restrict__ Dp,
                        double *__restrict__ w) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col < n) w[col] = Dp[perm[n - 1 - col]];
}

// Rows of A rotated back to front (DLASR('L', 'V', 'B'), the lower-to-upper
// rotations of DBDSDC applied to U): for j = n-2 .. 0, with c = cs[j],
// s = sn[j]: (A_j, A_{j+1}) <- (s A_{j+1} + c A_j, c A_{j+1} - s A_j).  One
// thread per column.
__global__ void k_rows_rotate_back(int n, int ncols, const double *__restrict__ cs,
                                   const double *__restrict__ sn, double *__restrict__ A,
                                   long long lda) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= ncols) return;
  double *a = A + (long long)col * lda;
  for (int j = n - 2; j >= 0; --j) {
    const double c = cs[j], s = sn[j];
    const double t = a[j + 1];
    a[j + 1] = c * t - s * a[j];
    a[j] = s * t + c * a[j];
  }
}

// ---------------------------------------------------------------- launch --
void launch_rows_rotate_back(int n, int ncols, const double *cs, const double *sn, double *A,
                             long long lda, cudaStream_t st) {
  if (n > 1 && ncols > 0) k_rows_rotate_back<<<(ncols + 127) / 128, 128, 0, st>>>(n, ncols, cs, sn, A, lda);
}

template <int G, int R>
static void svd_leaf_launch(int nleaf, const int *lstart, const int *lsize, const int *lsqre,
                            int rmax, const double *d, const double *e, double *U, long long ldu,
                            double *V, long long ldv, double *Dp, int *perm, int *status,
                            int2 *supU, int2 *supV, cudaStream_t st) {
  const size_t smem = svd_leaf_smem(rmax, R);
  static size_t attr = 48 * 1024;
  if (smem > attr) {
    cudaFuncSetAttribute(k_svd_leaf<G, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr = smem;
  }
  k_svd_leaf<G, R><<<(nleaf * G + 31) / 32, 32, smem, st>>>(nleaf, lstart, lsize, lsqre, rmax, d, e,
                                                            U, ldu, V, ldv, Dp, perm, status,
                                                            supU, supV);
}

void launch_svd_leaf(int nleaf, const int *lstart, const int *lsize, const int *lsqre, int rmax,
                     const double *d, const double *e, double *U, long long ldu, double *V,
                     long long ldv, double *Dp, int *perm, int *status, int2 *supU, int2 *supV,
                     cudaStream_t st) {
  if (nleaf <= 0) return;
  rmax = std::max(1, std::min(rmax, SVD_LEAF_MAX));
  // two blocks of vectors (shared memory): at most 8 rows of each per lane
  int G = leaf_lanes(nleaf, rmax + 1);
  while (G < 32 && (G < 2 || (rmax + G) / G > 8)) G *= 2;
  const int R = (rmax + G) / G;  // ceil((rmax + 1) / G)
#define SVDL_ARGS \
  nleaf, lstart, lsize, lsqre, rmax, d, e, U, ldu, V, ldv, Dp, perm, status, supU, supV, st
#define SVDL_TRY(g, r) if (G == g && R <= r) return svd_leaf_launch<g, r>(SVDL_ARGS)
  SVDL_TRY(2, 4);
  SVDL_TRY(2, 8);
  SVDL_TRY(4, 4);
  SVDL_TRY(4, 8);
  SVDL_TRY(8, 2);
  SVDL_TRY(8, 5);
  SVDL_TRY(16, 1);
  SVDL_TRY(16, 3);
  SVDL_TRY(32, 1);
  svd_leaf_launch<32, 2>(SVDL_ARGS);  // rmax + 1 <= 33 rows
#undef SVDL_TRY
#undef SVDL_ARGS
}

static int svd_threads(int maxn) {
  return maxn <= 64 ? 64 : maxn <= 256 ? 128 : maxn <= 2048 ? 256 : 512;
}

void launch_svd_prepare(int P, int maxn, const int *ms, const int *mnl, const int *mnr,
                        const int *msq, const double *d, const double *e, double *U,
                        long long ldu, double *V, long long ldv, const double *Dp, const int *perm,
                        const LevelScratch &w, int *out, double *onrm, int2 *supU, int2 *supV,
                        int2 *winU, int2 *winV, cudaStream_t st) {
  if (P <= 0) return;
#define SVDP_CASE(T)                                                                        \
  case T:                                                                                  \
    k_svd_prepare<T><<<P, T, 0, st>>>(P, ms, mnl, mnr, msq, d, e, U, ldu, V, ldv, Dp, perm, \
                                      w, out, onrm, supU, supV, winU, winV);               \
    break;
  switch (svd_threads(maxn)) {
    SVDP_CASE(64)
    SVDP_CASE(128)
    SVDP_CASE(256)
    default:
    SVDP_CASE(512)
  }
#undef SVDP_CASE
}

void launch_svd_vectors(const LevelView &lv, int total, const double *dl, const double *difl,
                        const double *difr, const double *zhat, const long long *boff, double *Ub,
                        double *Vb, cudaStream_t st, NewRows nu, NewRows nv) {
  if (total <= 0) return;
  k_svd_vectors<<<(unsigned)(((long long)total * 32 + 255) / 256), 256, 0, st>>>(
      lv, dl, difl, difr, zhat, boff, Ub, Vb, nu, nv);
}
void launch_svd_unscale(const LevelView &lv, int total, const double *onrm, double *lam,
                        cudaStream_t st) {
  if (total > 0) k_svd_unscale<<<(total + 255) / 256, 256, 0, st>>>(lv, onrm, lam);
}

void launch_svd_outputs(int n, const int *perm, const double *Dp, const double *Uq,
                        long long ldq, const double *V, long long ldv, double *Uo, long long ldu,
                        double *VT, long long ldvt, double *w, bool vectors, cudaStream_t st,
                        const int2 *supU, const int2 *supV) {
  if (n <= 0) return;
  if (vectors) {
    k_svd_u<<<n, 256, 0, st>>>(n, perm, Dp, Uq, ldq, Uo, ldu, w, supU);
    dim3 g((n + 31) / 32, (n + 31) / 32);
    k_svd_vt<<<g, dim3(32, 8), 0, st>>>(n, perm, V, ldv, VT, ldvt, supV);
  } else {
    k_svd_w<<<(n + 255) / 256, 256, 0, st>>>(n, perm, Dp, w);
  }
}

}  // namespace hss
