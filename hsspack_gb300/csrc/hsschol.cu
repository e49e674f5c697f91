// hsschol.cu -- HSS Cholesky factorisation of a dense SPD matrix and its solves
// on sm_103a (HssCholSolver, SRC/HssCholSolver.f90:1-139, with mat2hsscholsvd /
// mat2hsscholsvdr, solvecholsvd and cg of SRC/mat2hsssvd.f90).
//
// The method (Li, Gu, Wu, Xia, SIMAX 33, 2012): at a node with diagonal block
// D = L L^T and block column T (the node's variables against every other
// current variable), the scaled block column T L^{-T} is compressed: its right
// singular vectors V = [V1 V2] split at the singular values above tol (rank rk,
// at most ncol).  With Q = [V2 V1] and the QL factorisation L Q = Qt Lt, the
// node's variables in the basis Qt decouple: the first ir = m - rk of them touch
// nothing outside the node once T L^{-T} V2 is dropped, so they are eliminated
// by Lt11, and the remaining rk carry the Schur complement Lt22 Lt22^T and the
// block column T W with W = L^{-T} V1 Lt22^T.  Parents stack their children's
// remaining variables; the root is factored by a plain Cholesky.  The
// factorisation is SPD by construction (every Schur complement is Lt22 Lt22^T).
//
// The reference visits the nodes in post order, one at a time, packing the
// partially compressed matrix in a stack (mat2hsssvd.f90:117-264).  Here all
// nodes of one tree height are compressed at once on an explicit reduced matrix
// Ah in HBM (each active node owns a contiguous range, in leaf order): a batched
// Cholesky of the diagonal blocks, the scaled block columns Ah(:, I) L^{-T} as a
// grouped GEMM (the node's own rows zeroed), their right singular vectors by the
// TSQR / pivoted-QR / Jacobi kernels of the dense HSS construction (or, for the
// randomised variant, of the ps x m sketches Omega X), the per-node QL step, and
// the congruence Ah' = W^T Ah W (W block diagonal; W_i = I for nodes that keep
// their variables) as two grouped GEMMs around a transpose -- its diagonal
// blocks are exactly Lt22 Lt22^T.  Nodes of one height see each other's
// variables uncompressed, so the kept subspaces differ from the sequential
// order's by the truncation tolerance; with no truncation both are exact.
//
// Solves run level by level in the same order: forward, each compressed node
// applies Qt^T, eliminates its first ir entries with Lt11 and hands Lt21's
// update of the remaining rk to the next level; the root is solved with its
// Cholesky factor; backward reverses it (solvecholsvd, mat2hsssvd.f90:553-671).
// The preconditioned CG of the reference (cg, :674-726) runs on the device with
// a dense FP64 matrix-vector product.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "hss_common.cuh"
#include "hss_gemm.h"
#include "hss_hss.h"
#include "hss_plan.h"
#include "hss_pool.h"
#include "hss_chol.h"

namespace hss {

#define CCK(x)                                                                              \
  do {                                                                                      \
    cudaError_t e_ = (x);                                                                   \
    if (e_ != cudaSuccess) throw HssError{std::string(#x) + ": " + cudaGetErrorString(e_)}; \
  } while (0)

constexpr int CHT = 256;  // threads per node CTA
constexpr size_t CH_SLOT = (size_t)CH_MAXM * CH_MAXM;

// ------------------------------------------------------------- kernels ----

// Cholesky D = L L^T of each node's diagonal block (one CTA per node, the block
// in shared memory); L (lower, m x m) and It = L^{-T} (upper) to the node's
// scratch slot.  status |= 1 when a pivot is not positive.
//
// Bound by the serial chain of m steps, each a few FP64 instructions a warp.  The
// columns stay unscaled until the end, so a step needs one reciprocal and no root; the
// trailing triangle is folded into a rectangle, column c's part and column t-1-c's in
// one row of it, so no thread works above the diagonal.  The inverse runs by columns
// of L in the upper triangle, (column, row) pairs over all threads; it took a thread per
// column with a division per entry.  256 nodes of 32 rows: 147 -> 45 us.
__global__ void __launch_bounds__(CHT)
k_ch_chol(const ChNode *__restrict__ nd, const double *__restrict__ Ah, long long lda,
          double *__restrict__ Lb, double *__restrict__ Ib, int *__restrict__ status) {
  extern __shared__ double S[];  // column j at S + j * ld: L below, It above the diagonal
  __shared__ double rd[CH_MAXM];
  const ChNode q = nd[blockIdx.x];
  const int m = q.m, ld = m | 1, tid = threadIdx.x;
  const double *D = Ah + (long long)q.o * lda + q.o;
  for (int e = tid; e < m * m; e += CHT) {
    const int j = e / m, i = e - j * m;
    S[j * ld + i] = i >= j ? D[(long long)j * lda + i] : 0.0;
  }
  __syncthreads();
  for (int j = 0; j < m; ++j) {
    const double *Sj = S + j * ld;
    const double d = Sj[j];
    if (!(d > 0.0)) {
      if (tid == 0) atomicOr(status, 1);
      return;
    }
    const int hd = __double2hiint(d);  // 2^-960 <= d < 2^960
    const double di = hd >= 0x03f00000 && hd < 0x7bf00000 ? rcp_nr(d) : 1.0 / d;
    const int t = m - j - 1, w = t | 1, tot = w * ((t + 1) >> 1);
    for (int e = tid; e < tot; e += CHT) {
      int c = e / w, r = e - c * w;
      if (r >= t - c) {  // column t - c (t odd) or t - 1 - c
        r -= t - c;
        c = (t & 1 ? t : t - 1) - c;
      }
      const double *u = Sj + j + 1;
      double *x = S + (j + 1 + c) * ld + j + 1 + c + r;
      *x = fma(-u[c + r] * di, u[c], *x);
    }
    __syncthreads();
  }
  for (int j = tid; j < m; j += CHT) {
    const double r = sqrt(S[j * ld + j]);
    S[j * ld + j] = r;
    rd[j] = 1.0 / r;
  }
  __syncthreads();
  double *L = Lb + (size_t)q.slot * CH_SLOT, *It = Ib + (size_t)q.slot * CH_SLOT;
  for (int e = tid; e < m * m; e += CHT) {
    const int j = e / m, i = e - j * m;
    if (i > j) S[j * ld + i] *= rd[j];
    L[(long long)j * m + i] = i >= j ? S[j * ld + i] : 0.0;
  }
  __syncthreads();
  // It(c, i) = L^{-1}(i, c): row l of L^{-1} is final before step l, times rd[l]
  for (int l = 0; l < m - 1; ++l) {
    const int tot = (l + 1) * (m - l - 1);
    for (int e = tid; e < tot; e += CHT) {
      const int ii = e / (l + 1), c = e - ii * (l + 1), i = l + 1 + ii;
      const double x = c == l ? rd[l] : S[l * ld + c] * rd[l];
      S[i * ld + c] = fma(-S[l * ld + i], x, S[i * ld + c]);
    }
    __syncthreads();
  }
  for (int e = tid; e < m * m; e += CHT) {
    const int i = e / m, c = e - i * m;
    It[(long long)i * m + c] = c < i ? S[i * ld + c] * rd[i] : c == i ? rd[i] : 0.0;
  }
}

// Rows of the node's own range in its scaled block column X(:, I) set to zero.
__global__ void k_ch_zero_own(const ChNode *__restrict__ nd, double *__restrict__ X, long long ld) {
  const ChNode q = nd[blockIdx.x];
  for (int e = threadIdx.x; e < q.m * q.m; e += blockDim.x) {
    const int j = e / q.m, i = e - j * q.m;
    X[(long long)(q.o + j) * ld + q.o + i] = 0.0;
  }
}

// One reflector step.  Vector j sits at vec(j), entry i at stride s; the reflector is
// [1 at pv; v(t0:t1) * scale], its parameters in hp[k & 1].  The last warp takes the
// vector nxt alone (null: none) and forms the next reflector from it, entry npv and tail
// nt0:nt1; the other threads take cnt vectors, up to eight threads a vector.
template <class Vec>
__device__ void ch_reflect(double *v, double *nxt, int s, int t0, int t1, int pv, int nt0, int nt1,
                           int npv, HousePar *hp, int k, int cnt, Vec vec, double *part) {
  const int tid = threadIdx.x, lane = tid & 31;
  const HousePar h = hp[k & 1];
  double *pe = nullptr, ptw = 0.0;  // this thread's entry pv, and its change
  if (tid >= CHT) {
    if (nxt) {
      if (h.tau != 0.0) {
        double d = 0.0;
        for (int i = t0 + lane; i < t1; i += 32) d = fma(v[i * s], nxt[i * s], d);
        d = warp_sum(d);
        const double tw = h.tau * fma(h.scale, d, nxt[pv * s]), tws = tw * h.scale;
        for (int i = t0 + lane; i < t1; i += 32) nxt[i * s] = fma(-tws, v[i * s], nxt[i * s]);
        __syncwarp();
        if (lane == 0) nxt[pv * s] -= tw;
      }
      double a = 0.0;
      for (int i = nt0 + lane; i < nt1; i += 32) { const double x = nxt[i * s]; a = fma(x, x, a); }
      a = warp_sum(a);
      if (lane == 0) hp[(k + 1) & 1] = house_par(nxt[npv * s], a);
    }
  } else if (cnt > 0 && h.tau != 0.0) {
    if (cnt > CHT / 2) {
      for (int j = tid; j < cnt; j += CHT) {
        double *x = vec(j), d = 0.0;
        for (int i = t0; i < t1; ++i) d = fma(v[i * s], x[i * s], d);
        const double tw = h.tau * fma(h.scale, d, x[pv * s]), tws = tw * h.scale;
        for (int i = t0; i < t1; ++i) x[i * s] = fma(-tws, v[i * s], x[i * s]);
        x[pv * s] -= tw;
      }
    } else {
      const int nch = min(CHT / cnt, 8), ch = tid / cnt, j = tid - ch * cnt;
      const bool act = ch < nch;
      double *x = vec(j), d = 0.0;
      const int i0 = t0 + (t1 - t0) * ch / nch, i1 = act ? t0 + (t1 - t0) * (ch + 1) / nch : i0;
      for (int i = i0; i < i1; ++i) d = fma(v[i * s], x[i * s], d);
      if (act) part[ch * cnt + j] = d;
      asm volatile("bar.sync 1, %0;" ::"n"(CHT) : "memory");
      if (act) {
        d = 0.0;
        for (int c = 0; c < nch; ++c) d += part[c * cnt + j];
        const double tw = h.tau * fma(h.scale, d, x[pv * s]), tws = tw * h.scale;
        for (int i = i0; i < i1; ++i) x[i * s] = fma(-tws, v[i * s], x[i * s]);
        if (ch == 0) { pe = x + pv * s; ptw = tw; }
      }
    }
  }
  __syncthreads();
  if (pe) *pe -= ptw;  // (every chunk has read it, and no later step does)
  if (tid == 0) v[pv * s] = h.beta;
}

// The QL step of one compressed node (one CTA; m <= 128).  In: L (scratch slot), V1 =
// the first rk right singular vectors (P, ld m).  Out: Qt and Lt (m x m each, the
// factor store), W = L^{-T} V1 Lt22^T up to rounding (m x rk, scratch).
//   1. QL of L V1 = Qt2 Lt22 (rk reflectors from the last column up, DGEQL2's order),
//      each applied to L and to the identity as well: they end as Qt^T L = [L1; L2]
//      and Qt^T.  V2 is not formed: Qt1 spans the complement of L V1, so the rows of
//      L1 span that of V1.
//   2. LQ of L1 = Lt11 V2^T by ir reflectors on the right, L2 V2 = Lt21 with it.
//   3. The eliminated variables' Schur step: W = Qt [-Lt11^{-T} Lt21^T; I].
// That is m reflector steps (forming V2 first, then the QL of L [V2 V1], and Qt from
// its reflectors took 2 m + 2 rk, a thread per column: n = 8192 with 32-row leaves
// 3.08 -> 0.77 ms in all).  Bound by the steps' chains, about 20 FP64 instructions a warp each
// at m = 32.  L, L V1 and Qt^T sit in shared memory, the last two in global memory
// (sm = 0) where a level's nodes are too large.
__global__ void __launch_bounds__(CHT + 32)
k_ch_node(const ChNode *__restrict__ nd, const double *__restrict__ Lb,
          const double *__restrict__ Pb, double *__restrict__ Gb, double *__restrict__ fac,
          double *__restrict__ Wb, int sm) {
  extern __shared__ double S[];
  __shared__ double rd[CH_MAXM], part[CHT];
  __shared__ HousePar hp[2];
  const ChNode q = nd[blockIdx.x];
  const int m = q.m, rk = q.rk, ir = q.ir, ld = m | 1, tid = threadIdx.x, lane = tid & 31;
  constexpr int NT = CHT + 32;
  const size_t so = (size_t)q.slot * CH_SLOT;
  const double *L = Lb + so, *P = Pb + so;
  double *A2 = S;                                   // L, then [Lt11; Lt21] (columns < ir)
  double *T = sm ? S + (size_t)m * ld : Gb + 4 * so;  // I, then Qt^T
  double *A1 = T + (size_t)m * ld;                  // L V1, then Lt22 under Z
  double *Qt = fac + q.f, *Lt = Qt + (size_t)m * m;
  double *W = Wb + so;
  for (int e = tid; e < m * m; e += NT) {
    const int j = e / m, i = e - j * m;
    A2[j * ld + i] = L[e];
    T[j * ld + i] = i == j ? 1.0 : 0.0;
  }
  __syncthreads();
  for (int e = tid; e < m * rk; e += NT) {
    const int j = e / m, i = e - j * m;
    double s = 0.0;
    for (int l = 0; l <= i; ++l) s = fma(A2[l * ld + i], P[(long long)j * m + l], s);
    A1[j * ld + i] = s;
  }
  __syncthreads();
  // the first reflector of a sequence, by the last warp
  auto first = [&](const double *v, int s, int t0, int t1, int pv) {
    if (tid >= CHT) {
      double a = 0.0;
      for (int i = t0 + lane; i < t1; i += 32) a = fma(v[i * s], v[i * s], a);
      a = warp_sum(a);
      if (lane == 0) hp[0] = house_par(v[pv * s], a);
    }
    __syncthreads();
  };
  if (rk > 0) first(A1 + (rk - 1) * ld, 1, 0, m - 1, m - 1);
  for (int k = 0; k < rk; ++k) {
    const int c = rk - 1 - k, p = ir + c, ca = max(c - 1, 0);
    ch_reflect(A1 + c * ld, c > 0 ? A1 + (c - 1) * ld : nullptr, 1, 0, p, p, 0, p - 1, p - 1, hp, k,
               ca + 2 * m,
               [=](int j) { return j < ca ? A1 + j * ld : j < ca + m ? A2 + (j - ca) * ld : T + (j - ca - m) * ld; },
               part);
  }
  __syncthreads();
  first(A2, ld, 1, m, 0);
  for (int k = 0; k < ir; ++k) {
    const bool la = k + 1 < ir;  // (the rows from ir on form no reflector)
    const int j0 = la ? k + 2 : k + 1;
    ch_reflect(A2 + k, la ? A2 + k + 1 : nullptr, ld, k + 1, m, k, k + 2, m, k + 1, hp, k, m - j0,
               [=](int j) { return A2 + j0 + j; }, part);
  }
  __syncthreads();
  for (int e = tid; e < m * m; e += NT) {
    const int j = e / m, i = e - j * m;
    Lt[e] = i < j ? 0.0 : j < ir ? A2[j * ld + i] : A1[(j - ir) * ld + i];
    Qt[e] = T[i * ld + j];
  }
  for (int i = tid; i < ir; i += NT) rd[i] = 1.0 / A2[i * ld + i];
  // Z = Lt11^{-T} Lt21^T in rows 0 .. ir-1 of A1 (row i times rd[i])
  for (int e = tid; e < ir * rk; e += NT) {
    const int j = e / ir, i = e - j * ir;
    A1[j * ld + i] = A2[i * ld + ir + j];
  }
  __syncthreads();
  if (rk > 0) {
    const int nch = NT / rk, ch = tid / rk, j = tid - ch * rk;
    for (int i = ir - 1; i > 0; --i) {
      if (ch < nch) {
        const double z = A1[j * ld + i] * rd[i];
        for (int l = ch; l < i; l += nch) A1[j * ld + l] = fma(-A2[l * ld + i], z, A1[j * ld + l]);
      }
      __syncthreads();
    }
  }
  for (int e = tid; e < ir * rk; e += NT) {
    const int j = e / ir, i = e - j * ir;
    A1[j * ld + i] *= rd[i];
  }
  __syncthreads();
  for (int e = tid; e < m * rk; e += NT) {
    const int j = e / m, i = e - j * m;
    double s = T[i * ld + ir + j];
    for (int l = 0; l < ir; ++l) s = fma(-T[i * ld + l], A1[j * ld + l], s);
    W[(long long)j * m + i] = s;
  }
}

// Columns [o, o + m) of A (rows x ., lda) copied to columns [o2, o2 + m) of B
// for the nodes that keep their variables (ir = 0).
__global__ void k_ch_copy_cols(const ChNode *__restrict__ nd, int nn, int rows,
                               const double *__restrict__ A, long long lda, double *__restrict__ B,
                               long long ldb) {
  const ChNode q = nd[blockIdx.y];
  if (q.ir != 0) return;
  const long long tot = (long long)rows * q.m;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < tot;
       e += (long long)gridDim.x * blockDim.x) {
    const long long j = e / rows, i = e - j * rows;
    B[(q.o2 + j) * ldb + i] = A[(q.o + j) * lda + i];
  }
}

// ---- solves: Y (level vectors, ld) for each right-hand side column, a warp each
// (CHT / 32 of them at a time on a node's CTA).  The substitutions run column by
// column: lane i % 32 holds entry i, and every step is one shuffled value times a
// precomputed reciprocal and one multiply-add per 32 entries.  (Row by row, a
// dot product's warp reduction and a division took 22 FP64 instructions per entry,
// on one warp, one right-hand side after the other: n = 8192, 16 right-hand sides
// 4.9 -> 0.5 ms.)  The matrix that a warp reads across its columns sits in shared
// memory with an odd leading dimension.
constexpr int CHB = CH_MAXM / 32;  // entries per lane

// forward: u = Qt^T y(I); u1 = Lt11^{-1} u1 (kept in y(I) for the backward
// pass); y2(I') = u2 - Lt21 u1.  Nodes that keep their variables copy.
__global__ void __launch_bounds__(CHT)
k_ch_fwd(const ChNode *__restrict__ nd, const double *__restrict__ fac, double *__restrict__ Y,
         long long ldy, double *__restrict__ Y2, long long ldy2, int nrhs) {
  extern __shared__ double Qs[];
  __shared__ double v[CHT / 32][CH_MAXM], rd[CH_MAXM];
  const ChNode q = nd[blockIdx.x];
  const int m = q.m, ir = q.ir, ld = m | 1, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const double *Qt = fac + q.f, *Lt = Qt + (size_t)m * m;
  if (ir > 0) {
    for (int e = tid; e < m * m; e += CHT) Qs[e / m * ld + e % m] = Qt[e];
    for (int i = tid; i < ir; i += CHT) rd[i] = 1.0 / Lt[(long long)i * m + i];
  }
  __syncthreads();
  for (int r = w; r < nrhs; r += CHT / 32) {
    double *y = Y + (long long)r * ldy + q.o;
    double *y2 = Y2 + (long long)r * ldy2 + q.o2;
    if (ir == 0) {
      for (int i = lane; i < m; i += 32) y2[i] = y[i];
      continue;
    }
    for (int i = lane; i < m; i += 32) v[w][i] = y[i];
    __syncwarp();
    double u[CHB];
#pragma unroll
    for (int b = 0; b < CHB; ++b) {
      const int i = lane + 32 * b;
      u[b] = 0.0;
      if (i < m)
        for (int l = 0; l < m; ++l) u[b] = fma(Qs[i * ld + l], v[w][l], u[b]);
    }
    __syncwarp();
#pragma unroll
    for (int b = 0; b < CHB; ++b)
      for (int i = 32 * b; i < min(ir, 32 * b + 32); ++i) {
        const double x = __shfl_sync(HSS_FULL, u[b], i & 31) * rd[i];
        if (lane == (i & 31)) u[b] = x;
#pragma unroll
        for (int c = b; c < CHB; ++c) {
          const int l = lane + 32 * c;
          if (l > i && l < m) u[c] = fma(-Lt[(long long)i * m + l], x, u[c]);
        }
      }
#pragma unroll
    for (int b = 0; b < CHB; ++b) {
      const int i = lane + 32 * b;
      if (i < ir) y[i] = u[b];
      else if (i < m) y2[i - ir] = u[b];
    }
  }
}

// backward: u2 = x2(I'); u1 = Lt11^{-T} (u1 - Lt21^T u2); x(I) = Qt [u1; u2].
__global__ void __launch_bounds__(CHT)
k_ch_bwd(const ChNode *__restrict__ nd, const double *__restrict__ fac, double *__restrict__ Y,
         long long ldy, const double *__restrict__ Y2, long long ldy2, int nrhs) {
  extern __shared__ double Ls[];
  __shared__ double v[CHT / 32][CH_MAXM], rd[CH_MAXM];
  const ChNode q = nd[blockIdx.x];
  const int m = q.m, ir = q.ir, ld = m | 1, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const double *Qt = fac + q.f, *Lt = Qt + (size_t)m * m;
  if (ir > 0) {
    for (int e = tid; e < m * m; e += CHT) Ls[e / m * ld + e % m] = Lt[e];
    for (int i = tid; i < ir; i += CHT) rd[i] = 1.0 / Lt[(long long)i * m + i];
  }
  __syncthreads();
  for (int r = w; r < nrhs; r += CHT / 32) {
    double *y = Y + (long long)r * ldy + q.o;
    const double *y2 = Y2 + (long long)r * ldy2 + q.o2;
    if (ir == 0) {
      for (int i = lane; i < m; i += 32) y[i] = y2[i];
      continue;
    }
    double u[CHB];
#pragma unroll
    for (int b = 0; b < CHB; ++b) {
      const int i = lane + 32 * b;
      u[b] = i < ir ? y[i] : i < m ? y2[i - ir] : 0.0;
    }
#pragma unroll
    for (int b = CHB - 1; b >= 0; --b)
      for (int i = min(m, 32 * b + 32) - 1; i >= 32 * b; --i) {
        double x = __shfl_sync(HSS_FULL, u[b], i & 31);
        if (i < ir) {
          x *= rd[i];
          if (lane == (i & 31)) u[b] = x;
        }
#pragma unroll
        for (int c = 0; c <= b; ++c) {
          const int l = lane + 32 * c;
          if (l < i && l < ir) u[c] = fma(-Ls[l * ld + i], x, u[c]);
        }
      }
    __syncwarp();
#pragma unroll
    for (int b = 0; b < CHB; ++b)
      if (lane + 32 * b < m) v[w][lane + 32 * b] = u[b];
    __syncwarp();
    for (int i = lane; i < m; i += 32) {
      double s = 0.0;
      for (int l = 0; l < m; ++l) s = fma(Qt[(long long)l * m + i], v[w][l], s);
      y[i] = s;
    }
  }
}

// L L^T x = y for the root (n x n lower L), a one-warp CTA per column, in place.
__global__ void __launch_bounds__(32)
k_ch_root(int n, const double *__restrict__ L, double *__restrict__ Y, long long ldy) {
  const int lane = threadIdx.x;
  double *y = Y + (long long)blockIdx.x * ldy;
  for (int i = 0; i < n; ++i) {
    const double x = y[i] / L[(long long)i * n + i];
    __syncwarp();
    if (lane == 0) y[i] = x;
    for (int l = i + 1 + lane; l < n; l += 32) y[l] = fma(-L[(long long)i * n + l], x, y[l]);
    __syncwarp();
  }
  for (int i = n - 1; i >= 0; --i) {
    const double x = y[i] / L[(long long)i * n + i];
    __syncwarp();
    if (lane == 0) y[i] = x;
    for (int l = lane; l < i; l += 32) y[l] = fma(-L[(long long)l * n + i], x, y[l]);
    __syncwarp();
  }
}

// y = A x for column-major A (n x n, lda): partial sums over column chunks
// (grid.y), then a fixed-order reduction -- deterministic.
constexpr int GV_CHUNK = 256;
__global__ void k_gemv_part(int n, const double *__restrict__ A, long long lda,
                            const double *__restrict__ x, double *__restrict__ part) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int c0 = blockIdx.y * GV_CHUNK, c1 = min(n, c0 + GV_CHUNK);
  if (i >= n) return;
  double s = 0.0;
  for (int j = c0; j < c1; ++j) s = fma(A[(long long)j * lda + i], __ldg(x + j), s);
  part[(long long)blockIdx.y * n + i] = s;
}
__global__ void k_gemv_sum(int n, int nch, const double *__restrict__ part, double *__restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
  for (int c = 0; c < nch; ++c) s += part[(long long)c * n + i];
  y[i] = s;
}
// out[k] = a_k . b_k for up to three pairs (partials per block, then one block)
__global__ void k_dots(int n, const double *__restrict__ a0, const double *__restrict__ b0,
                       const double *__restrict__ a1, const double *__restrict__ b1,
                       double *__restrict__ part) {
  __shared__ double red[2][CHT / 32];
  double s0 = 0.0, s1 = 0.0;
  for (int i = blockIdx.x * CHT + threadIdx.x; i < n; i += gridDim.x * CHT) {
    s0 = fma(a0[i], b0[i], s0);
    if (a1) s1 = fma(a1[i], b1[i], s1);
  }
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = s0; red[1][threadIdx.x >> 5] = s1; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t0 = 0.0, t1 = 0.0;
    for (int w = 0; w < CHT / 32; ++w) { t0 += red[0][w]; t1 += red[1][w]; }
    part[2 * blockIdx.x] = t0;
    part[2 * blockIdx.x + 1] = t1;
  }
}
__global__ void k_dots_sum(int nb, const double *__restrict__ part, double *__restrict__ out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double t0 = 0.0, t1 = 0.0;
    for (int b = 0; b < nb; ++b) { t0 += part[2 * b]; t1 += part[2 * b + 1]; }
    out[0] = t0;
    out[1] = t1;
  }
}
// x += nu p; r -= nu z
__global__ void k_cg_update(int n, double nu, const double *__restrict__ p,
                            const double *__restrict__ z, double *__restrict__ x,
                            double *__restrict__ r) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  x[i] = fma(nu, p[i], x[i]);
  r[i] = fma(-nu, z[i], r[i]);
}
// p = y + mu p
__global__ void k_cg_dir(int n, double mu, const double *__restrict__ y, double *__restrict__ p) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = fma(mu, p[i], y[i]);
}
// uniform [0, 1) sketch entries from a counter hash (splitmix64), seeded
__global__ void k_ch_omega(long long count, unsigned long long seed, double *__restrict__ O) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  O[i] = (double)(z >> 11) * 0x1.0p-53;
}

// ---------------------------------------------------------------- host ----

template <class T>
static T *dev_alloc(CholFactor &F, size_t count) {
  void *p = nullptr;
  CCK(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T)));
  F.allocs.push_back(p);
  F.fac_bytes += (long long)(std::max<size_t>(count, 1) * sizeof(T));
  return (T *)p;
}

static void set_smem(const void *fn, size_t bytes) {
  CCK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

constexpr size_t CH_SMEM = (size_t)CH_MAXM * (CH_MAXM + 1) * sizeof(double);
constexpr size_t CH_NODE_SMEM = 220 * 1024;  // of the 227 KB a CTA can have

// Factor A (n x n, lda; read only), leaves of ni rows (npart's tree), singular
// values above tol kept, at most ncol per node.  ps = 0: the scaled block
// columns are compressed by their exact right singular vectors (RS = 'S');
// ps > 0: by those of a ps-row uniform [0, 1) sketch (RS = 'R', as the
// reference's random_number Omega).  Returns 0 or a status: 1 not positive
// definite, 2 a node of more than 128 rows.
int hss_chol_factor_core(int n, const double *A, long long lda, int ni, double tol, int ncol,
                         int ps, unsigned long long seed, CholFactor &F, cudaStream_t st) {
  F.n = n;
  const HostTree t = make_tree(n, ni);
  const int ltr = t.ltr;
  if (t.mmax > CH_MAXM) return 2;
  std::vector<int> height(ltr + 1, 0);
  for (int i = 1; i <= ltr; ++i)
    if (!t.leaf(i)) height[i] = 1 + std::max(height[t.c1[i]], height[t.c2[i]]);
  const int H = height[ltr];
  static bool attr = false;
  if (!attr) {
    set_smem((const void *)k_ch_chol, CH_SMEM);
    set_smem((const void *)k_ch_node, CH_NODE_SMEM);
    attr = true;
  }
  const size_t nn = (size_t)n * n;
  double *cur = pool<double>("hc_A0", nn), *nxt = pool<double>("hc_A1", nn);
  double *X = pool<double>("hc_X", nn), *Xt = pool<double>("hc_Xt", nn);
  const int nslot = t.lm;  // a level factors at most one node per leaf
  double *Lb = pool<double>("hc_L", nslot * CH_SLOT), *Ib = pool<double>("hc_I", nslot * CH_SLOT);
  double *Pb = pool<double>("hc_P", nslot * CH_SLOT), *PTb = pool<double>("hc_PT", nslot * CH_SLOT);
  double *Gb = pool<double>("hc_G", 4 * nslot * CH_SLOT), *Wb = pool<double>("hc_W", nslot * CH_SLOT);
  int *status = pool<int>("hc_status", 2);
  double *Om = nullptr, *Ys = nullptr;
  if (ps > 0) {
    Om = pool<double>("hc_omega", (size_t)ps * n);
    Ys = pool<double>("hc_sketch", (size_t)nslot * ps * CH_MAXM);
    const long long cnt = (long long)ps * n;
    k_ch_omega<<<(unsigned)((cnt + 255) / 256), 256, 0, st>>>(cnt, seed, Om);
  }
  CCK(cudaMemsetAsync(status, 0, 2 * sizeof(int), st));
  CCK(cudaMemcpy2DAsync(cur, sizeof(double) * n, A, sizeof(double) * lda, sizeof(double) * n, n,
                        cudaMemcpyDeviceToDevice, st));
  std::vector<int> ids, sizes;  // the active nodes, left to right
  for (int i = 1, it = 0; i <= ltr; ++i)
    if (t.leaf(i)) { ids.push_back(i); sizes.push_back(t.m[it++]); }
  int Nc = n;
  for (int h = 0; h <= H; ++h) {
    // the parents of this height take over their (adjacent) children's ranges
    for (int p = 1; p <= ltr; ++p) {
      if (t.leaf(p) || height[p] != h) continue;
      const int a = (int)(std::find(ids.begin(), ids.end(), t.c1[p]) - ids.begin());
      if (a + 1 >= (int)ids.size() || ids[a + 1] != t.c2[p])
        throw HssError{"hsschol: children not adjacent"};
      ids[a] = p;
      sizes[a] += sizes[a + 1];
      ids.erase(ids.begin() + a + 1);
      sizes.erase(sizes.begin() + a + 1);
    }
    if (h == H) break;
    const int na = (int)ids.size();
    std::vector<ChNode> nodes(na);
    std::vector<ChNode> cand;
    for (int k = 0, o = 0; k < na; ++k) {
      nodes[k] = ChNode{o, sizes[k], 0, sizes[k], 0, -1, 0};
      // mat2hsssvd.f90:136, :210: only blocks of 20 or more rows with 20 or
      // more other variables are compressed
      if (height[ids[k]] == h && sizes[k] >= 20 && Nc - sizes[k] >= 20) {
        if (sizes[k] > CH_MAXM) return 2;
        nodes[k].slot = (int)cand.size();
        cand.push_back(nodes[k]);
      }
      o += sizes[k];
    }
    std::vector<int> rk(cand.size(), 0);
    if (!cand.empty()) {
      ChNode *dc = pool<ChNode>("hc_cand", cand.size());
      stage_h2d(dc, cand.data(), cand.size() * sizeof(ChNode), st);
      int mm = 0;  // the shared memory of the level's largest block: more CTAs per SM
      for (auto &q : cand) mm = std::max(mm, q.m);
      k_ch_chol<<<(unsigned)cand.size(), CHT, sizeof(double) * mm * (mm | 1), st>>>(dc, cur, Nc, Lb,
                                                                                   Ib, status);
      std::vector<GemmDesc> g;  // X(:, I) = Ah(:, I) L^{-T}
      for (auto &q : cand)
        g.push_back(GemmDesc{cur + (long long)q.o * Nc, Ib + (size_t)q.slot * CH_SLOT,
                             X + (long long)q.o * Nc, Nc, q.m, Nc, Nc, q.m, q.m, 0, 0, 1});
      launch_gemm(g, 0, st);
      k_ch_zero_own<<<(unsigned)cand.size(), 256, 0, st>>>(dc, X, Nc);
      std::vector<const double *> xs;
      std::vector<int> rows, cols;
      std::vector<long long> lds;
      std::vector<double *> P, PT;
      if (ps > 0) {  // sketches Omega(:, 0:Nc) X(:, I), ps x m
        std::vector<GemmDesc> gs;
        for (auto &q : cand)
          gs.push_back(GemmDesc{Om, X + (long long)q.o * Nc, Ys + (size_t)q.slot * ps * CH_MAXM, ps,
                                Nc, ps, ps, q.m, Nc, 0, 0});
        launch_gemm(gs, 0, st);
      }
      for (auto &q : cand) {
        if (ps > 0) {
          xs.push_back(Ys + (size_t)q.slot * ps * CH_MAXM);
          rows.push_back(ps);
          lds.push_back(ps);
        } else {
          xs.push_back(X + (long long)q.o * Nc);
          rows.push_back(Nc);
          lds.push_back(Nc);
        }
        cols.push_back(q.m);
        P.push_back(Pb + (size_t)q.slot * CH_SLOT);
        PT.push_back(PTb + (size_t)q.slot * CH_SLOT);
      }
      int hs[2] = {0, 0};
      CCK(cudaMemcpyAsync(hs, status, sizeof hs, cudaMemcpyDeviceToHost, st));
      rk = tall_right_bases(xs, rows, cols, lds, P, PT, tol, st);  // synchronises
      if (hs[0]) return 1;
    }
    // ranks (at most ncol), the next level's ranges, the factor offsets
    ChLevel L;
    L.Nc = Nc;
    long long ftot = 0;
    std::vector<ChNode> comp;
    for (int k = 0, o2 = 0; k < na; ++k) {
      ChNode &q = nodes[k];
      const int r = q.slot >= 0 ? std::max(0, std::min(rk[q.slot], ncol)) : q.m;
      if (q.slot >= 0 && r < q.m) {
        q.rk = r;
        q.ir = q.m - r;
        q.f = ftot;
        ftot += 2LL * q.m * q.m;
        F.max_rank = std::max(F.max_rank, r);
      } else {
        q.rk = q.m;
        q.ir = 0;
      }
      q.o2 = o2;
      o2 += q.rk;
      sizes[k] = q.rk;
    }
    for (const ChNode &q : nodes)
      if (q.ir > 0) comp.push_back(q);
    const int Nc2 = nodes.empty() ? 0 : nodes.back().o2 + nodes.back().rk;
    L.Nc2 = Nc2;
    L.fac = dev_alloc<double>(F, (size_t)ftot);
    L.d_nodes = dev_alloc<ChNode>(F, nodes.size());
    CCK(cudaMemcpyAsync(L.d_nodes, nodes.data(), nodes.size() * sizeof(ChNode),
                        cudaMemcpyHostToDevice, st));
    if (!comp.empty()) {
      ChNode *dq = pool<ChNode>("hc_comp", comp.size());
      stage_h2d(dq, comp.data(), comp.size() * sizeof(ChNode), st);
      size_t all = 0, l2 = 0;
      for (auto &q : comp) {
        all = std::max(all, sizeof(double) * (q.m | 1) * (2 * q.m + q.rk));
        l2 = std::max(l2, sizeof(double) * (q.m | 1) * q.m);
      }
      const int sm = all <= CH_NODE_SMEM;
      k_ch_node<<<(unsigned)comp.size(), CHT + 32, sm ? all : l2, st>>>(dq, Lb, Pb, Gb, L.fac, Wb,
                                                                       sm);
    }
    // congruence Ah' = W^T Ah W: X2 = Ah W, Xt = X2^T, Ah' = Xt W
    {
      std::vector<GemmDesc> g1, g2;
      for (auto &q : comp) {
        if (q.rk == 0) continue;  // every variable of the node eliminated
        const double *Wq = Wb + (size_t)q.slot * CH_SLOT;
        g1.push_back(GemmDesc{cur + (long long)q.o * Nc, Wq, X + (long long)q.o2 * Nc, Nc, q.m, Nc,
                              Nc, q.rk, q.m, 0, 0});
        g2.push_back(GemmDesc{Xt + (long long)q.o * Nc2, Wq, nxt + (long long)q.o2 * Nc2, Nc2, q.m,
                              Nc2, Nc2, q.rk, q.m, 0, 0});
      }
      const unsigned gx = (unsigned)std::min<long long>(((long long)Nc * CH_MAXM + 255) / 256, 512);
      if (Nc2 > 0) {
        launch_gemm(g1, 0, st);
        k_ch_copy_cols<<<dim3(gx, (unsigned)na), 256, 0, st>>>(L.d_nodes, na, Nc, cur, Nc, X, Nc);
        transpose(Nc, Nc2, X, Nc, Xt, Nc2, st);
        launch_gemm(g2, 0, st);
        k_ch_copy_cols<<<dim3(gx, (unsigned)na), 256, 0, st>>>(L.d_nodes, na, Nc2, Xt, Nc2, nxt,
                                                                Nc2);
      }
    }
    L.nodes = nodes;
    F.lv.push_back(L);
    std::swap(cur, nxt);
    Nc = Nc2;
  }
  // the root: a plain Cholesky of what is left (mat2hsssvd.f90:266-278)
  F.Nroot = Nc;
  if (Nc > CH_MAXM) return 2;
  F.root = dev_alloc<double>(F, (size_t)Nc * Nc);
  if (Nc > 0) {
    std::vector<ChNode> r1{ChNode{0, Nc, 0, Nc, 0, 0, 0}};
    ChNode *dr = pool<ChNode>("hc_cand", 1);
    stage_h2d(dr, r1.data(), sizeof(ChNode), st);
    CCK(cudaMemsetAsync(status, 0, sizeof(int), st));
    k_ch_chol<<<1, CHT, CH_SMEM, st>>>(dr, cur, Nc, Lb, Ib, status);
    CCK(cudaMemcpyAsync(F.root, Lb, sizeof(double) * Nc * Nc, cudaMemcpyDeviceToDevice, st));
    int hs = 0;
    CCK(cudaMemcpyAsync(&hs, status, sizeof hs, cudaMemcpyDeviceToHost, st));
    CCK(cudaStreamSynchronize(st));
    if (hs) return 1;
  }
  CCK(cudaGetLastError());
  return 0;
}

// B (n x nrhs, ldb) <- A_hss^{-1} B with the factor (solvecholsvd).
void hss_chol_solve_core(const CholFactor &F, double *B, long long ldb, int nrhs, cudaStream_t st) {
  const int n = F.n, nl = (int)F.lv.size();
  std::vector<long long> off(nl + 2, 0);
  std::vector<int> dim(nl + 1);
  for (int h = 0; h < nl; ++h) dim[h] = F.lv[h].Nc;
  dim[nl] = F.Nroot;
  for (int h = 0; h <= nl; ++h) off[h + 1] = off[h] + (long long)dim[h] * nrhs;
  double *Y = pool<double>("hc_Y", (size_t)std::max<long long>(off[nl + 1], 1));
  CCK(cudaMemcpy2DAsync(Y, sizeof(double) * n, B, sizeof(double) * ldb, sizeof(double) * n, nrhs,
                        cudaMemcpyDeviceToDevice, st));
  static bool attr = false;
  if (!attr) {
    const int most = CH_MAXM * (CH_MAXM | 1) * (int)sizeof(double);
    CCK(cudaFuncSetAttribute(k_ch_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CCK(cudaFuncSetAttribute(k_ch_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    attr = true;
  }
  auto smem = [&](int h) {  // one matrix of the level's largest node
    size_t m = 1;
    for (const auto &q : F.lv[h].nodes)
      if (q.ir > 0) m = std::max<size_t>(m, q.m);
    return m * (m | 1) * sizeof(double);
  };
  for (int h = 0; h < nl; ++h)
    k_ch_fwd<<<(unsigned)F.lv[h].nodes.size(), CHT, smem(h), st>>>(
        F.lv[h].d_nodes, F.lv[h].fac, Y + off[h], dim[h], Y + off[h + 1], dim[h + 1], nrhs);
  if (F.Nroot > 0) k_ch_root<<<nrhs, 32, 0, st>>>(F.Nroot, F.root, Y + off[nl], F.Nroot);
  for (int h = nl - 1; h >= 0; --h)
    k_ch_bwd<<<(unsigned)F.lv[h].nodes.size(), CHT, smem(h), st>>>(
        F.lv[h].d_nodes, F.lv[h].fac, Y + off[h], dim[h], Y + off[h + 1], dim[h + 1], nrhs);
  CCK(cudaMemcpy2DAsync(B, sizeof(double) * ldb, Y, sizeof(double) * n, sizeof(double) * n, nrhs,
                        cudaMemcpyDeviceToDevice, st));
}

static void gemv(int n, const double *A, long long lda, const double *x, double *y, double *part,
                 cudaStream_t st) {
  const int nch = (n + GV_CHUNK - 1) / GV_CHUNK;
  k_gemv_part<<<dim3((n + 127) / 128, nch), 128, 0, st>>>(n, A, lda, x, part);
  k_gemv_sum<<<(n + 255) / 256, 256, 0, st>>>(n, nch, part, y);
}

// two dot products (the second optional) read back to the host
static void dots(int n, const double *a0, const double *b0, const double *a1, const double *b1,
                 double *out, double *part, double *dout, cudaStream_t st) {
  const int nb = std::min(256, (n + CHT - 1) / CHT);
  k_dots<<<nb, CHT, 0, st>>>(n, a0, b0, a1, b1, part);
  k_dots_sum<<<1, 32, 0, st>>>(nb, part, dout);
  CCK(cudaMemcpyAsync(out, dout, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
  CCK(cudaStreamSynchronize(st));
}

// Preconditioned CG (cg, mat2hsssvd.f90:674-726) on the device: x <- the
// solution of A x = b (A n x n, lda), preconditioner the HSS Cholesky solve
// when F is given.  Stops when |r| / |b| < tau or after maxit + 1 steps, as the
// reference's loop.  Returns the steps; *relres the last relative residual.
int hss_chol_pcg_core(const CholFactor *F, int n, const double *A, long long lda, const double *b,
                      double *x, double tau, int maxit, double *relres, cudaStream_t st) {
  double *v = pool<double>("hc_cg", (size_t)5 * n);
  double *r = v, *p = v + n, *y = v + 2 * n, *z = v + 3 * n;
  const int nch = (n + GV_CHUNK - 1) / GV_CHUNK;
  double *part = pool<double>("hc_cg_part", (size_t)std::max(nch * n, 512));
  double *dout = pool<double>("hc_cg_dot", 2);
  CCK(cudaMemcpyAsync(r, b, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
  CCK(cudaMemcpyAsync(p, b, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
  CCK(cudaMemsetAsync(x, 0, sizeof(double) * n, st));
  double h[2];
  dots(n, b, b, nullptr, nullptr, h, part, dout, st);
  const double tb = sqrt(h[0]);
  if (F) hss_chol_solve_core(*F, p, n, 1, st);
  CCK(cudaMemcpyAsync(y, p, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
  double res = tb > 0.0 ? 1.0 : 0.0;
  int it = 0;
  dots(n, y, r, nullptr, nullptr, h, part, dout, st);
  double dt = h[0];
  const unsigned g = (unsigned)((n + 255) / 256);
  while (res >= tau && it <= maxit) {
    ++it;
    gemv(n, A, lda, p, z, part, st);
    dots(n, p, z, nullptr, nullptr, h, part, dout, st);
    const double nu = dt / h[0];
    k_cg_update<<<g, 256, 0, st>>>(n, nu, p, z, x, r);
    CCK(cudaMemcpyAsync(y, r, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
    if (F) hss_chol_solve_core(*F, y, n, 1, st);
    dots(n, y, r, r, r, h, part, dout, st);
    const double mu = h[0] / dt;
    dt = h[0];
    k_cg_dir<<<g, 256, 0, st>>>(n, mu, y, p);
    res = sqrt(h[1]) / tb;
  }
  CCK(cudaStreamSynchronize(st));
  *relres = res;
  return it;
}

}  // namespace hss
