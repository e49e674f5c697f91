// The rounding helpers and the Jacobi angle of the kernels on arrays of operands, and the
// leaf solvers' iterations as plain loops, one thread per matrix (tests/test_gpu_bits.py).
#include "hss_common.cuh"
#include "hss_jacobi.cuh"

using namespace hss;

__global__ void k_ops(int op, int n, const double *a, const double *b, const double *c, double *x,
                      double *y, double *z) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (op == 0) sqrt_rcp_rn(a[i], x[i], y[i]);
  if (op == 1) x[i] = quot_rn(a[i], b[i]);
  if (op == 2) x[i] = rcp_rn(a[i]);
  if (op == 3) {
    const HousePar h = house_par(a[i], b[i]);
    x[i] = h.beta;
    y[i] = h.tau;
    z[i] = h.scale;
  }
  if (op == 4) {
    double t = 0.0;
    y[i] = jacobi_tan(a[i], b[i], c[i], z[i], t);
    x[i] = t;
  }
}

constexpr int M = 32;
struct Work {
  double D[M], E[M], U[M * M], V[M * M];
};
__device__ void sort_columns(int m, double *D, double *A, double *B) {
  for (int i = 0; i < m - 1; ++i) {
    int k = i;
    for (int j = i + 1; j < m; ++j)
      if (D[j] < D[k]) k = j;
    if (k == i) continue;
    const double t = D[i];
    D[i] = D[k];
    D[k] = t;
    for (int r = 0; r < m; ++r) {
      const double u = A[r + i * M];
      A[r + i * M] = A[r + k * M];
      A[r + k * M] = u;
      if (!B) continue;
      const double v = B[r + i * M];
      B[r + i * M] = B[r + k * M];
      B[r + k * M] = v;
    }
  }
}

// Implicit QL with Wilkinson's shift, matrix q of m[q] rows from d, e + off[q]: w ascending,
// vectors in Z + zoff[q] (m x m, by columns)
__global__ void k_ql(int n, const int *m_, const int *off, const long long *zoff, const double *d,
                     const double *e, Work *ws, double *w, double *Z) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int m = m_[q], o = off[q];
  double *D = ws[q].D, *E = ws[q].E, *V = ws[q].V;
  for (int i = 0; i < m; ++i) {
    D[i] = d[o + i];
    E[i] = i < m - 1 ? e[o + i] : 0.0;
    for (int r = 0; r < m; ++r) V[r + i * M] = r == i ? 1.0 : 0.0;
  }
  for (int l = 0; l < m; ++l)
    for (int it = 0; it < 30 * m; ++it) {
      int mm = l;
      while (mm < m - 1 && !(fabs(E[mm]) <= HSS_EPS * (fabs(D[mm]) + fabs(D[mm + 1])))) ++mm;
      if (mm == l) break;
      double g = (D[l + 1] - D[l]) / (2.0 * E[l]);
      double r = sqrt(fma(g, g, 1.0));
      g = D[mm] - D[l] + E[l] / (g + copysign(r, g));
      double sn = 1.0, cs = 1.0, p = 0.0;
      for (int i = mm - 1; i >= l; --i) {
        const double f = sn * E[i], b = cs * E[i];
        r = sqrt(fma(f, f, g * g));
        E[i + 1] = r;
        const double rinv = 1.0 / r;
        sn = f * rinv;
        cs = g * rinv;
        g = D[i + 1] - p;
        r = fma(2.0 * cs, b, (D[i] - g) * sn);
        p = sn * r;
        D[i + 1] = g + p;
        g = cs * r - b;
        for (int k = 0; k < m; ++k) {
          const double zi = V[k + i * M], zi1 = V[k + (i + 1) * M];
          V[k + (i + 1) * M] = fma(sn, zi, cs * zi1);
          V[k + i * M] = fma(cs, zi, -(sn * zi1));
        }
      }
      D[l] = __dsub_rn(D[l], p);
      E[l] = g;
      E[mm] = 0.0;
    }
  sort_columns(m, D, V, nullptr);
  for (int i = 0; i < m; ++i) {
    w[o + i] = D[i];
    for (int r = 0; r < m; ++r) Z[zoff[q] + (long long)i * m + r] = V[r + i * M];
  }
}

// Golub-Kahan steps of an upper bidiagonal with nonzero diagonal: w ascending, U and V as Z above
__global__ void k_gk(int n, const int *m_, const int *off, const long long *zoff, const double *d,
                     const double *e, Work *ws, double *w, double *Uo, double *Vo) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int m = m_[q], o = off[q];
  double *D = ws[q].D, *E = ws[q].E, *U = ws[q].U, *V = ws[q].V;
  for (int i = 0; i < m; ++i) {
    D[i] = d[o + i];
    E[i] = i < m - 1 ? e[o + i] : 0.0;
    for (int r = 0; r < m; ++r) U[r + i * M] = V[r + i * M] = r == i ? 1.0 : 0.0;
  }
  auto rotate = [&](double *X, int k, double cs, double sn) {
    for (int r = 0; r < m; ++r) {
      const double x = X[r + k * M], x1 = X[r + (k + 1) * M];
      X[r + k * M] = fma(cs, x, sn * x1);
      X[r + (k + 1) * M] = fma(cs, x1, -(sn * x));
    }
  };
  for (int it = 0; it < 30 * m * m; ++it) {
    for (int i = 0; i + 1 < m; ++i)
      if (fabs(E[i]) <= HSS_EPS * (fabs(D[i]) + fabs(D[i + 1]))) E[i] = 0.0;
    int hi = m - 1;
    while (hi > 0 && E[hi - 1] == 0.0) --hi;
    if (hi == 0) break;
    int lo = hi - 1;
    while (lo > 0 && E[lo - 1] != 0.0) --lo;
    const double e0 = hi - 1 > lo ? E[hi - 2] : 0.0, t11 = fma(D[hi - 1], D[hi - 1], e0 * e0);
    const double t12 = D[hi - 1] * E[hi - 1];
    const double t22 = fma(D[hi], D[hi], E[hi - 1] * E[hi - 1]);
    const double dd = 0.5 * (t11 - t22);
    double mu;
    if (dd == 0.0 && t12 == 0.0) mu = t22;
    else mu = t22 - t12 * t12 / (dd + copysign(hypot(dd, t12), dd != 0.0 ? dd : 1.0));
    double y = fma(D[lo], D[lo], -mu), z = D[lo] * E[lo], bulge = 0.0;
    for (int k = lo; k < hi; ++k) {
      double t = hypot(y, z), cs = t == 0.0 ? 1.0 : y / t, sn = t == 0.0 ? 0.0 : z / t;
      if (k > lo) E[k - 1] = t;
      const double dk = D[k], ek = E[k];
      D[k] = fma(cs, dk, sn * ek);
      E[k] = fma(cs, ek, -(sn * dk));
      z = sn * D[k + 1];
      D[k + 1] = cs * D[k + 1];
      rotate(V, k, cs, sn);
      y = D[k];
      t = hypot(y, z);
      cs = t == 0.0 ? 1.0 : y / t;
      sn = t == 0.0 ? 0.0 : z / t;
      D[k] = t;
      const double e2 = E[k], d2 = D[k + 1];
      E[k] = fma(cs, e2, sn * d2);
      D[k + 1] = fma(cs, d2, -(sn * e2));
      if (k + 1 < hi) {
        bulge = sn * E[k + 1];
        E[k + 1] = cs * E[k + 1];
      }
      rotate(U, k, cs, sn);
      y = E[k];
      z = bulge;
    }
  }
  for (int i = 0; i < m; ++i)
    if (D[i] < 0.0) {
      D[i] = -D[i];
      for (int r = 0; r < m; ++r) V[r + i * M] = -V[r + i * M];
    }
  sort_columns(m, D, U, V);
  for (int i = 0; i < m; ++i) {
    w[o + i] = D[i];
    for (int r = 0; r < m; ++r) {
      Uo[zoff[q] + (long long)i * m + r] = U[r + i * M];
      Vo[zoff[q] + (long long)i * m + r] = V[r + i * M];
    }
  }
}

extern "C" {
int check_ops(int op, int n, const double *a, const double *b, const double *c, double *x, double *y,
              double *z) {
  k_ops<<<(n + 255) / 256, 256>>>(op, n, a, b, c, x, y, z);
  return (int)cudaDeviceSynchronize();
}
long long check_work_bytes() { return (long long)sizeof(Work); }
int check_leaves(int svd, int n, const int *m, const int *off, const long long *zoff, const double *d,
                 const double *e, void *work, double *w, double *U, double *V) {
  if (svd) k_gk<<<(n + 31) / 32, 32>>>(n, m, off, zoff, d, e, (Work *)work, w, U, V);
  else k_ql<<<(n + 31) / 32, 32>>>(n, m, off, zoff, d, e, (Work *)work, w, U);
  return (int)cudaDeviceSynchronize();
}
}
