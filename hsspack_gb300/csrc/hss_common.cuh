// hss_common.cuh -- shared device helpers for the sm_103a HSS merge kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define HSS_EPS 1.1102230246251565e-16   /* 2^-53, LAPACK DLAMCH('Epsilon') */
#define HSS_WARP 32
#define HSS_FULL 0xffffffffu
// SMs of a GB300, for the rules that split work by them.  A constant, not the device's count:
// lanes per column and per leaf fix orders of summation, so results depend on it.
constexpr int HSS_SMS = 152;

// ---- warp all-reduce (butterfly: every lane ends with the same bits) --------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(HSS_FULL, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(HSS_FULL, v, o));
  return v;
}
__device__ __forceinline__ int warp_sum_int(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(HSS_FULL, v, o);
  return v;
}

// 1/x from the estimate y of the PTX instruction rcp.approx.ftz.f64 and one
// second-order correction: with e = 1 - x y (one fma, exact to ~2^-75),
// 1/x = y / (1 - e) = y (1 + e + e^2 + e^3 + ...), so y + y (e + e^2)
// leaves |e|^3 (far below an ulp for the estimate's accuracy) plus the final
// fma's rounding: within one ulp of 1/x for normal, finite, nonzero x (x = 0
// or infinite gives NaN).  Four FP64 instructions instead of a correctly
// rounded divide: the pole sums are FP64-pipe bound.
__device__ __forceinline__ double rcp_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// a / b within 1.5 ulp through rcp_nr (four FP64 instructions instead of a
// correctly rounded divide) for the FP64-pipe bound loops; b = 0 gives NaN.
__device__ __forceinline__ double qdiv(double a, double b) { return a * rcp_nr(b); }

// rinv = 1 / sqrt(x) and r = sqrt(x) for normal x in [2^-960, 2^960): the estimate y
// of the PTX instruction rsqrt.approx.ftz.f64 and Householder's third-order step
// y (1 + c), c = e/2 + 3 e^2 / 8 with e = 1 - x y^2; r is the same step on x y.
// Each within about one ulp, in six FP64 instructions; a correctly rounded root
// and then a reciprocal take four times that, in one dependent chain.
__device__ __forceinline__ void sqrt_pair(double x, double &r, double &rinv) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = x * y;
  const double e = fma(-h, y, 1.0);
  const double c = fma(0.375, e, 0.5) * e;
  rinv = fma(y, c, y);
  r = fma(h, c, h);
}

// Rounding to nearest from estimates within about an ulp, by Newton corrections whose
// residuals fused multiply-adds form exactly (Markstein, IBM J. Res. Dev. 34, 1990), for
// operands and results well inside the normal range.  The correction of a reciprocal
// is exact but for a divisor with a mantissa of ones: 1 / b is then a power of two and
// a little over half an ulp, the correction gives the power of two, and ones_bit adds
// the ulp.  A quotient within 2^-51 ulps of the middle of two doubles may be either.
__device__ __forceinline__ double ones_bit(double y, double b) {
  int lo = __double2loint(y);
  if ((__double2loint(b) & (__double2hiint(b) | (int)0xfff00000)) == -1) lo |= 1;
  return __hiloint2double(__double2hiint(y), lo);
}
// sqrt(x) for x in sqrt_pair's range, and y = 1 / sqrt(x) within about an ulp
__device__ __forceinline__ double sqrt_rn(double x, double &y) {
  double r0;
  sqrt_pair(x, r0, y);
  const double y2 = __hiloint2double(__double2hiint(y) - (1 << 20), __double2loint(y));  // y / 2
  return fma(fma(-r0, r0, x), y2, r0);
}
// r = sqrt(x) and 1 / r as the divide gives it: ten FP64 instructions
__device__ __forceinline__ void sqrt_rcp_rn(double x, double &r, double &rinv) {
  double y;
  r = sqrt_rn(x, y);
  rinv = ones_bit(fma(y, fma(-r, y, 1.0), y), r);
}
__device__ __forceinline__ double rcp_rn(double b) {
  const double y = rcp_nr(b);
  return ones_bit(fma(y, fma(-b, y, 1.0), y), b);
}
// a / b from y = 1 / b
__device__ __forceinline__ double div_rn(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(-q, b, a), y, q);
}
// a / b, by div_rn where both are within 2^+-480
__device__ __forceinline__ double quot_rn(double a, double b) {
  const unsigned ha = __double2hiint(a) & 0x7fffffff, hb = __double2hiint(b) & 0x7fffffff;
  constexpr unsigned lo = 0x21f00000, w = 0x5df00000 - lo;
  return ha - lo < w && hb - lo < w ? div_rn(a, b, rcp_nr(b)) : a / b;
}

// Householder reflector of (alpha, tail) with the tail's squared norm sg: beta, tau, and
// scale with v = [1; tail * scale]
struct HousePar {
  double beta, tau, scale;
};
// (one lane forms it, at a warp's FP64 price: the root and the reciprocal from estimates,
// rounded to nearest; tau = 1 + |alpha| / |beta| in one multiply-add, within 1.5 ulps where
// (beta - alpha) / beta has two)
__device__ __forceinline__ HousePar house_par(double alpha, double sg) {
  HousePar h{alpha, 0.0, 0.0};
  if (sg > 0.0) {
    const double x = fma(alpha, alpha, sg);
    const int hx = __double2hiint(x);
    if (hx >= 0x03f00000 && hx < 0x7bf00000) {  // 2^-960 <= x < 2^960
      double rt, ri;
      rt = sqrt_rn(x, ri);
      h.beta = -copysign(rt, alpha);
      h.tau = fma(fabs(alpha), ri, 1.0);
      h.scale = rcp_rn(alpha - h.beta);
    } else {
      h.beta = -copysign(sqrt(x), alpha);
      h.tau = (h.beta - alpha) / h.beta;
      h.scale = 1.0 / (alpha - h.beta);
    }
  }
  return h;
}

// |d| as FP32 rounded towards zero by integer operations (a conversion holds the
// FP64 pipe); 0 below FP32's range, infinity above
__device__ __forceinline__ float abs_f32(double d) {
  const unsigned hi = (unsigned)__double2hiint(d) & 0x7fffffffu, lo = (unsigned)__double2loint(d);
  const int e = (int)(hi >> 20) - 1023 + 127;
  if (e <= 0) return 0.f;
  if (e >= 255) return __int_as_float(0x7f800000);
  return __uint_as_float((unsigned)e << 23 | (hi & 0xfffffu) << 3 | lo >> 29);
}

// a normal FP32 number as FP64, likewise
__device__ __forceinline__ double f64_of_f32(float f) {
  const unsigned b = __float_as_uint(f);
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))),
                          (int)(b << 29));
}

// (float)d by integer operations, rounded to nearest even as the conversion is (which
// holds the FP64 pipe); results outside FP32's normal range, but 0, by the conversion
__device__ __forceinline__ float f32_of_f64(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const unsigned E = (hi >> 20) & 0x7ffu;
  if (E - 897u < 254u) {
    const unsigned u = ((E - 896u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29), rem = lo << 3;
    return __uint_as_float((hi & 0x80000000u) | (u + (rem > 0x80000000u - (u & 1u))));
  }
  if (((hi << 1) | lo) == 0) return __uint_as_float(hi);
  return (float)d;
}
// (double)f, 0 included; FP32 subnormals, infinities and NaN by the conversion
__device__ __forceinline__ double f64_from(float f) {
  const unsigned e = (__float_as_uint(f) >> 23) & 0xffu;
  if (e - 1u < 254u) return f64_of_f32(f);
  return (__float_as_uint(f) << 1) == 0 ? __hiloint2double(__float_as_int(f), 0) : (double)f;
}

// Differences of the old poles F and new roots lam = F + DIFL, formed from
// DIFL/DIFR so that no cancellation occurs near the poles
// (SRC/CauchyHssEig.f90:470-568, computfd / computdd).
//   fd(p, q) = F_p - lam_q ;  dd(p, q) = lam_p - lam_q
// Singular-value mode (sq = true, the SVD merge of MDLASD3/MDLASD8): F holds
// the poles d, lam = sigma with DIFL/DIFR = sigma - d, and the differences are
// of squares, d_p^2 - sigma_q^2 = (d_p - sigma_q)(d_p + sigma_q), each factor
// formed without cancellation (as DLASD8 does).
struct PoleDiff {
  const double *__restrict__ F;
  const double *__restrict__ difl;
  const double *__restrict__ difr;
  bool sq = false;
  __device__ __forceinline__ double fd(int p, int q) const {
    // (operands chosen before the subtractions: those take the FP64 pipe either way)
    const double lin = (__ldg(F + p) - __ldg(F + (p <= q ? q : q + 1))) - __ldg((p <= q ? difl : difr) + q);
    return sq ? lin * (__ldg(F + p) + (__ldg(F + q) + __ldg(difl + q))) : lin;
  }
  // a - b for two pole values (a^2 - b^2 in singular-value mode)
  __device__ __forceinline__ double fv(double a, double b) const {
    return sq ? (a - b) * (a + b) : a - b;
  }
  __device__ __forceinline__ double dd(int p, int q) const {
    const double lin = p < q ? (__ldg(F + p + 1) - __ldg(F + q)) + __ldg(difr + p) - __ldg(difl + q)
                             : (__ldg(F + p) - __ldg(F + q + 1)) + __ldg(difl + p) - __ldg(difr + q);
    return sq ? lin * ((__ldg(F + p) + __ldg(difl + p)) + (__ldg(F + q) + __ldg(difl + q))) : lin;
  }
};

// Merge of root r in a level batch: merge m owns positions [s[m], s[m] + K[m])
// of the level arrays; off is the prefix sum of K (P + 1 entries).
__device__ __forceinline__ int find_merge(const int *__restrict__ off, int P, int r) {
  int lo = 0, hi = P;  // off[lo] <= r < off[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (__ldg(off + mid) <= r) lo = mid; else hi = mid;
  }
  return lo;
}

// The same for one index per warp, all lanes probing (a batch's bottom levels hold
// tens of thousands of merges: 4 dependent loads instead of 16).
template <class T>
__device__ __forceinline__ int find_merge_warp(const T *__restrict__ off, int P, T r) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = P;  // off[lo] <= r < off[hi]
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) / 32;
    const int i = lo + lane * step;
    const unsigned in = __ballot_sync(HSS_FULL, i < hi && __ldg(off + i) <= r);  // lane 0 always
    const int t = 31 - __clz((int)in);
    lo = lo + t * step;
    hi = min(hi, lo + step);
  }
  return lo;
}

// Device status words written by kernels; the host maps them to INFO > 0.
enum HssStatus : int {
  HSS_OK = 0,
  HSS_SECULAR_NOCONV = 1,   // a secular root hit the iteration cap
  HSS_LEAF_NOCONV = 2,      // a leaf QL iteration hit its cap
  HSS_BAD_INPUT = 3,        // NaN / non-increasing poles
};
