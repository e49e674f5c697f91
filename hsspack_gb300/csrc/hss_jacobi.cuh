// hss_jacobi.cuh -- the rotation angle of the one-sided Jacobi (mat2hss.cu).
#pragma once
#include "hss_common.cuh"

namespace hss {

// Tangent of the Jacobi rotation of two rows with squared norms a, b > 0 and product c:
// the root of smaller modulus of c t^2 + x t - c = 0, x = b - a (t^2 + 2 zeta t = 1 with
// zeta = x / 2c), within two ulps.  False: c^2 <= jtol2 a b, nothing to rotate.  The test
// and the first estimate are FP32 on numbers brought to c's exponent by integer
// operations; two steps with FP64 residuals and an FP32 slope finish it (one leaves
// about 42 bits): seven FP64 instructions where a reciprocal, a root and a comparison in
// FP64 made it thirteen.  DHSSMM n = 2000: 16.66 ms (with one step 16.50).
__device__ __forceinline__ bool jacobi_tan(double a, double b, double c, double jtol2, double &t) {
  const int hc = __double2hiint(c), Ec = (hc >> 20) & 0x7ff;
  const int Ea = __double2hiint(a) >> 20, Eb = __double2hiint(b) >> 20;
  const double x = b - a;
  const int hx = __double2hiint(x), Ex = (hx >> 20) & 0x7ff;
  if (Ea >= 600 && Eb >= 600 && Ea < 1500 && Eb < 1500) {
    if (Ec < 450) return false;  // (c^2 / (a b) below 2^-300)
    auto mant = [](double v, int e) {  // |v| as FP32 with the exponent set to e
      return __int_as_float((e + 127) << 23 | (__double2hiint(v) & 0xfffff) << 3 |
                            (unsigned)__double2loint(v) >> 29);
    };
    const float mc = mant(c, 0);
    const int D = 2 * Ec - Ea - Eb;
    if (D < -100) return false;
    // (mantissas cut to 23 bits are within 1e-6, the factor is below that: no pair that
    // FP64 would rotate is left out)
    if (mc * mc * __int_as_float((D + 127) << 23) <= 0.99999f * (float)jtol2 * mant(a, 0) * mant(b, 0))
      return false;
    const int dx = Ex - Ec;
    if (dx < 120) {
      const float zf = dx < -120 ? 0.f : __fdividef(0.5f * mant(x, dx), mc);
      const float rf = zf < 1e15f ? sqrtf(fmaf(zf, zf, 1.f)) : zf;
      const int sg = (hx ^ hc) & 0x80000000;
      const double t0 = f64_of_f32(__fdividef(1.f, zf + rf));
      t = __hiloint2double(__double2hiint(t0) | sg, __double2loint(t0));
      // 1 / |2 c (t + zeta)| (c's sign x's)
      const double w = f64_of_f32(__fdividef(0.5f, rf * mc));
      const double sl = __hiloint2double((__double2hiint(w) - ((Ec - 1023) << 20)) | (~hx & 0x80000000),
                                         __double2loint(w));
      t = fma(fma(t, fma(t, c, x), -c), sl, t);
      t = fma(fma(t, fma(t, c, x), -c), sl, t);
      return true;
    }
  }
  if (!(c * c > jtol2 * a * b)) return false;
  const double zeta = x / (2.0 * c);
  t = copysign(1.0 / (fabs(zeta) + sqrt(fma(zeta, zeta, 1.0))), zeta);
  return true;
}

}  // namespace hss
