// cexp.cuh -- complex exponential and reciprocal square root of the Stokes
// kernels, FP64.
//
// The assembly and the interior points evaluate two complex exponentials and
// one reciprocal square root per Gauss point, on the FP64 pipe that bounds
// them.  exp and sincos here are table-driven (P. T. P. Tang, "Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic", ACM TOMS 1989; the same scheme for sine and cosine by the
// addition theorem), with Cody-Waite reduction in two FMAs: 16 FP64
// operations for a sine and cosine pair, 10 for an exponential, about half of
// the general functions', which also carry the code for huge arguments.
// Arguments outside the tables' reduction (|phase| above 1e7, |exponent|
// above 700, not finite) take the general functions.
//
// Accuracy, in u = 2^-53 of the modulus (tests/test_gpu_math.py derives and
// checks the bounds): undamped at most 2.7 (measured 2.1; the general
// functions with the same products 1.7), damped at most 6.1 (3.5; 2.7), sines
// below pi/128 2.1 relative, 1/sqrt at most 1.6 (1.24; CUDA's rsqrt 1.01).
// The results built on them are no further from 64-bit values than with the
// general functions, since the radial functions round fewer terms.
#pragma once

#include <cuda_runtime.h>

namespace bem {

// sin(j pi / 64), j = 0..32, and 2^(j / 64), j = 0..63, correctly rounded.
__device__ const double kSinTab[33] = {
    0x0.0p+0, 0x1.91f65f10dd814p-5, 0x1.917a6bc29b42cp-4,
    0x1.2c8106e8e613ap-3, 0x1.8f8b83c69a60bp-3, 0x1.f19f97b215f1bp-3,
    0x1.294062ed59f06p-2, 0x1.58f9a75ab1fddp-2, 0x1.87de2a6aea963p-2,
    0x1.b5d1009e15cc0p-2, 0x1.e2b5d3806f63bp-2, 0x1.073879922ffeep-1,
    0x1.1c73b39ae68c8p-1, 0x1.30ff7fce17035p-1, 0x1.44cf325091dd6p-1,
    0x1.57d69348ceca0p-1, 0x1.6a09e667f3bcdp-1, 0x1.7b5df226aafafp-1,
    0x1.8bc806b151741p-1, 0x1.9b3e047f38741p-1, 0x1.a9b66290ea1a3p-1,
    0x1.b728345196e3ep-1, 0x1.c38b2f180bdb1p-1, 0x1.ced7af43cc773p-1,
    0x1.d906bcf328d46p-1, 0x1.e212104f686e5p-1, 0x1.e9f4156c62ddap-1,
    0x1.f0a7efb9230d7p-1, 0x1.f6297cff75cb0p-1, 0x1.fa7557f08a517p-1,
    0x1.fd88da3d12526p-1, 0x1.ff621e3796d7ep-1, 0x1.0000000000000p+0,
};
__device__ const double kExpTab[64] = {
    0x1.0000000000000p+0, 0x1.02c9a3e778061p+0, 0x1.059b0d3158574p+0,
    0x1.0874518759bc8p+0, 0x1.0b5586cf9890fp+0, 0x1.0e3ec32d3d1a2p+0,
    0x1.11301d0125b51p+0, 0x1.1429aaea92de0p+0, 0x1.172b83c7d517bp+0,
    0x1.1a35beb6fcb75p+0, 0x1.1d4873168b9aap+0, 0x1.2063b88628cd6p+0,
    0x1.2387a6e756238p+0, 0x1.26b4565e27cddp+0, 0x1.29e9df51fdee1p+0,
    0x1.2d285a6e4030bp+0, 0x1.306fe0a31b715p+0, 0x1.33c08b26416ffp+0,
    0x1.371a7373aa9cbp+0, 0x1.3a7db34e59ff7p+0, 0x1.3dea64c123422p+0,
    0x1.4160a21f72e2ap+0, 0x1.44e086061892dp+0, 0x1.486a2b5c13cd0p+0,
    0x1.4bfdad5362a27p+0, 0x1.4f9b2769d2ca7p+0, 0x1.5342b569d4f82p+0,
    0x1.56f4736b527dap+0, 0x1.5ab07dd485429p+0, 0x1.5e76f15ad2148p+0,
    0x1.6247eb03a5585p+0, 0x1.6623882552225p+0, 0x1.6a09e667f3bcdp+0,
    0x1.6dfb23c651a2fp+0, 0x1.71f75e8ec5f74p+0, 0x1.75feb564267c9p+0,
    0x1.7a11473eb0187p+0, 0x1.7e2f336cf4e62p+0, 0x1.82589994cce13p+0,
    0x1.868d99b4492edp+0, 0x1.8ace5422aa0dbp+0, 0x1.8f1ae99157736p+0,
    0x1.93737b0cdc5e5p+0, 0x1.97d829fde4e50p+0, 0x1.9c49182a3f090p+0,
    0x1.a0c667b5de565p+0, 0x1.a5503b23e255dp+0, 0x1.a9e6b5579fdbfp+0,
    0x1.ae89f995ad3adp+0, 0x1.b33a2b84f15fbp+0, 0x1.b7f76f2fb5e47p+0,
    0x1.bcc1e904bc1d2p+0, 0x1.c199bdd85529cp+0, 0x1.c67f12e57d14bp+0,
    0x1.cb720dcef9069p+0, 0x1.d072d4a07897cp+0, 0x1.d5818dcfba487p+0,
    0x1.da9e603db3285p+0, 0x1.dfc97337b9b5fp+0, 0x1.e502ee78b3ff6p+0,
    0x1.ea4afa2a490dap+0, 0x1.efa1bee615a27p+0, 0x1.f50765b6e4540p+0,
    0x1.fa7c1819e90d8p+0,
};

// The constants as operands from constant memory: as literals each costs two
// moves per use, which was a third of the kernels' instructions.
__constant__ double kCx[14] = {
    0x1.45f306dc9c883p+4,  // 64 / pi
    0x1.921fb54442d18p-5,  // pi / 64, high part
    0x1.1a62633145c07p-59,  // ... low part
    0x1.71547652b82fep+6,  // 64 / ln 2
    0x1.62e42fefa39efp-7,  // ln 2 / 64, high part
    0x1.abc9e3b39803fp-62,  // ... low part
    6755399441055744.0,  // 1.5 * 2^52: adding it rounds to an integer in the low word
    -1.0 / 5040.0,
    1.0 / 120.0,
    -1.0 / 6.0,
    -1.0 / 720.0,
    1.0 / 24.0,
    1.0 / 6.0,
    0.375,
};

// A CTA's copy of the tables in shared memory: sine and cosine of j pi / 64.
struct CexpTable {
  double2 sc[128];
  double e2[64];
};
// By all threads of the CTA; the caller synchronises.
__device__ __forceinline__ void cexp_table_fill(CexpTable& t) {
  for (int j = threadIdx.x; j < 128; j += blockDim.x) {
    const int q = j >> 5, i = j & 31;  // quadrant, index inside it
    const double a = kSinTab[i], b = kSinTab[32 - i];  // sine and cosine in the first quadrant
    const double s = (q & 1) ? b : a, c = (q & 1) ? a : b;
    t.sc[j] = make_double2((q & 2) ? -s : s, (q == 1 || q == 2) ? -c : c);
  }
  for (int j = threadIdx.x; j < 64; j += blockDim.x) t.e2[j] = kExpTab[j];
}

static __device__ __noinline__ double2 cexp_general(double re, double im) {
  double s, c;
  sincos(im, &s, &c);
  const double e = exp(re);
  return make_double2(e * c, e * s);
}

// scale * exp(re + i im); damped = false when re is known to be zero.
__device__ __forceinline__ double2 cexp_tab(const CexpTable& tab, double re, double im, double scale, bool damped) {
  // high words of 1e7 and 700 (NaN and infinity are above)
  if ((unsigned)(__double2hiint(im) & 0x7fffffff) >= 0x416312d0u ||
      (unsigned)(__double2hiint(re) & 0x7fffffff) >= 0x4085e000u) {
    const double2 g = cexp_general(re, im);
    return make_double2(g.x * scale, g.y * scale);
  }
  const double kt = fma(im, kCx[0], kCx[6]);  // 64 / pi
  const int k = __double2loint(kt);
  const double kd = kt - kCx[6];
  double r = fma(-kd, kCx[1], im);  // pi / 64 in two parts
  r = fma(-kd, kCx[2], r);
  const double r2 = r * r;  // |r| <= pi / 128
  const double sp = fma(r2, fma(r2, kCx[7], kCx[8]), kCx[9]);
  const double sr = fma(r2 * r, sp, r);                                         // sin r
  const double cr = r2 * fma(r2, fma(r2, kCx[10], kCx[11]), -0.5);      // cos r - 1
  const double2 t = tab.sc[k & 127];
  double e = scale;
  if (damped) {
    const double mt = fma(re, kCx[3], kCx[6]);  // 64 / ln 2
    const int m = __double2loint(mt);
    const double md = mt - kCx[6];
    double x = fma(-md, kCx[4], re);  // ln 2 / 64 in two parts
    x = fma(-md, kCx[5], x);
    const double p = fma(x * x, fma(x, fma(x, fma(x, kCx[8], kCx[11]), kCx[12]), 0.5), x);  // exp x - 1
    const double f = tab.e2[m & 63];
    const double g = fma(f, p, f);
    e *= __hiloint2double(__double2hiint(g) + ((m >> 6) << 20), __double2loint(g));
  }
  return make_double2(e * fma(-t.x, sr, fma(t.y, cr, t.y)), e * fma(t.y, sr, fma(t.x, cr, t.x)));
}

// 1 / sqrt(x), x > 0 and normal: the hardware's approximation (measured within
// 2^-20.08) refined by one step of Householder's third-order iteration.
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rsqrt_fast(double x) {
  const double y = rsqrt_seed(x);
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(kCx[13], e, 0.5), y);
}

}  // namespace bem
