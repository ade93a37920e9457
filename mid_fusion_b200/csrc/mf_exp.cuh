// The bilateral filter's exponential and its argument's quotient.
#pragma once

namespace mf {

// 2^(j / 64), rounded to nearest
__constant__ double c_exp2_64[64] = {
    0x1.0000000000000p+0, 0x1.02c9a3e778061p+0, 0x1.059b0d3158574p+0, 0x1.0874518759bc8p+0,
    0x1.0b5586cf9890fp+0, 0x1.0e3ec32d3d1a2p+0, 0x1.11301d0125b51p+0, 0x1.1429aaea92de0p+0,
    0x1.172b83c7d517bp+0, 0x1.1a35beb6fcb75p+0, 0x1.1d4873168b9aap+0, 0x1.2063b88628cd6p+0,
    0x1.2387a6e756238p+0, 0x1.26b4565e27cddp+0, 0x1.29e9df51fdee1p+0, 0x1.2d285a6e4030bp+0,
    0x1.306fe0a31b715p+0, 0x1.33c08b26416ffp+0, 0x1.371a7373aa9cbp+0, 0x1.3a7db34e59ff7p+0,
    0x1.3dea64c123422p+0, 0x1.4160a21f72e2ap+0, 0x1.44e086061892dp+0, 0x1.486a2b5c13cd0p+0,
    0x1.4bfdad5362a27p+0, 0x1.4f9b2769d2ca7p+0, 0x1.5342b569d4f82p+0, 0x1.56f4736b527dap+0,
    0x1.5ab07dd485429p+0, 0x1.5e76f15ad2148p+0, 0x1.6247eb03a5585p+0, 0x1.6623882552225p+0,
    0x1.6a09e667f3bcdp+0, 0x1.6dfb23c651a2fp+0, 0x1.71f75e8ec5f74p+0, 0x1.75feb564267c9p+0,
    0x1.7a11473eb0187p+0, 0x1.7e2f336cf4e62p+0, 0x1.82589994cce13p+0, 0x1.868d99b4492edp+0,
    0x1.8ace5422aa0dbp+0, 0x1.8f1ae99157736p+0, 0x1.93737b0cdc5e5p+0, 0x1.97d829fde4e50p+0,
    0x1.9c49182a3f090p+0, 0x1.a0c667b5de565p+0, 0x1.a5503b23e255dp+0, 0x1.a9e6b5579fdbfp+0,
    0x1.ae89f995ad3adp+0, 0x1.b33a2b84f15fbp+0, 0x1.b7f76f2fb5e47p+0, 0x1.bcc1e904bc1d2p+0,
    0x1.c199bdd85529cp+0, 0x1.c67f12e57d14bp+0, 0x1.cb720dcef9069p+0, 0x1.d072d4a07897cp+0,
    0x1.d5818dcfba487p+0, 0x1.da9e603db3285p+0, 0x1.dfc97337b9b5fp+0, 0x1.e502ee78b3ff6p+0,
    0x1.ea4afa2a490dap+0, 0x1.efa1bee615a27p+0, 0x1.f50765b6e4540p+0, 0x1.fa7c1819e90d8p+0,
};

// exp of a float argument at most 0, rounded to the nearest float (what the
// host's expf returns in all but rare cases): the double exponential rounded
// to float.  Table-driven reduction (P. T. P. Tang, "Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic", 1989): x = k ln2 / 64 + r with |r| < 0.0055, exp(x) =
// 2^(k / 64) (1 + r + ... + r^5 / 120), good to about 2^-53.  Half the FP64
// instructions of the general double exp, whose results rounded to float it
// equals for every float argument at most 0 (NaN aside, which gives 0 here).
// `tab` is c_exp2_64 in shared memory.
__device__ __forceinline__ float exp_nearest(float x, const double* tab) {
  const double xd = (double)fmaxf(x, -110.f);   // exp(-104) rounds to 0
  const double kd = fma(xd, 0x1.71547652b82fep+6, 0x1.8p52);   // round to an integer
  const int k = __double2loint(kd);
  const double kf = kd - 0x1.8p52;
  double r = fma(kf, -0x1.62e42fefa39efp-7, xd);
  r = fma(kf, -0x1.abc9e3b39803fp-62, r);
  double q = fma(r, 1.0 / 120, 1.0 / 24);
  q = fma(q, r, 1.0 / 6);
  q = fma(q, r, 0.5);
  q = fma(q, r, 1.0);
  q = q * r;
  const double t = tab[k & 63];
  const double v = fma(t, q, t);
  return (float)__hiloint2double(__double2hiint(v) + ((k >> 6) << 20), __double2loint(v));
}

// x / 0.02f (0x1.47ae16p-6f, the float 0.1f * 0.1f * 2) with one correction
// step: equal to the IEEE quotient for every mantissa (checked over all 2^23;
// the exponent only scales it).  A quotient so small that the remainder
// underflows is off by less than exp() can show.
__device__ __forceinline__ float div_e2(float x) {
  const float rc = 0x1.8ffffep+5f, b = 0x1.47ae16p-6f;
  const float q = x * rc;
  return fmaf(fmaf(-q, b, x), rc, q);
}

}  // namespace mf
