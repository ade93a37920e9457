// IRLS weight and robust loss of one residual: the device's GN rows use it,
// and host builds of the same code check it against the reference.
//
// Tracking::calc_robust_weight / calc_robust_residual (apps/kfusion/src/cpp/
// tracking/tracking.cpp:1474-1532), evaluated in double and returned as float.
// None and Huber equal the reference bit for bit.  Tukey and Cauchy square in
// double here, where the reference squares through `float sq(float)`
// (utils/math_utils.h:92), i.e. rounds r / b and 1 - r^2 / b^2 to float
// first: their weights and losses differ from the reference's by at most one
// float ulp of 1 and a few ulps of the loss (the Tukey weight most, relative
// to itself, near its cutoff where it vanishes).
#pragma once
#include <cmath>
#include <cstring>

#if defined(__CUDACC__)
#define MF_ROBUST_HD __host__ __device__ __forceinline__
#else
#define MF_ROBUST_HD inline
#endif
// a table of the host's and, as name_dev, of the device's
#if defined(__CUDACC__)
#define MF_ROBUST_TABLE(type, name, ...) \
  static const type name[] = __VA_ARGS__; \
  static __device__ const type name##_dev[] = __VA_ARGS__
#else
#define MF_ROBUST_TABLE(type, name, ...) static const type name[] = __VA_ARGS__
#endif

namespace mf {

// r = 1 / (1 + j / 64) rounded to nearest, and -log(r)
struct alignas(16) LogEntry { double r, t; };
MF_ROBUST_TABLE(LogEntry, log_64, {
    {0x1p+0, 0x0p+0}, {0x1.f81f81f81f820p-1, 0x1.fc0a8b0fc03c4p-7},
    {0x1.f07c1f07c1f08p-1, 0x1.f829b0e7832f8p-6}, {0x1.e9131abf0b767p-1, 0x1.77458f632dcffp-5},
    {0x1.e1e1e1e1e1e1ep-1, 0x1.f0a30c01162a8p-5}, {0x1.dae6076b981dbp-1, 0x1.341d7961bd1d0p-4},
    {0x1.d41d41d41d41dp-1, 0x1.6f0d28ae56b4ep-4}, {0x1.cd85689039b0bp-1, 0x1.a926d3a4ad562p-4},
    {0x1.c71c71c71c71cp-1, 0x1.e27076e2af2eap-4}, {0x1.c0e070381c0e0p-1, 0x1.0d77e7cd08e5bp-3},
    {0x1.bacf914c1bad0p-1, 0x1.29552f81ff521p-3}, {0x1.b4e81b4e81b4fp-1, 0x1.44d2b6ccb7d1cp-3},
    {0x1.af286bca1af28p-1, 0x1.5ff3070a793d6p-3}, {0x1.a98ef606a63bep-1, 0x1.7ab890210d907p-3},
    {0x1.a41a41a41a41ap-1, 0x1.9525a9cf456b6p-3}, {0x1.9ec8e951033d9p-1, 0x1.af3c94e80bff3p-3},
    {0x1.999999999999ap-1, 0x1.c8ff7c79a9a20p-3}, {0x1.948b0fcd6e9e0p-1, 0x1.e27076e2af2e8p-3},
    {0x1.8f9c18f9c18fap-1, 0x1.fb9186d5e3e29p-3}, {0x1.8acb90f6bf3aap-1, 0x1.0a324e27390e2p-2},
    {0x1.8618618618618p-1, 0x1.1675cababa60fp-2}, {0x1.8181818181818p-1, 0x1.22941fbcf7966p-2},
    {0x1.7d05f417d05f4p-1, 0x1.2e8e2bae11d31p-2}, {0x1.78a4c8178a4c8p-1, 0x1.3a64c556945eap-2},
    {0x1.745d1745d1746p-1, 0x1.4618bc21c5ec2p-2}, {0x1.702e05c0b8170p-1, 0x1.51aad872df82ep-2},
    {0x1.6c16c16c16c17p-1, 0x1.5d1bdbf5809cap-2}, {0x1.6816816816817p-1, 0x1.686c81e9b14adp-2},
    {0x1.642c8590b2164p-1, 0x1.739d7f6bbd007p-2}, {0x1.6058160581606p-1, 0x1.7eaf83b82afc2p-2},
    {0x1.5c9882b931057p-1, 0x1.89a3386c1425bp-2}, {0x1.58ed2308158edp-1, 0x1.947941c2116fbp-2},
    {0x1.5555555555555p-1, 0x1.9f323ecbf984dp-2}, {0x1.51d07eae2f815p-1, 0x1.a9cec9a9a084ap-2},
    {0x1.4e5e0a72f0539p-1, 0x1.b44f77bcc8f64p-2}, {0x1.4afd6a052bf5bp-1, 0x1.beb4d9da71b7ap-2},
    {0x1.47ae147ae147bp-1, 0x1.c8ff7c79a9a21p-2}, {0x1.446f86562d9fbp-1, 0x1.d32fe7e00ebd5p-2},
    {0x1.4141414141414p-1, 0x1.dd46a04c1c4a1p-2}, {0x1.3e22cbce4a902p-1, 0x1.e744261d68789p-2},
    {0x1.3b13b13b13b14p-1, 0x1.f128f5faf06ecp-2}, {0x1.3813813813814p-1, 0x1.faf588f78f31dp-2},
    {0x1.3521cfb2b78c1p-1, 0x1.02552a5a5d0ffp-1}, {0x1.323e34a2b10bfp-1, 0x1.0723e5c1cdf41p-1},
    {0x1.2f684bda12f68p-1, 0x1.0be72e4252a83p-1}, {0x1.2c9fb4d812ca0p-1, 0x1.109f39e2d4c96p-1},
    {0x1.29e4129e4129ep-1, 0x1.154c3d2f4d5eap-1}, {0x1.27350b8812735p-1, 0x1.19ee6b467c96fp-1},
    {0x1.2492492492492p-1, 0x1.1e85f5e7040d1p-1}, {0x1.21fb78121fb78p-1, 0x1.23130d7bebf43p-1},
    {0x1.1f7047dc11f70p-1, 0x1.2795e1289b11bp-1}, {0x1.1cf06ada2811dp-1, 0x1.2c0e9ed448e8cp-1},
    {0x1.1a7b9611a7b96p-1, 0x1.307d7334f10bep-1}, {0x1.1811811811812p-1, 0x1.34e289d9ce1d2p-1},
    {0x1.15b1e5f75270dp-1, 0x1.393e0d3562a1ap-1}, {0x1.135c81135c811p-1, 0x1.3d9026a7156fbp-1},
    {0x1.1111111111111p-1, 0x1.41d8fe84672afp-1}, {0x1.0ecf56be69c90p-1, 0x1.4618bc21c5ec2p-1},
    {0x1.0c9714fbcda3bp-1, 0x1.4a4f85db03ebbp-1}, {0x1.0a6810a6810a7p-1, 0x1.4e7d811b75bb0p-1},
    {0x1.0842108421084p-1, 0x1.52a2d265bc5abp-1}, {0x1.0624dd2f1a9fcp-1, 0x1.56bf9d5b3f399p-1},
    {0x1.0410410410410p-1, 0x1.5ad404c359f2dp-1}, {0x1.0204081020408p-1, 0x1.5ee02a9241676p-1},
    {0x1.0000000000000p-1, 0x1.62e42fefa39efp-1},
});

// 1 / x up to about 2^-22, for x within [1, 1e30]
MF_ROBUST_HD float robust_rcp(float x) {
#if defined(__CUDA_ARCH__)
  return __fdividef(1.f, x);
#else
  return 1.f / x;
#endif
}

// Whether every double within 2000 units in the last place of v (normal in
// float) rounds to the same float: v is not that close to the middle between two.
MF_ROBUST_HD bool rounds_alike(double v) {
#if defined(__CUDA_ARCH__)
  const unsigned lo = (unsigned)__double2loint(v);
#else
  unsigned long long bits;
  std::memcpy(&bits, &v, 8);
  const unsigned lo = (unsigned)bits;
#endif
  return (lo & 0x1fffffffu) - (0x10000000u - 2048u) > 4096u;
}

// One correction of a quotient q ~ x / b, rc = 1 / b rounded: correctly
// rounded if q was within one unit in the last place (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990).
MF_ROBUST_HD double div_step(double x, double b, double rc, double q) {
  return fma(fma(-q, b, x), rc, q);
}

// log(s) for s in [1, 1e30], up to 2^-44 of it: s = 2^m (1 + j / 64) (1 + u)
// with |u| <= 2^-7 (P. T. P. Tang, "Table-driven implementation of the
// logarithm function in IEEE floating-point arithmetic", 1990).  u is the
// rounded difference of an exact product, and s - 1 exactly next to 1.
MF_ROBUST_HD double robust_log(double s) {
#if defined(__CUDA_ARCH__)
  const int hi = __double2hiint(s);
  const double f = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(s));
  const int j = ((hi & 0xfffff) + 0x2000) >> 14;
  const double2 e = __ldg(reinterpret_cast<const double2*>(log_64_dev) + j);
  const double r = e.x, t = e.y;
#else
  unsigned long long bits;
  std::memcpy(&bits, &s, 8);
  const int hi = (int)(bits >> 32);
  bits = (bits & 0xfffffffffffffULL) | 0x3ff0000000000000ULL;
  double f;
  std::memcpy(&f, &bits, 8);
  const int j = ((hi & 0xfffff) + 0x2000) >> 14;
  const double r = log_64[j].r, t = log_64[j].t;
#endif
  const double u = fma(f, r, -1.0);
  double p = fma(u, -1.0 / 6, 1.0 / 5);
  p = fma(u, p, -1.0 / 4);
  p = fma(u, p, 1.0 / 3);
  p = fma(u, p, -1.0 / 2);
  p = fma(u * u, p, u);
  return fma((double)((hi >> 20) - 1023), 0x1.62e42fefa39efp-1, t) + p;
}

// robust() below, for the arguments and kinds where a cheaper evaluation gives
// the same floats: the double quotients and logarithm are replaced either by
// ones that are correctly rounded too, or by approximations within 2^-44 where
// everything that close rounds to the same float (rounds_alike); false
// elsewhere (one residual in 10^4 or fewer, and extreme values).
MF_ROBUST_HD bool robust_fast(float e, int kind, float& w, float& loss) {
  const double r = e;
  const float ae = fabsf(e);
  if (kind == 3) {
    if (!(ae < 1e15f)) return false;
    // r / 2.3849 exactly rounded (one step suffices for every float mantissa)
    const double x = div_step(r, 2.3849, 1.0 / 2.3849, r * (1.0 / 2.3849));
    const double s = 1.0 + x * x;
    const double y0 = robust_rcp((float)s);
    const double wd = fma(fma(-s, y0, 1.0), y0, y0);
    const double l = 0.5 * 2.3849 * 2.3849 * robust_log(s);
    w = (float)wd;
    loss = (float)l;
    return rounds_alike(wd) && rounds_alike(l);
  }
  if (kind == 2) {
    const double b = 4.6851;
    if (!(fabs(r) <= b)) return false;
    const double rr = r * r;   // exact
    double q = rr * (1.0 / (b * b));
    q = div_step(rr, b * b, 1.0 / (b * b), q);
    q = div_step(rr, b * b, 1.0 / (b * b), q);
    const double u = 1.0 - q;
    const double x = div_step(r, b, 1.0 / b, r * (1.0 / b));
    const double v = 1.0 - x * x;
    w = (float)(u * u);
    loss = (float)(b * b / 6.0 * (1.0 - v * v * v));
    return true;
  }
  if (kind == 1) {
    if (!(ae > 0x1.5851eap+0f && ae < 1e30f)) return false;
    const double a = fabs(r), y0 = robust_rcp(ae);
    const double wd = 1.345 * fma(fma(-a, y0, 1.0), y0, y0);
    w = (float)wd;
    loss = (float)(1.345 * (a - 0.5 * 1.345));
    return rounds_alike(wd);
  }
  return false;
}

// kind: 0 none, 1 Huber (k 1.345), 2 Tukey (b 4.6851), 3 Cauchy (k 2.3849)
// (tracking.h:19-24, :343-345).
MF_ROBUST_HD void robust(float e, int kind, float& w, float& loss) {
  // Within the quadratic part the double loss is 0.5 e^2 exactly, rounded once:
  // 0.5f * (e * e), unless e * e leaves the normal range (the double path then).
  // 0x1.5851eap+0f is the largest float at most 1.345.
  if (kind <= 1) {
    const float q = e * e;
    if ((kind == 0 || fabsf(e) <= 0x1.5851eap+0f) && ((q >= 1e-30f && q <= 1e38f) || e == 0.f)) {
      w = 1.f;
      loss = 0.5f * q;
      return;
    }
  }
  if (robust_fast(e, kind, w, loss)) return;
  const double r = e;
  double wd = 1.0, l;
  switch (kind) {
    case 1: {
      const double a = fabs(r);
      if (a <= 1.345) { wd = 1.0; l = 0.5 * r * r; }
      else { wd = 1.345 / a; l = 1.345 * (a - 0.5 * 1.345); }
      break;
    }
    case 2: {
      const double b = 4.6851, a = fabs(r);
      if (a <= b) {
        const double u = 1.0 - r * r / (b * b);
        wd = u * u;
        const double v = 1.0 - (r / b) * (r / b);
        l = b * b / 6.0 * (1.0 - v * v * v);
      } else { wd = 0; l = b * b / 6.0; }
      break;
    }
    case 3: {
      const double q = (r / 2.3849) * (r / 2.3849);
      wd = 1 / (1 + q);
      l = 0.5 * 2.3849 * 2.3849 * log(1.0 + q);
      break;
    }
    default: l = 0.5 * r * r;
  }
  w = (float)wd;
  loss = (float)l;
}

}  // namespace mf

#undef MF_ROBUST_HD
#undef MF_ROBUST_TABLE
