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
    {1.0, 0.0}, {0.9846153846153847, 0.015504186535965199},
    {0.9696969696969697, 0.03077165866675366}, {0.9552238805970149, 0.04580953603129422},
    {0.9411764705882353, 0.060624621816434854}, {0.927536231884058, 0.07522342123758752},
    {0.9142857142857143, 0.08961215868968717}, {0.9014084507042254, 0.10379679368164355},
    {0.8888888888888888, 0.11778303565638351}, {0.8767123287671232, 0.13157635778871932},
    {0.8648648648648649, 0.14518200984449783}, {0.8533333333333334, 0.15860503017663852},
    {0.8421052631578947, 0.17185025692665928}, {0.8311688311688312, 0.18492233849401193},
    {0.8205128205128205, 0.19782574332991992}, {0.810126582278481, 0.21056476910734964},
    {0.8, 0.2231435513142097}, {0.7901234567901234, 0.23556607131276697},
    {0.7804878048780488, 0.2478361639045812}, {0.7710843373493976, 0.259957524436926},
    {0.7619047619047619, 0.2719337154836418}, {0.7529411764705882, 0.2837681731306446},
    {0.7441860465116279, 0.2954642128938359}, {0.735632183908046, 0.3070250352949119},
    {0.7272727272727273, 0.3184537311185346}, {0.7191011235955056, 0.32975328637246804},
    {0.7111111111111111, 0.3409265869705932}, {0.7032967032967034, 0.3519764231571781},
    {0.6956521739130435, 0.3629054936893685}, {0.6881720430107527, 0.373716409793584},
    {0.6808510638297872, 0.38441169891033206}, {0.6736842105263158, 0.394993808240869},
    {0.6666666666666666, 0.40546510810816444}, {0.6597938144329897, 0.415827895143711},
    {0.6530612244897959, 0.42608439531090014}, {0.6464646464646465, 0.43623676677491796},
    {0.64, 0.4462871026284195}, {0.6336633663366337, 0.4562374334815876},
    {0.6274509803921569, 0.46608972992459924}, {0.6213592233009708, 0.475845904869964},
    {0.6153846153846154, 0.48550781578170077}, {0.6095238095238096, 0.4950772667978514},
    {0.6037735849056604, 0.5045560107523953}, {0.5981308411214953, 0.5139457511022344},
    {0.5925925925925926, 0.5232481437645479}, {0.5871559633027523, 0.5324647988694717},
    {0.5818181818181818, 0.5415972824327444}, {0.5765765765765766, 0.5506471179526623},
    {0.5714285714285714, 0.5596157879354228}, {0.5663716814159292, 0.5685047353526688},
    {0.5614035087719298, 0.5773153650348236}, {0.5565217391304348, 0.5860490450035782},
    {0.5517241379310345, 0.5947071077466928}, {0.5470085470085471, 0.6032908514380841},
    {0.5423728813559322, 0.6118015411059929}, {0.5378151260504201, 0.6202404097518576},
    {0.5333333333333333, 0.6286086594223742}, {0.5289256198347108, 0.6369074622370692},
    {0.5245901639344263, 0.6451379613735847}, {0.5203252032520326, 0.6533012720127456},
    {0.5161290322580645, 0.661398482245365}, {0.512, 0.6694306539426292},
    {0.5079365079365079, 0.6773988235918061}, {0.5039370078740157, 0.6853040030989195},
    {0.5, 0.6931471805599453},
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
  return fma((double)((hi >> 20) - 1023), 0.6931471805599453, t) + p;
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
    if (!(ae > 1.34499991f && ae < 1e30f)) return false;
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
  // 1.34499991f is the largest float at most 1.345.
  if (kind <= 1) {
    const float q = e * e;
    if ((kind == 0 || fabsf(e) <= 1.34499991f) && ((q >= 1e-30f && q <= 1e38f) || e == 0.f)) {
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
