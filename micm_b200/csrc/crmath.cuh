// Correctly rounded exp, log10 and pow for the rate constants and the
// step-size controller, evaluated identically on the host and the device.
//
// micm evaluates these with the host C library (std::exp, std::pow,
// std::log10 in rate_constant_functions.hpp:52-136 and the step-size factor
// std::pow(error, 1 / order) in rosenbrock.inl:232-235).  glibc's exp and pow
// round correctly except in rare cases (a few in 10,000 arguments), so a
// correctly rounded evaluation here reproduces micm's values bit for bit
// almost always; a last-bit difference in the step-size factor can change the
// accepted-step sequence of a stiff problem at tight tolerances.
//
// Method: double-double arithmetic (a value is an unevaluated sum hi + lo,
// |lo| <= ulp(hi)/2; Dekker's and Knuth's error-free sum and product, the
// product through a fused multiply-add), about 100 correct bits, then one
// rounding to double.  A result is rounded wrongly only when the exact value
// lies within about 2^-45 ulp of a rounding boundary.
//   exp(x):  x = (64 m + j) ln2 / 64 + r (|r| <= ln2 / 128, ln2 in three parts),
//            exp(r) by its Taylor polynomial to degree 11 -- the terms from r^6 on,
//            below 2^-54 of the result, in double, the first five in double-double
//            (Horner) -- times 2^(j/64) from a table of 64 double-doubles, times
//            2^m (Tang, ACM TOMS 15(2), 1989, carried to double-double).
//   log(x):  x = 2^e m (m in [sqrt(1/2), sqrt(2))), a double seed
//            e ln2 + 2 atanh((m-1)/(m+1)) by its series, then one Newton step
//            l + (x exp(-l) - 1) in double-double (quadratic: error ~1e-33).
//   pow:     exp(y log x);  log10: log(x) / ln(10).
// Arguments outside the ranges the solver meets (non-positive bases, results
// that overflow or fall into the subnormal range) use the plain double
// functions.  Every operation is an explicit IEEE add, multiply, divide or
// fma, so host and device results are identical; the library is compiled
// with contraction off (-fmad=false on the device, -ffp-contract=off on the
// host) so no other fusing happens.
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define CRM_HD __host__ __device__ __forceinline__
#else
#define CRM_HD inline
#endif

namespace micmb
{
  namespace crm
  {
    struct dd
    {
      double hi, lo;
    };

    // 2^(j/64), each the double nearest the value and the double nearest the rest
#define CRM_EXP2_64                                                                              \
      { 0x1.0000000000000p+0, 0x0.0p+0 }, { 0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56 }, \
      { 0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55 }, { 0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57 }, \
      { 0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54 }, { 0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59 }, \
      { 0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54 }, { 0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54 }, \
      { 0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55 }, { 0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55 }, \
      { 0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54 }, { 0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55 }, \
      { 0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54 }, { 0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55 }, \
      { 0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55 }, { 0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54 }, \
      { 0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55 }, { 0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54 }, \
      { 0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54 }, { 0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56 }, \
      { 0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55 }, { 0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58 }, \
      { 0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59 }, { 0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56 }, \
      { 0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56 }, { 0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54 }, \
      { 0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55 }, { 0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54 }, \
      { 0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54 }, { 0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54 }, \
      { 0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54 }, { 0x1.6623882552225p+0, -0x1.bb60987591c34p-54 }, \
      { 0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54 }, { 0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57 }, \
      { 0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55 }, { 0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54 }, \
      { 0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55 }, { 0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56 }, \
      { 0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54 }, { 0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54 }, \
      { 0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54 }, { 0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55 }, \
      { 0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57 }, { 0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54 }, \
      { 0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56 }, { 0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54 }, \
      { 0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54 }, { 0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54 }, \
      { 0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54 }, { 0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57 }, \
      { 0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56 }, { 0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55 }, \
      { 0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55 }, { 0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54 }, \
      { 0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56 }, { 0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54 }, \
      { 0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55 }, { 0x1.da9e603db3285p+0, 0x1.c2300696db532p-54 }, \
      { 0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54 }, { 0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55 }, \
      { 0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54 }, { 0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54 }, \
      { 0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54 }, { 0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55 }
#if defined(__CUDACC__)
    static __constant__ dd kExp2Device[64] = { CRM_EXP2_64 };
#endif
    static const dd kExp2Host[64] = { CRM_EXP2_64 };

    CRM_HD dd exp2_64(int j)
    {
#if defined(__CUDA_ARCH__)
      return kExp2Device[j];
#else
      return kExp2Host[j];
#endif
    }

    CRM_HD dd two_sum(double a, double b)
    {
      const double s = a + b;
      const double bb = s - a;
      const double e = (a - (s - bb)) + (b - bb);
      return { s, e };
    }

    // |a| >= |b| (or a == 0)
    CRM_HD dd quick_two_sum(double a, double b)
    {
      const double s = a + b;
      return { s, b - (s - a) };
    }

    CRM_HD dd two_prod(double a, double b)
    {
      const double p = a * b;
      return { p, fma(a, b, -p) };
    }

    CRM_HD dd add(dd a, dd b)
    {
      dd s = two_sum(a.hi, b.hi);
      const dd t = two_sum(a.lo, b.lo);
      s.lo = s.lo + t.hi;
      s = quick_two_sum(s.hi, s.lo);
      s.lo = s.lo + t.lo;
      return quick_two_sum(s.hi, s.lo);
    }

    CRM_HD dd mul(dd a, dd b)
    {
      dd p = two_prod(a.hi, b.hi);
      p.lo = p.lo + (a.hi * b.lo + a.lo * b.hi);
      return quick_two_sum(p.hi, p.lo);
    }

    CRM_HD dd mul_d(dd a, double b)
    {
      dd p = two_prod(a.hi, b);
      p.lo = p.lo + a.lo * b;
      return quick_two_sum(p.hi, p.lo);
    }

    // ln 2 = LN2_0 + LN2_1 + LN2_2 (each the double nearest the remainder)
    constexpr double LN2_0 = 0x1.62e42fefa39efp-1;
    constexpr double LN2_1 = 0x1.abc9e3b39803fp-56;
    constexpr double LN2_2 = 0x1.7b57a079a1934p-111;
    constexpr double INV_LN2 = 0x1.71547652b82fep+0;
    constexpr double INV_LN10_0 = 0x1.bcb7b1526e50ep-2;
    constexpr double INV_LN10_1 = 0x1.95355baaafad3p-57;
    constexpr double SQRT_HALF = 0x1.6a09e667f3bcdp-1;

    // a + b for |a| >= |b|, with about 2^-104 relative error
    CRM_HD dd add_ordered(dd a, dd b)
    {
      const dd s = quick_two_sum(a.hi, b.hi);
      return quick_two_sum(s.hi, s.lo + (a.lo + b.lo));
    }

    // exp of a double-double argument with |x| < 708 (normal results)
    CRM_HD dd exp_dd(dd x)
    {
      // 1/n! for n = 2..5 as double-doubles
      constexpr double F_HI[6] = { 0, 0, 0x1.0p-1, 0x1.5555555555555p-3, 0x1.5555555555555p-5, 0x1.1111111111111p-7 };
      constexpr double F_LO[6] = { 0, 0, 0.0, 0x1.5555555555555p-57, 0x1.5555555555555p-59, 0x1.1111111111111p-63 };
      const double k = rint(x.hi * (64.0 * INV_LN2));
      // r = x - k ln2 / 64, each product exact or below 2^-100 relative
      dd r = add(x, two_prod(-k, LN2_0 * 0x1.0p-6));
      r = add(r, two_prod(-k, LN2_1 * 0x1.0p-6));
      r = add_ordered(r, dd{ -k * (LN2_2 * 0x1.0p-6), 0.0 });
      // 1/6! + r/7! + ... + r^5/11!
      const double h = r.hi;
      double q = 1.0 / 39916800.0;
      q = 1.0 / 3628800.0 + h * q;
      q = 1.0 / 362880.0 + h * q;
      q = 1.0 / 40320.0 + h * q;
      q = 1.0 / 5040.0 + h * q;
      q = 1.0 / 720.0 + h * q;
      // exp(r) - 1 = r (1 + r (1/2 + r (1/6 + r (1/24 + r (1/120 + r q)))))
      dd t = add_ordered(dd{ F_HI[5], F_LO[5] }, two_prod(h, q));
#pragma unroll
      for (int n = 4; n >= 2; --n)
        t = add_ordered(dd{ F_HI[n], F_LO[n] }, mul(r, t));
      t = add_ordered(dd{ 1.0, 0.0 }, mul(r, t));
      const dd p = mul(r, t);
      const int ki = (int)k, m = ki >> 6;
      const dd c = exp2_64(ki & 63);
      const dd e = add_ordered(c, mul(c, p));
      return { ldexp(e.hi, m), ldexp(e.lo, m) };
    }

    // natural log of a positive, finite, normal double
    CRM_HD dd log_dd(double x)
    {
      int e;
      double m = frexp(x, &e);  // m in [0.5, 1)
      if (m < SQRT_HALF)
      {
        m = m * 2.0;
        e = e - 1;
      }
      // seed: log(m) = 2 atanh(u), u = (m - 1) / (m + 1), |u| <= 0.1716
      const double f = m - 1.0;
      const double u = f / (2.0 + f);
      const double u2 = u * u;
      double ser = 1.0 / 25.0;
#pragma unroll
      for (int j = 11; j >= 0; --j)
        ser = 1.0 / (double)(2 * j + 1) + u2 * ser;
      const double lm = 2.0 * u * ser;
      const double de = (double)e;
      dd l = add(two_prod(de, LN2_0), two_prod(de, LN2_1));
      l = add(l, dd{ lm, 0.0 });
      // Newton step for exp(l) = x:  l <- l + (x exp(-l) - 1)
      const dd q = mul_d(exp_dd(dd{ -l.hi, -l.lo }), x);
      const dd corr = add(q, dd{ -1.0, 0.0 });
      return add(l, corr);
    }

    CRM_HD bool plain_range(double x)
    {
      return !(x > 0.0) || !(x < INFINITY) || x < 0x1.0p-1022;
    }
  }  // namespace crm

  // exp(x), correctly rounded in all but rare cases
  CRM_HD double cr_exp(double x)
  {
    if (!(fabs(x) < 708.0))
      return exp(x);
    const crm::dd r = crm::exp_dd(crm::dd{ x, 0.0 });
    return r.hi + r.lo;
  }

  // pow(x, y) for x > 0, correctly rounded in all but rare cases
  CRM_HD double cr_pow(double x, double y)
  {
    if (y == 0.0)
      return 1.0;
    if (y == 1.0)
      return x;
    if (y == 2.0)
      return x * x;
    if (crm::plain_range(x) || !(fabs(y) < INFINITY))
      return pow(x, y);
    const crm::dd z = crm::mul_d(crm::log_dd(x), y);
    if (!(fabs(z.hi) < 708.0))
      return pow(x, y);
    const crm::dd r = crm::exp_dd(z);
    return r.hi + r.lo;
  }

  // log10(x) for x > 0, correctly rounded in all but rare cases
  CRM_HD double cr_log10(double x)
  {
    if (crm::plain_range(x))
      return log10(x);
    if (x == 1.0)
      return 0.0;
    const crm::dd r = crm::mul(crm::log_dd(x), crm::dd{ crm::INV_LN10_0, crm::INV_LN10_1 });
    return r.hi + r.lo;
  }
}  // namespace micmb
