// igamma.cuh -- the reference's incomplete gamma functions on the device
// (uppergamma, lowergamma, gser/gserlog, gcf/gcflog, expint(1, x) and
// LogDiff; utilities.cpp:808-1130, imamp.hpp:257-262), shared by the p(G)
// integrals (k_treeweight.cu) and the 2NM densities (k_popmig.cu).  Both
// files are compiled with -fmad=false so that these add and multiply in the
// reference's order; log and exp are the device's.
#pragma once

#include "ff.cuh"
#include "internal.h"

namespace {

enum { IG_E_TERM = 4, IG_E_LF = 5 };  // a series or fraction that did not converge; a count past logfact

// The reference's incomplete gamma functions, restated from the published
// Numerical Recipes methods it uses (series, Lentz continued fraction, E1
// series / continued fraction) with its constants: EPS 3e-7, ITMAX 1000,
// FPMIN 1e-30, expint's MAXIT 100 and Euler constant 0.5772156649.
constexpr double IG_EPS = 3.0e-7, IG_FPMIN = 1.0e-30, EI_EULER = 0.5772156649;
constexpr int IG_ITMAX = 1000, EI_MAXIT = 100;
constexpr double LD_CUT = 7.0978271289338397e+02, MPRIORMIN = 0.000001;
constexpr double LOG2 = 0.69314718055994530941723212146;

// From IGF_AMIN on the series and the fraction run on the FP32 pipe in
// float-float (2^-46; FP64's exponent a ln x - x - gln, by which they are
// multiplied or to whose logarithm they are added, is off by more from a = 32
// on): its operations take a tenth of the time, and there are 64 of them for
// one of FP64.  One pass each, the sum or the convergents growing until the
// reference's rule stops them, which FP32 decides unless the ratio lies
// within IGF_TOL of EPS; that bounds what IGF_NMAX steps of a few roundings
// each can be off.  A stop that cannot be told is left to the FP64 loops.
constexpr int IGF_AMIN = 32, IGF_NMAX = 512;
constexpr float IGF_EPS = 3.0e-7f, IGF_TOL = 2e-4f, IGF_XMAX = 1e6f;

__device__ __forceinline__ ff igf_rcp(float a)  // 1 / a, 1 <= a < 2^24
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  r = __fmaf_rn(r, __fmaf_rn(-a, r, 1.f), r);
  return ff_make(r, __fmul_rn(__fmaf_rn(-a, r, 1.f), r));
}

// the sum of gser's series over its first term 1 / a: false where the number
// of terms cannot be told
__device__ __forceinline__ bool igf_series(float a, double x, double *s)
{
  const ff xf = ff_split(x);
  if (!(xf.hi < IGF_XMAX)) return false;
  float ap = a, sum = 1.f, rest = 0.f;
  ff del = ff_from(1.f);
  for (int n = 0; n < IGF_NMAX; n++) {
    ap = __fadd_rn(ap, 1.f);
    const ff r = igf_rcp(ap);
    const float q = __fmul_rn(xf.hi, r.hi);
    const float qe = __fmaf_rn(xf.hi, r.lo, __fmaf_rn(xf.lo, r.hi, __fmaf_rn(xf.hi, r.hi, -q)));
    const float p = __fmul_rn(del.hi, q);
    del.lo = __fmaf_rn(del.hi, qe, __fmaf_rn(del.lo, q, __fmaf_rn(del.hi, q, -p)));
    del.hi = p;
    const ff t = two_sum(sum, p);
    sum = t.hi;
    rest = __fadd_rn(rest, __fadd_rn(t.lo, del.lo));
    const float stop = __fmul_rn(sum, IGF_EPS);
    if (p < stop * (1.f + IGF_TOL)) {
      *s = (double)sum + (double)rest;
      return p < stop * (1.f - IGF_TOL);
    }
  }
  return false;
}

// gcf's fraction, A / B of the convergents A_n = b_n A_(n-1) + a_n A_(n-2) (B
// alike) in units that keep B near 1; b0 = x + 1 - a.  Convergents n and n - 1
// differ by D / (B B'), D the product of the -a_i.
__device__ __forceinline__ bool igf_fraction(float a, double b0, double *h)
{
  const ff bf = ff_split(b0);
  if (!(bf.hi < IGF_XMAX) || !(bf.hi >= 1.f)) return false;
  ff A = ff_from(1.f), Ap = ff_from(0.f), B = bf, Bp = ff_from(1.f);
  float D = 1.f;
  for (int n = 1; n <= IGF_NMAX; n++) {
    const float fn = (float)n;
    ff b = two_sum(bf.hi, __fadd_rn(fn, fn));
    b.lo = __fadd_rn(b.lo, bf.lo);
    const ff an = two_prod(fn, __fsub_rn(a, fn));
    auto next = [&](ff c, ff cp) {
      const float u = __fmul_rn(b.hi, c.hi), v = __fmul_rn(an.hi, cp.hi);
      const float ue = __fmaf_rn(b.hi, c.lo, __fmaf_rn(b.lo, c.hi, __fmaf_rn(b.hi, c.hi, -u)));
      const float ve = __fmaf_rn(an.hi, cp.lo, __fmaf_rn(an.lo, cp.hi, __fmaf_rn(an.hi, cp.hi, -v)));
      const ff t = two_sum(u, v);
      return ff_make(t.hi, __fadd_rn(t.lo, __fadd_rn(ue, ve)));
    };
    const ff An = next(A, Ap), Bn = next(B, Bp);
    D = __fmul_rn(D, an.hi);
    // |h / h_before - 1| = |D| / |A_before B|
    const float stop = fabsf(__fmul_rn(A.hi, Bn.hi)) * IGF_EPS;
    Ap = A;
    Bp = B;
    A = An;
    B = Bn;
    if (fabsf(D) < stop * (1.f + IGF_TOL)) {
      const ff r = ff_div(fast_two_sum(A.hi, A.lo), fast_two_sum(B.hi, B.lo));
      *h = (double)r.hi + (double)r.lo;
      return fabsf(D) < stop * (1.f - IGF_TOL);
    }
    if (fabsf(B.hi) > 1e6f) {  // by 1 / B's power of two
      const float q = __int_as_float((254 - ((__float_as_int(B.hi) >> 23) & 0xff)) << 23);
      auto scale = [&](ff &v) { v = ff_make(__fmul_rn(v.hi, q), __fmul_rn(v.lo, q)); };
      scale(A);
      scale(Ap);
      scale(B);
      scale(Bp);
      D = __fmul_rn(D, __fmul_rn(q, q));
    }
  }
  return false;
}

// The series and the fraction follow one another term by term, each at the
// latency of FP64 operations (the pipe issues at 1/64 of the FP32 rate), and
// a division is a dozen of them.  So the series divides once for four terms
// and the fraction not at all: it runs on numerators and denominators,
// h = A / B, and compares successive convergents crosswise.  Both stop at the
// term where the reference does.
struct IgBase {
  const double *lft;
  int st;
  __device__ double lf(int i)
  {
    if (i < 0 || i >= TW_LF_N) {
      st = IG_E_LF;
      return 0.0;
    }
    return lft[i];
  }
  __device__ double gser(int a, double x, double *gln, bool lg)
  {
    *gln = lf(a - 1);
    if (x <= 0.0) {
      if (x < 0.0) st = IG_E_TERM;
      return 0.0;
    }
    double sf;
    if (a >= IGF_AMIN && igf_series((float)a, x, &sf)) {
      sf /= a;
      return lg ? log(sf) + (-x + a * log(x) - (*gln)) : sf * exp(-x + a * log(x) - (*gln));
    }
    double ap = a, del = 1.0 / a, sum = del;
    static_assert(IG_ITMAX % 4 == 0, "four terms at a time");
    for (int n = 0; n < IG_ITMAX; n += 4) {
      const double q1 = ap + 1.0, q2 = ap + 2.0, q3 = ap + 3.0, q4 = ap + 4.0;
      const double p12 = q1 * q2, p34 = q3 * q4, r = x / (p12 * p34);
      const double r12 = r * p34, r34 = r * p12;  // x / p12, x / p34
      const double t[4] = {r12 * q2, r12 * q1, r34 * q4, r34 * q3};  // x / q1 .. x / q4
      ap = q4;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        del *= t[j];
        sum += del;
        if (fabs(del) < fabs(sum) * IG_EPS)
          return lg ? log(sum) + (-x + a * log(x) - (*gln)) : sum * exp(-x + a * log(x) - (*gln));
      }
    }
    st = IG_E_TERM;
    return 0.0;
  }
  __device__ double gcf(double a, double x, double *gln, bool lg)
  {
    *gln = lf((int)a - 1);
    double hf;
    if (a >= IGF_AMIN && igf_fraction((float)a, x + 1.0 - a, &hf))
      return lg ? (-x + a * log(x) - (*gln)) + log(hf) : exp(-x + a * log(x) - (*gln)) * hf;
    // convergents: A / B of this term and of the one before
    double b = x + 1.0 - a, A = 1.0, Am = 0.0, B = b, Bm = 1.0;
    int i;
    for (i = 1; i <= IG_ITMAX; i++) {
      const double an = -i * (i - a);
      b += 2.0;
      const double An = b * A + an * Am, Bn = b * B + an * Bm;
      Am = A;
      Bm = B;
      A = An;
      B = Bn;
      // |h / h_before - 1| < EPS
      const double m = Am * B;
      if (fabs(A * Bm - m) < IG_EPS * fabs(m)) break;
      const int e = (__double2hiint(B) >> 20) & 0x7ff;
      if (e > 1023 + 256) {  // back to the middle of the range
        const double q = __hiloint2double((2046 - e) << 20, 0);
        A *= q;
        Am *= q;
        B *= q;
        Bm *= q;
      }
    }
    if (i > IG_ITMAX) st = IG_E_TERM;
    const double h = A / B;
    return lg ? (-x + a * log(x) - (*gln)) + log(h) : exp(-x + a * log(x) - (*gln)) * h;
  }
  __device__ double expint1(double x, bool *islog)
  {
    *islog = false;
    if (x <= 0.0) {
      st = IG_E_TERM;
      return 0.0;
    }
    if (x > 1.0) {
      double b = x + 1, c = 1.0 / IG_FPMIN, d = 1.0 / b, h = d;
      for (int i = 1; i <= EI_MAXIT; i++) {
        const double an = -i * i;
        b += 2.0;
        d = 1.0 / (an * d + b);
        c = b + an / c;
        const double del = c * d;
        h *= del;
        if (fabs(del - 1.0) < IG_EPS) {
          *islog = true;
          return log(h) - x;
        }
      }
      st = IG_E_TERM;
      return 0.0;
    }
    double ans = -log(x) - EI_EULER, fact = 1.0;
    for (int i = 1; i <= EI_MAXIT; i++) {
      fact *= -x / i;
      const double del = -fact / i;
      ans += del;
      if (fabs(del) < fabs(ans) * IG_EPS) return ans;
    }
    st = IG_E_TERM;
    return ans;
  }
  // Whether the smaller of gamma(a, x) / Gamma(a) and Gamma(a, x) / Gamma(a),
  // e^(a ln x - x - gln) times a series below 1,000 / a (x < a + 1) or a
  // fraction below 1/2, leaves gln + ln(1 - it) at gln: below 2^-60, or where
  // gln >= 64, whose last bit is 2^-46, below 2^-49 (a > 30).  In FP32, whose
  // error is below 1e-6 of the terms: 0.2 up to NEGL_MAX.
  static constexpr float NEGL_MAX = 2.0e5f;
  __device__ bool negligible(int a, float x, double gln)
  {
    const float g = (float)gln, l = (float)a * logf(x);
    return l - x - g < (g > 64.f ? -38.0f : -54.0f) && fabsf(l) < NEGL_MAX && x < NEGL_MAX && g < NEGL_MAX;
  }
  __device__ double upper(int a, double x)  // uppergamma: log Gamma(a, x)
  {
    double p, gln;
    if (x < 0.0 || a < 0) {
      st = IG_E_TERM;
      return 0.0;
    }
    if (a == 0) {
      bool islog;
      const double t = expint1(x, &islog);
      p = islog ? t : log(t);
    } else if (x < (a + 1.0)) {
      gln = lf(a - 1);
      if (negligible(a, (float)x, gln)) return gln;
      const double gs = gser(a, x, &gln, false);
      p = gln + log(1.0 - gs);
    } else {
      p = gln_plus_gcf(a, x, true);
    }
    return p < -1e200 ? -1e200 : p;
  }
  __device__ double gln_plus_gcf(int a, double x, bool lg)
  {
    double gln;
    const double v = gcf((double)a, x, &gln, lg);
    return lg ? gln + v : gln + log(1 - v);
  }
  __device__ double lower(int a, double x)  // lowergamma: log gamma(a, x)
  {
    double p, gln;
    if (x < 0.0 || a <= 0) {
      st = IG_E_TERM;
      return 0.0;
    }
    if (x < (a + 1.0)) {
      const double gs = gser(a, x, &gln, true);
      p = gln + gs;
    } else if (negligible(a, (float)x, lf(a - 1))) {
      return lf(a - 1);
    } else {
      p = gln_plus_gcf(a, x, false);
    }
    return p < -1e200 ? -1e200 : p;
  }
  __device__ double logdiff(double a, double b)  // LogDiff, imamp.hpp:257-262
  {
    if (a <= b) {
      st = IG_E_TERM;
      return 0.0;
    }
    return (a - b < LD_CUT) ? b + log(exp(a - b) - 1.0) : a;
  }
};

// The integral terms of initialize_integrate_tree_prob
// (update_gtree_common.cpp:108-304, MORESTABLE) on the functions above.
struct Ig : IgBase {
  __device__ double coal(int cc, double fc, double hcc, double max, double min)
  {
    double p;
    if (cc > 0) {
      if (!(fc > 0)) {
        st = IG_E_TERM;
        return 0.0;
      }
      if (min == 0) {
        double ug, fullg = cc > 1 ? lf(cc - 2) : 0.0;
        const float xf = 2.0f * (float)fc / (float)max;
        // Far below the maximum Gamma(a, x) is Gamma(a).  (x < a + 1 whatever
        // xf's rounding.)  And where ug is fullg, the other form's ugalt
        // differs from it by rounding alone: its terms are below fullg + cc +
        // 800 (or logdiff returns fullg), each rounded to 1.1e-16 of itself, a
        // handful of roundings -- far less than 1e-10 for a sum up to 9e4.
        if (cc > 2 && xf < (float)(cc - 1) && fullg + cc < 9e4 && negligible(cc - 1, xf, fullg)) {
          ug = fullg;
        } else {
          ug = upper(cc - 1, 2 * fc / max);
          if (cc > 1 && ((fullg - ug < 1e-15 && !(ug == fullg && fullg + cc < 9e4)) || fullg - ug > LD_CUT)) {
            const double lg = lower(cc - 1, 2 * fc / max);
            if (fullg > lg) {
              const double ugalt = logdiff(fullg, lg);
              if (fabs(ugalt - ug) > 1e-10) ug = ugalt;
            }
          }
        }
        p = ug + LOG2 - hcc + (1 - cc) * log(fc);
      } else {
        const double aa = upper(cc - 1, 2 * fc / max), bb = upper(cc - 1, 2 * fc / min);
        p = logdiff(aa, bb);
        p += (LOG2 - hcc + (1 - cc) * log(fc));
      }
    } else if (2 * fc / max > 0) {
      if (min == 0) {
        const double aa = log(max) - 2.0 * fc / max;
        const double bb = LOG2 + log(fc) + upper(0, 2.0 * fc / max);
        p = logdiff(aa, bb);
      } else {
        double aa = upper(0, 2 * fc / max), bb = upper(0, 2 * fc / min);
        double c = logdiff(aa, bb);
        c += LOG2 + log(fc);
        aa = log(max) - 2.0 * fc / max;
        bb = log(min) - 2.0 * fc / min;
        const double d = logdiff(aa, bb);
        p = logdiff(d, c);
      }
    } else {
      p = log(max - min);
    }
    return p;
  }
  __device__ double mig(int cm, double fm, double max, double min)
  {
    double p;
    if (cm > 0) {
      if (!(fm > 0)) {
        st = IG_E_TERM;
        return 0.0;
      }
      if (min == 0) {
        double lg = lower(cm + 1, fm * max);
        const double fullg = lf(cm);
        if (fullg - lg < 1e-15 || fullg - lg > LD_CUT) {
          const double ug = upper(cm + 1, fm * max);
          if (fullg > ug) {
            const double lgalt = logdiff(fullg, ug);
            if (fabs(lgalt - lg) > 1e-12) lg = lgalt;
          }
        }
        p = (-1 - cm) * log(fm) + lg;
      } else {
        const double aa = upper(cm + 1, fm * min), bb = upper(cm + 1, fm * max);
        p = (-1 - cm) * log(fm) + logdiff(aa, bb);
      }
    } else if (fm > MPRIORMIN) {
      if (min == 0) {
        p = (max == MPRIORMIN) ? 0 : logdiff(0.0, -fm * max) - log(fm);
      } else {
        p = logdiff(-fm * min, -fm * max) - log(fm);
      }
    } else {
      p = log(max - min);
    }
    return p;
  }
  __device__ double mig_expo(int cm, double fm, double mean)
  {
    return -log(mean) + (-(cm + 1) * log(fm + 1.0 / mean)) + lf(cm);
  }
};

}  // namespace
