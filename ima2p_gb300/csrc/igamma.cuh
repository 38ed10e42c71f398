// igamma.cuh -- the reference's incomplete gamma functions on the device
// (uppergamma, lowergamma, gser/gserlog, gcf/gcflog, expint(1, x) and
// LogDiff; utilities.cpp:808-1130, imamp.hpp:257-262), shared by the p(G)
// integrals (k_treeweight.cu, k_updgen.cu) and the 2NM densities
// (k_popmig.cu).  All FP64; log and exp are the device's.  The series takes
// one division for four terms and gcf's fraction runs on numerators and
// denominators, so their roundings are not the reference's one by one: both
// stop at its term, and the sums are within 5e-15 of the same sums in quad
// precision, as its own are (60,000 random (a, x) in each of ten ranges of a up
// to 12,000; the logarithms' errors are equal in mean and maximum).  The other
// expressions keep its order of operations (-fmad=false).
#pragma once

#include "internal.h"

namespace {

enum { IG_E_TERM = 4, IG_E_LF = 5 };  // a series or fraction that did not converge; a count past logfact

// The reference's incomplete gamma functions, restated from the published
// Numerical Recipes methods it uses (series, continued fraction, E1 series /
// continued fraction by Lentz's method) with its constants: EPS 3e-7, ITMAX 1000,
// FPMIN 1e-30, expint's MAXIT 100 and Euler constant 0.5772156649.
constexpr double IG_EPS = 3.0e-7, IG_FPMIN = 1.0e-30, EI_EULER = 0.5772156649;
constexpr int IG_ITMAX = 1000, EI_MAXIT = 100;
constexpr double LD_CUT = 7.0978271289338397e+02, MPRIORMIN = 0.000001;
constexpr double LOG2 = 0.69314718055994530941723212146;

// The series and the fraction follow one another term by term, each at the
// latency of FP64 operations (the pipe issues at 1/64 of the FP32 rate), and
// a division is a dozen of them.  So the series divides once for four terms
// and the fraction not at all: it runs on numerators and denominators,
// h = A / B, and compares successive convergents crosswise.  Both stop at the
// term where the reference does.  (In float-float from a = 32 on, 2^-46, a
// genealogy update of 50 HKY loci x 32 chains took 1.24 ms where it takes 1.69,
// 128 chains' split times 0.85 and 0.96; but the logarithm was then off by
// 1.5e-14 on average and 4e-13 at most at a = 32 to 40, against 6e-15 and 3e-14.)
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
