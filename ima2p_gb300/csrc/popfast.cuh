// popfast.cuh -- calc_popmig's general term (popmig.cpp:60-84) without FP64
// logarithms, exponentials and divisions.  With a = cc + mc, z = fc + fm x,
// x1 = 2 z / qmax and x2 = mmax z / x the reference adds, per genealogy,
//   2 x^mc z^-a e^-(hc + q + m) (Gamma(a, x1) - Gamma(a, x2)),
// each Gamma(a, .) from its series (x < a + 1) or its continued fraction, cut
// at EPS, in logarithms.  Here the same truncated sums are multiplied out:
//   series:    Gamma(a, x) = Gamma(a) - x^a e^-x S(x)
//   fraction:  Gamma(a, x) = x^a e^-x H(x)
// and z^-a x1^a = (2 / qmax)^a, so that every factor is 2^(linear form of the
// genealogy's values), formed in fixed point (fxexp.cuh); only Gamma(a) z^-a
// needs a logarithm.  S and H are float-float, with the number of terms found
// beforehand in FP32: the reference's stopping rule is decided there unless
// the ratio lies within STOP_TOL of EPS.
//
// Terms the form does not cover (no events, a stop too near EPS, x1 >= x2, a
// difference below DIFF_MIN of its parts, exponents or counts out of range)
// are left to the caller's FP64 form.
#pragma once
#include "ff.cuh"
#include "fxexp.cuh"

namespace {

constexpr float PF_EPS = 3.0e-7f, PF_STOP_TOL = 2e-5f;
constexpr int PF_NMAX = 48;    // longest series or fraction taken here
constexpr int PF_AMAX = 192;   // counts below this
constexpr int PF_RCP = PF_AMAX + PF_NMAX;  // reciprocals 1 / k, k < PF_RCP
constexpr double PF_LOG2E = 1.4426950408889634074;

// log2 of a normal positive double: integer part, and fraction in units of
// 2^-64 within 2^-60.  1 + j/512 <= m < 1 + (j+1)/512: u = m R_j - 1 >= 0 with
// R_j = 2^-32 ceil(2^32 512 / (512 + j)), then -log2 R_j + log2(1 + u).
struct FxLogTab {
  uint32_t r[FX_TAB];   // R_j 2^32 - 1 (R_0 = 1)
  uint64_t l[FX_TAB];   // -log2(R_j) 2^64, R_j = (r + 1) 2^-32
};
constexpr uint64_t FX_P0 = 0xb8aa3b295c17f041ull;  // 2^63
constexpr uint64_t FX_P1 = 0xb8aa3b295bb827ull;    // 2^64
constexpr uint32_t FX_P2 = 0x7b1c276bu;            // 2^48
constexpr uint32_t FX_P3 = 0x5c54fcu;              // 2^48
constexpr uint32_t FX_P4 = 0x4991u;                // 2^48

__device__ __forceinline__ uint64_t fx_log2(double z, const FxLogTab &T, int *e)
{
  const uint64_t b = fx_bits(z);
  *e = (int)(b >> 52) - 1023;
  const int j = (int)(b >> 43) & (FX_TAB - 1);
  const uint64_t m = (b << 11) | (1ull << 63);  // 2^63
  const uint64_t u = fx_mul64(m, T.r[j]) + (m >> 32) - (1ull << 63);  // 2^63, below 2^-9 (1 + 2^-22)
  const uint64_t rho = u << 9;  // 2^8 u, 2^64
  const uint32_t r = (uint32_t)(rho >> 32), rl = (uint32_t)rho;
  const uint32_t g3 = FX_P2 - fx_mulhi(r, FX_P3 - fx_mulhi(r, FX_P4));
  const uint64_t g2 = FX_P1 - ((uint64_t)fx_mulhi(r, g3) << 16);
  const uint64_t g1 = FX_P0 - ((fx_mul64(g2, r) + fx_mulhi((uint32_t)(g2 >> 32), rl)) >> 1);
  const uint64_t y = fx_mul64(g1, r) + fx_mulhi((uint32_t)(g1 >> 32), rl);  // 2^63
  return T.l[j] + (y >> 7);
}

__device__ __forceinline__ float pf_rcp(float a)
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}

// The number of terms of gser (utilities.cpp: del < sum EPS), 0 when too
// long or too near to tell.
__device__ __forceinline__ int pf_series_terms(float a, float x)
{
  float ap = a, del = 1.f, sum = 1.f;
  for (int n = 1; n <= PF_NMAX; n++) {
    ap += 1.f;
    del *= x * pf_rcp(ap);
    sum += del;
    const float t = sum * PF_EPS;
    if (del < t * (1.f + PF_STOP_TOL)) return del < t * (1.f - PF_STOP_TOL) ? n : 0;
  }
  return 0;
}

// The same for gcf's modified Lentz fraction: |h_n / h_(n-1) - 1| < EPS, from
// the differences of its convergents (Steed), which do not cancel.
__device__ __forceinline__ int pf_fraction_terms(float a, float b0)
{
  float b = b0, d = pf_rcp(b), h = d, del = d;
  for (int n = 1; n <= PF_NMAX; n++) {
    const float an = (float)n * (a - (float)n);
    b += 2.f;
    const float dn = pf_rcp(fmaf(an, d, b));
    del *= -an * (d * dn);
    const float t = fabsf(h) * PF_EPS;
    if (fabsf(del) < t * (1.f + PF_STOP_TOL)) return fabsf(del) < t * (1.f - PF_STOP_TOL) ? n : 0;
    h += del;
    d = dn;
  }
  return 0;
}

// One step of the series by Horner's rule: t <- 1 + t x / k
__device__ __forceinline__ ff pf_series_step(ff t, ff x, float2 rk)
{
  // t x and x / k unnormalised: the TwoSum with 1 is exact whatever their lo
  const float q = __fmul_rn(x.hi, rk.x);
  const float qe = __fmaf_rn(x.hi, rk.y, __fmaf_rn(x.lo, rk.x, __fmaf_rn(x.hi, rk.x, -q)));
  const float u = __fmul_rn(t.hi, q);
  const float ue = __fmaf_rn(t.hi, qe, __fmaf_rn(t.lo, q, __fmaf_rn(t.hi, q, -u)));
  const ff s = two_sum(1.0f, u);
  return fast_two_sum(s.hi, __fadd_rn(s.lo, ue));
}

// One step of the fraction's numerators: p_k = b_k p_(k+1) + a_(k+1) p_(k+2),
// scaled by s (a power of two).  Beyond k = a the second term is negative, but
// the fraction converges there without losing more than a few bits.
__device__ __forceinline__ ff pf_fraction_step(ff b0, float k, float a, float s, ff p1, ff p2)
{
  const ff b2 = two_sum(b0.hi, k + k);
  const ff b = ff_make(b2.hi * s, (b2.lo + b0.lo) * s);
  const float ak = (k + 1.f) * (a - (k + 1.f)) * (s * s);
  // b p1 and ak p2 unnormalised, one TwoSum of their leading parts
  const float u = __fmul_rn(b.hi, p1.hi), v = __fmul_rn(ak, p2.hi);
  const float ue = __fmaf_rn(b.hi, p1.lo, __fmaf_rn(b.lo, p1.hi, __fmaf_rn(b.hi, p1.hi, -u)));
  const float ve = __fmaf_rn(ak, p2.lo, __fmaf_rn(ak, p2.hi, -v));
  const ff t = two_sum(u, v);
  return fast_two_sum(t.hi, __fadd_rn(t.lo, __fadd_rn(ue, ve)));
}

}  // namespace
