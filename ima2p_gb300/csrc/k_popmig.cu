// k_popmig.cu -- posterior densities of the population migration rate
// 2NM = theta_i m_j / 2 over the loaded genealogies: calc_popmig and, under
// an exponential migration prior, calc_pop_expomig (popmig.cpp:9-172), the
// functions print_populationmigrationrate_histograms evaluates on its grids
// (histograms.cpp:755-810).
//
// Under a uniform prior a genealogy's term is one or two incomplete gamma
// functions.  k_popmig_fast evaluates it by popfast.cuh: truncated series and
// fractions in float-float (their lengths decided in FP32), the powers and
// exponentials in fixed point, some 17 FP64 operations a term where the
// logarithmic form took about 760 (GB300 issues 1.6 per cycle and SM).  The
// terms popfast.cuh leaves out, and the exponential prior (k_popmig), take the
// FP64 form below, written in the reference's operation order but for the
// sums inside igamma.cuh.
//
// k_popmig_fast: a warp takes a block of 2^lognx points of one term and a
// chunk of genealogies, 32 at a time staged in its shared memory by the warp's
// lanes (converted once for all its points); the lanes are the block's points
// times 32 / 2^lognx strides over the genealogies, so a search's few points
// still use every lane.  Against truth computed in extended precision on
// 1.6 million random terms its mean relative error is 1e-14, that of the FP64
// form 9e-7 on the same terms (log(1 - P) loses what x2 - x1 needs).
// Measured on 8 curves of 1,000 points over 10,000 genealogies: 121.6 ms
// before, 21.4 with every piece of the term inlined twice (instruction cache
// misses were half of the stalls), 13.2 now.  k_popmig: a CTA is one warp of 32 points and one chunk, each lane
// walking the rows.
// Each (point, chunk) partial has its own slot.  calc_popmig's sum
// of exp(temp1 + temp2) (terms outside +-700 skipped) is kept per chunk;
// calc_pop_expomig's eexp mantissa / decimal-exponent terms are kept per
// chunk rescaled to the chunk's largest exponent.  The merge kernel adds the
// chunks in chunk order, rescales them to the overall largest exponent, and
// divides by G and, for likelihoods, by the prior density of 2NM.  The peak
// search's forms (marginpopmig, marginpop_expomig; :181-351) sum a range of
// genealogies and divide by its length (+1 when it starts at genealogy 0).
//
// This file is compiled with -fmad=false; log, exp and pow are the device's.
#include <cmath>

#include "internal.h"
#include "igamma.cuh"
#include "eexp.cuh"
#include "popfast.cuh"

namespace {

constexpr int PM_BS = 32;  // points per CTA (one warp)
constexpr double LOG10 = 2.3025850929940456840;
constexpr int OCUTOFF = 10;

// calc_popmig's term for one genealogy (popmig.cpp:33-84): temp1 + temp2, or
// NaN when the reference would skip it.
__device__ double popmig_term(IgBase &ig, int cc, double fc, double hc, int mc, double fm, double qintg,
                              double mintg, double x, double qmax, double mmax)
{
  double temp1, temp2;
  if (fc == 0 && cc == 0 && fm > 0) {
    temp1 = LOG2 - (mc * log(fm)) - hc - qintg - mintg;
    temp2 = log(exp(ig.upper(mc, 2 * fm * x / qmax)) - exp(ig.upper(mc, mmax * fm)));
  } else if (fm == 0 && mc == 0 && fc > 0) {
    temp1 = LOG2 - (cc * log(fc)) - hc - qintg - mintg;
    temp2 = log(exp(ig.upper(cc, 2 * fc / qmax)) - exp(ig.upper(cc, fc * mmax / x)));
  } else if (fc == 0 && cc == 0 && mc == 0 && fm == 0) {
    temp1 = log(2 * log(mmax * qmax / (2 * x))) - hc - qintg - mintg;
    temp2 = 0;
  } else {
    temp1 = LOG2 + (mc * log(x)) - ((cc + mc) * log(fc + fm * x)) - hc - qintg - mintg;
    double a = ig.upper(cc + mc, 2 * (fc + fm * x) / qmax);
    double b = ig.upper(cc + mc, mmax * (fm + fc / x));
    if (a == b) {  // both saturated: the lower functions separate them
      b = ig.lower(cc + mc, 2 * (fc + fm * x) / qmax);
      a = ig.lower(cc + mc, mmax * (fm + fc / x));
    }
    if (a > b) {
      temp2 = ig.logdiff(a, b);
    } else {
      temp1 = temp2 = 0.0;  // the reference adds exp(0) for these
    }
  }
  return temp1 + temp2;
}

// calc_pop_expomig's log term for one genealogy (popmig.cpp:114-147).
__device__ double popexpo_term(IgBase &ig, int cc, double fc, double hc, int mc, double fm, double qintg,
                               double mintg, double x, double qmax, double mmean)
{
  const double temp1 = x + fc * mmean + fm * mmean * x;
  double temp2 = LOG2 - hc - log(mmean) - qintg - mintg;
  double temp3 = 2 * temp1 / (mmean * qmax);
  if (mc == 0 && cc == 0) {
    temp3 = ig.upper(0, temp3);
    temp2 += temp3;
  } else if (cc == 0) {
    temp3 = ig.upper(mc, temp3);
    temp2 += temp3 - mc * log(fm + 1 / mmean);
  } else if (mc == 0) {
    temp3 = ig.upper(cc, temp3);
    temp2 += temp3 + -cc * log(fc + x * (fm + 1 / mmean));
  } else {
    temp3 = ig.upper(mc + cc, temp3);
    temp2 += temp3 - cc * log(x) + (cc + mc) * log(mmean * x / temp1);
  }
  return temp2;
}

// the FP64 form for one lane, out of line: few terms take it
__device__ __noinline__ double popmig_slow(const double *logfact, const float *r, int th, int mi, int np, int nm,
                                           double x, double qmax, double mmax, int *st)
{
  IgBase ig{logfact, 0};
  const float *m = r + 3 * np;
  const double t = popmig_term(ig, (int)r[th], r[np + th], r[2 * np + th], (int)m[mi], m[nm + mi], m[2 * nm + th],
                               m[2 * nm + np + mi], x, qmax, mmax);
  if (ig.st) *st = ig.st;
  return t < 700 && t > -700 ? exp(t) : 0.0;
}

constexpr int PF_WARPS = 4;  // warps per CTA, each with its own block of points and chunk

struct PfTables {
  uint64_t ex[FX_TAB];
  FxLogTab lg;
  float2 rcp[PF_RCP];
};
__device__ PfTables d_pf;  // filled by popmig_init_tables

// a genealogy's values as the fast form reads them
struct PfGen {
  double fc, fm, mc, a, base, baseg, gln;  // base = 1 - (hc + q + m) log2 e, gln = log Gamma(a), baseg = base + log2 Gamma(a)
  int na;                             // a, or 0: not for the fast form
};

// S(x) / a or H(x) with n terms
__device__ __forceinline__ ff pf_value(ff x, bool series, int na, int n, const float2 *rcp)
{
  if (series) {
    ff t = ff_from(1.f);
#pragma unroll 1
    for (int k = n; k >= 1; k--) t = pf_series_step(t, x, rcp[na + k]);
    return ff_mul(t, ffc(rcp[na]));
  }
  const ff b0 = ff_add_f(x, (float)(1 - na));
  const float sc = __int_as_float((254 - ((__float_as_int(b0.hi + (float)n) >> 23) & 0xff)) << 23);
  const ff bn = ff_add_f(b0, (float)(2 * n));
  ff p1 = ff_make(bn.hi * sc, bn.lo * sc), p2 = ff_from(1.f);
#pragma unroll 1
  for (int k = n - 1; k >= 0; k--) {
    const ff q = pf_fraction_step(b0, (float)k, (float)na, sc, p1, p2);
    p2 = p1;
    p1 = q;
  }
  const ff h = ff_div(p2, p1);
  return ff_make(h.hi * sc, h.lo * sc);
}

__device__ __forceinline__ double pf_double(uint64_t m, int i)  // m 2^(i - 63), |i| < 1000
{
  return __longlong_as_double((long long)(((uint64_t)(i + 1022) << 52) + (m >> 11)));
}
__device__ __forceinline__ bool pf_in(double e) { return (__double2hiint(e) & 0x7fffffff) < 0x408f3800; }  // |e| < 999

// |a - b| < 998 of two fixed-point values below 999 (their difference may pass 2^63)
__device__ __forceinline__ bool pf_sub_in(int64_t a, int64_t b) { return abs((int)(((a >> 1) - (b >> 1)) >> 52)) < 998; }
// inside (e^-700, e^700), where the reference adds the term (the two bounds'
// own binades' edges go to the FP64 form)
__device__ __forceinline__ bool pf_kept(double d)
{
  const int h = __double2hiint(d);
  return h > 0x00d14f2b && h < 0x7f0d945d;
}
// log of a double in (0, 1], to 2^-60 absolute
__device__ __forceinline__ double pf_ln(double q, const FxLogTab &T)
{
  int e;
  const uint64_t f = fx_log2(q, T, &e);
  return ((double)(e + 1) - (f ? (double)(0ull - f) * 5.421010862427522e-20 : 1.0)) * 0.69314718055994530942;
}
constexpr double DIFF_MIN = 1.0 / 128;

__global__ void __launch_bounds__(32 * PF_WARPS, 4) k_popmig_fast(PopmigArgs a, int lognx, int nblocks, int nchunks,
                                                               int chunk, double *part)
{
  __shared__ PfTables T;
  __shared__ PfGen gen[PF_WARPS][32];
  for (int i = threadIdx.x; i < (int)(sizeof(PfTables) / 4); i += 32 * PF_WARPS)
    reinterpret_cast<uint32_t *>(&T)[i] = reinterpret_cast<const uint32_t *>(&d_pf)[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long unit = (long long)blockIdx.x * PF_WARPS + warp;
  const int blk = (int)(unit % nblocks), ch = (int)(unit / nblocks);
  if (ch >= nchunks) return;
  const int nx = 1 << lognx, sub = lane >> lognx, nsub = 32 >> lognx;
  const int k = (blk << lognx) + (lane & (nx - 1));
  const int th = a.thetai[k], mi = a.mi[k], np = a.fcp - a.ccp, nm = a.fmp - a.mcp;
  const double x = a.x[k], qmax = a.qmax[k], mmax = a.mmax[k];
  // per-point factors: x1 = r1 z, x2 = r2 z
  const double r1 = 2.0 / qmax, r2 = mmax / x;
  const ff r1f = ff_make((float)r1, (float)(r1 - (double)(float)r1));
  const ff r2f = ff_make((float)r2, (float)(r2 - (double)(float)r2));
  const double lx = log2(x), l1 = log2(r1), l2 = log2(r2), c1 = -r1 * PF_LOG2E, c2 = -r2 * PF_LOG2E;
  // factors that leave the float range (or zero, infinite): every term to the FP64 form
  const bool fine = x > 1e-10 && x < 1e10 && r1 > 1e-10 && r1 < 1e10 && r2 > 1e-10 && r2 < 1e10;
  const int g0 = a.g_lo + ch * chunk, g1 = min(a.g_hi, g0 + chunk);
  double sum = 0.0;
  int st = 0;
  for (int t0 = g0; t0 < g1; t0 += 32) {
    __syncwarp();
    if (t0 + lane < g1) {
      const float *r = a.rows + (size_t)(t0 + lane) * a.rowlen;
      const int cc = (int)r[a.ccp + th], mc = (int)r[a.mcp + mi], na = cc + mc;
      const float fc = r[a.fcp + th], fm = r[a.fmp + mi];
      // the general branch only, in ranges where z, x1 and x2 are normal floats
      const bool ok = na >= 1 && na < PF_AMAX && cc >= 0 && mc >= 0 && !(fc == 0.f && cc == 0) &&
                      !(fm == 0.f && mc == 0) && fc >= 0.f && fm >= 0.f && fc + fm > 1e-6f && fc < 1e8f && fm < 1e8f;
      PfGen &G = gen[warp][lane];
      G.fc = fc;
      G.fm = fm;
      G.mc = mc;
      G.a = na;
      G.na = ok ? na : 0;
      G.base = __fma_rn(-((double)r[a.hccp + th] + (double)r[a.qip + th] + (double)r[a.mip + mi]), PF_LOG2E, 1.0);
      G.gln = ok ? a.logfact[na - 1] : 0.0;
      G.baseg = __fma_rn(G.gln, PF_LOG2E, G.base);
    }
    __syncwarp();
    const int nt = min(32, g1 - t0);
    for (int j = sub; j < nt; j += nsub) {
      const PfGen &G = gen[warp][j];
      const int na = G.na;
      double D = -1.0;  // < 0: left to the FP64 form
      if (na > 0 && fine) {
        const double z = __fma_rn(G.fm, x, G.fc);
        const ff zf = ff_split(z);
        const float fa = (float)na;
        const double K = __fma_rn(G.mc, lx, G.base);
        // x1 then x2 through the same instructions (the kernel's code would
        // not fit the instruction cache twice): value, exponent, kind
        double v[2];
        int64_t f[2];
        bool s[2], ok = true;
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
          const ff xh = ff_mul(zf, h ? r2f : r1f);
          const bool se = __fsub_rn(xh.hi, fa + 1.f) + xh.lo < 0.f;
          const int n = se ? pf_series_terms(fa, xh.hi) : pf_fraction_terms(fa, __fsub_rn(xh.hi, fa - 1.f) + xh.lo);
          const double e = __fma_rn(z, h ? c2 : c1, __fma_rn(G.a, h ? l2 : l1, K));
          ok = ok && n > 0 && pf_in(e);
          const ff vf = pf_value(xh, se, na, n, T.rcp);
          const double vd = (double)vf.hi + (double)vf.lo;
          const int64_t fe = fx_fix(e);
          if (h == 0) {
            v[0] = vd;
            f[0] = fe;
            s[0] = se;
          } else {
            v[1] = vd;
            f[1] = fe;
            s[1] = se;
          }
        }
        ok = ok && (s[0] || !s[1]);
        // everything relative to 2^w: Gamma(a) z^-a where x1 takes the series
        // (which needs log z), else x1's own factor
        int64_t w = f[0];
        if (s[0]) {
          const double kg = __fma_rn(G.mc, lx, G.baseg);
          int e;
          const uint64_t lf = fx_log2(z, T.lg, &e);
          const int ae = na * e;
          ok = ok && pf_in(kg) && abs(ae) < 999;
          const int64_t la = ((int64_t)ae << 53) +
                             (int64_t)((((uint64_t)(uint32_t)na * (uint32_t)(lf >> 32)) << 21) +
                                       (((uint64_t)(uint32_t)na * (uint32_t)lf) >> 11));
          const int64_t fk = fx_fix(kg);
          ok = ok && pf_sub_in(fk, la);
          w = fk - la;
        }
        ok = ok && pf_sub_in(f[0], w) && pf_sub_in(f[1], w);
        if (ok) {
          double g1s = 0.0, g2s = 0.0, big = 0.0;
#pragma unroll 1
          for (int h = 0; h < 3; h++) {
            int i;
            const uint64_t m = fx_exp2(h == 2 ? w : (h ? f[1] : f[0]) - w, T.ex, &i);
            const double e = pf_double(m, i);
            if (h == 0) g1s = e * v[0];
            else if (h == 1) g2s = e * v[1];
            else big = e;
          }
          double d = -1.0, rel;  // rel: the difference over its larger part
          if (!s[0]) {
            d = g1s - g2s;
            rel = d > DIFF_MIN * g1s ? 1.0 : 0.0;
            d *= big;
          } else if (!s[1]) {
            rel = 1.0 - g1s - g2s;
            d = rel * big;
          } else {
            // both from series: the reference subtracts two logarithms gln +
            // log(1 - P), and where P is small their rounding (an ulp of gln)
            // is what its difference keeps; rounded alike here
            rel = 1.0;
            double A[2];
            const double q2 = 1.0 - g2s;
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
              const double q = h ? q2 : 1.0 - g1s;
              rel = q > 0.0 ? rel : 0.0;
              const double l = G.gln + pf_ln(q, T.lg);
              if (h == 0) A[0] = l;
              else A[1] = l;
            }
            const double df = A[0] - A[1];
            if (df > 0.0) {
              int i;
              const uint64_t m = fx_exp2(fx_fix(df * PF_LOG2E), T.ex, &i);
              const double E = __longlong_as_double((long long)(((uint64_t)(i + 1022) << 52) + (m >> 11) +
                                                                ((m >> 10) & 1)));
              d = (E - 1.0) * q2 * big;
              if (E == 1.0) rel = 0.0;  // the reference takes log(0)
            } else {
              d = (g2s - g1s) * big;  // equal: it turns to the lower functions, which separate them
              if (df < 0.0) rel = 0.0;
            }
          }
          // below DIFF_MIN the rounding of the reference's logarithms shows
          if (rel > DIFF_MIN && pf_kept(d)) D = d;
        }
      }
      sum += D >= 0.0 ? D
                      : popmig_slow(a.logfact, a.rows + (size_t)(t0 + j) * a.rowlen, th, mi, np, nm, x, qmax, mmax, &st);
    }
  }
  if (st) atomicCAS(a.err, 0, st);
  for (int w = 1; w < nsub; w++) {  // the strides of a point, in order
    const double o = __shfl_sync(0xffffffffu, sum, (lane & (nx - 1)) + (w << lognx));
    if (sub == 0) sum += o;
  }
  if (sub == 0) {
    const size_t o = (size_t)k * nchunks + ch;
    part[2 * o] = sum;
    part[2 * o + 1] = 0.0;
  }
}

// the exponential prior: sum of m 10^(z - (maxz - OCUTOFF))
__global__ void __launch_bounds__(PM_BS) k_popmig(PopmigArgs a, int chunk, double *part)
{
  const int k = blockIdx.x * PM_BS + threadIdx.x;
  if (k >= a.n) return;
  const int th = a.thetai[k], mi = a.mi[k];
  const double x = a.x[k], qmax = a.qmax[k], mmean = a.mmean[k];
  const float *c_cc = a.rows + a.ccp + th, *c_fc = a.rows + a.fcp + th, *c_hc = a.rows + a.hccp + th;
  const float *c_qi = a.rows + a.qip + th, *c_mc = a.rows + a.mcp + mi, *c_fm = a.rows + a.fmp + mi;
  const float *c_mi = a.rows + a.mip + mi;
  IgBase ig{a.logfact, 0};
  double sum = 0.0;
  int maxz = -1000000000;  // the chunk's largest decimal exponent
  const int g0 = a.g_lo + blockIdx.y * chunk, g1 = min(a.g_hi, g0 + chunk);
  for (int g = g0; g < g1; g++) {
    const size_t o = (size_t)g * a.rowlen;
    const int cc = (int)__ldg(c_cc + o), mc = (int)__ldg(c_mc + o);
    const double fc = __ldg(c_fc + o), hc = __ldg(c_hc + o), fm = __ldg(c_fm + o);
    const double qintg = __ldg(c_qi + o), mintg = __ldg(c_mi + o);
    const double t = popexpo_term(ig, cc, fc, hc, mc, fm, qintg, mintg, x, qmax, mmean);
    double m;
    int z;
    eexp_dev(t, &m, &z);
    if (z > maxz) {  // a new largest exponent: earlier terms rescale to it
      if (sum != 0.0) sum *= pow(10.0, (double)(maxz - z));
      maxz = z;
    }
    sum += m * pow(10.0, (double)(z - (maxz - OCUTOFF)));
  }
  const size_t o = (size_t)k * gridDim.y + blockIdx.y;
  part[2 * o] = sum;
  part[2 * o + 1] = (double)maxz;
  if (ig.st) atomicCAS(a.err, 0, ig.st);
}

__global__ void k_popmig_merge(PopmigArgs a, int nchunks, const double *part, double *out)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= a.n) return;
  const double *w = part + 2 * (size_t)k * nchunks;
  const double x = a.x[k], qmax = a.qmax[k], mmax = a.mmax[k];
  double sum = 0.0;
  if (!a.expo) {
    for (int c = 0; c < nchunks; c++) sum += w[2 * c];
    sum /= a.div;
    if (a.prob_or_like) {
      const double temp = 2 * (log(qmax) + log(mmax) - log(2 * x)) / (qmax * mmax);
      sum /= temp;
    }
  } else {
    const double mmean = a.mmean[k];
    int maxz = -1000000000;
    for (int c = 0; c < nchunks; c++) maxz = max(maxz, (int)w[2 * c + 1]);
    double acumm = 0.0;
    for (int c = 0; c < nchunks; c++)
      if (w[2 * c] != 0.0) acumm += w[2 * c] * pow(10.0, (double)((int)w[2 * c + 1] - maxz));
    sum = log(acumm) + (maxz - OCUTOFF) * LOG10;
    sum -= log(a.div);
    sum = exp(sum);
    if (a.prob_or_like) {
      IgBase ig{a.logfact, 0};
      const double temp = 2 * exp(ig.upper(0, 2 * x / (mmean * qmax))) / (qmax * mmean);
      sum /= temp;
      if (ig.st) atomicCAS(a.err, 0, ig.st);
    }
  }
  out[k] = sum;
}

}  // namespace

// the tables, made once per process (long double is slow in software on aarch64)
static const PfTables &pf_tables()
{
  static const PfTables t = [] {
    PfTables v{};
    for (int j = 0; j < FX_TAB; j++) {
      v.ex[j] = (uint64_t)(exp2l((long double)j / FX_TAB) * 9223372036854775808.0L);
      const uint64_t r = (4294967296ull * FX_TAB + FX_TAB + j - 1) / (FX_TAB + j);  // ceil
      v.lg.r[j] = (uint32_t)(r - 1);
      v.lg.l[j] = j ? (uint64_t)(-log2l((long double)r / 4294967296.0L) * 18446744073709551616.0L) : 0ull;
    }
    for (int k = 1; k < PF_RCP; k++) {
      const long double w = 1.0L / k;
      v.rcp[k] = make_float2((float)w, (float)(w - (long double)(float)w));
    }
    return v;
  }();
  return t;
}

int popmig_init_tables()
{
  return cudaMemcpyToSymbol(d_pf, &pf_tables(), sizeof(PfTables)) == cudaSuccess ? 0 : -1;
}

int popmig_log_block(int most)
{
  int l = 0;
  while ((1 << l) < most && l < 5) l++;
  return l;
}

int popmig_chunks(int G, int nblocks, int expo)
{
  // about 16 waves of warps (16 to 20 resident per SM), chunks of at least 64
  // genealogies (128 in the fast form, whose CTAs load 13 KB of tables)
  long long nchunks = (16LL * 152 * 20 + nblocks - 1) / nblocks;
  const long long maxc = expo ? (G + 63) / 64 : (G + 127) / 128;
  if (nchunks > maxc) nchunks = maxc;
  if (nchunks > 65535) nchunks = 65535;  // grid y limit
  return nchunks < 1 ? 1 : (int)nchunks;
}

int launch_popmig(const PopmigArgs &a, int lognx, double *part, int nchunks, double *out, cudaStream_t st)
{
  const int ng = a.g_hi - a.g_lo;
  if (a.n < 1 || ng < 1) return 2;
  const int quantum = a.expo ? 1 : 32;
  const int chunk = ((ng + nchunks - 1) / nchunks + quantum - 1) / quantum * quantum;
  nchunks = (ng + chunk - 1) / chunk;
  if (a.expo) {
    k_popmig<<<dim3((a.n + PM_BS - 1) / PM_BS, nchunks), PM_BS, 0, st>>>(a, chunk, part);
  } else {
    const int nb = a.n >> lognx;
    const long long units = (long long)nb * nchunks;
    k_popmig_fast<<<(unsigned)((units + PF_WARPS - 1) / PF_WARPS), 32 * PF_WARPS, 0, st>>>(a, lognx, nb, nchunks, chunk,
                                                                                   part);
  }
  k_popmig_merge<<<(a.n + 127) / 128, 128, 0, st>>>(a, nchunks, part, out);
  return 0;
}
