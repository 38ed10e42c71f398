// k_margin.cu -- 1-D marginal posterior densities (margincalc,
// surface_call_functions.cpp:119-175; fillvec, histograms.cpp:82-99).
//
// For parameter p at x the density is (1/G) sum_g exp(term_g):
//   population size p:  -qi_p + round(cc_p) (ln 2 - ln x) - hcc_p - 2 fc_p / x
//   migration rate p:   -mi_p + round(mc_p) ln x - fm_p x
//                       (+ ln(1/mean) - x / mean under an exponential prior)
// summed in FP64 without a shift, as the reference sums it (the values span
// hundreds of orders of magnitude and the reference returns them as they are).
// marginp (surface_call_functions.cpp:25-80), the peak searches' form, sums a
// range of genealogies, takes the theta term's cc as stored and divides by
// the range's length (+1 when it starts at genealogy 0).
//
// A term is c a(x) + f b(x) + base: c the count, f the rate and base
// everything that does not depend on x, all of one genealogy.  A CTA takes
// requests of one parameter, so a tile's (c, f, base) go to shared memory as
// doubles once for all its requests, in units of ln 2, and a term costs two
// FP64 FMAs (three under an exponential prior); 2^term is formed in fixed
// point on the integer pipe and summed in 96-bit integers (fxexp.cuh).  GB300
// issues about 1.6 FP64 operations or conversions per cycle and SM: the
// former kernel (conversions, six operations and an FP64 exponential per
// term) spent 20 cycles a term, 83.5 ms for 13,000 points x 100,000
// genealogies; now 6.9 ms, 5.2 of them the two FMAs of each term.  (6.8 while
// the products with log2 e were left rounded: on the rows of a run the
// densities were off by 3.2e-16 to 4.2e-16 of their mean from an FP64
// evaluation, now by 1.4e-16, with FP64 exponentials by 2.0e-16 to 2.8e-16.)
// Adding the doubles instead (a third FP64 operation) measured 14.6 ms against 11.9 for
// the integer sums before the last two steps (integer compare, shorter tail).
//
// Threads: `nx` requests by MG_BS / nx genealogy strides, nx the power of two
// that holds the largest parameter's requests, so a search's few points
// still use every lane.  Partial sums per chunk are added in a fixed order by
// the merge kernel.
#include <cfloat>
#include <cmath>

#include "fxexp.cuh"
#include "internal.h"

namespace {

constexpr int MG_BS = 128;  // threads per CTA
constexpr int MG_TG = 128;  // genealogies per shared-memory tile
constexpr double LOG2 = 0.69314718055994530942;
constexpr double LOG2E = 1.4426950408889634074, LOG2E_LO = 2.0355273740931033e-17;  // log2 e, and the rest of it
constexpr double FX_ONE = 9007199254740992.0;  // 2^53: fx_fix's fraction bits
constexpr int FX_LIMIT_HI = 0x408f4000;  // high word of 1000.0, the bound of the fixed-point form's argument

__constant__ uint64_t c_fxtab[FX_TAB];

__device__ __forceinline__ double intround(float v)  // INTEGERROUND (imamp.hpp:180)
{
  return v >= 0.f ? (double)(long long)((double)v + 0.5) : (double)(long long)((double)v - 0.5);
}

template <bool EXPO>
__global__ void __launch_bounds__(MG_BS) k_margin(MarginArgs a, int lognx, int chunk, double *part)
{
  __shared__ uint64_t tab[FX_TAB];
  __shared__ double sc[MG_TG], sf[MG_TG], sb[MG_TG];
  __shared__ float4 sl[MG_TG];  // c and f in FP32, and what the rounding of base leaves (2^-53)
  const int tid = threadIdx.x, nx = 1 << lognx;
  const int k = blockIdx.x * nx + (tid & (nx - 1));  // this thread's request
  const int sub = tid >> lognx, nsub = MG_BS >> lognx;
  for (int i = tid; i < FX_TAB; i += MG_BS) tab[i] = c_fxtab[i];
  const int pi = a.param[blockIdx.x * nx];
  const double x = a.x[k];
  const bool theta = pi < a.np;
  // The term's coefficients, as the reference rounds them, in units of ln 2;
  // and in units of 2^-53 what that product's rounding leaves.  (That is the
  // same for every genealogy, or of base for every x, and where few
  // genealogies make the sum neither averages out.)
  const double a_ = theta ? LOG2 - log(x) : log(x), b_ = theta ? 1.0 / x : x;
  const double A = a_ * LOG2E, B = b_ * LOG2E;
  const float Al = (float)((__fma_rn(a_, LOG2E, -A) + a_ * LOG2E_LO) * FX_ONE);
  const float Bl = (float)((__fma_rn(b_, LOG2E, -B) + b_ * LOG2E_LO) * FX_ONE);
  double cst = 0.0;
  float cl = 0.f;
  if (EXPO && !theta) {
    const double meani = 1.0 / a.expo_mean[pi - a.np], c_ = log(meani) - x * meani;
    cst = c_ * LOG2E;
    cl = (float)((__fma_rn(c_, LOG2E, -cst) + c_ * LOG2E_LO) * FX_ONE);
  }
  const int p = pi - a.np;  // columns: (qi, cc, hcc, fc) or (mi, mc, fm)
  const int c0 = theta ? a.qip + pi : a.mip + p, c1 = theta ? a.ccp + pi : a.mcp + p,
            c2 = theta ? a.hccp + pi : a.fmp + p, c3 = theta ? a.fcp + pi : c2;
  const int g0 = a.g_lo + blockIdx.y * chunk, g1 = min(a.g_hi, g0 + chunk);
  FxSum sum;
  sum.init();
  int since = 0;  // terms since the last flush
  for (int t0 = g0; t0 < g1; t0 += MG_TG) {
    const int nt = min(MG_TG, g1 - t0);
    __syncthreads();
    if (tid < nt) {
      const float *r = a.rows + (size_t)(t0 + tid) * a.rowlen;
      const float r0 = r[c0], r1 = r[c1], r2 = r[c2], r3 = r[c3];
      sc[tid] = theta && a.raw_cc ? (double)r1 : intround(r1);
      sf[tid] = theta ? -2.0 * (double)r3 : -(double)r2;
      const double base = theta ? -(double)r0 - (double)r2 : -(double)r0;
      sb[tid] = base * LOG2E;
      sl[tid] = make_float4((float)sc[tid], (float)sf[tid],
                            (float)((__fma_rn(base, LOG2E, -sb[tid]) + base * LOG2E_LO) * FX_ONE), 0.f);
    }
    __syncthreads();
    for (int j = sub; j < nt; j += nsub) {
      double v = __fma_rn(sf[j], B, __fma_rn(sc[j], A, sb[j]));
      if (EXPO) v += cst;
      // |v| < 1000, compared as bits: a DSETP would be a third FP64 operation
      if ((__double2hiint(v) & 0x7fffffff) < FX_LIMIT_HI) {
        int i;
        const float4 l = sl[j];
        const uint64_t m = fx_exp2(fx_fix(v) + __float2int_rn(__fmaf_rn(l.x, Al, __fmaf_rn(l.y, Bl, EXPO ? l.z + cl : l.z))), tab, &i);
        sum.add(m, i);
      } else {  // beyond it, infinite or NaN
        sum.total += exp2(v);
      }
    }
    since += (nt - sub + nsub - 1) / nsub;
    if (since > 512 - MG_TG) {
      sum.flush();
      since = 0;
    }
  }
  sum.flush();
  double s = sum.total;
  if (nsub > 1) {  // the strides of a request, pairwise
    __shared__ double red[MG_BS];
    red[tid] = s;
    for (int o = nsub >> 1; o; o >>= 1) {
      __syncthreads();
      if (sub < o) red[tid] = s += red[tid + (o << lognx)];
    }
  }
  if (sub == 0) part[(size_t)k * gridDim.y + blockIdx.y] = s;
}

// a warp per request: its chunks by lane, then the lanes pairwise (fewer
// roundings follow one another than chunk by chunk)
__global__ void __launch_bounds__(128) k_margin_merge(MarginArgs a, int nchunks, const double *part, double *out)
{
  const int k = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k >= a.n) return;
  double s = 0.0;
  for (int c = lane; c < nchunks; c += 32) s += part[(size_t)k * nchunks + c];
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane) return;
  s /= a.div;
  if (a.logi) s = (s <= 0.0) ? -1e200 : log(s);  // LOWLOG
  out[k] = s - a.yadjust;
}

}  // namespace

int margin_init_tables()
{
  struct Tab {
    uint64_t t[FX_TAB];
  };
  static const Tab tab = [] {  // once per process (long double is slow in software on aarch64)
    Tab v;
    for (int j = 0; j < FX_TAB; j++) v.t[j] = (uint64_t)(exp2l((long double)j / FX_TAB) * 9223372036854775808.0L);
    return v;
  }();
  return cudaMemcpyToSymbol(c_fxtab, tab.t, sizeof(tab.t)) == cudaSuccess ? 0 : -1;
}

int margin_chunks(int G, int nblocks)
{
  // about six waves of eight resident CTAs per SM: the last one is then a
  // small share (two waves left a quarter of the kernel to its tail)
  int nchunks = (48 * 152 + nblocks - 1) / nblocks;
  const int maxc = (G + 2 * MG_TG - 1) / (2 * MG_TG);  // at least two tiles per chunk
  if (nchunks > maxc) nchunks = maxc;
  return nchunks < 1 ? 1 : nchunks;
}

int margin_log_block(int most)
{
  int l = 0;
  while ((1 << l) < most && (1 << l) < MG_BS) l++;
  return l;
}

int launch_margin(const MarginArgs &a, int lognx, double *part, int nchunks, double *out, cudaStream_t st)
{
  if (a.n < 1) return 2;
  const int ng = a.g_hi - a.g_lo;
  if (ng < 1) return 2;
  const int chunk = ((ng + nchunks - 1) / nchunks + MG_TG - 1) / MG_TG * MG_TG;
  nchunks = (ng + chunk - 1) / chunk;
  const dim3 grid(a.n >> lognx, nchunks);
  if (a.expo_mean) k_margin<true><<<grid, MG_BS, 0, st>>>(a, lognx, chunk, part);
  else k_margin<false><<<grid, MG_BS, 0, st>>>(a, lognx, chunk, part);
  k_margin_merge<<<(a.n + 3) / 4, 128, 0, st>>>(a, nchunks, part, out);
  return 0;
}
