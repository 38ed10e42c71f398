// surf_common.cuh -- shared pieces of the split-precision surface: the
// prepared operands, the exact recomputation of one term, the online
// log-sum-exp state, shared per-point thresholds and the FP64 merge of
// per-chunk partials.
#pragma once
#include <cstdint>

#include "ff.cuh"
#include "internal.h"

constexpr int SURF_K = 30;          // exact terms: 2 (theta + migration parameters)
constexpr int SURF_KP = 32;         // screened columns: the terms, the bias (tensor-core screen: in two), zero padding
constexpr int SURF_MAX_CHUNKS = 64;
constexpr float SURF_MARGIN = 32.0f;  // nats below the running max that still count
constexpr int SURF_SEED = 256;      // genealogies sampled per point for the seed maximum (FP32 screen)
constexpr int SURF_SAMPLES = 256;   // evenly spaced genealogies whose terms decide how a point is taken
constexpr int SURF_DENSE_TILE = 64; // genealogies per tile of the direct form
constexpr int SURF_TC_M = 128;      // tensor-core screen: points per A tile
constexpr int SURF_TC_N = 256;      // tensor-core screen: genealogies per B tile

// Operands prepared once per evaluation (model type and points fixed).
struct SurfPrep {
  int G, Gpad, K, np, nm;
  float *samp;      // [SURF_SAMPLES][SURF_KP] columns of the sampled genealogies
  float *sT;        // [SURF_KP][Gpad] statistics (exact floats), column K = bias (rounded)
  float2 *biasff;   // [Gpad] bias as float-float
  float2 *phiff;    // [npoints][SURF_K] phi as float-float
  float *phi32;     // [npoints][SURF_KP] phi rounded, 1 in the bias column
  float *mag;       // [npoints] sum_k colmax_k |phi_k|: scale of screening errors
  float *err;       // [npoints] error bound of the tensor-core screen
  float *seed;      // [npoints] exact max over a sample of genealogies
  unsigned *best;   // [npoints] best exact maximum found so far (ordered bits), shared by chunks
  unsigned *xmax;   // [npoints] largest exact value the refinement met (ordered bits; tensor-core screen)
  unsigned *colmax; // [SURF_KP] max |column| as float bits
  unsigned *emax;   // [SURF_KP] max |column - its FP16 form| as float bits (tensor-core screen)
  uint16_t *sh;     // FP16 statistics in 256-row MMA tiles (tensor-core screen)
  uint16_t *ph;     // FP16 phi in 128-row MMA tiles (tensor-core screen)
  float4 *sR;       // [Gpad][SURF_KP / 4] a genealogy's statistics in one line, columns 30, 31 its bias
                    // as float-float (tensor-core form: single terms)
};

// Per (point, chunk) partial of the online log-sum-exp.
struct SurfPart {
  float mh, ml;  // running maximum (float-float)
  float sh, sl;  // sum of exp(p - max) (float-float)
  float s2;      // sum of exp(2 (p - max)) for the effective sample size
  float pad;
};

// exact p_g(x) = bias + sum_k s_k phi_k, s_k exact floats, phi_k float-float:
// compensated dot product (Ogita, Rump & Oishi 2005, Dot2) on the high parts,
// the low parts and all error terms gathered in one float
__device__ __forceinline__ ff surf_exact(const SurfPrep &S, int g, const float *col, int stride,
                                         const float2 *phi)
{
  float2 b = S.biasff[g];
  float sum = b.x, comp = b.y;
  // fully unrolled with a bound check: phi stays in registers and the
  // column loads issue together
#pragma unroll
  for (int k = 0; k < SURF_K; k++) {
    if (k >= S.K) break;
    float s = col[k * stride];
    float2 f = phi[k];
    float p = __fmul_rn(s, f.x);
    float pe = __fmaf_rn(s, f.x, -p);
    float t = __fadd_rn(sum, p);
    float bb = __fsub_rn(t, sum);
    float te = __fadd_rn(__fsub_rn(sum, __fsub_rn(t, bb)), __fsub_rn(p, bb));
    sum = t;
    comp = __fadd_rn(comp, __fadd_rn(te, __fmaf_rn(s, f.y, pe)));
  }
  return fast_two_sum(sum, comp);
}

// the same from the genealogy's line: seven or eight 16-byte loads issued
// together where the columns of sT would be as many sectors as statistics
__device__ __forceinline__ ff surf_exact_row(const SurfPrep &S, int g, const float2 *phi)
{
  const float4 *r = S.sR + (size_t)g * (SURF_KP / 4);
  float v[SURF_KP];
#pragma unroll
  for (int q = 0; q < SURF_KP / 4; q++) {
    const float4 t = 4 * q < S.K || q == SURF_KP / 4 - 1 ? __ldg(r + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    v[4 * q] = t.x;
    v[4 * q + 1] = t.y;
    v[4 * q + 2] = t.z;
    v[4 * q + 3] = t.w;
  }
  float sum = v[SURF_KP - 2], comp = v[SURF_KP - 1];
#pragma unroll
  for (int q = 0; q < (SURF_K + 3) / 4; q++) {
    if (4 * q >= S.K) break;
#pragma unroll
    for (int k = 4 * q; k < 4 * q + 4 && k < SURF_K; k++) {
      const float2 f = phi[k];
      const float p = __fmul_rn(v[k], f.x);
      const float pe = __fmaf_rn(v[k], f.x, -p);
      const ff t = two_sum(sum, p);
      sum = t.hi;
      comp = __fadd_rn(comp, __fadd_rn(t.lo, __fmaf_rn(v[k], f.y, pe)));
    }
  }
  return fast_two_sum(sum, comp);
}

// e^(dh + dl) for |dh| <= 86: d = k ln2 / 64 + r, |r| <= ln2 / 128, e^r from
// its series (r and r^2/2 in float-float, r^3 .. r^5 in FP32), times tab[k &
// 63] = 2^((k & 63)/64) (float-float).  Relative error below 2e-14 for |d| < 1
// and 3e-14 |d| beyond.
__device__ __forceinline__ ff exp_tab(float dh, float dl, const float2 *tab)
{
  const float z = __fmaf_rn(dh, 92.33248262f, 12582912.f);
  const float kf = __fsub_rn(z, 12582912.f);
  const int k = __float_as_int(z) - 0x4B400000;
  float h = __fmaf_rn(-kf, L64_B, __fmaf_rn(-kf, L64_A, dh));  // both exact
  const ff r = two_sum(h, __fmaf_rn(-kf, L64_C, dl));
  h = r.hi;
  const float p = __fmul_rn(h, h), pe = __fmaf_rn(h, h, -p);
  const float q = __fmul_rn(__fmul_rn(p, h), __fmaf_rn(h, __fmaf_rn(h, 1.f / 120, 1.f / 24), 1.f / 6));
  const ff u = fast_two_sum(h, 0.5f * p);  // r + r^2/2
  const float w = __fadd_rn(u.lo, __fmaf_rn(u.hi, r.lo, __fadd_rn(r.lo, __fmaf_rn(0.5f, pe, q))));
  const float2 T = tab[k & 63];
  const float a = __fmul_rn(T.x, u.hi), ae = __fmaf_rn(T.x, u.hi, -a);
  const float lo = __fadd_rn(__fmaf_rn(T.x, w, __fmaf_rn(T.y, u.hi, ae)), T.y);
  const ff s = fast_two_sum(T.x, a);
  const float sc = __int_as_float((127 + (k >> 6)) << 23);
  return ff_make(s.hi * sc, __fadd_rn(s.lo, lo) * sc);
}

struct LseState {
  ff m, s;
  float s2;
  __device__ __forceinline__ void init()
  {
    m = ff_make(-INFINITY, 0.f);
    s = ff_from(0.f);
    s2 = 0.f;
  }
  __device__ __forceinline__ void add(ff y)
  {
    if (m.hi == -INFINITY) {
      m = y;
      s = ff_from(1.f);
      s2 = 1.f;
      return;
    }
    ff d = ff_sub(y, m);
    float dd = d.hi + d.lo;
    if (dd > 0.f) {
      float e = expf(-dd);
      s = ff_add_f(ff_mul_f(s, e), 1.0f);
      s2 = s2 * e * e + 1.0f;
      m = y;
    } else {
      float e = expf(dd);
      s = ff_add_f(s, e);
      s2 += e * e;
    }
  }
  __device__ __forceinline__ SurfPart pack() const
  {
    SurfPart p;
    p.mh = m.hi;
    p.ml = m.lo;
    p.sh = s.hi;
    p.sl = s.lo;
    p.s2 = s2;
    p.pad = 0.f;
    return p;
  }
  __device__ __forceinline__ void unpack(const SurfPart &o)
  {
    m = ff_make(o.mh, o.ml);
    s = ff_make(o.sh, o.sl);
    s2 = o.s2;
  }
  // fold another partial (same point) into this one
  __device__ __forceinline__ void merge(const SurfPart &o)
  {
    if (o.mh == -INFINITY) return;
    if (m.hi == -INFINITY) {
      m = ff_make(o.mh, o.ml);
      s = ff_make(o.sh, o.sl);
      s2 = o.s2;
      return;
    }
    ff om = ff_make(o.mh, o.ml);
    ff d = ff_sub(om, m);
    float dd = d.hi + d.lo;
    ff os = ff_make(o.sh, o.sl);
    if (dd > 0.f) {
      float e = expf(-dd);
      s = ff_add(ff_mul_f(s, e), os);
      s2 = s2 * e * e + o.s2;
      m = om;
    } else {
      float e = expf(dd);
      s = ff_add(s, ff_mul_f(os, e));
      s2 += o.s2 * e * e;
    }
  }
};

// order-preserving float <-> uint for atomicMax on shared thresholds
__device__ __forceinline__ unsigned f2ord(float f)
{
  unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned u)
{
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

size_t surf_prep_bytes(int G, int npoints);
SurfPart *surf_prep_carve(SurfPrep *S, char *base, int G, int npoints);
// The operands.  tc: the tensor-core ones too.  rows_ready: the row-derived
// ones (sT, biasff, colmax, samp; tc: emax, sh, sR) are already in place from
// an earlier evaluation of the same rows and model type.  nseed > 0: seed,
// best and xmax from the exact terms of that many evenly spaced genealogies
// (32 or 256).  z0, z1: words to clear on the way.  Returns the kernels queued.
struct SurfZero {
  int *z0 = nullptr, n0 = 0, *z1 = nullptr, n1 = 0;
};
int surf_prep(const SurfArgs &a, SurfPrep &S, bool tc, bool rows_ready, int nseed, const SurfZero &z, cudaStream_t st);
void surf_merge(const SurfArgs &a, const SurfPart *part, int nchunks, cudaStream_t st);

// How the points of an evaluation are taken (k_surf_dense.cu): dense[p] = 1
// where every term is evaluated directly, the list of those points,
// counts[0] = their number and counts[1 + t] = points of tensor-core tile t
// left to the screen.
struct SurfSplit {
  uint8_t *dense;
  int *list, *counts;
};
int surf_init_tables();
float2 *surf_exp_table();  // device address of 2^(j/64), j < 64, as float-float
void surf_split(const SurfPrep &S, int npoints, const SurfSplit &D, cudaStream_t st);
int surf_dense_grid(const SurfArgs &a, int nsm);
// the chunking of nd dense points over a grid of nb CTAs: about three equal
// rounds of (32 points, chunk) units, at most SURF_MAX_CHUNKS chunks of whole
// tiles; the merge recomputes it from the same two numbers
__host__ __device__ inline int surf_dense_chunks(int nd, int nb, int G, int *per)
{
  const int ntiles = (G + SURF_DENSE_TILE - 1) / SURF_DENSE_TILE;
  const int groups = (nd + 31) / 32;
  int n = groups > 0 ? 3 * nb / groups : 1;
  const int lim = ntiles < SURF_MAX_CHUNKS ? ntiles : SURF_MAX_CHUNKS;
  n = n < 1 ? 1 : n > lim ? lim : n;
  *per = (ntiles + n - 1) / n;
  return (ntiles + *per - 1) / *per;
}
void surf_dense(const SurfArgs &a, const SurfPrep &S, const SurfSplit &D, int nb, double2 *part, cudaStream_t st);
