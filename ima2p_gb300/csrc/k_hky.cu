// k_hky.cu -- HKY85 Felsenstein pruning over site patterns (makefrac,
// calc_prob_data.cpp:118-471; likelihoodHKY :583-607) and the accept/reject of
// its partial likelihoods (copyfraclike / storescalefactors /
// restorescalefactors, update_gtree_common.cpp:2140-2181).
//
// One CTA per chain-locus.  Internal nodes are visited level by level (the
// host supplies, with each genealogy, its internal nodes sorted by height);
// inside a level every (node, pattern) pair is independent, so the CTA's
// threads sweep them with one barrier per level.  A node is recomputed when
// it is on the dirty list, when the list is -1 (full), or when a daughter is
// dirty or recomputed -- the reference's propagation rule (:137-163).
//
// Partial likelihoods are resident state in two slots per node: slot[node]
// names the committed one ("frac"), the other receives new values
// ("newfrac").  Accept flips the slot of every recomputed node, reject keeps
// it; this replaces the reference's buffer copies with a one-byte flip.
//
// FP32 form: partials are float4, rescaled after every node by an exact
// power of two whose exponent is kept as an integer, so the log scale factor
// carries no rounding; the root sum log(sum_j pi_j L_j) is formed from an
// FP32 mantissa log and the integer exponent, accumulated in FP64.
// Float-float form (the default fast precision): the same kernel with every
// partial, coefficient and product as a float-float pair (about 46 bits):
// the hi parts in the FP32 partial array, the lo parts in a second one, the
// exponents shared.  An FP32 partial's rounding (6e-8) repeats in every
// site of a pattern, so a 1000-bp locus of FP32 pruning is off by ~1e-4 in
// log L; the pairs bring that below 1e-8.
// FP64 form: the reference's arithmetic -- partials divided by their maximum,
// log(max) accumulated into an FP64 scale factor.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ff.cuh"
#include "internal.h"

namespace {

__constant__ FFConsts c_ffh;     // ln 2 and the log table (filled by hky_init_tables)
__device__ float2 d_exp64m1[64];  // 2^((j - 32) / 64) - 1 as float-float

constexpr int HKY_BS = 128;
constexpr double LN2 = 0.69314718055994530941723212146;

__device__ __forceinline__ float branch_ff(const NodeRec *nd, const float2 *t, int c)
{
  int u = nd[c].up0;
  if (u < 0) return t[c].x + t[c].y;
  return (t[c].x - t[u].x) + (t[c].y - t[u].y);
}

__device__ __forceinline__ double branch_64(const NodeRec *nd, const double *t, int c)
{
  int u = nd[c].up0;
  return (u < 0) ? t[c] : t[c] - t[u];
}

// HKY85 transition matrix P[j][k] = P(j -> k | b), Pi and A from the class
// (purine / pyrimidine) of the target state k.
template <typename T>
__device__ __forceinline__ void hky_p(const T *pi, T kpa, T b, T *P)
{
  T e1 = exp(-b);
  T PR = pi[0] + pi[2], PY = pi[1] + pi[3];
  T eR = exp(-b * (T(1) + PR * kpa)), eY = exp(-b * (T(1) + PY * kpa));
#pragma unroll
  for (int k = 0; k < 4; k++) {
    T Pk = (k == 0 || k == 2) ? PR : PY;
    T e2 = (k == 0 || k == 2) ? eR : eY;
    T base = pi[k] + pi[k] * e1 * (T(1) / Pk - T(1));
#pragma unroll
    for (int j = 0; j < 4; j++) {
      T v;
      if (j == k) v = base + e2 * ((Pk - pi[k]) / Pk);
      else if (j + k == 2 || j + k == 4) v = base - (pi[k] / Pk) * e2;
      else v = pi[k] * (T(1) - e1);
      P[j * 4 + k] = v;
    }
  }
}

// The same matrix for FP32 as five coefficients per branch.  With
// E1 = 1 - exp(-b) and E2_c = 1 - exp(-b A_c), A_c = 1 + Pi_c (kappa - 1),
// both taken from expm1 so that short branches do not cancel, the entries are
//   transversion  pi_k E1
//   transition    (pi_k / Pi_c) (E2_c - E1 (1 - Pi_c))
//   identity      the transition value plus 1 - E2_c
// and with the states ordered A, C, G, T (purines R = {A, G}, pyrimidines
// Y = {C, T}) the product of P(b) with a partial L is, for j in class c and
// the other class o,
//   v_j = E1 S_o + b_c S_c + d_c L_j,   S_c = sum_{k in c} pi_k L_k,
//   b_c = (E2_c - E1 (1 - Pi_c)) / Pi_c,   d_c = 1 - E2_c.
// K = {E1, b_R, b_Y, d_R, d_Y}.
__device__ __forceinline__ void hky_coef_fast(const float *pi, float kpa, float b, float *K)
{
  const float E1 = -expm1f(-b);
  const float PR = pi[0] + pi[2], PY = pi[1] + pi[3];
  const float ER = -expm1f(-b * (1.0f + PR * kpa)), EY = -expm1f(-b * (1.0f + PY * kpa));
  K[0] = E1;
  K[1] = (ER - E1 * (1.0f - PR)) / PR;
  K[2] = (EY - E1 * (1.0f - PY)) / PY;
  K[3] = 1.0f - ER;
  K[4] = 1.0f - EY;
}

// P(b) L for one child at one pattern: a tip observed in state st, or an
// internal node's partial Lc
struct HkyCoef {
  float a, bR, bY, dR, dY;
};
__device__ __forceinline__ void hky_apply_tip(const HkyCoef &K, const float *pi, int st, float *v)
{
  const float p = pi[st];
  const bool isR = (st & 1) == 0;
  const float tR = (isR ? K.bR : K.a) * p, tY = (isR ? K.a : K.bY) * p;
  v[0] = tR + (st == 0 ? K.dR : 0.0f);
  v[2] = tR + (st == 2 ? K.dR : 0.0f);
  v[1] = tY + (st == 1 ? K.dY : 0.0f);
  v[3] = tY + (st == 3 ? K.dY : 0.0f);
}
__device__ __forceinline__ void hky_apply(const HkyCoef &K, const float *pi, float4 L, float *v)
{
  const float SR = fmaf(pi[2], L.z, pi[0] * L.x), SY = fmaf(pi[3], L.w, pi[1] * L.y);
  const float tR = fmaf(K.bR, SR, K.a * SY), tY = fmaf(K.bY, SY, K.a * SR);
  v[0] = fmaf(K.dR, L.x, tR);
  v[2] = fmaf(K.dR, L.z, tR);
  v[1] = fmaf(K.dY, L.y, tY);
  v[3] = fmaf(K.dY, L.w, tY);
}

// e^x and e^x - 1 of x <= 0 in float-float: x = k ln2 / 64 + r, |r| <= ln2 /
// 128, y = 2^(j/64) e^r - 1 from its table t_j = 2^(j/64) - 1, j in [-32, 32)
// (signed, so that a short branch has j = 0 and keeps its relative accuracy),
// and m = e^r - 1: y = t + m + t m; then e^x = 2^e (1 + y).  About 75
// instructions (a series to degree 7 and four doublings took 110); relative errors
// within 3e-14 of e^x - 1 and of e^x.
__device__ __forceinline__ void hky_exp(ff x, const float2 *tab, ff *ex, ff *em1)
{
  if (x.hi < -86.0f) {
    *ex = ff_from(0.0f);
    *em1 = ff_from(-1.0f);
    return;
  }
  const float z = __fmaf_rn(x.hi, 92.33248262f, 12582912.f);
  const float kf = __fsub_rn(z, 12582912.f);
  const int k = __float_as_int(z) - 0x4B400000;
  const float c = __fmul_rn(-kf, L64_C);
  ff r = two_sum(__fmaf_rn(-kf, L64_B, __fmaf_rn(-kf, L64_A, x.hi)), c);
  r.lo = __fadd_rn(r.lo, __fadd_rn(x.lo, __fmaf_rn(-kf, L64_C, -c)));
  const float h = r.hi;
  // m = r (1 + r (1/2 + r (1/6 + r (1/24 + r / 120))))
  const float g = __fmaf_rn(h, 1.f / 120, 1.f / 24);
  const float s3 = __fmaf_rn(h, g, 0.16666667f), s3l = __fmaf_rn(h, g, 0.16666667f - s3) - 4.967054e-09f;
  const float a1 = __fmul_rn(h, s3), a1e = __fmaf_rn(h, s3, -a1) + __fmaf_rn(h, s3l, r.lo * s3);
  const ff s2 = fast_two_sum(0.5f, a1);
  const float s2l = __fadd_rn(s2.lo, a1e);
  const float a2 = __fmul_rn(h, s2.hi), a2e = __fmaf_rn(h, s2.hi, -a2) + __fmaf_rn(h, s2l, r.lo * s2.hi);
  const ff s1 = fast_two_sum(1.0f, a2);
  const ff m = ff_mul(r, ff_make(s1.hi, __fadd_rn(s1.lo, a2e)));
  const int j = (k + 32) & 63, e = (k + 32 - j) >> 6;
  const ff t = ffc(tab[j]);
  const ff y = ff_add(ff_add(t, m), ff_mul(t, m));
  const float p2 = __int_as_float((127 + e) << 23);
  const ff one_y = ff_add_f(y, 1.0f);
  *ex = ff_make(one_y.hi * p2, one_y.lo * p2);
  *em1 = e == 0 ? y : ff_add_f(*ex, -1.0f);
}

// What the branches of a chain-locus share: A_c = 1 + Pi_c (kappa - 1),
// 1 / Pi_c and 1 - Pi_c of the two classes.
struct HkyShared {
  float2 AR, AY, iR, iY, oR, oY;
};

// Float-float coefficients of one branch, K = {E1, b_R, b_Y, d_R, d_Y} as
// (hi, lo) pairs: E1 = 1 - e^-b, E2_c = 1 - e^(-b A_c), d_c = e^(-b A_c)
// taken directly (1 - E2_c would cancel on long branches).
__device__ __forceinline__ void hky_coef_ff(const HkyShared &H, const float2 *tab, ff b, float *K)
{
  ff e1, m1, eR, mR, eY, mY;
  hky_exp(ff_neg(b), tab, &e1, &m1);
  hky_exp(ff_neg(ff_mul(b, ffc(H.AR))), tab, &eR, &mR);
  hky_exp(ff_neg(ff_mul(b, ffc(H.AY))), tab, &eY, &mY);
  const ff E1 = ff_neg(m1), ER = ff_neg(mR), EY = ff_neg(mY);
  const ff bR = ff_mul(ff_sub(ER, ff_mul(E1, ffc(H.oR))), ffc(H.iR));
  const ff bY = ff_mul(ff_sub(EY, ff_mul(E1, ffc(H.oY))), ffc(H.iY));
  K[0] = E1.hi; K[1] = E1.lo;
  K[2] = bR.hi; K[3] = bR.lo;
  K[4] = bY.hi; K[5] = bY.lo;
  K[6] = eR.hi; K[7] = eR.lo;
  K[8] = eY.hi; K[9] = eY.lo;
}

// Every operand of the pruning products is >= 0, so these sums never cancel.
// a*b + c:
__device__ __forceinline__ ff ff_fma_pos(ff a, ff b, ff c)
{
  const float p = __fmul_rn(a.hi, b.hi);
  const float pe = __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.hi, -p)));
  const ff s = two_sum(p, c.hi);
  return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(pe, c.lo)));
}

// Two float-floats at once, in the packed FP32 instructions: states are
// taken as the pairs (A, C) and (G, T), so that a pair holds one purine and
// one pyrimidine and the two classes' sums and coefficients are pairs too.
// A packed instruction takes one issue slot for two results (measured 105-119
// results per cycle and SM against 83 of the scalar ones).
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_pack(float x, float y)
{
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 f2_un(f2 a)
{
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b)
{
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b)
{
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c)
{
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 f2_neg(f2 a) { return a ^ 0x8000000080000000ull; }
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) { return f2_add(a, f2_neg(b)); }
struct ff2 {
  f2 hi, lo;
};
__device__ __forceinline__ ff2 ff2_make(f2 h, f2 l)
{
  ff2 r;
  r.hi = h;
  r.lo = l;
  return r;
}
// a b and a b + c, every operand >= 0, left unnormalised (|lo| may reach a few
// ulp(hi)): the next step's TwoSum is exact whatever lo is
__device__ __forceinline__ ff2 ff2_mul_u(ff2 a, ff2 b)
{
  const f2 p = f2_mul(a.hi, b.hi);
  return ff2_make(p, f2_fma(a.hi, b.lo, f2_fma(a.lo, b.hi, f2_fma(a.hi, b.hi, f2_neg(p)))));
}
__device__ __forceinline__ ff2 ff2_fma_u(ff2 a, ff2 b, ff2 c)
{
  const ff2 p = ff2_mul_u(a, b);
  const f2 s = f2_add(p.hi, c.hi), bb = f2_sub(s, p.hi);
  const f2 e = f2_add(f2_sub(p.hi, f2_sub(s, bb)), f2_sub(c.hi, bb));
  return ff2_make(s, f2_add(e, f2_add(p.lo, c.lo)));
}
// the product renormalised; of unnormalised factors, so lo x lo counts
__device__ __forceinline__ ff2 ff2_mul(ff2 a, ff2 b)
{
  const f2 p = f2_mul(a.hi, b.hi);
  const f2 e = f2_fma(a.hi, b.lo, f2_fma(a.lo, b.hi, f2_fma(a.lo, b.lo, f2_fma(a.hi, b.hi, f2_neg(p)))));
  const f2 s = f2_add(p, e);
  return ff2_make(s, f2_sub(e, f2_sub(s, p)));
}
__device__ __forceinline__ void ff2_load(const float4 &hi, const float4 &lo, ff2 *v)
{
  v[0] = ff2_make(f2_pack(hi.x, hi.y), f2_pack(lo.x, lo.y));
  v[1] = ff2_make(f2_pack(hi.z, hi.w), f2_pack(lo.z, lo.w));
}

// An internal branch's coefficients as pairs: (E1, E1), (b_R, b_Y), (d_R,
// d_Y), hi parts then lo parts (12 floats).  v_j = E1 S_o + b_c S_c + d_c L_j,
// left unnormalised: its only use is the product of the two daughters.
__device__ __forceinline__ void hky_apply_ff(const float *K, const ff2 *pi, const ff2 *L, ff2 *v)
{
  const float4 k0 = reinterpret_cast<const float4 *>(K)[0], k1 = reinterpret_cast<const float4 *>(K)[1],
               k2 = reinterpret_cast<const float4 *>(K)[2];
  const ff2 a = ff2_make(f2_pack(k0.x, k0.y), f2_pack(k1.z, k1.w)), b = ff2_make(f2_pack(k0.z, k0.w), f2_pack(k2.x, k2.y)),
            d = ff2_make(f2_pack(k1.x, k1.y), f2_pack(k2.z, k2.w));
  const ff2 S = ff2_fma_u(pi[1], L[1], ff2_mul_u(pi[0], L[0]));  // (S_R, S_Y)
  const float2 sh = f2_un(S.hi), sl = f2_un(S.lo);
  const ff2 O = ff2_make(f2_pack(sh.y, sh.x), f2_pack(sl.y, sl.x));
  const ff2 t = ff2_fma_u(b, S, ff2_mul_u(a, O));
  v[0] = ff2_fma_u(d, L[0], t);
  v[1] = ff2_fma_u(d, L[1], t);
}

// P(b) applied to a tip observed in state st: column st of P(b), (b_R, E1) or
// (E1, b_Y) times pi_st, and d of its class added at st itself.  (Columns made
// once per branch took 144 bytes of shared memory a tip, which cost more
// resident CTAs than these thirty instructions do.)
__device__ __forceinline__ void hky_apply_tip_ff(const float *K, float2 p, int st, ff2 *v)
{
  const float4 k0 = reinterpret_cast<const float4 *>(K)[0], k1 = reinterpret_cast<const float4 *>(K)[1],
               k2 = reinterpret_cast<const float4 *>(K)[2];
  const bool isR = (st & 1) == 0;
  const ff2 c = ff2_make(f2_pack(isR ? k0.z : k0.x, isR ? k0.x : k0.w), f2_pack(isR ? k2.x : k1.z, isR ? k1.z : k2.y));
  const ff2 t = ff2_mul_u(c, ff2_make(f2_pack(p.x, p.x), f2_pack(p.y, p.y)));
  const float2 th = f2_un(t.hi), tl = f2_un(t.lo);
  const ff s = two_sum(isR ? th.x : th.y, isR ? k1.x : k1.y);
  const float oh = s.hi, ol = __fadd_rn(s.lo, __fadd_rn(isR ? tl.x : tl.y, isR ? k2.z : k2.w));
  v[0] = ff2_make(f2_pack(st == 0 ? oh : th.x, st == 1 ? oh : th.y), f2_pack(st == 0 ? ol : tl.x, st == 1 ? ol : tl.y));
  v[1] = ff2_make(f2_pack(st == 2 ? oh : th.x, st == 3 ? oh : th.y), f2_pack(st == 2 ? ol : tl.x, st == 3 ? ol : tl.y));
}
__device__ __forceinline__ ff ff_of(float2 v) { return ff_make(v.x, v.y); }

// Shared-memory carve-up, identical on host (sizing) and device.
// coef: bytes of the branches' coefficients; fast: with the node times, the
// tips and the list's offsets of k_hky_fast.
struct HkyLayout {
  size_t nd, times, fresh, order, tip, off, total;
};
__host__ __device__ inline HkyLayout hky_layout(int maxnl, size_t coef, bool fast)
{
  const size_t nl = (size_t)maxnl;
  HkyLayout l;
  l.nd = coef;
  l.times = l.nd + sizeof(NodeRec) * nl;
  l.fresh = l.times + (fast ? sizeof(float2) * nl : 0);
  l.order = (l.fresh + 3 * nl + 15) & ~size_t(15);
  l.tip = l.order + sizeof(int16_t) * (nl + 3);
  l.off = fast ? (l.tip + sizeof(int16_t) * nl + 3) & ~size_t(3) : l.tip;
  l.total = (l.off + (fast ? sizeof(int32_t) * (nl / 2 + 2) : 0) + 15) & ~size_t(15);
  return l;
}
__host__ __device__ inline HkyLayout hky_layout64(int maxnl)  // k_hky_fp64: a 4 x 4 matrix per branch
{
  return hky_layout(maxnl, 16 * sizeof(double) * (size_t)maxnl, false);
}
// k_hky_fast: floats per branch (5 coefficients, as pairs in float-float) and
// per tip's branch (float-float with every pattern kept: the four columns of
// P(b) as pairs)
__host__ __device__ constexpr int hky_floats(bool ff) { return ff ? 12 : 8; }
__host__ __device__ constexpr int hky_tip_floats(bool uni, bool ff) { return ff && !uni ? 32 : hky_floats(ff); }
__host__ __device__ inline HkyLayout hky_layout_fast(int maxnl, bool uni, bool ff)
{
  const size_t maxn = (size_t)(maxnl + 1) / 2;
  return hky_layout(maxnl, 4 * (maxn * hky_tip_floats(uni, ff) + (maxn - 1) * hky_floats(ff)), true);
}

// ----------------------------------------------------- uniform patterns
// Where every tip below a node shows the same state x, the node's partial at
// that pattern depends on x alone.  So a node keeps one partial per pattern
// that is mixed below it (in pattern order from entry 4 on) and one per state x
// (at entry x) for all the others: on
// sequences simulated on their genealogies 8-26% of the (node, pattern) pairs,
// on random genealogies 33-49%.  Which patterns are mixed depends only on the
// tips below, so a clean node's stored partials stay addressable whatever
// happens above.  Masks of mixed patterns come bottom-up from the tips' states,
// kept as two bit planes per tip (P.planes): mixed(v) = mixed(a) | mixed(b) |
// (planes of a tip below a != planes of a tip below b).  The tasks (one per
// recomputed node and entry) are listed in schedule order, x = (node - n) |
// entry << 16, y = the daughters' entries (a tip's state), the internal
// daughter first.  A full evaluation's list depends on the topology alone: it
// is kept per item and read back while P.is_valid says so.  The list of an
// evaluation from edited edges is shorter; what of it does not fit in shared
// memory goes to the same place, which ends the kept list.
// Loci whose masks pass HKY_MASK_WORDS, or whose patterns 16 bits, keep every
// pattern and have no list (UNI false in the kernel), and so do those where
// most tips differ (hky_uniform_entries).
constexpr int HKY_MASK_WORDS = 8192;
__device__ __forceinline__ int2 hky_children(const NodeRec &nd, int n)  // the internal daughter first
{
  return nd.up0 < n && nd.up1 >= n ? make_int2(nd.up1, nd.up0) : make_int2(nd.up0, nd.up1);
}

// Per-CTA shared state common to both precisions.
struct Tree {
  NodeRec *nd;
  uint8_t *fresh;
  uint8_t *dirty;
  uint8_t *slot;
  int16_t *order;
  int16_t *lstart;
};

__device__ double standfactor(const double *pi, double kappa)
{
  double p = 0.0;
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < 4; j++) {
      if (i == j) continue;
      p += (i + j == 2 || i + j == 4) ? pi[i] * pi[j] * kappa : pi[i] * pi[j];
    }
  return p;
}

// Loads topology and schedule, marks dirty nodes and decides which internal
// nodes are recomputed.  Returns after a barrier.
__device__ void load_tree(const Pools &P, const ItemDev &it, const ReqDev &R, int nlev, Tree &T,
                          const uint8_t *gslot)
{
  const int n = it.n, nl = 2 * n - 1;
  for (int k = threadIdx.x; k < nl; k += blockDim.x) {
    T.nd[k] = P.nodes[it.node_off + k];
    T.dirty[k] = 0;
    T.slot[k] = gslot[it.node_off + k];
  }
  for (int k = threadIdx.x; k < n - 1 + nlev + 1; k += blockDim.x)
    T.order[k] = P.sched[it.sched_off + k];
  __syncthreads();
  if (threadIdx.x == 0) {
    bool full = (R.e[0] == -1);
    for (int q = 0; q < 4; q++)
      if (R.e[q] >= 0 && R.e[q] < nl) T.dirty[R.e[q]] = 1;
    for (int k = 0; k < n - 1; k++) {
      int node = T.order[k];
      int a = T.nd[node].up0, b = T.nd[node].up1;
      bool f = full || T.dirty[node] || T.dirty[a] || T.dirty[b] ||
               (a >= n && T.fresh[a]) || (b >= n && T.fresh[b]);
      T.fresh[node] = f ? 1 : 0;
    }
  }
  __syncthreads();
}

__device__ __forceinline__ float pow2f(int k)  // 2^k for -126 <= k <= 127
{
  return __int_as_float((127 + k) << 23);
}

__device__ __forceinline__ int expo_of(float m)  // floor(log2(m)) for normal m > 0
{
  return ((__float_as_int(m) >> 23) & 0xff) - 127;
}

// ------------------------------------------------------------------ FP32
// One CTA per chain-locus, internal nodes level by level.  Each branch gets
// the five coefficients of hky_coef_fast (in place of a 4 x 4 matrix).  UNI: a
// node's partials are those of its mixed patterns and of the four states, and
// a thread takes a task of the list at a time.  Otherwise a node keeps every
// pattern and a warp takes one node and 32 of its patterns at a time, so that
// the children's coefficients are warp-uniform and no warp mixes tip and
// internal children.  BS threads per CTA, registers for MINB resident CTAs per
// SM.  FF: every value a float-float pair (the lo parts of the partials in
// P.partlo); otherwise FP32 (which clears the lo parts of what it writes when
// they exist, so a later FF evaluation reads its partials as exact pairs).
template <bool UNI, bool FF, int BS, int MINB>
__global__ void __launch_bounds__(BS, MINB) k_hky_fast(Pools P, const ReqDev *reqs,
                                                     double *result, int32_t *status, int maxnl,
                                                     int mcap, int pcap, int tcap)
{
  extern __shared__ __align__(16) char smem[];
  // the request carries the item's offsets and sizes, so the tree loads
  // below wait on this one load only
  const ReqDev R = reqs[blockIdx.x];
  const int n = R.n, nl = 2 * n - 1, S = R.nsites, nint = n - 1;
  constexpr int PB = hky_floats(FF), PT = hky_tip_floats(UNI, FF);
  const HkyLayout lay = hky_layout_fast(maxnl, UNI, FF);
  float *Pt = reinterpret_cast<float *>(smem);  // [n][PT], a tip's branch
  float *Pm = Pt + (PT - PB) * n;               // [2n - 1][PB], from n on: the other branches
  float2 *stm = reinterpret_cast<float2 *>(smem + lay.times);        // node times
  Tree T;
  T.nd = reinterpret_cast<NodeRec *>(smem + lay.nd);
  T.fresh = reinterpret_cast<uint8_t *>(smem + lay.fresh);
  T.dirty = T.fresh + maxnl;
  T.slot = T.dirty + maxnl;
  T.order = reinterpret_cast<int16_t *>(smem + lay.order);
  int16_t *tipof = reinterpret_cast<int16_t *>(smem + lay.tip);  // a tip below each node
  int32_t *toff = reinterpret_cast<int32_t *>(smem + lay.off);   // tasks before the k-th node of the schedule
  // the last tcap tasks (the narrow levels, where an L2 round trip of about
  // 1,000 cycles would be the level), the masks of mixed patterns [nint][W],
  // the tips' planes [n][2][W] where they fit in pcap words
  uint2 *stask = reinterpret_cast<uint2 *>(smem + lay.total);
  uint32_t *mixed = reinterpret_cast<uint32_t *>(stask + tcap);
  uint32_t *splane = mixed + mcap;
  uint16_t *ahead = reinterpret_cast<uint16_t *>(splane + pcap);  // mixed patterns of a node before each mask word
  __shared__ double red_d[BS / 32];
  __shared__ long long red_e[BS / 32];
  __shared__ float2 spi[4];   // pi (FP32: .x only)
  __shared__ float2 smu, skpa, stab[FF ? 64 : 1];
  __shared__ HkyShared sH;

  const int tid = threadIdx.x;
  const bool full = (R.e[0] == -1);
  for (int k = tid; k < nl; k += BS) {
    T.nd[k] = P.nodes[R.node_off + k];
    stm[k] = P.tff[R.node_off + k];
    T.slot[k] = P.slot32[R.node_off + k];
    T.dirty[k] = 0;
    T.fresh[k] = full ? 1 : 0;
  }
  // the schedule (n-1 + nlev+1 entries, nlev <= n-1) in its 2n-entry slot,
  // without waiting for the level count
  for (int k = tid; k < 2 * n; k += BS) T.order[k] = P.sched[R.sched_off + k];
  const int nlev = P.nlev[R.item];
  T.lstart = T.order + nint;
  const int W = (S + 31) >> 5, S4 = S + 4;  // S4: partials stored per node
  const int lw = W > 1 ? 32 - __clz(W - 1) : 0;  // words per node rounded up to 2^lw
  const uint32_t *plane = P.planes + R.plane_off;
  uint2 *task = P.task + R.part_off / 2;
  int32_t *gtoff = P.toff + R.sched_off;
  const bool listed = UNI && full && P.is_valid[R.item];
  // the list's offsets are loaded beside the flag that says whether they hold
  if (UNI && full)
    for (int k = tid; k < n; k += BS) toff[k] = gtoff[k];
  if (UNI && !listed && n * 2 * W <= pcap) {
    for (int k = tid; k < n * 2 * W; k += BS) splane[k] = plane[k];
    plane = splane;
  }
  if (tid == 0) {
    // mu = u / (totsites standfactor) in FP64, the standard factor as 2 kappa
    // (pA pG + pC pT) + 2 (pA + pG) (pC + pT): its sum of twelve products held
    // up the CTA for some 3,000 cycles
    const double *pid = P.pi + 4 * (size_t)R.item;
    const double p0 = pid[0], p1 = pid[1], p2 = pid[2], p3 = pid[3];
    smu = ff_round(R.u / (2.0 * R.totsites * fma(R.par, fma(p0, p2, p1 * p3), (p0 + p2) * (p1 + p3))));
  } else if (tid == 32) {
    const double *pid = P.pi + 4 * (size_t)R.item;
    ff pj[4];
    for (int j = 0; j < 4; j++) {
      spi[j] = ff_round(pid[j]);
      pj[j] = ff_of(spi[j]);
    }
    skpa = ff_round(R.par - 1.0);
    const ff PR = ff_add(pj[0], pj[2]), PY = ff_add(pj[1], pj[3]), kp = ff_of(skpa), one = ff_from(1.0f);
    auto put = [](ff v) { return make_float2(v.hi, v.lo); };
    sH.AR = put(ff_add_f(ff_mul(PR, kp), 1.0f));
    sH.AY = put(ff_add_f(ff_mul(PY, kp), 1.0f));
    sH.iR = put(ff_div(one, PR));
    sH.iY = put(ff_div(one, PY));
    sH.oR = put(ff_add_f(ff_neg(PR), 1.0f));
    sH.oY = put(ff_add_f(ff_neg(PY), 1.0f));
  }
  if (FF)
    for (int k = tid; k < 64; k += BS) stab[k] = d_exp64m1[k];
  __syncthreads();
  if (!full && tid < 32) {  // the reference's propagation rule, a level at a time
    const int ed = tid == 0 ? R.e[0] : tid == 1 ? R.e[1] : tid == 2 ? R.e[2] : R.e[3];
    if (tid < 4 && ed >= 0 && ed < nl) T.dirty[ed] = 1;
    __syncwarp();
    for (int lv = 0; lv < nlev; lv++) {
      for (int k = T.lstart[lv] + tid; k < T.lstart[lv + 1]; k += 32) {
        const int node = T.order[k], a = T.nd[node].up0, b = T.nd[node].up1;
        T.fresh[node] = (T.dirty[node] || T.dirty[a] || T.dirty[b] || (a >= n && T.fresh[a]) || (b >= n && T.fresh[b])) ? 1 : 0;
      }
      __syncwarp();
    }
  }
  if (!full) __syncthreads();
  // the masks and the nodes' task counts by the first warp, the branches'
  // coefficients by the others
  const bool build = UNI && !listed;
  if (listed) {  // the copies land during the coefficients
    const int tbase = max(0, toff[nint] - tcap);
    for (int k = tbase + tid; k < toff[nint]; k += BS)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(stask + k - tbase)),
                   "l"(task + k)
                   : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  if (build && tid < 32) {
    for (int k = tid; k < n; k += 32) tipof[k] = (int16_t)k;
    __syncwarp();
    for (int lv = 0; lv < nlev; lv++) {
      const int beg = T.lstart[lv], cnt = (T.lstart[lv + 1] - beg) << lw;
      for (int q = tid; q < cnt; q += 32) {
        const int w = q & ((1 << lw) - 1), node = T.order[beg + (q >> lw)];
        if (w >= W) continue;
        const int a = T.nd[node].up0, b = T.nd[node].up1, ta = tipof[a], tb = tipof[b];
        uint32_t m = (plane[2 * W * ta + w] ^ plane[2 * W * tb + w]) | (plane[2 * W * ta + W + w] ^ plane[2 * W * tb + W + w]);
        if (a >= n) m |= mixed[(a - n) * W + w];
        if (b >= n) m |= mixed[(b - n) * W + w];
        mixed[(node - n) * W + w] = m;
        if (w == 0) tipof[node] = (int16_t)ta;
      }
      __syncwarp();
    }
    int before = 0;
    for (int k0 = 0; k0 < nint; k0 += 32) {
      int c = 0;
      if (k0 + tid < nint) {
        const int node = T.order[k0 + tid];
        for (int w = 0; w < W; w++) {
          ahead[(node - n) * W + w] = (uint16_t)c;
          c += __popc(mixed[(node - n) * W + w]);
        }
        c = !T.fresh[node] ? 0 : T.nd[node].down < 0 ? S : c + 4;  // the root: every pattern, for the sum
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, c, o);
        if (tid >= o) c += v;
      }
      if (k0 + tid < nint) toff[k0 + tid + 1] = before + c;
      before += __shfl_sync(0xffffffffu, c, 31);
    }
    if (tid == 0) toff[0] = 0;
  }
  for (int c = build ? tid - 32 : tid; c < nl; c += build ? BS - 32 : BS) {
    if (c < 0) break;
    int d = T.nd[c].down;
    if (d < 0 || !T.fresh[d]) continue;
    if constexpr (FF) {
      const int u = T.nd[c].up0;
      const ff tc = ff_of(stm[c]);
      const ff br = (u < 0) ? tc : ff_sub(tc, ff_of(stm[u]));
      float Kc[10];
      hky_coef_ff(sH, stab, ff_mul(ff_of(smu), br), Kc);
      float4 *dst = reinterpret_cast<float4 *>(UNI || c >= n ? Pm + PB * c : Pt + PT * c);
      dst[0] = make_float4(Kc[0], Kc[0], Kc[2], Kc[4]);
      dst[1] = make_float4(Kc[6], Kc[8], Kc[1], Kc[1]);
      dst[2] = make_float4(Kc[3], Kc[5], Kc[7], Kc[9]);
      if (!UNI && c < n) {  // the four columns, over the coefficients they come from
        ff2 col[4][2];
#pragma unroll
        for (int st = 0; st < 4; st++) hky_apply_tip_ff(Pt + PT * c, spi[st], st, col[st]);
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const float2 h = f2_un(col[k >> 1][k & 1].hi), l = f2_un(col[k >> 1][k & 1].lo);
          dst[k] = make_float4(h.x, h.y, l.x, l.y);
        }
      }
    } else {
      float pil[4] = {spi[0].x, spi[1].x, spi[2].x, spi[3].x};
      hky_coef_fast(pil, skpa.x, smu.x * branch_ff(T.nd, stm, c), Pm + PB * c);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int tbase = UNI ? max(0, toff[nint] - tcap) : 0;
  if (build) {
    // a thread takes eight patterns of a node
    for (int q = tid; q < nint << (lw + 2); q += BS) {
      const int j = q >> (lw + 2), b8 = q & ((4 << lw) - 1), w = b8 >> 2, node = T.order[j];
      int at = toff[j];
      if (w >= W || toff[j + 1] == at) continue;  // no such word; not recomputed
      const int2 ch = hky_children(T.nd[node], n);
      auto put = [&](int ea, int eb) {
        const uint2 t = make_uint2((uint32_t)(node - n) | (uint32_t)(at - toff[j]) << 16, (uint32_t)ea | (uint32_t)eb << 16);
        if (at >= tbase) stask[at - tbase] = t;
        if (full || at < tbase) task[at] = t;
        at++;
      };
      const int sh = 8 * (b8 & 3);
      uint32_t m;
      if (j == nint - 1) {
        m = w == W - 1 && (S & 31) ? (1u << (S & 31)) - 1u : 0xffffffffu;
        at += 32 * w;
      } else {
        m = mixed[(node - n) * W + w];
        if (b8 == 0)
          for (int x = 0; x < 4; x++) put(x, x);
        else at += 4;
        at += ahead[(node - n) * W + w];
      }
      at += __popc(m & ((1u << sh) - 1u));
      m &= 0xffu << sh;
      if (!m) continue;
      // the daughters' entries: a tip's state, a mixed pattern's, or the state
      // of the tips below
      const int ta = tipof[ch.x], tb = tipof[ch.y];
      const uint32_t a0 = plane[2 * W * ta + w], a1 = plane[2 * W * ta + W + w], b0 = plane[2 * W * tb + w],
                     b1 = plane[2 * W * tb + W + w];
      const uint32_t ma = ch.x < n ? 0u : mixed[(ch.x - n) * W + w], mb = ch.y < n ? 0u : mixed[(ch.y - n) * W + w];
      const int pa = ch.x < n ? 0 : 4 + ahead[(ch.x - n) * W + w], pb = ch.y < n ? 0 : 4 + ahead[(ch.y - n) * W + w];
      for (; m; m &= m - 1) {
        const int k = __ffs(m) - 1;
        const uint32_t below = (1u << k) - 1u;
        put((ma >> k) & 1u ? pa + __popc(ma & below) : (int)((a0 >> k) & 1u) + 2 * (int)((a1 >> k) & 1u),
            (mb >> k) & 1u ? pb + __popc(mb & below) : (int)((b0 >> k) & 1u) + 2 * (int)((b1 >> k) & 1u));
      }
    }
    if (full)
      for (int k = tid; k < n; k += BS) gtoff[k] = toff[k];
    __syncthreads();
    // read by later launches only (an item is in a launch once)
    if (tid == 0 && (full || tbase > 0)) P.is_valid[R.item] = full;
  }

  const size_t slot_stride = (size_t)nint * S4;
  float4 *part = P.part + R.part_off;
  float4 *partlo = P.partlo ? P.partlo + R.part_off : nullptr;
  int32_t *pexp = P.pexp + R.part_off;
  const int8_t *seq = P.seq + R.seq_off;
  const float pi4[4] = {spi[0].x, spi[1].x, spi[2].x, spi[3].x};
  const ff2 pi2[2] = {ff2_make(f2_pack(spi[0].x, spi[1].x), f2_pack(spi[0].y, spi[1].y)),
                      ff2_make(f2_pack(spi[2].x, spi[3].x), f2_pack(spi[2].y, spi[3].y))};
  // A level's tasks are independent; the threads take them in turn.  Without a
  // list the warps take (node, 32 patterns) in turn: warp w starts at node j0 of
  // the level and chunk c0 and advances by NW chunks (no division in the loop).
  constexpr int NW = BS / 32;
  const int jstep = UNI ? 0 : NW / W, cstep = UNI ? 0 : NW - jstep * W, j0 = UNI ? 0 : (tid >> 5) / W,
            c0 = UNI ? 0 : (tid >> 5) - j0 * W;
  for (int lv = 0; lv < nlev; lv++) {
    const int beg = UNI ? toff[T.lstart[lv]] + tid : tid >> 5,
              end = UNI ? toff[T.lstart[lv + 1]] : (T.lstart[lv + 1] - T.lstart[lv]) * W;
    int jj = j0, chunk = c0;
    for (int q = beg; q < end; q += UNI ? BS : NW) {
      int node, i, ic[2];  // the daughters' entries
      if (UNI) {
        const uint2 t = q >= tbase ? stask[q - tbase] : task[q];
        node = n + (int)(t.x & 0xffffu);
        i = (int)(t.x >> 16);
        ic[0] = (int)(t.y & 0xffffu);
        ic[1] = (int)(t.y >> 16);
      } else {
        node = T.order[T.lstart[lv] + jj];
        i = chunk * 32 + (tid & 31);
        jj += jstep;
        chunk += cstep;
        if (chunk >= W) {
          chunk -= W;
          jj++;
        }
        if (!T.fresh[node] || i >= S) continue;
      }
      const int2 ch = hky_children(T.nd[node], n);
      const int cc[2] = {ch.x, ch.y};
      if (!UNI)
        for (int h = 0; h < 2; h++) ic[h] = cc[h] < n ? seq[(size_t)cc[h] * S + i] : i;
      int e = 0;
      float4 ov, ol = make_float4(0.f, 0.f, 0.f, 0.f);
      if constexpr (FF) {
        ff2 v[2][2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int c = cc[h];
          if (!UNI && c < n) {
            const float4 *col = reinterpret_cast<const float4 *>(Pt + PT * c) + 2 * ic[h];
            const float4 a = col[0], b = col[1];
            v[h][0] = ff2_make(f2_pack(a.x, a.y), f2_pack(a.z, a.w));
            v[h][1] = ff2_make(f2_pack(b.x, b.y), f2_pack(b.z, b.w));
          } else if (c < n) {
            hky_apply_tip_ff(Pm + PB * c, spi[ic[h]], ic[h], v[h]);
          } else {
            const int rs = T.fresh[c] ? 1 - T.slot[c] : T.slot[c];
            const size_t idx = rs * slot_stride + (size_t)(c - n) * S4 + ic[h];
            ff2 L[2];
            ff2_load(part[idx], partlo[idx], L);
            e += pexp[idx];
            hky_apply_ff(Pm + PB * c, pi2, L, v[h]);
          }
        }
        const ff2 o0 = ff2_mul(v[0][0], v[1][0]), o1 = ff2_mul(v[0][1], v[1][1]);
        const float2 h0 = f2_un(o0.hi), h1 = f2_un(o1.hi), l0 = f2_un(o0.lo), l1 = f2_un(o1.lo);
        ov = make_float4(h0.x, h0.y, h1.x, h1.y);
        ol = make_float4(l0.x, l0.y, l1.x, l1.y);
        // normalise by an exact power of two when the largest entry drops
        // below 2^-20: the lo parts (2^-24 below) stay far from subnormal
        const float m = fmaxf(fmaxf(ov.x, ov.y), fmaxf(ov.z, ov.w));
        if (m < 9.5367432e-07f && m > 0.f) {
          const int k = expo_of(m);
          const float sc = pow2f(-k);
          ov = make_float4(ov.x * sc, ov.y * sc, ov.z * sc, ov.w * sc);
          ol = make_float4(ol.x * sc, ol.y * sc, ol.z * sc, ol.w * sc);
          e += k;
        }
      } else {
        float v[2][4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int c = cc[h];
          const float *Kp = Pm + PB * c;
          const HkyCoef K = {Kp[0], Kp[1], Kp[2], Kp[3], Kp[4]};
          if (c < n) {
            hky_apply_tip(K, pi4, ic[h], v[h]);
          } else {
            float4 Lc;
            const int rs = T.fresh[c] ? 1 - T.slot[c] : T.slot[c];
            const size_t idx = rs * slot_stride + (size_t)(c - n) * S4 + ic[h];
            Lc = part[idx];
            e += pexp[idx];
            hky_apply(K, pi4, Lc, v[h]);
          }
        }
        ov = make_float4(v[0][0] * v[1][0], v[0][1] * v[1][1], v[0][2] * v[1][2], v[0][3] * v[1][3]);
        // rescale by an exact 2^40 only when the largest entry drops below
        // 2^-40: products of two daughters then stay above 2^-80 (normal)
        const float m = fmaxf(fmaxf(ov.x, ov.y), fmaxf(ov.z, ov.w));
        if (m < 9.094947e-13f) {
          const float up = 1.0995116e12f;  // 2^40
          ov.x *= up; ov.y *= up; ov.z *= up; ov.w *= up;
          e -= 40;
          if (m * up < 9.094947e-13f) {  // very small value: normalise exactly
            const float mm = m * up;
            const int k = (mm > 0.f) ? expo_of(mm) : 0;
            const float sc = pow2f(-k);
            ov.x *= sc; ov.y *= sc; ov.z *= sc; ov.w *= sc;
            e += k;
          }
        }
      }
      const size_t widx = (1 - T.slot[node]) * slot_stride + (size_t)(node - n) * S4 + i;
      part[widx] = ov;
      if (partlo) partlo[widx] = ol;
      pexp[widx] = e;
    }
    __syncthreads();
  }

  // root: sum_i mult_i * (log(sum_j pi_j L_j) + scale_i)
  const int root = T.order[nint - 1];
  const int rs = T.fresh[root] ? 1 - T.slot[root] : T.slot[root];
  const int32_t *mult = P.mult + R.mult_off;
  double acc = 0.0;
  long long acce = 0;
  for (int i = tid; i < S; i += BS) {
    float4 Lr, Ll = make_float4(0.f, 0.f, 0.f, 0.f);
    int er;
    const size_t idx = rs * slot_stride + (size_t)(root - n) * S4 + i;
    Lr = part[idx];
    if (FF) Ll = partlo[idx];
    er = pexp[idx];
    const int mlt = mult[i];
    if constexpr (FF) {
      ff f = ff_mul(ff_of(spi[0]), ff_make(Lr.x, Ll.x));
      f = ff_fma_pos(ff_of(spi[1]), ff_make(Lr.y, Ll.y), f);
      f = ff_fma_pos(ff_of(spi[2]), ff_make(Lr.z, Ll.z), f);
      f = ff_fma_pos(ff_of(spi[3]), ff_make(Lr.w, Ll.w), f);
      const int k = expo_of(f.hi);
      const float sc = pow2f(-k);
      const ff lg = ff_log(ff_make(f.hi * sc, f.lo * sc), c_ffh);
      acc += (double)mlt * ((double)lg.hi + (double)lg.lo);
      acce += (long long)mlt * (long long)(er + k);
    } else {
      float f = spi[0].x * Lr.x + spi[1].x * Lr.y + spi[2].x * Lr.z + spi[3].x * Lr.w;
      int k = expo_of(f);
      float mant = f * pow2f(-k);
      acc += (double)mlt * (double)logf(mant);
      acce += (long long)mlt * (long long)(er + k);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    acc += __shfl_xor_sync(0xffffffffu, acc, o);
    acce += __shfl_xor_sync(0xffffffffu, acce, o);
  }
  if ((tid & 31) == 0) {
    red_d[tid >> 5] = acc;
    red_e[tid >> 5] = acce;
  }
  // recomputed marks for the commit step
  for (int k = tid; k < nl; k += BS) P.fresh32[R.node_off + k] = (k >= n) ? T.fresh[k] : 0;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    long long se = 0;
    for (int w = 0; w < BS / 32; w++) { s += red_d[w]; se += red_e[w]; }
    result[blockIdx.x] = s + (double)se * LN2;
    P.pdg_new[R.item] = result[blockIdx.x];
    status[blockIdx.x] = IMA_EVAL_OK;
  }
}

// ------------------------------------------------------------------ FP64
__global__ void __launch_bounds__(HKY_BS) k_hky_fp64(Pools P, const ReqDev *reqs,
                                                     double *result, int32_t *status, int maxnl)
{
  extern __shared__ __align__(16) char smem[];
  const ReqDev R = reqs[blockIdx.x];
  const ItemDev it = P.items[R.item];
  const LocusDev L = P.loci[it.locus];
  const int n = it.n, nl = 2 * n - 1, S = L.nsites, nint = n - 1;
  const int nlev = P.nlev[R.item];
  const HkyLayout lay = hky_layout64(maxnl);
  double *Pm = reinterpret_cast<double *>(smem);  // [maxnl][16]
  Tree T;
  T.nd = reinterpret_cast<NodeRec *>(smem + lay.nd);
  T.fresh = reinterpret_cast<uint8_t *>(smem + lay.fresh);
  T.dirty = T.fresh + maxnl;
  T.slot = T.dirty + maxnl;
  T.order = reinterpret_cast<int16_t *>(smem + lay.order);
  __shared__ double red_d[HKY_BS / 32];
  __shared__ double spi[4];
  __shared__ double smu;

  load_tree(P, it, R, nlev, T, P.slot64);
  T.lstart = T.order + nint;
  if (threadIdx.x == 0) {
    const double *pid = P.pi + 4 * (size_t)R.item;
    smu = R.u / ((double)L.totsites * standfactor(pid, R.par));
    for (int j = 0; j < 4; j++) spi[j] = pid[j];
  }
  __syncthreads();
  const double *t64 = P.t64 + it.node_off;
  double kpa = R.par - 1.0;
  for (int c = threadIdx.x; c < nl; c += blockDim.x) {
    int d = T.nd[c].down;
    if (d < 0 || !T.fresh[d]) continue;
    double pil[4] = {spi[0], spi[1], spi[2], spi[3]};
    hky_p<double>(pil, kpa, smu * branch_64(T.nd, t64, c), Pm + 16 * c);
  }
  __syncthreads();

  const size_t slot_stride = (size_t)nint * S;
  double *part = P.part64 + it.part64_off * 4;
  double *psf = P.psf64 + it.part64_off;
  const int8_t *seq = P.seq + L.seq_off;
  for (int lv = 0; lv < nlev; lv++) {
    int beg = T.lstart[lv], cnt = T.lstart[lv + 1] - beg;
    for (int w = threadIdx.x; w < cnt * S; w += blockDim.x) {
      int node = T.order[beg + w / S];
      int i = w - (w / S) * S;
      if (!T.fresh[node]) continue;
      double v[2][4];
      double sf = 0.0;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        int c = h ? T.nd[node].up1 : T.nd[node].up0;
        const double *Pc = Pm + 16 * c;
        if (c < n) {
          int s = seq[(size_t)c * S + i];
#pragma unroll
          for (int j = 0; j < 4; j++) v[h][j] = Pc[j * 4 + s];
        } else {
          int rs = T.fresh[c] ? 1 - T.slot[c] : T.slot[c];
          size_t idx = rs * slot_stride + (size_t)(c - n) * S + i;
          const double2 *Lp = reinterpret_cast<const double2 *>(part + 4 * idx);
          double2 a = Lp[0], b = Lp[1];
          sf += psf[idx];
#pragma unroll
          for (int j = 0; j < 4; j++)
            v[h][j] = Pc[j * 4 + 0] * a.x + Pc[j * 4 + 1] * a.y + Pc[j * 4 + 2] * b.x +
                      Pc[j * 4 + 3] * b.y;
        }
      }
      double o[4];
      double m = 0.0;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        o[j] = v[0][j] * v[1][j];
        if (o[j] > m) m = o[j];
      }
      size_t widx = (1 - T.slot[node]) * slot_stride + (size_t)(node - n) * S + i;
      double2 *W = reinterpret_cast<double2 *>(part + 4 * widx);
      W[0] = make_double2(o[0] / m, o[1] / m);
      W[1] = make_double2(o[2] / m, o[3] / m);
      psf[widx] = sf + log(m);
    }
    __syncthreads();
  }

  int root = T.order[nint - 1];
  int rs = T.fresh[root] ? 1 - T.slot[root] : T.slot[root];
  const int32_t *mult = P.mult + L.mult_off;
  double acc = 0.0;
  for (int i = threadIdx.x; i < S; i += blockDim.x) {
    size_t idx = rs * slot_stride + (size_t)(root - n) * S + i;
    const double2 *Lp = reinterpret_cast<const double2 *>(part + 4 * idx);
    double2 a = Lp[0], b = Lp[1];
    double f = spi[0] * a.x + spi[1] * a.y + spi[2] * b.x + spi[3] * b.y;
    acc += mult[i] * (log(f) + psf[idx]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red_d[threadIdx.x >> 5] = acc;
  for (int k = threadIdx.x; k < nl; k += blockDim.x)
    P.fresh64[it.node_off + k] = (k >= n) ? T.fresh[k] : 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < HKY_BS / 32; w++) s += red_d[w];
    result[blockIdx.x] = s;
    P.pdg_new[R.item] = s;
    status[blockIdx.x] = IMA_EVAL_OK;
  }
}

// accept: recomputed nodes' new slot becomes the committed one; reject: the
// committed slot stays.  Either way the recomputed marks are cleared, so a
// repeated accept is a no-op as the reference's repeated copy is.
__global__ void k_hky_commit(Pools P, const int32_t *items, const uint8_t *accept)
{
  const ItemDev it = P.items[items[blockIdx.x]];
  const bool acc = accept[blockIdx.x] != 0;
  const int nl = 2 * it.n - 1;
  for (int k = threadIdx.x; k < nl; k += blockDim.x) {
    size_t g = (size_t)it.node_off + k;
    if (P.fresh32[g]) {
      if (acc) P.slot32[g] ^= 1;
      P.fresh32[g] = 0;
    }
    if (P.slot64 && P.fresh64[g]) {
      if (acc) P.slot64[g] ^= 1;
      P.fresh64[g] = 0;
    }
  }
}

}  // namespace

constexpr size_t HKY_TASK_CAP = 640, HKY_PLANE_CAP = 1024;  // tasks and words kept in shared memory
constexpr int HKY_FEW = 4 * 152;
constexpr size_t HKY_FEW_SMEM = 56 * 1024;  // so that four CTAs fit an SM

template <bool UNI, bool FF, int BS, int MINB>
static void hky_fast_launch(const Pools &P, const ReqDev *reqs, int nreq, int maxnl, int maxS, double *result,
                            int32_t *status, cudaStream_t st)
{
  const size_t maxn = (size_t)(maxnl + 1) / 2, W = ((size_t)maxS + 31) / 32;
  const size_t mcap = UNI ? std::min((size_t)HKY_MASK_WORDS, (maxn - 1) * W) : 0;
  const size_t tcap = UNI ? std::min(HKY_TASK_CAP, (maxn - 1) * (maxS + 4)) : 0;
  const size_t base = hky_layout_fast(maxnl, UNI, FF).total + 4 * mcap + 2 * ((mcap + 1) & ~size_t(1)) + tcap * sizeof(uint2);
  // few CTAs take all of the tips' planes, which one warp reads for the masks
  const size_t planes = UNI ? 2 * maxn * W : 0;
  const size_t pcap = nreq <= HKY_FEW && base + 4 * planes <= HKY_FEW_SMEM ? planes : std::min(HKY_PLANE_CAP, planes);
  const size_t sm = base + 4 * pcap;
  if (sm > 40 * 1024)  // (48 KB with the static part)
    cudaFuncSetAttribute(k_hky_fast<UNI, FF, BS, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX - 1024);
  k_hky_fast<UNI, FF, BS, MINB><<<nreq, BS, sm, st>>>(P, reqs, result, status, maxnl, (int)mcap, (int)pcap, (int)tcap);
}

template <bool FF, int BS, int MINB>
static void hky_fast_bs(const Pools &P, const ReqDev *reqs, int nreq, int maxnl, int maxS, bool uni, double *result,
                        int32_t *status, cudaStream_t st)
{
  if (uni) hky_fast_launch<true, FF, BS, MINB>(P, reqs, nreq, maxnl, maxS, result, status, st);
  else hky_fast_launch<false, FF, BS, MINB>(P, reqs, nreq, maxnl, maxS, result, status, st);
}

// One entry per state pays where the tips below a node often agree.  Where
// few pairs of tips do, the list's loads and the mixed daughters of a warp
// cost more than the entries save: with 44% of the pairs alike 1,280
// chain-loci of 100 genes x 300 patterns take 389 us either way and 12,800 of
// 96 x 80 836 and 806, with 25% (unrelated sequences) 433 and 374, 927 and 804;
// with 57% 345 and 374, 757 and 804.  That is of states drawn tip by tip; along a
// genealogy equal states lie together, and simulated sequences have 64-94%.
constexpr double HKY_AGREE = 0.4;

bool hky_uniform_entries(int n, int S, const int8_t *seq)
{
  if ((long long)(n - 1) * ((S + 31) / 32) > HKY_MASK_WORDS || S > 65531 || n > 32768) return false;
  // pairs of tips with the same state, over the patterns
  std::vector<int> f(4 * (size_t)S, 0);
  for (int t = 0; t < n; t++)
    for (int k = 0; k < S; k++) f[4 * (size_t)k + seq[(size_t)t * S + k]]++;
  double same = 0.0;
  for (int v : f) same += (double)v * (v - 1);
  return same >= HKY_AGREE * S * (double)n * (n - 1);
}

void launch_hky_fast(const Pools &P, const ReqDev *reqs, int nreq, int maxn, int maxS, bool uni, int variant,
                     double *result, int32_t *status, cudaStream_t st)
{
  if (nreq <= 0) return;
  const int maxnl = 2 * maxn - 1;
  switch (variant) {
    case 1: hky_fast_bs<true, 64, 16>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
    case 2: hky_fast_bs<true, 256, 4>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
    case 3: hky_fast_bs<true, 128, 10>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
    case 4: hky_fast_bs<true, 128, 8>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
    case 5: hky_fast_bs<true, 96, 11>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
    default: hky_fast_bs<true, 128, 6>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
  }
}

void launch_hky_fp32(const Pools &P, const ReqDev *reqs, int nreq, int maxn, int maxS, bool uni, int variant,
                     double *result, int32_t *status, cudaStream_t st)
{
  if (nreq <= 0) return;
  const int maxnl = 2 * maxn - 1;
  switch (variant) {
    case 1: hky_fast_bs<false, 64, 24>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
    case 2: hky_fast_bs<false, 256, 6>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
    case 3: hky_fast_bs<false, 128, 6>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
    case 4: hky_fast_bs<false, 128, 8>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
    case 5: hky_fast_bs<false, 96, 16>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
    default: hky_fast_bs<false, 128, 12>(P, reqs, nreq, maxnl, maxS, uni, result, status, st); break;
  }
}

// ln 2 and the log table of the float-float root sum (once per device)
int hky_init_tables()
{
  FFConsts K{};
  for (int i = 0; i < 64; i++) {
    const double v = std::log(1.0 + (2.0 * i + 1.0) / 128.0);
    K.logtab[i] = make_float2((float)v, (float)(v - (double)(float)v));
  }
  const double ln2 = 0.69314718055994530941723212146;
  const double a = 355.0 / 512.0;
  K.ln2a = make_float2((float)a, (float)(ln2 - a));
  K.ln2b = (float)(ln2 - a - (double)(float)(ln2 - a));
  float2 t[64];
  for (int j = 0; j < 64; j++) {
    const double v = std::expm1((j - 32) * (0.69314718055994530942 / 64));
    t[j] = make_float2((float)v, (float)(v - (double)(float)v));
  }
  return cudaMemcpyToSymbol(c_ffh, &K, sizeof(K)) == cudaSuccess &&
                 cudaMemcpyToSymbol(d_exp64m1, t, sizeof(t)) == cudaSuccess
             ? 0
             : -1;
}

void launch_hky_fp64(const Pools &P, const ReqDev *reqs, int nreq, int maxn, double *result,
                     int32_t *status, cudaStream_t st)
{
  if (nreq <= 0) return;
  size_t sm = hky_layout64(2 * maxn - 1).total;
  if (sm > 48 * 1024)
    cudaFuncSetAttribute(k_hky_fp64, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX - 128);
  k_hky_fp64<<<nreq, HKY_BS, sm, st>>>(P, reqs, result, status, 2 * maxn - 1);
}

void launch_hky_commit(const Pools &P, const int32_t *items, const uint8_t *accept, int n,
                       cudaStream_t st)
{
  if (n <= 0) return;
  k_hky_commit<<<n, 128, 0, st>>>(P, items, accept);
}
