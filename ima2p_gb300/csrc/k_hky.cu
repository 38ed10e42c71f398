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
// instructions (ff_exp_expm1's four doublings take 110); relative errors
// within 3e-14 of e^x - 1 and of e^x.
constexpr float L64_A = 0.01082611083984375f;     // ln 2 / 64 = A + B + C: k A and k B exact for |k| < 2^13
constexpr float L64_B = 4.3101608753204346e-06f;
constexpr float L64_C = 3.695530104153022e-09f;
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

struct HkyCoefFF {
  ff a, bR, bY, dR, dY;
};
__device__ __forceinline__ HkyCoefFF load_coef_ff(const float *Kp)  // 16-byte aligned
{
  const float4 a = reinterpret_cast<const float4 *>(Kp)[0], b = reinterpret_cast<const float4 *>(Kp)[1];
  const float2 c = reinterpret_cast<const float2 *>(Kp)[4];
  HkyCoefFF K;
  K.a = ff_make(a.x, a.y);
  K.bR = ff_make(a.z, a.w);
  K.bY = ff_make(b.x, b.y);
  K.dR = ff_make(b.z, b.w);
  K.dY = ff_make(c.x, c.y);
  return K;
}
// P(b) applied to a tip observed in state st: column st of P(b)
__device__ __forceinline__ void hky_apply_tip_ff(const HkyCoefFF &K, const ff *pi, int st, ff *v)
{
  const ff p = st == 0 ? pi[0] : st == 1 ? pi[1] : st == 2 ? pi[2] : pi[3];
  const bool isR = (st & 1) == 0;
  const ff tR = ff_mul(isR ? K.bR : K.a, p), tY = ff_mul(isR ? K.a : K.bY, p);
  const ff own = ff_add(isR ? tR : tY, isR ? K.dR : K.dY);  // the observed state's entry
  v[0] = st == 0 ? own : tR;
  v[2] = st == 2 ? own : tR;
  v[1] = st == 1 ? own : tY;
  v[3] = st == 3 ? own : tY;
}
// The same steps leaving the pair unnormalised (|lo| may reach a few
// ulp(hi)), for intermediate values: the next step's TwoSum is exact
// whatever lo is, so only the values that leave the apply are renormalised.
__device__ __forceinline__ ff ff_mul_u(ff a, ff b)
{
  const float p = __fmul_rn(a.hi, b.hi);
  return ff_make(p, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.hi, -p))));
}
__device__ __forceinline__ ff ff_fma_pos_u(ff a, ff b, ff c)
{
  const float p = __fmul_rn(a.hi, b.hi);
  const float pe = __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.hi, -p)));
  const ff s = two_sum(p, c.hi);
  return ff_make(s.hi, __fadd_rn(s.lo, __fadd_rn(pe, c.lo)));
}

// v_j = E1 S_o + b_c S_c + d_c L_j, left unnormalised too: its only use is
// the product of the two daughters, whose ff_mul renormalises
__device__ __forceinline__ void hky_apply_ff(const HkyCoefFF &K, const ff *pi, const ff *L, ff *v)
{
  const ff SR = ff_fma_pos_u(pi[2], L[2], ff_mul_u(pi[0], L[0]));
  const ff SY = ff_fma_pos_u(pi[3], L[3], ff_mul_u(pi[1], L[1]));
  const ff tR = ff_fma_pos_u(K.bR, SR, ff_mul_u(K.a, SY));
  const ff tY = ff_fma_pos_u(K.bY, SY, ff_mul_u(K.a, SR));
  v[0] = ff_fma_pos_u(K.dR, L[0], tR);
  v[2] = ff_fma_pos_u(K.dR, L[2], tR);
  v[1] = ff_fma_pos_u(K.dY, L[1], tY);
  v[3] = ff_fma_pos_u(K.dY, L[3], tY);
}

__device__ __forceinline__ ff ff_of(float2 v) { return ff_make(v.x, v.y); }

// Shared-memory carve-up, identical on host (sizing) and device.
// tip, inner: bytes of one branch's coefficients below a tip and below an
// internal node; times: bytes of one node's time.
struct HkyLayout {
  size_t inner, nd, times, fresh, order, lev, total;
};
__host__ __device__ inline HkyLayout hky_layout(int maxnl, size_t tip, size_t inner, size_t time)
{
  const size_t maxn = (size_t)(maxnl + 1) / 2;
  HkyLayout l;
  l.inner = tip * maxn;
  l.nd = l.inner + inner * maxn;
  l.times = l.nd + sizeof(NodeRec) * (size_t)maxnl;
  l.fresh = l.times + time * (size_t)maxnl;
  l.order = (l.fresh + 3 * (size_t)maxnl + 15) & ~size_t(15);
  l.lev = (l.order + sizeof(int16_t) * (size_t)(maxnl + 3) + 15) & ~size_t(15);
  l.total = (l.lev + sizeof(int32_t) * (size_t)(maxnl / 2 + 2) + 15) & ~size_t(15);
  return l;
}
__host__ __device__ inline HkyLayout hky_layout64(int maxnl)  // k_hky_fp64: a 4 x 4 matrix per branch
{
  return hky_layout(maxnl, 16 * sizeof(double), 16 * sizeof(double), 0);
}
// k_hky_fast, in floats: a tip branch's 32 are padded so that lanes on
// different branches of a level start in different banks
__host__ __device__ constexpr int hky_tip_floats(bool ff) { return ff ? 36 : 8; }
__host__ __device__ constexpr int hky_inner_floats(bool ff) { return ff ? 12 : 8; }
__host__ __device__ inline HkyLayout hky_layout_fast(int maxnl, bool ff)
{
  return hky_layout(maxnl, 4 * hky_tip_floats(ff), 4 * hky_inner_floats(ff), sizeof(float2));
}

// ----------------------------------------------------- pattern classes
// Below a node, site patterns that agree on its tips have the same partial.
// A node's classes are numbered in the order of their first patterns, which
// depends only on the tips below it, so that a clean node's stored partials
// (one per class, at the class's number) stay addressable whatever happens
// above.  k_hky_classes lists, per level, one task per class of each node: x =
// (node - n) | class << 16, y = the index of either daughter's value (a tip's
// state, or the class in the daughter), the internal daughter first.  The
// root keeps every pattern, for the sum.  On sequences simulated on their
// genealogies 8-20% of the (node, pattern) pairs remain, on random ones 30-40%.
// Loci of more than CLS_MAXS patterns keep every pattern (CLS_MAXS bounds a
// warp's hash table).
constexpr int CLS_MAXS = 2048;
constexpr int CLS_WARPS = 8;
constexpr size_t CLS_SHARED = 32 * 1024;  // class numbers of all nodes and patterns kept in shared memory up to this
constexpr uint32_t CLS_EMPTY = 0xffffffffu;

__device__ __forceinline__ int2 hky_children(const NodeRec &nd, int n)
{
  return nd.up0 < n && nd.up1 >= n ? make_int2(nd.up1, nd.up0) : make_int2(nd.up0, nd.up1);
}

__global__ void __launch_bounds__(32 * CLS_WARPS) k_hky_classes(Pools P, const ReqDev *reqs, int maxnl, int logh, int cap)
{
  extern __shared__ __align__(16) char smem[];
  const ReqDev R = reqs[blockIdx.x];
  const int n = R.n, nl = 2 * n - 1, S = R.nsites, nint = n - 1;
  if (S > CLS_MAXS || P.is_valid[R.item]) return;
  const int H = 1 << logh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  NodeRec *nd = reinterpret_cast<NodeRec *>(smem);
  int16_t *order = reinterpret_cast<int16_t *>(nd + maxnl);
  uint32_t *keys = reinterpret_cast<uint32_t *>(smem + ((sizeof(NodeRec) * maxnl + 2 * (maxnl + 3) + 15) & ~size_t(15))) +
                   (size_t)warp * (H + H / 2);
  uint16_t *vals = reinterpret_cast<uint16_t *>(keys + H);
  __shared__ int count;  // tasks listed so far
  for (int k = threadIdx.x; k < nl; k += 32 * CLS_WARPS) nd[k] = P.nodes[R.node_off + k];
  for (int k = threadIdx.x; k < 2 * n; k += 32 * CLS_WARPS) order[k] = P.sched[R.sched_off + k];
  if (threadIdx.x == 0) count = 0;
  const int nlev = P.nlev[R.item];
  const int16_t *lstart = order + nint;
  const int8_t *seq = P.seq + R.seq_off;
  // the classes of every node and pattern, read back by the parents
  uint16_t *rep = nint * S <= cap ? reinterpret_cast<uint16_t *>(keys + (size_t)(CLS_WARPS - warp) * (H + H / 2))
                                  : P.crep + R.part_off / 2;
  uint2 *task = P.ctask + R.part_off / 2;
  int32_t *clev = P.clev + R.sched_off;
  __syncthreads();
  for (int lv = 0; lv < nlev; lv++) {
    if (threadIdx.x == 0) clev[lv] = count;
    __syncthreads();
    const int cnt = lstart[lv + 1] - lstart[lv];
    for (int j = warp; j < cnt; j += CLS_WARPS) {
      const int node = order[lstart[lv] + j];
      const int2 c = hky_children(nd[node], n);
      const bool root = nd[node].down < 0;  // its patterns are summed one by one
      if (!root)
        for (int h = lane; h < H; h += 32) keys[h] = CLS_EMPTY;
      __syncwarp();
      int ncls = 0;  // classes so far
      for (int p0 = 0; p0 < S; p0 += 32) {
        const int p = p0 + lane;
        const bool in = p < S;
        uint32_t ia = 0, ib = 0;
        if (in) {
          ia = c.x < n ? (uint32_t)seq[(size_t)c.x * S + p] : rep[(size_t)(c.x - n) * S + p];
          ib = c.y < n ? (uint32_t)seq[(size_t)c.y * S + p] : rep[(size_t)(c.y - n) * S + p];
        }
        const uint32_t key = ia | ib << 16;
        bool first = in;
        unsigned f;
        int r = p;
        if (root) {
          f = __ballot_sync(0xffffffffu, in);
        } else {
          const unsigned m = __match_any_sync(0xffffffffu, in ? key : CLS_EMPTY);
          const int lead = __ffs(m) - 1;
          first = false;
          uint32_t h = 0;
          if (in && lane == lead) {
            // one lane per distinct key of these 32: find it or claim a slot
            for (h = (key * 2654435761u) >> (32 - logh);; h = (h + 1) & (H - 1)) {
              const uint32_t old = atomicCAS(&keys[h], CLS_EMPTY, key);
              if (old == CLS_EMPTY) first = true;
              else if (old == key) r = vals[h];
              else continue;
              break;
            }
          }
          f = __ballot_sync(0xffffffffu, first);
          if (first) {
            r = ncls + __popc(f & ((1u << lane) - 1u));
            vals[h] = (uint16_t)r;
          }
          ncls += __popc(f);
          __syncwarp();
          r = __shfl_sync(0xffffffffu, r, lead);
          if (in) rep[(size_t)(node - n) * S + p] = (uint16_t)r;
        }
        int base = 0;
        if (lane == 0) base = atomicAdd(&count, __popc(f));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (first) task[base + __popc(f & ((1u << lane) - 1u))] = make_uint2((uint32_t)(node - n) | (uint32_t)r << 16, key);
      }
    }
    __syncthreads();  // the level's classes before its parents
  }
  if (threadIdx.x == 0) {
    clev[nlev] = count;
    P.is_valid[R.item] = 1;
  }
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
// the five coefficients of hky_coef_fast (in place of a 4 x 4 matrix), and a
// warp works on one node and 32 of its patterns at a time, so the children's
// coefficients are warp-uniform and no warp mixes tip and internal children.
// With CACHE, the partials this launch computes are also kept in shared
// memory ([internal node][pattern]) and daughters are read from there instead
// of making an L2 round trip per level.  BS threads per CTA, registers for
// MINB resident CTAs per SM.  FF: every value a float-float pair (the lo
// parts of the partials in P.partlo); otherwise FP32 (which clears the lo
// parts of what it writes when they exist, so a later FF evaluation reads
// its partials as exact pairs).
template <bool FF, bool CACHE, int BS, int MINB>
__global__ void __launch_bounds__(BS, MINB) k_hky_fast(Pools P, const ReqDev *reqs,
                                                     double *result, int32_t *status, int maxnl,
                                                     int cache_S, int task_cap)
{
  extern __shared__ __align__(16) char smem[];
  // the request carries the item's offsets and sizes, so the tree loads
  // below wait on this one load only
  const ReqDev R = reqs[blockIdx.x];
  const int n = R.n, nl = 2 * n - 1, S = R.nsites, nint = n - 1;
  // per branch 5 coefficients (FF: pairs); FF tip branches hold instead the
  // columns of P(b) for the four observed states, [4][4] pairs, so a tip
  // daughter costs two loads
  constexpr int PT = hky_tip_floats(FF), PI = hky_inner_floats(FF);
  const HkyLayout lay = hky_layout_fast(maxnl, FF);
  float *Pt = reinterpret_cast<float *>(smem);                       // [tip][PT]
  float *Pi = reinterpret_cast<float *>(smem + lay.inner) - n * PI;  // [internal node][PI]
  float2 *stm = reinterpret_cast<float2 *>(smem + lay.times);        // node times
  Tree T;
  T.nd = reinterpret_cast<NodeRec *>(smem + lay.nd);
  T.fresh = reinterpret_cast<uint8_t *>(smem + lay.fresh);
  T.dirty = T.fresh + maxnl;
  T.slot = T.dirty + maxnl;
  T.order = reinterpret_cast<int16_t *>(smem + lay.order);
  int32_t *lev = reinterpret_cast<int32_t *>(smem + lay.lev);
  // the first task_cap tasks staged in shared memory
  uint2 *stask = reinterpret_cast<uint2 *>(smem + lay.total);
  float4 *cpart = reinterpret_cast<float4 *>(stask + task_cap);         // [nint][cache_S]
  float4 *cpartlo = cpart + (FF ? (size_t)(maxnl / 2) * cache_S : 0);   // FF: lo parts
  int32_t *cexp = reinterpret_cast<int32_t *>(cpartlo + (size_t)(maxnl / 2) * cache_S);
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
  const bool cls = S <= CLS_MAXS;
  const uint2 *task = P.ctask + R.part_off / 2;
  const int staged = cls ? (int)min((long long)task_cap, (long long)nint * S) : 0;
  for (int k = tid; k < staged; k += BS) stask[k] = task[k];
  if (cls)
    for (int k = tid; k < n; k += BS) lev[k] = P.clev[R.sched_off + k];  // nlev + 1 <= n of them are meant
  if (tid == 0) {
    // mu = u / (totsites standfactor): 2 kappa (pA pG + pC pT) + 2 (pA + pG)
    // (pC + pT), in float-float (in FP64 one thread's fifty operations held up
    // the CTA for some 3,000 cycles)
    const double *pid = P.pi + 4 * (size_t)R.item;
    ff pj[4];
    for (int j = 0; j < 4; j++) {
      pj[j] = ff_split(pid[j]);
      spi[j] = make_float2(pj[j].hi, pj[j].lo);
    }
    const ff kap = ff_split(R.par);
    ff sf = ff_mul(kap, ff_add(ff_mul(pj[0], pj[2]), ff_mul(pj[1], pj[3])));
    sf = ff_add(sf, ff_mul(ff_add(pj[0], pj[2]), ff_add(pj[1], pj[3])));
    const ff mu = ff_div(ff_split(R.u), ff_mul(ff_make(2.f * sf.hi, 2.f * sf.lo), ff_split((double)R.totsites)));
    smu = make_float2(mu.hi, mu.lo);
  } else if (tid == 32) {
    const double *pid = P.pi + 4 * (size_t)R.item;
    const ff PR = ff_add(ff_split(pid[0]), ff_split(pid[2])), PY = ff_add(ff_split(pid[1]), ff_split(pid[3]));
    const ff kp = ff_add_f(ff_split(R.par), -1.0f), one = ff_from(1.0f);
    auto put = [](ff v) { return make_float2(v.hi, v.lo); };
    skpa = put(kp);
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
  if (!full && tid == 0) {  // the reference's propagation rule, bottom-up
    for (int q = 0; q < 4; q++)
      if (R.e[q] >= 0 && R.e[q] < nl) T.dirty[R.e[q]] = 1;
    for (int k = 0; k < nint; k++) {
      int node = T.order[k];
      int a = T.nd[node].up0, b = T.nd[node].up1;
      T.fresh[node] = (T.dirty[node] || T.dirty[a] || T.dirty[b] || (a >= n && T.fresh[a]) ||
                       (b >= n && T.fresh[b])) ? 1 : 0;
    }
  }
  if (!full) __syncthreads();
  for (int c = tid; c < nl; c += BS) {
    int d = T.nd[c].down;
    if (d < 0 || !T.fresh[d]) continue;
    if constexpr (FF) {
      const ff pif[4] = {ff_of(spi[0]), ff_of(spi[1]), ff_of(spi[2]), ff_of(spi[3])};
      const int u = T.nd[c].up0;
      const ff tc = ff_of(stm[c]);
      const ff br = (u < 0) ? tc : ff_sub(tc, ff_of(stm[u]));
      float Kc[10];
      hky_coef_ff(sH, stab, ff_mul(ff_of(smu), br), Kc);
      float *dst = c < n ? Pt + PT * c : Pi + PI * c;
      if (c < n) {
        const HkyCoefFF K = {ff_make(Kc[0], Kc[1]), ff_make(Kc[2], Kc[3]), ff_make(Kc[4], Kc[5]), ff_make(Kc[6], Kc[7]),
                             ff_make(Kc[8], Kc[9])};
#pragma unroll
        for (int st = 0; st < 4; st++) {
          ff v[4];
          hky_apply_tip_ff(K, pif, st, v);
#pragma unroll
          for (int j = 0; j < 4; j++) reinterpret_cast<float2 *>(dst)[4 * st + j] = make_float2(v[j].hi, v[j].lo);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 10; j++) dst[j] = Kc[j];
      }
    } else {
      float pil[4] = {spi[0].x, spi[1].x, spi[2].x, spi[3].x};
      hky_coef_fast(pil, skpa.x, smu.x * branch_ff(T.nd, stm, c), c < n ? Pt + PT * c : Pi + PI * c);
    }
  }
  __syncthreads();

  const size_t slot_stride = (size_t)nint * S;
  float4 *part = P.part + R.part_off;
  float4 *partlo = P.partlo ? P.partlo + R.part_off : nullptr;
  int32_t *pexp = P.pexp + R.part_off;
  const int8_t *seq = P.seq + R.seq_off;
  const float pi4[4] = {spi[0].x, spi[1].x, spi[2].x, spi[3].x};
  // a level's tasks (one per node and class, or per node and pattern) are
  // independent; the threads take them in turn
  for (int lv = 0; lv < nlev; lv++) {
    const int beg = cls ? lev[lv] : 0, end = cls ? lev[lv + 1] : (T.lstart[lv + 1] - T.lstart[lv]) * S;
    for (int q = beg + tid; q < end; q += BS) {
      int node, i, ic[2];
      if (cls) {
        const uint2 t = q < staged ? stask[q] : task[q];
        node = n + (int)(t.x & 0xffffu);
        i = (int)(t.x >> 16);
        ic[0] = (int)(t.y & 0xffffu);
        ic[1] = (int)(t.y >> 16);
      } else {
        node = T.order[T.lstart[lv] + q / S];
        i = q % S;
      }
      if (!T.fresh[node]) continue;
      const int2 ch = hky_children(T.nd[node], n);
      const int cc[2] = {ch.x, ch.y};
      if (!cls)
        for (int h = 0; h < 2; h++) ic[h] = cc[h] < n ? seq[(size_t)cc[h] * S + i] : i;
      int e = 0;
      float4 ov, ol = make_float4(0.f, 0.f, 0.f, 0.f);
      if constexpr (FF) {
        const ff pif[4] = {ff_of(spi[0]), ff_of(spi[1]), ff_of(spi[2]), ff_of(spi[3])};
        ff v[2][4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int c = cc[h];
          if (c < n) {
            const float4 *col = reinterpret_cast<const float4 *>(Pt + PT * c) + 2 * ic[h];
            const float4 a = col[0], b = col[1];
            v[h][0] = ff_make(a.x, a.y);
            v[h][1] = ff_make(a.z, a.w);
            v[h][2] = ff_make(b.x, b.y);
            v[h][3] = ff_make(b.z, b.w);
          } else {
            const HkyCoefFF K = load_coef_ff(Pi + PI * c);
            float4 hi, lo;
            if (CACHE && T.fresh[c]) {
              const size_t ci = (size_t)(c - n) * cache_S + ic[h];
              hi = cpart[ci];
              lo = cpartlo[ci];
              e += cexp[ci];
            } else {
              const int rs = T.fresh[c] ? 1 - T.slot[c] : T.slot[c];
              const size_t idx = rs * slot_stride + (size_t)(c - n) * S + ic[h];
              hi = part[idx];
              lo = partlo[idx];
              e += pexp[idx];
            }
            const ff Lc[4] = {ff_make(hi.x, lo.x), ff_make(hi.y, lo.y), ff_make(hi.z, lo.z), ff_make(hi.w, lo.w)};
            hky_apply_ff(K, pif, Lc, v[h]);
          }
        }
        ff o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) o[j] = ff_mul(v[0][j], v[1][j]);
        // normalise by an exact power of two when the largest entry drops
        // below 2^-20: the lo parts (2^-24 below) stay far from subnormal
        const float m = fmaxf(fmaxf(o[0].hi, o[1].hi), fmaxf(o[2].hi, o[3].hi));
        if (m < 9.5367432e-07f && m > 0.f) {
          const int k = expo_of(m);
          const float sc = pow2f(-k);
#pragma unroll
          for (int j = 0; j < 4; j++) o[j] = ff_make(o[j].hi * sc, o[j].lo * sc);
          e += k;
        }
        ov = make_float4(o[0].hi, o[1].hi, o[2].hi, o[3].hi);
        ol = make_float4(o[0].lo, o[1].lo, o[2].lo, o[3].lo);
      } else {
        float v[2][4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int c = cc[h];
          const float *Kp = c < n ? Pt + PT * c : Pi + PI * c;
          const HkyCoef K = {Kp[0], Kp[1], Kp[2], Kp[3], Kp[4]};
          if (c < n) {
            hky_apply_tip(K, pi4, ic[h], v[h]);
          } else {
            float4 Lc;
            if (CACHE && T.fresh[c]) {
              const size_t ci = (size_t)(c - n) * cache_S + ic[h];
              Lc = cpart[ci];
              e += cexp[ci];
            } else {
              const int rs = T.fresh[c] ? 1 - T.slot[c] : T.slot[c];
              const size_t idx = rs * slot_stride + (size_t)(c - n) * S + ic[h];
              Lc = part[idx];
              e += pexp[idx];
            }
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
      const size_t widx = (1 - T.slot[node]) * slot_stride + (size_t)(node - n) * S + i;
      part[widx] = ov;
      if (partlo) partlo[widx] = ol;
      pexp[widx] = e;
      if (CACHE) {
        const size_t ci = (size_t)(node - n) * cache_S + i;
        cpart[ci] = ov;
        if (FF) cpartlo[ci] = ol;
        cexp[ci] = e;
      }
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
    if (CACHE && T.fresh[root]) {
      size_t ci = (size_t)(root - n) * cache_S + i;
      Lr = cpart[ci];
      if (FF) Ll = cpartlo[ci];
      er = cexp[ci];
    } else {
      size_t idx = rs * slot_stride + (size_t)(root - n) * S + i;
      Lr = part[idx];
      if (FF) Ll = partlo[idx];
      er = pexp[idx];
    }
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

// Partials stay in shared memory when the largest chain-locus of the batch
// fits in this budget (keeps >= 3 CTAs per SM).
constexpr size_t HKY_CACHE_BUDGET = 64 * 1024;
constexpr int HKY_TASK_CAP = 768;  // tasks staged in shared memory (6 KB)

template <bool FF, int BS, int MINB>
static void hky_fast_bs(const Pools &P, const ReqDev *reqs, int nreq, int maxnl, int maxS, bool cache_ok,
                        double *result, int32_t *status, cudaStream_t st)
{
  const size_t maxn = (size_t)(maxnl + 1) / 2;
  const int task_cap = (int)std::min((size_t)HKY_TASK_CAP, (maxn - 1) * maxS + 1) & ~1;
  const size_t base = hky_layout_fast(maxnl, FF).total + task_cap * sizeof(uint2);
  size_t cache = (size_t)(maxnl / 2) * maxS * ((FF ? 2 : 1) * sizeof(float4) + sizeof(int32_t));
  if (cache_ok && cache <= HKY_CACHE_BUDGET) {
    size_t sm = base + cache;
    if (sm > 48 * 1024)
      cudaFuncSetAttribute(k_hky_fast<FF, true, BS, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_hky_fast<FF, true, BS, MINB><<<nreq, BS, sm, st>>>(P, reqs, result, status, maxnl, maxS, task_cap);
  } else {
    if (base > 48 * 1024)
      cudaFuncSetAttribute(k_hky_fast<FF, false, BS, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)base);
    k_hky_fast<FF, false, BS, MINB><<<nreq, BS, base, st>>>(P, reqs, result, status, maxnl, 0, task_cap);
  }
}

void launch_hky_classes(const Pools &P, const ReqDev *reqs, int nreq, int maxn, int maxS, cudaStream_t st)
{
  if (nreq <= 0) return;
  const int maxnl = 2 * maxn - 1, S = std::min(maxS, CLS_MAXS);
  int logh = 6;
  while ((1 << logh) < 2 * S) logh++;
  const size_t hash = ((sizeof(NodeRec) * maxnl + 2 * (maxnl + 3) + 15) & ~size_t(15)) + CLS_WARPS * 6ul * (1ul << logh);
  size_t sm = hash;
  const size_t all = 2ul * (maxn - 1) * S;
  if (all <= CLS_SHARED) sm += all;
  if (sm > 48 * 1024) cudaFuncSetAttribute(k_hky_classes, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_hky_classes<<<nreq, 32 * CLS_WARPS, sm, st>>>(P, reqs, maxnl, logh, all <= CLS_SHARED ? (int)(all / 2) : 0);
}

void launch_hky_fast(const Pools &P, const ReqDev *reqs, int nreq, int maxn, int maxS, int variant,
                     double *result, int32_t *status, cudaStream_t st)
{
  if (nreq <= 0) return;
  const int maxnl = 2 * maxn - 1;
  switch (variant) {
    case 1: hky_fast_bs<true, 64, 16>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
    case 2: hky_fast_bs<true, 256, 4>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
    case 3: hky_fast_bs<true, 128, 10>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
    case 4: hky_fast_bs<true, 128, 6>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
    case 5: hky_fast_bs<true, 96, 11>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
    default: hky_fast_bs<true, 128, 8>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
  }
}

void launch_hky_fp32(const Pools &P, const ReqDev *reqs, int nreq, int maxn, int maxS, int variant,
                     double *result, int32_t *status, cudaStream_t st)
{
  if (nreq <= 0) return;
  const int maxnl = 2 * maxn - 1;
  switch (variant) {
    case 1: hky_fast_bs<false, 64, 24>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
    case 2: hky_fast_bs<false, 256, 6>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
    case 3: hky_fast_bs<false, 128, 12>(P, reqs, nreq, maxnl, maxS, false, result, status, st); break;
    case 4: hky_fast_bs<false, 128, 8>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
    case 5: hky_fast_bs<false, 96, 16>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
    default: hky_fast_bs<false, 128, 12>(P, reqs, nreq, maxnl, maxS, true, result, status, st); break;
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
    cudaFuncSetAttribute(k_hky_fp64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_hky_fp64<<<nreq, HKY_BS, sm, st>>>(P, reqs, result, status, 2 * maxn - 1);
}

void launch_hky_commit(const Pools &P, const int32_t *items, const uint8_t *accept, int n,
                       cudaStream_t st)
{
  if (n <= 0) return;
  k_hky_commit<<<n, 128, 0, st>>>(P, items, accept);
}
