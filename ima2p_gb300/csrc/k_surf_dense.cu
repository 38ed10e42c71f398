// k_surf_dense.cu -- the split-precision surface where most terms count.
//
// The tensor-core screen (k_surf_tc.cu) pays when few genealogies lie within
// MARGIN of a point's maximum.  On a run's own saved genealogies, whose p(G)
// follows the statistics, most of them do, and every term then went through
// the candidate rings of two refine warps per SM: 9.1 ms for 500 points x
// 100,000 genealogies of a two-population run, 5.5e9 terms/s.  For such
// points this file evaluates every term directly.
//
// k_surf_split counts, per point, how many of up to 256 evenly spaced
// genealogies lie within MARGIN of the point's bound.  A point with at least
// one in DENSE_FRAC is taken here, the others by the screen.  The line lies
// where a refined candidate costs as much as twelve terms here: 500 points x
// 100,000 genealogies of three widths take 544, 482 and 368 us with one in 12,
// 559, 543 and 399 with one in 16, 596, 556 and 296 with one in 8 (all here:
// 518, 519, 470; 1,300 points of 26 columns 1,670, 1,100 and 398 against 1,930,
// 1,790 and 1,790).
//
// k_surf_dense: lanes are points, phi in registers; a CTA's 8 warps share 32
// points and take a tile's 64 genealogies by turns, reading each statistic
// as a warp-wide broadcast.  A term is the same compensated dot product as
// surf_exact (started at bias - ref, so it gives p - ref), a float-float
// exponential (a 64-entry table of 2^(j/64) and four terms of e^r, within
// 1e-14 of the sum's largest weight), and float-float sums of w and w^2 over
// 64 terms at a time, added to FP64 sums.  About 170 FP32 instructions per
// term at 10 columns, FP32-issue bound: 385 us for the case above (1.3e11
// terms/s; the whole evaluation 9.40 -> 0.60 ms).  Units of (32 points, genealogy
// chunk) are dealt to a persistent grid; a point's chunk sums depend on the
// number of dense points only, so results repeat bit for bit.
#include <algorithm>
#include <cmath>

#include "surf_common.cuh"

namespace {

constexpr int DT = SURF_DENSE_TILE;
constexpr int DW = 8;            // warps per CTA, sharing 32 points
constexpr int DENSE_FRAC = 12;   // dense from one sampled genealogy in 12 within MARGIN
constexpr float DENSE_OVF = 40.0f;  // nats above ref at which a point is left to the retake: w^2 and its sums stay in FP32's range
__device__ float2 d_exp64[64];  // 2^(j/64) as float-float

constexpr int FLUSH = 8;         // tiles (of DT / DW terms per warp) between FP64 flushes

// One warp per sample group, lanes are points; counts[0] = dense points
// (their list in any order: each is evaluated on its own), sparse[t] = points
// of tensor-core tile t left to the screen.
__global__ void __launch_bounds__(256) k_surf_split(SurfPrep S, int npoints, uint8_t *dense, int *list, int *counts,
                                                    int *sparse)
{
  __shared__ float4 sm[SURF_SAMPLES * SURF_KP / 4];
  __shared__ int cnt[8][32];
  const int n = min(SURF_SAMPLES, S.G);
  const float4 *src = reinterpret_cast<const float4 *>(S.samp);
  for (int i = threadIdx.x; i < n * SURF_KP / 4; i += 256) sm[i] = src[i];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p = blockIdx.x * 32 + lane;
  float phi[SURF_KP];
  float thr = INFINITY;
  if (p < npoints) {
    const float b = ord2f(S.best[p]);
    if (fabsf(b) < INFINITY) thr = b - SURF_MARGIN;
    const float4 *f = reinterpret_cast<const float4 *>(S.phi32 + (size_t)p * SURF_KP);
#pragma unroll
    for (int k = 0; k < SURF_KP / 4; k++) {
      const float4 v = f[k];
      phi[4 * k] = v.x;
      phi[4 * k + 1] = v.y;
      phi[4 * k + 2] = v.z;
      phi[4 * k + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < SURF_KP; k++) phi[k] = 0.f;
  }
  __syncthreads();
  int c = 0;
  for (int i = warp; i < n; i += 8) {
    float v0 = 0.f, v1 = 0.f;
#pragma unroll
    for (int k = 0; k < SURF_KP / 4; k++) {
      const float4 s = sm[i * (SURF_KP / 4) + k];
      v0 = __fmaf_rn(s.x, phi[4 * k], v0);
      v1 = __fmaf_rn(s.y, phi[4 * k + 1], v1);
      v0 = __fmaf_rn(s.z, phi[4 * k + 2], v0);
      v1 = __fmaf_rn(s.w, phi[4 * k + 3], v1);
    }
    c += v0 + v1 > thr;
  }
  cnt[warp][lane] = c;
  __syncthreads();
  if (warp == 0) {
    int t = 0;
    for (int w = 0; w < 8; w++) t += cnt[w][lane];
    const bool d = p < npoints && t * DENSE_FRAC >= n;
    const unsigned m = __ballot_sync(0xffffffffu, d), sp = __ballot_sync(0xffffffffu, p < npoints && !d);
    int base = 0;
    if (lane == 0) {
      if (m) base = atomicAdd(counts, __popc(m));
      if (sp) atomicAdd(&sparse[blockIdx.x * 32 / SURF_TC_M], __popc(sp));
    }
    base = __shfl_sync(0xffffffffu, base, 0);
    if (d) list[base + __popc(m & ((1u << lane) - 1u))] = p;
    if (p < npoints) dense[p] = d;
  }
}

template <int KC>
__global__ void __launch_bounds__(32 * DW, KC <= 12 ? 3 : KC <= 20 ? 2 : 1)
    k_surf_dense(SurfPrep S, int col0, int ncols, const int *list, const int *counts, double2 *part)
{
  // a tile row: KC statistics, the bias (hi, lo), padding; an odd number of
  // 16-byte units, so the transposing stores conflict 4 ways at most
  constexpr int KS = ((KC + 4) / 4) % 2 ? KC + 4 : KC + 8;
  constexpr int NL = (DT * (KC + 2) + 32 * DW - 1) / (32 * DW);  // tile values each thread loads
  __shared__ __align__(16) float tile[DT * KS];
  __shared__ double red[2][DW][32];
  __shared__ int sovf[32];
  __shared__ float2 tab[64];
  const int nd = counts[0];
  if (nd == 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ntiles = (S.G + DT - 1) / DT;
  int per;
  const int nch = surf_dense_chunks(nd, gridDim.x, S.G, &per);
  const int groups = (nd + 31) / 32;
  if (tid < 64) tab[tid] = d_exp64[tid];
  const float2 *bias = S.biasff;
  for (int u = blockIdx.x; u < groups * nch; u += gridDim.x) {
    const int grp = u % groups, chunk = u / groups;
    const int t0 = chunk * per, t1 = min(ntiles, t0 + per);
    const bool live = grp * 32 + lane < nd;
    const int p = live ? list[grp * 32 + lane] : 0;
    float2 phi[KC];
#pragma unroll
    for (int k = 0; k < KC; k++)
      phi[k] = live && k < ncols ? S.phiff[(size_t)p * SURF_K + col0 + k] : make_float2(0.f, 0.f);
    const float ref = live ? ord2f(S.best[p]) : 0.f;
    if (tid < 32) sovf[tid] = 0;
    double dsum = 0.0, dsum2 = 0.0;
    ff a = ff_from(0.f), a2 = ff_from(0.f);
    float top = -INFINITY;
    // values of the tile at t, one genealogy per lane (coalesced)
    float v[NL];
    auto fetch = [&](int t) {
#pragma unroll
      for (int i = 0; i < NL; i++) {
        const int e = tid + i * 32 * DW, k = e / DT, g = t * DT + e % DT;
        float x = 0.f;
        if (e < DT * (KC + 2)) {
          if (k < KC) {
            if (k < ncols) x = S.sT[(size_t)(col0 + k) * S.Gpad + g];
          } else {
            const float2 b = bias[g];
            x = k > KC ? b.y : g < S.G ? b.x : -INFINITY;  // padding: weight 0
          }
        }
        v[i] = x;
      }
    };
    fetch(t0);
    for (int t = t0; t < t1; t++) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < NL; i++) {
        const int e = tid + i * 32 * DW;
        if (e < DT * (KC + 2)) tile[(e % DT) * KS + e / DT] = v[i];
      }
      __syncthreads();
      if (t + 1 < t1) fetch(t + 1);
#pragma unroll 2
      for (int j = warp; j < DT; j += DW) {
        const float4 *row = reinterpret_cast<const float4 *>(tile + j * KS);
        const float4 b = row[KC / 4];
        ff s0 = two_sum(b.x, -ref);
        float sum = s0.hi, comp = __fadd_rn(s0.lo, b.y);
#pragma unroll
        for (int kk = 0; kk < KC / 4; kk++) {
          const float4 s4 = row[kk];
          const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
          for (int h = 0; h < 4; h++) {  // Dot2, as surf_exact
            const float s = sv[h];
            const float2 f = phi[4 * kk + h];
            const float q = __fmul_rn(s, f.x);
            const float qe = __fmaf_rn(s, f.x, -q);
            const ff ts = two_sum(sum, q);
            sum = ts.hi;
            comp = __fadd_rn(comp, __fadd_rn(ts.lo, __fmaf_rn(s, f.y, qe)));
          }
        }
        const ff d = fast_two_sum(sum, comp);
        // below -80 nats (and NaN, as in the screen): no weight
        const bool in = d.hi > -80.f && d.hi <= DENSE_OVF;
        if (d.hi > top) top = d.hi;
        const ff w = exp_tab(in ? d.hi : 0.f, in ? d.lo : 0.f, tab);
        const float wh = in ? w.hi : 0.f, wl = in ? w.lo : 0.f;
        const ff t1s = two_sum(a.hi, wh);
        a = ff_make(t1s.hi, __fadd_rn(a.lo, __fadd_rn(t1s.lo, wl)));
        const float w2 = __fmul_rn(wh, wh), w2e = __fmaf_rn(2.f * wh, wl, __fmaf_rn(wh, wh, -w2));
        const ff t2s = two_sum(a2.hi, w2);
        a2 = ff_make(t2s.hi, __fadd_rn(a2.lo, __fadd_rn(t2s.lo, w2e)));
      }
      if ((t - t0) % FLUSH == FLUSH - 1 || t + 1 == t1) {
        dsum += (double)a.hi + (double)a.lo;
        dsum2 += (double)a2.hi + (double)a2.lo;
        a = a2 = ff_from(0.f);
      }
    }
    red[0][warp][lane] = dsum;
    red[1][warp][lane] = dsum2;
    if (top > DENSE_OVF && live) {
      sovf[lane] = 1;
      atomicMax(&S.xmax[p], f2ord(top + ref));
    }
    __syncthreads();
    if (warp == 0 && live) {
      double s = 0.0, s2 = 0.0;
      for (int w = 0; w < DW; w++) {
        s += red[0][w][lane];
        s2 += red[1][w][lane];
      }
      part[(size_t)p * SURF_MAX_CHUNKS + chunk] = make_double2(sovf[lane] ? -1.0 : s, s2);
    }
    __syncthreads();  // red and sovf are reused
  }
}

int g_dense_blocks(int kc, int nsm)
{
  return nsm * (kc <= 12 ? 3 : kc <= 20 ? 2 : 1);
}

}  // namespace

int surf_init_tables()
{
  float2 t[64];
  for (int j = 0; j < 64; j++) {
    const double v = std::exp2(j / 64.0);
    t[j] = make_float2((float)v, (float)(v - (double)(float)v));
  }
  return cudaMemcpyToSymbol(d_exp64, t, sizeof(t)) == cudaSuccess ? 0 : -1;
}

float2 *surf_exp_table()
{
  void *p = nullptr;
  return cudaGetSymbolAddress(&p, d_exp64) == cudaSuccess ? static_cast<float2 *>(p) : nullptr;
}

int surf_dense_cols(const SurfArgs &a, int *col0)
{
  *col0 = a.modeltype == 2 ? 2 * a.np : 0;
  return a.modeltype == 0 ? 2 * (a.np + a.nm) : a.modeltype == 1 ? 2 * a.np : 2 * a.nm;
}

void surf_split(const SurfPrep &S, int npoints, const SurfSplit &D, cudaStream_t st)
{
  k_surf_split<<<(npoints + 31) / 32, 256, 0, st>>>(S, npoints, D.dense, D.list, D.counts, D.counts + 1);
}

int surf_dense_grid(const SurfArgs &a, int nsm)
{
  int col0;
  return g_dense_blocks((surf_dense_cols(a, &col0) + 3) / 4 * 4, nsm);
}

void surf_dense(const SurfArgs &a, const SurfPrep &S, const SurfSplit &D, int nb, double2 *part, cudaStream_t st)
{
  int col0;
  const int nc = surf_dense_cols(a, &col0);
  switch ((nc + 3) / 4) {
#define IMA_DENSE(N) \
  case N: k_surf_dense<4 * N><<<nb, 32 * DW, 0, st>>>(S, col0, nc, D.list, D.counts, part); break;
    IMA_DENSE(1) IMA_DENSE(2) IMA_DENSE(3) IMA_DENSE(4) IMA_DENSE(5) IMA_DENSE(6) IMA_DENSE(7) IMA_DENSE(8)
#undef IMA_DENSE
  }
}
