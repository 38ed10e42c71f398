// surf_common.cu -- operand preparation and the FP64 merge of the
// split-precision surface (see k_surf_fast.cu).
#include <cuda_fp16.h>

#include "surf_common.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr double LOG2 = 0.69314718055994530941723212146;

__host__ __device__ inline size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

// a maximum kept by many warps: an atomic only where it would change something
__device__ __forceinline__ void raise_max(unsigned *p, unsigned v)
{
  if (v > __ldcg(p)) atomicMax(p, v);
}

constexpr int PR_G = 128;  // genealogies per CTA of k_prep_rows

// Statistics of every genealogy in exact floats and its bias in float-float.
// Columns: cc_i, 2 fc_i (theta terms), mc_j, fm_j (migration terms); the
// bias is the reference's -probg (2 populations), -sum qi / -sum mi (model
// types 1 / 2) or the supplied FP64 normaliser, minus sum hcc_i.  A CTA's rows
// pass through shared memory, so that both the rows' reads and the columns'
// writes are whole lines (2,097,152 rows of 48: 1.32 ms with a thread walking
// its row, an eighth of that now).
__global__ void __launch_bounds__(PR_G) k_prep_rows(SurfArgs a, SurfPrep S)
{
  extern __shared__ float rows[];  // [PR_G][rowlen | 1]
  const int t = threadIdx.x, g0 = blockIdx.x * PR_G, g = g0 + t, stride = a.rowlen | 1;
  const int np = a.np, nm = a.nm, K = S.K;
  const int nr = min(PR_G, a.G - g0);
  for (int i = t; i < nr * a.rowlen; i += PR_G)
    rows[i / a.rowlen * stride + i % a.rowlen] = a.rows[(size_t)g0 * a.rowlen + i];
  __syncthreads();
  const bool in = g < a.G;
  const float *r = rows + t * stride;
  const int fc = np, hcc = 2 * np, mc = 3 * np, qi = 3 * np + 2 * nm, mi = 4 * np + 2 * nm, probg = 4 * np + 3 * nm + 1;
  double bias = 0.0;
  if (in) {
    if (a.lognorm) bias = a.lognorm[g];
    else if (a.npops == 2) bias = -(double)r[probg];
    else {
      double s = 0.0;
      if (a.modeltype == 1) for (int i = 0; i < np; i++) s += r[qi + i];
      else for (int i = 0; i < nm; i++) s += r[mi + i];
      bias = -s;
    }
    if (a.modeltype != 2)
      for (int i = 0; i < np; i++) bias -= r[hcc + i];
  }
  const float bh = (float)bias;
  S.biasff[g] = make_float2(bh, (float)(bias - (double)bh));
  // the genealogies floor(i G / n), i < n
  const int n = min(SURF_SAMPLES, a.G);
  const int i = (int)(((long long)g * n + a.G - 1) / a.G);
  const bool sampled = in && i < n && (int)((long long)i * a.G / n) == g;
  unsigned top = 0;
  for (int k = 0; k < SURF_KP; k++) {
    float v = 0.f;
    if (in && k < K) v = k < np ? r[k] : k < 2 * np ? 2.0f * r[fc + k - np] : r[mc + k - 2 * np];
    if (in && k == K) v = bh;
    S.sT[(size_t)k * S.Gpad + g] = v;
    if (sampled) S.samp[i * SURF_KP + k] = v;
    const unsigned m = __reduce_max_sync(0xffffffffu, in ? __float_as_uint(fabsf(v)) : 0u);
    if ((t & 31) == k) top = m;
  }
  raise_max(&S.colmax[t & 31], top);
}

// The tensor-core operand of a column is in units of 2^e, e such that its
// largest statistic lies in [64, 128): FP16 then holds counts exactly, and
// phi 2^e far from its ends.
__device__ __forceinline__ int col_exp(const SurfPrep &S, int k)
{
  const int e = (int)(S.colmax[k] >> 23) - 127 - 6;
  return e < -110 ? -110 : e > 110 ? 110 : e;
}
__device__ __forceinline__ float exp2i(int e) { return __int_as_float((127 + e) << 23); }

// FP16 statistics in the MMA's tile layout and FP32 ones as a line per
// genealogy, a thread per genealogy; in FP16 the bias (column K) leaves its
// rounding error in column K + 1.  emax: the columns' largest rounding errors.
__global__ void __launch_bounds__(256) k_prep_tiles(SurfPrep S)
{
  const int g = blockIdx.x * 256 + threadIdx.x;
  char *tile = reinterpret_cast<char *>(S.sh) + (size_t)(g / SURF_TC_N) * SURF_TC_N * SURF_KP * 2;
  float4 *line = S.sR + (size_t)g * (SURF_KP / 4);
  const float2 bias = S.biasff[g];
  float left = 0.f;  // the bias's rounding error
  unsigned top = 0;
  for (int q = 0; q < SURF_KP / 8; q++) {
    __align__(16) __half2 h[4];
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int k = 8 * q + j;
      const int e = col_exp(S, k == S.K + 1 ? S.K : k);
      const float v = k == S.K + 1 ? left : S.sT[(size_t)k * S.Gpad + g];
      f[j] = k < S.K ? v : 0.f;
      const __half x = __float2half_rn(v * exp2i(-e));
      const float d = v - __half2float(x) * exp2i(e);
      // no weight, or no bound: infinite, so that every other term passes the
      // screen (a value that is not a number leaves none, its own or a point's)
      const float r = isinf(k == S.K + 1 ? bias.x : v) ? INFINITY : d;
      if (k == S.K) left = d;
      if (j & 1) h[j >> 1] = __halves2half2(__low2half(h[j >> 1]), x);
      else h[j >> 1] = __halves2half2(x, x);
      const unsigned m = k == S.K ? 0u : __reduce_max_sync(0xffffffffu, g < S.G ? __float_as_uint(fabsf(r)) : 0u);
      if ((threadIdx.x & 31) == k) top = m;
    }
    if (q == SURF_KP / 8 - 1) {
      f[6] = bias.x;
      f[7] = bias.y;
    }
    *reinterpret_cast<uint4 *>(tile + tc::tile_off(g % SURF_TC_N, 8 * q)) = *reinterpret_cast<uint4 *>(h);
    line[2 * q] = make_float4(f[0], f[1], f[2], f[3]);
    line[2 * q + 1] = make_float4(f[4], f[5], f[6], f[7]);
  }
  raise_max(&S.emax[threadIdx.x & 31], top);
}

// Error of the tensor-core screen beyond the operands' rounding: 32 exact FP16
// products added in FP32, even if every addition truncates, at most 33 2^-22
// = 8e-6 of sum_k |s_k phi_k|.
constexpr float TC_ACC_ERR = 2e-5f;

// phi(x) of every point, a warp per two points: half a warp for the
// parameters of each (FP64 logarithms and reciprocals), then a lane per
// column of one and of the other; terms outside the model type get
// coefficient 0.  Then, a lane per genealogy, the exact maximum over nseed <= 32
// evenly spaced ones, the starting value of the maximum shared by chunks.
__global__ void __launch_bounds__(256) k_prep_points(SurfArgs a, SurfPrep S, int npad, int nseed, SurfZero z)
{
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i < z.n0; i += 256) z.z0[i] = 0;
    for (int i = threadIdx.x; i < z.n1; i += 256) z.z1[i] = 0;
  }
  const int p0 = (blockIdx.x * 256 + threadIdx.x) >> 5 << 1, k = threadIdx.x & 31;
  if (p0 >= npad) return;
  const int np = a.np, nm = a.nm, K = S.K;
  const int lo = (a.modeltype == 2) ? np : 0, hi = (a.modeltype == 1) ? np : np + nm;
  double plog = 0.0, pinv = 0.0;  // ln x, and -1/x (theta) or -x (m)
  {
    const int p = p0 + (k >> 4), j = k & 15;
    if (p < a.npoints && j >= lo && j < hi) {
      const double v = a.x[(size_t)p * (np + nm) + j];
      plog = log(v);
      pinv = j < np ? -1.0 / v : -v;
    }
  }
  const int j = k < np ? k : k < 2 * np ? k - np : k < 2 * np + nm ? k - np : k - np - nm;  // the column's parameter
  const float top = __uint_as_float(S.colmax[k]);
#pragma unroll 1
  for (int h = 0; h < 2; h++) {
    const int p = p0 + h;
    const double vl = __shfl_sync(0xffffffffu, plog, 16 * h + (j & 15)), vi = __shfl_sync(0xffffffffu, pinv, 16 * h + (j & 15));
    const bool in = p < a.npoints;
    double phi = 0.0;
    if (in && k < K && j >= lo && j < hi)
      phi = k < np ? LOG2 - vl : k >= 2 * np && k < 2 * np + nm ? vl : vi;
    if (in && k == K) phi = 1.0;
    const float v = (float)phi, vlo = (float)(phi - (double)v);
    if (in) {
      S.phi32[(size_t)p * SURF_KP + k] = v;
      if (k < SURF_K) S.phiff[(size_t)p * SURF_K + k] = make_float2(v, vlo);
    }
    float mag = top * fabsf(v), err = 0.f;
    if (S.ph) {  // the MMA's tile layout, 128 points per tile
      const int e = col_exp(S, k == K + 1 ? K : k);
      const float w = k == K + 1 ? (in ? 1.0f : 0.f) : v;
      const __half x = __float2half_rn(fminf(fmaxf(w * exp2i(e), -60000.f), 60000.f));
      char *tile = reinterpret_cast<char *>(S.ph) + (size_t)(p / SURF_TC_M) * SURF_TC_M * SURF_KP * 2;
      *reinterpret_cast<__half *>(tile + tc::tile_off(p % SURF_TC_M, k)) = x;
      const float y = __half2float(x) * exp2i(-e);
      // |sum s phi - sum s^ phi^| <= sum colmax |phi - phi^| + |phi^| max |s - s^|;
      // NaN where a coefficient is not finite: nothing passes the screen
      err = top * (fabsf(w - y) + 6e-8f * fabsf(w)) + fabsf(y) * __uint_as_float(S.emax[k]) + (w - w);
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      mag += __shfl_xor_sync(0xffffffffu, mag, o);
      err += __shfl_xor_sync(0xffffffffu, err, o);
    }
    if (in && k == 0) {
      S.mag[p] = mag;
      S.err[p] = 1.001f * (err + TC_ACC_ERR * mag);
    }
    if (nseed > 0 && in) {
      float2 f[SURF_K];
#pragma unroll
      for (int q = 0; q < SURF_K; q++)
        f[q] = make_float2(__shfl_sync(0xffffffffu, v, q), __shfl_sync(0xffffffffu, vlo, q));
      float best = -INFINITY;
      const int n = min(nseed, S.G);
      for (int i = k; i < n; i += 32) {
        const int g = (int)(((long long)i * S.G) / n);
        const int s = S.G >= SURF_SAMPLES ? i * (SURF_SAMPLES / n) : g;
        best = fmaxf(best, surf_exact(S, g, S.samp + s * SURF_KP, 1, f).hi);
      }
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
      if (k == 0) {
        S.seed[p] = best;
        S.best[p] = f2ord(best);
        S.xmax[p] = f2ord(best);
      }
    }
  }
}

// the same maximum from more genealogies than a lane each, a warp per point
// (256 of them by the kernel above, two points a warp, took 190 us more for
// 16,384 points)
__global__ void __launch_bounds__(256) k_surf_seed(SurfPrep S, int npoints, int nseed)
{
  const int p = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (p >= npoints) return;  // warp-uniform
  float2 phi[SURF_K];
#pragma unroll
  for (int k = 0; k < SURF_K; k++) phi[k] = S.phiff[(size_t)p * SURF_K + k];
  float best = -INFINITY;
  const int n = min(nseed, S.G);
  for (int i = lane; i < n; i += 32) {
    const int g = (int)(((long long)i * S.G) / n);
    best = fmaxf(best, surf_exact(S, g, S.sT + g, S.Gpad, phi).hi);
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
  if (lane == 0) {
    S.seed[p] = best;
    S.best[p] = f2ord(best);
    S.xmax[p] = f2ord(best);
  }
}

__global__ void k_surf_merge_ff(SurfArgs a, const SurfPart *part, int nchunks)
{
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.npoints) return;
  const SurfPart *w = part + (size_t)p * nchunks;
  double M = -INFINITY;
  for (int c = 0; c < nchunks; c++)
    if (w[c].mh != -INFINITY) M = fmax(M, (double)w[c].mh + (double)w[c].ml);
  double s = 0.0, s2 = 0.0;
  for (int c = 0; c < nchunks; c++) {
    if (w[c].mh == -INFINITY) continue;
    double f = exp((double)w[c].mh + (double)w[c].ml - M);
    s += ((double)w[c].sh + (double)w[c].sl) * f;
    s2 += (double)w[c].s2 * f * f;
  }
  a.q[p] = log((double)a.G) - (M + log(s));
  if (a.ess) a.ess[p] = s * s / s2;
}

}  // namespace

size_t surf_prep_bytes(int G, int npoints)
{
  size_t Gpad = ((size_t)G + 255) / 256 * 256;
  size_t npad = ((size_t)npoints + 255) / 256 * 256;
  size_t b = 0;
  b += align256(sizeof(float) * SURF_KP * Gpad);
  b += align256(sizeof(float2) * Gpad);
  b += align256(sizeof(float2) * SURF_K * npad);
  b += align256(sizeof(float) * SURF_KP * npad);
  b += align256(sizeof(float) * npad);
  b += align256(sizeof(float) * npad);
  b += align256(sizeof(unsigned) * npad);
  b += align256(sizeof(unsigned) * npad);
  b += align256(sizeof(float) * npad);
  b += 2 * align256(sizeof(unsigned) * SURF_KP);
  b += align256(sizeof(uint16_t) * SURF_KP * Gpad);
  b += align256(sizeof(float) * SURF_KP * Gpad);
  b += align256(sizeof(float) * SURF_KP * SURF_SAMPLES);
  b += align256(sizeof(uint16_t) * SURF_KP * npad);
  return b;
}

SurfPart *surf_prep_carve(SurfPrep *S, char *base, int G, int npoints)
{
  size_t Gpad = ((size_t)G + 255) / 256 * 256;
  size_t npad = ((size_t)npoints + 255) / 256 * 256;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    char *p = base + o;
    o += align256(bytes);
    return p;
  };
  S->G = G;
  S->Gpad = (int)Gpad;
  // operands derived from the rows alone come first, at offsets that do not
  // depend on the number of points, so they survive between evaluations
  S->sT = reinterpret_cast<float *>(take(sizeof(float) * SURF_KP * Gpad));
  S->biasff = reinterpret_cast<float2 *>(take(sizeof(float2) * Gpad));
  S->colmax = reinterpret_cast<unsigned *>(take(sizeof(unsigned) * SURF_KP));
  S->emax = reinterpret_cast<unsigned *>(take(sizeof(unsigned) * SURF_KP));
  S->sh = reinterpret_cast<uint16_t *>(take(sizeof(uint16_t) * SURF_KP * Gpad));
  S->sR = reinterpret_cast<float4 *>(take(sizeof(float) * SURF_KP * Gpad));
  S->samp = reinterpret_cast<float *>(take(sizeof(float) * SURF_KP * SURF_SAMPLES));
  S->phiff = reinterpret_cast<float2 *>(take(sizeof(float2) * SURF_K * npad));
  S->phi32 = reinterpret_cast<float *>(take(sizeof(float) * SURF_KP * npad));
  S->mag = reinterpret_cast<float *>(take(sizeof(float) * npad));
  S->err = reinterpret_cast<float *>(take(sizeof(float) * npad));
  S->seed = reinterpret_cast<float *>(take(sizeof(float) * npad));
  S->best = reinterpret_cast<unsigned *>(take(sizeof(unsigned) * npad));
  S->xmax = reinterpret_cast<unsigned *>(take(sizeof(unsigned) * npad));
  S->ph = reinterpret_cast<uint16_t *>(take(sizeof(uint16_t) * SURF_KP * npad));
  return reinterpret_cast<SurfPart *>(base + o);
}

int surf_prep(const SurfArgs &a, SurfPrep &S, bool tc, bool rows_ready, int nseed, const SurfZero &z, cudaStream_t st)
{
  S.np = a.np;
  S.nm = a.nm;
  S.K = 2 * (a.np + a.nm);
  if (!tc) S.ph = nullptr;
  int nk = 1;
  if (!rows_ready) {
    // colmax and emax
    cudaMemsetAsync(S.colmax, 0, reinterpret_cast<char *>(S.emax + SURF_KP) - reinterpret_cast<char *>(S.colmax), st);
    k_prep_rows<<<S.Gpad / PR_G, PR_G, PR_G * (a.rowlen | 1) * sizeof(float), st>>>(a, S);
    nk++;
    if (tc) {
      k_prep_tiles<<<S.Gpad / 256, 256, 0, st>>>(S);
      nk++;
    }
  }
  const int npad = (a.npoints + 255) / 256 * 256;
  k_prep_points<<<npad / 16, 256, 0, st>>>(a, S, npad, nseed > 32 ? 0 : nseed, z);
  if (nseed > 32) {
    k_surf_seed<<<(a.npoints + 7) / 8, 256, 0, st>>>(S, a.npoints, nseed);
    nk++;
  }
  return nk;
}

void surf_merge(const SurfArgs &a, const SurfPart *part, int nchunks, cudaStream_t st)
{
  k_surf_merge_ff<<<(a.npoints + 127) / 128, 128, 0, st>>>(a, part, nchunks);
}
