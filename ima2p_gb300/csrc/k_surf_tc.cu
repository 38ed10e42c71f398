// k_surf_tc.cu -- tensor-core screen of the L-mode surface (tcgen05, sm_103a).
//
// The screen of the split-precision surface (see k_surf_fast.cu) as a GEMM on
// the 5th-generation tensor cores: D[point][genealogy] = phi(x_point) .
// s_genealogy over 32 columns (up to 30 statistics, the bias in two parts),
// FP16 operands in units that suit each column and FP32 accumulation in
// tensor memory.  The screen only has to tell which terms may lie within
// MARGIN of the maximum: the statistics are counts and rates that FP16 holds
// exactly or to 2^-12, so one product is enough, and every point carries a
// bound on its error (S.err, from the columns' largest rounding errors and
// its own coefficients') that widens its threshold.
//
// One CTA owns 128 points (the A operand, loaded once) and streams tiles of
// 256 genealogies (the B operand) through an 8-stage shared-memory ring
// filled by 1-D bulk copies (the TMA engine; the prepared operand is already
// in the tile layout, so one copy per tile).  Warp roles:
//   warp 0     issues the bulk copies;
//   warps 1-2  issue, each for its half of every tile, two K=16 MMAs into one
//              of four 128-column TMEM accumulators (the tensor cores hold few
//              instructions: one warp's waits would leave them idle);
//   warps 3-6  take the rings' candidates 32 at a time, recompute them
//              exactly (phi of every point is staged in shared memory) and
//              add exp(p - ref) to the point's sums;
//   warps 7-22 drain the accumulators, four warps to each: a warp reads TMEM
//              lane quarter w % 4 (32 points, one per thread) by
//              tcgen05.ld.red of 32 columns, which return the maximum of
//              their 32 values too; where it lies within MARGIN +
//              screen error of the point's lower bound, the values above that
//              become candidates and go to a ring.
//
// 7.1 ms a call, 2.9 in the first pass and 3.6 in the second, against 20.3 with
// bf16 operands split into two halves (three products), two 256-column
// accumulators and one issuing thread; the first pass's products alone are 2.1.
//
// Results are bit-for-bit reproducible.  Two things would otherwise follow
// timing: which terms pass the screen, and the order in which they are added.
//   * The set: a drain warp's threshold is the point's lower bound from the
//     max-only pre-pass (a maximum over a fixed set of values, so fixed);
//     without a pre-pass it is raised by the screened maxima of the warp's own
//     earlier values.  Nothing another warp or chunk found moves it, so every
//     warp screens the same terms on every run.
//   * The order: each term's weight w = exp(p - ref), with ref the pre-pass
//     bound, is added as a 256-bit fixed-point integer (w * 2^64) by 64-bit
//     shared-memory atomics with exact carries.  Integer addition is
//     associative, so the sum does not depend on arrival order; the chunk
//     sums are merged in chunk order.
// A term with w >= 2^80 (the pre-pass bound more than 55 nats below the
// term) would leave the fixed-point range: the point is flagged.  The pass
// also keeps each point's largest exact value, a maximum and so the same on
// every run; the flagged points are then taken again by a second pass over
// just them, with that value as the reference, where no term can exceed it.
//
// Every wait is bounded: a wait that runs out sets the error word, the CTA
// stops issuing work, waits (bounded) for the copies and MMAs it started,
// frees its TMEM and returns.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "surf_common.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr int TC_M = SURF_TC_M;  // points per CTA (TMEM lanes)
constexpr int TC_N = SURF_TC_N;  // genealogies per tile (accumulator columns)
constexpr int ACC_N = TC_N / 2;       // genealogies per accumulator: half a tile
constexpr int NACC = 512 / ACC_N;    // TMEM accumulators
constexpr uint32_t A_BYTES = TC_M * SURF_KP * 2;   // 8 KB
constexpr uint32_t B_BYTES = TC_N * SURF_KP * 2;   // 16 KB
constexpr int TC_STAGES = (128 * 1024) / B_BYTES;  // operand ring stages (128 KB of B tiles)
// shared memory requested per CTA: more than half an SM's, so one CTA holds
// an SM and its 512 TMEM columns at a time (the operand ring, phi of the
// CTA's points, the candidate rings and the per-point log-sum-exp states)
constexpr size_t TC_SMEM = 212 * 1024;
constexpr uint32_t WAIT_LIMIT = 1u << 24;          // try_wait rounds before a wait gives up

constexpr int PHI_STRIDE = SURF_K + 1;   // float2 per point row of staged phi (padded)
constexpr int REF_WARPS = 4;             // warps recomputing candidates exactly
constexpr int MMA_WARPS = 2;             // a warp issues the products of one half of every tile
constexpr int REF_WARP0 = 1 + MMA_WARPS; // the first of the refining warps
constexpr int EPI_WARP0 = REF_WARP0 + REF_WARPS;
constexpr int EPI_WARPS = 16;            // warps draining the accumulators
constexpr int ACC_WARPS = EPI_WARPS / NACC;  // warps of an accumulator: its 4 lane quarters
constexpr int TC_THREADS = 32 * (EPI_WARP0 + EPI_WARPS);
static_assert(ACC_WARPS == 4 && NACC == 4 && ACC_N % 64 == 0, "a warp drains a lane quarter of one accumulator");
constexpr int RING = 256;                // candidate slots per epilogue warp
static_assert(REF_WARPS == 4, "refine warp r takes the candidates of epilogue warps r, r + 4, ...: one lane quarter");

constexpr int FIXW = 4;  // 64-bit words of the fixed-point sums

struct TcSmem {
  // full[s]: B tile of stage s landed; done[s]: its MMAs completed (stage
  // free); accfull[a], accempty[a]: accumulator a complete, drained
  uint64_t full[TC_STAGES], done[TC_STAGES], accfull[NACC], accempty[NACC], abar;
  uint32_t tmem;
  int err;
  int epi_done;                       // epilogue warps that have finished
  unsigned head[EPI_WARPS], tail[EPI_WARPS];  // candidates put into and taken from each ring
  int ring[EPI_WARPS][RING];          // candidates: genealogy << 7 | point
  unsigned long long sum[TC_M][FIXW];   // sum of w * 2^64, w = exp(p - ref), 256-bit fixed point
  unsigned long long sum2[TC_M][FIXW];  // sum of w^2 * 2^64
  float ref[TC_M];                    // the point's lower bound after the pre-pass
  unsigned xmax[TC_M];                // largest exact value refined (ordered bits)
  int ovf[TC_M];                      // a term left the fixed-point range
  float2 phi[TC_M * PHI_STRIDE];      // float-float phi of the CTA's points
  float2 etab[64];                    // 2^(j/64)
};

// w >= 2^80 (55.45 nats above ref) leaves the range the sums are sized for:
// 2^24 genealogies of w^2 * 2^64 < 2^160 * 2^64 stay below 2^248
constexpr double OVF_NATS = 55.0;

// w * 2^64 as a 256-bit integer, truncated (0 <= w < 2^180)
__device__ __forceinline__ void fixw(double w, unsigned long long o[FIXW])
{
#pragma unroll
  for (int i = 0; i < FIXW; i++) o[i] = 0ull;
  const unsigned long long b = (unsigned long long)__double_as_longlong(w);
  const int e = (int)((b >> 52) & 0x7ff);
  if (!(w > 0.0) || e == 0) return;  // zero or subnormal: nothing at this scale
  const unsigned long long m = (b & 0xfffffffffffffull) | (1ull << 52);
  const int s = e - 1023 - 52 + 64;  // w * 2^64 = m * 2^s
  if (s <= -53) return;
  if (s < 0) {
    o[0] = m >> (-s);
    return;
  }
  const int wd = s >> 6, bit = s & 63;
  if (wd < FIXW) o[wd] = m << bit;
  if (bit && wd + 1 < FIXW) o[wd + 1] = m >> (64 - bit);
}

// acc += x on a 256-bit integer in shared memory, word by word with 64-bit
// atomics; a word that wraps carries one into the next.  Every wrap is seen
// by exactly one atomic, so the sum is exact whatever the interleaving.
__device__ __forceinline__ void atomic_addw(unsigned long long *acc, const unsigned long long x[FIXW])
{
  unsigned long long carry = 0ull;
#pragma unroll
  for (int i = 0; i < FIXW; i++) {
    unsigned long long out = 0ull;
    if (x[i]) {
      const unsigned long long old = atomicAdd(&acc[i], x[i]);
      out += (old + x[i] < old) ? 1ull : 0ull;
    }
    if (carry) {
      const unsigned long long old = atomicAdd(&acc[i], carry);
      out += (old + carry < old) ? 1ull : 0ull;
    }
    carry = out;
  }
}

__device__ __forceinline__ double fixw_to_double(const unsigned long long w[FIXW])
{
  // powers of two are exact; the order of the additions is fixed
  double v = 0.0;
#pragma unroll
  for (int i = FIXW - 1; i >= 0; i--) v = v * 18446744073709551616.0 + (double)w[i];
  return v * 5.421010862427522e-20;  // 2^-64
}

__device__ __forceinline__ void set_err(int *err_shared, int *err_global, int code)
{
  atomicCAS(err_shared, 0, code);
  atomicCAS(err_global, 0, code);
}

// An epilogue warp's side of its candidate ring.  The ring has one writing
// and one reading warp, so its ends are plain counters.
struct CandidateRing {
  unsigned head = 0, tail = 0;  // put so far; taken, as last seen

  // the warp's lanes hand over (point pl, genealogies g0 + the set bits of mask)
  __device__ __forceinline__ void put(TcSmem &sh, int *gerr, int ew, int lane, int pl, int g0, unsigned mask)
  {
    for (;;) {
      const unsigned b = __ballot_sync(0xffffffffu, mask != 0);
      if (!b) return;
      const unsigned n = __popc(b);
      for (uint32_t it = 0; head + n - tail > RING; it++) {
        tail = __shfl_sync(0xffffffffu, *(volatile unsigned *)&sh.tail[ew], 0);
        if (head + n - tail <= RING) break;
        if (__any_sync(0xffffffffu, it > WAIT_LIMIT || *(volatile int *)&sh.err)) {
          set_err(&sh.err, gerr, 6);
          return;
        }
        __nanosleep(32);
      }
      if (mask) {
        *(volatile int *)&sh.ring[ew][(head + __popc(b & ((1u << lane) - 1u))) % RING] = ((g0 + __ffs(mask) - 1) << 7) | pl;
        mask &= mask - 1;
      }
      head += n;
      __threadfence_block();
      __syncwarp();
      if (lane == 0) *(volatile unsigned *)&sh.head[ew] = head;
    }
  }
};

// below w = exp(d) < 2^-66 a term adds nothing at the sums' scale of 2^-64
constexpr float ZERO_NATS = -46.0f;

// One candidate per lane, recomputed exactly; its weight is added to its
// point's sums.
__device__ __forceinline__ void refine(const SurfPrep &S, TcSmem &sh, int e)
{
  const int pl = e & (TC_M - 1), g = e >> 7;
  const ff y = surf_exact_row(S, g, &sh.phi[pl * PHI_STRIDE]);
  const unsigned yo = f2ord(y.hi);
  if (yo > *(volatile unsigned *)&sh.xmax[pl]) atomicMax(&sh.xmax[pl], yo);
  const ff d = ff_sub(y, ff_from(sh.ref[pl]));
  if (d.hi > (float)OVF_NATS) {
    sh.ovf[pl] = 1;
  } else if (!(d.hi < ZERO_NATS)) {
    // w = e^d in float-float (FP32 pipes: GB300 runs FP64 at 1/64 of the FP32
    // rate); hi + lo is exact in a double, and w^2 (up to 2^160, beyond FP32's
    // range) is squared there
    const ff x = exp_tab(d.hi, d.lo, sh.etab);
    const double w = (double)x.hi + (double)x.lo;
    unsigned long long f[FIXW];
    fixw(w, f);
    atomic_addw(sh.sum[pl], f);
    fixw(w * w, f);
    atomic_addw(sh.sum2[pl], f);
  }
}

// Refine warp r: takes the candidates of its four rings 32 at a time.  It
// stops when every epilogue warp has finished and the rings are drained.
__device__ void refine_loop(const SurfPrep &S, TcSmem &sh, int *gerr, int r, int lane)
{
  constexpr int NR = EPI_WARPS / REF_WARPS;
  unsigned tail = 0;  // lane j < NR: of ring r + REF_WARPS j
  for (uint32_t idle = 0;;) {
    const bool last = __shfl_sync(0xffffffffu, *(volatile int *)&sh.epi_done, 0) == EPI_WARPS;
    __threadfence_block();
    const unsigned have = *(volatile unsigned *)&sh.head[r + REF_WARPS * (lane % NR)] - tail;
    __threadfence_block();
    const unsigned ready = __ballot_sync(0xffffffffu, lane < NR && (have >= 32 || (last && have > 0)));
    if (ready) {
      idle = 0;
      const int j = __ffs(ready) - 1, ew = r + REF_WARPS * j;
      const unsigned n = min(32u, __shfl_sync(0xffffffffu, have, j)), t = __shfl_sync(0xffffffffu, tail, j);
      const int e = *(volatile int *)&sh.ring[ew][(t + lane) % RING];
      __syncwarp();
      if (lane == j) *(volatile unsigned *)&sh.tail[ew] = tail += n;
      if (lane < n) refine(S, sh, e);
      __syncwarp();
      continue;
    }
    if (last) break;
    if (__any_sync(0xffffffffu, ++idle > WAIT_LIMIT || *(volatile int *)&sh.err)) {
      if (idle > WAIT_LIMIT) set_err(&sh.err, gerr, 7);
      break;
    }
    __nanosleep(64);
  }
}

// MAXONLY: a pass that only raises the per-point lower bounds S.best (no
// candidates, no partials); otherwise the full pass, which reads S.best and
// leaves it unchanged (raise: there was no pre-pass).  Over every 2nd or 4th
// tile the first pass would be cheaper and its bounds lower: where the terms
// are alike it would pay (32,768 points x 2,097,152 genealogies: 7.7 ms, 6.3
// with every 4th), where a few genealogies dominate a point it would not
// (8,192 x 1,048,576: 1.35 ms, 1.83 with every 2nd).  dense, sparse (may be null: every point): the
// full pass leaves the points with dense[p] = 1 to k_surf_dense, and skips
// the tiles without others (sparse[tile] = 0).
template <bool MAXONLY>
__global__ void __launch_bounds__(TC_THREADS, 1)
    k_surf_tc(SurfPrep S, int npoints, int tiles_per_chunk, bool raise, const float2 *etab,
              const uint8_t *dense, const int *sparse, double2 *part, int *gerr)
{
  extern __shared__ __align__(1024) char smem[];
  if (sparse && sparse[blockIdx.x] == 0) return;
  char *bufA = smem;
  char *bufB = smem + A_BYTES;
  TcSmem &sh = *reinterpret_cast<TcSmem *>(smem + A_BYTES + TC_STAGES * B_BYTES);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int ptile = blockIdx.x;
  const int ntiles_all = S.Gpad / TC_N;
  const int t0 = blockIdx.y * tiles_per_chunk, t1 = min(ntiles_all, t0 + tiles_per_chunk);
  const int ntiles = max(0, t1 - t0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < TC_STAGES; s++) {
      tc::mbar_init(&sh.full[s], 1);
      tc::mbar_init(&sh.done[s], MMA_WARPS);
    }
    for (int a = 0; a < NACC; a++) {
      tc::mbar_init(&sh.accfull[a], 1);
      tc::mbar_init(&sh.accempty[a], ACC_WARPS);  // one arrival per warp draining it
    }
    tc::mbar_init(&sh.abar, 1);
    sh.err = 0;
    sh.epi_done = 0;
    tc::fence_barrier_init();
  }
  // every thread stages phi, the rings and the per-point states
  for (int i = threadIdx.x; i < TC_M * SURF_K; i += TC_THREADS) {
    const int pl = i / SURF_K, k = i % SURF_K, p = ptile * TC_M + pl;
    sh.phi[pl * PHI_STRIDE + k] = p < npoints ? S.phiff[(size_t)p * SURF_K + k] : make_float2(0.f, 0.f);
  }
  if (threadIdx.x < EPI_WARPS) sh.head[threadIdx.x] = sh.tail[threadIdx.x] = 0;
  if (threadIdx.x < 64) sh.etab[threadIdx.x] = etab[threadIdx.x];
  for (int pl = threadIdx.x; pl < TC_M; pl += TC_THREADS) {
    for (int w = 0; w < FIXW; w++) sh.sum[pl][w] = sh.sum2[pl][w] = 0ull;
    const int p = ptile * TC_M + pl;
    sh.ref[pl] = p < npoints ? ord2f(S.best[p]) : -INFINITY;
    sh.xmax[pl] = f2ord(-INFINITY);
    sh.ovf[pl] = 0;
  }
  if (warp == 0) {
    tc::tmem_alloc(&sh.tmem, 512);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = sh.tmem;

  if (warp == 0) {
    // ------------------------------------------------------------ loader
    if (tc::elect_one()) {
      tc::mbar_expect_tx(&sh.abar, A_BYTES);
      tc::bulk_g2s(bufA, S.ph + (size_t)ptile * (A_BYTES / 2), A_BYTES, &sh.abar);
    }
    __syncwarp();
    int issued = 0;
    for (int i = 0; i < ntiles; i++) {
      const int s = i % TC_STAGES;
      const bool ok = i < TC_STAGES || tc::mbar_wait(&sh.done[s], ((i / TC_STAGES) - 1) & 1, WAIT_LIMIT);
      if (!ok) set_err(&sh.err, gerr, 1);
      if (!__all_sync(0xffffffffu, ok && !*(volatile int *)&sh.err)) break;
      if (tc::elect_one()) {
        tc::mbar_expect_tx(&sh.full[s], B_BYTES);
        tc::bulk_g2s(bufB + s * B_BYTES, S.sh + (size_t)(t0 + i) * (B_BYTES / 2), B_BYTES, &sh.full[s]);
      }
      __syncwarp();
      issued = i + 1;
    }
    // copies this warp started must land before the CTA can leave
    for (int i = max(0, issued - TC_STAGES); i < issued; i++)
      tc::mbar_wait(&sh.full[i % TC_STAGES], (i / TC_STAGES) & 1, WAIT_LIMIT);
    tc::mbar_wait(&sh.abar, 0, WAIT_LIMIT);
  } else if (warp < REF_WARP0) {
    // --------------------------------------------------------------- MMA
    const int half = warp - 1;
    const uint32_t idesc = tc::idesc_f16_f32(TC_M, ACC_N);
    // descriptors: the address field counts 16-byte units, so offsets add
    const uint64_t ad = tc::sdesc(tc::smem_u32(bufA), 128, 512);
    const uint64_t bd0 = tc::sdesc(tc::smem_u32(bufB) + half * (B_BYTES / 2), 128, 512);
    bool ok = tc::mbar_wait(&sh.abar, 0, WAIT_LIMIT);
    if (!ok) set_err(&sh.err, gerr, 2);
    int ndone = 0;
    for (int i = 0; i < ntiles; i++) {
      const int s = i % TC_STAGES, h = 2 * i + half, a = h % NACC;
      if (ok && !tc::mbar_wait(&sh.full[s], (i / TC_STAGES) & 1, WAIT_LIMIT)) {
        set_err(&sh.err, gerr, 3);
        ok = false;
      }
      if (ok && h >= NACC && !tc::mbar_wait(&sh.accempty[a], ((h / NACC) - 1) & 1, WAIT_LIMIT)) {
        set_err(&sh.err, gerr, 4);
        ok = false;
      }
      // all of the warp goes on or none
      if (!__all_sync(0xffffffffu, ok && !*(volatile int *)&sh.err)) break;
      tc::fence_after_sync();
      const uint32_t d = tmem + (uint32_t)(a * ACC_N);
      const uint64_t bd = bd0 + (uint64_t)((s * B_BYTES) >> 4);
      if (tc::elect_one()) {
#pragma unroll
        for (int kh = 0; kh < 2; kh++) tc::mma_f16(d, ad + kh * 16, bd + kh * 16, idesc, kh);
        tc::mma_commit(&sh.accfull[a]);
        tc::mma_commit(&sh.done[s]);  // and, with the other half's, stage s free
      }
      __syncwarp();
      ndone = i + 1;
    }
    // the products this warp started end before the CTA frees its TMEM
    if (ndone > 0) {
      const int h = 2 * (ndone - 1) + half;
      tc::mbar_wait(&sh.accfull[h % NACC], (h / NACC) & 1, WAIT_LIMIT);
    }
  } else if (warp >= REF_WARP0 && warp < EPI_WARP0) {
    // ------------------------------------------------------------ refine
    if (!MAXONLY) refine_loop(S, sh, gerr, warp - REF_WARP0, lane);
  } else if (warp >= EPI_WARP0) {
    // ---------------------------------------------------------- epilogue
    const int ew = warp - EPI_WARP0;
    const int q = warp & 3;             // TMEM lane quarter of this warp
    const int a = ew / ACC_WARPS;       // its accumulator: half a & 1 of the tiles a / 2, a / 2 + 2, ...
    const int pl = q * 32 + lane;       // point within the tile = TMEM lane
    const int p = ptile * TC_M + pl;
    const bool live = p < npoints && !(dense && dense[p]);
    const float err = live ? S.err[p] : 0.f;  // screen error bound
    // lb: a lower bound on the point's maximum
    float lb = live ? sh.ref[pl] : -INFINITY;
    float thr = live ? lb - (err + SURF_MARGIN) : INFINITY;
    const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * ACC_N);
    float mx = -INFINITY;  // pre-pass: largest screened value
    CandidateRing ring;
    uint32_t parity = 0;
    int gc = (t0 + a / 2) * TC_N + (a & 1) * ACC_N;  // genealogy of the first column
    for (int i = a / 2; i < ntiles; i += NACC / 2, gc += (NACC / 2) * TC_N, parity ^= 1) {
      if (!tc::mbar_wait(&sh.accfull[a], parity, WAIT_LIMIT)) {
        set_err(&sh.err, gerr, 5);
        break;
      }
      tc::fence_after_sync();
#pragma unroll
      for (int c = 0; c < ACC_N; c += 64) {
        // two loads in flight; nothing but straight-line code runs before
        // they have landed
        uint32_t r[2][32], m[2];
        tc::tmem_ld32_max_nowait(tl + c, r[0], m[0]);
        tc::tmem_ld32_max_nowait(tl + c + 32, r[1], m[1]);
        tc::tmem_wait_ld(r[0]);
        tc::reg_fence32(r[1]);
        tc::reg_fence(m[0]);
        tc::reg_fence(m[1]);
        if (c + 64 == ACC_N) {  // the accumulator has been read
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&sh.accempty[a]);
        }
        const float m0 = __uint_as_float(m[0]), m1 = __uint_as_float(m[1]);
        if (MAXONLY) {
          // padded genealogies (g >= G) screen to 0 and must not count
          if (gc + ACC_N <= S.G) {
            mx = fmaxf(mx, fmaxf(m0, m1));
          } else {
            if (gc + c + 32 <= S.G) mx = fmaxf(mx, m0);
            if (gc + c + 64 <= S.G) mx = fmaxf(mx, m1);
          }
          continue;
        }
        if (raise) {
          if (gc + c + 32 <= S.G) lb = fmaxf(lb, m0 - err);
          if (gc + c + 64 <= S.G) lb = fmaxf(lb, m1 - err);
          if (live) thr = lb - (err + SURF_MARGIN);
        }
        if (!__any_sync(0xffffffffu, fmaxf(m0, m1) > thr)) continue;
#pragma unroll
        for (int j = 0; j < 2; j++) {
          if (!__any_sync(0xffffffffu, __uint_as_float(m[j]) > thr)) continue;
          unsigned mask = 0;
#pragma unroll
          for (int b = 0; b < 32; b++)
            if (__uint_as_float(r[j][b]) > thr) mask |= 1u << b;
          const int gj = gc + c + 32 * j, nv = S.G - gj;
          if (nv < 32) mask &= nv > 0 ? (1u << nv) - 1u : 0u;
          ring.put(sh, gerr, ew, lane, pl, gj, mask);
        }
      }
    }
    if (MAXONLY) lb = fmaxf(lb, mx - err);
    // the pre-pass publishes its bound once: a maximum, whatever the order
    if (MAXONLY && live) atomicMax(&S.best[p], f2ord(lb));
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();
      atomicAdd(&sh.epi_done, 1);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 512);
  }
  if (threadIdx.x < TC_M && !MAXONLY) {
    const int p = ptile * TC_M + threadIdx.x;
    const bool mine = p < npoints && !(dense && dense[p]);
    if (mine) atomicMax(&S.xmax[p], sh.xmax[threadIdx.x]);
    if (mine)
      part[(size_t)p * SURF_MAX_CHUNKS + blockIdx.y] =
          make_double2(sh.ovf[threadIdx.x] ? -1.0 : fixw_to_double(sh.sum[threadIdx.x]),
                       fixw_to_double(sh.sum2[threadIdx.x]));
  }
}

// Chunk sums added in chunk order: q = ln G - (ref + ln sum).  A point with
// a flagged chunk goes to the list of points to take again (flag[0] = list
// length, flag[1..] = points; the list's order does not matter, each point
// is taken on its own).
__global__ void k_surf_tc_merge(SurfArgs a, SurfPrep S, const double2 *part, int nchunks, const uint8_t *dense,
                                const int *counts, int dense_blocks, int *flag)
{
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.npoints) return;
  const double2 *w = part + (size_t)p * SURF_MAX_CHUNKS;
  int per;
  if (dense && dense[p]) nchunks = surf_dense_chunks(counts[0], dense_blocks, a.G, &per);
  double s = 0.0, s2 = 0.0;
  int ovf = 0;
  for (int c = 0; c < nchunks; c++) {
    if (w[c].x < 0.0) ovf = 1;
    s += w[c].x;
    s2 += w[c].y;
  }
  if (ovf) {
    flag[1 + atomicAdd(&flag[0], 1)] = p;
    return;
  }
  const double ref = (double)ord2f(S.best[p]);
  a.q[p] = log((double)a.G) - (ref + log(s));
  if (a.ess) a.ess[p] = s * s / s2;
}

// The flagged points as a problem of their own: their coordinates and, as
// the reference, the largest exact value the first pass met.
__global__ void k_surf_tc_gather(const double *x, int npar, const unsigned *xmax, const int *flag, double *xs,
                                 unsigned *refs)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= flag[0]) return;
  const int p = flag[1 + k];
  for (int j = 0; j < npar; j++) xs[(size_t)k * npar + j] = x[(size_t)p * npar + j];
  refs[k] = xmax[p];
}

__global__ void k_surf_tc_setref(unsigned *best, unsigned *xmax, const unsigned *refs, int n)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) best[k] = xmax[k] = refs[k];
}

__global__ void k_surf_tc_scatter(const int *flag, const double *qs, const double *es, double *q, double *ess)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= flag[0]) return;
  const int p = flag[1 + k];
  q[p] = qs[k];
  if (ess) ess[p] = es[k];
}

// ------------------------------------------------------------ self-test
// One 128 x 256 x 32 tile of small integers (exact in FP16 and FP32),
// checked element by element against CUDA cores.
__global__ void __launch_bounds__(128, 1) k_tc_selftest(const uint16_t *A, const uint16_t *B, float *D,
                                                         int *err)
{
  extern __shared__ __align__(1024) char smem[];
  char *bufA = smem, *bufB = smem + A_BYTES;
  __shared__ uint64_t bar, mbar;
  __shared__ uint32_t tslot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tc::mbar_init(&bar, 1);
    tc::mbar_init(&mbar, 1);
    tc::fence_barrier_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(&tslot, 256);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tslot;
  __shared__ int ok;
  if (threadIdx.x == 0) {
    ok = 1;
    tc::mbar_expect_tx(&bar, A_BYTES + B_BYTES);
    tc::bulk_g2s(bufA, A, A_BYTES, &bar);
    tc::bulk_g2s(bufB, B, B_BYTES, &bar);
    if (!tc::mbar_wait(&bar, 0, WAIT_LIMIT)) {
      ok = 0;
      atomicCAS(err, 0, 1);
    } else {
      tc::fence_after_sync();
      const uint32_t idesc = tc::idesc_f16_f32(TC_M, TC_N);
      const uint32_t aa = tc::smem_u32(bufA), bb = tc::smem_u32(bufB);
      for (int kh = 0; kh < 2; kh++)
        tc::mma_f16(tmem, tc::sdesc(aa + kh * 256, 128, 512), tc::sdesc(bb + kh * 256, 128, 512), idesc, kh);
      tc::mma_commit(&mbar);
    }
  }
  __syncthreads();
  if (ok) {
    if (!tc::mbar_wait(&mbar, 0, WAIT_LIMIT)) {
      atomicCAS(err, 0, 2);
    } else {
      tc::fence_after_sync();
      const int row = warp * 32 + lane;
      for (int c = 0; c < TC_N / 32; c++) {
        float v[32];
        tc::tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c * 32), v);
        for (int j = 0; j < 32; j++) D[(size_t)row * TC_N + c * 32 + j] = v[j];
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 256);
  }
}

__device__ __forceinline__ int st_a(int r, int k) { return ((r * 7 + k * 3) % 17) - 8; }
__device__ __forceinline__ int st_b(int n, int k) { return ((n * 5 + k * 11) % 13) - 6; }

__global__ void k_tc_selftest_fill(uint16_t *A, uint16_t *B)
{
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < TC_M * SURF_KP) {
    int r = i / SURF_KP, k = i % SURF_KP;
    const __half v = __float2half_rn((float)st_a(r, k));
    *reinterpret_cast<__half *>(reinterpret_cast<char *>(A) + tc::tile_off(r, k)) = v;
  }
  if (i < TC_N * SURF_KP) {
    int n = i / SURF_KP, k = i % SURF_KP;
    const __half v = __float2half_rn((float)st_b(n, k));
    *reinterpret_cast<__half *>(reinterpret_cast<char *>(B) + tc::tile_off(n, k)) = v;
  }
}

__global__ void k_tc_selftest_check(const float *D, int *bad, float *maxerr)
{
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= TC_M * TC_N) return;
  int r = i / TC_N, n = i % TC_N;
  int want = 0;
  for (int k = 0; k < SURF_KP; k++) want += st_a(r, k) * st_b(n, k);
  float e = fabsf(D[i] - (float)want);
  if (e != 0.f) atomicAdd(bad, 1);
  atomicMax(reinterpret_cast<int *>(maxerr), __float_as_int(e));
}

}  // namespace

// ---------------------------------------------------------------- host
size_t surface_tc_scratch_bytes(int G, int npoints)
{
  // prepared operands | chunk sums (double2 per point and chunk) | the list
  // of points to retake (a count, then points) | their coordinates,
  // references, densities, sample sizes and the retake's own list | how each
  // point is taken (SurfSplit: counts, list, flags)
  const size_t np = (size_t)npoints;
  return surf_prep_bytes(G, npoints) + np * SURF_MAX_CHUNKS * sizeof(double2) + 2 * (np + 1) * sizeof(int) +
         np * (SURF_K / 2) * sizeof(double) + np * sizeof(unsigned) + 2 * np * sizeof(double) +
         (1 + np / TC_M + 1 + np) * sizeof(int) + np + 4096;
}

namespace {

constexpr int SEED_TC = 32;    // exact samples per point before the pre-pass (one per lane)

// genealogy chunks for a pass over `ntiles` tiles: one CTA holds an SM, so
// pick the chunk count whose CTA total fills its last wave best (at least
// 8 tiles per CTA); returns the chunk count, tiles per chunk in *per
int surf_tc_chunks(int ptiles, int ntiles, int nsm, int *per)
{
  const int maxch = std::max(1, std::min(SURF_MAX_CHUNKS, ntiles / 8));
  int nchunks = 1;
  *per = ntiles;
  double best_eff = -1.0;
  for (int c = 1; c <= maxch; c++) {
    const int pc = (ntiles + c - 1) / c, cc = (ntiles + pc - 1) / pc;
    const double waves = (double)ptiles * cc / nsm;
    const double eff = waves / std::ceil(waves);
    if (eff > best_eff + 0.02) {  // fewer chunks unless clearly better filled
      best_eff = eff;
      nchunks = cc;
      *per = pc;
    }
  }
  return nchunks;
}

}  // namespace

// One evaluation of the points of `a` on prepared operands S: the optional
// max-only pre-pass, the choice between the screen and the direct form per
// point (D null: the screen for all), the full pass, the direct form and the
// merge; returns the kernels queued.
static int tc_passes(const SurfArgs &a, const SurfPrep &S, const SurfSplit *D, double2 *part, int *flag, int *d_err,
                     int nsm, bool pre, cudaStream_t st)
{
  const float2 *etab = surf_exp_table();
  const int ntiles = S.Gpad / TC_N;
  const int ptiles = (a.npoints + TC_M - 1) / TC_M;
  int per = 0, nk = 0;
  const int nchunks = surf_tc_chunks(ptiles, ntiles, nsm, &per);
  if (pre) {
    k_surf_tc<true><<<dim3(ptiles, nchunks), TC_THREADS, TC_SMEM, st>>>(S, a.npoints, per, false, etab, nullptr, nullptr,
                                                                        part, d_err);
    nk++;
  }
  const uint8_t *dense = nullptr;
  const int *counts = nullptr;
  int db = 0;
  if (D) {
    dense = D->dense;
    counts = D->counts;
    db = surf_dense_grid(a, nsm);
    surf_split(S, a.npoints, *D, st);
    surf_dense(a, S, *D, db, part, st);
    nk += 2;
  }
  k_surf_tc<false><<<dim3(ptiles, nchunks), TC_THREADS, TC_SMEM, st>>>(S, a.npoints, per, !pre, etab,
                                                                dense, counts ? counts + 1 : nullptr, part, d_err);
  k_surf_tc_merge<<<(a.npoints + 127) / 128, 128, 0, st>>>(a, S, part, nchunks, dense, counts, db, flag);
  return nk + 2;
}

int launch_surface_tc(const SurfArgs &a, void *scratch, size_t scratch_bytes, int *d_err, bool rows_ready,
                      int *nkernels, int *nretaken, cudaStream_t st)
{
  if (a.np + a.nm > SURF_K / 2) return 2;
  if (scratch_bytes < surface_tc_scratch_bytes(a.G, a.npoints)) return 3;
  if (a.G >= (1 << 24)) return 4;  // candidate entries pack the genealogy index into 24 bits
  const size_t np = (size_t)a.npoints;
  const int npar = a.np + a.nm;
  char *base = static_cast<char *>(scratch);
  SurfPrep S;
  double2 *part = reinterpret_cast<double2 *>(surf_prep_carve(&S, base, a.G, a.npoints));
  // the retake's buffers sit past everything the first evaluation uses
  int *flag = reinterpret_cast<int *>(part + np * SURF_MAX_CHUNKS);
  double *xs = reinterpret_cast<double *>(
      (reinterpret_cast<uintptr_t>(flag + np + 1) + 255) & ~static_cast<uintptr_t>(255));
  unsigned *refs = reinterpret_cast<unsigned *>(xs + np * (SURF_K / 2));
  double *qs = reinterpret_cast<double *>((reinterpret_cast<uintptr_t>(refs + np) + 255) & ~static_cast<uintptr_t>(255));
  double *es = qs + np;
  int *flag2 = reinterpret_cast<int *>(es + np);  // the retake's own list (always empty)
  SurfSplit D;
  D.counts = flag2 + np + 1;
  D.list = D.counts + 2 + np / TC_M;
  D.dense = reinterpret_cast<uint8_t *>(D.list + np);
  static_assert(A_BYTES + TC_STAGES * B_BYTES + sizeof(TcSmem) + 1024 <= TC_SMEM, "smem");
  cudaFuncSetAttribute(k_surf_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM);
  cudaFuncSetAttribute(k_surf_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM);
  int nsm = 152;
  {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  }
  SurfZero z;
  z.z0 = flag;
  z.n0 = 1;
  z.z1 = D.counts;
  z.n1 = 1 + (a.npoints + TC_M - 1) / TC_M;
  int nk = surf_prep(a, S, true, rows_ready, SEED_TC, z, st);
  // a max-only pre-pass gives every point a lower bound at (or near) its
  // screened maximum before the full pass
  const bool pre = S.Gpad / TC_N >= 4;
  nk += tc_passes(a, S, &D, part, flag, d_err, nsm, pre, st);
  // points whose terms left the fixed-point range: a second evaluation of
  // just them, referenced to their exact maxima
  int nflag = 0;
  if (cudaMemcpyAsync(&nflag, flag, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return 5;
  *nretaken = nflag;
  if (nflag > 0) {
    k_surf_tc_gather<<<(nflag + 127) / 128, 128, 0, st>>>(a.x, npar, S.xmax, flag, xs, refs);
    SurfArgs b = a;
    b.npoints = nflag;
    b.x = xs;
    b.q = qs;
    b.ess = a.ess ? es : nullptr;
    SurfPrep S2;
    double2 *part2 = reinterpret_cast<double2 *>(surf_prep_carve(&S2, base, a.G, nflag));
    SurfZero z2;
    z2.z0 = flag2;
    z2.n0 = 1;
    surf_prep(b, S2, true, true, 0, z2, st);
    k_surf_tc_setref<<<(nflag + 127) / 128, 128, 0, st>>>(S2.best, S2.xmax, refs, nflag);
    nk += 3 + tc_passes(b, S2, nullptr, part2, flag2, d_err, nsm, false, st);
    k_surf_tc_scatter<<<(nflag + 127) / 128, 128, 0, st>>>(flag, qs, es, a.q, a.ess);
    nk++;
  }
  *nkernels = nk;
  return 0;
}

int tc_selftest(cudaStream_t st, void *scratch, size_t bytes, int *h_bad, float *h_maxerr)
{
  // scratch: A (8 KB) | B (16 KB) | D (128 KB) | bad, maxerr, err
  const size_t need = A_BYTES + B_BYTES + (size_t)TC_M * TC_N * 4 + 16;
  if (bytes < need) return 3;
  char *p = static_cast<char *>(scratch);
  uint16_t *A = reinterpret_cast<uint16_t *>(p);
  uint16_t *B = reinterpret_cast<uint16_t *>(p + A_BYTES);
  float *D = reinterpret_cast<float *>(p + A_BYTES + B_BYTES);
  int *bad = reinterpret_cast<int *>(p + A_BYTES + B_BYTES + (size_t)TC_M * TC_N * 4);
  float *mx = reinterpret_cast<float *>(bad + 1);
  int *err = bad + 2;
  cudaMemsetAsync(p, 0, need, st);
  k_tc_selftest_fill<<<(TC_N * SURF_KP + 255) / 256, 256, 0, st>>>(A, B);
  const size_t sm = A_BYTES + B_BYTES + 1024;
  cudaFuncSetAttribute(k_tc_selftest, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_tc_selftest<<<1, 128, sm, st>>>(A, B, D, err);
  k_tc_selftest_check<<<(TC_M * TC_N + 255) / 256, 256, 0, st>>>(D, bad, mx);
  int out[3];
  cudaMemcpyAsync(out, bad, sizeof(out), cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) return 4;
  *h_bad = out[2] ? -out[2] : out[0];
  memcpy(h_maxerr, &out[1], sizeof(float));
  return 0;
}
