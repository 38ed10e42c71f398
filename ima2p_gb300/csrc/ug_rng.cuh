// ug_rng.cuh -- a chain's generators for the genealogy-update kernels
// (k_updgen.cu): the reference's uniform() (MT19937, utilities.cpp:323-427)
// and bitran (:438-455), staged for one kernel.
#pragma once

#include "internal.h"

namespace {

// The chain's generators for one kernel: MT19937 (Matsumoto & Nishimura
// 1998) with its 624 words in shared memory and the rest in thread 0's
// registers, so that a draw costs a shared-memory read, not a dependent
// round trip to global memory.  The threads that load it twist the state once ahead into a
// second set of words, 227 at a time (word k needs words k, k + 1 and k + 397
// of the old state, or k - 227 of the new): thread 0 by itself takes 18 us
// for the 624.
struct LocalRng {
  uint32_t *mt;    // [2][624]
  int mti, iset;
  double gset;
  unsigned long long iseed;
  int twists;      // since the load
  // the next draws, made beforehand (rng_ahead): the deviate of word i, its
  // logarithm, and the polar method's two normal deviates from words i and
  // i + 1 (both 0: outside the circle)
  int at, ahead;   // words drawn; words made
  const double *u, *lu, *v1, *v2;
};

constexpr int RNG_N = 624, RNG_M = 397;

__device__ __forceinline__ uint32_t mt_mix(uint32_t a, uint32_t b, uint32_t far)
{
  const uint32_t y = (a & 0x80000000u) | (b & 0x7fffffffu);
  return far ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
}

// barrier number 1 for nt threads, whole warps
__device__ __forceinline__ void rng_barrier(int nt) { asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory"); }

// nt threads, tid of them; smt: 2 x 624 words
__device__ void rng_load(LocalRng &r, const ima_ug_rng *g, uint32_t *smt, int tid, int nt)
{
  const uint2 *src = reinterpret_cast<const uint2 *>(g->mt.mt);  // the state is 8-byte aligned
  uint2 *dst = reinterpret_cast<uint2 *>(smt);
  for (int k = tid; k < RNG_N / 2; k += nt) dst[k] = src[k];
  r.mt = smt;
  r.mti = (int)min((unsigned)g->mt.mti, (unsigned)RNG_N);  // a count outside the state: all words are drawn
  r.iset = g->iset;
  r.gset = g->gset;
  r.iseed = g->iseed;
  r.twists = 0;
  r.at = r.ahead = 0;
  rng_barrier(nt);
  uint32_t *nx = smt + RNG_N;
  constexpr int D = RNG_N - RNG_M;  // 227
  for (int b = 0; b < RNG_N; b += D) {
    for (int k = b + tid; k < min(b + D, RNG_N); k += nt)
      nx[k] = mt_mix(smt[k], k + 1 < RNG_N ? smt[k + 1] : nx[0], k < D ? smt[k + RNG_M] : nx[k - D]);
    rng_barrier(nt);
  }
}

// the CTA writes the generator back, after a barrier: thread 0's registers,
// and the words when thread 0 moved to the next state
__device__ void rng_store(const LocalRng &r, ima_ug_rng *g, const int *twists, int tid, int nt)
{
  if (*twists) {
    const uint2 *src = reinterpret_cast<const uint2 *>(r.mt + (*twists & 1 ? RNG_N : 0));
    uint2 *dst = reinterpret_cast<uint2 *>(g->mt.mt);
    for (int k = tid; k < RNG_N / 2; k += nt) dst[k] = src[k];
  }
  if (tid == 0) {
    g->mt.mti = r.mti;
    g->iset = r.iset;
    g->gset = r.gset;
    g->iseed = r.iseed;
  }
}

__device__ __forceinline__ uint32_t mt_temper(uint32_t y)
{
  y ^= y >> 11;
  y ^= (y << 7) & 0x9d2c5680u;
  y ^= (y << 15) & 0xefc60000u;
  y ^= y >> 18;
  return y;
}
// genrand_real3, in (0, 1)
__device__ __forceinline__ double mt_real3(uint32_t y) { return ((double)y + 0.5) * (1.0 / 4294967296.0); }

// the nt threads make the next `words` (< 624) draws, a thread each, after
// rng_load: four FP64 functions that would follow one another in the thread
// that draws.  buf: 4 x words
__device__ void rng_ahead(LocalRng &r, double *buf, int words, int tid, int nt)
{
  for (int i = tid; i < words; i += nt) {
    const double u1 = mt_real3(mt_temper(r.mt[r.mti + i])), u2 = mt_real3(mt_temper(r.mt[r.mti + i + 1]));
    const double v1 = 2.0 * u1 - 1.0, v2 = 2.0 * u2 - 1.0, rsq = v1 * v1 + v2 * v2;
    double w1 = 0.0, w2 = 0.0;
    if (!(rsq >= 1.0 || rsq == 0.0)) {
      const double fac = sqrt(-2.0 * log(rsq) / rsq);
      w1 = v1 * fac;
      w2 = v2 * fac;
    }
    buf[i] = u1;
    buf[words + i] = log(u1);
    buf[2 * words + i] = w1;
    buf[3 * words + i] = w2;
  }
  r.u = buf;
  r.lu = buf + words;
  r.v1 = buf + 2 * words;
  r.v2 = buf + 3 * words;
  r.ahead = words;
}

// thread 0 only: the generator's next word, by its index in r.mt
__device__ int mt_step(LocalRng &r)
{
  r.at++;
  if (r.mti >= RNG_N) {
    // to the state made ahead; past that one (more than 624 draws in one
    // launch), over the words that are done with
    const uint32_t *mt = r.mt + (r.twists & 1 ? RNG_N : 0);
    uint32_t *nx = r.mt + (r.twists & 1 ? 0 : RNG_N);
    if (r.twists++ > 0)
      for (int k = 0; k < RNG_N; k++)
        nx[k] = mt_mix(mt[k], k + 1 < RNG_N ? mt[k + 1] : nx[0], k < RNG_N - RNG_M ? mt[k + RNG_M] : nx[k - (RNG_N - RNG_M)]);
    r.mti = 0;
  }
  return (r.twists & 1 ? RNG_N : 0) + r.mti++;
}

// uniform() = genrand_real3, in (0, 1)
__device__ double uniform(LocalRng &r)
{
  const int at = r.at, k = mt_step(r);
  return at < r.ahead ? r.u[at] : mt_real3(mt_temper(r.mt[k]));
}

// the word behind uniform()
__device__ uint32_t uniform_word(LocalRng &r) { return mt_temper(r.mt[mt_step(r)]); }

// log(uniform())
__device__ double log_uniform(LocalRng &r)
{
  if (r.at >= r.ahead) return log(uniform(r));
  const double v = r.lu[r.at];
  mt_step(r);
  return v;
}

// bitran (utilities.cpp:438-455): Press et al.'s irbit2 on its own register
__device__ int bitran(LocalRng &r)
{
  if (r.iseed & 131072ull) {
    r.iseed = ((r.iseed ^ 19ull) << 1) | 1ull;
    return 1;
  }
  r.iseed <<= 1;
  return 0;
}

}  // namespace
