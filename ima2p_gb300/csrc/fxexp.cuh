// fxexp.cuh -- 2^a in fixed point on the integer pipe, and sums of such
// values, for loops that are bound by FP64 exponentials: GB300 runs FP64
// (and FP64 conversions) at 1/64 of the FP32 rate, 32-bit integer multiplies
// at a quarter.  The argument stays FP64 and exact; the value carries 63
// bits with a relative error below 2^-53.
#pragma once
#include <cstdint>

namespace {

constexpr int FX_TAB = 512;  // 2^(j / 512) for j < FX_TAB, as 2^63 times the value, truncated

// 2^(rho / 512) - 1 = 2^-9 rho (L1 + rho (L2 + rho (L3 + rho L4))), rho in
// [0, 1): interpolation at four Chebyshev nodes, within 2^-61
constexpr uint64_t FX_L1 = 0xb17217f7d1cf6ebeull;  // 2^64
constexpr uint64_t FX_L2 = 0x1ebfbdff84233eull;    // 2^64
constexpr uint32_t FX_L3 = 3814212867u;            // 2^54
constexpr uint32_t FX_L4 = 1291623u;               // 2^54

#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint32_t fx_mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
__device__ __forceinline__ uint64_t fx_bits(double a) { return (uint64_t)__double_as_longlong(a); }
#else
inline uint32_t fx_mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline uint64_t fx_bits(double a)
{
  uint64_t u;
  __builtin_memcpy(&u, &a, 8);
  return u;
}
#endif

// a x b / 2^32 of a 64-bit a = (ah, al) and 32-bit b, truncated
__host__ __device__ __forceinline__ uint64_t fx_mul64(uint64_t a, uint32_t b)
{
  return (uint64_t)(uint32_t)(a >> 32) * b + fx_mulhi((uint32_t)a, b);
}

// a in fixed point with 53 fraction bits, |a| < 1000 (exact for |a| >= 1/2,
// within 2^-54 below)
__host__ __device__ __forceinline__ int64_t fx_fix(double a)
{
  const uint64_t b = fx_bits(a);
  const int hi = (int)(b >> 32);
  const uint64_t man = (b << 11) | (1ull << 63);
  int sh = 1033 - ((hi >> 20) & 0x7ff);  // 10 - E
  sh = sh < 63 ? sh : 63;
  const uint64_t v = man >> sh;
  return (int64_t)(hi < 0 ? 0ull - v : v);
}

// 2^(v 2^-53) = m 2^(i - 63), m in [2^63, 2^64)
__host__ __device__ __forceinline__ uint64_t fx_exp2(int64_t v, const uint64_t *tab, int *i)
{
  const int vh = (int)(v >> 32);
  *i = vh >> 21;
  const uint64_t T = tab[(vh >> 12) & (FX_TAB - 1)];
  const uint64_t rho = (uint64_t)v << 20;  // the low 44 bits: rho in [0, 1), 2^64
  const uint32_t r = (uint32_t)(rho >> 32), rl = (uint32_t)rho;
  const uint32_t g3 = FX_L3 + fx_mulhi(r, FX_L4);
  const uint64_t g2 = FX_L2 + ((uint64_t)fx_mulhi(r, g3) << 10);
  const uint64_t g1 = FX_L1 + fx_mul64(g2, r) + fx_mulhi((uint32_t)(g2 >> 32), rl);
  const uint64_t z = fx_mul64(g1, r) + fx_mulhi((uint32_t)(g1 >> 32), rl);
  const uint64_t y = fx_mul64(z, (uint32_t)(T >> 32)) + fx_mulhi((uint32_t)(z >> 32), (uint32_t)T);
  return T + (y >> 9);
}

// A sum of values m 2^(i - 63): 96 bits below 2^9 times the largest term, so
// 512 terms fit and each is truncated below 2^-86 of the largest.  A term
// that exceeds the largest so far moves the sum to the FP64 total first.
struct FxSum {
  uint32_t w0, w1, w2;
  int top;       // exponent of the largest term
  double total;  // what was moved out
#ifdef __CUDACC__
  __device__ __forceinline__ void init()
  {
    w0 = w1 = w2 = 0u;
    top = -100000;
    total = 0.0;
  }
  // to be called at least once every 512 terms
  __device__ __forceinline__ void flush()
  {
    if (w0 | w1 | w2) {
      const double v = (double)w2 * 18446744073709551616.0 + (double)(((uint64_t)w1 << 32) | w0);
      total += scalbn(v, top - 86);
    }
    w0 = w1 = w2 = 0u;
  }
  __device__ __forceinline__ void add(uint64_t m, int i)
  {
    if (i > top) {
      flush();
      top = i;
    }
    uint32_t a2 = (uint32_t)(m >> 32), a1 = (uint32_t)m, a0 = 0u;
    int s = top - i + 9;
    if (s >= 32) {
      a0 = a1;
      a1 = a2;
      a2 = 0u;
      s -= 32;
      if (s >= 32) {
        a0 = a1;
        a1 = 0u;
        s -= 32;
        if (s >= 32) return;  // below 2^-86 of the largest
      }
    }
    a0 = __funnelshift_r(a0, a1, s);
    a1 = __funnelshift_r(a1, a2, s);
    a2 >>= s;
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(w0), "+r"(w1), "+r"(w2) : "r"(a0), "r"(a1), "r"(a2));
  }
#endif
};

}  // namespace
