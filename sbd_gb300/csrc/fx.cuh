// Fixed-point arithmetic for FP64 sums of products.
//
// On this GPU an FP64 multiply-add issues at 2 per clock and SM, a 32 x 32 ->
// 64-bit integer multiply-add at 32 of unsigned operands (measured 1.97 and 29.4;
// signed ones, which these are, 19.0 as compiled).  A sum over a pair list whose
// operands are integers on a common scale takes three of the latter per term:
//
//   X = round(x 2^(55 - ex)), |x| < 2^ex for every x of the sum
//   V = round(v 2^(57 - ev)),  |v| < 2^ev for every v of the table
//
// each split into a high and a 27-bit low part, and the partial products but
// low x low are added exactly, so a sum's value does not depend on the order of
// its terms.  A term's error is that of the two conversions (2^-56 of the
// largest |x| of the sum, 2^-58 of the largest |v|) and the product left out
// (2^-59 of the largest |x| times the largest |v|, of either sign; 2^-58 where v is
// a sum of two); an FP64 sum's is 2^-53 of each partial sum.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#ifdef __CUDACC__
#include "df.cuh"
#endif

namespace sbdgb {
namespace fx {

constexpr int kXBits = 55, kVBits = 57;  // |X| <= 2^55, |V| <= 2^57
constexpr int kLow = 27;                 // bits of the low parts
constexpr int kMaxTerms = 4096;          // terms of one sum
constexpr int kZero = -(1 << 20);        // exponent of an all-zero vector
constexpr int kBad = 1 << 20;            // exponent of one that is not finite, or too large or small
constexpr int kMaxExp = 800;             // |exponent| of the operands that this arithmetic takes

// ex with |x| < 2^ex, for the largest high word (sign bit cleared) of a set of
// doubles; kZero and kBad as above.
__host__ __device__ __forceinline__ int exponent_of(uint32_t hi, bool nonzero) {
  if (!nonzero) return kZero;
  const int e = (int)(hi >> 20) - 1022;
  return (e > kMaxExp || e < -kMaxExp) ? kBad : e;
}

// round(x 2^s) for |x 2^s| <= 2^57 (half away from zero).
__device__ __forceinline__ long long from_double(double x, int s) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)(b >> 52) & 0x7ff;
  unsigned long long m = b & 0xfffffffffffffull;
  if (e) m |= 1ull << 52;
  const int sh = (e ? e : 1) - 1075 + s;
  if (sh >= 0)
    m <<= sh;
  else
    m = sh > -63 ? (m + (1ull << (-sh - 1))) >> -sh : 0ull;
  return (long long)b < 0 ? -(long long)m : (long long)m;
}
// A table value's (high, low) parts: value = high 2^27 + low, |low| <= 2^26.
__device__ __forceinline__ int2 split(long long v) {
  const int lo = (int)((uint32_t)v << (32 - kLow)) >> (32 - kLow);
  return make_int2((int)((v - lo) >> kLow), lo);
}
__device__ __forceinline__ int2 make(double x, int s) { return split(from_double(x, s)); }

// A vector element's parts, both with its sign (|low| < 2^27), from the words of
// a double and the exponent of its sum, rounded half away from zero.  32-bit
// shifts only (about 22 instructions; the general conversion above takes twice
// that).
__device__ __forceinline__ int2 vector_parts(uint32_t lo, uint32_t hi, int ex) {
  const int e = (int)(hi >> 20) & 0x7ff;  // a subnormal is shifted out whatever its leading bit
  const uint32_t a1 = ((hi & 0xfffffu) | 0x100000u) << 3 | lo >> 29, a0 = lo << 3;  // 56 bits
  const uint32_t d = (uint32_t)min(ex + 1022 - e, 62);                              // 0 for the largest binade
  const uint32_t d1 = min(d, 31u), d2 = d - d1;
  const uint32_t b0 = __funnelshift_r(a0, a1, d1), b1 = a1 >> d1;
  const unsigned long long c =
      ((unsigned long long)(b1 >> d2) << 32 | __funnelshift_r(b0, b1, d2)) + 1ull;  // one bit below the unit
  const int s = (int)hi >> 31;
  const int h = (int)(uint32_t)(c >> (kLow + 1)), l = (int)((uint32_t)(c >> 1) & ((1u << kLow) - 1u));
  return make_int2((h ^ s) - s, (l ^ s) - s);
}

#ifdef __CUDACC__
// A double-float's, from the bits of hi and lo: their integers on the sum's
// scale, added (|hi| + |lo| < 2^ex).
__device__ __forceinline__ int2 vector_parts_df(uint32_t lo, uint32_t hi, int ex) {
  auto fixed = [&](uint32_t b) {
    const int e = (int)(b >> 23) & 0xff;
    const unsigned long long m = (unsigned long long)((b & 0x7fffffu) | (e ? 0x800000u : 0u)) << 32;
    const int d = min(ex + 126 - max(e, 1), 62);  // 2^32 m: 56 bits, the last one below the unit, for e = ex + 126
    const long long v = (long long)(m >> d);
    return (int)b < 0 ? -v : v;
  };
  return split((fixed(hi) + fixed(lo) + 1) >> 1);
}
#endif

// A sum: (m + hh 2^27 + top 2^59) 2^27.
struct Acc {
  long long m, hh, top;
};
__device__ __forceinline__ void zero(Acc &a) { a.m = a.hh = a.top = 0; }
__device__ __forceinline__ void mac(Acc &a, int xh, int xl, int vh, int vl) {
  a.hh += (long long)xh * vh;
  a.m += (long long)xh * vl;
  a.m += (long long)xl * vh;
}
// Carries.  A term is at most 2^58 in hh and 2^55 + 2^57 in m (where V may be a
// sum of two, |low| <= 2^27): carry_high() at least every 16 terms, carry() at
// least every 32.
constexpr int kChunkHigh = 16, kChunk = 32;
__device__ __forceinline__ void carry_high(Acc &a) {
  a.top += a.hh >> 32;
  a.hh &= 0xffffffffll;
}
__device__ __forceinline__ void carry(Acc &a) {
  a.hh += a.m >> kLow;
  a.m &= (1ll << kLow) - 1;
  carry_high(a);
}
constexpr int kUnit = kLow - kXBits - kVBits;  // a sum's value is its integer times 2^(ex + ev + kUnit)

// |a| (after carry()) with its leading one in bit 63, the rest cut off: the sign
// in neg, that bit's exponent in top.  0 for a zero sum.
__device__ __forceinline__ unsigned long long normalised(const Acc &a, bool &neg, int &top) {
  // 128-bit two's complement (hi, lo)
  unsigned long long lo =
      (unsigned long long)a.m | ((unsigned long long)a.hh << kLow) | ((unsigned long long)a.top << (kLow + 32));
  unsigned long long hi = (unsigned long long)(a.top >> (32 - kLow));
  neg = (long long)hi < 0;
  if (neg) {
    lo = ~lo + 1ull;
    hi = ~hi + (lo == 0ull ? 1ull : 0ull);
  }
  top = 127;
  if (hi == 0ull) {
    hi = lo;
    lo = 0ull;
    top = 63;
  }
  if (hi == 0ull) return 0ull;
  const int lz = __clzll((long long)hi);
  top -= lz;
  return lz ? hi << lz | lo >> (64 - lz) : hi;
}
// A sum's value times 2^e, rounded to FP64 (integer instructions only: a
// conversion of a 64-bit integer costs an FP64 issue).
__device__ __forceinline__ double value(const Acc &a, int e) {
  bool neg;
  int top;
  const unsigned long long t = normalised(a, neg, top);
  if (t == 0ull) return 0.0;
  const unsigned long long mant = (t >> 11) + ((t >> 10) & 1ull);  // 53 bits, or 2^53 after rounding up
  const unsigned long long bits = ((unsigned long long)(1022 + top + e) << 52) + mant;
  return __longlong_as_double((long long)(bits | (neg ? 1ull << 63 : 0ull)));
}
#ifdef __CUDACC__
// x 2^k in two steps, so that no factor leaves FP32's range where the result does not.
__device__ __forceinline__ float scaled(float x, int k) {
  k = max(-250, min(250, k));
  const int h = k >> 1;
  return x * __int_as_float((h + 127) << 23) * __int_as_float((k - h + 127) << 23);
}
// The same as a double-float: 24 bits in hi, the next 31 in lo.
__device__ __forceinline__ dfloat value_df(const Acc &a, int e) {
  bool neg;
  int top;
  const unsigned long long t = normalised(a, neg, top);
  if (t == 0ull) return dfloat(0.f, 0.f);
  int h = (int)(t >> 40), l = (int)((uint32_t)(t >> 8) >> 1);  // l: 31 bits below h's last
  if (l >> 30) {  // nearest: lo may be negative
    h += 1;
    l = -(int)((1u << 31) - (uint32_t)l);
  }
  if (neg) {
    h = -h;
    l = -l;
  }
  const int k = top + e - 23;
  return dfloat(scaled((float)h, k), scaled((float)l, k - 31));
}
#endif

}  // namespace fx
}  // namespace sbdgb
