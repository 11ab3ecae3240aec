// fp64_int.cuh -- correctly rounded FP64 multiplication and division on the integer pipes.
//
// GB300 runs 2 FP64 lanes per clock per SM against 64 integer lanes and 64 of 32 x 32 -> 64-bit
// IMAD, so a multiplication (about 22 integer instructions) or a division (about 50) costs
// less there than on the FP64 pipe (1 and 9-10 instructions of 16 clocks per warp and SM), and
// runs beside the FP64 additions that stay.  Both return exactly what IEEE round-to-nearest-even
// does, for operands within the exponent ranges that their callers check; the plain functions of
// 32- and 64-bit integers below also compile for the host, where a test holds them to the
// hardware's own results.
//  - Product: the 53-bit mantissas, aligned to the top of 64 bits, are multiplied exactly into
//    128 bits; the upper 64 are normalised by 0 or 1 bit and rounded on bit 11, the lower 64
//    only enter as a sticky bit.
//  - Quotient: long division in three digits (20, 16 and 16 bits) with an FP32 reciprocal of the
//    divisor (high-radix digit recurrence, as in Ercegovac and Lang, Division and Square Root,
//    1994), each remainder exact modulo 2^64; the last remainder decides the rounding.  A
//    quotient of two 53-bit integers is never a tie.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define LPM_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#include <cstring>
#define LPM_HD inline
#endif

namespace lpm {

constexpr uint32_t kBias20 = 1023u << 20;

// A nonzero normal double taken apart: the mantissa's upper 32 bits with the leading one at bit
// 31, its lower 21 bits, and the sign and biased exponent in the bits they have in the high word.
struct F64Parts {
  uint32_t lo, hi, x;
};

LPM_HD uint64_t f64_bits(double v) {
#ifdef __CUDA_ARCH__
  return static_cast<uint64_t>(__double_as_longlong(v));
#else
  uint64_t b;
  memcpy(&b, &v, 8);
  return b;
#endif
}

LPM_HD double f64_from(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
#else
  const uint64_t b = (static_cast<uint64_t>(hi) << 32) | lo;
  double v;
  memcpy(&v, &b, 8);
  return v;
#endif
}

// Whether 2^lo <= |v| < 2^(hi + 1) (false for zero, infinities and NaN).
LPM_HD bool f64_in_range(double v, int lo, int hi) {
  const int e = static_cast<int>((f64_bits(v) >> 52) & 0x7ffu) - 1023;
  return e >= lo && e <= hi;
}

LPM_HD bool f64_is_zero(double v) { return (f64_bits(v) << 1) == 0; }

// Zero or subnormal, tested on the exponent field: an integer test that stays one (a comparison
// of the whole value with zero compiles to an FP64 instruction).
LPM_HD bool f64_tiny(double v) { return (static_cast<uint32_t>(f64_bits(v) >> 32) & 0x7ff00000u) == 0; }

LPM_HD F64Parts f64_parts(double v) {
  const uint64_t b = f64_bits(v);
  const uint32_t h = static_cast<uint32_t>(b >> 32), l = static_cast<uint32_t>(b);
  F64Parts p;
  p.lo = l & 0x1fffffu;
  p.hi = static_cast<uint32_t>(b >> 21) | 0x80000000u;
  p.x = h & 0xfff00000u;
  return p;
}

// The double whose parts these are.
LPM_HD double f64_whole(const F64Parts& p) {
  return f64_from(p.x | ((p.hi >> 11) & 0xfffffu), (p.hi << 21) | p.lo);
}

// The second factor of a product: its parts with the exponent's bias taken off, so that the
// product's exponent field is one sum of three.
struct F64Factor {
  uint32_t lo, hi, x;
};

LPM_HD F64Factor f64_factor(const F64Parts& p) { return F64Factor{p.lo, p.hi, p.x - kBias20}; }
LPM_HD double f64_whole(const F64Factor& f) { return f64_whole(F64Parts{f.lo, f.hi, f.x + kBias20}); }

// The words of the double nearest a * b (round to nearest even), for nonzero normal factors with
// a normal product.  TIES = false leaves out the test for an exact half: such a product has 54
// significant bits, so the factors' mantissas (as 53-bit integers) end in 51 or 52 zeros together
// (f64_short tells a factor with 26 or more).
struct F64Words {
  uint32_t lo, hi;
};

template <bool TIES>
LPM_HD F64Words mul_words(const F64Parts& a, const F64Factor& b) {
  // a b = hi hi 2^42 + (hi lo + lo hi) 2^21 + lo lo; the middle sum stays below 2^55
  const uint64_t y = static_cast<uint64_t>(a.lo) * b.lo;
  uint64_t x = static_cast<uint64_t>(a.hi) * b.lo + static_cast<uint32_t>(y >> 21);
  x = static_cast<uint64_t>(a.lo) * b.hi + x;
  uint64_t u = static_cast<uint64_t>(a.hi) * b.hi + (x >> 21);
  // the leading one is at bit 63 (a product in [2, 4)) or 62
  const bool top = static_cast<int64_t>(u) < 0;
  const uint32_t half = top ? 0x400u : 0x200u, sh = top ? 11u : 10u;
  u += half;  // no carry out: a product in [2, 4) is below 4 - 2^-51
  F64Words r;
  const uint32_t ul = static_cast<uint32_t>(u), uh = static_cast<uint32_t>(u >> 32);
#ifdef __CUDA_ARCH__
  r.lo = __funnelshift_r(ul, uh, sh);
#else
  r.lo = static_cast<uint32_t>(u >> sh);
#endif
  if (TIES) {
    const uint32_t rest = (static_cast<uint32_t>(x) | static_cast<uint32_t>(y)) & 0x1fffffu;  // below bit 0 of u
    if (((ul & (2u * half - 1u)) | rest) == 0) r.lo &= ~1u;  // an exact half goes to even
  }
  // the leading one adds 1 to the exponent field (2 after rounding up to the next power); the
  // signs add modulo 2^32
  r.hi = (uh >> sh) + a.x + b.x;
  if (!top) r.hi -= 1u << 20;
  return r;
}

template <bool TIES>
LPM_HD double mul_rn_int(const F64Parts& a, const F64Factor& b) {
  const F64Words w = mul_words<TIES>(a, b);
  return f64_from(w.hi, w.lo);
}

// Whether a mantissa ends in 26 or more zeros.
LPM_HD bool f64_short(double v) { return (static_cast<uint32_t>(f64_bits(v)) & 0x3ffffffu) == 0; }

LPM_HD float rcp_fp32(float v) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
#else
  return 1.0f / v;
#endif
}

LPM_HD int32_t to_int_rn(float v) {
#ifdef __CUDA_ARCH__
  return __float2int_rn(v);
#else
  return static_cast<int32_t>(std::nearbyint(v));
#endif
}

// The quotient n / d rounded to the nearest double, as parts, for a nonzero numerator n (its parts) and a nonzero divisor d (its
// words), both normal and their exponents such that the quotient is normal.
// With N and D the 53-bit mantissas, N doubled if below D, the quotient is in [1, 2).  An FP32
// reciprocal y of D's leading 24 bits is within 2^-22 of 2^52 / D, so
//   q1 = round(2^20 N / D) within 0.5 + 2, R1 = 2^20 N - q1 D, |R1| < 2.5 D,
//   q2 = round(2^16 R1 / D) within 0.5 + 0.13, R2 = 2^16 R1 - q2 D, |R2| < 0.63 D,
//   q3 = round(2^16 R2 / D - 0.55) in (q - 1.1, q), R3 = 2^16 R2 - q3 D in (0, 1.1 D);
// 2^32 q1 + 2^16 q2 + q3, plus one when 2 R3 > D, is the nearest integer to 2^52 N / D.  The
// remainders fit in 56 bits, so arithmetic modulo 2^64 is exact.
LPM_HD F64Parts div_parts(const F64Parts& n, const F64Words& d) {
  const uint64_t D = (static_cast<uint64_t>((d.hi & 0xfffffu) | 0x100000u) << 32) | d.lo;
  uint64_t N = (static_cast<uint64_t>(n.hi) << 21) | n.lo;
  uint32_t x = n.x - (d.hi & 0xfff00000u) + kBias20;  // signs subtract modulo 2^32
  if (N < D) {
    N <<= 1;
    x -= 1u << 20;
  }
  const float y = rcp_fp32(static_cast<float>(static_cast<int32_t>(D >> 29)));  // 2^29 / D
  const int32_t q1 =
      to_int_rn(static_cast<float>(static_cast<int32_t>(N >> 29)) * (y * 1048576.0f));
  const uint64_t nd = 0 - D;
  const uint64_t r1 = (N << 20) + static_cast<uint64_t>(q1) * nd;
  const float ys = y * 524288.0f;  // 2^16 2^32 / 2^29
  const int32_t q2 = to_int_rn(static_cast<float>(static_cast<int32_t>(r1 >> 32)) * ys);
  const uint64_t r2 = (r1 << 16) + static_cast<uint64_t>(static_cast<int64_t>(q2)) * nd;
  const int32_t q3 = to_int_rn(static_cast<float>(static_cast<int32_t>(r2 >> 32)) * ys - 0.55f);
  const uint64_t r3 = (r2 << 16) + static_cast<uint64_t>(static_cast<int64_t>(q3)) * nd;
  uint64_t q = (static_cast<uint64_t>(q1) << 32) + static_cast<uint64_t>(static_cast<int64_t>(q2) * 65536) +
               static_cast<uint64_t>(static_cast<int64_t>(q3));
  if (static_cast<int64_t>(2 * r3) > static_cast<int64_t>(D)) ++q;
  // no carry to 2^53: a quotient in [1, 2) of N < 2 D is at most 2 - 2^-52
  return F64Parts{static_cast<uint32_t>(q) & 0x1fffffu, static_cast<uint32_t>(q >> 21), x};
}

LPM_HD double div_rn_int(const F64Parts& n, const F64Words& d) { return f64_whole(div_parts(n, d)); }

}  // namespace lpm
