// xg_dcmp.cuh — FP64 tests, signs and shared-divisor quotients that spare the
// FP64 pipe.
//
// GB300 issues an FP64 instruction to a sub-partition in 66 cycles however
// few lanes need it, a comparison (DSETP) included; the integer pipe takes
// one or two.  The comparisons of device models are therefore made on the
// bits, with IEEE's results for every operand (signed zeros equal, NaN
// unordered), and multiplication by a polarity of +-1 is a sign flip.
#pragma once

namespace xg {

__device__ __forceinline__ unsigned long long dbits(double x) { return (unsigned long long)__double_as_longlong(x); }
constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;
constexpr unsigned long long kSignBit = 0x8000000000000000ull;

// x > 0, x >= 0, x < 0, x <= 0, x != 0 (true for NaN), x == 0, finite
__device__ __forceinline__ bool gt0(double x) { return dbits(x) - 1ull < kInfBits; }
__device__ __forceinline__ bool lt0(double x) { return (dbits(x) ^ kSignBit) - 1ull < kInfBits; }
__device__ __forceinline__ bool ge0(double x) { return dbits(x) <= kInfBits || dbits(x) == kSignBit; }
__device__ __forceinline__ bool le0(double x) { return (dbits(x) ^ kSignBit) <= kInfBits || dbits(x) == 0ull; }
__device__ __forceinline__ bool ne0(double x) { return (dbits(x) << 1) != 0ull; }
__device__ __forceinline__ bool eq0(double x) { return (dbits(x) << 1) == 0ull; }
__device__ __forceinline__ bool finite_bits(double x) { return ((unsigned(__double2hiint(x)) >> 20) & 0x7ffu) != 0x7ffu; }

// The magnitude with its sign as a two's-complement number: ordered as the
// doubles are, both zeros 0, NaN outside +-kInfBits.
__device__ __forceinline__ long long dkey(double x) {
  const long long v = __double_as_longlong(x), m = v >> 63;
  return (v ^ (m & 0x7fffffffffffffffll)) - m;
}
__device__ __forceinline__ bool lt(double a, double b) {
  const long long x = dkey(a), y = dkey(b);
  return x < y && x >= -(long long)kInfBits && y <= (long long)kInfBits;
}
__device__ __forceinline__ bool le(double a, double b) {
  const long long x = dkey(a), y = dkey(b);
  return x <= y && x >= -(long long)kInfBits && y <= (long long)kInfBits;
}
__device__ __forceinline__ bool gt(double a, double b) { return lt(b, a); }
__device__ __forceinline__ bool ge(double a, double b) { return le(b, a); }
// a != b (true for NaN)
__device__ __forceinline__ bool ne(double a, double b) {
  const long long x = dkey(a);
  return x != dkey(b) || x > (long long)kInfBits || x < -(long long)kInfBits;
}

__device__ __forceinline__ bool eq(double a, double b) { return !ne(a, b); }

// x or -x by a mask of 0 or kSignBit's high word
__device__ __forceinline__ double flip(double x, int sign) {
  return __hiloint2double(__double2hiint(x) ^ sign, __double2loint(x));
}
__device__ __forceinline__ double magnitude(double x) {
  return __hiloint2double(__double2hiint(x) & 0x7fffffff, __double2loint(x));
}

// A parameter that holds a small non-negative integer, as one.
__device__ __forceinline__ int small_int(double x) {
  const int hi = __double2hiint(x), e = (hi >> 20) - 1023;
  return e < 0 ? 0 : (1 << e) | ((hi & 0xfffff) >> (20 - e));
}

// How far x's exponent lies above 2^-480, in units of 2^21; at most kMiddling
// for 2^-480 <= |x| < 2^480 (an integer instruction each).
constexpr unsigned kMiddling = (960u << 21) - 1u;
__device__ __forceinline__ unsigned above_low(double x) { return 2u * unsigned(__double2hiint(x)) - (543u << 21); }

// The division where the three instructions of quotient() do not do, out of
// line: inline it stood between the quotients, and a warp ran them one by one.
static __device__ __noinline__ double plain_quotient(double a, double b) { return a / b; }

// a / b from y, the correctly rounded reciprocal of b: the quotient a y and
// one correction by its remainder, which gives IEEE's rounding (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34(1), 1990) where nothing on the way leaves
// the normal numbers: three FP64 instructions where the division takes 8.6 of
// their time.  With a and b between 2^-480 and 2^480 all of it is well inside
// (the remainder's last bit is at least 2^-105 of a); a zero over such a b is
// the product, and the rest is left to the division.  The tests cost exact
// BSIM3 loads 1.5% (300,000 devices: 1.635 ms against 1.611; 1.789 with the
// division inline, 1.745 with the zeros out of line too).
__device__ __forceinline__ double quotient(double a, double b, double y) {
  const double q = a * y, r = fma(-b, q, a), z = fma(r, y, q);
  const unsigned ha = above_low(a), hb = above_low(b);
  if ((ha > hb ? ha : hb) > kMiddling) return eq0(a) && hb <= kMiddling ? q : plain_quotient(a, b);
  return z;
}

}  // namespace xg
