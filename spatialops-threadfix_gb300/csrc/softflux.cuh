// The heat operators' face flux  RN(s * RN(b - a))  of three doubles on the integer pipe, bit for
// bit what the FP64 subtraction and multiplication give.
//
// This GPU starts one FP64 operation per 64 clocks and SM partition, so the exact FP64 heat
// kernels (16 FP64 operations per cell) leave most issue slots empty.  Doing the flux's two
// operations in 64-bit integers beside the FP64 operations that remain uses them.  The method is
// the IEEE definition itself: align the two signed significands to the larger exponent, keeping
// everything below as one sticky bit (round to odd), subtract, normalise, round to 53 bits (ties
// to even); multiply the two 53-bit significands exactly and round again.
//
// A value is unpacked once (SoftVal) and used by the faces on both of its sides.  soft_flux
// reports the operands it does not cover, whose flux the caller computes with the FP64 unit:
// infinities, NaNs, -0 and values of the largest binade among a and b, a zero, subnormal or
// non-finite s, and results outside the normal range.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include <spatialops/NeboFixMath.h>

namespace nebo {
namespace softfp {

// A double as m 2^(e - 1084): m the signed significand with 9 fraction bits below it (|m| < 2^62),
// e the biased exponent (1 for subnormals and zero).  -0, which a significand cannot carry, takes
// m = 0 and the exponent of the non-finite values.
struct SoftVal {
  long long m;
  int e;
};

__host__ __device__ __forceinline__ SoftVal unpack(double x) {
  const unsigned long long b = fixmath::bits(x);
  const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b;
  const int ef = (int)((hi >> 20) & 0x7ffu);
  unsigned mh = (hi & 0xfffffu) | 0x100000u;
  int e = ef;
  if (ef == 0) {  // zero or subnormal
    mh = hi & 0xfffffu;
    e = (b == (1ull << 63)) ? 2047 : 1;
  }
  const unsigned long long m = (((unsigned long long)mh << 32) | lo) << 9;
  SoftVal v;
  v.m = (int)hi < 0 ? -(long long)m : (long long)m;
  v.e = e;
  return v;
}

// The double a SoftVal was unpacked from.
__host__ __device__ __forceinline__ double pack(SoftVal v) {
  if (v.m == 0 && v.e == 2047) return fixmath::from_bits(1ull << 63);
  const unsigned long long neg = v.m < 0 ? 1ull << 63 : 0ull;
  const unsigned long long m = (unsigned long long)(v.m < 0 ? -v.m : v.m) >> 9;
  const unsigned long long ef = (m >> 52) ? (unsigned long long)v.e : 0ull;
  return fixmath::from_bits(neg | (ef << 52) | (m & 0xFFFFFFFFFFFFFull));
}

// The high word of (hi:lo) << n for 0 <= n < 32.
__host__ __device__ __forceinline__ unsigned shl_hi(unsigned hi, unsigned lo, int n) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, n);
#else
  return n ? (hi << n) | (lo >> (32 - n)) : hi;
#endif
}

// d as a normalised 53-bit significand: dq 2^(ed - 1085), dq in [2^62, 2^63] a multiple of 2^10
// (0 for d = 0, whose ed is meaningless).
struct SoftDiff {
  unsigned long long dq;
  int ed;
  unsigned sign;  // bit 31
};

// RN(b - a), for exponents below 2046
__host__ __device__ __forceinline__ SoftDiff soft_diff(SoftVal a, SoftVal b, int& E) {
  // align to the larger exponent; bits shifted out leave the low bit set (round to odd)
  const int D0 = a.e - b.e;
  const bool sw = D0 > 0;
  const long long big = sw ? a.m : b.m, small = sw ? b.m : a.m;
  E = sw ? a.e : b.e;
  int D = D0 < 0 ? -D0 : D0;
  D = D < 63 ? D : 63;
  long long t = small >> D;
  if ((long long)((unsigned long long)t << D) != small) t |= 1;
  const long long S = big - t;  // +-(b - a), |S| < 2^63
  const unsigned long long U = (unsigned long long)(S < 0 ? -S : S);
  const unsigned uh = (unsigned)(U >> 32), ul = (unsigned)U;
  const int lz = uh ? fixmath::clz32(uh) : 32 + fixmath::clz32(ul);  // 1 .. 64
  const unsigned long long n = U << (lz - 1);
  const unsigned long long r = n + (0x1ffu + (((unsigned)n >> 10) & 1u));
  SoftDiff d;
  d.dq = r & ~0x3ffull;
  d.ed = E + 2 - lz;
  d.sign = ((unsigned)(S >> 32) ^ (sw ? 0x80000000u : 0u));
  return d;
}

// RN(s d).  covered = false: the caller evaluates the product in FP64.
__host__ __device__ __forceinline__ double soft_mul(double s, SoftDiff d, bool& covered) {
  const unsigned long long sb = fixmath::bits(s);
  const unsigned sh = (unsigned)(sb >> 32), s0 = (unsigned)sb;
  const int es = (int)((sh >> 20) & 0x7ffu);
  const unsigned s1 = (sh & 0xfffffu) | 0x100000u;
  const unsigned d0 = (unsigned)d.dq, d1 = (unsigned)(d.dq >> 32);
  const unsigned long long p0 = (unsigned long long)s0 * d0;
  // s1 < 2^21, d1 <= 2^31: the middle sum stays below 2^64
  const unsigned long long mid = (unsigned long long)s0 * d1 + ((unsigned long long)s1 * d0 + (p0 >> 32));
  const unsigned long long hi = (unsigned long long)s1 * d1 + (mid >> 32);  // [2^50, 2^52)
  const unsigned h1 = (unsigned)(hi >> 32), h0 = (unsigned)hi, m0 = (unsigned)mid;
  const int c = (int)(h1 >> 19);  // 1: the product's top bit is the higher one
  const int n = 2 - c;
  const unsigned r1 = shl_hi(h1, h0, n), r0 = shl_hi(h0, m0, n);  // [2^52, 2^53)
  const unsigned rest = (m0 << n) | ((unsigned)p0 ? 1u : 0u);     // what follows, with a sticky bit
  const int er = d.ed + es + (c - 1024);                  // biased exponent - 1
  const bool zero = d.dq == 0;
  covered = (unsigned)(es - 1) < 2046u && (zero || (unsigned)er < 2045u);
  const unsigned sign = (d.sign ^ sh) & 0x80000000u;
  const unsigned long long up = ((unsigned long long)rest + (0x7fffffffu + (r0 & 1u))) >> 32;
  const unsigned long long r = (((unsigned long long)(r1 + (zero ? 0u : (unsigned)er << 20)) << 32) | r0) + up;
  return fixmath::from_bits(r | ((unsigned long long)sign << 32));
}

__host__ __device__ __forceinline__ double soft_flux(double s, SoftVal a, SoftVal b, bool& covered) {
  int E;
  const SoftDiff d = soft_diff(a, b, E);
  const double f = soft_mul(s, d, covered);
  covered = covered && E < 2046;
  return f;
}

// RN(b - a) as a double.  covered = false: an operand of the largest binade, non-finite or -0, or a
// subnormal result; the caller subtracts in FP64.
__host__ __device__ __forceinline__ double soft_sub(SoftVal a, SoftVal b, bool& covered) {
  int E;
  const SoftDiff d = soft_diff(a, b, E);
  const bool zero = d.dq == 0;
  covered = E < 2046 && (zero || d.ed > 0);
  unsigned long long r = (d.dq >> 10) + ((unsigned long long)(unsigned)(d.ed - 1) << 52);
  if (zero) r = 0;
  return fixmath::from_bits(r | (zero ? 0ull : (unsigned long long)(d.sign & 0x80000000u) << 32));
}

}  // namespace softfp
}  // namespace nebo
