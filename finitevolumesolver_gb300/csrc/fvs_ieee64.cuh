// fvs_ieee64.cuh -- IEEE double-precision quotients and square roots on the
// integer and FP32 pipes.
//
// What bounds the FP64 flavours is the FP64 pipe: 2 lanes per SM and clock
// (16 clocks per warp instruction, measured), against 64-128 for integer and
// FP32 instructions.  A correctly rounded division costs that pipe 137 clocks
// per warp and a square root 143 (measured), because both are sequences of
// FP64 multiply-adds.  Here they are long division and digit-by-digit square
// root in 32-bit integer arithmetic, round to nearest even, so every result
// is the same bits as the IEEE operation's: about 50 instructions that
// overlap with the FP64 pipe's work.
//
// Division: mantissas ma, mb in [2^52, 2^53).  Y = 2^32 * (2^52 / mb),
// rounded down by at most 6 units, comes from an FP32 reciprocal seed and one
// Newton step.  Two quotient digits, each the product of a remainder's upper
// 32 bits with Y, give Q' = 2^59 * ma / mb rounded down by less than 8 units;
// its upper 54 bits are the quotient's floor F (53 bits and the rounding bit)
// or F - 1, and the sign of one remainder in 64-bit wraparound arithmetic
// tells which.  A quotient of two 53-bit numbers is never half way between
// two 53-bit numbers, so (F + 1) >> 1 is the rounded mantissa.
// Square root: the same with Y = 2^32 / sqrt(m), m = mantissa scaled to
// [1, 4).
// Zero numerators are handled here; operands outside [2^-510, 2^511)
// (subnormal, infinite and NaN among them) take the IEEE operation.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

namespace fvs {
namespace ieee64 {

__host__ __device__ __forceinline__ uint32_t Hi(double x) {
#ifdef __CUDA_ARCH__
  return static_cast<uint32_t>(__double2hiint(x));
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return static_cast<uint32_t>(b >> 32);
#endif
}
__host__ __device__ __forceinline__ uint32_t Lo(double x) {
#ifdef __CUDA_ARCH__
  return static_cast<uint32_t>(__double2loint(x));
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return static_cast<uint32_t>(b);
#endif
}
__host__ __device__ __forceinline__ double Make(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
#else
  const uint64_t b = (uint64_t(hi) << 32) | lo;
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
__host__ __device__ __forceinline__ uint32_t MulHi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return static_cast<uint32_t>((uint64_t(a) * b) >> 32);
#endif
}
// bits [32 - s, 64 - s) of hi:lo (0 < s < 32)
__host__ __device__ __forceinline__ uint32_t ShiftLeft(uint32_t hi, uint32_t lo, int s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return (hi << s) | (lo >> (32 - s));
#endif
}
__host__ __device__ __forceinline__ float FloatOf(uint32_t bits) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(bits);
#else
  float f;
  memcpy(&f, &bits, 4);
  return f;
#endif
}
// FP32 seeds, within 2^-22 of the exact value.  On the host (the test of the
// digit bounds) an approximate one: off by `seed_error` ulp.
inline int seed_error = 0;
inline float HostSeed(double exact) {
  float f = static_cast<float>(exact);
  uint32_t b;
  memcpy(&b, &f, 4);
  b += uint32_t(seed_error);
  memcpy(&f, &b, 4);
  return f;
}
__host__ __device__ __forceinline__ float RcpSeed(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return HostSeed(1.0 / double(x));
#endif
}
__host__ __device__ __forceinline__ float RsqrtSeed(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return HostSeed(1.0 / __builtin_sqrt(double(x)));
#endif
}
// floor of a float in [0, 2^32], 2^32 as 2^32 - 1
__host__ __device__ __forceinline__ uint32_t ToUint(float x) {
#ifdef __CUDA_ARCH__
  return __float2uint_rz(x);
#else
  return x >= 4294967296.0f ? 0xFFFFFFFFu : static_cast<uint32_t>(x);
#endif
}

// The IEEE operations, out of line: operands outside the range below are rare,
// and inlined they would double the kernels' code (instruction fetch bounds a
// lone warp).
static __host__ __device__ __noinline__ double IeeeDiv(double a, double b) { return a / b; }
static __host__ __device__ __noinline__ double IeeeSqrt(double a) { return sqrt(a); }

// Unsigned distance of a high word's exponent into [2^-510, 2^511): below
// kSpan inside, at or above it outside (the sign bit drops out).
constexpr uint32_t kSpan = 1021u << 21;
__host__ __device__ __forceinline__ uint32_t Span(uint32_t hi) { return hi * 2u - (513u << 21); }

// Comparisons on the integer pipes (an FP64 comparison takes the FP64 pipe
// as long as an addition), false for NaN operands like the IEEE ones.
__host__ __device__ __forceinline__ uint64_t Bits(double x) {
  return (uint64_t(Hi(x)) << 32) | Lo(x);
}
constexpr uint64_t kInf = 0x7FF0000000000000ull;
constexpr uint64_t kSign = 0x8000000000000000ull;
__host__ __device__ __forceinline__ bool Positive(double x) { return Bits(x) - 1u < kInf; }
__host__ __device__ __forceinline__ bool Negative(double x) {
  return Bits(x) - (kSign + 1u) < kInf;
}
__host__ __device__ __forceinline__ bool IsNan(double x) { return (Bits(x) & ~kSign) > kInf; }
__host__ __device__ __forceinline__ bool IsZero(double x) { return (Bits(x) & ~kSign) == 0u; }
// a < b, and -0 < +0 (its callers differ by the sign of a zero at most; MinMod
// avoids that)
__host__ __device__ __forceinline__ bool Less(double a, double b) {
  const int64_t x = static_cast<int64_t>(Bits(a)), y = static_cast<int64_t>(Bits(b));
  const int64_t kx = x ^ static_cast<int64_t>(static_cast<uint64_t>(x >> 63) >> 1);
  const int64_t ky = y ^ static_cast<int64_t>(static_cast<uint64_t>(y >> 63) >> 1);
  return kx < ky && !IsNan(a) && !IsNan(b);
}

// The reference's MinMod, (sR > 0) ? max(0, min(sL, sR)) : min(0, max(sL, sR))
// with its a < b ? a : b and a > b ? a : b: which of two zeros, and which side
// of a NaN, comes out as there.
__host__ __device__ __forceinline__ double MinMod(double sL, double sR) {
  const bool up = Positive(sR);
  const bool left = up ? Less(sL, sR) : Less(sR, sL) && !(IsZero(sL) && IsZero(sR));
  const double m = left ? sL : sR;
  return (up ? Negative(m) : Positive(m)) ? 0.0 : m;
}

// A factor y with the bits of (0.5 x) x in y x, off the FP64 pipe: x / 2, or x
// itself below 2^-1021, where either product is zero.
__host__ __device__ __forceinline__ double HalfFactor(double x) {
  const uint32_t h = Hi(x);
  return (h & 0x7FE00000u) ? Make(h - (1u << 20), Lo(x)) : x;
}

// A divisor prepared for several quotients.
struct Divisor {
  double b;
  uint32_t hi, lo;  // mantissa with its leading bit
  uint32_t y;       // 2^32 * 2^52 / mantissa, rounded down by at most 6
  uint32_t exp;     // (1022 << 20) - exponent field
  uint32_t span;
};

__host__ __device__ __forceinline__ Divisor MakeDivisor(double b) {
  Divisor d;
  d.b = b;
  const uint32_t h = Hi(b);
  d.lo = Lo(b);
  d.hi = (h & 0x000FFFFFu) | 0x00100000u;
  d.exp = (1022u << 20) - (h & 0x7FF00000u);
  d.span = Span(h);
  const uint32_t top = ShiftLeft(d.hi, d.lo, 11);  // mantissa * 2^-21 in [2^31, 2^32)
  const float f = FloatOf(0x3F800000u | ((top >> 8) & 0x007FFFFFu));
  const uint32_t y0 = ToUint(RcpSeed(f) * 4294967296.0f);
  // Newton: y0 (1 + e 2^-31), e = 2^31 - top y0 / 2^32, low by 2 so that the
  // roundings (top and the product are rounded down) leave y below 1/b
  const int32_t e = static_cast<int32_t>(0x7FFFFFFEu - MulHi(top, y0));
  d.y = y0 + static_cast<uint32_t>((static_cast<int32_t>(y0 >> 11) * e) >> 20);
  return d;
}

// The correctly rounded 53-bit mantissa of ma / mb from Q' (al: ma's low word).
__host__ __device__ __forceinline__ uint64_t RoundedQuotient(uint64_t q, bool ge1, uint32_t al,
                                                             const Divisor& d) {
  const uint64_t f1 = (q >> (ge1 ? 6 : 5)) + 1;  // the floor F, or F + 1
  const uint32_t f1l = static_cast<uint32_t>(f1), f1h = static_cast<uint32_t>(f1 >> 32);
  const uint64_t p = uint64_t(f1l) * d.lo + (uint64_t(f1l * d.hi + f1h * d.lo) << 32);
  const uint64_t rem = (uint64_t(al << (ge1 ? 21 : 22)) << 32) - p;  // 2^53|54 ma - f1 mb
  // F = f1 - (rem < 0); the rounded mantissa (F + 1) >> 1
  return (f1 + 1 + static_cast<uint64_t>(static_cast<int64_t>(rem) >> 63)) >> 1;
}

// a / d.b, or with kHalf (0.5 a) / d.b.  kNear: without the remainder that
// decides the rounding; Q' plus its mean error rounded at the mantissa's last
// bit, within 0.57 ulp (exact quotients stay exact).
template <bool kHalf = false, bool kNear = false>
__host__ __device__ __forceinline__ double Div(double a, const Divisor& d) {
  const uint32_t ah = Hi(a), al = Lo(a);
  const uint32_t mh = (ah & 0x000FFFFFu) | 0x00100000u;
  // first digit: q1 = 2^31 ma / mb, rounded down by less than 8
  const uint32_t q1 = MulHi(ShiftLeft(mh, al, 11), d.y);
  // remainder 2^31 ma - q1 mb, in [0, 2^56)
  const uint64_t r = ((uint64_t(ShiftLeft(mh, al, 31)) << 32) | (al << 31)) -
                     (uint64_t(q1) * d.lo + (uint64_t(q1 * d.hi) << 32));
  const uint64_t q = uint64_t(q1) * (1u << 28) + MulHi(static_cast<uint32_t>(r >> 24), d.y);
  const bool ge1 = (q >> 59) != 0;  // quotient of the mantissas >= 1
  uint64_t n;
  if constexpr (kNear) {
    n = (q + (ge1 ? 64u + 4u : 32u + 4u)) >> (ge1 ? 7 : 6);
  } else {
    n = RoundedQuotient(q, ge1, al, d);
  }
  const uint32_t ea = (ah & 0x7FF00000u) + d.exp - (ge1 ? 0u : 1u << 20) -
                      (kHalf ? 1u << 20 : 0u);
  const uint32_t sign = (ah ^ Hi(d.b)) & 0x80000000u;
  uint32_t hi = (static_cast<uint32_t>(n >> 32) + ea) | sign;
  uint32_t lo = static_cast<uint32_t>(n);
  const bool zero = ((ah * 2u) | al) == 0u;
  hi = zero ? sign : hi;
  lo = zero ? 0u : lo;
  if (d.span >= kSpan || !(Span(ah) < kSpan || zero)) return IeeeDiv(kHalf ? 0.5 * a : a, d.b);
  return Make(hi, lo);
}
__host__ __device__ __forceinline__ double Div(double a, double b) { return Div(a, MakeDivisor(b)); }

// kNear: without the deciding remainder, within 0.75 ulp.
template <bool kNear = false> __host__ __device__ __forceinline__ double Sqrt(double a) {
  const uint32_t h = Hi(a), l = Lo(a);
  const uint32_t odd = (~h >> 20) & 1u;  // odd exponent: m = 2 * 1.f in [2, 4)
  const uint32_t mh = (h & 0x000FFFFFu) | 0x00100000u;
  // x = m 2^62
  const int sh = 10 + static_cast<int>(odd);
  const uint32_t xh = ShiftLeft(mh, l, sh), xl = l << sh;
  const float f = FloatOf((0x3F800000u + (odd << 23)) | ((ShiftLeft(mh, l, 11) >> 8) & 0x007FFFFFu));
  const uint32_t y0 = ToUint(RsqrtSeed(f) * 4294967296.0f);
  // Newton: y0 (1 + e 2^-31), e = 2^30 (1 - m y0^2), low by 3
  const int32_t e = static_cast<int32_t>(0x3FFFFFFDu - MulHi(MulHi(y0, y0), xh));
  const uint32_t y = y0 + static_cast<uint32_t>((static_cast<int32_t>(y0 >> 11) * e) >> 20);
  // first digit: s1 = 2^31 sqrt(m), rounded down
  const uint32_t s1 = static_cast<uint32_t>((uint64_t(xh) * y) >> 31);
  const uint64_t r = ((uint64_t(xh) << 32) | xl) - uint64_t(s1) * s1;
  const uint64_t s = uint64_t(s1) * (1u << 26) + MulHi(static_cast<uint32_t>(r >> 6), y);
  uint64_t n;
  if constexpr (kNear) {
    n = (s + 16u + 5u) >> 5;  // s is low by 5 of 2^-57 on average
  } else {
    const uint64_t f1 = (s >> 4) + 1;  // floor(2^53 sqrt(m)) or one more
    const uint32_t f1l = static_cast<uint32_t>(f1), f1h = static_cast<uint32_t>(f1 >> 32);
    const uint64_t p = uint64_t(f1l) * f1l + (uint64_t(f1l * (f1h * 2u)) << 32);
    const uint64_t rem = (uint64_t(l << (22 + static_cast<int>(odd))) << 32) - p;
    n = (f1 + 1 + static_cast<uint64_t>(static_cast<int64_t>(rem) >> 63)) >> 1;
  }
  const uint32_t er = ((h + (1021u << 20)) >> 1) & 0x7FF00000u;  // floor((e + 1021) / 2)
  if (h - 0x00100000u >= 0x7FE00000u) {  // zero, subnormal, negative, infinite, NaN
    return IeeeSqrt(a);
  }
  return Make(static_cast<uint32_t>(n >> 32) + er, static_cast<uint32_t>(n));
}

}  // namespace ieee64
}  // namespace fvs
