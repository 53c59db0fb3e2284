// soft64.cuh -- IEEE-754 binary64 addition, subtraction, multiplication,
// division and square root carried out with integer instructions, correctly
// rounded (round to nearest, ties to even), with signed zeros, subnormal
// operands and results, and infinities as IEEE-754 (2008) specifies.  NaN
// results are a quiet NaN (the first NaN operand made quiet, or the default
// NaN for an invalid operation); their payload is not that of any hardware.
//
// Why: GB300 executes FP64 at 1/54 of its FP32 rate (measured over its 152
// SMs: DFMA 525 G op/s, DDIV and DSQRT 70 G op/s), while its integer pipes
// issue several warp instructions per clock per SM.  An exact binary64
// operation built from 32- and 64-bit integer arithmetic therefore runs beside
// the FP64 pipe.  Measured on the same part (agx_soft64_throughput): division
// 320 G op/s and square root 356 G op/s this way; multiplication 429 against
// the FP64 pipe's 525, and 839 with half of the products on each; addition
// 262.  So the FP64 kernels divide and take square roots with these
// functions, and large meshes form part of their products so.  Every non-NaN
// result is bitwise the IEEE result; tests/cpp/check_soft64.cpp checks that on
// the host against the processor's own IEEE arithmetic, agx_soft64_check on
// the device against the FP64 pipe.
//
// Methods.  Addition aligns the significands in 64-bit integers, multiplication
// forms their exact product; a sticky bit stands for everything shifted out
// and the result is rounded once with guard, round and sticky bits (Goldberg,
// "What every computer scientist should know about floating-point
// arithmetic", 1991).  Division and square root take a few digits guessed in
// FP32 with exact remainders (the schoolbook digit recurrences with a large
// radix and nearest digits), whose last remainder gives the floor and the
// sticky bit.
#pragma once
#include <stdint.h>
#include <string.h>
#include <math.h>

#ifdef __CUDACC__
#define SF_HD __host__ __device__ __forceinline__
#else
#define SF_HD inline
#endif

namespace soft64 {

constexpr uint64_t SIGN = 0x8000000000000000ull;
constexpr uint64_t EXP_MASK = 0x7ff0000000000000ull;
constexpr uint64_t FRAC = 0x000fffffffffffffull;
constexpr uint64_t HIDDEN = 0x0010000000000000ull;
constexpr uint64_t QUIET = 0x0008000000000000ull;
constexpr uint64_t DEFAULT_NAN = 0x7ff8000000000000ull;

// On the device the 64 bits are taken and put together as two 32-bit words: a
// sign or exponent mask on the whole word is turned into an FP64 absolute
// value or comparison by the compiler (two FP64 instructions a division and a
// square root, counted with sm__thread_inst_executed_pipe_fp64), which is the
// pipe these functions keep free.
SF_HD uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  return ((uint64_t)(uint32_t)__double2hiint(x) << 32) | (uint32_t)__double2loint(x);
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return b;
#endif
}
SF_HD double from_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)(b >> 32), (int)(uint32_t)b);
#else
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}

SF_HD int clz64(uint64_t x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}

// x >> n with every bit shifted out ORed into bit 0 (n >= 0)
SF_HD uint64_t shr_jam(uint64_t x, int n) {
  if (n <= 0) return x;
  if (n >= 64) return x != 0;
  return (x >> n) | ((x << (64 - n)) != 0);
}

// Round to 53 bits and pack.  The exact result is (-1)^sign * sig * 2^(e - 1085):
// when sig's leading one is at bit 62, e is the result's biased exponent.  sig
// is non-zero with its leading one at bit 62 or below; bit 0 is a sticky bit
// (set when any non-zero bits lay below it).
SF_HD uint64_t round_pack(uint64_t sign, int e, uint64_t sig) {
  const int lz = clz64(sig) - 1;
  if (lz > 0) {                       // leading one to bit 62
    sig <<= lz;
    e -= lz;
  }
  if (e <= 0) {                       // below the normal range: as if e were 1
    sig = shr_jam(sig, 1 - e);
    e = 1;
  }
  const uint64_t low = sig & 0x3ff;   // the 10 bits below the 53-bit significand
  uint64_t r = (sig + 0x200) >> 10;   // add half an ulp, truncate
  if (low == 0x200) r &= ~1ull;       // exactly half: to even
  // r: the significand with its hidden bit at bit 52 (bit 53 when rounding
  // carried, bit 52 clear for a subnormal result); the sum carries into the
  // exponent field where needed
  const uint64_t out = ((uint64_t)(e - 1) << 52) + r;
  if (out >= EXP_MASK) return sign | EXP_MASK;      // overflow: infinity
  return sign | out;
}

// A finite non-zero operand as significand m (leading one at bit 52) and
// biased exponent e (below 1 for subnormal operands).
SF_HD void unpack(uint64_t a, uint64_t& m, int& e) {
  e = (int)((a >> 52) & 0x7ff);
  m = a & FRAC;
  if (e == 0) {
    const int s = clz64(m) - 11;
    m <<= s;
    e = 1 - s;
  } else {
    m |= HIDDEN;
  }
}

SF_HD uint64_t nan_of(uint64_t a, uint64_t b) {
  if ((a & ~SIGN) > EXP_MASK) return a | QUIET;
  if ((b & ~SIGN) > EXP_MASK) return b | QUIET;
  return DEFAULT_NAN;
}

SF_HD uint64_t add_bits(uint64_t a, uint64_t b) {
  const uint64_t aa = a & ~SIGN, ab = b & ~SIGN;
  if (aa >= EXP_MASK || ab >= EXP_MASK) {
    if (aa > EXP_MASK || ab > EXP_MASK) return nan_of(a, b);
    if (aa == EXP_MASK && ab == EXP_MASK) return ((a ^ b) & SIGN) ? DEFAULT_NAN : a;   // inf - inf
    return aa == EXP_MASK ? a : b;
  }
  if (aa == 0) return ab == 0 ? (a & b) : b;        // +0 + -0 = +0
  if (ab == 0) return a;
  uint64_t x = a, y = b;                            // |x| >= |y|
  if (ab > aa) {
    x = b;
    y = a;
  }
  uint64_t mx, my;
  int ex, ey;
  unpack(x, mx, ex);
  unpack(y, my, ey);
  mx <<= 10;                                        // leading ones at bit 62
  my = shr_jam(my << 10, ex - ey);
  uint64_t s;
  if ((x ^ y) & SIGN) {
    s = mx - my;
    if (s == 0) return 0;                           // exact cancellation: +0
  } else {
    s = mx + my;
    if (s >> 63) {
      s = shr_jam(s, 1);
      ex += 1;
    }
  }
  return round_pack(x & SIGN, ex, s);
}

SF_HD uint64_t sub_bits(uint64_t a, uint64_t b) { return add_bits(a, b ^ SIGN); }

// FP32 approximations of 1 / x, sqrt(x) and 1 / sqrt(x) for the digits below
// (a few units in the last place are enough), conversions to the nearest
// integer and of 32-bit integers only: conversions of 64-bit integers run on
// the FP64 pipe.
SF_HD float recip_approx(float x) {
#ifdef __CUDA_ARCH__
  return __fdividef(1.0f, x);
#else
  return 1.0f / x;
#endif
}
SF_HD float rsqrt_approx(float x) {
#ifdef __CUDA_ARCH__
  return rsqrtf(x);
#else
  return 1.0f / sqrtf(x);
#endif
}
SF_HD int nearest_int(float x) {
#ifdef __CUDA_ARCH__
  return __float2int_rn(x);
#else
  return (int)lrintf(x);
#endif
}

// What the integer forms below do not take (NaNs, infinities, subnormal
// operands or results, negative roots), out of line.
#ifdef __CUDACC__
#define SF_COLD static __host__ __device__ __noinline__
#else
#define SF_COLD static __attribute__((noinline))
#endif
SF_COLD double div_rare(double a, double b) {
#ifdef __CUDA_ARCH__
  return __ddiv_rn(a, b);
#else
  return a / b;
#endif
}
SF_COLD double sqrt_rare(double a) {
#ifdef __CUDA_ARCH__
  return __dsqrt_rn(a);
#else
  return ::sqrt(a);
#endif
}

// The 55-bit value q in [2^54, 2^55) with its low bit set for anything below,
// rounded to 53 bits and packed with biased exponent e (1 .. 2046).
SF_HD double pack55(uint64_t sign, int e, uint64_t q) {
  const uint64_t r = (q + 1 + ((q >> 2) & 1)) >> 2;      // to nearest, ties to even
  return from_bits(sign | (((uint64_t)(uint32_t)(e - 1) << 52) + r));
}

SF_COLD double mul_rare(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}

// x << s with y's top bits shifted in (0 < s < 32)
SF_HD uint32_t shl_in(uint32_t x, uint32_t y, int s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(y, x, s);
#else
  return (x << s) | (y >> (32 - s));
#endif
}

// a * b: the exact product of the significands from four 32-bit ones.
SF_HD double mul(double a, double b) {
  const uint64_t ua = bits(a), ub = bits(b);
  const uint64_t sign = (ua ^ ub) & SIGN;
  const int ea = (int)((uint32_t)(ua >> 52) & 0x7ffu), eb = (int)((uint32_t)(ub >> 52) & 0x7ffu);
  const int e = ea + eb - 1023;
  if ((unsigned)(ea - 1) >= 2046u || (unsigned)(eb - 1) >= 2046u || (unsigned)(e - 1) >= 2045u) {
    if (((ua << 1) == 0 && eb < 2047) || ((ub << 1) == 0 && ea < 2047)) return from_bits(sign);
    return mul_rare(a, b);
  }
  const uint64_t x = (ua & FRAC) | HIDDEN, y = ((ub & FRAC) | HIDDEN) << 11;     // product in [2^115, 2^117)
  const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32), y0 = (uint32_t)y, y1 = (uint32_t)(y >> 32);
  const uint64_t p = (uint64_t)x0 * y0;
  const uint64_t m = (uint64_t)x0 * y1 + (p >> 32);
  const uint64_t n = (uint64_t)x1 * y0 + (uint32_t)m;
  const uint64_t hi = (uint64_t)x1 * y1 + (m >> 32) + (n >> 32);                 // leading one at bit 51 or 52
  const int top = (int)(hi >> 52), s = 3 - top;
  // hi : lo shifted left by s (2 or 3): the 55 bits, and whether any are set below
  const uint32_t h1 = (uint32_t)(hi >> 32), h0 = (uint32_t)hi, l1 = (uint32_t)n, l0 = (uint32_t)p;
  const uint32_t q1 = shl_in(h1, h0, s), q0 = shl_in(h0, l1, s);
  const bool below = (shl_in(l1, l0, s) | (l0 << s)) != 0;
  return pack55(sign, e + top, ((uint64_t)q1 << 32) | q0 | (below ? 1u : 0u));
}

// a / b by three digits of the quotient n / d in [1, 2) (n, d the
// significands): each digit is the nearest integer to the FP32 quotient of the remainder's
// leading 31 bits and d, scaled by 2^17, 2^18 and 2^19.  The FP32 relative
// error is below 2^-21 (the quotient's 2 ulp 2^-22, two conversions and a
// product 2^-24 each, two cuts 2^-30), so a digit is off by less than 0.5 + 2^-2 of the scaled quotient,
// the remainders (exact in 64-bit wrap-around arithmetic) stay below d in
// magnitude, the next digits below 2^19, and the last remainder gives the
// floor after one correction and the sticky bit.
SF_HD double div(double a, double b) {
  const uint64_t ua = bits(a), ub = bits(b);
  const uint64_t sign = (ua ^ ub) & SIGN;
  const int ea = (int)((uint32_t)(ua >> 52) & 0x7ffu), eb = (int)((uint32_t)(ub >> 52) & 0x7ffu);
  uint64_t n = (ua & FRAC) | HIDDEN;
  const uint64_t d = (ub & FRAC) | HIDDEN;
  const int less = n < d ? 1 : 0;
  const int e = ea - eb + 1023 - less;
  if ((unsigned)(eb - 1) >= 2046u || (unsigned)(ea - 1) >= 2046u || (unsigned)(e - 1) >= 2046u) {
    if ((ua << 1) == 0 && (unsigned)(eb - 1) < 2046u) return from_bits(sign);      // 0 / x
    return div_rare(a, b);
  }
  n = less ? n + n : n;
  const float r = recip_approx((float)(int)(uint32_t)(d >> 22));                 // 2^22 / d
  const int q1 = nearest_int((float)(int)(uint32_t)(n >> 23) * (r * 262144.0f));  // n / d * 2^17
  int64_t rem = (int64_t)((n << 17) - (uint64_t)(uint32_t)q1 * d);
  const int q2 = nearest_int((float)(int)(rem >> 23) * (r * 524288.0f));          // rem / d * 2^18
  rem = (int64_t)(((uint64_t)rem << 18) - (uint64_t)(int64_t)q2 * d);
  const int q3 = nearest_int((float)(int)(rem >> 23) * (r * 1048576.0f));         // rem / d * 2^19
  rem = (int64_t)(((uint64_t)rem << 19) - (uint64_t)(int64_t)q3 * d);
  uint64_t q = ((uint64_t)(uint32_t)q1 << 37) + ((uint64_t)(int64_t)q2 << 19) + (uint64_t)(int64_t)q3;
  const bool low = rem < 0;                       // floor
  q -= low ? 1 : 0;
  rem += low ? (int64_t)d : 0;
  return pack55(sign, e, q | (rem != 0 ? 1u : 0u));
}

// sqrt(a): s in [2^52, 2^54) is the significand at an even exponent; the root
// of s is taken to 27 bits in FP32 (off by less than 2^6) and refined by two
// digits d = remainder / (2 root), of 13 and 15 more bits, to the nearest
// integer, with exact remainders (s scaled minus root squared): after the
// first the root is off by less than 1 (digit below 2^19, FP32 relative
// error below 2^-20, second-order term d^2 / (2 root) below 2^-4), after the
// second likewise, and one correction gives the floor and the sticky bit.
SF_HD double sqrt(double a) {
  const uint64_t ua = bits(a);
  const int ea = (int)(uint32_t)(ua >> 52);              // the sign too: negative operands are rare
  if ((unsigned)(ea - 1) >= 2046u) {
    if ((ua << 1) == 0) return a;                        // +0, -0
    return sqrt_rare(a);
  }
  const int odd = (ea & 1) ^ 1;                          // ea - 1023 odd
  const uint64_t m = (ua & FRAC) | HIDDEN;
  const uint64_t s = odd ? m + m : m;
  const float x = (float)(int)(uint32_t)(s >> 24);       // s / 2^24, below 2^30
  const float y = rsqrt_approx(x);                       // 2^12 / sqrt(s)
  const int r0 = nearest_int(x * y * 4096.0f);           // sqrt(s): 2^26 .. 2^27
  int64_t rem = (int64_t)(s - (uint64_t)(uint32_t)r0 * (uint32_t)r0);
  const int d1 = nearest_int((float)(int)(rem >> 4) * (y * 16.0f));      // rem 2^13 / (2 r0)
  const uint64_t r1 = ((uint64_t)(uint32_t)r0 << 13) + (uint64_t)(int64_t)d1;
  rem = (int64_t)(((uint64_t)rem << 26) - (r1 + ((uint64_t)(uint32_t)r0 << 13)) * (uint64_t)(int64_t)d1);
  const int d2 = nearest_int((float)(int)(rem >> 13) * (y * 4.0f));      // rem 2^15 / (2 r1)
  const uint64_t r2 = (r1 << 15) + (uint64_t)(int64_t)d2;
  rem = (int64_t)(((uint64_t)rem << 30) - (r2 + (r1 << 15)) * (uint64_t)(int64_t)d2);
  uint64_t q = r2;
  const bool low = rem < 0;
  q -= low ? 1 : 0;
  return pack55(0, ((ea - 1023 - odd) >> 1) + 1023, q | (rem != 0 ? 1u : 0u));
}

SF_HD double add(double a, double b) { return from_bits(add_bits(bits(a), bits(b))); }
SF_HD double sub(double a, double b) { return from_bits(sub_bits(bits(a), bits(b))); }

}  // namespace soft64
