// ttfld_fp64.cuh -- FP64 products, quotients and square roots, rounded to
// nearest even, computed on the integer and FP32 pipes.
//
// GB300 issues FP64 arithmetic two lanes per clock and SM (measured: 515-605
// G fused multiply-adds per second; a quotient costs 7.3 of them, a square
// root 7.5), while integer and FP32 instructions issue at up to 128 lanes.
// A correctly rounded product of two normal numbers is four 32 x 32 -> 64
// multiplications and some 30 other integer instructions, a quotient or a
// square root 70 to 90, so on this chip the integer pipes do a product in
// about the FP64 pipe's own time, beside it, and a quotient in a fifth of
// it: measured alone, in G per second, mul_rn 570 (hardware 494), div_rn 335
// (67), sqrt_rn 306 (68).  The
// kernels of the FP64 path, which were bound by the FP64 pipe, use these for
// their quotients and about half of their products and leave the sums to the
// FP64 pipe: at 100x256x128 a face pass (FLIM, DIFF, flux of one direction)
// takes 248 us instead of 777, the outer iteration's rows 427 instead of
// 982, the stellar heating 118 instead of 418, KAPPA 45 instead of 184,
// delta Q 120 instead of 355 and the FP32 compaction 81 instead of 123.
//
// Every result is the IEEE round-to-nearest-even one, bit for bit the result
// of `*`, `/` and sqrt(): operands or results that are subnormal, infinite,
// NaN or near the ends of the exponent range take the hardware operation.
// The header also compiles for the host, where tests/test_fp64_pipe.py
// checks it against the machine's own arithmetic.
//
// The methods are from the definitions: the product is formed exactly and
// rounded; the quotient and the root are long division (and digit-by-digit
// root) in three digits of about 26 bits, each guessed in FP32 from the
// leading bits of the exact integer remainder, so that the remainder after
// the last digit decides the rounding.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define TT_FP_HD __host__ __device__ __forceinline__
#else
#include <math.h>
#include <string.h>
#define TT_FP_HD static inline
#endif
#ifndef TT_GUESS_ERROR  // on the host: a test's stand-in for the error of the approximate instructions
#define TT_GUESS_ERROR(v) (v)
#endif

namespace ttfld {

TT_FP_HD uint64_t f64_bits(double v) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(v);
#else
  union { double d; uint64_t u; } b;
  b.d = v;
  return b.u;
#endif
}
TT_FP_HD double f64_of(uint64_t v) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)v);
#else
  union { double d; uint64_t u; } b;
  b.u = v;
  return b.d;
#endif
}
TT_FP_HD float f32_of(uint32_t v) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(v);
#else
  union { float d; uint32_t u; } b;
  b.u = v;
  return b.d;
#endif
}
TT_FP_HD uint32_t f32_bits(float v) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(v);
#else
  union { float d; uint32_t u; } b;
  b.d = v;
  return b.u;
#endif
}
// (hi:lo) >> s for s in 0..31, low word
TT_FP_HD uint32_t shr64_lo(uint32_t lo, uint32_t hi, int s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(lo, hi, s);
#else
  return s ? (lo >> s) | (hi << (32 - s)) : lo;
#endif
}
TT_FP_HD uint64_t wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
TT_FP_HD uint32_t hi32(uint64_t v) { return (uint32_t)(v >> 32); }
TT_FP_HD uint32_t lo32(uint64_t v) { return (uint32_t)v; }
// FP32 reciprocal and reciprocal square root, a few ulp: first guesses only
TT_FP_HD float rcp_guess(float v) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
#else
  return TT_GUESS_ERROR(1.0f / v);
#endif
}
TT_FP_HD float rsqrt_guess(float v) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
#else
  return TT_GUESS_ERROR(1.0f / sqrtf(v));
#endif
}
TT_FP_HD int32_t round_i32(float v) {
#if defined(__CUDA_ARCH__)
  return __float2int_rn(v);
#else
  return (int32_t)lrintf(v);
#endif
}

#if defined(__CUDA_ARCH__)
static __device__ __noinline__ double hw_mul(double a, double b) { return __dmul_rn(a, b); }
static __device__ __noinline__ double hw_div(double a, double b) { return __ddiv_rn(a, b); }
static __device__ __noinline__ double hw_sqrt(double a) { return __dsqrt_rn(a); }
#else
TT_FP_HD double hw_mul(double a, double b) { return a * b; }
TT_FP_HD double hw_div(double a, double b) { return a / b; }
TT_FP_HD double hw_sqrt(double a) { return sqrt(a); }
#endif

// a b.  The 106-bit product P of the mantissas is P2 (from bit 64 up), P1, P0;
// c is 1 if it is 2^105 or more, and its leading 53 bits m and the part that
// is rounded away, top-aligned in rh:rl, come by shifts of 20 + c and 12 - c.
// m is rounded up if rh:rl is above half, or half with m odd: then
// rh + 2^31 - 1 + odd carries (the bits of rl joined to rh's last one).  The
// fast path is for operands and results in [2^-511, 2^512): the first two
// exponent bits differ.
TT_FP_HD double mul_rn(double a, double b) {
  const uint64_t ua = f64_bits(a), ub = f64_bits(b);
  const uint32_t ah = hi32(ua), al = lo32(ua), bh = hi32(ub), bl = lo32(ub);
  const uint32_t mh = (ah & 0xfffffu) | 0x100000u, nh = (bh & 0xfffffu) | 0x100000u;
  const uint64_t t0 = wide(al, bl), t1 = wide(mh, bl) + wide(al, nh), t2 = wide(mh, nh);  // t1 < 2^54
  uint32_t p1, p2l, p2h;
#if defined(__CUDA_ARCH__)
  asm("add.cc.u32 %0, %3, %4;\n\taddc.cc.u32 %1, %5, %6;\n\taddc.u32 %2, %7, 0;"
      : "=&r"(p1), "=&r"(p2l), "=r"(p2h)
      : "r"(hi32(t0)), "r"(lo32(t1)), "r"(lo32(t2)), "r"(hi32(t1)), "r"(hi32(t2)));
#else
  const uint64_t w = (uint64_t)hi32(t0) + lo32(t1), v = t2 + hi32(t1) + (w >> 32);
  p1 = lo32(w);
  p2l = lo32(v);
  p2h = hi32(v);
#endif
  const uint32_t c = p2h >> 9;
  const uint32_t ml = shr64_lo(p1, p2l, (int)(20u + c));
  const uint32_t mu = shr64_lo(p2l, p2h, (int)(20u + c));
  const uint32_t rl = lo32(t0) << (12u - c);
  const uint32_t rest = shr64_lo(lo32(t0), p1, (int)(20u + c)) | (rl < 1u ? rl : 1u);
  const uint32_t half = 0x7fffffffu + (ml & 1u);
  const uint32_t e = (ah & 0x7ff00000u) + (bh & 0x7ff00000u) + (c << 20) - (1024u << 20) + ((ah ^ bh) & 0x80000000u);
  uint32_t ol, oh;
#if defined(__CUDA_ARCH__)
  asm("{\n\t.reg .u32 drop;\n\tadd.cc.u32 drop, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, %6;\n\t}"
      : "=&r"(ol), "=r"(oh)
      : "r"(rest), "r"(half), "r"(ml), "r"(mu), "r"(e));
#else
  const uint64_t o = (((uint64_t)(mu + e) << 32) | ml) + (((uint64_t)rest + half) >> 32);
  ol = lo32(o);
  oh = hi32(o);
#endif
  if (((ah ^ (ah << 1)) & (bh ^ (bh << 1)) & (oh ^ (oh << 1)) & 0x40000000u) != 0u)
    return f64_of(((uint64_t)oh << 32) | ol);
  // a zero operand (no flow across a face, a boundary row) needs no product
  const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
  const bool za = (al | (ah << 1)) == 0u, zb = (bl | (bh << 1)) == 0u;
  if ((za && eb < 2047u) || (zb && ea < 2047u)) return f64_of((uint64_t)((ah ^ bh) & 0x80000000u) << 32);
  return hw_mul(a, b);
}

// a / b.  With A in [B, 2 B), B in [2^52, 2^53), the quotient
// Q = floor(A 2^53 / B) has 54 bits, and the nearest 53-bit one is
// (Q + 1) >> 1 (a quotient of two 53-bit numbers is never half way between
// two).  Signed digits with 26, 24 and 3 bits after the point; r is the
// remainder, exact modulo 2^64.  y is within 2^-24 of 2^52 / B (the guess's
// error enters squared) and each FP32 rounding adds 2^-24, so q1 < 2^27 is
// within 25 units, |q2| < 2^28.7 and within 90 units, r / B then below 90:
// r stays below 2^62.6 and the last digit is off by less than one.
TT_FP_HD double div_rn(double a, double b) {
  const uint64_t ua = f64_bits(a), ub = f64_bits(b);
  const uint32_t ah = hi32(ua), bh = hi32(ub);
  const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
  const uint64_t B = (ub & 0xfffffffffffffull) | 0x10000000000000ull;
  uint64_t A = (ua & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint32_t c = A < B ? 1u : 0u;
  const int32_t e = (int32_t)(ea - eb - c) + 1022;
  // B 2^-52 in [1, 2): leading 24 bits and the 23 after them
  const uint32_t bt = (uint32_t)(B >> 29);
  const float b0 = f32_of(0x3f800000u | (bt & 0x7fffffu));
  const float b1 = f32_of(0x34000000u | ((uint32_t)(B >> 6) & 0x7fffffu)) - f32_of(0x34000000u);
  float y = rcp_guess(b0);
  y = fmaf(y, fmaf(-b1, y, fmaf(-b0, y, 1.0f)), y);  // 2^52 / B within about 2^-23
  A <<= c;
  const float af = (float)(uint32_t)(A >> 23);  // A 2^-23, below 2^31
  const uint32_t q1 = (uint32_t)round_i32(af * (y * 0.125f));  // A 2^-23 y 2^-3 = (A / B) 2^26
  int64_t r = (int64_t)((A << 26) - B * q1);
  const int32_t q2 = round_i32((float)(int32_t)(r >> 32) * (y * 16.0f));  // r / B 2^24 = r 2^-32 y 2^4
  r = (int64_t)(((uint64_t)r << 27) - ((B * (uint64_t)(int64_t)q2) << 3));
  const int32_t q3 = round_i32((float)(int32_t)(r >> 32) * (y * 9.5367431640625e-7f));  // r / B = r 2^-32 y 2^-20
  r = r - (int64_t)(B * (uint64_t)(int64_t)q3);
  const uint64_t q = ((uint64_t)q1 << 27) + (uint64_t)(((int64_t)q2 << 3) + (q3 - (r < 0 ? 1 : 0)));
  if (ea - 1u < 2046u && eb - 1u < 2046u && (uint32_t)(e - 1) < 2043u) {
    const uint32_t sign = (ah ^ bh) & 0x80000000u;
    return f64_of(((uint64_t)((uint32_t)e << 20 | sign) << 32) + ((q + 1) >> 1));
  }
  if ((ua << 1) == 0u && eb - 1u < 2046u) return f64_of((uint64_t)((ah ^ bh) & 0x80000000u) << 32);
  return hw_div(a, b);
}

// sqrt(a).  With M in [2^52, 2^54) (the mantissa, doubled for odd
// exponents) the root S = floor(sqrt(M 2^54)) has 54 bits and the nearest
// 53-bit one is (S + 1) >> 1 (a root is never half way between two).
// Digits: s1 of 27 bits within 40 units, then two signed ones of 14 and 13
// bits within one unit each; r = M 4^k - s^2 is exact at every step and the
// last one settles the floor (or, never seen, hands over to the hardware).
TT_FP_HD double sqrt_rn(double a) {
  const uint64_t ua = f64_bits(a);
  const uint32_t e = (uint32_t)(ua >> 52);  // with the sign: negative values fail the test below
  const uint32_t odd = (e & 1u) ^ 1u;       // a = M 2^(e - 1075): e odd has an even power of two
  const uint64_t M = ((ua & 0xfffffffffffffull) | 0x10000000000000ull) << odd;
  const float mf = (float)(uint32_t)(M >> 23);                    // M 2^-23, below 2^31
  float y = rsqrt_guess(mf);                                      // 2^11.5 / sqrt(M)
  y = fmaf(y * 0.5f, fmaf(-mf * y, y, 1.0f), y);
  const float root = mf * y;                                      // sqrt(M) 2^-11.5
  const uint32_t s1 = (uint32_t)round_i32(root * 2896.30937574009925f);  // times 2^11.5
  int64_t r = (int64_t)(M - wide(s1, s1));                        // below 2^34
  // s2 = r 2^14 / (2 s1), 1 / s1 = y 2^-11.5
  const float h = y * 3.4526698300124393e-4f;                     // 1 / sqrt(M)
  const int32_t s2 = round_i32((float)(int32_t)(r >> 8) * (h * 2097152.0f));
  // s = s1 2^14 + s2: M 4^14 - s^2 = r 2^28 - 2 s1 s2 2^14 - s2^2
  const int64_t w = (int64_t)s2 * s2;
  r = (int64_t)(((uint64_t)r << 28) - (((uint64_t)s1 * (uint64_t)(int64_t)s2) << 15) - (uint64_t)w);
  const uint64_t s12 = ((uint64_t)s1 << 14) + (uint64_t)(int64_t)s2;
  // s3 = r 2^13 / (2 s12), s12 = sqrt(M) 2^14; r is below 2^43
  const int32_t s3 = round_i32((float)(int32_t)(r >> 16) * (h * 16384.0f));
  // s = s12 2^13 + s3
  int64_t s = (int64_t)((s12 << 13) + (uint64_t)(int64_t)s3);
  r = (int64_t)(((uint64_t)r << 26) - ((s12 * (uint64_t)(int64_t)s3) << 14) - (uint64_t)((int64_t)s3 * s3));
  // r = M 4^27 - s^2, |r| below a few times 2 s: settle the floor
  if (r < 0) { s -= 1; r += 2 * s + 1; }
  else if (r > 2 * s) { r -= 2 * s + 1; s += 1; }
  if (e - 1u < 2046u && r >= 0 && r <= 2 * s) {
    return f64_of(((uint64_t)((e + 1021u + 1u - odd) >> 1) << 52) + ((uint64_t)(s + 1) >> 1));
  }
  return hw_sqrt(a);
}

// The conversions between FP64 and FP32 run on the FP64 pipe too (measured:
// 604 G per second); these are the same values from integer instructions.
TT_FP_HD float f32_rn(double v) {
  const uint64_t u = f64_bits(v);
  const uint32_t h = hi32(u), l = lo32(u);
  const uint32_t e = (h >> 20) & 0x7ffu;
  if (e - 897u < 253u) {  // a normal FP32 result, clear of overflow
    const uint32_t m = ((h & 0x7fffffffu) - (896u << 20)) << 3 | l >> 29;
    const uint32_t rest = l << 3, up = rest > 0x80000000u - (m & 1u) ? 1u : 0u;
    return f32_of((m + up) | (h & 0x80000000u));
  }
  return (float)v;
}
TT_FP_HD double f64_of_f32(float v) {
  const uint32_t u = f32_bits(v);
  const uint32_t e = (u >> 23) & 0xffu;
  if (e - 1u < 254u) return f64_of(((uint64_t)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))) << 32) | ((uint64_t)(u << 29)));
  return (double)v;
}

// Unsigned 32-bit division by a divisor fixed before the launch (Granlund and
// Montgomery's invariant division): q = n m >> sh with m = ceil(2^(31+s) / d),
// s = ceil(log2 d), exact for every n < 2^31.  The kernels split their linear
// index with it: a 64-bit `/` or `%` takes some 70 integer instructions and
// conversions that run on the FP64 pipe (277 G per second), the pipes that
// the functions above load.
// Linear indexes fit: a context keeps 57 FP64 arrays, so one of 2^31 cells
// could not be allocated.
struct FastDiv {
  unsigned int d, m;
  int sh;
};
static inline FastDiv fast_div(int d) {
  int s = 0;
  while ((1ull << s) < (unsigned long long)d) ++s;
  const unsigned long long p = 1ull << (31 + s);
  return FastDiv{(unsigned int)d, (unsigned int)((p + (unsigned int)d - 1) / (unsigned int)d), 31 + s};
}
TT_FP_HD unsigned int div_of(const FastDiv& f, unsigned int n) {
  return (unsigned int)(((unsigned long long)n * f.m) >> f.sh);
}
// n = q d + r
TT_FP_HD unsigned int div_rem(const FastDiv& f, unsigned int n, unsigned int& r) {
  const unsigned int q = div_of(f, n);
  r = n - q * f.d;
  return q;
}

}  // namespace ttfld
