// Correctly rounded FP64 operations that keep off the FP64 pipe.
//
// GB300 issues about two FP64 operations per clock and SM (1.06 TFLOP/s against
// 78 TFLOP/s of FP32, measured with independent FMA chains), so one FP64
// instruction costs a warp as much issue time as some 30 integer or 60 FP32
// instructions.  The exact kernels must return the reference's FP64 bits, but
// nothing says that the FP64 pipe has to form them: the functions here work on the
// significands with the integer and FP32 pipes and round as IEEE 754 does.  They
// state the operand ranges they need; callers check those ranges (on the integer
// pipes) and use the plain operators outside them.
#pragma once

#include <stdint.h>
#ifdef __CUDACC__
#include <cuda_runtime.h>
#define GB_HD __host__ __device__ __forceinline__
#else
#include <math.h>
#include <string.h>
#define GB_HD inline
#endif

namespace gb2d {

// Bit casts and FP32 steps, on the device and (for the CPU checks) on the host.
#ifdef __CUDA_ARCH__
GB_HD uint64_t dbits(double x) {  // opaque: the compiler must not recognise FP64 operations in what follows
  uint64_t b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
  return b;
}
GB_HD double bitsd(uint64_t b) {
  double x;
  asm("mov.b64 %0, %1;" : "=d"(x) : "l"(b));
  return x;
}
GB_HD uint32_t fbits(float x) { return __float_as_uint(x); }
GB_HD float bitsf(uint32_t b) { return __uint_as_float(b); }
GB_HD float fma32(float a, float b, float c) { return __fmaf_rn(a, b, c); }
GB_HD float mul32(float a, float b) { return __fmul_rn(a, b); }
GB_HD float u32f(uint32_t u) { return __uint2float_rn(u); }
GB_HD float i32f(int32_t u) { return __int2float_rn(u); }
GB_HD int32_t f32i(float x) { return __float2int_rn(x); }
GB_HD float rcp32(float x) {  // within 1 ulp
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
GB_HD float rsqrt32(float x) {  // within 2 ulp
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// (hi:lo) << n, upper word, 0 <= n < 32.
GB_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t n) { return __funnelshift_l(lo, hi, n); }
// m + the carry out of rem + (2^63 - 1 + odd): round to nearest even by the discarded
// bits rem (left aligned) of a significand whose last bit is odd.
GB_HD uint64_t round_even(uint64_t m, uint64_t rem) {
  uint32_t lo, hi, odd = (uint32_t)m & 1u;
  asm("{\n\t.reg .u32 t;\n\t"
      "add.cc.u32 t, %2, %4;\n\t"
      "addc.cc.u32 t, %3, %5;\n\t"
      "addc.cc.u32 %0, %6, 0;\n\t"
      "addc.u32 %1, %7, 0;\n\t}"
      : "=&r"(lo), "=&r"(hi)
      : "r"((uint32_t)rem), "r"((uint32_t)(rem >> 32)), "r"(odd - 1u), "r"(0x7fffffffu + odd), "r"((uint32_t)m), "r"((uint32_t)(m >> 32)));
  return (uint64_t)hi << 32 | lo;
}
GB_HD uint64_t mulhi64(uint64_t a, uint64_t b) { return __umul64hi(a, b); }
#else
GB_HD uint64_t dbits(double x) { uint64_t b; __builtin_memcpy(&b, &x, 8); return b; }
GB_HD double bitsd(uint64_t b) { double x; __builtin_memcpy(&x, &b, 8); return x; }
GB_HD uint32_t fbits(float x) { uint32_t b; __builtin_memcpy(&b, &x, 4); return b; }
GB_HD float bitsf(uint32_t b) { float x; __builtin_memcpy(&x, &b, 4); return x; }
GB_HD float fma32(float a, float b, float c) { return __builtin_fmaf(a, b, c); }
GB_HD float mul32(float a, float b) { return a * b; }
GB_HD float u32f(uint32_t u) { return (float)u; }
GB_HD float i32f(int32_t u) { return (float)u; }
GB_HD int32_t f32i(float x) { return (int32_t)__builtin_rintf(x); }
extern int g_rcp_ulp;  // the CPU checks perturb the seed by this many ulps
GB_HD float rcp32(float x) { return bitsf(fbits(1.0f / x) + (uint32_t)g_rcp_ulp); }
GB_HD float rsqrt32(float x) { return bitsf(fbits((float)(1.0 / __builtin_sqrt((double)x))) + (uint32_t)g_rcp_ulp); }
GB_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t n) { return (uint32_t)((((uint64_t)hi << 32) | lo) << n >> 32); }
GB_HD uint64_t round_even(uint64_t m, uint64_t rem) {
  const uint64_t half = 0x8000000000000000ull;
  return m + (rem > half || (rem == half && (m & 1)) ? 1 : 0);
}
GB_HD uint64_t mulhi64(uint64_t a, uint64_t b) { return (uint64_t)((unsigned __int128)a * b >> 64); }
#endif

constexpr uint64_t kFracBits = 0x000fffffffffffffull, kHidden = 0x0010000000000000ull;

// a / b, correctly rounded to nearest, for positive normal a and b whose quotient
// is normal; no FP64 instruction.  With the significands ma, mb in [2^52, 2^53)
// the result's significand is the integer nearest to N / mb, N = ma 2^(52 + sh),
// sh = 1 where ma < mb:
//  1. r0 = 1/bh in FP32 (bh: mb's leading 24 bits), e = 1 - b r0 and r0 (1 + e + e^2)
//     as two FP32 words; times a as two FP32 words: a quotient estimate good to
//     2^-44, i.e. qi within 2^9 of N / mb;
//  2. R = N - qi mb, formed modulo 2^64 (|R| < 2^63, so the wrapped value is R);
//     dq = R / mb rounded in FP32, and the remainder follows: |R| <= (1/2 + 2^-12) mb;
//  3. one exact comparison of 2 R with mb settles the rounding.  A quotient of two
//     53-bit significands is never a midpoint of two 53-bit numbers (a midpoint
//     times mb has more than 53 significant bits), so there are no ties.
// About 55 integer and FP32 instructions in place of a dozen on the FP64 pipe; the
// terms of b alone are formed once where several quotients share a divisor.
GB_HD double div_pos(double a, double b) {
  const uint64_t ab = dbits(a), bb = dbits(b);
  const uint64_t ma = (ab & kFracBits) | kHidden, mb = (bb & kFracBits) | kHidden;
  const float ah = bitsf(((uint32_t)(ab >> 29) & 0x7fffffu) | 0x3f800000u), al = u32f((uint32_t)ab & 0x1fffffffu);
  const float bh = bitsf(((uint32_t)(bb >> 29) & 0x7fffffu) | 0x3f800000u), bl = u32f((uint32_t)bb & 0x1fffffffu);
  const float r0 = rcp32(bh), r0s = mul32(r0, 2.220446049250313e-16f);  // 2^-52: the scale of al, bl
  float e = fma32(-bh, r0, 1.0f);
  e = fma32(-bl, r0s, e);
  const float rl = mul32(r0, fma32(e, e, e));
  const float p = mul32(ah, r0);
  float t = fma32(ah, rl, fma32(ah, r0, -p));
  t = fma32(al, r0s, t);
  const uint32_t sh = ma < mb ? 1u : 0u;
  const uint32_t pb = fbits(p), s = (pb >> 23) - (127u - 29u) + sh;  // 27..31
  const uint32_t pi = (pb & 0x7fffffu) | 0x800000u;
  const int32_t ti = f32i(mul32(t, sh ? 562949953421312.0f : 281474976710656.0f));  // 2^49 : 2^48
  uint64_t q = ((uint64_t)(pi >> (32u - s)) << 32 | (uint32_t)(pi << s)) + (uint64_t)((int64_t)ti << 4);
  uint64_t R = (ma << (52u + sh)) - q * mb;
  const int32_t dq = f32i(mul32(i32f((int32_t)(R >> 32)), mul32(r0, 9.5367431640625e-07f)));  // 2^-20
  q += (uint64_t)(int64_t)dq;
  R -= (uint64_t)(int64_t)dq * mb;
  const int64_t R2 = (int64_t)(R << 1);
  q += R2 > (int64_t)mb ? 1u : 0u;
  q -= R2 < -(int64_t)mb ? 1u : 0u;
  return bitsd(((uint64_t)((uint32_t)(ab >> 52) - (uint32_t)(bb >> 52) + 1022u - sh) << 52) + q);
}

// a b, correctly rounded, for zero or normal a and b whose product is zero or normal:
// the 106-bit product of the significands from 32-bit parts, normalised by one bit
// and rounded by its discarded bits.  About 28 integer instructions (fewer where b is
// a constant with few bits), a little less issue time than the FP64 multiply has in
// the FP64 pipe, and beside it.
GB_HD double mul_rn(double a, double b) {
  const uint64_t ab = dbits(a), bb = dbits(b);
  const uint32_t ah = (uint32_t)(ab >> 32), bh = (uint32_t)(bb >> 32), al = (uint32_t)ab, bl = (uint32_t)bb;
  const uint32_t am = (ah & 0xfffffu) | 0x100000u, bm = (bh & 0xfffffu) | 0x100000u;
  const uint64_t ll = (uint64_t)al * bl;
  const uint64_t t1 = (uint64_t)am * bl + (ll >> 32);
  const uint64_t t2 = (uint64_t)al * bm + (uint32_t)t1;
  const uint64_t hh = (uint64_t)am * bm + (t1 >> 32) + (t2 >> 32);
  const uint32_t top = (uint32_t)(hh >> 41), n = 12u - top, p0 = (uint32_t)ll, p1 = (uint32_t)t2, h0 = (uint32_t)hh;
  uint64_t m = (uint64_t)shl_hi(h0, (uint32_t)(hh >> 32), n) << 32 | shl_hi(p1, h0, n);
  m = round_even(m, (uint64_t)shl_hi(p0, p1, n) << 32 | (p0 << n));
  const uint32_t ae = ah & 0x7ff00000u, be = bh & 0x7ff00000u;
  uint32_t hi = (uint32_t)(m >> 32) + (ae + be - (1024u << 20)) + (top << 20), lo = (uint32_t)m;
  if (ae == 0u || be == 0u) hi = lo = 0u;
  hi |= (ah ^ bh) & 0x80000000u;
  return bitsd((uint64_t)hi << 32 | lo);
}

// a / 3 (HALF = 0) or a / 6 (HALF = 1), correctly rounded, for zero or normal a with a
// normal quotient: the significand m, shifted to N = 2 m or 4 m so that N / 3 has 53
// bits, gives floor((N + 1) / 3), the nearest integer to N / 3 (whose fraction is 0,
// 1/3 or 2/3); the division by 3 is a multiplication by (2^64 + 2) / 3, exact below 2^63.
template <int HALF>
GB_HD double third_rn(double a) {
  const uint64_t ab = dbits(a);
  const uint32_t ah = (uint32_t)(ab >> 32);
  const uint64_t m = (ab & kFracBits) | kHidden;
  const uint32_t sh = (ah & 0x80000u) ? 1u : 2u;  // m >= 1.5 2^52
  const uint64_t q = mulhi64((m << sh) + 1u, 0x5555555555555556ull);
  uint32_t hi = (uint32_t)(q >> 32) + (ah & 0x7ff00000u) - ((sh + 1u + HALF) << 20), lo = (uint32_t)q;
  if ((ah & 0x7ff00000u) == 0u) hi = lo = 0u;
  hi |= ah & 0x80000000u;
  return bitsd((uint64_t)hi << 32 | lo);
}

// sqrt(a), correctly rounded, for zero or positive normal a.  With a = M 2^(2k - 104),
// M in [2^104, 2^106), the root's significand is the integer nearest to sqrt(M): an
// FP32 estimate s0 + c (s0 = x y, y = rsqrt(x), after one Newton step, c = (x - s0^2) y / 2)
// good to 2^-45, the remainder R = M - q^2 modulo 2^64 corrects it, and R against q
// settles the rounding ((q + 1/2)^2 = q^2 + q + 1/4, never equal to M).
GB_HD double sqrt_rn(double a) {
  const uint64_t ab = dbits(a);
  const uint32_t ea = (uint32_t)(ab >> 52), od = (ea & 1u) ^ 1u;  // od: an extra factor 2 makes the exponent even
  const uint64_t ma = (ab & kFracBits) | kHidden;
  const float xh = bitsf((((uint32_t)(ab >> 29) & 0x7fffffu) | 0x3f800000u) + (od << 23));
  const float xl = mul32(u32f((uint32_t)ab & 0x1fffffffu), od ? 4.440892098500626e-16f : 2.220446049250313e-16f);
  const float y = rsqrt32(xh), yh = mul32(0.5f, y), s1 = mul32(xh, y);
  const float s0 = fma32(fma32(-s1, s1, xh) + xl, yh, s1);
  const float c = mul32(fma32(-s0, s0, xh) + xl, yh);
  const uint32_t sb = fbits(s0);  // in [1, 2), or a few ulps outside
  const uint32_t pi = (sb & 0x7fffffu) | 0x800000u, s = (sb >> 23) - (127u - 29u);
  const int32_t ti = f32i(mul32(c, 281474976710656.0f));  // 2^48
  uint64_t q = ((uint64_t)(pi >> (32u - s)) << 32 | (uint32_t)(pi << s)) + (uint64_t)((int64_t)ti << 4);
  uint64_t R = (ma << (52u + od)) - q * q;
  const int32_t dq = f32i(mul32(i32f((int32_t)(R >> 32)), mul32(y, 4.76837158203125e-07f)));  // 2^-21
  R -= (uint64_t)(int64_t)dq * (2u * q + (uint64_t)(int64_t)dq);
  q += (uint64_t)(int64_t)dq;
  const int64_t Rs = (int64_t)R;
  const uint64_t up = Rs > (int64_t)q ? 1u : 0u, dn = Rs <= -(int64_t)q ? 1u : 0u;
  q += up;
  q -= dn;
  const uint64_t r = ((uint64_t)((ea + 1023u - od) / 2u - 1u) << 52) + q;
  return ea == 0u ? 0.0 : bitsd(r);
}

}  // namespace gb2d
