// Device forms of the reference's upwind schemes.  Expressions keep the
// reference's association order; the translation unit that instantiates the
// FP64 versions is compiled with --fmad=false so that they round exactly as the
// reference's FP64 CPU code (ADVECTION_METHOD_2D.h).
#pragma once

#include <cuda_runtime.h>

#include "gb2d_exact_math.cuh"
#include "gb2d_internal.cuh"

namespace gb2d {

// The two words of a double, and back.  The moves are opaque to the compiler, which
// otherwise recognises integer tests and masks of a double's bits and turns them into FP64
// comparisons and additions (a fabs or a negation is an FP64 addition on this part: the
// right-hand side kernel issued 15 FP64 instructions a node, 3 of them its sums).
struct Words {
  unsigned lo, hi;
};
__device__ __forceinline__ Words words(double x) {
  Words w;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(w.lo), "=r"(w.hi) : "d"(x));
  return w;
}
__device__ __forceinline__ double from_words(unsigned lo, unsigned hi) {
  double x;
  asm("mov.b64 %0, {%1, %2};" : "=d"(x) : "r"(lo), "r"(hi));
  return x;
}
__device__ __forceinline__ double absd(double x) {
  const Words w = words(x);
  return from_words(w.lo, w.hi & 0x7fffffffu);
}
__device__ __forceinline__ double negd(double x) {
  const Words w = words(x);
  return from_words(w.lo, w.hi ^ 0x80000000u);
}
__device__ __forceinline__ bool is_zero(double x) {
  const Words w = words(x);
  return ((w.hi << 1) | w.lo) == 0u;
}
// |x| as an integer (ordered as the magnitudes are; above kInfBits: NaN).
constexpr long long kAbsBits = 0x7fffffffffffffffLL, kInfBits = 0x7ff0000000000000LL;
__device__ __forceinline__ long long mag_bits(double x) {
  const Words w = words(x);
  return (long long)((unsigned long long)(w.hi & 0x7fffffffu) << 32 | w.lo);
}

// IEEE comparisons with zero.  FP64: on the integer pipes (an FP64 compare takes
// one of the part's few FP64 issue slots), exact for every input, NaN and
// infinities included.  FP32: the native compare.
__device__ __forceinline__ bool nan_words(Words w) {
  const unsigned h = w.hi & 0x7fffffffu;
  return h > 0x7ff00000u || (h == 0x7ff00000u && w.lo != 0u);
}
__device__ __forceinline__ bool gtz(double x) {  // x > 0
  const Words w = words(x);
  return (int)w.hi >= 0 && (w.hi | w.lo) != 0u && !nan_words(w);
}
__device__ __forceinline__ bool gez(double x) {  // x >= 0
  const Words w = words(x);
  return ((int)w.hi >= 0 || ((w.hi << 1) | w.lo) == 0u) && !nan_words(w);
}
__device__ __forceinline__ bool lez(double x) {  // x <= 0
  const Words w = words(x);
  return ((int)w.hi < 0 || (w.hi | w.lo) == 0u) && !nan_words(w);
}
__device__ __forceinline__ bool ltz(double x) {  // x < 0
  const Words w = words(x);
  return (int)w.hi < 0 && ((w.hi << 1) | w.lo) != 0u && !nan_words(w);
}
// |a| <= |b| (false when either is NaN), on the integer pipes.
__device__ __forceinline__ bool abs_le(double a, double b) {
  const long long ma = mag_bits(a), mb = mag_bits(b);
  return ma <= mb && mb <= kInfBits;
}
// x < -e and x > e for a finite e > 0, on the integer pipes (false for NaN).
__device__ __forceinline__ bool lt_neg(double x, double e) {
  const long long m = mag_bits(x);
  return (int)words(x).hi < 0 && m > mag_bits(e) && m <= kInfBits;
}
__device__ __forceinline__ bool gt_pos(double x, double e) {
  const long long m = mag_bits(x);
  return (int)words(x).hi >= 0 && m > mag_bits(e) && m <= kInfBits;
}

// Smeared Heaviside inside its band |phi| <= eps (HeavisideFunction,
// PROJECTION_2D.h:1441-1461 and VISCOSITY_2D.h:688-708), with the reference's
// PI = 3.141592 (MACROS.h:5); oe = 1/eps taken on the host.
__device__ __forceinline__ double heaviside_band(double phi, double oe) {
  const double PI_REF = 3.141592, opi = 1.0 / PI_REF;
  return 0.5 + phi * oe * 0.5 + 0.5 * opi * sin(PI_REF * phi * oe);
}
__device__ __forceinline__ double heaviside(double phi, double eps, double oe) {
  if (lt_neg(phi, eps)) return 0;
  if (gt_pos(phi, eps)) return 1;
  return heaviside_band(phi, oe);
}

// Maximum of non-negative doubles by their bit patterns (which order as
// integers): a warp's maximum, then one atomicMax into *out.
__device__ __forceinline__ void block_max_bits(unsigned long long b, unsigned long long* out) {
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long w = __shfl_xor_sync(0xffffffffu, b, o);
    b = w > b ? w : b;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(out, b);
}
// max(|x|, m) as the reference's `if (m <= |x|) m = |x|`: NaN never replaces m.
__device__ __forceinline__ unsigned long long abs_max_bits(double x, unsigned long long m) {
  const unsigned long long ab = (unsigned long long)mag_bits(x);
  return (ab > m && ab <= (unsigned long long)kInfBits) ? ab : m;
}

__device__ __forceinline__ bool gtz(float x) { return x > 0.0f; }
__device__ __forceinline__ bool gez(float x) { return x >= 0.0f; }
__device__ __forceinline__ bool lez(float x) { return x <= 0.0f; }
__device__ __forceinline__ bool ltz(float x) { return x < 0.0f; }

// a / 3 and a / 6, correctly rounded (IEEE binary64, round to nearest), in three
// FP64 operations instead of a division: with z = RN(1/d), q = RN(a z) lies within
// two ulps of a/d; the residual r = a - d q is then exactly representable and the
// FMA forms it exactly; RN(q + r z) has an error below 1e-15 ulp against a/d
// (the FMA correction step of P. Markstein, IBM J. Res. Dev. 34(1), 1990).  Since
// a is a multiple of 2 (d = 3) or 4 (d = 6) ulps of the quotient's binade, a/d
// sits at 0, 1/3 or 2/3 of an ulp from a representable number, never within 1/6
// ulp of a rounding midpoint, so that RN is the correctly rounded quotient.
// Magnitudes that could leave the normal range, zeros, infinities and NaN take
// the division.
template <int D>
__device__ __forceinline__ double div_by(double a) {
  static_assert(D == 3 || D == 6, "exact for 3 and 6");
  constexpr double z = D == 3 ? 0.33333333333333331483 : 0.16666666666666665741;  // RN(1/D)
  const int e = (int)((__double_as_longlong(a) >> 52) & 0x7ff);
  if (e < 64 || e > 1984) return a / (double)D;
  const double q = __dmul_rn(a, z);
  const double r = __fma_rn(-q, (double)D, a);
  return __fma_rn(r, z, q);
}

// Divisions in the type of the expression.  The exact FP64 path keeps IEEE
// quotients (div_by for the constants 3 and 6).  The FP32 flux path is an
// approximation of the scheme anyway: constants become reciprocal multiplies and
// the weights use the fast division (about 2 ulp).
__device__ __forceinline__ double cdiv3(double a) { return div_by<3>(a); }
__device__ __forceinline__ double cdiv6(double a) { return div_by<6>(a); }
__device__ __forceinline__ float cdiv3(float a) { return a * (1.0f / 3.0f); }
__device__ __forceinline__ float cdiv6(float a) { return a * (1.0f / 6.0f); }
__device__ __forceinline__ double vdiv(double a, double b) { return a / b; }
__device__ __forceinline__ float vdiv(float a, float b) { return __fdividef(a, b); }

// WENO5 one-sided derivative from five first differences (ADVECTION_METHOD_2D.h:545-619).
template <typename R>
__device__ __forceinline__ R weno5_side(R a1, R a2, R a3, R a4, R a5, R eps) {
  const R c13 = R(13.0 / 12.0);
  const R q = R(0.25);
  R A1 = a1 - R(2) * a2 + a3, B1 = a1 - R(4) * a2 + R(3) * a3;
  R A2 = a2 - R(2) * a3 + a4, B2 = a2 - a4;
  R A3 = a3 - R(2) * a4 + a5, B3 = R(3) * a3 - R(4) * a4 + a5;
  R s1 = c13 * A1 * A1 + q * B1 * B1;
  R s2 = c13 * A2 * A2 + q * B2 * B2;
  R s3 = c13 * A3 * A3 + q * B3 * B3;
  R al1 = vdiv(R(1.0 / 10.0), (eps + s1) * (eps + s1));
  R al2 = vdiv(R(6.0 / 10.0), (eps + s2) * (eps + s2));
  R al3 = vdiv(R(3.0 / 10.0), (eps + s3) * (eps + s3));
  R sum = al1 + al2 + al3;
  R w1 = vdiv(al1, sum), w2 = vdiv(al2, sum), w3 = vdiv(al3, sum);
  const R cm16 = R((-1.0) / 6.0);
  return w1 * (cdiv3(a1) - cdiv6(a2 * R(7)) + cdiv6(a3 * R(11))) + w2 * (a2 * cm16 + cdiv6(a3 * R(5)) + cdiv3(a4)) +
         w3 * (cdiv3(a3) + cdiv6(a4 * R(5)) - cdiv6(a5));
}

// Zero, or a magnitude in [2^-E, 2^E): operands in this range keep every product and
// quotient of the fast forms below normal (each caller states its E).
template <int E>
__device__ __forceinline__ bool mid_range(double d) {
  const Words w = words(d);
  return (w.hi & 0x7fffffffu) - ((1023u - E) << 20) < ((2u * E) << 20) || ((w.hi << 1) | w.lo) == 0u;
}

// The plain FP64 product, for operands outside a fast form's range.  Out of line:
// inlined, the compiler evaluates both forms and selects.
static __device__ __noinline__ double plain_mul(double a, double b) { return a * b; }
// a b for b in [2^-100, 2^100] on the integer pipes; where the product may leave the
// normal range the FP64 multiply.  An FP64 instruction takes an SM's FP64 pipe 16 cycles a
// warp and mul_rn its integer pipes about 14, so a kernel is fastest with its products
// shared out between the two.
__device__ __forceinline__ double mul_wide(double a, double b) { return mid_range<900>(a) ? mul_rn(a, b) : plain_mul(a, b); }

// weno5_side<float> with the same bits and ten operations fewer, for differences below
// 1e30 and epsilon >= 1e-15 (which absorbs a B B that underflows): doublings, quadruplings
// and quarters are exact and join their sums as FMAs, 3 a3 is formed once.
__device__ __forceinline__ float weno5_side_f32(float a1, float a2, float a3, float a4, float a5, float eps) {
  const float c13 = 13.0 / 12.0, cm16 = (-1.0) / 6.0;
  const float t3 = 3.0f * a3;
  const float A1 = __fmaf_rn(-2.0f, a2, a1) + a3, B1 = __fmaf_rn(-4.0f, a2, a1) + t3;
  const float A2 = __fmaf_rn(-2.0f, a3, a2) + a4, B2 = a2 - a4;
  const float A3 = __fmaf_rn(-2.0f, a4, a3) + a5, B3 = __fmaf_rn(-4.0f, a4, t3) + a5;
  const float e1 = eps + __fmaf_rn(0.25f, B1 * B1, c13 * A1 * A1);
  const float e2 = eps + __fmaf_rn(0.25f, B2 * B2, c13 * A2 * A2);
  const float e3 = eps + __fmaf_rn(0.25f, B3 * B3, c13 * A3 * A3);
  const float al1 = vdiv(float(1.0 / 10.0), e1 * e1), al2 = vdiv(float(6.0 / 10.0), e2 * e2), al3 = vdiv(float(3.0 / 10.0), e3 * e3);
  const float sum = al1 + al2 + al3;
  return vdiv(al1, sum) * (cdiv3(a1) - cdiv6(a2 * 7.0f) + cdiv6(a3 * 11.0f)) + vdiv(al2, sum) * (a2 * cm16 + cdiv6(a3 * 5.0f) + cdiv3(a4)) +
         vdiv(al3, sum) * (cdiv3(a3) + cdiv6(a4 * 5.0f) - cdiv6(a5));
}

// Range of the differences (and of epsilon) in which weno5_side_fast equals
// weno5_side<double> bit for bit: zero, or a magnitude in [2^-300, 2^100);
// epsilon in [2^-100, 2^100].
__device__ __forceinline__ bool weno5_in_range(double d) {
  const Words w = words(d);
  return (w.hi & 0x7fffffffu) - ((1023u - 300u) << 20) < (400u << 20) || ((w.hi << 1) | w.lo) == 0u;
}

// weno5_side<double> with the same bits and a fifth of its FP64 operations (27
// against 140 and more), for differences and epsilon in the range above: no
// intermediate result overflows, and none but an exact zero is below 2^-1022.
//   * Every product, the six divisions and the constant thirds and sixths run on the
//     integer and FP32 pipes (gb2d_exact_math.cuh), correctly rounded; only the sums
//     are left to the FP64 pipe.
//   * Doubling and quadrupling are exact: RN(a1 - RN(2 a2)) is one FMA, and
//     0.25 B B = RN(B B) / 4 joins its sum as an FMA.
__device__ __forceinline__ double weno5_side_fast(double a1, double a2, double a3, double a4, double a5, double eps) {
  const double c13 = 13.0 / 12.0, cm16 = (-1.0) / 6.0;
  const double t3 = mul_rn(a3, 3.0);
  const double A1 = __fma_rn(-2.0, a2, a1) + a3, B1 = __fma_rn(-4.0, a2, a1) + t3;
  const double A2 = __fma_rn(-2.0, a3, a2) + a4, B2 = a2 - a4;
  const double A3 = __fma_rn(-2.0, a4, a3) + a5, B3 = __fma_rn(-4.0, a4, t3) + a5;
  const double e1 = eps + __fma_rn(0.25, mul_rn(B1, B1), mul_rn(mul_rn(A1, c13), A1));
  const double e2 = eps + __fma_rn(0.25, mul_rn(B2, B2), mul_rn(mul_rn(A2, c13), A2));
  const double e3 = eps + __fma_rn(0.25, mul_rn(B3, B3), mul_rn(mul_rn(A3, c13), A3));
  const double al1 = div_pos(1.0 / 10.0, mul_rn(e1, e1)), al2 = div_pos(6.0 / 10.0, mul_rn(e2, e2)),
               al3 = div_pos(3.0 / 10.0, mul_rn(e3, e3));
  const double sum = al1 + al2 + al3;
  const double p1 = third_rn<0>(a1) - third_rn<1>(mul_rn(a2, 7.0)) + third_rn<1>(mul_rn(a3, 11.0));
  const double p2 = mul_rn(a2, cm16) + third_rn<1>(mul_rn(a3, 5.0)) + third_rn<0>(a4);
  const double p3 = third_rn<0>(a3) + third_rn<1>(mul_rn(a4, 5.0)) - third_rn<1>(a5);
  return mul_rn(div_pos(al1, sum), p1) + mul_rn(div_pos(al2, sum), p2) + mul_rn(div_pos(al3, sum), p3);
}

// Sign of a WENO5 one-sided derivative from FP32 copies of its differences, or 0
// where that is not certain.  The derivative is a convex combination of three
// candidate stencils, so it has their sign when they agree; the margin 2^-13 max|a|
// on six times a candidate is 16 times the error of the truncated inputs and the
// FP32 sums (20 max|a| 2^-21.6).
__device__ __forceinline__ int weno5_sign(float a1, float a2, float a3, float a4, float a5) {
  const float p1 = fmaf(11.0f, a3, fmaf(-7.0f, a2, 2.0f * a1));
  const float p2 = fmaf(2.0f, a4, fmaf(5.0f, a3, -a2));
  const float p3 = fmaf(5.0f, a4, fmaf(2.0f, a3, -a5));
  const float m = fmaxf(fmaxf(fmaxf(fabsf(a1), fabsf(a2)), fmaxf(fabsf(a3), fabsf(a4))), fabsf(a5));
  const float thr = m * 1.220703125e-4f;
  if (!(m > 1e-25f)) return 0;
  return fminf(fminf(p1, p2), p3) > thr ? 1 : fmaxf(fmaxf(p1, p2), p3) < -thr ? -1 : 0;
}

// Mixed pair: differences of the FP64 state formed in FP64, everything after in
// FP32 (the FP64 -> FP32 moves by truncation on the integer pipes).
__device__ __forceinline__ void weno5_pair_f32(const double q[7], float o, float eps, float& dm, float& dp) {
  float d[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) d[k] = narrow(q[k + 1] - q[k]) * o;
  dm = weno5_side<float>(d[0], d[1], d[2], d[3], d[4], eps);
  dp = weno5_side<float>(d[5], d[4], d[3], d[2], d[1], eps);
}

// Godunov selection of WENO5thReinitialization (ADVECTION_METHOD_2D.h:1505-1655).
// Returns false where the reference leaves phi unchanged (tie sss == 0 or NaN);
// otherwise h = |grad phi| - 1 over the selected one-sided derivatives.
// godunov_pick: one direction's choice from its one-sided derivatives m, p: 0 m, 1 p, 2 neither,
// -1 unchanged.  along_x: only there a tie of the shock rule leaves phi unchanged.
template <typename R>
__device__ __forceinline__ int godunov_pick(R s, R m, R p, bool along_x) {
  const R sm = s * m, sp = s * p;
  if (gez(sp) && gez(sm)) return 0;
  if (lez(sp) && lez(sm)) return 1;
  if (gtz(sp) && ltz(sm)) return 2;
  if (ltz(sp) && gtz(sm)) {
    const R sss = s * (fabs(p) - fabs(m)) / (p - m);
    if (gtz(sss)) return 0;
    return along_x && !ltz(sss) ? -1 : 1;
  }
  return -1;
}
template <typename R>
__device__ __forceinline__ bool godunov_h(R s, R mx, R px, R my, R py, R& h) {
  const int xs = godunov_pick(s, mx, px, true);
  if (xs < 0) return false;
  const int ys = godunov_pick(s, my, py, false);
  if (ys < 0) return false;
  R gx = xs == 0 ? mx : px, gy = ys == 0 ? my : py;
  if (xs != 2 && ys != 2)
    h = sqrt(gx * gx + gy * gy) - R(1);
  else if (xs != 2)
    h = sqrt(gx * gx) - R(1);
  else if (ys != 2)
    h = sqrt(gy * gy) - R(1);
  else
    h = R(-1);
  return true;
}

// ENO3 one-sided derivatives by divided-difference selection (ADVECTION_METHOD_2D.h:2054-2111),
// from the six first divided differences d[0..5] (offsets -3..+2).
__device__ __forceinline__ bool mag_le(double a, double b) { return abs_le(a, b); }
__device__ __forceinline__ bool mag_le(float a, float b) { return fabsf(a) <= fabsf(b); }
template <typename R>
__device__ __forceinline__ void eno3_select(const R d[6], R o2, R o3, R h, R& dm, R& dp) {
  const R d1n1 = d[2], d10 = d[3];
  R d2n2 = o2 * (d[1] - d[0]), d2n1 = o2 * (d[2] - d[1]), d20 = o2 * (d[3] - d[2]);
  R d2p1 = o2 * (d[4] - d[3]), d2p2 = o2 * (d[5] - d[4]);
  R d3n2 = o3 * (d2n1 - d2n2), d3n1 = o3 * (d20 - d2n1), d30 = o3 * (d2p1 - d20), d3p1 = o3 * (d2p2 - d2p1);
  if (mag_le(d2n1, d20)) {
    if (mag_le(d3n2, d3n1))
      dm = d1n1 + d2n1 * h + R(2) * d3n2 * h * h;
    else
      dm = d1n1 + d2n1 * h + R(2) * d3n1 * h * h;
  } else {
    if (mag_le(d3n1, d30))
      dm = d1n1 + d20 * h - d3n1 * h * h;
    else
      dm = d1n1 + d20 * h - d30 * h * h;
  }
  if (mag_le(d20, d2p1)) {
    if (mag_le(d3n1, d30))
      dp = d10 - d20 * h - d3n1 * h * h;
    else
      dp = d10 - d20 * h - d30 * h * h;
  } else {
    if (mag_le(d30, d3p1))
      dp = d10 - d2p1 * h + R(2) * d30 * h * h;
    else
      dp = d10 - d2p1 * h + R(2) * d3p1 * h * h;
  }
}

// Exact FP64 pair: q[0..6] are values at offsets -3..+3.
__device__ __forceinline__ void eno3_pair(const double q[7], double o, double o2, double o3, double h, double& dm, double& dp) {
  double d[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) d[k] = o * (q[k + 1] - q[k]);
  eno3_select<double>(d, o2, o3, h, dm, dp);
}

}  // namespace gb2d
