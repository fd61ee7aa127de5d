// wf_int64.cuh — products, quotients and square roots of doubles in integer
// operations, rounded to nearest even, for the FP64 passes (wf_step_fp64.cu).
//
// A warp's FP64 addition or multiplication takes ~19 cycles of an SM, a
// division ~140 and a square root ~140 (measured, 1.92 GHz); in 32-bit integer
// operations a product takes 12, a quotient 17 (known divisor) to 21 and a
// root 23, on pipes that are otherwise idle here and beside FP64 additions
// nearly for free.  The results are those of IEEE arithmetic to the
// bit; tests/test_34_gpu_int_arith.py compares them on ties, neighbours of
// products, quotients and squares, and the ends of the operands' range.
#pragma once
#include <cstdint>

// a b rounded to nearest even: the 53-bit significands' 106-bit product (one of
// them shifted up by 11, so that the upper 64 bits hold the 52 or 53 result
// bits), normalised by one bit, rounded by a carry out of the bits below, the
// exponents and signs added as one word.  For operands that are zero (a zero
// result is +0) or whose exponents keep the product inside the normal range.
__device__ __forceinline__ double mul_int(double a, double b) {
  const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
  const unsigned bh = (unsigned)__double2hiint(b), bl = (unsigned)__double2loint(b);
  const unsigned ua = (ah & 0xfffffu) | 0x100000u, ub = (bh & 0xfffffu) | 0x100000u;
  const unsigned xh = __funnelshift_l(al, ua, 11), xl = al << 11;
  const uint64_t p = (uint64_t)xl * bl;
  const uint64_t t = (uint64_t)xh * bl + (p >> 32);
  const uint64_t u = (uint64_t)xl * ub + (uint32_t)t;
  const uint64_t v = (uint64_t)xh * ub + (t >> 32) + (u >> 32);
  const unsigned w0 = (unsigned)p, w1 = (unsigned)u, w2 = (unsigned)v, w3 = (unsigned)(v >> 32);
  const unsigned k = w3 < 0x100000u ? 1u : 0u;          // 52 bits: shift up by one
  const unsigned mh = __funnelshift_l(w2, w3, k), ml = __funnelshift_l(w1, w2, k);
  const unsigned r1 = __funnelshift_l(w0, w1, k), r0 = w0 << k;
  const unsigned e = (ah & 0xfff00000u) + (bh & 0xfff00000u) - 0x3ff00000u - (k << 20);
  // up: the bits below (r1, r0) are over a half, or a half with an odd result:
  // r1 + 0x7fffffff + (r0 != 0 or odd) carries; the carry runs into the exponent
  unsigned lo, hi;
  asm("{\n\t.reg .u32 d;\n\t"
      "add.cc.u32 d, %2, 0xffffffff;\n\taddc.cc.u32 d, %3, 0x7fffffff;\n\t"
      "addc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, %6;\n\t}"
      : "=r"(lo), "=r"(hi)
      : "r"((ml & 1u) | r0), "r"(r1), "r"(ml), "r"(mh), "r"(e));
  const bool zero = (ah << 1) == 0u || (bh << 1) == 0u;
  return __hiloint2double(zero ? 0 : (int)hi, zero ? 0 : (int)lo);
}

// The significand of a normal number with its hidden bit, and its 24 upper
// bits as a float of [1, 2)
__device__ __forceinline__ uint64_t whole_bits(double x) {
  return (uint64_t)(((unsigned)__double2hiint(x) & 0xfffffu) | 0x100000u) << 32 |
         (unsigned)__double2loint(x);
}
__device__ __forceinline__ unsigned lead_bits(double x) {
  return (__funnelshift_l((unsigned)__double2loint(x), (unsigned)__double2hiint(x), 3) &
          0x7fffffu) | 0x3f800000u;
}
__device__ __forceinline__ unsigned word(uint64_t v, int shift) {   // bits shift .. shift + 31
  return __funnelshift_r((unsigned)v, (unsigned)(v >> 32), shift);
}
// 2^32 y of a float approximation 0.5 < y <= 1, from below: y (1 - 2^-21) + 1
// has its bits in the fraction field
__device__ __forceinline__ unsigned seed(float y) {
  return __float_as_uint(__fmaf_rn(y, 1.0f - 4.76837158203125e-7f, 1.0f)) << 9;
}

// a / b rounded to nearest even by long division with digits of 31 and 23
// bits (Knuth, The Art of Computer Programming 2, 4.3.1): the reciprocal of b
// to 29 bits from the float one and a Newton step, always from below, so a
// digit is at most a few units low; the next remainder takes them up, the last
// one decides the last bit.  q = N 2^-53 is then floored and N + 1 >> 1 is the
// rounded significand (a quotient of 53-bit numbers never lies in the middle).
// Operands as for mul_int, b not zero.
__device__ __forceinline__ double div_int(double a, double b) {
  const unsigned ah = (unsigned)__double2hiint(a), bh = (unsigned)__double2hiint(b);
  const uint64_t B = whole_bits(b);
  uint64_t A = whole_bits(a);
  const unsigned c = A < B ? 1u : 0u;
  A <<= c;                                              // A / B in [1, 2)
  float y0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(__uint_as_float(lead_bits(b))));
  const unsigned Y = seed(y0);
  const unsigned y = Y + __umulhi(Y, 0u - 2u * __umulhi(Y, word(B, 21)) - 4u);
  const unsigned q1 = __umulhi(word(A, 22), y);         // at most 5 low
  const uint64_t R = (A << 30) - (uint64_t)q1 * B;
  const unsigned q2 = __umulhi(word(R, 24), y) >> 5;    // at most 1 low
  const uint64_t R2 = (R << 23) - (uint64_t)q2 * B;
  const uint64_t M = (((uint64_t)q1 << 23) + q2 + (R2 >= B ? 2u : 1u)) >> 1;
  const unsigned e = (ah & 0xfff00000u) - (bh & 0xfff00000u) + 0x3fe00000u - (c << 20);
  const bool zero = (ah << 1) == 0u;
  return __hiloint2double(zero ? 0 : (int)((unsigned)(M >> 32) + e), zero ? 0 : (int)(unsigned)M);
}

// sqrt(x) rounded to nearest even, digit by digit the same way (x = 0 or
// normal): s1 of 31 bits from x / sqrt(x), the rest from the remainder over
// 2 s1, and N^2 <= x < (N + 1)^2 settled with the last remainder.
__device__ __forceinline__ double sqrt_int(double x) {
  const unsigned xh = (unsigned)__double2hiint(x);
  const unsigned odd = ~(xh >> 20) & 1u;                // of the unbiased exponent
  const uint64_t X = whole_bits(x) << odd;             // [1, 4) 2^52
  float y0;
  asm("rsqrt.approx.ftz.f32 %0, %1;"
      : "=f"(y0) : "f"(__uint_as_float(lead_bits(x) + (odd << 23))));
  const unsigned Y = seed(y0), x32 = word(X, 22);
  const unsigned y =
      Y + __umulhi(Y, 0x80000000u - 6u - 2u * __umulhi(__umulhi(Y, Y), x32));
  const unsigned s1 = __umulhi(x32, y);                 // at most 6 low
  const uint64_t R = (X << 8) - (uint64_t)s1 * s1;
  const int s2 = (int)(__umulhi(word(R, 3), y) - 8u) >> 5;   // at most 1 low, may be -1
  const uint64_t K = ((uint64_t)s1 << 24) + (uint64_t)(int64_t)s2;
  const uint64_t R2 = ((uint64_t)((unsigned)R << 14) << 32) - K * (uint64_t)(int64_t)s2;
  const uint64_t N = ((uint64_t)s1 << 23) + (uint64_t)(int64_t)s2;
  const uint64_t M = (N + (R2 > 2 * N ? 2u : 1u)) >> 1;
  const unsigned e = ((((xh >> 20) + 1023u) >> 1) - 1u) << 20;
  return __hiloint2double(xh == 0u ? 0 : (int)((unsigned)(M >> 32) + e),
                          xh == 0u ? 0 : (int)(unsigned)M);
}
