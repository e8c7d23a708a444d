/*
 * axg_soft64.h -- IEEE double products on the integer pipes, correctly
 * rounded (round to nearest, ties to even), bit for bit the hardware's; and
 * the split of a double into two floats there (axs_split).
 *
 * GB300 issues FP64 at 1/64 of the FP32 rate: measured, an SM retires 1.7
 * FP64 operations a clock against 57 32 x 32 -> 64-bit integer products, 57
 * logic operations or shifts and 110 integer adds, and the integer pipes are
 * idle in an FP64 stencil.  A product written out in integers is about 26
 * instructions, some 31 clocks of the busiest integer pipe per warp against
 * 75 on the FP64 pipe, and runs beside it.  Sums stay on the FP64 pipe: the
 * alignment and normalising shifts make an integer sum as long as an FP64 one.
 *
 * The fast path takes operands with exponents in [-511, 512] (axs_in_window):
 * then the operands are normal and so is the product.  Anything else (zeros,
 * subnormals, infinities, NaN, extreme exponents) clears a bit of `ok`, and
 * the caller redoes its block of arithmetic with hardware operations.
 *
 * Method: the operands' significands A, C (53 bits, A shifted left by 11) are
 * multiplied exactly; the upper 64 bits hold 52 or 53 bits of the quotient
 * A C / 2^53, the lower 64 the fraction F.  With the significand normalised
 * to 53 bits M, rounding to nearest even adds the carry of
 * F + 2^63 - 1 + (M mod 2) over 64 bits; a carry out of M increments the
 * exponent field it is added beside.
 *
 * Plain C++ (no CUDA needed) except for the carry chain in device code, so a
 * CPU test compiles it and compares it with the host's multiplication.
 */
#ifndef AXG_SOFT64_H
#define AXG_SOFT64_H

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define AXS_FN static __host__ __device__ __forceinline__
#else
#define AXS_FN static inline
#endif

/* A factor that many products share, taken apart once on the host: the
 * significand, the exponent field less 1024 and the sign, in place. */
typedef struct {
  uint32_t lo, hi, exp, sign;
  double v;
  uint32_t ok; /* 0: outside the window (axs_mulc must not be used) */
} axs_const;

AXS_FN uint32_t axs_hi(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2hiint(x);
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return (uint32_t)(b >> 32);
#endif
}
AXS_FN uint32_t axs_lo(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2loint(x);
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return (uint32_t)b;
#endif
}
AXS_FN double axs_make(uint32_t hi, uint32_t lo) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t b = (uint64_t)hi << 32 | lo;
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}

/* bit 30 is set when the exponent of the double with high word h lies in
 * [-511, 512], i.e. when the top two bits of its exponent field differ */
AXS_FN uint32_t axs_in_window(uint32_t h) { return h ^ (h + h); }
#define AXS_WINDOW 0x40000000u
AXS_FN uint32_t axs_window2(double a, double b) { return axs_in_window(axs_hi(a)) & axs_in_window(axs_hi(b)); }

AXS_FN axs_const axs_const_of(double v) {
  const uint32_t h = axs_hi(v);
  axs_const c;
  c.lo = axs_lo(v);
  c.hi = (h & 0xfffffu) | 0x100000u;
  c.exp = (h & 0x7ff00000u) - (1024u << 20);
  c.sign = h & 0x80000000u;
  c.v = v;
  /* below 2^476: the product with an operand in the window stays finite */
  c.ok = ((axs_in_window(h) & AXS_WINDOW) && (h & 0x7ff00000u) < (1500u << 20)) ? 1u : 0u;
  return c;
}

/* the product of the significands ah:al 2^11 and ch:cl, rounded to 53 bits;
 * exp: the exponent fields' sum less 1024.  Returns the double's magnitude */
AXS_FN double axs_mul_core(uint32_t ah, uint32_t al, uint32_t ch, uint32_t cl, uint32_t exp, uint32_t sign,
                           uint32_t *hi_out) {
  const uint64_t t0 = (uint64_t)al * cl;
  const uint64_t t1 = (uint64_t)al * ch + (uint32_t)(t0 >> 32);
  const uint64_t t2 = (uint64_t)ah * cl + (uint32_t)t1;
  const uint64_t H = (uint64_t)ah * ch + (uint32_t)(t1 >> 32) + (uint32_t)(t2 >> 32);
  uint32_t hh = (uint32_t)(H >> 32), hl = (uint32_t)H, lt = (uint32_t)t2, ll = (uint32_t)t0;
  const uint32_t e = exp + (hh & 0x100000u); /* one more when the quotient has 53 bits */
#if defined(__CUDA_ARCH__)
  asm("{\n\t.reg .pred p;\n\t.reg .u32 t;\n\t"
      "setp.lt.u32 p, %0, 0x100000;\n\t" /* 52 bits: one place to the left */
      "@p add.cc.u32 %3, %3, %3;\n\t"
      "@p addc.cc.u32 %2, %2, %2;\n\t"
      "@p addc.cc.u32 %1, %1, %1;\n\t"
      "@p addc.u32 %0, %0, %0;\n\t"
      "and.b32 t, %1, 1;\n\t"
      "add.cc.u32 t, t, 0xffffffff;\n\t"
      "addc.cc.u32 t, %3, 0xffffffff;\n\t"
      "addc.cc.u32 t, %2, 0x7fffffff;\n\t"
      "addc.cc.u32 %1, %1, 0;\n\t"
      "addc.u32 %0, %0, %4;\n\t}"
      : "+r"(hh), "+r"(hl), "+r"(lt), "+r"(ll)
      : "r"(e));
#else
  if (hh < 0x100000u) {
    hh = hh << 1 | hl >> 31;
    hl = hl << 1 | lt >> 31;
    lt = lt << 1 | ll >> 31;
    ll <<= 1;
  }
  {
    const uint64_t F = (uint64_t)lt << 32 | ll, add = 0x7fffffffffffffffull + (hl & 1u);
    const uint64_t M = ((uint64_t)hh << 32 | hl) + (F + add < F ? 1u : 0u);
    hl = (uint32_t)M;
    hh = (uint32_t)(M >> 32) + e;
  }
#endif
  *hi_out = hh;
  return axs_make(hh | sign, hl);
}

/* a c; clears bit 30 of *ok when a is outside the window (c.ok must hold) */
AXS_FN double axs_mulc(double a, const axs_const *c, uint32_t *ok) {
  const uint32_t h = axs_hi(a), l = axs_lo(a), m = (h & 0xfffffu) | 0x100000u;
  uint32_t rh;
  *ok &= axs_in_window(h);
  return axs_mul_core(m << 11 | l >> 21, l << 11, c->hi, c->lo, (h & 0x7ff00000u) + c->exp, (h ^ c->sign) & 0x80000000u,
                      &rh);
}

/* a b; clears bit 30 of *ok when a or b is outside the window or the product
 * overflows */
AXS_FN double axs_mul(double a, double b, uint32_t *ok) {
  const uint32_t h = axs_hi(a), l = axs_lo(a), m = (h & 0xfffffu) | 0x100000u;
  const uint32_t g = axs_hi(b);
  uint32_t rh;
  const double r = axs_mul_core(m << 11 | l >> 21, l << 11, (g & 0xfffffu) | 0x100000u, axs_lo(b),
                                (h & 0x7ff00000u) + (g & 0x7ff00000u) - (1024u << 20), (h ^ g) & 0x80000000u, &rh);
  *ok &= axs_in_window(h) & axs_in_window(g);
  if (rh >= 0x7ff00000u) *ok = 0;
  return r;
}

/* x as the sum of two floats, the bits of (float)x and (float)(x - (float)x):
 * h is x rounded to 24 bits (a tie away from zero, which moves h and l but not
 * their sum), l the low 29 bits less what h took, as a signed integer converted
 * to float and scaled by the power of two of its place.  |x - h - l| <= 2^-49
 * |x|.  0: outside [2^-74, 2^127) (zeros, subnormals, non-finite x too), where
 * the conversions have to do it. */
AXS_FN int axs_split(double x, float *h, float *l) {
  const uint32_t hi = axs_hi(x), lo = axs_lo(x), e = (hi >> 20) & 0x7ffu, sign = hi & 0x80000000u;
  const uint32_t hb = sign | ((((e - 896u) << 23) | (hi & 0xfffffu) << 3 | lo >> 29) + (lo >> 28 & 1u));
  const float r = (float)((int32_t)(lo << 3) >> 3);
#if defined(__CUDA_ARCH__)
  *h = __uint_as_float(hb);
  *l = __uint_as_float(__float_as_uint(__fmul_rn(r, __uint_as_float((e - 948u) << 23))) ^ sign);
#else
  const uint32_t sb = ((e - 948u) & 0xffu) << 23;
  uint32_t lb;
  float scale, v;
  memcpy(h, &hb, 4);
  memcpy(&scale, &sb, 4);
  v = r * scale;
  memcpy(&lb, &v, 4);
  lb ^= sign;
  memcpy(l, &lb, 4);
#endif
  return e >= 949u && e <= 1149u;
}

#endif
