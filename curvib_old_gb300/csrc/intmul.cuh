// FP64 products on the integer pipe.
//
// GB300 issues about two FP64 operations per SM per clock, 1/32 of what its
// integer pipe does, and the momentum kernels, whose every product and sum
// must round on its own as the reference's C does, are bound by it.  The
// product of two doubles rounded to nearest even is integer arithmetic by its
// definition (IEEE 754-2008, 5.4.1 and 4.3.1): the exact 106-bit product of
// the two significands, shifted so that its leading bit is the 53rd, rounded
// on the bits below, and the sum of the exponents.  So the products go to the
// integer pipe, the sums stay on the FP64 one, and both run at once.  Measured
// on a GB300 (six blocks of 256 threads per SM): 20.3 SM clocks a warp for an
// FP64 multiply, 16.7 for int_mul with one operand split on the way, 10.3 a
// product with every other one on either pipe.
//
// Operands are split once and used in several products.  They must be zero
// (of either sign) or have an exponent field of 513 .. 1534 (2^-510 to
// 2^511), so that every product's field is within 2 .. 2046; int_split_a says
// where one is not, and the caller then takes the FP64 multiplies.  The
// results are the FP64 multiply's bit for bit.
#pragma once

namespace cvb {

// A split operand: the significand with its leading one, shifted left by 5
// (left operand) or 6 (right), and the sign and exponent field in place.  A
// zero has a zero significand.
struct IntMulA {
  unsigned lo, hi, se;
};
struct IntMulB {
  unsigned lo, hi, se;
};

__device__ __forceinline__ bool int_mul_in_range(unsigned h) {
  return (h & 0x7fffffffu) - (513u << 20) < (1022u << 20);
}

__device__ __forceinline__ IntMulA int_split_a(double x, bool &out_of_range) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const bool zero = ((h & 0x7fffffffu) | l) == 0;
  out_of_range = out_of_range || (!zero && !int_mul_in_range(h));
  const unsigned m = zero ? 0u : (h & 0xfffffu) | 0x100000u;
  return {l << 5, __funnelshift_l(l, m, 5), h & 0xfff00000u};
}
// The range of a right operand is the caller's to know (the metrics' is
// checked once per grid).
__device__ __forceinline__ IntMulB int_split_b(double x) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const unsigned m = ((h & 0x7fffffffu) | l) == 0 ? 0u : (h & 0xfffffu) | 0x100000u;
  return {l << 6, __funnelshift_l(l, m, 6), h & 0xfff00000u};
}

// a * b rounded to nearest even.  The shifted significands A < 2^58, B < 2^59
// give A B = S_a S_b 2^11 in [2^115, 2^117): bits 64 .. 116 are the 53-bit
// significand of the result (one bit short where the product of the
// significands is below 2), the bits below decide the rounding.  A's and B's
// low words end in 5 and 6 zeros, so the product's lowest word ends in 11 and
// its other bits fit below the rounding bit of the word above (sticky).
__device__ __forceinline__ double int_mul(const IntMulA &a, const IntMulB &b) {
  const unsigned long long t = (unsigned long long)a.lo * b.lo;
  const unsigned long long u = (unsigned long long)a.hi * b.lo + (t >> 32);
  const unsigned long long v = (unsigned long long)a.lo * b.hi + u;  // < 2^61: no carry out
  const unsigned long long w = (unsigned long long)a.hi * b.hi + (v >> 32);
  unsigned r = (unsigned)v | ((unsigned)t >> 11), wl = (unsigned)w, wh = (unsigned)(w >> 32);
  const unsigned top = wh & 0x100000u;
  const int sh = top ? 0 : 1;
  wh = __funnelshift_l(wl, wh, sh);
  wl = __funnelshift_l(r, wl, sh);
  r <<= sh;
  // up where the rest is above 1/2, or is 1/2 and the last bit odd: the carry
  // out of rest + (2^31 - 1) + (last bit)
  unsigned lo, hi;
  asm("{ .reg .u32 t; add.cc.u32 t, %2, %3; addc.cc.u32 %0, %4, 0; addc.u32 %1, %5, 0; }"
      : "=r"(lo), "=r"(hi)
      : "r"(r), "r"(0x7fffffffu + (wl & 1u)), "r"(wl), "r"(wh));
  // exponents add (bias 1023, one less for the leading bit of hi, one more
  // where the product was 2 or above) and the signs with them, modulo 2^32
  const unsigned se = hi + a.se + b.se + (top - (1024u << 20));
  return __hiloint2double(hi ? se : (a.se ^ b.se) & 0x80000000u, lo);
}

}  // namespace cvb
