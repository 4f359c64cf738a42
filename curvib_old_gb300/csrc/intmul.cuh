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

__device__ __forceinline__ IntMulB int_split_b(double x, bool &out_of_range) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const bool zero = ((h & 0x7fffffffu) | l) == 0;
  out_of_range = out_of_range || (!zero && !int_mul_in_range(h));
  const unsigned m = zero ? 0u : (h & 0xfffffu) | 0x100000u;
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

// 3 x and 9 x rounded to nearest even: the significand's multiple has one or two
// (three or four) bits too many.  Other than normal numbers with a normal result
// and zeros go through the multiply, out of line.
static __device__ __noinline__ double times_slow(double x, double k) { return __dmul_rn(k, x); }
template <int K>
__device__ __forceinline__ double int_times(double x) {
  static_assert(K == 3 || K == 9, "");
  constexpr int S = K == 3 ? 1 : 3;
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
  if (e - 1u >= 2045u - S) return (b << 1) == 0 ? x : times_slow(x, K);
  const unsigned long long m = (b & 0xfffffffffffffULL) | 0x10000000000000ULL, t = K * m;
  const int s = t >> (53 + S) ? S + 1 : S;
  const unsigned long long r = (t + ((1u << (s - 1)) - 1) + ((t >> s) & 1)) >> s;
  return __longlong_as_double((long long)((b & 0x8000000000000000ULL) + r + ((unsigned long long)(e + s - 1) << 52)));
}
__device__ __forceinline__ double int_triple(double x) { return int_times<3>(x); }

// x 2^-K as the FP64 multiply gives it: K less in the exponent field while the
// result stays normal; a zero stays itself; subnormal results, inf and NaN go
// through the multiply, out of line.
static __device__ __noinline__ double scale_slow(double x, int K) {
  return __dmul_rn(x, __longlong_as_double((long long)(1023 - K) << 52));
}
__device__ __forceinline__ double scale_down(double x, int K) {
  const long long b = __double_as_longlong(x), e = (b >> 52) & 0x7ff;
  if (e > K && e < 0x7ff) return __longlong_as_double(b - ((long long)K << 52));
  if ((b & 0x7fffffffffffffffLL) == 0) return x;
  return scale_slow(x, K);
}
template <int K>
__device__ __forceinline__ double scale_down(double x) {
  return scale_down(x, K);
}

// Whether v can be a right operand of int_mul (host).
inline bool int_mul_factor(double v) {
  const double a = v < 0 ? -v : v;
  return a >= 0x1p-510 && a < 0x1p511;
}

// (double)f and (float)v on the integer pipe (a conversion costs an FP64 operation):
// the same bits for zeros and numbers with a normal result, others go through the
// conversion, out of line.
static __device__ __noinline__ double widen_slow(float f) { return (double)f; }
__device__ __forceinline__ double int_widen(float f) {
  const unsigned u = __float_as_uint(f), m = u & 0x7fffffffu;
  if (m - 0x00800000u >= 0x7f000000u && m) return widen_slow(f);
  const unsigned h = (((unsigned)((int)u >> 3)) & 0x8fffffffu) + (896u << 20);
  return __hiloint2double((int)(m ? h : u), (int)(u << 29));
}
static __device__ __noinline__ float narrow_slow(double v) { return (float)v; }
__device__ __forceinline__ float int_narrow(double v) {
  const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v), e = (h >> 20) & 0x7ffu;
  if (e - 897u < 254u - 1u) {  // a rounding up stays finite
    const unsigned m = __funnelshift_l(l, h & 0x7fffffffu, 3) - (896u << 23), rest = l << 3;
    // up where the rest is above half a unit, or is half and m odd
    return __uint_as_float((h & 0x80000000u) | (m + (rest > 0x80000000u || (rest == 0x80000000u && (m & 1)))));
  }
  return ((h & 0x7fffffffu) | l) == 0 ? __uint_as_float(h) : narrow_slow(v);
}

// x / y rounded to nearest even for a divisor used many times, from rcp = 1 / y
// rounded to nearest: x rcp, then twice the residual x - y q added back through
// rcp.  The residual of a quotient within an ulp is exact in one fused
// multiply-add, and a quotient within an ulp so corrected with a correctly
// rounded reciprocal is the correctly rounded one (P. W. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34, 1990); x rcp itself may be off by more than an ulp, the
// first correction makes it so.  Five FP64 operations.  For y and rcp within
// int_mul's range and |x| within 2^-400 .. 2^400 (nothing over- or underflows
// on the way), or x zero; other x take the division, out of line.
static __device__ __noinline__ double quot_slow(double x, double y) { return __ddiv_rn(x, y); }
__device__ __forceinline__ double quot_known(double x, double y, double rcp) {
  const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
  if ((h | (unsigned)__double2loint(x)) == 0)
    return __hiloint2double((__double2hiint(x) ^ __double2hiint(y)) & 0x80000000, 0);
  if (h - (623u << 20) >= (800u << 20)) return quot_slow(x, y);
  double q = __dmul_rn(x, rcp);
  q = __fma_rn(__fma_rn(-y, q, x), rcp, q);
  return __fma_rn(__fma_rn(-y, q, x), rcp, q);
}

}  // namespace cvb
