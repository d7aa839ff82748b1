// fvm_ieee64.h -- binary64 products and quotients in integer arithmetic,
// equal bit for bit to the IEEE round-to-nearest-even operations.
//
// This GPU's FP64 pipe passes 2 lanes per SM and clock: a warp instruction
// every 64 cycles of an SM quarter, a division or square root about 7.5 of
// them (measured: 500, 68 and 65 G operations/s).  Its integer pipes pass 64
// lanes and stand idle meanwhile.  In integer instructions a product runs at
// 620, a quotient at 340 and a square root at 310 G/s, beside the sums on the
// FP64 pipe (a product and a sum together: 500 G pairs/s against 250).
//
// The operations below are schoolbook integer arithmetic on the significands;
// operands outside a window of exponents (zeros, subnormals, very large or
// small values, infinities, NaN) take the hardware operation, so nothing
// special is decided here.
//
// Plain C++: the same functions compile for the host, where they are tested
// against the machine's own operations.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define FVM_I64 __host__ __device__ __forceinline__
#else
#define FVM_I64 inline
#endif

namespace fvm {

FVM_I64 uint64_t i64_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
FVM_I64 double i64_double(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t u = ((uint64_t)hi << 32) | lo;
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
FVM_I64 float i64_float(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  memcpy(&x, &u, 4);
  return x;
#endif
}
// high word of (hi:lo) << s, 0 <= s < 32
FVM_I64 uint32_t i64_shl(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return (uint32_t)(((((uint64_t)hi << 32) | lo) << s) >> 32);
#endif
}
FVM_I64 uint32_t i64_mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
// 1/x and 1/sqrt(x) of a float, to 2^-22 (FVM_I64_OFF: a relative error that
// the host test adds to its own)
#ifndef FVM_I64_OFF
#define FVM_I64_OFF 0.0f
#endif
FVM_I64 float i64_rcp(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  const float r = 1.0f / x;
  return x == 1.0f ? r : r + r * (FVM_I64_OFF);
#endif
}
FVM_I64 float i64_rsqrt(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  const float r = 1.0f / sqrtf(x);
  return x == 1.0f ? r : r + r * (FVM_I64_OFF);
#endif
}

// Window of all operations: both operands' magnitudes in [2^-255, 2^257), so
// that the result is a normal number.  x: the exponent field less 768.
FVM_I64 bool i64_outside(uint32_t x) { return (x & 0xe0000000u) != 0u; }

// The hardware operations, for operands outside the window.  Not inlined: the
// compiler would otherwise issue the FP64 instruction for every lane and
// select, which is the cost to avoid (measured: no gain at all).
#ifdef __CUDACC__
#define FVM_I64_CALL inline __host__ __device__ __noinline__
#else
#define FVM_I64_CALL inline
#endif
FVM_I64_CALL double i64_hw_mul(double a, double b) { return a * b; }
FVM_I64_CALL double i64_hw_div(double a, double b) { return a / b; }
FVM_I64_CALL double i64_hw_sqrt(double a) { return sqrt(a); }

// Product.
FVM_I64 double mul64(double a, double b) {
  const uint64_t ua = i64_bits(a), ub = i64_bits(b);
  const uint32_t ah = (uint32_t)(ua >> 32), al = (uint32_t)ua;
  const uint32_t bh = (uint32_t)(ub >> 32), bl = (uint32_t)ub;
  const uint32_t ea = (ah & 0x7ff00000u) - 0x30000000u, eb = (bh & 0x7ff00000u) - 0x30000000u;
  if (i64_outside(ea | eb)) return i64_hw_mul(a, b);
  const uint32_t ma = (ah & 0xfffffu) | 0x100000u, mb = (bh & 0xfffffu) | 0x100000u;
  // 53 x 53 bits: p3 holds bits 64..105, low word of p2 bits 32..63
  const uint64_t p0 = (uint64_t)al * bl;
  const uint64_t p1 = (uint64_t)ma * bl + (p0 >> 32);
  const uint64_t p2 = (uint64_t)al * mb + p1;
  const uint64_t p3 = (uint64_t)ma * mb + (p2 >> 32);
  const uint32_t h = (uint32_t)(p3 >> 32), m = (uint32_t)p3, l = (uint32_t)p2;
  const uint32_t n = h >> 9;            // 1: the product is in [2, 4)
  const uint32_t s = 12u - n;
  const uint32_t hi = i64_shl(m, h, s), lo = i64_shl(l, m, s);
  // the bits below the result's last, the last of them sticky; round to even
  const uint32_t rem = (l << s) | ((uint32_t)p0 != 0u ? 1u : 0u);
  const uint64_t up = (uint64_t)rem + 0x7fffffffu + (lo & 1u);
  const uint32_t e = ea + eb + (n << 20) + (0x60000000u - (1024u << 20));
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  const uint64_t r = (((uint64_t)(hi + e + sign) << 32) | lo) + (up >> 32);
  return i64_double((uint32_t)(r >> 32), (uint32_t)r);
}

// Quotient.  With the significands A, B in [2^52, 2^53) the quotient to 56
// binary places comes in two digits from a reciprocal X that is 2 to 4 units
// below 2^31 / (B / 2^52), each with its exact remainder:
//   q1 <= A 2^30 / B < q1 + 5.5,  r1 = A 2^30 - q1 B;
//   q2 <= r1 2^26 / B < q2 + 3,   r2 = r1 2^26 - q2 B.
// The last remainder decides the rounding (a quotient of two 53-bit numbers
// is never halfway between two others).
FVM_I64 double div64(double a, double b) {
  const uint64_t ua = i64_bits(a), ub = i64_bits(b);
  const uint32_t ah = (uint32_t)(ua >> 32), al = (uint32_t)ua;
  const uint32_t bh = (uint32_t)(ub >> 32), bl = (uint32_t)ub;
  const uint32_t ea = (ah & 0x7ff00000u) - 0x30000000u, eb = (bh & 0x7ff00000u) - 0x30000000u;
  if (i64_outside(ea | eb)) return i64_hw_div(a, b);
  const uint32_t ma = (ah & 0xfffffu) | 0x100000u, mb = (bh & 0xfffffu) | 0x100000u;
  // X from a float reciprocal of B's first 24 bits and one Newton step with
  // the other 29
  const uint32_t b24 = i64_shl(bl, mb, 3);                         // [2^23, 2^24)
  const float fh = i64_float(0x3f800000u | (b24 & 0x7fffffu));
  const float fl = (float)(int)(bl & 0x1fffffffu) * 0x1p-52f;
  const float r = i64_rcp(fh);
  const float er = fmaf(-fl, r, fmaf(-fh, r, 1.0f));
  const uint32_t X = (uint32_t)(r * 0x1p31f) + (uint32_t)(int)(er * r * 0x1p31f) - 3u;
  // first digit
  const uint32_t a32 = i64_shl(al, ma, 11);                        // A / 2^21
  const uint32_t q1 = i64_mulhi(a32, X);                           // (A/B) 2^30
  const uint64_t A = ((uint64_t)ma << 32) | al, B = ((uint64_t)mb << 32) | bl;
  const uint64_t r1 = (A << 30) - (uint64_t)q1 * B;
  // second digit
  const uint32_t q2 = i64_mulhi((uint32_t)(r1 >> 25), X);          // (r1/B) 2^26
  const uint64_t r2 = (r1 << 26) - (uint64_t)q2 * B;
  const uint64_t q = ((uint64_t)q1 << 26) + q2;                    // A/B to 2^-56, from below
  const uint32_t one = (uint32_t)(q >> 56);                        // A/B >= 1
  const uint32_t g = 3u + one;
  const uint32_t low = (uint32_t)q & ((1u << g) - 1u);
  const int64_t d = (int64_t)((uint64_t)(int64_t)((int)low - (int)(4u << one)) * B + r2);
  const uint64_t m0 = (q >> g) + (d > 0 ? 1u : 0u);
  const uint32_t e = ea - eb + (one << 20) + ((1022u - 1u) << 20);
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  return i64_double((uint32_t)(m0 >> 32) + e + sign, (uint32_t)m0);
}

// Square root.  M, the significand (doubled for odd exponents), in
// [2^52, 2^54); z = M / 2^52.  Two digits as above, from Y, 2 to 4 units below
// 2^31 / sqrt(z):
//   s1 <= sqrt(z) 2^29 < s1 + 6,  r1 = M 2^6 - s1^2;
//   s = s1 2^26 + q2, q2 <= r1 2^26 / (2 sqrt(z) 2^29): s <= sqrt(z) 2^55 < s + 5.
// The exact remainder at the midpoint decides the rounding (a square root of
// a 53-bit number is never a midpoint).
FVM_I64 double sqrt64(double a) {
  const uint64_t ua = i64_bits(a);
  const uint32_t ah = (uint32_t)(ua >> 32), al = (uint32_t)ua;
  const uint32_t ea = ah - 0x30000000u;           // a sign bit is outside too
  if (i64_outside(ea)) return i64_hw_sqrt(a);
  const uint32_t odd = ~(ah >> 20) & 1u;          // the field's bias is odd
  const uint32_t m = (ah & 0xfffffu) | 0x100000u;
  const uint64_t M = (((uint64_t)m << 32) | al) << odd;
  const uint32_t mh = (uint32_t)(M >> 32), ml = (uint32_t)M;
  // Y: float 1/sqrt of the first 24 bits of a's significand, one Newton step
  // with the others
  const float fh = i64_float((0x3f800000u + (odd << 23)) | (i64_shl(al, m, 3) & 0x7fffffu));
  const float fl = (float)(int)(al & 0x1fffffffu) * (odd ? 0x1p-51f : 0x1p-52f);
  const float y = i64_rsqrt(fh);
  const float t = fh * y;
  const float tl = fmaf(fl, y, fmaf(fh, y, -t));
  const float er = fmaf(-tl, y, fmaf(-t, y, 1.0f));
  const uint32_t Y = (uint32_t)(y * 0x1p31f) + (uint32_t)(int)(er * y * 0x1p30f) - 3u;
  const uint32_t z32 = i64_shl(ml, mh, 10);                        // z 2^30
  const uint32_t s1 = i64_mulhi(z32, Y);
  const uint64_t r1 = (M << 6) - (uint64_t)s1 * s1;
  const uint32_t q2 = i64_mulhi((uint32_t)(r1 >> 3), Y);
  const uint64_t s = ((uint64_t)s1 << 26) + q2;
  const uint64_t r2 = (r1 << 52) - (((uint64_t)s1 * q2) << 27) - (uint64_t)q2 * q2;
  const int low = (int)((uint32_t)s & 7u), dm = 4 - low;           // midpoint: s + dm
  const int64_t d = (int64_t)(r2 - (uint64_t)(int64_t)(2 * dm) * s - (uint64_t)(dm * dm));
  const uint64_t m0 = (s >> 3) + (d > 0 ? 1u : 0u);
  // exponent: half of the unbiased one, rounded down; the field without the
  // significand's own leading one
  const uint32_t e = (((ah >> 20) - 1023u - odd) << 19) + (1022u << 20);
  return i64_double((uint32_t)(m0 >> 32) + e, (uint32_t)m0);
}

// 0.5 a: exact, the exponent less one.  p + 0.5 a: one fused operation, whose
// product is exact (a subnormal a apart, where half an ulp of 2^-1074 is lost).
FVM_I64 double half64(double a) {
  const uint64_t u = i64_bits(a);
  const uint32_t h = (uint32_t)(u >> 32);
  if (i64_outside((h & 0x7ff00000u) - 0x30000000u)) return i64_hw_mul(0.5, a);
  return i64_double(h - 0x00100000u, (uint32_t)u);
}

// a < 0, a > 0 (false for NaN and zeros)
FVM_I64 bool neg64(double a) {
  const uint64_t u = i64_bits(a);
  return u > 0x8000000000000000ull && u <= 0xfff0000000000000ull;
}
FVM_I64 bool pos64(double a) {
  const uint64_t u = i64_bits(a);
  return u - 1u < 0x7ff0000000000000ull;
}

// The operations inlined (C = 0) or as functions (C = 1).  Inlined they are the
// quicker way for a warp alone; but long kernels of them wait for their own
// instructions once many warps stream through the code (16 bytes per
// instruction), and functions stay in the nearest instruction cache.  C = 2:
// products on the FP64 pipe, for work so little that the pipe is never full.
FVM_I64_CALL double i64_mul_call(double a, double b) { return mul64(a, b); }
FVM_I64_CALL double i64_div_call(double a, double b) { return div64(a, b); }
FVM_I64_CALL double i64_sqrt_call(double a) { return sqrt64(a); }
// FVM_FP64_CONTRACT (the library with contracted FP64 kernels): products on the
// FP64 pipe in every form, where the compiler can join them with sums.
template <int C>
FVM_I64 double mul_as(double a, double b) {
#ifdef FVM_FP64_CONTRACT
  return a * b;
#else
  return C == 2 ? a * b : C ? i64_mul_call(a, b) : mul64(a, b);
#endif
}
template <int C>
FVM_I64 double div_as(double a, double b) { return C ? i64_div_call(a, b) : div64(a, b); }
template <int C>
FVM_I64 double sqrt_as(double a) { return C ? i64_sqrt_call(a) : sqrt64(a); }

// A double whose products, quotients and square roots are the ones above and
// whose sums are the FP64 pipe's; the arithmetic of fvm_device.cuh compiles
// for it as for double.  The / operator always calls (the HLLC flux, which
// divides 25 times, 639 -> 597 us on 768 x 256), mdiv follows C.
template <int C>
struct F64T {
  double v;
  F64T() = default;
  FVM_I64 F64T(double x) : v(x) {}
  FVM_I64 explicit operator double() const { return v; }
  FVM_I64 friend F64T operator+(F64T a, F64T b) { return F64T(a.v + b.v); }
  FVM_I64 friend F64T operator-(F64T a, F64T b) { return F64T(a.v - b.v); }
  FVM_I64 friend F64T operator-(F64T a) { return F64T(-a.v); }
  FVM_I64 friend F64T operator*(F64T a, F64T b) { return F64T(mul_as<C>(a.v, b.v)); }
  FVM_I64 friend F64T operator/(F64T a, F64T b) { return F64T(i64_div_call(a.v, b.v)); }
  FVM_I64 friend bool operator<(F64T a, F64T b) { return a.v < b.v; }
  FVM_I64 friend bool operator>(F64T a, F64T b) { return a.v > b.v; }
  FVM_I64 friend bool operator<=(F64T a, F64T b) { return a.v <= b.v; }
  FVM_I64 friend bool operator>=(F64T a, F64T b) { return a.v >= b.v; }
  FVM_I64 friend bool operator!=(F64T a, F64T b) { return a.v != b.v; }
};
using F64 = F64T<0>;

}  // namespace fvm
