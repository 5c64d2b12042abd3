// Correctly rounded FP64 square root and division in integer arithmetic.
//
// GB300's FP64 unit does one warp instruction per quarter-SM every 64 cycles,
// and CUDA's own sqrt and division are about nine such instructions each: 24
// divisions and 12 square roots were more than half of a ring's 509.  The
// integer units issue a warp instruction every cycle or two and are idle
// beside it, so the functions here take an approximation from the FP32
// reciprocal square root, improve it by one Newton step in fixed point, and
// decide the rounding from the exact remainder.  The results are the correctly
// rounded ones (IEEE round-to-nearest-even), so they are the bits of sqrt() and
// of the division operator.
//
// With the significand of x scaled to X in [2^62, 2^64) so that its exponent is
// even, r = sqrt(X / 2^62) lies in [1, 2):
//   Y ~ 2^31 / r       from rsqrtf, then Y += Y (1 - r^2 Y^2) / 2 (error < 2^-28)
//   S ~ 2^31 r         = X Y, and D = X - S^2 exactly
//   R ~ 2^63 r         = 2^32 S + 2^32 D / (2 S)            (error < 2^10 of 2^63)
//   N = R / 2^11 rounded, off from the correctly rounded root by at most one,
// and with the exact remainder e = 2^42 X - N^2 the root rounds to N iff
// -N < e <= N (the root of a 53-bit number is never halfway between two).
// For a division by that N, or by the 53-bit significand N of any divisor,
//   Z ~ 2^115 / N      from Y by one Newton step            (error < 2^-56)
//   q = A Z            rounded to 53 bits, off by at most one,
// and A 2^s - q N decides (a quotient is never halfway either: 2 A 2^s = q N
// with an odd q would need 2^53 to divide N < 2^53).  The remainders fit 64 bits, so
// they are computed modulo 2^64.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#include "vlm_math.h"

namespace vlm {
namespace exact64 {

VLM_HD uint32_t mulhi32(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
VLM_HD int32_t mulhi32s(int32_t a, int32_t b) {
#if defined(__CUDA_ARCH__)
  return __mulhi(a, b);
#else
  return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
VLM_HD uint64_t bits(double x) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
VLM_HD double from_bits(uint64_t u) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
VLM_HD uint32_t high(double x) { return (uint32_t)(bits(x) >> 32); }
// 1/sqrt(v) in FP32, v in [1, 4)
VLM_HD float rsqrt32(float v) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
#else
#if defined(VLM_RSQRT32_FACTOR)
  return (1.0f / sqrtf(v)) * (VLM_RSQRT32_FACTOR);  // a test stands in for the unit's approximation error
#else
  return 1.0f / sqrtf(v);
#endif
#endif
}
VLM_HD float float_bits(uint32_t u) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}
VLM_HD uint32_t bits_float(float f) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(f);
#else
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
#endif
}

// The significand N (bit 52 set) and the exponent of a number, and Y ~ 2^83 / N.
struct Root {
  uint64_t N;
  int32_t exp;  // the number is N 2^(exp - 52)
  uint32_t Y;
};

// Square roots are taken of numbers in [2^-400, 2^400) and give numbers in
// [2^-200, 2^200): in_range.  Dividends are zero or in [2^-800, 2^700):
// div_in_range.  Every exponent below then stays normal.
constexpr uint32_t kSqrtLo = (1023u - 400u) << 20, kSqrtHi = (1023u + 400u) << 20;
VLM_HD bool in_range(double x) { return high(x) - kSqrtLo < kSqrtHi - kSqrtLo; }
constexpr uint32_t kDivLo = (1023u - 800u) << 20, kDivHi = (1023u + 700u) << 20;
// whether a is +-0, told from its two words (a comparison of the whole would
// become one on the FP64 unit)
VLM_HD bool is_zero(double a) {
  const uint64_t u = bits(a);
  return (((uint32_t)(u >> 32) << 1) | (uint32_t)u) == 0u;
}
VLM_HD bool div_in_range(double a) { return (high(a) & 0x7fffffffu) - kDivLo < kDivHi - kDivLo || is_zero(a); }

// sqrt(x), in_range(x)
VLM_HD Root root_of(double x) {
  const uint64_t u = bits(x);
  const uint32_t hx = (uint32_t)(u >> 32);
  const int32_t E = (int32_t)(hx >> 20) - 1023;
  const uint32_t odd = (uint32_t)E & 1u;
  const uint64_t m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint64_t X = m << (10 + odd);
  const uint32_t Xh = (uint32_t)(X >> 32);
  // v = X / 2^62 in FP32 (its significand cut to 23 bits), 1/sqrt(v) in (1/2, 1]
  const float v = float_bits(((127u + odd) << 23) | (uint32_t)((u >> 29) & 0x7fffffu));
  uint32_t rb = bits_float(rsqrt32(v));
  rb = rb < 0x3f000000u ? 0x3f000000u : rb;  // 1/2, in case the approximation falls short of it
  uint32_t Y = rb >= 0x3f800000u ? 0x80000000u : ((rb & 0x7fffffu) | 0x800000u) << 7;  // 2^31 / r
  // 1 - r^2 Y^2, scaled by 2^28
  const int32_t e = (1 << 28) - (int32_t)mulhi32(mulhi32(Y, Y), Xh);
  Y += (uint32_t)(mulhi32s((int32_t)((uint32_t)e << 14), (int32_t)(Y >> 1)) >> 10);
  const uint64_t S = ((uint64_t)Xh * Y) >> 30;  // 2^32 at most, for r next to 2
  const uint32_t S0 = S >> 32 ? 0xffffffffu : (uint32_t)S;
  const int64_t D = (int64_t)(X - (uint64_t)S0 * S0);
  const int64_t d = (int64_t)(int32_t)(D >> 7) * (int64_t)(int32_t)(Y >> 1);  // D Y / 2^8
  const uint64_t R = ((uint64_t)S0 << 32) + (uint64_t)(d >> 23);
  uint64_t N = (R + 1024) >> 11;
  const int64_t rem = (int64_t)((X << 42) - N * N);
  if (rem > (int64_t)N) ++N;
  if (rem <= -(int64_t)N) --N;
  Root r;
  r.N = N;
  r.exp = E >> 1;
  r.Y = Y;
  return r;
}
VLM_HD double value(const Root& r) { return from_bits(((uint64_t)(uint32_t)(r.exp + 1022) << 52) + r.N); }

// Z ~ 2^115 / N
VLM_HD uint64_t reciprocal(const Root& r) {
  const int64_t Er = (int64_t)(0 - r.N * (uint64_t)r.Y);  // 2^83 - N Y
  const int64_t c = (int64_t)(int32_t)(Er >> 26) * (int64_t)(int32_t)(r.Y >> 1);
  return ((uint64_t)r.Y << 32) + (uint64_t)(c >> 24);
}

// a / n, n the number of r and Z its reciprocal, div_in_range(a)
VLM_HD double divide(double a, const Root& r, uint64_t Z) {
  const uint64_t u = bits(a);
  const uint64_t A = (u & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint32_t up = A >= r.N ? 0u : 1u;  // the quotient's exponent is one lower
  // (A 2^11 Z) / 2^64 ~ 2^62 A / N, its lowest partial product left out (error < 4)
  const uint64_t As = A << 11;
  const uint32_t ah = (uint32_t)(As >> 32), al = (uint32_t)As, zh = (uint32_t)(Z >> 32), zl = (uint32_t)Z;
  const uint64_t Q = (uint64_t)ah * zh + mulhi32(ah, zl) + mulhi32(al, zh);
  uint64_t q = (((Q << up) >> 9) + 1) >> 1;
  const int64_t rem2 = (int64_t)(((A << 52) << (1 + up)) - 2 * (q * r.N));
  if (rem2 > (int64_t)r.N) ++q;
  if (rem2 < -(int64_t)r.N) --q;
  const uint32_t e = ((uint32_t)(u >> 52) & 0x7ffu) - (uint32_t)r.exp - up - 1u;
  const uint64_t w = (((uint64_t)e << 52) + q) | (u & 0x8000000000000000ull);
  return is_zero(a) ? a : from_bits(w);
}

// 1/r in FP32, r in [1, 2)
VLM_HD float rcp32(float r) {
#if defined(__CUDA_ARCH__)
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(r));
  return y;
#elif defined(VLM_RSQRT32_FACTOR)
  return (1.0f / r) * (VLM_RSQRT32_FACTOR);
#else
  return 1.0f / r;
#endif
}
// Any divisor d with |d| in [2^-200, 2^200) (divisor_in_range): as root_of, with
// one Newton step Y += Y (1 - r Y) in 32 bits (error < 2^-28).
VLM_HD bool divisor_in_range(double d) {
  const uint32_t lo = (1023u - 200u) << 20, hi = (1023u + 200u) << 20;
  return (high(d) & 0x7fffffffu) - lo < hi - lo;
}
VLM_HD Root divisor_of(double d) {
  const uint64_t u = bits(d);
  Root r;
  r.N = (u & 0xfffffffffffffull) | 0x10000000000000ull;
  r.exp = (int32_t)((u >> 52) & 0x7ffu) - 1023;
  uint32_t rb = bits_float(rcp32(float_bits(0x3f800000u | (uint32_t)((u >> 29) & 0x7fffffu))));
  rb = rb < 0x3f000000u ? 0x3f000000u : rb;
  uint32_t Y = rb >= 0x3f800000u ? 0x80000000u : ((rb & 0x7fffffu) | 0x800000u) << 7;
  const int32_t e = (1 << 30) - (int32_t)mulhi32(Y, (uint32_t)(r.N >> 21));
  Y += (uint32_t)(mulhi32s((int32_t)((uint32_t)e << 16), (int32_t)(Y >> 1)) >> 13);
  r.Y = Y;
  return r;
}
VLM_HD double with_sign(double a, double d) { return from_bits(bits(a) ^ (bits(d) & 0x8000000000000000ull)); }
// a / d
VLM_HD double quotient(double a, double d) {
  if (!divisor_in_range(d) || !div_in_range(a)) return a / d;
  const Root r = divisor_of(d);
  return with_sign(divide(a, r, reciprocal(r)), d);
}
VLM_HD d3 quotient(d3 a, double d) {
  if (!divisor_in_range(d) || !div_in_range(a.x) || !div_in_range(a.y) || !div_in_range(a.z)) return a / d;
  const Root r = divisor_of(d);
  const uint64_t Z = reciprocal(r);
  return mk3(with_sign(divide(a.x, r, Z), d), with_sign(divide(a.y, r, Z), d), with_sign(divide(a.z, r, Z), d));
}
VLM_HD double root(double x) { return in_range(x) ? value(root_of(x)) : sqrt(x); }
// vlm_math.h's norm3, unit3, proj3, noproj3
VLM_HD double norm(d3 a) { return root(sumsq3(a)); }
VLM_HD d3 unit(d3 a) {
  const double n = norm(a);
  return n > kEps ? quotient(a, n) : zero3();
}
VLM_HD d3 proj(d3 a, d3 d) {
  const double ns = sumsq3(d);
  return ns > kEps ? quotient(dot3(a, d) * d, ns) : zero3();
}
VLM_HD d3 noproj(d3 a, d3 d) {
  const double ns = sumsq3(d);
  return ns > kEps ? a - quotient(dot3(a, d) * d, ns) : a;
}

// ---- the Biot-Savart functions of vlm_math.h with these roots and divisions ----
// The same operations in the same order, so the same bits; numbers outside the
// ranges above (a target on a corner, coordinates beyond 1e60) take
// vlm_math.h's own functions.
//
// Every sum and product is a fused multiply-add of three registers, a 1 + b and
// a b - 0, which round the same: the FP64 unit takes those in 64 cycles a warp
// and quarter-SM, but an add, a multiply, or a fused multiply-add with a
// constant operand in 76 (measured).  Unit holds the 1 and the -0 in registers
// the compiler cannot see into; device code fills it with load_unit().
struct Unit {
  double one, nz;
};
#if defined(__CUDACC__)
static __device__ double g_unit64[2] = {1.0, -0.0};
__device__ __forceinline__ Unit load_unit() {
  const volatile double* p = g_unit64;
  Unit k;
  k.one = p[0];
  k.nz = p[1];
  return k;
}
#endif
VLM_HD double add(const Unit& k, double a, double b) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, k.one, b);
#else
  (void)k;
  return a + b;
#endif
}
VLM_HD double mul(const Unit& k, double a, double b) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, k.nz);
#else
  (void)k;
  return a * b;
#endif
}
VLM_HD double sub(const Unit& k, double a, double b) { return add(k, a, -b); }
VLM_HD d3 add(const Unit& k, d3 a, d3 b) { return mk3(add(k, a.x, b.x), add(k, a.y, b.y), add(k, a.z, b.z)); }
VLM_HD d3 sub(const Unit& k, d3 a, d3 b) { return mk3(sub(k, a.x, b.x), sub(k, a.y, b.y), sub(k, a.z, b.z)); }
VLM_HD d3 mul(const Unit& k, d3 a, double s) { return mk3(mul(k, a.x, s), mul(k, a.y, s), mul(k, a.z, s)); }
VLM_HD double dot(const Unit& k, d3 a, d3 b) {
  return add(k, add(k, mul(k, a.x, b.x), mul(k, a.y, b.y)), mul(k, a.z, b.z));
}
VLM_HD d3 cross(const Unit& k, d3 a, d3 b) {
  return mk3(sub(k, mul(k, a.y, b.z), mul(k, a.z, b.y)), sub(k, mul(k, a.z, b.x), mul(k, a.x, b.z)),
             sub(k, mul(k, a.x, b.y), mul(k, a.y, b.x)));
}
// x > kEps^2 for x >= 0 or NaN (false), compared as integers
VLM_HD bool above_eps2(double x) {
  const uint64_t lo = 0x3970000000000000ull;  // 2^-104
  return bits(x) - (lo + 1) <= 0x7ff0000000000000ull - (lo + 1);
}

VLM_HD corner64 make_corner(const Unit& k, d3 P, d3 c) {
  corner64 o;
  o.r = sub(k, P, c);
  const double x = dot(k, o.r, o.r);
  if (in_range(x) && div_in_range(o.r.x) && div_in_range(o.r.y) && div_in_range(o.r.z)) {
    const Root n = root_of(x);
    // |r| > kEps = 2^-52
    if (n.exp > -52 || (n.exp == -52 && n.N > 0x10000000000000ull)) {
      const uint64_t Z = reciprocal(n);
      o.u = mk3(divide(o.r.x, n, Z), divide(o.r.y, n, Z), divide(o.r.z, n, Z));
    } else {
      o.u = zero3();
    }
  } else {
    o.u = unit3(o.r);
  }
  return o;
}
VLM_HD d3 vf_vind(const Unit& k, const corner64& a, const corner64& b, double rvc) {
  const d3 r0 = sub(k, a.r, b.r);
  const d3 c = cross(k, a.r, b.r);
  const double c2 = dot(k, c, c);
  if (!above_eps2(c2)) return zero3();
  const double d = dot(k, r0, sub(k, a.u, b.u));
  const double s = mul(k, rvc, root(dot(k, r0, r0)));
  const double s2 = mul(k, s, s);
  const double den2 = add(k, mul(k, s2, s2), mul(k, c2, c2));
  const d3 v = mul(k, mul(k, c, kInv4Pi), d);
  if (in_range(den2) && div_in_range(v.x) && div_in_range(v.y) && div_in_range(v.z)) {
    const Root n = root_of(den2);
    const uint64_t Z = reciprocal(n);
    return mk3(divide(v.x, n, Z), divide(v.y, n, Z), divide(v.z, n, Z));
  }
  return v / sqrt(den2);
}
VLM_HD d3 vr_vind(const Unit& k, d3 P, const d3* c, const double* rvc) {
  const corner64 k0 = make_corner(k, P, c[0]), k1 = make_corner(k, P, c[1]);
  d3 v = vf_vind(k, k0, k1, rvc[0]);
  const corner64 k2 = make_corner(k, P, c[2]);
  v = add(k, v, vf_vind(k, k1, k2, rvc[1]));
  const corner64 k3 = make_corner(k, P, c[3]);
  v = add(k, v, vf_vind(k, k2, k3, rvc[2]));
  v = add(k, v, vf_vind(k, k3, k0, rvc[3]));
  return v;
}
VLM_HD d3 fil_vind(const Unit& k, d3 P, d3 a, d3 b, double rvc) {
  return vf_vind(k, make_corner(k, P, a), make_corner(k, P, b), rvc);
}

}  // namespace exact64
}  // namespace vlm
