// Binary64 division, square root and their reciprocals on the integer pipe.
//
// GB300's FP64 unit takes 64-76 cycles per warp instruction whatever the
// number of active lanes (two results per clock and SM), its integer pipes 2.
// An IEEE binary64 division takes 560 cycles there, a square root 597
// (measured, one warp or a full SM alike).  The functions below do the same on
// 64-bit fixed-point significands with 32-bit multiplies, about 40 integer
// instructions for a reciprocal or a reciprocal square root and 65 for a
// division or a square root:
//   seed       the binary32 hardware estimate of 1/d or 1/sqrt(m) (2^-22.5);
//   refinement one step of the binomial series to second order (an extension
//              of Newton's iteration): r (1 + e + e^2), e = 1 - d r, or
//              y (1 + e/2 + 3 e^2 / 8), e = 1 - m y^2, with e kept to 2^-63:
//              the neglected e^3 is below 2^-65;
//   rounding   ddiv and dsqrt: the quotient's or root's first 54 bits from
//              the refined value, made exact by the sign of the exact
//              remainder (computed modulo 2^64), then rounded to nearest; a
//              quotient or root of binary64 numbers is never half-way, so the
//              result is the correctly rounded one, bit for bit.
//              rcp_int and rsqrt_int: the refined 62 bits rounded once (error
//              below 0.51 ulp).
// Operands outside the normal range, or results near the exponent limits,
// take the FP64 instructions.  Fixed-point numbers: d in [1, 2) as D = d 2^63.
//
// The header compiles for the host as well (tests check it there against the
// host's IEEE operations): a host build defines the two seed functions first.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define M2CG_INT __device__ __forceinline__
#define M2CG_INT_SLOW static __device__ __noinline__
namespace m2cg {
M2CG_INT uint32_t if_mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
M2CG_INT uint32_t if_hi(double x) { return (uint32_t)__double2hiint(x); }
M2CG_INT uint32_t if_lo(double x) { return (uint32_t)__double2loint(x); }
M2CG_INT double if_dbl(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }
M2CG_INT int if_clz(uint32_t x) { return __clz((int)x); }
// bits of the binary32 estimate of 1/f and 1/sqrt(f), f given by its bits
M2CG_INT uint32_t if_seed_rcp(uint32_t f) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
  return __float_as_uint(r);
}
M2CG_INT uint32_t if_seed_rsqrt(uint32_t f) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
  return __float_as_uint(r);
}
M2CG_INT double if_mul(double a, double b) { return __dmul_rn(a, b); }
}  // namespace m2cg
#endif

namespace m2cg {

// hi 64 bits of a * b without the low-by-low product: in (a b / 2^64 - 2, a b / 2^64]
M2CG_INT uint64_t if_mulhi64(uint64_t a, uint64_t b) {
  const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
  const uint64_t t = (uint64_t)ah * bl;
  const uint64_t w = (uint64_t)al * bh + (uint32_t)t;
  return (uint64_t)ah * bh + (t >> 32) + (w >> 32);
}
M2CG_INT uint64_t if_sqrhi64(uint64_t a) {
  const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32);
  const uint64_t t = (uint64_t)ah * al;
  return (uint64_t)ah * ah + (t >> 31);
}
// significand of a normal double as 1.f 2^63
M2CG_INT uint64_t if_sig(uint32_t hi, uint32_t lo) {
  const uint32_t h = (hi << 11) | (lo >> 21) | 0x80000000u;
  return ((uint64_t)h << 32) | (lo << 11);
}

// 2^126 / D for D = d 2^63, d in [1, 2): at most the true value, at least it - 5.
M2CG_INT uint64_t if_recip(uint64_t D) {
  const uint32_t Dh = (uint32_t)(D >> 32), Dl = (uint32_t)D;
  // the seed's argument lies just above d, so that the seed stays below 1
  uint32_t rb = if_seed_rcp((Dh >> 8) + 0x3f000001u);
  rb = rb > 0x3f000000u ? rb : 0x3f000000u;
  const uint32_t r24 = (rb & 0x7fffffu) | 0x800000u;      // r 2^24, r in [0.5, 1)
  const uint32_t R0 = r24 << 8;
  const uint64_t P = (uint64_t)Dh * R0 + if_mulhi(Dl, R0);   // d r 2^63, cut
  int64_t es = (int64_t)(0x7ffffffffffffffdull - P) << 20;   // e 2^83, |e| < 2^-21; 3 units low on purpose
  const int32_t eh = (int32_t)(es >> 32);
  es += ((int64_t)eh * eh) >> 19;
  const int64_t c = (int64_t)(int32_t)r24 * (int32_t)(es >> 32) + if_mulhi(r24, (uint32_t)es);
  return ((uint64_t)r24 << 39) + (uint64_t)(c >> 12);
}

// 2^63 / sqrt(m) for M = m 2^62, m in [1, 4): at most the true value, at least
// it - 10.
M2CG_INT uint64_t if_rsqrt(uint64_t M) {
  // binary32 argument just above m, exponent 127 or 128
  const uint32_t Mh = (uint32_t)(M >> 32);
  const uint32_t two = Mh >> 31;                             // m >= 2
  const uint32_t f = (Mh >> (7 + two)) + (two ? 0x3f800001u : 0x3f000001u);
  uint32_t rb = if_seed_rsqrt(f);
  rb = rb > 0x3f000000u ? rb : 0x3f000000u;
  rb = rb < 0x3f7fffffu ? rb : 0x3f7fffffu;
  const uint32_t r24 = (rb & 0x7fffffu) | 0x800000u;
  const uint64_t S = ((uint64_t)r24 * r24) << 16;            // y^2 2^64
  const uint64_t P = if_mulhi64(M, S);                       // m y^2 2^62, cut
  int64_t es = (int64_t)(0x3ffffffffffffffaull - P) << 20;   // (e / 2) 2^83
  const int32_t eh = (int32_t)(es >> 32);                    // e 2^50
  es += ((int64_t)eh * (eh * 3)) >> 20;                      // + 3 e^2 / 8
  const int64_t c = (int64_t)(int32_t)r24 * (int32_t)(es >> 32) + if_mulhi(r24, (uint32_t)es);
  return ((uint64_t)r24 << 39) + (uint64_t)(c >> 12);
}

// value (hi part of the exponent and sign) + rounded 53-bit significand
M2CG_INT double if_pack(uint32_t base_hi, uint64_t m) {
  return if_dbl(base_hi + (uint32_t)(m >> 32), (uint32_t)m);
}

// ---- approximate (0.51 ulp) reciprocal and reciprocal square root ----------
// in range: |x| normal and below 2^1022 (rcp), x > 0 normal (rsqrt)
M2CG_INT bool if_rcp_range(uint32_t hi) { return ((hi & 0x7fffffffu) - 0x00100000u) < 0x7fc00000u; }
M2CG_INT bool if_rsqrt_range(uint32_t hi) { return (hi - 0x00100000u) < 0x7fe00000u; }
M2CG_INT double if_rcp_core(uint32_t hi, uint32_t lo) {
  const uint64_t R = if_recip(if_sig(hi, lo));
  // exponent field 2045 - E, less one for the significand's leading bit
  const uint32_t base = (hi & 0x80000000u) + (0x7fc00000u - (hi & 0x7ff00000u));
  return if_pack(base, (R + 512u) >> 10);
}
M2CG_INT double if_rsqrt_core(uint32_t hi, uint32_t lo) {
  const uint64_t D = if_sig(hi, lo);
  const uint32_t E = hi >> 20;
  const uint64_t Y = if_rsqrt(D >> (E & 1u));                // E - 1023 even: m = 1.f
  const uint32_t base = (1021u - (uint32_t)(((int32_t)E - 1023) >> 1)) << 20;
  return if_pack(base, (Y + 512u) >> 10);
}

// ---- correctly rounded division --------------------------------------------
// Quotient of two significands (D's reciprocal R from if_recip): the 53-bit
// rounded significand, and s = 1 when a < d (the exponent is one lower).
M2CG_INT uint64_t if_quot(uint64_t A, uint32_t a_lo, uint64_t D, uint64_t R, uint32_t& s) {
  const uint64_t T = if_mulhi64(A, R);                       // (a / d) 2^62, up to 8 units low
  s = ((uint32_t)(T >> 62) ^ 1u) & 1u;
  const uint64_t Q = T >> (9u - s);                          // 54 bits, exact floor or one less
  const uint64_t D53 = D >> 11;
  // remainder a 2^(53+s) - Q d modulo 2^64 (a_lo: the low word of the 53-bit a)
  const uint64_t rem = ((uint64_t)(a_lo << (21u + s)) << 32) - Q * D53;
  return (Q + 1u + (rem >= D53 ? 1u : 0u)) >> 1;
}
M2CG_INT bool if_normal(uint32_t hi) { return ((hi & 0x7fffffffu) - 0x00100000u) < 0x7fe00000u; }

M2CG_INT_SLOW double if_div_slow(double a, double b) { return a / b; }
// whether a / b is in range: both normal, the quotient's exponent field in [2, 2045]
M2CG_INT bool if_div_range(double a, double b) {
  const uint32_t ah = if_hi(a), bh = if_hi(b);
  const uint32_t eq = ((ah >> 20) & 0x7ffu) - ((bh >> 20) & 0x7ffu) + 1023u;
  return if_normal(ah) && if_normal(bh) && eq - 2u <= 2043u;
}
// a / b in range, from D = if_sig(b) and R = if_recip(D)
M2CG_INT double if_div_core(double a, double b, uint64_t D, uint64_t R) {
  const uint32_t ah = if_hi(a), al = if_lo(a), bh = if_hi(b);
  uint32_t s;
  const uint64_t m = if_quot(if_sig(ah, al), al, D, R, s);
  return if_pack(((ah ^ bh) & 0x80000000u) + ((((ah >> 20) & 0x7ffu) - ((bh >> 20) & 0x7ffu) + 1022u - s) << 20), m);
}
// ddiv is a call (one copy of its code per kernel unit: the solver's straight-
// line code has dozens of divisions); ddiv2 forms two independent quotients
// in line, their integer chains interleaved.
M2CG_INT_SLOW double ddiv(double a, double b) {
  if (!if_div_range(a, b)) return a / b;
  const uint64_t D = if_sig(if_hi(b), if_lo(b));
  return if_div_core(a, b, D, if_recip(D));
}
// The same for a chain that waits for each result (one problem per warp): the
// estimate is rounded at once, and the exact remainder is formed only where the
// estimate's error bound reaches the rounding boundary (8 of 512 or 1024
// values); 250 cycles of latency against 385.  D and R as in if_div_core, so
// that a divisor's reciprocal can be started before the dividend is known.
M2CG_INT_SLOW double if_div_edge(double a, double b, uint64_t D, uint64_t R) {
  return if_div_range(a, b) ? if_div_core(a, b, D, R) : a / b;
}
M2CG_INT double if_div_lat(double a, double b, uint64_t D, uint64_t R) {
  const uint32_t ah = if_hi(a), bh = if_hi(b);
  const uint64_t T = if_mulhi64(if_sig(ah, if_lo(a)), R);     // in (a / d 2^62 - 8, a / d 2^62]
  const bool one = (uint32_t)(T >> 32) >= 0x40000000u;        // a / d >= 1
  const uint64_t X0 = T + 512u, X1 = T + 256u;
  const uint64_t m = one ? X0 >> 10 : X1 >> 9;
  const bool edge = one ? (((uint32_t)X0 + 8u) & 1023u) < 8u : (((uint32_t)X1 + 8u) & 511u) < 8u;
  const uint32_t ex = ((ah >> 20) & 0x7ffu) - ((bh >> 20) & 0x7ffu);
  double r = if_pack(((ah ^ bh) & 0x80000000u) + ((ex + (one ? 1022u : 1021u)) << 20), m);
  if (edge || !if_div_range(a, b)) r = if_div_edge(a, b, D, R);
  return r;
}
M2CG_INT double if_div_lat(double a, double b) {
  const uint64_t D = if_sig(if_hi(b), if_lo(b));
  return if_div_lat(a, b, D, if_recip(D));
}
M2CG_INT_SLOW double ddiv_lat(double a, double b) { return if_div_lat(a, b); }
M2CG_INT void ddiv2(double a, double b, double c, double d, double& q, double& r) {
  const bool ok = if_div_range(a, b) && if_div_range(c, d);
  const uint64_t D = if_sig(if_hi(b), if_lo(b)), E = if_sig(if_hi(d), if_lo(d));
  q = if_div_core(a, b, D, if_recip(D));
  r = if_div_core(c, d, E, if_recip(E));
  if (!ok) { q = if_div_slow(a, b); r = if_div_slow(c, d); }
}

// ---- correctly rounded square root -------------------------------------------
#ifdef __CUDACC__
M2CG_INT_SLOW double if_sqrt_slow(double x) { return sqrt(x); }
#endif
M2CG_INT_SLOW double dsqrt(double x) {
  const uint32_t hi = if_hi(x), lo = if_lo(x);
  if (!if_rsqrt_range(hi)) return if_sqrt_slow(x);
  const uint32_t E = hi >> 20, even = E & 1u;                // E odd: E - 1023 even
  const uint64_t M = if_sig(hi, lo) >> even;
  const uint64_t T = if_mulhi64(M, if_rsqrt(M));             // sqrt(m) 2^61, up to 10 units low
  const uint64_t Q = T >> 8;                                 // 54 bits, exact floor or one less
  const uint64_t rem = ((uint64_t)(lo << (23u - even)) << 32) - Q * Q;   // m 2^106 - Q^2 modulo 2^64
  const uint64_t m = (Q + 1u + (rem > 2u * Q ? 1u : 0u)) >> 1;
  return if_pack((1022u + (uint32_t)(((int32_t)E - 1023) >> 1)) << 20, m);
}

M2CG_INT double if_sqrt_lat(double x) {   // as if_div_lat
  const uint32_t hi = if_hi(x), lo = if_lo(x), E = hi >> 20;
  const uint64_t M = if_sig(hi, lo) >> (E & 1u);
  const uint64_t X = if_mulhi64(M, if_rsqrt(M)) + 256u;       // T in (sqrt(m) 2^61 - 13, sqrt(m) 2^61]
  double r = if_pack((1022u + (uint32_t)(((int32_t)E - 1023) >> 1)) << 20, X >> 9);
  if ((((uint32_t)X + 13u) & 511u) < 13u || !if_rsqrt_range(hi)) r = dsqrt(x);
  return r;
}

// ---- van Albada's limited slope ------------------------------------------------
// (b a^2 + a b^2) / (a^2 + b^2) for two differences of the same sign, with a
// the smaller: a h, h = b (a + b) / (a^2 + b^2) in [1, 1.21], h in fixed point
// from the significands (a's shifted to b's exponent: h depends on a / b to
// 2^-60) and one binary64 multiplication; 0 for opposite signs and for a
// product below 1e-16.  Returns 1 with the slope, or 0 where the product rounds
// at 1e-16 or an operand is special (the caller's FP64 form decides).
M2CG_INT int if_van_albada(double x, double y, double& out) {
  const uint32_t xh = if_hi(x), yh = if_hi(y);
  const uint32_t ux = xh & 0x7fffffffu, uy = yh & 0x7fffffffu;
  const bool xs = ux < uy || (ux == uy && if_lo(x) < if_lo(y));   // |x| < |y|
  const uint32_t ah = xs ? xh : yh, al = xs ? if_lo(x) : if_lo(y);
  const uint32_t bh = xs ? yh : xh, bl = xs ? if_lo(y) : if_lo(x);
  const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
  out = 0.0;
  if (eb > 2000u) return 0;
  // the product lies in [2^(ea + eb - 2046), 4 x that); 1e-16 = 2^-53.15
  if (ea + eb <= 1990u) return 1;
  if ((int32_t)(ah ^ bh) < 0) return 1;
  if (ea + eb < 1993u) {
    // next to the threshold: the product to 2^-62 against 1e-16, undecided only
    // within the rounding of the product
    const uint64_t t = if_mulhi64(if_sig(ah, al), if_sig(bh, bl)), c = 16615349947311448064ull >> (ea + eb - 1991u);
    if (t + 2048u < c) return 1;
    if (t < c + 2048u) return 0;
  }
  if (ea == 0u) return 0;
  const uint32_t sh = eb - ea;
  const uint64_t B = if_sig(bh, bl), A = if_sig(ah, al) >> (sh < 63u ? sh : 63u);
  const uint64_t b2 = if_sqrhi64(B) >> 2;                    // b^2 2^60
  const uint64_t den = b2 + (if_sqrhi64(A) >> 2);
  const uint64_t num = b2 + (if_mulhi64(A, B) >> 2);
  const int z = if_clz((uint32_t)(den >> 32));               // 0 < z < 4
  const uint64_t h = if_mulhi64(num << (z - 1), if_recip(den << z));   // h 2^61
  out = if_mul(if_dbl(ah, al), if_pack(1022u << 20, (h + 256u) >> 9));
  return 1;
}

// ---- ordering and one-sided differences ----------------------------------------
// order-preserving integer of a double that is not NaN (-0 just below +0)
M2CG_INT int64_t if_key(double x) {
  const uint32_t m = (uint32_t)((int32_t)if_hi(x) >> 31);
  return (int64_t)(((uint64_t)(if_hi(x) ^ (m & 0x7fffffffu)) << 32) | (if_lo(x) ^ m));
}
// bit 31 set for an infinity or a NaN (several operands: or them, one test)
M2CG_INT uint32_t if_special_bit(double x) { return (if_hi(x) & 0x7fffffffu) + 0x00100000u; }
// x, negated where sb (0 or the sign bit) is set
M2CG_INT double if_flip(double x, uint32_t sb) { return if_dbl(if_hi(x) ^ sb, if_lo(x)); }

// Godunov's one-sided difference along one axis: max(p - m, p - n, 0), for
// phi < 0 (sb set) max(m - p, n - p, 0), the maximum taken over the bit patterns
// as signed integers (a NaN with a clear sign bit wins, one with a set sign bit
// counts as negative).  Rounding is monotone, so for finite operands the larger
// difference is that of the smaller (larger) neighbour, chosen on the integer
// pipe: one subtraction instead of two, the same bits (if_one_sided; the caller
// has seen to the operands with if_special_bit).  if_one_sided_any forms both.
M2CG_INT double if_one_sided(double p, double m, double n, uint32_t sb) {
  const double x = if_flip(m, sb), y = if_flip(n, sb);
  const double d = if_flip(p, sb) - (if_key(x) <= if_key(y) ? x : y);
  return (int32_t)if_hi(d) < 0 ? 0.0 : d;
}
M2CG_INT double if_one_sided_any(double p, double m, double n, uint32_t sb) {
  const double a = if_flip(p - m, sb), b = if_flip(p - n, sb);
  const int64_t x = (int64_t)(((uint64_t)if_hi(a) << 32) | if_lo(a)), y = (int64_t)(((uint64_t)if_hi(b) << 32) | if_lo(b));
  return x > y ? (x > 0 ? a : 0.0) : (y > 0 ? b : 0.0);
}

}  // namespace m2cg
