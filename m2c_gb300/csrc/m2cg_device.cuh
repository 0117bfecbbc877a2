// Device-side equations of state, numerical fluxes and slope limiters for the
// GB300 finite-volume step.  All arithmetic is IEEE binary64.
//
// Reference formulas: VarFcnSG.h:64-68, VarFcnNASG.h:55-59, VarFcnMG.h:70-87,
// VarFcnBase.h:120-298, FluxFcnBase.h:82-123, FluxFcnHLLC.h:51-245,
// FluxFcnLLF.h:46-185, FluxFcnGenRoe.h:63-221, Reconstructor.h:96-111.
#pragma once
#include <cstdint>
#include <cfloat>
#include "../../include/m2cg.h"
#include "m2cg_intfp.cuh"

#define M2CG_DEV __device__ __forceinline__

namespace m2cg {

// Material constants precomputed on the host (one entry per material ID).
struct DevMat {
  int type;                      // M2CG_EOS_*
  int clip_default;              // rhomin = 0, pmin = -DBL_MAX, rhomax = pmax = DBL_MAX
  double gam, gam1, Pstiff, gamPs, invgam1;   // SG / NASG (Pstiff = pc for NASG)
  double b, q;                                // NASG
  double rho0, s, e0, rho0_c0_c0, G0_half, G0_rho0;  // MG
  double rhomin, pmin, rhomax, pmax;
};

struct Mats {
  DevMat m[M2CG_MAX_MATERIALS];
};

// ---- binary64 building blocks on the integer and FP64 pipes -----------------
// GB300 runs binary64 at 2 FMA/clk/SM; comparisons, min/max and divisions cost
// FP64-pipe slots too.  Sign and range tests on a double's bit pattern run on
// the integer pipe instead (IEEE-754 binary64 orders like a sign-magnitude
// integer).
// The tests read the two 32-bit words: the compiler turns the same tests on the
// 64-bit pattern back into FP64 comparisons (78 FP64 instructions per cell in
// the reconstruction).
M2CG_DEV long long bits(double x) { return __double_as_longlong(x); }
M2CG_DEV int hi_word(double x) { return __double2hiint(x); }
M2CG_DEV unsigned lo_word(double x) { return (unsigned)__double2loint(x); }
M2CG_DEV bool is_finite_bits(double x) { return (hi_word(x) & 0x7ff00000) != 0x7ff00000; }
// x <= 0 (both zeros included)
M2CG_DEV bool le_zero_bits(double x) { return hi_word(x) < 0 || ((unsigned)hi_word(x) | lo_word(x)) == 0u; }
// x < 0 (negative zero excluded)
M2CG_DEV bool lt_zero_bits(double x) { return hi_word(x) < 0 && (((unsigned)hi_word(x) << 1) | lo_word(x)) != 0u; }
// |x| < c for a positive constant c
M2CG_DEV bool abs_lt_bits(double x, double c) { return (bits(x) & 0x7fffffffffffffffll) < bits(c); }
M2CG_DEV bool is_pos_inf(double x) { return hi_word(x) == 0x7ff00000 && lo_word(x) == 0u; }
M2CG_DEV bool is_neg_inf(double x) { return hi_word(x) == (int)0xfff00000 && lo_word(x) == 0u; }
// Comparisons, minima and maxima of any two doubles on the integer pipe: the
// results of the FP64 instructions for every operand (an FP64 comparison costs
// a full slot of the FP64 pipe, and 115 cycles of latency on a dependent chain).
M2CG_DEV bool is_nan_bits(double x) {
  const int h = hi_word(x) & 0x7fffffff;
  return h > 0x7ff00000 || (h == 0x7ff00000 && lo_word(x) != 0u);
}
M2CG_DEV bool i_eq0(double x) { return (((unsigned)hi_word(x) << 1) | lo_word(x)) == 0u; }
M2CG_DEV bool i_lt0(double x) { return hi_word(x) < 0 && !i_eq0(x) && !is_nan_bits(x); }             // x < 0
M2CG_DEV bool i_le0(double x) { return i_eq0(x) || (hi_word(x) < 0 && !is_nan_bits(x)); }            // x <= 0
M2CG_DEV bool i_gt0(double x) { return hi_word(x) >= 0 && !i_eq0(x) && !is_nan_bits(x); }            // x > 0
M2CG_DEV bool i_ge0(double x) { return i_eq0(x) || (hi_word(x) >= 0 && !is_nan_bits(x)); }           // x >= 0
M2CG_DEV double flip_sign(double x) { return __hiloint2double(hi_word(x) ^ (int)0x80000000, __double2loint(x)); }
M2CG_DEV long long i_key(double x) { return if_key(x); }
M2CG_DEV bool i_special(double a, double b) {   // an infinity or NaN among the two
  return (__double2hiint(a) & 0x7ff00000) == 0x7ff00000 || (__double2hiint(b) & 0x7ff00000) == 0x7ff00000;
}
static __device__ __noinline__ bool lt_fp64(double a, double b) { return a < b; }
static __device__ __noinline__ bool le_fp64(double a, double b) { return a <= b; }
static __device__ __noinline__ double max_fp64(double a, double b) { return fmax(a, b); }
static __device__ __noinline__ double min_fp64(double a, double b) { return fmin(a, b); }
M2CG_DEV bool i_lt(double a, double b) {
  if (i_special(a, b)) return lt_fp64(a, b);
  return i_key(a) < i_key(b) && ((bits(a) | bits(b)) << 1) != 0;
}
M2CG_DEV bool i_le(double a, double b) {
  if (i_special(a, b)) return le_fp64(a, b);
  return i_key(a) <= i_key(b) || ((bits(a) | bits(b)) << 1) == 0;
}
M2CG_DEV double i_min(double a, double b) {
  if (i_special(a, b)) return min_fp64(a, b);
  return i_key(a) <= i_key(b) ? a : b;
}
M2CG_DEV double i_max(double a, double b) {
  if (i_special(a, b)) return max_fp64(a, b);
  return i_key(a) >= i_key(b) ? a : b;
}
// a b < 0: opposite signs, unless the product underflows to zero or an operand is zero or NaN
M2CG_DEV bool i_prod_lt0(double a, double b) {
  const unsigned ea = (unsigned)(bits(a) >> 52) & 0x7ffu, eb = (unsigned)(bits(b) >> 52) & 0x7ffu;
  if (ea + eb < 1100u || ea - 1u > 2045u || eb - 1u > 2045u) return i_lt0(__dmul_rn(a, b));
  return (bits(a) ^ bits(b)) < 0;
}

// a b > 0 likewise
M2CG_DEV bool i_prod_gt0(double a, double b) {
  const unsigned ea = (unsigned)(bits(a) >> 52) & 0x7ffu, eb = (unsigned)(bits(b) >> 52) & 0x7ffu;
  if (ea + eb < 1100u || ea - 1u > 2045u || eb - 1u > 2045u) return __dmul_rn(a, b) > 0.0;
  return (bits(a) ^ bits(b)) >= 0;
}
// Reciprocal and reciprocal square root to 0.51 ulp on the integer pipe
// (m2cg_intfp.cuh: 68 and 99 cycles per warp against 204 and 369 for the
// refined FP64 estimates, and none of them on the FP64 pipe that bounds the
// stage kernels).  Operands outside the normal range -- zero, subnormal,
// infinite, NaN, a negative argument of the root -- take the FP64 form: the
// hardware estimate of the PTX ISA refined by one third-order Householder step.
static __device__ __noinline__ double rcp_fp64(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
static __device__ __noinline__ double rsqrt_fp64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double e = fma(-x, y * y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}
M2CG_DEV double rcp_fast(double x) {
  if (!if_rcp_range(if_hi(x))) return rcp_fp64(x);
  return if_rcp_core(if_hi(x), if_lo(x));
}
M2CG_DEV double rsqrt_fast(double x) {
  if (!if_rsqrt_range(if_hi(x))) return rsqrt_fp64(x);
  return if_rsqrt_core(if_hi(x), if_lo(x));
}

// The same as calls, for kernels whose straight-line code would not fit the
// instruction cache with dozens of copies.
static __device__ __noinline__ double rcp_call(double x) { return rcp_fast(x); }
static __device__ __noinline__ double rsqrt_call(double x) { return rsqrt_fast(x); }

// Quotients of several numerators over one divisor: the divisor's fixed-point
// reciprocal (m2cg_intfp.cuh) is formed once, each quotient takes the
// remaining 40 integer instructions of ddiv.  Correctly rounded, equal to a / b
// bit for bit (m2cg_selftest_quotient checks that on random and edge-case
// operands); operands or results outside the normal range take the IEEE
// division out of line.
struct Quot {
  double b;
  uint64_t D, R;
};
M2CG_DEV Quot quot_of(double b) {
  Quot q;
  q.b = b;
  q.D = if_sig(if_hi(b), if_lo(b));
  q.R = if_recip(q.D);
  return q;
}
M2CG_DEV bool qfast(double a, const Quot& d) { return if_div_range(a, d.b); }
static __device__ __noinline__ double qdiv_call(double a, double b, uint64_t D, uint64_t R) {
  return if_div_range(a, b) ? if_div_core(a, b, D, R) : a / b;
}
M2CG_DEV double qdiv(double a, const Quot& d) { return qdiv_call(a, d.b, d.D, d.R); }

// ---- equation of state ----------------------------------------------------
M2CG_DEV double eos_p(const DevMat& M, double rho, double e) {
  if (M.type == M2CG_EOS_SG) return M.gam1 * rho * e - M.gamPs;   // gamPs = RN(gamma * pc), the same product
  if (M.type == M2CG_EOS_NASG) return ddiv(M.gam1 * (e - M.q), ddiv(1.0, rho) - M.b) - M.gamPs;
  double eta = 1.0 - ddiv(M.rho0, rho);
  return ddiv(M.rho0_c0_c0 * eta * (1.0 - M.G0_half * eta), (1.0 - M.s * eta) * (1.0 - M.s * eta)) + M.G0_rho0 * (e - M.e0);
}
M2CG_DEV double eos_e(const DevMat& M, double rho, double p) {
  if (M.type == M2CG_EOS_SG) return ddiv(p + M.gamPs, M.gam1 * rho);
  if (M.type == M2CG_EOS_NASG) return M.invgam1 * (p + M.gamPs) * (ddiv(1.0, rho) - M.b) + M.q;
  double eta = 1.0 - ddiv(M.rho0, rho);
  return ddiv(p - ddiv(M.rho0_c0_c0 * eta * (1.0 - M.G0_half * eta), (1.0 - M.s * eta) * (1.0 - M.s * eta)), M.G0_rho0) + M.e0;
}
M2CG_DEV double eos_dpdrho(const DevMat& M, double rho, double e) {
  if (M.type == M2CG_EOS_SG) return M.gam1 * e;
  if (M.type == M2CG_EOS_NASG) { double V = ddiv(1.0, rho); return ddiv(M.gam1 * V * V * (e - M.q), (V - M.b) * (V - M.b)); }
  double eta = 1.0 - ddiv(M.rho0, rho);
  double S = 1.0 - M.s * eta;
  return ddiv(ddiv(M.rho0_c0_c0 * (1.0 + (M.s - 2.0 * M.G0_half) * eta), S * S * S) * M.rho0, rho * rho);
}
M2CG_DEV double eos_Gamma(const DevMat& M, double rho) {
  if (M.type == M2CG_EOS_SG) return M.gam1;
  if (M.type == M2CG_EOS_NASG) return ddiv(M.gam1, 1.0 - M.b * rho);
  return ddiv(M.G0_rho0, rho);
}
// VarFcnBase.h:219-223.  The quotients that share a divisor or an operand are
// formed once (NASG's 1/rho enters p, dp/drho and, through p / rho, c^2).
M2CG_DEV double eos_c2(const DevMat& M, double rho, double e) {
  if (M.type == M2CG_EOS_NASG) {
    const double eq = M.gam1 * (e - M.q);
    const Quot R = quot_of(rho);
    const double V = qdiv(1.0, R);
    const double p = ddiv(eq, V - M.b) - M.gamPs;
    const double dpdrho = ddiv(M.gam1 * V * V * (e - M.q), (V - M.b) * (V - M.b));
    return dpdrho + qdiv(p, R) * ddiv(M.gam1, 1.0 - M.b * rho);
  }
  return eos_dpdrho(M, rho, e) + ddiv(eos_p(M, rho, e), rho) * eos_Gamma(M, rho);
}
// eos_c2 with its divisions by rho through a reciprocal the caller shares (same bits)
M2CG_DEV double eos_c2_q(const DevMat& M, double rho, const Quot& R, double e) {
  if (M.type == M2CG_EOS_NASG) {
    const double V = qdiv(1.0, R);
    const double p = ddiv(M.gam1 * (e - M.q), V - M.b) - M.gamPs;
    const double dpdrho = ddiv(M.gam1 * V * V * (e - M.q), (V - M.b) * (V - M.b));
    return dpdrho + qdiv(p, R) * ddiv(M.gam1, 1.0 - M.b * rho);
  }
  return eos_dpdrho(M, rho, e) + qdiv(eos_p(M, rho, e), R) * eos_Gamma(M, rho);
}
// CheckState: true = nonphysical (VarFcnSG.h:96-108, VarFcnNASG.h:73-85, VarFcnBase.h:120-140)
M2CG_DEV bool eos_bad(const DevMat& M, double rho, double p) {
  if (!is_finite_bits(rho) || !is_finite_bits(p)) return true;
  if (M.type == M2CG_EOS_SG || M.type == M2CG_EOS_NASG) return i_le0(rho) || i_le0(p + M.Pstiff);
  if (i_le0(rho)) return true;
  double e = eos_e(M, rho, p);
  return eos_dpdrho(M, rho, e) + ddiv(p, rho) * eos_Gamma(M, rho) <= 0.0;
}
M2CG_DEV bool eos_bad5(const DevMat& M, const double* V) {
  if (!isfinite(V[1]) || !isfinite(V[2]) || !isfinite(V[3])) return true;
  return eos_bad(M, V[0], V[4]);
}
// VarFcnBase.h:262-298 (returns whether it clipped)
M2CG_DEV bool eos_clip(const DevMat& M, double* V) {
  bool c = false;
  if (V[0] < M.rhomin) { V[0] = M.rhomin; c = true; }
  if (V[4] < M.pmin) { V[4] = M.pmin; c = true; }
  if (V[0] > M.rhomax) { V[0] = M.rhomax; c = true; }
  if (V[4] > M.pmax) { V[4] = M.pmax; c = true; }
  return c;
}
// CheckState and ClipDensityAndPressure with the integer-pipe tests above
// (same results for finite and infinite inputs).
M2CG_DEV bool eos_bad5_fast(const DevMat& M, const double* V) {
  if (!is_finite_bits(V[0]) || !is_finite_bits(V[1]) || !is_finite_bits(V[2]) || !is_finite_bits(V[3]) ||
      !is_finite_bits(V[4]))
    return true;
  if (M.type == M2CG_EOS_SG || M.type == M2CG_EOS_NASG) return le_zero_bits(V[0]) || i_le(V[4], flip_sign(M.Pstiff));   // p + Pstiff <= 0 without the addition
  return eos_bad(M, V[0], V[4]);
}
M2CG_DEV bool eos_clip_fast(const DevMat& M, double* V) {
  if (!M.clip_default) return eos_clip(M, V);
  bool c = false;
  if (lt_zero_bits(V[0])) { V[0] = 0.0; c = true; }
  if (is_neg_inf(V[4])) { V[4] = M.pmin; c = true; }
  if (is_pos_inf(V[0])) { V[0] = M.rhomax; c = true; }
  if (is_pos_inf(V[4])) { V[4] = M.pmax; c = true; }
  return c;
}

// VarFcnBase.h:190-201
M2CG_DEV void prim_to_cons(const DevMat& M, const double* V, double* U) {
  U[0] = V[0];
  U[1] = V[0] * V[1]; U[2] = V[0] * V[2]; U[3] = V[0] * V[3];
  double e = eos_e(M, V[0], V[4]);
  U[4] = V[0] * (e + 0.5 * (V[1] * V[1] + V[2] * V[2] + V[3] * V[3]));
}
// Conversions with one reciprocal and no division (SG and NASG closed forms);
// equal to prim_to_cons / cons_to_prim to rounding.
M2CG_DEV void prim_to_cons_fast(const DevMat& M, const double* V, double* U) {
  double k2 = V[1] * V[1] + V[2] * V[2] + V[3] * V[3];
  U[0] = V[0];
  U[1] = V[0] * V[1]; U[2] = V[0] * V[2]; U[3] = V[0] * V[3];
  if (M.type == M2CG_EOS_SG) U[4] = fma(0.5 * V[0], k2, (V[4] + M.gamPs) * M.invgam1);
  else U[4] = V[0] * (eos_e(M, V[0], V[4]) + 0.5 * k2);
}
M2CG_DEV void cons_to_prim_fast(const DevMat& M, const double* U, double* V) {
  V[0] = U[0];
  double ir = rcp_fast(U[0]);
  V[1] = U[1] * ir; V[2] = U[2] * ir; V[3] = U[3] * ir;
  double rhoe = U[4] - 0.5 * V[0] * (V[1] * V[1] + V[2] * V[2] + V[3] * V[3]);
  if (M.type == M2CG_EOS_SG) V[4] = fma(M.gam1, rhoe, -M.gamPs);
  else V[4] = eos_p(M, V[0], rhoe * ir);
}
// VarFcnBase.h:173-186
M2CG_DEV void cons_to_prim(const DevMat& M, const double* U, double* V) {
  V[0] = U[0];
  double invRho = ddiv(1.0, U[0]);
  V[1] = U[1] * invRho; V[2] = U[2] * invRho; V[3] = U[3] * invRho;
  double e = (U[4] - 0.5 * V[0] * (V[1] * V[1] + V[2] * V[2] + V[3] * V[3])) * invRho;
  V[4] = eos_p(M, V[0], e);
}
M2CG_DEV double total_enthalpy(const DevMat& M, const double* V) {
  double e = eos_e(M, V[0], V[4]);
  return e + 0.5 * (V[1] * V[1] + V[2] * V[2] + V[3] * V[3]) + ddiv(V[4], V[0]);
}

// ---- physical flux (FluxFcnBase.h:82-123) ------------------------------------
M2CG_DEV void phys_flux(const DevMat& M, int dir, const double* V, double* F) {
  double H = total_enthalpy(M, V);
  double vn = V[1 + dir];
  double rhou = V[0] * vn;
  F[0] = rhou;
  F[1] = rhou * V[1]; F[2] = rhou * V[2]; F[3] = rhou * V[3];
  F[1 + dir] = rhou * vn + V[4];
  F[4] = rhou * H;
}

M2CG_DEV double avg(double w1, double f1, double w2, double f2) { return ddiv(w1 * f1 + w2 * f2, w1 + w2); }

// Generalized Roe-averaged state of Hu et al. (FluxFcnHLLC.h:57-126)
struct RoeHat {
  double rho_hat, srm, srp, em, ep, e_hat, c_hat, c2_hat, dpdrho_hat, Gamma_hat, p_over_rho_hat;
};
M2CG_DEV void roe_hat(const DevMat& M, int dir, const double* Vm, const double* Vp, RoeHat& r) {
  const double eps = 1e-10;
  r.rho_hat = dsqrt(Vm[0] * Vp[0]);
  r.srm = dsqrt(Vm[0]);
  r.srp = dsqrt(Vp[0]);
  double drho = Vp[0] - Vm[0];
  double dp = Vp[4] - Vm[4];
  double diff = ddiv(Vp[1 + dir] - Vm[1 + dir], r.srm + r.srp);
  r.p_over_rho_hat = avg(r.srm, ddiv(Vm[4], Vm[0]), r.srp, ddiv(Vp[4], Vp[0])) + 0.5 * diff * diff;
  r.em = eos_e(M, Vm[0], Vm[4]);
  r.ep = eos_e(M, Vp[0], Vp[4]);
  double de = r.ep - r.em;
  r.e_hat = avg(r.srm, r.em, r.srp, r.ep);
  double w_rho = ddiv(drho * drho, r.rho_hat * r.rho_hat);
  double w_e = ddiv(de * de, r.e_hat * r.e_hat);
  double denom = w_rho + w_e + eps;
  double dpdrho_avg = avg(r.srm, eos_dpdrho(M, Vm[0], r.em), r.srp, eos_dpdrho(M, Vp[0], r.ep));
  double Gamma_avg = avg(r.srm, eos_Gamma(M, Vm[0]), r.srp, eos_Gamma(M, Vp[0]));
  double t1 = (w_e + eps) * dpdrho_avg;
  double t2 = ddiv((dp - Gamma_avg * r.rho_hat * de) * drho, r.rho_hat * r.rho_hat);
  r.dpdrho_hat = ddiv(t1 + t2, denom);
  double g1 = (w_rho + eps) * Gamma_avg;
  double g2 = ddiv((dp - dpdrho_avg * drho) * de, r.rho_hat * r.e_hat * r.e_hat);
  r.Gamma_hat = ddiv(g1 + g2, denom);
  r.c2_hat = r.dpdrho_hat + r.Gamma_hat * r.p_over_rho_hat;
  if (r.c2_hat <= 0) { r.c_hat = eps; r.c2_hat = eps * eps; }
  else r.c_hat = dsqrt(r.c2_hat);
}

// FluxFcnHLLC.h:158-192
M2CG_DEV void hllc_fstar(const DevMat& M, int dir, const double* V, double S, double Sstar, double* F) {
  double velo = V[1 + dir];
  double rhostar = ddiv(V[0] * (S - velo), S - Sstar);
  double U[5];
  prim_to_cons(M, V, U);
  double Us[5];
  Us[0] = 1.0; Us[1] = V[1]; Us[2] = V[2]; Us[3] = V[3];
  Us[1 + dir] = Sstar;
  Us[4] = ddiv(U[4], V[0]) + (Sstar - velo) * (Sstar + ddiv(V[4], V[0] * (S - velo)));
  phys_flux(M, dir, V, F);
#pragma unroll
  for (int i = 0; i < 5; i++) F[i] += S * (Us[i] * rhostar - U[i]);
}

// FluxFcnHLLC.h:196-245.  Returns false if c^2 < 0 on either side.
M2CG_DEV bool flux_hllc(const DevMat& M, int dir, const double* Vm, const double* Vp, double* F) {
  RoeHat r;
  roe_hat(M, dir, Vm, Vp, r);
  double cm = eos_c2(M, Vm[0], r.em);
  double cp = eos_c2(M, Vp[0], r.ep);
  bool ok = !(cm < 0.0) && !(cp < 0.0);
  cm = dsqrt(fmax(cm, 0.0));
  cp = dsqrt(fmax(cp, 0.0));
  double vm = Vm[1 + dir], vp = Vp[1 + dir];
  double vh = avg(r.srm, vm, r.srp, vp);
  double Sm = fmin(vm - cm, vh - r.c_hat);
  double Sp = fmax(vp + cp, vh + r.c_hat);
  if (0.0 <= Sm) phys_flux(M, dir, Vm, F);
  else if (0.0 >= Sp) phys_flux(M, dir, Vp, F);
  else {
    double Sstar = ddiv(Vp[4] - Vm[4] + Vm[0] * vm * (Sm - vm) - Vp[0] * vp * (Sp - vp),
                        Vm[0] * (Sm - vm) - Vp[0] * (Sp - vp));
    if (Sstar >= 0.0) hllc_fstar(M, dir, Vm, Sm, Sstar, F);
    else hllc_fstar(M, dir, Vp, Sp, Sstar, F);
  }
  return ok;
}

// ---- HLLC for the FP64 pipe ---------------------------------------------------
// The same flux as flux_hllc (FluxFcnHLLC.h:57-245) in the fewest FP64
// instructions (57 for a stiffened gas; the FP64 pipe bounds the stage
// kernels): reciprocals and roots on the integer pipe, 1/rho and sqrt(rho) from
// one reciprocal root per side, the Roe weight shared by all averages,
// comparisons and selections on the integer pipe.  Results agree with the
// reference's order to a few ulps.
struct Side {
  double rho, vn, p, inv_rho, sr, e, dpdrho, Gamma, c2, c;
};
M2CG_DEV void side_eos(const DevMat& M, const double* V, int dir, Side& S) {
  S.rho = V[0];
  S.vn = V[1 + dir];
  S.p = V[4];
  double y = rsqrt_call(S.rho);
  S.sr = S.rho * y;
  S.inv_rho = y * y;
  if (M.type == M2CG_EOS_SG) {
    // c^2 = dp/drho + p/rho Gamma = gamma (p + p_inf) / rho (VarFcnSG.h:64-68,
    // VarFcnBase.h:219-223), the same value to rounding without the
    // cancellation of the two terms near p = -p_inf.  e follows where it is used.
    S.e = 0.0;
    S.c2 = M.gam * (S.p + M.Pstiff) * S.inv_rho;
    S.c = i_gt0(S.c2) ? S.c2 * rsqrt_call(S.c2) : 0.0;
    return;
  } else if (M.type == M2CG_EOS_NASG) {
    double vb = S.inv_rho - M.b;
    S.e = M.invgam1 * (S.p + M.gamPs) * vb + M.q;
    double r = S.inv_rho * rcp_call(vb);
    S.dpdrho = M.gam1 * (S.e - M.q) * r * r;
    S.Gamma = M.gam1 * rcp_call(1.0 - M.b * S.rho);
  } else {
    S.e = eos_e(M, S.rho, S.p);
    S.dpdrho = eos_dpdrho(M, S.rho, S.e);
    S.Gamma = eos_Gamma(M, S.rho);
  }
  S.c2 = S.dpdrho + S.p * S.inv_rho * S.Gamma;
  S.c = i_gt0(S.c2) ? S.c2 * rsqrt_call(S.c2) : 0.0;
}
M2CG_DEV bool flux_hllc_fast(const DevMat& M, int dir, const double* Vm, const double* Vp, double* F) {
  const double eps = 1e-10;
  Side A, B;
  side_eos(M, Vm, dir, A);
  side_eos(M, Vp, dir, B);
  const double inv_s = rcp_call(A.sr + B.sr);
  const double dp = B.p - A.p;
  const double diff = (B.vn - A.vn) * inv_s;
  double c2_hat;
  if (M.type == M2CG_EOS_SG) {
    // Stiffened gas: p is linear in rho e with the constant Gamma = gamma - 1,
    // and the Roe-averaged jumps satisfy d(rho e) = rho_hat de + e_hat drho
    // exactly, so the generalized averages of FluxFcnHLLC.h:99-119 reduce to
    // Gamma_hat = gamma - 1 and dp/drho_hat = (gamma - 1) e_hat; with
    // (gamma - 1)(e + p / rho) = c^2, c_hat^2 is the average of the two c^2 plus
    // (gamma - 1) diff^2 / 2 (the reference's form carries its rounding through
    // a cancellation when dp ~ Gamma rho_hat de).
    c2_hat = fma(0.5 * M.gam1 * diff, diff, (A.sr * A.c2 + B.sr * B.c2) * inv_s);
  } else {
    const double p_over_rho_hat = (A.sr * (A.p * A.inv_rho) + B.sr * (B.p * B.inv_rho)) * inv_s + 0.5 * diff * diff;
    const double e_hat = (A.sr * A.e + B.sr * B.e) * inv_s;
    const double rho_hat = A.sr * B.sr;
    const double irr = A.inv_rho * B.inv_rho;          // 1 / rho_hat^2
    const double drho = B.rho - A.rho;
    double de = B.e - A.e;
    double inv_e = rcp_call(e_hat);
    double w_rho = drho * drho * irr;
    double de_e = de * inv_e;
    double w_e = de_e * de_e;
    double inv_den = rcp_call(w_rho + w_e + eps);
    double dpdrho_avg = (A.sr * A.dpdrho + B.sr * B.dpdrho) * inv_s;
    double Gamma_avg = (A.sr * A.Gamma + B.sr * B.Gamma) * inv_s;
    double dpdrho_hat = ((w_e + eps) * dpdrho_avg + (dp - Gamma_avg * rho_hat * de) * drho * irr) * inv_den;
    double Gamma_hat = ((w_rho + eps) * Gamma_avg + (dp - dpdrho_avg * drho) * de_e * inv_e * (A.inv_rho * B.sr * B.inv_rho * A.sr)) * inv_den;
    c2_hat = dpdrho_hat + Gamma_hat * p_over_rho_hat;
  }
  const double c_hat = i_le0(c2_hat) ? eps : c2_hat * rsqrt_call(c2_hat);
  const double vh = (A.sr * A.vn + B.sr * B.vn) * inv_s;
  const double Sm = i_min(A.vn - A.c, vh - c_hat);
  const double Sp = i_max(B.vn + B.c, vh + c_hat);
  const bool ok = !i_lt0(A.c2) && !i_lt0(B.c2);
  // FluxFcnHLLC.h:226-241: F_L, F_R, F*_L or F*_R.  The side K and its state --
  // (rho, vn, p) or the star state (rho*, S*, p*) -- are selected first and the
  // flux evaluated once, so lanes of a warp whose faces differ do not run
  // several branches.  F* = F + S (U* - U) is the physical flux of the star
  // state with energy E* (the jump conditions across S): no cancellation
  // between S U* and S U.
  const bool sup_l = i_ge0(Sm), sup_r = i_le0(Sp);
  const double am = A.rho * (Sm - A.vn), bp = B.rho * (Sp - B.vn);
  const double Sstar = (dp + am * A.vn - bp * B.vn) * rcp_call(am - bp);
  const bool left = sup_l || (!sup_r && i_ge0(Sstar)), sup = sup_l || sup_r;
  // value selects (no pointer to either side, which would put them in memory)
  double V[5];
#pragma unroll
  for (int i = 0; i < 5; i++) V[i] = left ? Vm[i] : Vp[i];
  const double inv_rho = left ? A.inv_rho : B.inv_rho;
  const double vn = V[1 + dir], p = V[4];
  const double e = M.type == M2CG_EOS_SG ? (p + M.gamPs) * M.invgam1 * inv_rho : (left ? A.e : B.e);
  const double a = left ? am : bp;                    // rho (S - vn)
  const double Sw = left ? Sm : Sp;
  const double rs = a * rcp_call(Sw - Sstar);
  const double w = sup ? vn : Sstar, rw = sup ? V[0] : rs;
  const double dv = w - vn;
  const double ps = fma(a, dv, p), de = dv * fma(p, rcp_call(a), w);
  const double pw = sup ? p : ps;
  const double E = fma(0.5, V[1] * V[1] + V[2] * V[2] + V[3] * V[3], e) + (sup ? 0.0 : de);
  const double m = rw * w;
  F[0] = m;
  F[1] = m * V[1]; F[2] = m * V[2]; F[3] = m * V[3];
  F[1 + dir] = fma(m, w, pw);
  F[4] = fma(m, E, pw * w);
  return ok;
}

// FluxFcnLLF.h:46-111 and 118-185 (two materials)
M2CG_DEV bool flux_llf2(const DevMat& Mm, const DevMat& Mp, int dir, const double* Vm, const double* Vp, double* F) {
  double em = eos_e(Mm, Vm[0], Vm[4]);
  double ep = eos_e(Mp, Vp[0], Vp[4]);
  double cm = eos_c2(Mm, Vm[0], em);
  double cp = eos_c2(Mp, Vp[0], ep);
  bool ok = !(cm < 0.0) && !(cp < 0.0);
  cm = dsqrt(fmax(cm, 0.0));
  cp = dsqrt(fmax(cp, 0.0));
  double a = fmax(fabs(Vm[1 + dir]) + cm, fabs(Vp[1 + dir]) + cp);
  double fm[5], fp[5], Um[5], Up[5];
  phys_flux(Mm, dir, Vm, fm);
  phys_flux(Mp, dir, Vp, fp);
  prim_to_cons(Mm, Vm, Um);
  prim_to_cons(Mp, Vp, Up);
#pragma unroll
  for (int i = 0; i < 5; i++) F[i] = 0.5 * ((fm[i] + fp[i]) - a * (Up[i] - Um[i]));
  return ok;
}

// FluxFcnGenRoe.h:63-221 with the eigenvectors of FluxFcnBase.h:154-176 (F),
// 203-225 (G), 252-274 (H).
M2CG_DEV bool flux_genroe(const DevMat& M, int dir, const double* Vm, const double* Vp, double del, double* F) {
  double srm = dsqrt(Vm[0]), srp = dsqrt(Vp[0]);
  double rho_hat = dsqrt(Vm[0] * Vp[0]);
  double vel[3];
#pragma unroll
  for (int m = 0; m < 3; m++) vel[m] = avg(srm, Vm[1 + m], srp, Vp[1 + m]);
  double H_hat = avg(srm, total_enthalpy(M, Vm), srp, total_enthalpy(M, Vp));
  double dvel[3] = {Vp[1] - Vm[1], Vp[2] - Vm[2], Vp[3] - Vm[3]};
  double dp = Vp[4] - Vm[4], drho = Vp[0] - Vm[0];
  RoeHat r;
  roe_hat(M, dir, Vm, Vp, r);
  double c = r.c_hat, c2 = r.c2_hat;
  double vn = vel[dir];
  double vel2 = vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2];
  double e_term = r.e_hat + 0.5 * vel2 - ddiv(r.dpdrho_hat, r.Gamma_hat);
  double lam[5] = {vn - c, vn, vn, vn, vn + c};
  double a[5];
  a[0] = ddiv(dp - rho_hat * c * dvel[dir], 2 * c2);
  a[4] = ddiv(dp + rho_hat * c * dvel[dir], 2 * c2);
#pragma unroll
  for (int p = 1; p <= 3; p++) a[p] = (p - 1 == dir) ? (ddiv(-dp, c2) + drho) : rho_hat * dvel[p - 1];
  double tol = lam[0];
#pragma unroll
  for (int i = 1; i < 5; i++) if (fabs(lam[i]) > tol) tol = fabs(lam[i]);
  tol *= del;
#pragma unroll
  for (int i = 0; i < 5; i++) if (fabs(lam[i]) < tol) lam[i] = ddiv(lam[i] * lam[i] + tol * tol, 2 * tol);
  double fm[5], fp[5];
  phys_flux(M, dir, Vm, fm);
  phys_flux(M, dir, Vp, fp);
#pragma unroll
  for (int i = 0; i < 5; i++) F[i] = 0.5 * (fm[i] + fp[i]);
  // subtract 0.5|lam_p| a_p r_p in the order p = 0..4 for every component
#pragma unroll
  for (int p = 0; p < 5; p++) {
    double coef = 0.5 * fabs(lam[p]) * a[p];
    double R[5] = {0, 0, 0, 0, 0};
    if (p == 0 || p == 4) {
      R[0] = 1; R[1] = vel[0]; R[2] = vel[1]; R[3] = vel[2];
      R[1 + dir] = (p == 0) ? vn - c : vn + c;
      R[4] = (p == 0) ? H_hat - vn * c : H_hat + vn * c;
    } else if (p - 1 == dir) {
      R[0] = 1; R[1] = vel[0]; R[2] = vel[1]; R[3] = vel[2]; R[4] = e_term;
    } else {
      R[p] = 1; R[4] = vel[p - 1];
    }
#pragma unroll
    for (int i = 0; i < 5; i++) F[i] -= coef * R[i];
  }
  return true;
}

// ---- slope limiters (Reconstructor.h:96-111) ------------------------------------
// The candidate of smallest magnitude on the integer pipe (equal signs order
// like the bit patterns, and alpha min(|dq0|, |dq1|) rounds like the smaller of
// the two products): two FP64 instructions against nine.  The same value as the
// reference's form, whose comparisons make NaN differences give 0.
static __device__ __noinline__ double gen_minmod_fp64(double alpha, double dq0, double dq1) {
  // uniform mesh: A = B = 1, so B/(A+1) = 0.5
  if (dq0 < 0.0 && dq1 < 0.0) return fmax(alpha * dq0, fmax(0.5 * (dq0 + dq1), alpha * dq1));
  if (dq0 > 0.0 && dq1 > 0.0) return fmin(alpha * dq0, fmin(0.5 * (dq0 + dq1), alpha * dq1));
  return 0.0;
}
static __device__ __noinline__ double gen_minmod(double alpha, double dq0, double dq1) {
  const unsigned long long MAG = 0x7fffffffffffffffull;
  const unsigned long long u0 = (unsigned long long)bits(dq0) & MAG, u1 = (unsigned long long)bits(dq1) & MAG;
  if ((bits(dq0) ^ bits(dq1)) < 0 || u0 == 0ull || u1 == 0ull || is_nan_bits(dq0) || is_nan_bits(dq1)) return 0.0;
  const double s = __dadd_rn(dq0, dq1);
  const int es = __double2hiint(s) & 0x7ff00000;
  if (es <= 0x00100000 || es == 0x7ff00000 || !(bits(alpha) > 0)) return gen_minmod_fp64(alpha, dq0, dq1);
  const double h = __hiloint2double(__double2hiint(s) - 0x00100000, __double2loint(s));   // s / 2
  const double t = __dmul_rn(alpha, u0 < u1 ? dq0 : dq1);
  return ((unsigned long long)bits(h) & MAG) < ((unsigned long long)bits(t) & MAG) ? h : t;
}
// van Albada on the integer pipe (if_van_albada: 182 cycles per warp with one
// FP64 multiplication, against 666 for the FP64 form with its ten); products
// next to the 1e-16 threshold and special operands take the FP64 form.  Every
// operation is pinned (no contraction), so every caller gets the same bits.
static __device__ __noinline__ double van_albada_fp64(double dq0, double dq1) {
  double pr = __dmul_rn(dq0, dq1);
  if (le_zero_bits(pr) || abs_lt_bits(pr, 1e-16)) return 0.0;
  const double a = __dmul_rn(dq0, dq0), b = __dmul_rn(dq1, dq1);
  return __dmul_rn(fma(dq1, a, __dmul_rn(dq0, b)), rcp_fast(__dadd_rn(a, b)));
}
static __device__ __noinline__ double van_albada_fast(double dq0, double dq1) {
  double s;
  if (!if_van_albada(dq0, dq1, s)) s = van_albada_fp64(dq0, dq1);
  return s;
}
}  // namespace m2cg
