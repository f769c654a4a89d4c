// physics.cuh -- pointwise state math and Riemann solvers of the fv2d hydro
// step, for device code (and host code where marked __host__).
//
// Every expression keeps the operand order of the reference so that, built
// with -fmad=false, binary64 results are bit-identical to it:
//   primToCons / consToPrim / speedOfSound   States.h:19-46
//   hll                                      RiemannSolvers.h:7-51
//   hllc                                     RiemannSolvers.h:53-128
//   fslp                                     RiemannSolvers.h:130-171
//   minmod                                   Update.h:77-85
// Differences from the reference are in control flow only: the Riemann
// solvers evaluate their candidate fluxes without data-dependent branches
// and select at the end (same values, no warp divergence), and constants such
// as 1/(gamma-1) are computed once by the caller with the same operation.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "softfp.cuh"
#include "step_common.cuh"

namespace fv2d {

// Division and square root: binary64 on the device goes through the
// integer-pipe routines (same correctly rounded bits as the hardware
// instructions, off the FP64 pipe); binary32 and host code use the operators.
__host__ __device__ __forceinline__ double fv_div(double a, double b) {
#ifdef __CUDA_ARCH__
  return softfp::div_rn(a, b);
#else
  return a / b;
#endif
}
__host__ __device__ __forceinline__ float fv_div(float a, float b) { return a / b; }
// a1 / b and a2 / b (one reciprocal of b on the device)
__host__ __device__ __forceinline__ void fv_div2(double a1, double a2, double b, double &q1, double &q2) {
#ifdef __CUDA_ARCH__
  const double2 q = softfp::div2_rn(a1, a2, b);
  q1 = q.x;
  q2 = q.y;
#else
  q1 = a1 / b;
  q2 = a2 / b;
#endif
}
__host__ __device__ __forceinline__ void fv_div2(float a1, float a2, float b, float &q1, float &q2) {
  q1 = a1 / b;
  q2 = a2 / b;
}
__host__ __device__ __forceinline__ double fv_sqrt(double x) {
#ifdef __CUDA_ARCH__
  return softfp::sqrt_rn(x);
#else
  return sqrt(x);
#endif
}
__host__ __device__ __forceinline__ float fv_sqrt(float x) { return sqrtf(x); }
// Several quotients by one divisor: r = fv_recip(b) once, fv_div_by(a, b, r)
// per dividend (binary64 on the device: the reciprocal word of b is formed
// once; the quotients are the same correctly rounded values as a / b).
__host__ __device__ __forceinline__ uint32_t fv_recip(double b) {
#ifdef __CUDA_ARCH__
  return softfp::recip_of(b);
#else
  (void)b;
  return 0u;
#endif
}
__host__ __device__ __forceinline__ double fv_div_by(double a, double b, uint32_t r) {
#ifdef __CUDA_ARCH__
  return softfp::div_by(a, b, r);
#else
  (void)r;
  return a / b;
#endif
}
__host__ __device__ __forceinline__ uint32_t fv_recip(float) { return 0u; }
__host__ __device__ __forceinline__ float fv_div_by(float a, float b, uint32_t) { return a / b; }

// Comparisons, fmin / fmax and scalings by 1/2: on the device, binary64 goes
// through the bit-pattern forms of softfp.cuh (IEEE results, integer pipe).
#ifdef __CUDA_ARCH__
#define FV2D_D(dev, host) return dev
#else
#define FV2D_D(dev, host) return host
#endif
__host__ __device__ __forceinline__ bool fv_gt0(double x) { FV2D_D(softfp::gt0(x), x > 0.0); }
__host__ __device__ __forceinline__ bool fv_lt0(double x) { FV2D_D(softfp::lt0(x), x < 0.0); }
__host__ __device__ __forceinline__ bool fv_ge0(double x) { FV2D_D(softfp::ge0(x), x >= 0.0); }
__host__ __device__ __forceinline__ bool fv_le0(double x) { FV2D_D(softfp::le0(x), x <= 0.0); }
__host__ __device__ __forceinline__ bool fv_lt(double x, double y) { FV2D_D(softfp::lt(x, y), x < y); }
__host__ __device__ __forceinline__ bool fv_lt_abs(double x, double y) {
  FV2D_D(softfp::lt_abs(x, y), fabs(x) < fabs(y));
}
__host__ __device__ __forceinline__ bool fv_prod_neg(double x, double y) {
  FV2D_D(softfp::prod_neg(x, y), x * y < 0.0);
}
__host__ __device__ __forceinline__ double fv_fmax(double x, double y) { FV2D_D(softfp::fmax_nm(x, y), fmax(x, y)); }
__host__ __device__ __forceinline__ double fv_fmin(double x, double y) { FV2D_D(softfp::fmin_nm(x, y), fmin(x, y)); }
__host__ __device__ __forceinline__ double fv_half(double x) { FV2D_D(softfp::half(x), 0.5 * x); }
__host__ __device__ __forceinline__ double fv_mul(double x, double y) { FV2D_D(softfp::mul_rn(x, y), x * y); }
__host__ __device__ __forceinline__ bool fv_isnan(double x) { FV2D_D(softfp::isnan_b(softfp::bits(x)), isnan(x)); }
#undef FV2D_D
__host__ __device__ __forceinline__ bool fv_gt0(float x) { return x > 0.0f; }
__host__ __device__ __forceinline__ bool fv_lt0(float x) { return x < 0.0f; }
__host__ __device__ __forceinline__ bool fv_ge0(float x) { return x >= 0.0f; }
__host__ __device__ __forceinline__ bool fv_le0(float x) { return x <= 0.0f; }
__host__ __device__ __forceinline__ bool fv_lt(float x, float y) { return x < y; }
__host__ __device__ __forceinline__ bool fv_lt_abs(float x, float y) { return fabsf(x) < fabsf(y); }
__host__ __device__ __forceinline__ bool fv_prod_neg(float x, float y) { return x * y < 0.0f; }
__host__ __device__ __forceinline__ float fv_fmax(float x, float y) { return fmaxf(x, y); }
__host__ __device__ __forceinline__ float fv_fmin(float x, float y) { return fminf(x, y); }
__host__ __device__ __forceinline__ float fv_half(float x) { return 0.5f * x; }
__host__ __device__ __forceinline__ float fv_mul(float x, float y) { return x * y; }
__host__ __device__ __forceinline__ bool fv_isnan(float x) { return isnan(x); }

// Products moved from the binary64 pipe to the integer pipes (softfp::mul_rn),
// by group: a product holds the binary64 pipe for 76 cycles of an SM
// sub-partition, an integer-pipe one the ALU for about 80, so the set that
// balances the two is the fastest.  The sets are masks (bit GROUP - 1: that
// group on the integer pipes); the groups are
//   1  HLLC: squared velocities
//   2  HLLC: total energy (rho/2 (u^2 + v^2), p / (gamma - 1))
//   3  the update's dt (F_L - F_R) products
//   4  consToPrim: kinetic energy and (E - Ek)(gamma - 1)
//   5  HLLC: rho (u - S)
//   6  HLLC: p* numerator
//   7  HLLC: star energy
//   8  HLLC: fluxes
//   9  HLL: products of each side's state (kinetic energy, fluxes, momenta)
//  10  HLL: the HLL average's products by the wave speeds
//  11  viscous face terms
//  12  conduction fluxes and the conduction / viscosity update products
//  13  MUSCL-Hancock predictor
//  14  FSLP
//  15  HLLC: u* numerator
// Measured (ms a step; group on the binary64 pipe | on the integer pipes):
// Sedov 2048^2 HLLC: 1 0.96 | 0.94, 3 1.00 | 0.94, 8 1.00 | 0.96; KH 2048^2
// HLLC: 4 1.02 | 1.07, 6 1.02 | 1.06, 7 1.05 | 1.06; its PCM form: 5 0.80 | 0.77;
// HLL: 9 1.58 | 1.40; FSLP RK2 777 x 1501: 3 0.327 | 0.334 a stage; RT
// 1024 x 3072: 10 1.64 | 1.60, 12 1.48 | 1.46.
template <int... GROUPS>
constexpr int soft_groups = ((1 << (GROUPS - 1)) | ...);
constexpr int kSoftMulHllc = soft_groups<1, 2, 3, 5, 8, 9, 12, 13, 14, 15>;
constexpr int kSoftMul = soft_groups<1, 2, 5, 8, 9, 12, 13, 14, 15>;          // HLL and FSLP
constexpr int kSoftMulVisc = soft_groups<1, 2, 5, 8, 9, 10, 12, 13, 14, 15>;  // the same with viscosity
// Sums and differences.  In binary64 on the device a + b is issued as the
// multiply-add a * one + b, with `one` = 1 in a register that the compiler
// cannot see through: the same correctly rounded sum (signed zeros, infinities
// and NaNs included), but GB300 takes a warp's three-register DFMA every 64
// cycles of an SM sub-partition and a DADD or DMUL (or a DFMA with a constant
// operand) only every 76 (measured: 100 % against 84 % of the pipe's peak), and
// the step is bound by that pipe: KH 2048^2 1.08 -> 1.02 ms a step, Sedov 0.99 ->
// 0.94, RT 1024 x 3072 1.54 -> 1.48.  Products stay DMULs: a register pair for
// their -0 addend cost as much as it gave.
template <class R>
struct Adder {
  R one = R(1);
  __host__ __device__ __forceinline__ R operator()(R a, R b) const { return a + b; }
  __host__ __device__ __forceinline__ R sub(R a, R b) const { return a - b; }
};
template <>
struct Adder<double> {
  double one = 1.0;
  __host__ __device__ __forceinline__ double operator()(double a, double b) const {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, one, b);
#else
    return a + b;
#endif
  }
  __host__ __device__ __forceinline__ double sub(double a, double b) const {
#ifdef __CUDA_ARCH__
    return __fma_rn(-b, one, a);
#else
    return a - b;
#endif
  }
};

template <int GROUP, int SOFT, class R>
__host__ __device__ __forceinline__ R mulx(R a, R b) {
  if constexpr ((SOFT >> (GROUP - 1)) & 1) return fv_mul(a, b);
  else return a * b;
}
// {x0 y0, x1 y1} of one group: on the integer pipes in one call
template <int GROUP, int SOFT, class R>
__host__ __device__ __forceinline__ void mulx2(R x0, R y0, R x1, R y1, R &r0, R &r1) {
#ifdef __CUDA_ARCH__
  if constexpr (sizeof(R) == 8 && ((SOFT >> (GROUP - 1)) & 1)) {
    const double2 r = softfp::mul2_rn(x0, y0, x1, y1);
    r0 = r.x;
    r1 = r.y;
    return;
  }
#endif
  r0 = x0 * y0;
  r1 = x1 * y1;
}
// {a1 / b1, a2 / b2}; {a1 / b, a2 / b} with b's reciprocal word r
__host__ __device__ __forceinline__ void fv_quot2(double a1, double b1, double a2, double b2, double &q1, double &q2) {
#ifdef __CUDA_ARCH__
  const double2 q = softfp::quot2_rn(a1, b1, a2, b2);
  q1 = q.x;
  q2 = q.y;
#else
  q1 = a1 / b1;
  q2 = a2 / b2;
#endif
}
__host__ __device__ __forceinline__ void fv_div2_by(double a1, double a2, double b, uint32_t r, double &q1, double &q2) {
#ifdef __CUDA_ARCH__
  const double2 q = softfp::div2_by(a1, a2, b, r);
  q1 = q.x;
  q2 = q.y;
#else
  (void)r;
  q1 = a1 / b;
  q2 = a2 / b;
#endif
}

enum { IR = 0, IU = 1, IV = 2, IP = 3, IE = 3 };

template <class R>
struct S4 {
  R r, u, v, p;  // (rho, u, v, p) or (rho, rho u, rho v, E)
};

// Per-simulation constants used by the pointwise functions.
template <class R>
struct Gas {
  R gamma;   // gamma0
  R gm1;     // gamma0 - 1.0
  R entho;   // 1.0 / (gamma0 - 1.0)               (RiemannSolvers.h:76)
  R fslp_K;  // FSLP K                              (SimInfo.h:399)
  uint32_t rgm1;  // fv_recip(gm1): the divisions by gamma0 - 1 (set by make_gas)
  Adder<R> add;
};

template <class R>
__host__ __device__ __forceinline__ Gas<R> make_gas(R gamma, R gm1, R entho, R fslp_K, Adder<R> add = Adder<R>()) {
  return Gas<R>{gamma, gm1, entho, fslp_K, fv_recip(gm1), add};
}

// States.h:19-30
template <class R>
__host__ __device__ __forceinline__ S4<R> prim_to_cons(const S4<R> &q, const Gas<R> &g) {
  S4<R> s;
  s.r = q.r;
  s.u = q.r * q.u;
  s.v = q.r * q.v;
  R Ek = fv_div(fv_half(s.u * s.u + s.v * s.v), q.r);
  s.p = (Ek + fv_div_by(q.p, g.gm1, g.rgm1));
  return s;
}

// States.h:32-43
template <int SOFT = kSoftMul, class R>
__host__ __device__ __forceinline__ S4<R> cons_to_prim(const S4<R> &u, const Gas<R> &g) {
  S4<R> q;
  q.r = u.r;
  fv_div2(u.u, u.v, u.r, q.u, q.v);
  R uu, vv;
  mulx2<4, SOFT>(q.u, q.u, q.v, q.v, uu, vv);
  R Ek = mulx<4, SOFT>(fv_half(q.r), g.add(uu, vv));
  q.p = mulx<4, SOFT>(g.add.sub(u.p, Ek), g.gm1);
  return q;
}

template <class R>
__device__ __forceinline__ R dsqrt(R x) {
  return fv_sqrt(x);
}

// States.h:45-46
template <int SOFT = kSoftMul, class R>
__device__ __forceinline__ R sound_speed(const S4<R> &q, const Gas<R> &g) {
  return dsqrt(fv_div(mulx<1, SOFT>(q.p, g.gamma), q.r));
}
// the same with the reciprocal of q.r already formed (fv_recip)
template <int SOFT = kSoftMul, class R>
__device__ __forceinline__ R sound_speed_r(const S4<R> &q, const Gas<R> &g, uint32_t rr) {
  return dsqrt(fv_div_by(mulx<1, SOFT>(q.p, g.gamma), q.r, rr));
}

// ---------------------------------------------------------------- CFL filter
// The CFL reduction needs the largest inverse hyperbolic dt of a grid
// exactly, so a cell's value only matters when it can exceed a maximum already
// reached.  inv_dt_bound gives an upper bound of a cell's value in binary32
// (30-40 instructions and no binary64 ones, against ~350 and 3 for the exact
// value): the fields truncated to binary32 (relative error below 2^-23 each),
// the approximate reciprocal and square root (2^-22), half a dozen roundings,
// all of one sign, within a factor 1 + 2^-18.  States the bound does not cover
// (negative, infinite, NaN, outside binary32's range) give a NaN, which no
// test passes over.
__device__ __forceinline__ float truncated_f32(double x) {  // |x|; 0 below 2^-126, NaN from 2^127 up
  const uint64_t b = softfp::bits(x);
  const uint32_t h = (uint32_t)(b >> 32) & 0x7FFFFFFFu;
  const uint32_t f = h < 0x38100000u ? 0u : ((h - 0x38000000u) << 3) | ((uint32_t)b >> 29);
  return __uint_as_float(h >= 0x47E00000u ? 0x7FC00000u : f);
}
__device__ __forceinline__ float inv_dt_bound(const S4<double> &q, const DtBound &d) {
  float rr, cs;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rr) : "f"(truncated_f32(q.r)));
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(cs) : "f"(__fmul_rn(__fmul_rn(truncated_f32(q.p), d.gamma), rr)));
  const float b = __fmul_rn(__fadd_rn(__fmul_rn(__fadd_rn(cs, truncated_f32(q.u)), d.inv_dx),
                                      __fmul_rn(__fadd_rn(cs, truncated_f32(q.v)), d.inv_dy)),
                            1.0f + 0x1p-18f);
  const bool negative = (int32_t)((softfp::bits(q.r) | softfp::bits(q.p)) >> 32) < 0;
  // a vanishing sound speed may have lost a factor to underflow
  return negative || !(cs > 0x1p-40f) || !(cs < 0x1p40f) ? __uint_as_float(0x7FC00000u) : b;
}
// whether a cell with that bound can exceed the maximum reached so far (the
// bits of a non-negative double)
__device__ __forceinline__ bool may_exceed(float bound, uint64_t max_bits) {
  return !(bound < truncated_f32(softfp::from_bits(max_bits)));
}
inline DtBound dt_bound_of(double gamma, double dx, double dy) {
  const double lo = 1e-30, hi = 1e30;
  const bool ok = dx > lo && dx < hi && dy > lo && dy < hi && gamma > 1e-6 && gamma < 1e6;
  return ok ? DtBound{(float)gamma, (float)(1.0 / dx), (float)(1.0 / dy)} : DtBound{NAN, NAN, NAN};
}

// Update.h:77-85
template <class R>
__host__ __device__ __forceinline__ R minmod(R dL, R dR) {
  R m = fv_lt_abs(dL, dR) ? dL : dR;
  return fv_prod_neg(dL, dR) ? R(0) : m;
}

template <class R>
__device__ __forceinline__ R sel(bool c, R a, R b) {
  return c ? a : b;
}

// RiemannSolvers.h:7-51.  All three candidates are evaluated, then selected
// in the reference's branch order (SL >= 0, SR <= 0, else the HLL state).
template <class R>
__device__ __forceinline__ void riemann_hll(const S4<R> &qL, const S4<R> &qR, S4<R> &f, R &pout, const Gas<R> &g) {
  // every quotient by rho_L (rho_R) shares one reciprocal
  const uint32_t rL = fv_recip(qL.r), rR = fv_recip(qR.r);
  const R aL = sound_speed_r(qL, g, rL);
  const R aR = sound_speed_r(qR, g, rR);
  const R sminL = qL.u - aL;
  const R smaxL = qL.u + aL;
  const R sminR = qR.u - aR;
  const R smaxR = qR.u + aR;
  const R SL = fv_fmin(sminL, sminR);
  const R SR = fv_fmax(smaxL, smaxR);
  // computeFlux (RiemannSolvers.h:133-141).  p/(gamma-1) is also the pressure
  // term of primToCons below: the same division, evaluated once.
  const R peL = fv_div_by(qL.p, g.gm1, g.rgm1);
  const R peR = fv_div_by(qR.p, g.gm1, g.rgm1);
  const R EkL = (fv_half(qL.r) * ((qL.u * qL.u) + (qL.v * qL.v)));
  const R EkR = (fv_half(qR.r) * ((qR.u * qR.u) + (qR.v * qR.v)));
  const R EL = (peL + EkL);
  const R ER = (peR + EkR);
  const R ruL = (qL.r * qL.u), ruR = (qR.r * qR.u);
  S4<R> FL{ruL, (ruL * qL.u) + qL.p, (ruL * qL.v), ((qL.p + EL) * qL.u)};
  S4<R> FR{ruR, (ruR * qR.u) + qR.p, (ruR * qR.v), ((qR.p + ER) * qR.u)};
  // primToCons (States.h:19-30) of both states
  const R mvL = (qL.r * qL.v), mvR = (qR.r * qR.v);
  const R uEL = (fv_div_by(fv_half((ruL * ruL) + (mvL * mvL)), qL.r, rL) + peL);
  const R uER = (fv_div_by(fv_half((ruR * ruR) + (mvR * mvR)), qR.r, rR) + peR);
  const R SLSR = (SL * SR);
  const R den = SR - SL;
  const uint32_t rden = fv_recip(den);
  S4<R> FM;
  FM.r = fv_div_by((SR * FL.r) - (SL * FR.r) + (SLSR * (qR.r - qL.r)), den, rden);
  FM.u = fv_div_by((SR * FL.u) - (SL * FR.u) + (SLSR * (ruR - ruL)), den, rden);
  FM.v = fv_div_by((SR * FL.v) - (SL * FR.v) + (SLSR * (mvR - mvL)), den, rden);
  FM.p = fv_div_by((SR * FL.p) - (SL * FR.p) + (SLSR * (uER - uEL)), den, rden);
  const R pM = fv_half(qL.p + qR.p);
  const bool left = fv_ge0(SL);
  const bool right = !left && fv_le0(SR);
  f.r = left ? FL.r : (right ? FR.r : FM.r);
  f.u = left ? FL.u : (right ? FR.u : FM.u);
  f.v = left ? FL.v : (right ? FR.v : FM.v);
  f.p = left ? FL.p : (right ? FR.p : FM.p);
  pout = left ? qL.p : (right ? qR.p : pM);
}

// The same in binary64, its independent products, quotients and sound speeds
// taken in pairs (one call and two chains each).
template <int SOFT = kSoftMul>
__device__ __forceinline__ void riemann_hll(const S4<double> &qL, const S4<double> &qR, S4<double> &f, double &pout,
                                            const Gas<double> &g) {
  const double2 c = softfp::sound2(qL.p, qL.r, qR.p, qR.r, g.gamma);
  const Adder<double> add = g.add;
  const double SL = fv_fmin(add.sub(qL.u, c.x), add.sub(qR.u, c.y));
  const double SR = fv_fmax(add(qL.u, c.x), add(qR.u, c.y));
  double peL, peR, uuL, vvL, uuR, vvR, EkL, EkR, EL, ER;
  fv_div2_by(qL.p, qR.p, g.gm1, g.rgm1, peL, peR);
  mulx2<9, SOFT>(qL.u, qL.u, qL.v, qL.v, uuL, vvL);
  mulx2<9, SOFT>(qR.u, qR.u, qR.v, qR.v, uuR, vvR);
  mulx2<9, SOFT>(fv_half(qL.r), add(uuL, vvL), fv_half(qR.r), add(uuR, vvR), EkL, EkR);
  EL = add(peL, EkL);
  ER = add(peR, EkR);
  S4<double> FL, FR;
  double a, b, mvL, mvR;
  mulx2<9, SOFT>(qL.r, qL.u, qR.r, qR.u, FL.r, FR.r);
  mulx2<9, SOFT>(FL.r, qL.u, FR.r, qR.u, a, b);
  FL.u = add(a, qL.p);
  FR.u = add(b, qR.p);
  mulx2<9, SOFT>(FL.r, qL.v, FR.r, qR.v, FL.v, FR.v);
  mulx2<9, SOFT>(add(qL.p, EL), qL.u, add(qR.p, ER), qR.u, FL.p, FR.p);
  mulx2<9, SOFT>(qL.r, qL.v, qR.r, qR.v, mvL, mvR);
  mulx2<9, SOFT>(FL.r, FL.r, mvL, mvL, uuL, vvL);
  mulx2<9, SOFT>(FR.r, FR.r, mvR, mvR, uuR, vvR);
  double wL, wR;
  fv_quot2(fv_half(add(uuL, vvL)), qL.r, fv_half(add(uuR, vvR)), qR.r, wL, wR);
  const double duE = add.sub(add(wR, peR), add(wL, peL));
  const double SLSR = mulx<10, SOFT>(SL, SR);
  const double den = add.sub(SR, SL);
  const uint32_t rden = fv_recip(den);
  auto average = [&](double fL, double fR, double du) {
    double x, y;
    mulx2<10, SOFT>(SR, fL, SL, fR, x, y);
    return add(add.sub(x, y), mulx<10, SOFT>(SLSR, du));
  };
  S4<double> FM;
  fv_div2_by(average(FL.r, FR.r, add.sub(qR.r, qL.r)), average(FL.u, FR.u, add.sub(FR.r, FL.r)), den, rden, FM.r, FM.u);
  fv_div2_by(average(FL.v, FR.v, add.sub(mvR, mvL)), average(FL.p, FR.p, duE), den, rden, FM.v, FM.p);
  const double pM = fv_half(add(qL.p, qR.p));
  const bool left = fv_ge0(SL);
  const bool right = !left && fv_le0(SR);
  f.r = left ? FL.r : (right ? FR.r : FM.r);
  f.u = left ? FL.u : (right ? FR.u : FM.u);
  f.v = left ? FL.v : (right ? FR.v : FM.v);
  f.p = left ? FL.p : (right ? FR.p : FM.p);
  pout = left ? qL.p : (right ? qR.p : pM);
}

// RiemannSolvers.h:53-128.  The star state is evaluated once, for the side
// the reference would pick if it reaches the star branches (uS > 0 -> left,
// otherwise right), then the final state is chosen in the reference's order.
template <class R>
__device__ __forceinline__ void riemann_hllc(const S4<R> &qL, const S4<R> &qR, S4<R> &f, R &pout, const Gas<R> &g) {
  const R rL = qL.r, uL = qL.u, vL = qL.v, pL = qL.p;
  const R rR = qR.r, uR = qR.u, vR = qR.v, pR = qR.p;
  const R ekL = (fv_half(rL) * ((uL * uL) + (vL * vL)));
  const R EL = ekL + (pL * g.entho);
  const R ekR = (fv_half(rR) * ((uR * uR) + (vR * vR)));
  const R ER = ekR + (pR * g.entho);
  const R cL = sound_speed(qL, g);
  const R cR = sound_speed(qR, g);
  const R cmax = fv_fmax(cL, cR);
  const R SL = fv_fmin(uL, uR) - cmax;
  const R SR = fv_fmax(uL, uR) + cmax;
  const R rcL = (rL * (uL - SL));
  const R rcR = (rR * (SR - uR));
  R uS, pS;
  fv_div2((rcR * uR) + (rcL * uL) + (pL - pR),
          (rcR * pL) + (rcL * pR) + ((rcL * rcR) * (uL - uR)), rcR + rcL, uS, pS);
  const bool sideL = fv_gt0(uS);
  const R rK = sideL ? rL : rR;
  const R uK = sideL ? uL : uR;
  const R pK = sideL ? pL : pR;
  const R EK = sideL ? EL : ER;
  const R SK = sideL ? SL : SR;
  R rS, ES;
  fv_div2((rK * (SK - uK)), ((SK - uK) * EK) - (pK * uK) + (pS * uS), SK - uS, rS, ES);
  // branch order of RiemannSolvers.h:89-112
  const bool bL = fv_gt0(SL);
  const bool bStar = !bL && (sideL || fv_gt0(SR));
  R sr, su, sv, sp, E;
  if (bL) {
    sr = rL; su = uL; sv = vL; sp = pL; E = EL;
  } else if (bStar) {
    sr = rS; su = uS; sv = sideL ? vL : vR; sp = pS; E = ES;
  } else {
    sr = rR; su = uR; sv = vR; sp = pR; E = ER;
  }
  pout = sp;
  f.r = (sr * su);
  f.u = ((sr * su) * su) + sp;
  f.v = (f.r * sv);
  f.p = ((E + sp) * su);
}

// x with its sign changed, a zero as it is: (b - a) from (a - b), whose zero
// is +0 either way.
__device__ __forceinline__ double negated_difference(double x) {
  const uint64_t b = softfp::bits(x);
  return (b & softfp::MAG) == 0 ? x : softfp::from_bits(b ^ softfp::SIGN);
}

// The same in binary64, with fewer operations for the same bits:
//   - max(cL, cR) is the square root of the larger quotient (a correctly
//     rounded square root is monotone; negative and NaN quotients lose to any
//     other in both orders);
//   - S_K - u_K and rho_K (S_K - u_K) of the star state are the negated (left)
//     or the same (right) difference and product of the wave speeds' step;
//   - the total energy is formed for the side the flux is taken from only.
template <int SOFT = kSoftMul>
__device__ __forceinline__ void riemann_hllc(const S4<double> &qL, const S4<double> &qR, S4<double> &f, double &pout,
                                             const Gas<double> &g) {
  const double rL = qL.r, uL = qL.u, vL = qL.v, pL = qL.p;
  const double rR = qR.r, uR = qR.u, vR = qR.v, pR = qR.p;
  const double cmax = softfp::sound_max(pL, rL, pR, rR, g.gamma);
  const double2 um = softfp::minmax_nm(uL, uR);
  const Adder<double> add = g.add;
  const double SL = add.sub(um.x, cmax), SR = add(um.y, cmax);
  const double dL = add.sub(uL, SL), dR = add.sub(SR, uR);
  double rcL, rcR, a, b, c, d;
  mulx2<5, SOFT>(rL, dL, rR, dR, rcL, rcR);
  mulx2<15, SOFT>(rcR, uR, rcL, uL, a, b);
  mulx2<6, SOFT>(rcR, pL, rcL, pR, c, d);
  double uS, pS;
  fv_div2(add(add(a, b), add.sub(pL, pR)),
          add(add(c, d), mulx<6, SOFT>(mulx<6, SOFT>(rcL, rcR), add.sub(uL, uR))), add(rcR, rcL), uS, pS);
  const bool sideL = fv_gt0(uS);
  // branch order of RiemannSolvers.h:89-112
  const bool bL = fv_gt0(SL);
  const bool bStar = !bL && (sideL || fv_gt0(SR));
  const bool left = bL || (bStar && sideL);
  double sr = left ? rL : rR;
  double su = left ? uL : uR;
  const double sv = left ? vL : vR;
  double sp = left ? pL : pR;
  const double SK = left ? SL : SR;
  const double dK = left ? negated_difference(dL) : dR;   // S_K - u_K
  const double rcK = left ? negated_difference(rcL) : rcR;  // rho_K (S_K - u_K)
  double E;
  mulx2<1, SOFT>(su, su, sv, sv, a, b);
  mulx2<2, SOFT>(fv_half(sr), add(a, b), sp, g.entho, c, d);
  E = add(c, d);
  double rS, ES;
  mulx2<7, SOFT>(dK, E, sp, su, a, b);
  fv_div2(rcK, add(add.sub(a, b), mulx<7, SOFT>(pS, uS)), add.sub(SK, uS), rS, ES);
  if (bStar) {
    sr = rS; su = uS; sp = pS; E = ES;
  }
  pout = sp;
  mulx2<8, SOFT>(sr, su, add(E, sp), su, f.r, f.p);
  mulx2<8, SOFT>(f.r, su, f.r, sv, a, f.v);
  f.u = add(a, sp);
}

// RiemannSolvers.h:130-171 (Kokkos::max / min as (a<b)?b:a and (b<a)?b:a).
template <class R>
__device__ __forceinline__ void riemann_fslp(const S4<R> &qL, const S4<R> &qR, S4<R> &f, R &pout, R gdx,
                                             const Gas<R> &g) {
  const R rhoL = qL.r, uL = qL.u, pL = qL.p;
  const R csL = dsqrt(fv_div((g.gamma * pL), rhoL));
  const R rhoR = qR.r, uR = qR.u, pR = qR.p;
  const R csR = dsqrt(fv_div((g.gamma * pR), rhoR));
  const R zL = (rhoL * csL), zR = (rhoR * csR);
  const R ai = (g.fslp_K * (fv_lt(zL, zR) ? zR : zL));
  const R mL = fv_div(fabs(uL), csL), mR = fv_div(fabs(uR), csR);
  const R mx = fv_lt(mL, mR) ? mR : mL;
  const R theta = fv_lt(mx, R(1)) ? mx : R(1);
  const R ustar = fv_half(uR + uL) - ((fv_div(R(0.5), ai)) * (pR - pL - (fv_half(rhoL + rhoR) * gdx)));
  const R Pi = fv_half(pR + pL) - (((fv_half(theta) * ai)) * (uR - uL));
  const bool up = fv_gt0(ustar);
  const R sr = up ? qL.r : qR.r;
  const R su = up ? qL.u : qR.u;
  const R sv = up ? qL.v : qR.v;
  const R sp = up ? qL.p : qR.p;
  const R Ekstar = (fv_half(sr) * ((su * su) + (sv * sv)));
  const R Estar = Ekstar + fv_div_by(sp, g.gm1, g.rgm1);
  const R usr = (ustar * sr);
  f.r = usr;
  f.u = (usr * su) + Pi;
  f.v = (usr * sv);
  f.p = (ustar * (Estar + Pi));
  pout = Pi;
}

// The same in binary64, in pairs as above.
template <int SOFT = kSoftMul>
__device__ __forceinline__ void riemann_fslp(const S4<double> &qL, const S4<double> &qR, S4<double> &f, double &pout,
                                             double gdx, const Gas<double> &g) {
  const double uL = qL.u, pL = qL.p, uR = qR.u, pR = qR.p;
  const double2 c = softfp::sound2(pL, qL.r, pR, qR.r, g.gamma);
  const Adder<double> add = g.add;
  double zL, zR, mL, mR;
  mulx2<14, SOFT>(qL.r, c.x, qR.r, c.y, zL, zR);
  const double ai = mulx<14, SOFT>(g.fslp_K, fv_lt(zL, zR) ? zR : zL);
  fv_quot2(fabs(uL), c.x, fabs(uR), c.y, mL, mR);
  const double mx = fv_lt(mL, mR) ? mR : mL;
  const double theta = fv_lt(mx, 1.0) ? mx : 1.0;
  double a, b, uu, vv, w, z;
  mulx2<14, SOFT>(fv_half(add(qL.r, qR.r)), gdx, fv_half(theta), ai, a, b);
  mulx2<14, SOFT>(fv_div(0.5, ai), add.sub(add.sub(pR, pL), a), b, add.sub(uR, uL), a, b);
  const double ustar = add.sub(fv_half(add(uR, uL)), a);
  const double Pi = add.sub(fv_half(add(pR, pL)), b);
  const bool up = fv_gt0(ustar);
  const double sr = up ? qL.r : qR.r;
  const double su = up ? uL : uR;
  const double sv = up ? qL.v : qR.v;
  const double sp = up ? pL : pR;
  mulx2<14, SOFT>(su, su, sv, sv, uu, vv);
  mulx2<14, SOFT>(fv_half(sr), add(uu, vv), ustar, sr, w, z);
  const double Estar = add(w, fv_div_by(sp, g.gm1, g.rgm1));
  f.r = z;
  mulx2<14, SOFT>(z, su, z, sv, a, f.v);
  f.u = add(a, Pi);
  f.p = mulx<14, SOFT>(ustar, add(Estar, Pi));
  pout = Pi;
}

enum { RS_HLL = 0, RS_HLLC = 1, RS_FSLP = 2 };

// SOFT: which products run on the integer pipes (binary64)
template <int RS, int SOFT = kSoftMul>
__device__ __forceinline__ void riemann(const S4<double> &qL, const S4<double> &qR, S4<double> &f, double &pout,
                                        double gdx, const Gas<double> &g) {
  if constexpr (RS == RS_HLL)
    riemann_hll<SOFT>(qL, qR, f, pout, g);
  else if constexpr (RS == RS_FSLP)
    riemann_fslp<SOFT>(qL, qR, f, pout, gdx, g);
  else
    riemann_hllc<SOFT>(qL, qR, f, pout, g);
}
template <int RS>
__device__ __forceinline__ void riemann(const S4<float> &qL, const S4<float> &qR, S4<float> &f, float &pout, float gdx,
                                        const Gas<float> &g) {
  if constexpr (RS == RS_HLL)
    riemann_hll(qL, qR, f, pout, g);
  else if constexpr (RS == RS_FSLP)
    riemann_fslp(qL, qR, f, pout, gdx, g);
  else
    riemann_hllc(qL, qR, f, pout, g);
}

// Extension (no reference counterpart): primitive-variable MUSCL-Hancock
// half-step qh = q - (dt/2dx) A(q) sx - (dt/2dy) B(q) sy, with ax = 0.5 dt/dx,
// ay = 0.5 dt/dy and sx, sy the full minmod slopes.
template <class R>
__host__ __device__ __forceinline__ S4<R> hancock(const S4<R> &q, const S4<R> &sx, const S4<R> &sy, R ax, R ay,
                                                  R gamma) {
  S4<R> h;
  h.r = q.r - ((ax * ((q.u * sx.r) + (q.r * sx.u))) +
               (ay * ((q.v * sy.r) + (q.r * sy.v))));
  h.u = q.u - ((ax * ((q.u * sx.u) + fv_div(sx.p, q.r))) + (ay * (q.v * sy.u)));
  h.v = q.v - ((ax * (q.u * sx.v)) + (ay * ((q.v * sy.v) + fv_div(sy.p, q.r))));
  h.p = q.p - ((ax * (((gamma * q.p) * sx.u) + (q.u * sx.p))) +
               (ay * (((gamma * q.p) * sy.v) + (q.v * sy.p))));
  return h;
}

template <int SOFT = kSoftMul>
__device__ __forceinline__ S4<double> hancock(const S4<double> &q, const S4<double> &sx, const S4<double> &sy,
                                              double ax, double ay, double gamma, const Adder<double> &add) {
  auto m = [](double a, double b) { return mulx<13, SOFT>(a, b); };
  S4<double> h;
  h.r = add.sub(q.r, add(m(ax, add(m(q.u, sx.r), m(q.r, sx.u))), m(ay, add(m(q.v, sy.r), m(q.r, sy.v)))));
  h.u = add.sub(q.u, add(m(ax, add(m(q.u, sx.u), fv_div(sx.p, q.r))), m(ay, m(q.v, sy.u))));
  h.v = add.sub(q.v, add(m(ax, m(q.u, sx.v)), m(ay, add(m(q.v, sy.v), fv_div(sy.p, q.r)))));
  h.p = add.sub(q.p, add(m(ax, add(m(m(gamma, q.p), sx.u), m(q.u, sx.p))),
                         m(ay, add(m(m(gamma, q.p), sy.v), m(q.v, sy.p)))));
  return h;
}

// ---------------------------------------------------------------- boundaries
// Source (interior index, 0-based) of ghost `k` along one axis of length N,
// for the boundary fills of BoundaryConditions.h:13-71.  Ghost indices are
// interior-relative: -2, -1 on the low side, N, N+1 on the high side.
// Returns the source index and sets *neg when the normal velocity flips
// (reflecting walls).
__host__ __device__ __forceinline__ int ghost_source(int k, int N, int bc, bool *neg) {
  *neg = false;
  if (k < 0) {
    if (bc == 1) {  // reflecting: 2*ibeg - i - 1
      *neg = true;
      return -k - 1;
    }
    if (bc == 2) return k + N;  // periodic
    return 0;                   // absorbing: copy ibeg
  }
  if (bc == 1) {
    *neg = true;
    return 2 * N - k - 1;
  }
  if (bc == 2) return k - N;
  return N - 1;
}

// Ghost positions (interior-relative) whose source is interior index s;
// returns their count (<= 4) in out[], with the matching negation flags.
__host__ __device__ __forceinline__ int ghost_targets(int s, int N, int bc, int out[4], bool neg[4]) {
  const int ks[4] = {-2, -1, N, N + 1};
  int n = 0;
  for (int t = 0; t < 4; ++t) {
    bool ng;
    if (ghost_source(ks[t], N, bc, &ng) == s) {
      out[n] = ks[t];
      neg[n] = ng;
      ++n;
    }
  }
  return n;
}

}  // namespace fv2d
